"""The grid-wide one-kernel form of large channels-last BatchNorm layers against the
CPU oracle and the chain of kernels (tuning key 26: 1 takes the form at every size, 4, 8 and 16 in column blocks
of that many packs)."""
import numpy as np
import pytest
import torch

from oracle import np_ref
from helpers import bn_inputs, to_numpy, to_torch
from tensorflow_musa_extension_b200 import raw_ops
from test_batchnorm_gpu import EPS, _rms, check_forward, check_grad, launch_ops, tuned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,rows,c,tx", [
    # One row, and fewer rows than a CTA has row lanes: a column block per CTA (c = 0: as many
    # blocks of 16 packs as SMs).  The scratch holds no other cut of so few rows.
    ("float32", 1, 0, 1), ("bfloat16", 7, 0, 1),
    # Fewer rows than there are row lanes in all (CTAs without a row); one more than that.
    ("float16", 300, 64, 1), ("bfloat16", 9473, 64, 1),
    # A last column block that is partly empty, at 4, 8 and 16 packs a block.
    ("float32", 3001, 20, 4), ("float32", 3001, 20, 8), ("float32", 3001, 20, 16),
    ("bfloat16", 5000, 40, 4), ("bfloat16", 5000, 40, 8), ("bfloat16", 5000, 40, 16),
    ("bfloat16", 777, 4104, 1), ("float32", 1025, 2052, 1),
    # Widths that the rule cuts without a remainder.
    ("float16", 4099, 96, 1), ("float32", 2500, 160, 1),
    # Rows that are not whole lines: split between CTAs, and in one block.
    ("bfloat16", 44001, 200, 1), ("float32", 30011, 100, 1), ("float16", 61001, 136, 1),
    ("bfloat16", 90001, 72, 1),
    # The rings to the last row, one row more, and several rings.
    ("float32", 113664, 64, 1), ("bfloat16", 227329, 64, 1), ("float16", 500001, 32, 1)])
def test_against_oracle_and_chain(kernel_lib, dtype, rows, c, tx):
    if c == 0:
        c = torch.cuda.get_device_properties(0).multi_processor_count * (64 if dtype == "float32" else 128)
    x, s, o, dy = bn_inputs(rows + c, (rows, c), dtype, 1.0, 3.0)
    gen = np.random.default_rng(c)
    est = gen.standard_normal(c).astype(np.float32), (gen.random(c) + 0.5).astype(np.float32)
    want = np_ref.fused_batch_norm(x, s, o, *est, epsilon=EPS, exponential_avg_factor=0.25)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))
    # (Key 25 = 3 shuts the cluster form out: one kernel per pass is this form, more is the chain.)
    with tuned(kernel_lib, (26, tx), (25, 3)):
        before = kernel_lib.MusaKernelsLaunchCount()
        got = launch_ops(kernel_lib, x, s, o, dy, est=est, factor=0.25)
        assert kernel_lib.MusaKernelsLaunchCount() - before == 3
        again = launch_ops(kernel_lib, x, s, o, dy, est=est, factor=0.25, scratch=0x5A)
    with tuned(kernel_lib, (24, -1)):
        chain = launch_ops(kernel_lib, x, s, o, dy, est=est, factor=0.25)
    check_forward(got[0], want, dtype)
    check_grad(got[1], wg, dtype, dx_scale=terms)
    check_grad(got[2], tuple(to_numpy(t) for t in chain[2][:3]), dtype, dx_scale=terms)
    for a, b in zip((t for out in got for t in out), (t for out in again for t in out)):
        assert torch.equal(a, b)
    # Statistics and per-channel sums: fp32 sums in another order.
    for a, b in zip((*got[0][1:], *got[1][1:], *got[2][1:]),
                    (*chain[0][1:], *chain[1][1:], *chain[2][1:])):
        a, b = to_numpy(a).astype(np.float64), to_numpy(b).astype(np.float64)
        assert np.all(np.abs(a - b) <= 1e-5 * np.abs(b) + 1e-5 * max(_rms(b), 1e-12))


@pytest.mark.parametrize("rows,c,kernels", [
    # 16 MiB of inputs and more, narrow and wide: one kernel a pass.
    (262144, 32, (1, 1)), (200000, 64, (1, 1)), (100352, 64, (3, 1)), (25088, 256, (3, 1)),
    (4096, 2048, (1, 1)), (3136, 2048, (2, 1)),
    # One row less than that: the chain.
    (131071, 64, (3, 1)), (65535, 64, (3, 3)),
    # Rows that are not whole lines, up to their limits and one row beyond: 64-byte multiples, others,
    # 17 to 31 packs.
    (1398101, 96, (1, 1)), (1398102, 96, (3, 3)), (67108, 1000, (1, 1)), (67109, 1000, (2, 2)),
    (932067, 72, (1, 1)), (932068, 72, (3, 3)), (209715, 200, (1, 1)), (209716, 200, (3, 3)),
    # Whole lines have no limit.
    (1100000, 128, (1, 1))])
def test_rule(kernel_lib, rows, c, kernels):
    """Kernels of the forward and the gradient by the rule, with the cluster form shut out."""
    x = torch.zeros(rows, c, device="cuda", dtype=torch.bfloat16)
    dy, s, o = torch.zeros_like(x), torch.ones(c, device="cuda"), torch.ones(c, device="cuda")
    e = torch.empty(0, device="cuda")
    with tuned(kernel_lib, (25, 3)):
        counts = [kernel_lib.MusaKernelsLaunchCount()]
        f = raw_ops.FusedBatchNormV3(x, s, o, e, e, epsilon=EPS)
        counts.append(kernel_lib.MusaKernelsLaunchCount())
        raw_ops.FusedBatchNormGradV3(dy, x, s, f.reserve_space_1, f.reserve_space_2, None, EPS)
        counts.append(kernel_lib.MusaKernelsLaunchCount())
    assert (counts[1] - counts[0], counts[2] - counts[1]) == kernels


@pytest.mark.parametrize("rows,c", [(200000, 64), (4096, 2048)])
def test_refused_launch(kernel_lib, rows, c):
    """A context that owns fewer SMs than the device refuses the launch (key 28 stands in for that):
    the chain of kernels takes the call."""
    x, s, o, dy = bn_inputs(9, (rows, c), "bfloat16", 1.0, 3.0)
    with tuned(kernel_lib, (24, -1)):
        before = kernel_lib.MusaKernelsLaunchCount()
        want = launch_ops(kernel_lib, x, s, o, dy)
        kernels = kernel_lib.MusaKernelsLaunchCount() - before
    with tuned(kernel_lib, (28, 1)):
        before = kernel_lib.MusaKernelsLaunchCount()
        got = launch_ops(kernel_lib, x, s, o, dy)
        assert kernel_lib.MusaKernelsLaunchCount() - before == kernels > 3
    for a, b in zip((t for out in got for t in out), (t for out in want for t in out)):
        assert torch.equal(a, b)


def test_in_place_streams_and_capture(kernel_lib):
    """Large layers by the rule: y on top of x, two streams at once, a call beside another stream's
    kernel, and a captured call give the bits of a plain call."""
    e = torch.empty(0, device="cuda")
    x, s, o, dy = (to_torch(a) for a in bn_inputs(1, (60000, 256), "bfloat16", 1.0, 3.0))

    def step():
        f = raw_ops.FusedBatchNormV3(x, s, o, e, e, epsilon=EPS)
        g = raw_ops.FusedBatchNormGradV3(dy, x, s, f.reserve_space_1, f.reserve_space_2, None, EPS)
        return (*f, *g)

    before = kernel_lib.MusaKernelsLaunchCount()
    want = step()
    assert kernel_lib.MusaKernelsLaunchCount() - before == 2
    z = x.clone()
    ws = torch.empty(kernel_lib.BnWorkspaceBytes(60000, 256, 1), dtype=torch.uint8, device="cuda")
    stats = [torch.empty(256, device="cuda") for _ in range(4)]
    assert kernel_lib.LaunchBnFwdTrain_BF16(
        z.data_ptr(), s.data_ptr(), o.data_ptr(), None, None, z.data_ptr(),
        *(t.data_ptr() for t in stats), 60000, 256, 1, EPS, 1.0, ws.data_ptr(), ws.numel(),
        torch.cuda.current_stream().cuda_stream) == 0
    assert torch.equal(z, want[0])
    torch.cuda.synchronize()
    streams, outs = [torch.cuda.Stream() for _ in range(2)], []
    for _ in range(4):
        for st in streams:
            with torch.cuda.stream(st):
                outs.append(step())
    torch.cuda.synchronize()
    with torch.cuda.stream(streams[0]):
        torch.cuda._sleep(2_000_000)   # about a millisecond on one SM
    outs.append(step())
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for out in (*outs, captured):
        for a, b in zip(out, want):
            assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,c,tx,big,small", [
    ("float32", 32, 8, 40, 0), ("bfloat16", 64, 8, 40, 0), ("float32", 64, 16, 40, 0),
    ("float16", 32, 4, 14, -14),
    # Sums of the ones below the normal range of fp32; sums of `big` next to its end.
    ("float32", 32, 8, -100, -140), ("float32", 32, 8, 118, 90)])
def test_partial_sums_add_in_64_bits(kernel_lib, dtype, c, tx, big, small):
    """CTAs whose sums cancel: their rows hold `big`, -`big` and 1 in turn, an fp64 total leaves the
    exact sum of the ones, an fp32 sum of two of them rounds it away.  An infinity and a
    NaN stay in their channels."""
    ctas = torch.cuda.get_device_properties(0).multi_processor_count
    lanes, each = 512 // tx, 4
    big, small = 2.0 ** big, 2.0 ** small
    kind = torch.arange(lanes * each * ctas, device="cuda") // lanes % ctas
    kind = torch.where(kind >= ctas // 3 * 3, 3, kind % 3)
    value = torch.tensor([big, -big, small, 0.0], device="cuda")[kind]
    dy = value[:, None].repeat(1, c).to(getattr(torch, dtype))
    x = torch.ones_like(dy)
    ones, zeros = torch.ones(c, device="cuda"), torch.zeros(c, device="cuda")
    suffix = {"float32": "F32", "float16": "F16", "bfloat16": "BF16"}[dtype]
    want = float(lanes * each * (ctas // 3)) * small

    def grad():
        dx, ds, do = torch.empty_like(x), torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
        ws = torch.empty(kernel_lib.BnWorkspaceBytes(len(x), c, 1), dtype=torch.uint8, device="cuda")
        with tuned(kernel_lib, (26, tx)):
            assert getattr(kernel_lib, "LaunchBnGrad_" + suffix)(
                dy.data_ptr(), x.data_ptr(), ones.data_ptr(), zeros.data_ptr(), ones.data_ptr(),
                dx.data_ptr(), ds.data_ptr(), do.data_ptr(), len(x), c, 1, 0.0, True, ws.data_ptr(),
                ws.numel(), torch.cuda.current_stream().cuda_stream) == 0
        torch.cuda.synchronize()
        return ds, do

    # x - mean and 1 / std are one: both sums are the sum of dy.
    for t in grad():
        assert torch.equal(t, torch.full_like(t, want))
    dy[5, 3], dy[lanes * 7 + 1, 9] = float("inf"), float("nan")
    for t in grad():
        assert t[3] == float("inf") and torch.isnan(t[9])
        t[3] = t[9] = want
        assert torch.equal(t, torch.full_like(t, want))
