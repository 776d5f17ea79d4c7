"""The grid-wide one-kernel form of large channels-last BatchNorm layers against the
CPU oracle and the chain of kernels (tuning key 26: 1 takes the form at every size)."""
import numpy as np
import pytest
import torch

from oracle import np_ref
from helpers import bn_inputs, to_numpy, to_torch
from tensorflow_musa_extension_b200 import raw_ops
from test_batchnorm_gpu import EPS, _rms, check_forward, check_grad, launch_ops, tuned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,rows,c", [
    # One row; fewer rows than a CTA has row lanes; fewer than there are row lanes in all
    # (CTAs without a row); one more than that; the narrowest column count; a last
    # column block that is partly empty, at 4, 8 and 16 packs a block.
    ("bfloat16", 1, 32), ("float32", 7, 16), ("float16", 300, 64), ("bfloat16", 9473, 64),
    ("float32", 3001, 20), ("bfloat16", 5000, 40), ("float16", 4099, 96), ("float32", 2500, 160),
    ("bfloat16", 777, 4104), ("float32", 1025, 2052),
    # The rings to the last row, one row more, and several rings.
    ("float32", 113664, 64), ("bfloat16", 227329, 64), ("float16", 500001, 32)])
def test_against_oracle_and_chain(kernel_lib, dtype, rows, c):
    x, s, o, dy = bn_inputs(rows + c, (rows, c), dtype, 1.0, 3.0)
    gen = np.random.default_rng(c)
    est = gen.standard_normal(c).astype(np.float32), (gen.random(c) + 0.5).astype(np.float32)
    want = np_ref.fused_batch_norm(x, s, o, *est, epsilon=EPS, exponential_avg_factor=0.25)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))
    with tuned(kernel_lib, (26, 1)):
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


def test_in_place_streams_and_capture(kernel_lib):
    """Large layers by the rule: y on top of x, two streams at once, and a captured call give the
    bits of a plain call."""
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
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        captured = step()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for out in (*outs, captured):
        for a, b in zip(out, want):
            assert torch.equal(a, b)
