"""FusedBatchNorm forward / gradient on the GPU (through the C ABI) against the
CPU oracle and the committed golden vectors."""
import contextlib
import ctypes

import numpy as np
import pytest
import torch

from oracle import c_ref, np_ref
from helpers import NP_BF16, RTOL, assert_close, bn_inputs, np_dtype, to_numpy, to_torch
from tensorflow_musa_extension_b200 import errors, raw_ops

pytestmark = pytest.mark.gpu

EPS = 1e-3


def _rt(dtype):
    return RTOL["f32_bn"] if dtype == "float32" else RTOL["lowp"]


def _rms(a):
    a = np.asarray(a).astype(np.float64)
    return float(np.sqrt(np.mean(a * a))) if a.size else 0.0


def check_forward(got, want, dtype, what=""):
    rt = _rt(dtype)
    assert_close(to_numpy(got.y), want[0], rt, rt * max(_rms(want[0]), 1e-6), what + " y")
    names = ["batch_mean", "batch_variance", "reserve_space_1", "reserve_space_2"]
    for i, n in enumerate(names, start=1):
        # Statistics are fp32 for every x dtype.
        assert_close(to_numpy(got[i]), want[i], RTOL["f32_bn"],
                     RTOL["f32_bn"] * max(_rms(want[i]), 1e-6), what + " " + n)
    assert tuple(got.reserve_space_3.shape) == () and float(got.reserve_space_3) == 0.0


def check_grad(got, want, dtype, what="", dx_scale=None):
    """`dx_scale`: magnitude of the terms dx is a difference of (|dy| * scale *
    inv_std); with a handful of rows dx is what is left after they cancel, so
    the absolute tolerance follows the terms, not the residue."""
    rt = _rt(dtype)
    floor = max(_rms(want[0]), 1e-12) if dx_scale is None else max(dx_scale, _rms(want[0]))
    assert_close(to_numpy(got.x_backprop), want[0], rt, rt * floor, what + " dx")
    srt = RTOL["f32_bn"]
    assert_close(to_numpy(got.scale_backprop), want[1], srt,
                 srt * max(_rms(want[1]), 1e-12), what + " dscale")
    assert_close(to_numpy(got.offset_backprop), want[2], srt,
                 srt * max(_rms(want[2]), 1e-12), what + " doffset")
    c = want[1].shape[0]
    assert tuple(got.reserve_space_4.shape) == (c,) and not to_numpy(got.reserve_space_4).any()
    assert tuple(got.reserve_space_5.shape) == (c,) and not to_numpy(got.reserve_space_5).any()


def run_both(x, scale, offset, dy, fmt):
    tx = to_torch(x)
    fwd = raw_ops.FusedBatchNormV3(tx, to_torch(scale), to_torch(offset),
                                   torch.empty(0, device="cuda"),
                                   torch.empty(0, device="cuda"), epsilon=EPS,
                                   data_format=fmt, is_training=True)
    grad = raw_ops.FusedBatchNormGradV3(to_torch(dy), tx, to_torch(scale),
                                        fwd.reserve_space_1, fwd.reserve_space_2,
                                        fwd.reserve_space_3, epsilon=EPS, data_format=fmt,
                                        is_training=True)
    return fwd, grad


@contextlib.contextmanager
def tuned(lib, *pairs):
    """Tuning keys set for the length of the block; (24, -1) is the chain of kernels
    at every size."""
    old = [(k, lib.MusaKernelsSetTuning(k, v)) for k, v in pairs]
    try:
        yield
    finally:
        for k, v in reversed(old):
            lib.MusaKernelsSetTuning(k, v)


def launch_ops(lib, x, scale, offset, dy, fmt="NHWC", est=None, factor=1.0, scratch=0xA5):
    """Training forward, training gradient and frozen gradient (about the running
    statistics `est` where given, else the batch's) through the C entry points,
    with scratch and outputs that arrive holding arbitrary bytes."""
    tx, tdy, ts, to_ = (to_torch(a) for a in (x, dy, scale, offset))
    c = tx.shape[-1] if fmt == "NHWC" else tx.shape[1]
    outer, inner = (tx.numel() // c, 1) if fmt == "NHWC" else (tx.shape[0], tx[0, 0].numel())
    code, st = raw_ops._DT_CODE[tx.dtype], torch.cuda.current_stream().cuda_stream
    need = max(lib.BnWorkspaceBytes(outer, c, inner), 16)

    def ptrs(ts_):
        return [t.data_ptr() for t in ts_]

    def dirty():
        return torch.full((need,), scratch, dtype=torch.uint8, device="cuda")

    def outputs():
        return [torch.full_like(tx, 999.0)] + [torch.full((c,), 999.0, device="cuda")
                                               for _ in range(4)]

    run = [to_torch(a) for a in est] if est is not None else None
    out, r3, ws = outputs(), torch.full((), 999.0, device="cuda"), dirty()
    assert lib.LaunchBnFwdTrainOp(code, *ptrs((tx, ts, to_)), *(ptrs(run) if run else (None, None)),
                                  *ptrs(out), r3.data_ptr(), outer, c, inner, EPS, factor,
                                  ws.data_ptr(), ws.numel(), st) == 0
    fwd = raw_ops.FusedBatchNormV3Output(*out, r3)
    results = [fwd]
    for training in (True, False):
        stats = (fwd.reserve_space_1, fwd.reserve_space_2) if training or not run else run
        out, ws = outputs(), dirty()
        assert lib.LaunchBnGradOp(code, *ptrs((tdy, tx, ts, *stats)), *ptrs(out), outer, c, inner,
                                  EPS, training, ws.data_ptr(), ws.numel(), st) == 0
        results.append(raw_ops.FusedBatchNormGradV3Output(*out))
    torch.cuda.synchronize()
    return results


def test_golden_vectors(golden, kernel_lib):
    g = golden["bn_torch_cpu"]
    for n in sorted({k.split("/")[0] for k in g.files}):
        fmt = str(g[n + "/format"])
        fwd, grad = run_both(g[n + "/x"], g[n + "/scale"], g[n + "/offset"], g[n + "/dy"], fmt)
        want = (g[n + "/y"], g[n + "/mean"], g[n + "/var_unbiased"], g[n + "/mean"],
                g[n + "/var_pop"])
        check_forward(fwd, want, "float32", n)
        check_grad(grad, (g[n + "/dx"], g[n + "/dscale"], g[n + "/doffset"]), "float32", n)


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("c", [1, 3, 8, 64, 65, 256, 520])
@pytest.mark.parametrize("rows", [2, 31, 32, 33, 1000])
def test_nhwc_shape_matrix(kernel_lib, dtype, c, rows):
    x, s, o, dy = bn_inputs(100 + c + rows, (rows, 1, 1, c), dtype, 1.0, 3.0)
    fwd, grad = run_both(x, s, o, dy, "NHWC")
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS)
    check_forward(fwd, want, dtype)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))
    check_grad(grad, wg, dtype, dx_scale=terms)


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("shape", [(2, 3, 4, 5), (2, 32, 1, 1), (5, 16, 8, 8), (3, 7, 7, 7),
                                   (16, 64, 14, 14), (1, 4, 3, 3),
                                   # planes that are not whole packs, channels in whole groups:
                                   (4, 16, 7, 7), (3, 8, 5, 5), (2, 8, 3, 3), (37, 64, 7, 7),
                                   (2, 8, 17, 19), (3, 16, 31, 33), (70, 24, 3, 5)])
def test_nchw_shapes(kernel_lib, dtype, shape):
    x, s, o, dy = bn_inputs(200 + shape[1], shape, dtype, 0.5, 2.0, channel_axis=1)
    fwd, grad = run_both(x, s, o, dy, "NCHW")
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS, data_format="NCHW")
    check_forward(fwd, want, dtype)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS, "NCHW")
    check_grad(grad, wg, dtype)


def test_keras_2d_batchnorm_shape(kernel_lib):
    # Keras feeds 2-D inputs as [N, 1, 1, C]; a plain 2-D tensor works as well.
    x, s, o, dy = bn_inputs(7, (512, 64), "float32", 0.0, 1.0, dy_std=1.0)
    fwd, grad = run_both(x, s, o, dy, "NHWC")
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS)
    check_forward(fwd, want, "float32")
    check_grad(grad, np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS), "float32")


def test_one_value_per_channel(kernel_lib):
    x = np.array([[[[1.0, -2.0, 3.0, 0.5]]]], np.float32)
    s, o = np.full(4, 2.0, np.float32), np.full(4, 0.25, np.float32)
    fwd, _ = run_both(x, s, o, np.ones_like(x), "NHWC")
    assert_close(to_numpy(fwd.batch_variance), np.zeros(4), 0)      # no 0/0
    assert_close(to_numpy(fwd.reserve_space_2), np.zeros(4), 0)
    assert_close(to_numpy(fwd.y), np.full((1, 1, 1, 4), 0.25), 1e-6)


def test_large_mean_small_spread_is_stable(kernel_lib):
    """mean 1000, std 1: a sum-of-squares variance in fp32 would lose every
    digit; the shifted sums keep rtol 1e-4 on the variance."""
    x, s, o, dy = bn_inputs(9, (64, 8, 8, 32), "float32", 1000.0, 1.0)
    fwd, _ = run_both(x, s, o, dy, "NHWC")
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS)
    assert_close(to_numpy(fwd.reserve_space_2), want[4], 1e-4, 0, "variance")
    assert_close(to_numpy(fwd.reserve_space_1), want[3], 1e-6, 0, "mean")


def test_large_variance_gradient(kernel_lib):
    # The gradient takes a VARIANCE (std 30 here), not an inverse std-dev.
    for dtype in ("float32", "bfloat16"):
        x, s, o, dy = bn_inputs(10, (8, 6, 16, 16), dtype, 3.0, 30.0, dy_std=1.0,
                                channel_axis=1)
        fwd, grad = run_both(x, s, o, dy, "NCHW")
        want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS, data_format="NCHW")
        wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS, "NCHW")
        check_grad(grad, wg, dtype)
        assert np.abs(to_numpy(grad.x_backprop).astype(np.float64)).max() < 1.0


def test_outputs_do_not_depend_on_stale_memory(kernel_lib):
    """Poison the allocator pool with 999, free it, then run the ops: every
    output element must be written by the kernels."""
    x, s, o, dy = bn_inputs(11, (16, 9, 9, 40), "float32", 0.0, 1.0, dy_std=1.0)
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    for _ in range(3):
        junk = [torch.full((16, 9, 9, 40), 999.0, device="cuda") for _ in range(4)]
        junk += [torch.full((40,), 999.0, device="cuda") for _ in range(16)]
        del junk
        fwd, grad = run_both(x, s, o, dy, "NHWC")
        check_forward(fwd, want, "float32")
        check_grad(grad, wg, "float32")


def test_exponential_avg_factor(kernel_lib):
    x, s, o, _ = bn_inputs(12, (4, 5, 5, 24), "float32", 0.5, 2.0)
    rm = np.random.default_rng(1).normal(0, 1, 24).astype(np.float32)
    rv = np.random.default_rng(2).uniform(0.5, 2, 24).astype(np.float32)
    got = raw_ops.FusedBatchNormV3(to_torch(x), to_torch(s), to_torch(o), to_torch(rm),
                                   to_torch(rv), epsilon=EPS, exponential_avg_factor=0.1)
    want = np_ref.fused_batch_norm(x, s, o, rm, rv, EPS, 0.1)
    check_forward(got, want, "float32")
    with pytest.raises(errors.InvalidArgumentError):
        raw_ops.FusedBatchNormV3(to_torch(x), to_torch(s), to_torch(o),
                                 torch.empty(0, device="cuda"), torch.empty(0, device="cuda"),
                                 exponential_avg_factor=0.1)


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("fmt,shape", [("NHWC", (4, 6, 6, 48)), ("NCHW", (4, 12, 6, 6))])
def test_inference_mode(kernel_lib, dtype, fmt, shape):
    ax = 3 if fmt == "NHWC" else 1
    x, s, o, dy = bn_inputs(13, shape, dtype, 0.5, 2.0, dy_std=1.0, channel_axis=ax)
    rng = np.random.default_rng(3)
    mean = rng.normal(0.5, 0.2, shape[ax]).astype(np.float32)
    var = rng.uniform(2, 6, shape[ax]).astype(np.float32)
    got = raw_ops.FusedBatchNormV3(to_torch(x), to_torch(s), to_torch(o), to_torch(mean),
                                   to_torch(var), epsilon=EPS, data_format=fmt,
                                   is_training=False)
    want = np_ref.fused_batch_norm(x, s, o, mean, var, EPS, data_format=fmt,
                                   is_training=False)
    rt = _rt(dtype)
    assert_close(to_numpy(got.y), want[0], rt, rt * _rms(want[0]), "y")
    g = raw_ops.FusedBatchNormGradV3(to_torch(dy), to_torch(x), to_torch(s), to_torch(mean),
                                     to_torch(var), None, epsilon=EPS, data_format=fmt,
                                     is_training=False)
    check_grad(g, np_ref.fused_batch_norm_grad(dy, x, s, mean, var, EPS, fmt, False), dtype)


def test_op_versions_and_errors(kernel_lib):
    x, s, o, dy = bn_inputs(14, (2, 3, 3, 8), "float32", 0.0, 1.0)
    e = torch.empty(0, device="cuda")
    v1 = raw_ops.FusedBatchNorm(to_torch(x), to_torch(s), to_torch(o), e, e, epsilon=EPS)
    v2 = raw_ops.FusedBatchNormV2(to_torch(x), to_torch(s), to_torch(o), e, e, epsilon=EPS)
    assert len(v1) == 5 and len(v2) == 5 and torch.equal(v1.y, v2.y)
    with pytest.raises(errors.InvalidArgumentError, match="scale must have 8 elements"):
        raw_ops.FusedBatchNormV3(to_torch(x), to_torch(s[:4]), to_torch(o), e, e)
    with pytest.raises(errors.InvalidArgumentError, match="float, half, bfloat16"):
        raw_ops.FusedBatchNormV3(to_torch(x).double(), to_torch(s), to_torch(o), e, e)
    with pytest.raises(errors.InvalidArgumentError, match="is_training=False"):
        raw_ops.FusedBatchNormV3(to_torch(x), to_torch(s), to_torch(o), e, e,
                                 is_training=False)
    with pytest.raises(errors.InvalidArgumentError, match="same shape"):
        raw_ops.FusedBatchNormGradV3(to_torch(dy[:1]), to_torch(x), to_torch(s),
                                     v1.reserve_space_1, v1.reserve_space_2)
    with pytest.raises(errors.InvalidArgumentError):
        raw_ops.FusedBatchNormV3(to_torch(x), to_torch(s), to_torch(o), e, e,
                                 data_format="NDHWC")


def test_workspace_contract(kernel_lib):
    x = torch.randn(64, 16, device="cuda")
    outs = [torch.empty(16, device="cuda") for _ in range(4)]
    s = torch.ones(16, device="cuda")
    y = torch.empty_like(x)
    need = kernel_lib.BnWorkspaceBytes(64, 16, 1)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    args = [x.data_ptr(), s.data_ptr(), s.data_ptr(), None, None, y.data_ptr()] + \
        [t.data_ptr() for t in outs] + [64, 16, 1, EPS, 1.0]
    assert kernel_lib.LaunchBnFwdTrain_F32(*args, ws.data_ptr(), need - 1, st) == -2
    assert kernel_lib.LaunchBnFwdTrain_F32(*args, None, need, st) == -2
    assert kernel_lib.LaunchBnFwdTrain_F32(*args, ws.data_ptr(), need, st) == 0
    torch.cuda.synchronize()
    assert torch.allclose(outs[2], x.mean(0), atol=1e-6)


def test_host_buffers_round_trip(kernel_lib):
    x, s, o, dy = bn_inputs(15, (8, 4, 4, 32), "bfloat16", 0.0, 1.0)
    got = raw_ops.FusedBatchNormV3(x, s, o, np.empty(0, np.float32), np.empty(0, np.float32),
                                   epsilon=EPS)
    assert isinstance(got.y, np.ndarray) and got.y.dtype == NP_BF16
    check_forward(got, np_ref.fused_batch_norm(x, s, o, epsilon=EPS), "bfloat16")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,c", [(2, 8), (33, 64), (5000, 256), (70000, 128), (3000, 2048),
                                    (9000, 520), (1200, 4104)])
def test_dirty_workspace_and_launch_shapes(kernel_lib, dtype, rows, c):
    """The workspace arrives with arbitrary contents (a framework hands out
    temporary memory as it finds it); the same call twice gives the same bits;
    column blocks as wide as the row, or 8 packs wide (both passes), the 256-thread finalize
    kernel and the other row map (contiguous ranges / interleaved tiles) agree
    with the default shapes to rounding."""
    x, s, o, dy = bn_inputs(300 + rows, (rows, c), dtype, 1.0, 3.0)
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))

    def run(*pairs, scratch=0xA5):
        with tuned(kernel_lib, *pairs):
            return launch_ops(kernel_lib, x, s, o, dy, scratch=scratch)

    chain = (24, -1)    # the keys below are the chain's
    for pairs in ((), (chain,)):
        fwd, grad, _ = run(*pairs)
        fwd2, grad2, _ = run(*pairs, scratch=0x5A)
        for a, b in zip(list(fwd)[:5] + list(grad)[:3], list(fwd2)[:5] + list(grad2)[:3]):
            assert torch.equal(a, b)
        check_forward(fwd, want, dtype)
        check_grad(grad, wg, dtype, dx_scale=terms)
    for key, value in ((14, 256), (14, 8), (19, 32), (22, 0), (22, 8),
                       (21, 1 - kernel_lib.MusaKernelsGetTuning(21)),
                       (23, 1 - kernel_lib.MusaKernelsGetTuning(23))):
        fwd3, grad3, _ = run(chain, (key, value))
        check_forward(fwd3, want, dtype)
        check_grad(grad3, wg, dtype, dx_scale=terms)
        assert_close(to_numpy(fwd.batch_mean), to_numpy(fwd3.batch_mean), 1e-5, 1e-6)
        assert_close(to_numpy(fwd.reserve_space_2), to_numpy(fwd3.reserve_space_2), 1e-5, 1e-7)


def test_bessel_and_inv_std_launchers(kernel_lib):
    """The two fix-up launchers kept from the reference boundary
    (musa_ext/kernels/nn/musa_fused_batchnorm_kernel.mu:38-56)."""
    rng = np.random.default_rng(5)
    st = torch.cuda.current_stream().cuda_stream
    for count in (1, 7, 256, 1000):
        var = rng.uniform(0.0, 4.0, count).astype(np.float32)
        data = to_torch(var.copy())
        factor = np.float32(50176.0 / 50175.0)
        kernel_lib.LaunchBesselCorrection(data.data_ptr(), float(factor), count, st)
        assert np.array_equal(to_numpy(data), var * factor)          # one fp32 multiply
        inv = torch.empty(count, device="cuda")
        kernel_lib.LaunchVarianceToInvStd(to_torch(var).data_ptr(), inv.data_ptr(), EPS,
                                          count, st)
        want = 1.0 / np.sqrt(var.astype(np.float64) + np.float64(np.float32(EPS)))
        assert_close(to_numpy(inv), want, 1e-6, 0)
    keep = torch.full((4,), 3.0, device="cuda")
    kernel_lib.LaunchBesselCorrection(keep.data_ptr(), 2.0, 0, st)      # empty: untouched
    torch.cuda.synchronize()
    assert float(keep.sum()) == 12.0


# ------------------------------------------------ cross-replica (split) API --

def _split_forward_and_grad(lib, x, dy, scale, offset, parts, fused=False):
    """Runs the SyncBN halves on `parts` row blocks as if they were replicas
    and sums the per-replica sums on the host side of the all-reduce.
    fused="moments": the replicas' [mean, M2, count] vectors are gathered and
    merged instead (LaunchBnStatsMoments / MergeMoments / ApplyFromMoments)."""
    if fused == "moments":
        return _split_with_moments(lib, x, dy, scale, offset, parts)
    dt = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[x.dtype]
    rows, c = x.shape
    st = torch.cuda.current_stream().cuda_stream
    bounds = np.linspace(0, rows, parts + 1).astype(int)
    need = lib.BnWorkspaceBytes(rows, c, 1)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
    total = torch.zeros(2 * c + 1, device="cuda")
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        sums = torch.zeros(2 * c + 1, device="cuda")
        fn = lib.LaunchBnStatsSumsCount if fused else lib.LaunchBnStatsSums
        rc = fn(dt, x[lo:hi].data_ptr(), sums.data_ptr(), int(hi - lo), c, 1,
                ws.data_ptr(), ws.numel(), st)
        assert rc == 0
        total += sums
    if fused:   # the row count rode along with the sums
        assert float(total[2 * c]) == float(rows)
    bm, bv, sm, sv = (torch.empty(c, device="cuda") for _ in range(4))
    if not fused:
        assert lib.LaunchBnFinalizeFromSums(total.data_ptr(), float(rows), None, None,
                                            bm.data_ptr(), bv.data_ptr(), sm.data_ptr(),
                                            sv.data_ptr(), c, 1.0, st) == 0
    y = torch.empty_like(x)
    gtotal = torch.zeros(2 * c, device="cuda")
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        if fused:
            assert lib.LaunchBnApplyFromSums(
                dt, x[lo:hi].data_ptr(), scale.data_ptr(), offset.data_ptr(),
                total.data_ptr(), float(rows), None, None, 1.0, y[lo:hi].data_ptr(),
                bm.data_ptr(), bv.data_ptr(), sm.data_ptr(), sv.data_ptr(), int(hi - lo),
                c, 1, EPS, st) == 0
        else:
            assert lib.LaunchBnApply(dt, x[lo:hi].data_ptr(), scale.data_ptr(),
                                     offset.data_ptr(), sm.data_ptr(), sv.data_ptr(),
                                     y[lo:hi].data_ptr(), int(hi - lo), c, 1, EPS, st) == 0
        sums = torch.empty(2 * c, device="cuda")
        assert lib.LaunchBnGradStatsSums(dt, dy[lo:hi].data_ptr(), x[lo:hi].data_ptr(),
                                         sm.data_ptr(), sums.data_ptr(), int(hi - lo), c, 1,
                                         ws.data_ptr(), ws.numel(), st) == 0
        gtotal += sums
    dx = torch.empty_like(x)
    dscale, doffset = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        assert lib.LaunchBnGradApplyFromSums(
            dt, dy[lo:hi].data_ptr(), x[lo:hi].data_ptr(), scale.data_ptr(), sm.data_ptr(),
            sv.data_ptr(), gtotal.data_ptr(), float(rows), dx[lo:hi].data_ptr(),
            dscale.data_ptr(), doffset.data_ptr(), int(hi - lo), c, 1, EPS, st) == 0
    return y, bm, bv, sm, sv, dx, dscale, doffset


def _split_with_moments(lib, x, dy, scale, offset, parts):
    dt = {torch.float32: 0, torch.float16: 1, torch.bfloat16: 2}[x.dtype]
    rows, c = x.shape
    st = torch.cuda.current_stream().cuda_stream
    bounds = np.linspace(0, rows, parts + 1).astype(int)
    need = lib.BnWorkspaceBytes(rows, c, 1)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
    gathered = torch.zeros(parts, 2 * c + 1, device="cuda")
    for q, (lo, hi) in enumerate(zip(bounds[:-1], bounds[1:])):
        assert lib.LaunchBnStatsMoments(dt, x[lo:hi].data_ptr(), gathered[q].data_ptr(),
                                        int(hi - lo), c, 1, ws.data_ptr(), ws.numel(), st) == 0
    merged = torch.empty(2 * c + 1, device="cuda")
    assert lib.LaunchBnMergeMoments(gathered.data_ptr(), parts, c, merged.data_ptr(), st) == 0
    assert float(merged[2 * c]) == float(rows)
    bm, bv, sm, sv = (torch.empty(c, device="cuda") for _ in range(4))
    y = torch.empty_like(x)
    gtotal = torch.zeros(2 * c, device="cuda")
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        assert lib.LaunchBnApplyFromMoments(
            dt, x[lo:hi].data_ptr(), scale.data_ptr(), offset.data_ptr(), merged.data_ptr(),
            float(rows), None, None, 1.0, y[lo:hi].data_ptr(), bm.data_ptr(), bv.data_ptr(),
            sm.data_ptr(), sv.data_ptr(), int(hi - lo), c, 1, EPS, st) == 0
        sums = torch.empty(2 * c, device="cuda")
        assert lib.LaunchBnGradStatsSums(dt, dy[lo:hi].data_ptr(), x[lo:hi].data_ptr(),
                                         sm.data_ptr(), sums.data_ptr(), int(hi - lo), c, 1,
                                         ws.data_ptr(), ws.numel(), st) == 0
        gtotal += sums
    dx = torch.empty_like(x)
    dscale, doffset = torch.empty(c, device="cuda"), torch.empty(c, device="cuda")
    for lo, hi in zip(bounds[:-1], bounds[1:]):
        assert lib.LaunchBnGradApplyFromSums(
            dt, dy[lo:hi].data_ptr(), x[lo:hi].data_ptr(), scale.data_ptr(), sm.data_ptr(),
            sv.data_ptr(), gtotal.data_ptr(), float(rows), dx[lo:hi].data_ptr(),
            dscale.data_ptr(), doffset.data_ptr(), int(hi - lo), c, 1, EPS, st) == 0
    return y, bm, bv, sm, sv, dx, dscale, doffset


@pytest.mark.parametrize("layout", ["NHWC", "NCHW"])
def test_merged_moments_keep_the_variance_when_the_mean_is_large(kernel_lib, layout):
    """|mean| / std = 1000, four replicas: the statistics of the merged
    moments meet the tolerance of the single-GPU op (raw fp32 [sum x, sum x^2]
    would have no correct digit left in the variance)."""
    rng = np.random.default_rng(77)
    rows, c = 4096, 64
    x = (rng.standard_normal((rows, c)) + 1e3).astype(np.float32)
    want = np_ref.fused_batch_norm(x, np.ones(c, np.float32), np.zeros(c, np.float32),
                                   epsilon=EPS)
    st = torch.cuda.current_stream().cuda_stream
    parts = 4
    gathered = torch.zeros(parts, 2 * c + 1, device="cuda")
    per = rows // parts
    for q in range(parts):
        blk = x[q * per:(q + 1) * per]
        if layout == "NCHW":     # [n, C, 4] view of the same values per channel
            t = to_torch(np.ascontiguousarray(blk.reshape(per // 4, 4, c).transpose(0, 2, 1)))
            outer, inner = per // 4, 4
        else:
            t = to_torch(blk)
            outer, inner = per, 1
        need = kernel_lib.BnWorkspaceBytes(outer, c, inner)
        ws = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
        assert kernel_lib.LaunchBnStatsMoments(0, t.data_ptr(), gathered[q].data_ptr(), outer,
                                               c, inner, ws.data_ptr(), ws.numel(), st) == 0
    merged = torch.empty(2 * c + 1, device="cuda")
    assert kernel_lib.LaunchBnMergeMoments(gathered.data_ptr(), parts, c, merged.data_ptr(),
                                           st) == 0
    m = to_numpy(merged)
    assert m[2 * c] == rows
    assert_close(m[:c], want[3], 1e-6, 0, "mean")
    assert_close(m[c:2 * c] / rows, want[4], 1e-4, 0, "variance")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("parts", [1, 2, 8])
@pytest.mark.parametrize("fused", [False, True, "moments"])
def test_split_api_equals_global_batchnorm(kernel_lib, dtype, parts, fused):
    x, s, o, dy = bn_inputs(16, (4096, 64), dtype, 0.0, 1.0)
    got = _split_forward_and_grad(kernel_lib, to_torch(x), to_torch(dy), to_torch(s),
                                  to_torch(o), parts, fused)
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    rt = _rt(dtype)
    assert_close(to_numpy(got[0]), want[0], rt, rt * _rms(want[0]), "y")
    for i in range(1, 5):
        assert_close(to_numpy(got[i]), want[i], 1e-4, 1e-4 * max(_rms(want[i]), 1e-6))
    assert_close(to_numpy(got[5]), wg[0], rt, rt * _rms(wg[0]), "dx")
    assert_close(to_numpy(got[6]), wg[1], 1e-4, 1e-4 * _rms(wg[1]), "dscale")
    assert_close(to_numpy(got[7]), wg[2], 1e-4, 1e-4 * _rms(wg[2]), "doffset")


def test_empty_replica_contributes_zero_sums(kernel_lib):
    sums = torch.full((16,), 7.0, device="cuda")
    st = torch.cuda.current_stream().cuda_stream
    assert kernel_lib.LaunchBnStatsSums(0, None, sums.data_ptr(), 0, 8, 1, None, 0, st) == 0
    torch.cuda.synchronize()
    assert not sums.any()


# ------------------------------------------------------- benchmark shapes --

def test_config1_fp32_full_size(kernel_lib):
    x, s, o, dy = bn_inputs(0, (32, 56, 56, 64), "float32", 0.5, 2.0)
    fwd, grad = run_both(x, s, o, dy, "NHWC")
    x2 = x.reshape(-1, 64)
    want = c_ref.bn_fwd_train(x2, s, o, EPS)
    check_forward(fwd, (want[0].reshape(x.shape),) + tuple(want[1:]), "float32")
    wg = c_ref.bn_grad(dy.reshape(-1, 64), x2, s, want[3], want[4], EPS)
    check_grad(grad, (wg[0].reshape(x.shape), wg[1], wg[2]), "float32")


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
def test_config2_16bit_full_size(kernel_lib, dtype):
    x, s, o, dy = bn_inputs(1, (256, 28, 28, 256), dtype, 1.0, 3.0)
    fwd, grad = run_both(x, s, o, dy, "NHWC")
    x2 = x.reshape(-1, 256)
    want = c_ref.bn_fwd_train(x2, s, o, EPS)
    check_forward(fwd, (want[0].reshape(x.shape),) + tuple(want[1:]), dtype)
    wg = c_ref.bn_grad(dy.reshape(-1, 256), x2, s, want[3], want[4], EPS)
    check_grad(grad, (wg[0].reshape(x.shape), wg[1], wg[2]), dtype)
    # Size-independent properties: y has zero mean / unit variance per channel
    # before scale and offset; dx sums to zero per channel.
    y = fwd.y.float().reshape(-1, 256)
    z = (y - to_torch(o)) / to_torch(s)
    assert float(z.mean(0).abs().max()) < 5e-3
    assert float((z.var(0, unbiased=False) - 1).abs().max()) < 2e-2
    # dx sums to zero per channel in exact arithmetic; after rounding dx to 16
    # bits the sum is whatever the rounding leaves, which the oracle shares.
    dxs = grad.x_backprop.double().reshape(-1, 256).sum(0).cpu().numpy()
    want_dxs = wg[0].astype(np.float64).sum(0)
    assert float(np.abs(dxs - want_dxs).max()) < 5e-2


@pytest.mark.parametrize("fold", [0, 2, 4, 8])
@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("rows,c", [(2, 8), (33, 64), (1000, 520), (5000, 256), (70000, 128),
                                    (3000, 2048), (20000, 64), (1200, 4104), (40000, 32)])
def test_chain_without_finalize_kernel(kernel_lib, fold, dtype, rows, c):
    """The element-wise kernel adds the partial rows itself when few enough are
    left (tuning key 13: here any number that fits its shared memory), with
    and without clusters of the statistics kernel adding theirs on chip first
    (key 5) - no finalize kernel: training forward with running statistics,
    training gradient and inference gradient against the oracle, from a
    workspace with arbitrary contents, the same bits on a second call, and the
    same numbers (to rounding) as the chain with the finalize kernel."""
    x, s, o, dy = bn_inputs(900 + rows + c, (rows, c), dtype, 1.0, 3.0)
    gen = np.random.default_rng(rows + c)
    rm = gen.standard_normal(c).astype(np.float32)
    rv = (gen.random(c) + 0.5).astype(np.float32)
    want = np_ref.fused_batch_norm(x, s, o, rm, rv, epsilon=EPS, exponential_avg_factor=0.25)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    wi = np_ref.fused_batch_norm_grad(dy, x, s, rm, rv, EPS, is_training=False)
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))

    def run(*pairs, scratch=0x5A):
        with tuned(kernel_lib, (24, -1), *pairs):
            return launch_ops(kernel_lib, x, s, o, dy, est=(rm, rv), factor=0.25, scratch=scratch)

    base = run((13, 0))
    got = run((13, 4096), (5, fold))
    again = run((13, 4096), (5, fold), scratch=0xA5)
    check_forward(got[0], want, dtype)
    check_grad(got[1], wg, dtype, dx_scale=terms)
    check_grad(got[2], wi, dtype, dx_scale=terms)
    for a, b in zip(list(got[0])[:5] + list(got[1])[:3] + list(got[2])[:3],
                    list(again[0])[:5] + list(again[1])[:3] + list(again[2])[:3]):
        assert torch.equal(a, b)
    for a, b in zip(list(got[0])[1:5] + list(got[1])[1:3], list(base[0])[1:5] + list(base[1])[1:3]):
        a, b = to_numpy(a).astype(np.float64), to_numpy(b).astype(np.float64)
        assert np.all(np.abs(a - b) <= 1e-5 * np.abs(b) + 1e-5 * max(_rms(b), 1e-12))


def test_tracing_counts_the_kernels_of_a_chain(kernel_lib):
    """The tracing counters tell how many kernels a launcher call made: three
    for a BatchNorm pass (statistics, finalize, element-wise), two when the
    element-wise kernel adds the partial rows itself (few rows are left: a
    wide or a small layer)."""
    from tensorflow_musa_extension_b200 import _capi
    was = kernel_lib.MusaKernelsTraceEnable(1)
    try:
        for rows, c, want in ((200000, 64, 3), (4096, 2048, 2)):
            x, s_, o, dy = bn_inputs(5, (rows, c), "bfloat16", 0.0, 1.0)
            with tuned(kernel_lib, (24, -1)):
                run_both(x, s_, o, dy, "NHWC")          # per-device set-up happens here
                torch.cuda.synchronize()
                kernel_lib.MusaKernelsTraceReset()
                launched = kernel_lib.MusaKernelsLaunchCount()
                run_both(x, s_, o, dy, "NHWC")
                torch.cuda.synchronize()
            assert kernel_lib.MusaKernelsLaunchCount() - launched == 2 * want
            snap = _capi.trace_snapshot(kernel_lib)
            assert snap["LaunchBnFwdTrain"]["calls"] == 1
            assert snap["LaunchBnFwdTrain"]["kernels"] == want
            assert snap["LaunchBnGrad"]["kernels"] == want
    finally:
        kernel_lib.MusaKernelsTraceEnable(was)
        kernel_lib.MusaKernelsTraceReset()


@pytest.mark.parametrize("rows,c", [(5000, 256), (4096, 2048), (300, 64)])
def test_forward_in_place(kernel_lib, rows, c):
    """y may be x itself (every element is read and written by one thread):
    the same bits as the out-of-place call, statistics included - also for the
    layers whose element-wise kernel would add the partial rows itself."""
    x, s_, o, _ = bn_inputs(77 + c, (rows, c), "bfloat16", 1.0, 3.0)
    st = torch.cuda.current_stream().cuda_stream
    need = kernel_lib.BnWorkspaceBytes(rows, c, 1)
    ws = torch.empty(max(need, 16), dtype=torch.uint8, device="cuda")
    ts, to_ = to_torch(s_), to_torch(o)

    def run(tx, ty):
        stats = [torch.empty(c, device="cuda") for _ in range(4)]
        assert kernel_lib.LaunchBnFwdTrain_BF16(
            tx.data_ptr(), ts.data_ptr(), to_.data_ptr(), None, None, ty.data_ptr(),
            *[t.data_ptr() for t in stats], rows, c, 1, EPS, 1.0, ws.data_ptr(), ws.numel(),
            st) == 0
        torch.cuda.synchronize()
        return stats

    tx = to_torch(x)
    ty = torch.empty_like(tx)
    want = run(tx, ty)
    tz = to_torch(x)
    got = run(tz, tz)
    assert torch.equal(tz, ty)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,shape,layout", [
    ("bfloat16", (3, 5, 7, 64), "NHWC"),     # whole packs, one column block
    ("float32", (2, 3, 3, 2056), "NHWC"),    # many column blocks, the last one partly filled
    ("float16", (4, 3, 5, 37), "NHWC"),      # single elements
    ("bfloat16", (3, 16, 7, 7), "NCHW"),     # channel groups
    ("float16", (2, 12, 8, 8), "NCHW"),      # whole planes
    ("float32", (1, 1, 3, 5), "NCHW"),       # one channel
])
def test_outputs_beside_the_statistics(kernel_lib, dtype, shape, layout):
    """The zeros (reserve_space_3 .. 5) and the passed-through statistics of the
    inference form come from the op's own kernels, in every geometry and from
    buffers with arbitrary contents."""
    c = shape[-1] if layout == "NHWC" else shape[1]
    x, s_, o, dy = bn_inputs(41, shape, dtype, 0.5, 2.0)
    gen = np.random.default_rng(c)
    rm = to_torch(gen.standard_normal(c).astype(np.float32))
    rv = to_torch((gen.random(c) + 0.5).astype(np.float32))
    tx, tdy, ts, to_ = to_torch(x), to_torch(dy), to_torch(s_), to_torch(o)
    outer, inner = (tx.numel() // c, 1) if layout == "NHWC" else (shape[0], shape[2] * shape[3])
    code = raw_ops._DT_CODE[tx.dtype]
    st = torch.cuda.current_stream().cuda_stream
    need = kernel_lib.BnWorkspaceBytes(outer, c, inner)
    ws = torch.full((max(need, 16),), 0x5A, dtype=torch.uint8, device="cuda")

    def fresh(n):
        return [torch.full((c,), float("nan"), device="cuda") for _ in range(n)]

    def ptrs(ts_):
        return [t.data_ptr() for t in ts_]

    def run_all():
        y, stats, r3 = torch.empty_like(tx), fresh(4), torch.full((), float("nan"), device="cuda")
        assert kernel_lib.LaunchBnFwdInferOp(
            code, *ptrs((tx, ts, to_, rm, rv, y, *stats, r3)), outer, c, inner, EPS, st) == 0
        for got, want in zip(stats, (rm, rv, rm, rv)):
            assert torch.equal(got, want)
        assert float(r3) == 0.0
        stats, r3 = fresh(4), torch.full((), float("nan"), device="cuda")
        assert kernel_lib.LaunchBnFwdTrainOp(
            code, *ptrs((tx, ts, to_)), None, None, *ptrs((y, *stats, r3)), outer, c, inner, EPS, 1.0,
            ws.data_ptr(), ws.numel(), st) == 0
        assert float(r3) == 0.0 and all(bool(torch.isfinite(t).all()) for t in stats)
        for training in (True, False):
            dx, outs = torch.empty_like(tx), fresh(4)
            assert kernel_lib.LaunchBnGradOp(
                code, *ptrs((tdy, tx, ts, stats[2], stats[3], dx, *outs)), outer, c, inner, EPS,
                training, ws.data_ptr(), ws.numel(), st) == 0
            assert all(bool(torch.isfinite(t).all()) for t in outs[:2])
            assert not outs[2].any() and not outs[3].any()

    for pairs in ((), ((24, -1),)):      # by rule (mostly one kernel), and the chain
        with tuned(kernel_lib, *pairs):
            run_all()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("cluster", [0, 1, 2, 8, 16])
@pytest.mark.parametrize("shape,layout", [
    ((1, 8), "NHWC"), ((2, 16), "NHWC"), ((511, 24), "NHWC"), ((1000, 520), "NHWC"),
    ((6272, 64), "NHWC"), ((12800, 16), "NHWC"), ((12801, 16), "NHWC"),
    ((1, 16, 7, 7), "NCHW"), ((3, 8, 4, 4), "NCHW"), ((37, 24, 3, 5), "NCHW"),
    ((64, 32, 14, 14), "NCHW"), ((20, 2, 28, 28), "NCHW"), ((6, 2, 56, 56), "NCHW"), ((3, 5, 8, 11), "NCHW"), ((250, 8, 7, 7), "NCHW"),
])
def test_one_kernel_form(kernel_lib, dtype, cluster, shape, layout):
    """The one-kernel form (inputs held in shared memory, sums met over a
    cluster) against the oracle and against the chain of kernels, at the edges
    of its cuts: a single row, partly filled column blocks, CTAs without rows,
    the last row slot; key 25 forces the cluster size (sizes that cannot hold
    the layer fall back to the chain), key 24 = -1 turns the form off."""
    c = shape[-1] if layout == "NHWC" else shape[1]
    axis = -1 if layout == "NHWC" else 1
    x, s, o, dy = bn_inputs(70 + c, shape, dtype, 1.0, 3.0, channel_axis=axis)
    gen = np.random.default_rng(c)
    rm = gen.standard_normal(c).astype(np.float32)
    rv = (gen.random(c) + 0.5).astype(np.float32)
    want = np_ref.fused_batch_norm(x, s, o, rm, rv, epsilon=EPS, exponential_avg_factor=0.25,
                                   data_format=layout)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS, layout)
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))

    def run():
        tx = to_torch(x)
        fwd = raw_ops.FusedBatchNormV3(tx, to_torch(s), to_torch(o), to_torch(rm), to_torch(rv),
                                       epsilon=EPS, exponential_avg_factor=0.25,
                                       data_format=layout)
        args = (to_torch(dy), tx, to_torch(s), fwd.reserve_space_1, fwd.reserve_space_2, None,
                EPS, layout)
        grad = raw_ops.FusedBatchNormGradV3(*args)
        frozen = raw_ops.FusedBatchNormGradV3(*args, is_training=False)
        torch.cuda.synchronize()
        return fwd, grad, frozen

    old = kernel_lib.MusaKernelsSetTuning(25, cluster)
    try:
        before = kernel_lib.MusaKernelsLaunchCount()
        fwd, grad, frozen = run()
        launches = kernel_lib.MusaKernelsLaunchCount() - before
        again = run()
    finally:
        kernel_lib.MusaKernelsSetTuning(25, old)
    if cluster == 0:
        assert launches == 3     # every shape of this list takes the form
    off = kernel_lib.MusaKernelsSetTuning(24, -1)
    try:
        chain = run()
    finally:
        kernel_lib.MusaKernelsSetTuning(24, off)
    check_forward(fwd, want, dtype)
    check_grad(grad, wg, dtype, dx_scale=terms)
    for a, b in zip((*fwd, *grad, *frozen), (t for out in again for t in out)):
        assert torch.equal(a, b)
    for a, b in zip((*fwd[1:], *grad[1:], *frozen[1:]),
                    (t for out in chain for t in out[1:])):
        a, b = to_numpy(a).astype(np.float64), to_numpy(b).astype(np.float64)
        assert np.all(np.abs(a - b) <= 1e-5 * np.abs(b) + 1e-5 * max(_rms(b), 1e-12))
    check_grad(frozen, tuple(to_numpy(t) for t in chain[2][:3]), dtype, dx_scale=terms)


@pytest.mark.parametrize("dtype", ["float32", "float16", "bfloat16"])
@pytest.mark.parametrize("rows,c", [(8, 1), (9, 37), (15, 3), (4099, 100), (7001, 6), (2051, 1001),
                                    (300, 4099), (70001, 5), (9, 70001)])
def test_rows_that_are_not_whole_packs(kernel_lib, dtype, rows, c):
    """Odd channel counts: several rows together are whole packs and take the
    vector kernels, the rows left over are added by the finalize kernel and
    written element by element.  Against the oracle, and against the element
    kernels (the same values off a 16-byte boundary): training forward with
    running statistics, inference, both gradients, the raw sums of the
    cross-replica form."""
    x, s, o, dy = bn_inputs(17 + c, (rows, c), dtype, 1.0, 3.0)
    gen = np.random.default_rng(c)
    rm = gen.standard_normal(c).astype(np.float32)
    rv = (gen.random(c) + 0.5).astype(np.float32)
    want = np_ref.fused_batch_norm(x, s, o, rm, rv, epsilon=EPS, exponential_avg_factor=0.25)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))
    ts, to_, tm, tv = to_torch(s), to_torch(o), to_torch(rm), to_torch(rv)
    st = torch.cuda.current_stream().cuda_stream

    def run(tx, tdy):
        fwd = raw_ops.FusedBatchNormV3(tx, ts, to_, tm, tv, epsilon=EPS,
                                       exponential_avg_factor=0.25)
        infer = raw_ops.FusedBatchNormV3(tx, ts, to_, tm, tv, epsilon=EPS, is_training=False)
        args = (tdy, tx, ts, fwd.reserve_space_1, fwd.reserve_space_2, None, EPS)
        grad = raw_ops.FusedBatchNormGradV3(*args)
        frozen = raw_ops.FusedBatchNormGradV3(*args, is_training=False)
        sums = torch.empty(2 * c, device="cuda")
        ws = torch.empty(max(kernel_lib.BnWorkspaceBytes(rows, c, 1), 16), dtype=torch.uint8,
                         device="cuda")
        assert kernel_lib.LaunchBnGradStatsSums(
            raw_ops._DT_CODE[tx.dtype], tdy.data_ptr(), tx.data_ptr(),
            fwd.reserve_space_1.data_ptr(), sums.data_ptr(), rows, c, 1, ws.data_ptr(),
            ws.numel(), st) == 0
        torch.cuda.synchronize()
        return fwd, infer, grad, frozen, (sums,)

    def unaligned(a):
        t = to_torch(a)
        return torch.cat((t.new_zeros(1), t.reshape(-1)))[1:].view(t.shape)

    old = kernel_lib.MusaKernelsSetTuning(24, -1)   # the chain, whatever the size
    try:
        got = run(to_torch(x), to_torch(dy))
        again = run(to_torch(x), to_torch(dy))
        base = run(unaligned(x), unaligned(dy))
    finally:
        kernel_lib.MusaKernelsSetTuning(24, old)
    check_forward(got[0], want, dtype)
    check_grad(got[2], wg, dtype, dx_scale=terms)
    for out, same in zip(got, again):
        for a, b in zip(out, same):
            assert torch.equal(a, b)
    for i, (out, ref) in enumerate(zip(got, base)):
        for k, (a, b) in enumerate(zip(out, ref)):
            a, b = to_numpy(a).astype(np.float64), to_numpy(b).astype(np.float64)
            # Element-wise results: one rounding of T on statistics that agree
            # to 1e-5; the others are fp32 sums in another order.
            rt = _rt(dtype) if k == 0 and i < 4 else 1e-5
            floor = max(_rms(b), terms if i in (2, 3) and k == 0 else 1e-12)
            assert np.all(np.abs(a - b) <= rt * np.abs(b) + rt * floor), (i, k)


@pytest.mark.parametrize("dtype,rows,c,one_kernel", [
    ("bfloat16", 49152, 64, True),      # 64 CTAs of 12 slots
    ("bfloat16", 49153, 64, False),     # 13 slots, or 32 CTAs of 25
    ("float16", 51200, 64, False), ("bfloat16", 50176, 32, False), ("float32", 50176, 32, False),
    ("bfloat16", 49153, 40, False), ("float16", 50176, 72, False),
    ("float32", 50176, 48, True)])      # 48 CTAs of 25
def test_long_narrow_layers(kernel_lib, dtype, rows, c, one_kernel):
    """A forward of few channels and many rows leaves the one-kernel form where its
    cuts are too few CTAs, whichever way the columns are cut."""
    x, s, o, dy = bn_inputs(rows + c, (rows, c), dtype, 1.0, 3.0)
    tx, e = to_torch(x), torch.empty(0, device="cuda")
    before = kernel_lib.MusaKernelsLaunchCount()
    fwd = raw_ops.FusedBatchNormV3(tx, to_torch(s), to_torch(o), e, e, epsilon=EPS)
    launches = kernel_lib.MusaKernelsLaunchCount() - before
    assert (launches == 1) == one_kernel
    check_forward(fwd, np_ref.fused_batch_norm(x, s, o, epsilon=EPS), dtype)


def test_retired_tuning_numbers_have_no_effect(kernel_lib):
    """Keys 2 and 3 were the bias chains' launch shape: a program that still
    sets them gets the same kernels as one that does not."""
    x, s, o, dy = bn_inputs(3, (1000, 64), "float32", 1.0, 3.0)

    def launches():
        before = kernel_lib.MusaKernelsLaunchCount()
        out = run_both(x, s, o, dy, "NHWC")
        return kernel_lib.MusaKernelsLaunchCount() - before, out

    want = launches()
    old = [kernel_lib.MusaKernelsSetTuning(k, v) for k, v in ((2, -1), (3, 8))]
    try:
        got = launches()
    finally:
        for k, v in zip((2, 3), old):
            kernel_lib.MusaKernelsSetTuning(k, v)
    assert got[0] == want[0]
    for a, b in zip((t for out in got[1] for t in out), (t for out in want[1] for t in out)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("shape", [
    # Planes of the channel-group kernels beyond four packs a thread (1025 .. 2816
    # elements), several images a CTA: 5, 6, 7, 10 and 11 packs a thread, planes of
    # single elements, of 4-byte, 8-byte and whole packs.
    (16, 512, 33, 33), (16, 512, 34, 33), (16, 512, 40, 40), (24, 256, 47, 51), (12, 512, 44, 64),
    # The longest plane, and the first that is too long; one image a CTA.
    (2, 16, 44, 64), (2, 16, 1, 2817), (1, 8, 50, 50),
    # One to four packs a thread, whole and not.
    (40, 256, 14, 14), (9, 64, 18, 18), (24, 128, 24, 24), (33, 64, 28, 28), (17, 64, 32, 32),
    (33, 64, 29, 31), (5, 2048, 7, 14)])
def test_channel_major_chain(kernel_lib, dtype, shape):
    """Channel-major planes through the chain of kernels (group and plane kernels as
    the rule has it for each pass), inference too, against the oracle."""
    c = shape[1]
    x, s, o, dy = bn_inputs(500 + c + shape[3], shape, dtype, 1.0, 3.0, channel_axis=1)
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS, data_format="NCHW")
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS, "NCHW")
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))
    with tuned(kernel_lib, (24, -1)):
        fwd, grad, _ = launch_ops(kernel_lib, x, s, o, dy, "NCHW")
    check_forward(fwd, want, dtype)
    check_grad(grad, wg, dtype, dx_scale=terms)
    infer = raw_ops.FusedBatchNormV3(to_torch(x), to_torch(s), to_torch(o), fwd.reserve_space_1,
                                     fwd.reserve_space_2, epsilon=EPS, data_format="NCHW",
                                     is_training=False)
    rt = _rt(dtype)
    assert_close(to_numpy(infer.y), want[0], rt, rt * _rms(want[0]), "inference")


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("rows,parts", [(4099, 1), (4096, 4), (4099, 4)])
@pytest.mark.parametrize("fused", [False, True, "moments"])
@pytest.mark.parametrize("c", [37, 101])
def test_split_api_with_odd_channel_counts(kernel_lib, dtype, rows, parts, fused, c):
    """The cross-replica forms where several rows make one whole-pack row: the rows
    left over (4099 = 4096 + 3) are added by the finalize kernel of every form; row
    blocks that start inside a pack take the element kernels."""
    x, s, o, dy = bn_inputs(18 + c, (rows, c), dtype, 0.0, 1.0)
    got = _split_forward_and_grad(kernel_lib, to_torch(x), to_torch(dy), to_torch(s),
                                  to_torch(o), parts, fused)
    want = np_ref.fused_batch_norm(x, s, o, epsilon=EPS)
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS)
    rt = _rt(dtype)
    assert_close(to_numpy(got[0]), want[0], rt, rt * _rms(want[0]), "y")
    for i in range(1, 5):
        assert_close(to_numpy(got[i]), want[i], 1e-4, 1e-4 * max(_rms(want[i]), 1e-6))
    assert_close(to_numpy(got[5]), wg[0], rt, rt * _rms(wg[0]), "dx")
    assert_close(to_numpy(got[6]), wg[1], 1e-4, 1e-4 * _rms(wg[1]), "dscale")
    assert_close(to_numpy(got[7]), wg[2], 1e-4, 1e-4 * _rms(wg[2]), "doffset")
