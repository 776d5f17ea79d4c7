"""Channel-major BatchNorm layers of more channels than CTAs are resident at once: one kernel per
pass, in waves (tuning key 26: 1 takes the form wherever it is possible)."""
import numpy as np
import pytest
import torch

from oracle import np_ref
from helpers import bn_inputs, to_numpy
from test_batchnorm_gpu import EPS, _rms, check_forward, check_grad, launch_ops, tuned

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shape", [
    # One image and many; planes longer and shorter than a CTA has threads; a walk that ends
    # inside a slot; waves that are full, half full and nearly empty.
    ("bfloat16", (20, 600, 28, 28)), ("float32", (11, 520, 32, 32)), ("float32", (100, 500, 10, 10)),
    ("float16", (1, 700, 120, 120)), ("bfloat16", (5, 560, 56, 56)), ("bfloat16", (13, 700, 31, 32)),
    ("float32", (2, 297, 76, 76)), ("float16", (1536, 592, 4, 4))])
def test_against_oracle_and_chain(kernel_lib, dtype, shape):
    x, s, o, dy = bn_inputs(sum(shape), shape, dtype, 1.0, 3.0, channel_axis=1)
    c = shape[1]
    gen = np.random.default_rng(c)
    est = gen.standard_normal(c).astype(np.float32), (gen.random(c) + 0.5).astype(np.float32)
    want = np_ref.fused_batch_norm(x, s, o, *est, epsilon=EPS, exponential_avg_factor=0.25,
                                   data_format="NCHW")
    wg = np_ref.fused_batch_norm_grad(dy, x, s, want[3], want[4], EPS, data_format="NCHW")
    terms = _rms(dy) * float(np.max(s / np.sqrt(want[4] + EPS)))
    with tuned(kernel_lib, (26, 1)):
        before = kernel_lib.MusaKernelsLaunchCount()
        got = launch_ops(kernel_lib, x, s, o, dy, fmt="NCHW", est=est, factor=0.25)
        assert kernel_lib.MusaKernelsLaunchCount() - before == 3
        again = launch_ops(kernel_lib, x, s, o, dy, fmt="NCHW", est=est, factor=0.25, scratch=0x5A)
    with tuned(kernel_lib, (24, -1)):
        chain = launch_ops(kernel_lib, x, s, o, dy, fmt="NCHW", est=est, factor=0.25)
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
