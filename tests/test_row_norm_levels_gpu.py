"""The second level of the LayerNorm gradient (column sums over the partial rows of the CTAs):
from one partial row to more than one thread requests at once, columns that do not fill a
CTA, rows in slab order and in plain order."""
import numpy as np
import pytest
import torch

from oracle import np_ref
from helpers import assert_close, np_dtype, to_numpy, to_torch
from tensorflow_musa_extension_b200 import raw_ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
# Row lengths: one pack and two, a last CTA of 8 columns, warp groups, wide groups; rows that
# start inside a pack; rows longer than the register layouts.
@pytest.mark.parametrize("n", [8, 20, 24, 512, 1024, 2048, 37, 777, 20000])
# Row blocks (1 to 16 rows each): one partial row, a lane each, more than a lane requests at once.
@pytest.mark.parametrize("blocks", [1, 64, 65, 300, 2400])
def test_column_sums(kernel_lib, dtype, n, blocks):
    if n * blocks > 3_000_000:
        blocks = 3_000_000 // n
    for rows in {blocks, 4 * blocks - 1}:
        rng = np.random.default_rng(n + rows)
        dt = np_dtype(dtype)
        x = (rng.standard_normal((rows, n)) * 2 + 1).astype(dt)
        dy = rng.standard_normal((rows, n)).astype(dt)
        gamma = rng.uniform(0.5, 1.5, n).astype(dt)
        beta = np.zeros(n, dt)
        tx, td, tg, tb = (to_torch(a) for a in (x, dy, gamma, beta))
        got = raw_ops.MusaLayerNormGrad(td, tx, tg, tb)
        again = raw_ops.MusaLayerNormGrad(td, tx, tg, tb)
        want = np_ref.layer_norm_grad(dy, x, gamma)
        # |x_hat| and |dy| are O(1): a sum of `rows` terms has fp32 roundings of at most 2^-22 of
        # the sum of magnitudes and a few ulps of its own size.  Both sides are rounded to bf16: next
        # to a tie they are neighbours, one ulp or at most 2^-7 of the value apart.
        at = rows * 2.0 ** -22 + np.sqrt(rows) * 2.0 ** -20
        rt = 1e-5 if dtype == "float32" else 2.0 ** -7
        for k, name in ((1, "dgamma"), (2, "dbeta")):
            assert_close(to_numpy(got[k]), want[k], rt, at, name)
        for a, b in zip(got, again):
            assert (to_numpy(a) == to_numpy(b)).all()


# One row a CTA: rows in slab order, rows that start inside a pack, rows beyond the register layouts.
@pytest.mark.parametrize("dtype,n", [("float32", 4096), ("float32", 4097), ("float32", 20000),
                                     ("bfloat16", 8192), ("bfloat16", 8191)])
def test_partial_rows_add_in_64_bits(kernel_lib, dtype, n):
    """Partial rows that cancel: of 2^30, -2^30 and 1, in turn, an fp64 sum leaves the exact number of
    ones, an fp32 sum of two of them rounds the one away.  An infinity and a NaN stay in their
    columns."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    rows = min(sms, 140) // 3 * 3
    dt = getattr(torch, dtype)
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn(rows, n, device="cuda", generator=gen).to(dt)
    dy = torch.tensor([2.0 ** 30, -2.0 ** 30, 1.0], device="cuda").repeat(rows // 3)[:, None]
    dy = dy.repeat(1, n).to(dt)
    gamma, beta = torch.ones(n, device="cuda", dtype=dt), torch.zeros(n, device="cuda", dtype=dt)
    db = raw_ops.MusaLayerNormGrad(dy, x, gamma, beta)[2]
    assert torch.equal(db, torch.full_like(db, rows // 3))
    dy[5, 3], dy[70, 9] = float("inf"), float("nan")
    db = raw_ops.MusaLayerNormGrad(dy, x, gamma, beta)[2].float()
    assert db[3] == float("inf") and torch.isnan(db[9])
    db[3] = db[9] = rows // 3
    assert torch.equal(db, torch.full_like(db, rows // 3))
