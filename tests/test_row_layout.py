"""Rows that are not whole 128-bit packs: the arithmetic that the row kernels use
(csrc/row_layout.h), compiled for the host and checked for every small shape."""
import os
import subprocess

import numpy as np
import pytest
import torch

from conftest import ROOT
from oracle import np_ref
from helpers import NP_BF16
from tensorflow_musa_extension_b200 import raw_ops

PROGRAM = r"""
#include <cstdio>
#include "row_layout.h"
using namespace musa_b200;
// Every copy of every row of a [rows, n] tensor, as the kernels of kTailRows make them.
template <int vec, int kTailRows>
bool Inside(int n, int64_t rows) {
  bool ok = true;
  for (int64_t row = 0; row < rows; ++row) {
    const int shift = RowShift<vec>(row, n);
    const int packs = ShiftedPacks<vec>(n, shift);
    const int64_t first = ShiftedRowPack<vec>(row, n, shift) * vec;
    ok = ok && first >= 0 && first + shift == row * n && shift == RowShift<vec>(row + vec, n);
    int64_t end = first;
    for (int p = 0; p < packs; ++p) {
      const int e = MayEndTensor<kTailRows>(row, rows, p, packs)
                        ? PackElements<vec, kTailRows>(row, rows, n, shift, p) : vec;
      ok = ok && e > 0 && e <= vec && first + p * vec + e <= rows * n;
      end = first + p * vec + e;
    }
    ok = ok && end >= (row + 1) * n;
  }
  if (!ok) std::printf("vec %d, tail rows %d: [%d, %d]\n", vec, kTailRows, (int)rows, n);
  return ok;
}
int main() {
  bool ok = true;
  for (int n = 1; n <= 24; ++n)
    for (int64_t rows = 1; rows <= 24; ++rows) {
      ok = Inside<4, 4>(n, rows) && Inside<8, 8>(n, rows) && ok;
      if (n >= 4) ok = Inside<4, 1>(n, rows) && ok;
      if (n >= 8) ok = Inside<8, 1>(n, rows) && ok;
    }
  return !ok;
}
"""


def test_copies_stay_inside_the_tensor(tmp_path):
    src, exe = tmp_path / "rows.cc", tmp_path / "rows"
    src.write_text(PROGRAM)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(
        ROOT, "tensorflow_musa_extension_b200", "csrc"), str(src), "-o", str(exe)], check=True)
    got = subprocess.run([str(exe)], capture_output=True, text=True)
    assert got.returncode == 0, got.stdout


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("n", [1, 2, 3, 5, 7])
@pytest.mark.parametrize("rows", [1, 2, 3, 5, 1000])
def test_rows_shorter_than_a_pack(kernel_lib, dtype, n, rows):
    """Rows of one to seven elements, several of them in the tensor's last pack:
    all four ops against the oracle."""
    rng = np.random.default_rng(rows * 8 + n)
    np_t = np.float32 if dtype == "float32" else NP_BF16
    x, dy = (rng.standard_normal((rows, n)).astype(np_t) for _ in range(2))
    g, b = (rng.uniform(0.5, 1.5, n).astype(np_t) for _ in range(2))
    y = raw_ops.MusaLayerNorm(x, g, b, 1e-2)
    dx, dgamma, dbeta = raw_ops.MusaLayerNormGrad(dy, x, g, b, 1e-2)
    rms = raw_ops.MusaRmsNorm(x, g, 1e-2)
    rdx = raw_ops.MusaRmsNormGradDx(x, rms.inv_rms, g, dy)
    wx, wg, wb = np_ref.layer_norm_grad(dy, x, g, 1e-2)
    wr = np_ref.rms_norm(x, g, 1e-2)
    wrx = np_ref.rms_norm_grad_dx(x, rms.inv_rms, g, dy)
    # One rounding of T on the result beside fp32 arithmetic on terms that are at
    # most 1 / sqrt(epsilon) = 10 times the inputs.
    rt, at = (1e-5, 1e-4) if dtype == "float32" else (2.0 ** -7, 1e-4)
    for got, want in ((y, np_ref.layer_norm(x, g, b, 1e-2)), (dx, wx), (dgamma, wg), (dbeta, wb),
                      (rms.y, wr[0]), (rdx, wrx)):
        got, want = (np.asarray(t).astype(np.float64) for t in (got, want))
        terms = 1e-6 * rows ** 0.5 * 40 + at
        assert np.all(np.abs(got - want) <= rt * np.abs(want) + terms)
