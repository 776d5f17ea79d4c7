// Where the rows of a [rows, row_size] tensor lie against packs of kVec elements
// (a power of two) when row_size is not a multiple of kVec.  Plain integer
// arithmetic: the kernels and host code share it.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MUSA_HOST_DEVICE __host__ __device__
#else
#define MUSA_HOST_DEVICE
#endif

namespace musa_b200 {

// Elements of the row's first pack that belong to the rows before it.  Rows a
// multiple of kVec apart share it.
template <int kVec>
MUSA_HOST_DEVICE constexpr int RowShift(int64_t row, int row_size) {
  return static_cast<int>((row % kVec) * (row_size % kVec) % kVec);
}

// Packs that hold a row which starts `shift` elements into a pack.
template <int kVec>
MUSA_HOST_DEVICE constexpr int ShiftedPacks(int row_size, int shift) {
  return (row_size + shift + kVec - 1) / kVec;
}

// The row's first pack, counted from the tensor's start.
template <int kVec>
MUSA_HOST_DEVICE constexpr int64_t ShiftedRowPack(int64_t row, int row_size, int shift) {
  return (row * row_size - shift) / kVec;
}

// Whether the row's pack p (of `packs`) can be the tensor's last one.  kTailRows: 1
// for rows of at least a pack, kVec for rows that may be shorter (several of them
// can share the last pack).
template <int kTailRows>
MUSA_HOST_DEVICE constexpr bool MayEndTensor(int64_t row, int64_t rows, int p, int packs) {
  return p == packs - 1 && (kTailRows == 1 ? row == rows - 1 : rows - row <= kTailRows);
}

// Elements of such a pack that lie inside the tensor.
template <int kVec, int kTailRows>
MUSA_HOST_DEVICE constexpr int PackElements(int64_t row, int64_t rows, int row_size, int shift,
                                            int p) {
  if (kTailRows == 1) return row_size + shift - p * kVec;
  const int left = static_cast<int>(rows - row) * row_size + shift - p * kVec;
  return left < kVec ? left : kVec;
}

}  // namespace musa_b200
