// Sliced-ELL copy of a CSR matrix with its columns shared by blocks of
// unknowns, for the products of the Krylov solver.
//
// The unknowns of a velocity node are consecutive, their rows have the same
// columns and those columns come in runs of one node's unknowns, so a node's
// D x D entries need one column index: 5 (D = 2) or 4.4 (D = 3) bytes per
// FP32 entry instead of 8, one gather of D consecutive entries of x for D^2
// products, and the threads of a node hold its D row sums.  The blocks are found in the
// pattern itself (rows with equal columns; runs of columns), not in the
// numbering, so any pattern is accepted: rows and columns that do not pair
// up stay single.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "fe_krylov.h"

namespace feng {

class BlockSell {
 public:
  BlockSell() = default;
  BlockSell(const BlockSell &) = delete;
  BlockSell &operator=(const BlockSell &) = delete;
  ~BlockSell();
  // Builds the layout of the pattern on the device (values FP32 or FP64).
  int build(const DeviceCSR &A, bool fp32, cudaStream_t s);
  // Copies the CSR values (of the type given to build) into the layout.
  void gather(const void *vals);
  // FP32 values: y = A x in FP32; r = b - A x with FP64 x and FP64
  // accumulation, or with x split into two floats and double-float
  // accumulation (fe_df.h).
  void mul32(const float *x, float *y, const int *done) const;
  void resid32(const double *x, const double *b, double *r) const;
  void resid32_df(const float2 *xs, const double *b, double *r) const;
  // FP64 values: y = A x; r = b - A x.  x 16-byte aligned (all of these).
  void mul64(const double *x, double *y, const int *done) const;
  void resid64(const double *x, const double *b, double *r) const;
  bool built() const { return built_; }
  int blockSize() const { return D_; }
  // Bytes of the layout that one product reads (values, columns, slices).
  int64_t bytes() const;

  // A set of row groups (NR = D rows each, or single rows): groups in slices
  // of 32, one or more threads per group; a slice's entries are padded to its longest
  // group and stored step by step (entry k of the 32 groups together).
  struct Part {
    int64_t n = 0;                                   // groups
    int32_t *row = nullptr;                          // [n] first row of the group
    int32_t *pPtr = nullptr, *sPtr = nullptr;        // [slices + 1] steps: block entries (D columns), single columns
    int32_t *pCol = nullptr, *sCol = nullptr;        // first column of the entry
    int32_t *pOff = nullptr, *sOff = nullptr;        // its offset in the CSR row (-1: padding)
    void *pVal = nullptr, *sVal = nullptr;           // NR x D, NR x 1 values
    int64_t pSteps = 0, sSteps = 0;
  };

 private:
  int fill(Part &P, const std::vector<int32_t> &rows, const uint8_t *dStart);
  template <int MODE, typename VA, typename X, typename Y>
  void launch(const X *x, const double *b, Y *y, const int *done) const;
  DeviceCSR A_;
  cudaStream_t s_ = 0;
  Part grp_, one_;  // groups of D rows; single rows
  int D_ = 1;
  int lanes_ = 1;      // threads per row group
  bool even_ = false;  // D = 2: every block starts at an even column
  bool fp32_ = false, built_ = false;
};

}  // namespace feng
