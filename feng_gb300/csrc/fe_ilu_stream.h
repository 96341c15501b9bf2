// Triangular solves of the block-Jacobi ILU(0) with the vector in shared
// memory: one thread block per diagonal block, whose levels follow one
// another with a block barrier between them, and the factor's entries packed
// in the order in which the solve uses them, so that one warp copies them into
// shared memory ahead of the dependences.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

namespace feng {

class IluStream {
 public:
  IluStream() = default;
  IluStream(const IluStream &) = delete;
  IluStream &operator=(const IluStream &) = delete;
  ~IluStream();
  // Packs the pattern (block-local CSR lia / lja / ldiag by row, global
  // columns; rows of block b: perm[start[b]] .. perm[start[b + 1] - 1]).
  // Returns FE_OK with usable() false when a block does not fit.
  int build(const std::vector<int32_t> &lia, const std::vector<int32_t> &lja, const std::vector<int32_t> &ldiag,
            const std::vector<int32_t> &perm, const std::vector<int32_t> &start, bool fp32, cudaStream_t s);
  bool usable() const { return usable_; }
  // Takes over the factor's values (FP32 or FP64 as built; lia, ldiag: build's,
  // on the device).
  void gather(const void *f, const int32_t *lia, const int32_t *ldiag);
  // z = U^-1 L^-1 r on the factor's own precision; r and z FP32 or FP64.
  void solve(const float *r, float *z, const int *done) const;
  void solve(const double *r, double *z, const int *done) const;

  // One step of a block's stream: `warps` warps of slots, the longest chains
  // first; warp w holds rows of four slots where bit w of wide is set, else of
  // two, and in nibble w of chains the entries of its longest slot (the others
  // padded with zeros).  Entry k of the warps that have one: from entry + lanes
  // (the warps with an entry 0, .. k - 1) on.  A warp alone (small blocks: a
  // level is a few rows) is stored with the lanes that it uses.
  static constexpr int E = 5;  // entries of a slot per step
  struct Step {
    int32_t entry;      // first entry
    int32_t slot;       // first slot (columns)
    uint32_t chains;
    uint8_t warps, wide;
    uint8_t flags;      // STEP_*
    uint8_t lanes;      // stored of a warp
  };

 private:
  template <typename V> void launch(const V *r, V *z, const int *done) const;
  cudaStream_t s_ = 0;
  bool usable_ = false, fp32_ = false;
  int64_t nBlocks_ = 0, nSteps_ = 0, nEntries_ = 0, nRows_ = 0;
  int maxWarps_ = 1;               // of a step
  size_t smem_ = 0;
  int lateStep_ = -1;
  Step *steps_ = nullptr;          // all blocks' steps
  int2 *from_ = nullptr;           // [steps] the block's first row; 2 times the chunk of its rows, + 1 for L
  int32_t *stepStart_ = nullptr;   // [nBlocks + 1]
  int32_t *start_ = nullptr;
  int32_t *perm_ = nullptr;        // rows in the vector's order
  uint4 *col_ = nullptr;           // [slots] local indices of its E entries and its row (16 bits each)
  void *val_ = nullptr;            // [entries]
  void *scale_ = nullptr;          // [rows, as perm] inverse diagonal of U
};

}  // namespace feng
