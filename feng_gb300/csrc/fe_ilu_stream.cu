// Triangular solves with the vector in shared memory (see fe_ilu_stream.h).
#include "fe_ilu_stream.h"

#include <algorithm>

#include "fe_common.h"
#include "fe_launch.h"

namespace feng {

#define CKI(x)                                                                         \
  do {                                                                                 \
    cudaError_t _e = (x);                                                              \
    if(_e != cudaSuccess) {                                                            \
      set_error("CUDA error %s at %s:%d", cudaGetErrorString(_e), __FILE__, __LINE__); \
      return FE_CUDA_FAIL;                                                             \
    }                                                                                  \
  } while(0)

namespace {

constexpr int E = IluStream::E;
constexpr int WORKERS = 256;       // threads that solve: 128 rows per step
constexpr int THREADS = 512;       // the others copy the next steps' operands
constexpr int STAGES = 3;
constexpr int MAX_STEPS = 4096;    // of one block (shared memory)
constexpr size_t MAX_SMEM = 226 * 1024;
enum : uint8_t { STEP_FIRST = 1, STEP_LAST = 2 };

// A step's operands in shared memory.
template <typename V>
struct Stage {
  uint4 col[WORKERS];
  V val[E][WORKERS];
  V scale[WORKERS];
  int32_t row[WORKERS];
};

template <int BYTES>
__device__ __forceinline__ void copy_async(void *dst, const void *src)
{
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr(BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}

// z = U^-1 L^-1 r on one diagonal block, z in shared memory.  Two slots
// (neighbouring lanes) per row: the row's entries alternate between them, the
// first starts from the row's right-hand side, and one exchange adds the two.
// (More lanes per row would only queue at the FP64 pipe, which takes 64
// cycles per warp; the rows of a step are sorted by length, so that a warp
// runs no further than its own longest row.)  U's entries are scaled by the
// inverse diagonal beforehand, so a row ends with an addition.  The upper
// half of the threads copies the operands of the step after next while the
// lower half solves; a block barrier ends every step.
// Bound: the chain of levels (their products on one SM's FP64 pipe, an
// exchange and a barrier).  64 x 64 P2 diffusion (16 k rows, 254 levels per
// triangle): 0.42 ms per application against 3.75 ms with a warp per row and
// the vector in global memory.
template <typename V>
__global__ void __launch_bounds__(THREADS) k_ilu_stream(const IluStream::Step *__restrict__ steps,
                                                        const int32_t *__restrict__ stepStart,
                                                        const int32_t *__restrict__ start,
                                                        const int32_t *__restrict__ perm,
                                                        const uint4 *__restrict__ col, const V *__restrict__ val,
                                                        const int32_t *__restrict__ row, const V *__restrict__ scale,
                                                        const V *__restrict__ r, V *__restrict__ z,
                                                        const int *__restrict__ done)
{
  FE_PDL_ENTRY();
  if(done && *done) return;
  extern __shared__ __align__(16) unsigned char smem[];
  const int b = blockIdx.x, tid = threadIdx.x;
  const int32_t p0 = start[b], n = start[b + 1] - p0;
  const int32_t s0 = stepStart[b], ns = stepStart[b + 1] - s0;
  Stage<V> *stage = reinterpret_cast<Stage<V> *>(smem);
  V *x = reinterpret_cast<V *>(smem + STAGES * sizeof(Stage<V>));
  IluStream::Step *st = reinterpret_cast<IluStream::Step *>(
      smem + STAGES * sizeof(Stage<V>) + (((size_t)n * sizeof(V) + 15) & ~(size_t)15));
  for(int i = tid; i < ns; i += THREADS) st[i] = steps[s0 + i];
  for(int i0 = tid; i0 < n; i0 += 8 * THREADS) {
    V t[8];
#pragma unroll
    for(int u = 0; u < 8; ++u) t[u] = i0 + u * THREADS < n ? r[perm[p0 + i0 + u * THREADS]] : (V)0;
#pragma unroll
    for(int u = 0; u < 8; ++u)
      if(i0 + u * THREADS < n) x[i0 + u * THREADS] = t[u];
  }
  __syncthreads();
  // the copying threads: one commit group per step, empty past the end
  const int h = tid - WORKERS;
  auto copy = [&](int q) {
    if(q < ns) {
      const IluStream::Step s = st[q];
      Stage<V> &g = stage[q % STAGES];
      int64_t e = s.entry;
#pragma unroll
      for(int k = 0; k < E; ++k) {
        if(h < 32 * s.groups[k]) copy_async<sizeof(V)>(&g.val[k][h], val + e + h);
        e += 32 * s.groups[k];
      }
      if(h < s.n) {
        copy_async<16>(&g.col[h], col + s.slot + h);
        copy_async<sizeof(V)>(&g.scale[h], scale + s.slot + h);
        copy_async<4>(&g.row[h], row + s.slot + h);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if(h >= 0) {
#pragma unroll
    for(int q = 0; q < STAGES - 1; ++q) copy(q);
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
  }
  __syncthreads();
  V acc = 0;
  for(int q = 0; q < ns; ++q) {
    if(h >= 0) {
      // into the stage that the last step has left
      copy(q + STAGES - 1);
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    } else {
      const IluStream::Step &s = st[q];
      if((tid & ~31) < s.n) {  // whole warps take part in the exchange
        const Stage<V> &g = stage[q % STAGES];
        const bool live = tid < s.n;
        const int row = live ? g.row[tid] : 0;
        const uint4 c4 = live ? g.col[tid] : make_uint4(0, 0, 0, 0);
        if(s.flags & STEP_FIRST) acc = live && !(tid & 1) ? x[row] * g.scale[tid] : (V)0;
        const unsigned cw[4] = {c4.x, c4.y, c4.z, c4.w};
        V xv[E], v[E];
#pragma unroll
        for(int k = 0; k < E; ++k) {
          const bool on = (tid >> 5) < s.groups[k];
          v[k] = on ? g.val[k][tid] : (V)0;
          xv[k] = on ? x[(cw[k >> 1] >> (16 * (k & 1))) & 0xffffu] : (V)0;
        }
#pragma unroll
        for(int k = 0; k < E; ++k)
          if((tid >> 5) < s.groups[k]) acc -= v[k] * xv[k];
        if(s.flags & STEP_LAST) {
          const V other = __shfl_xor_sync(0xffffffffu, acc, 1);
          if(live && !(tid & 1)) x[row] = acc + other;
        }
      }
    }
    __syncthreads();
  }
  for(int i = tid; i < n; i += THREADS) z[perm[p0 + i]] = x[i];
}

// The packed values: L as it is, U divided by its row's diagonal, and the
// slots' scales (1 / diagonal for the first slot of a U row).
template <typename V>
__global__ void k_ilu_pack(int64_t ne, const int32_t *__restrict__ pos, const int32_t *__restrict__ dpos,
                           const V *__restrict__ f, V *__restrict__ val, int64_t nslots,
                           const int32_t *__restrict__ slotDiag, V *__restrict__ scale)
{
  FE_PDL_ENTRY();
  for(int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
    V v = pos[e] >= 0 ? f[pos[e]] : (V)0;
    if(pos[e] >= 0 && dpos[e] >= 0) v /= f[dpos[e]];
    val[e] = v;
  }
  for(int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nslots; q += (int64_t)gridDim.x * blockDim.x)
    scale[q] = slotDiag[q] >= 0 ? (V)1 / f[slotDiag[q]] : (V)1;
}

template <typename T>
int to_device(T **dst, const std::vector<T> &v)
{
  CKI(cudaMalloc(dst, sizeof(T) * std::max<size_t>(1, v.size())));
  CKI(cudaMemcpy(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

}  // namespace

IluStream::~IluStream()
{
  cudaFree(steps_); cudaFree(stepStart_); cudaFree(start_); cudaFree(perm_);
  cudaFree(col_); cudaFree(pos_); cudaFree(dpos_); cudaFree(val_);
  cudaFree(row_); cudaFree(slotDiag_); cudaFree(scale_);
}

int IluStream::build(const std::vector<int32_t> &lia, const std::vector<int32_t> &lja,
                     const std::vector<int32_t> &ldiag, const std::vector<int32_t> &perm,
                     const std::vector<int32_t> &start, bool fp32, cudaStream_t s)
{
  s_ = s;
  fp32_ = fp32;
  nBlocks_ = (int64_t)start.size() - 1;
  const size_t vs = fp32 ? sizeof(float) : sizeof(double);
  const size_t stages = STAGES * (fp32 ? sizeof(Stage<float>) : sizeof(Stage<double>));
  const int64_t n = (int64_t)perm.size();
  for(int64_t b = 0; b < nBlocks_; ++b) {
    const int64_t rows = start[b + 1] - start[b];
    if(rows > 65535 || stages + rows * vs > MAX_SMEM) return FE_OK;  // the level kernels
  }
  std::vector<int32_t> local(n);
  for(int64_t b = 0; b < nBlocks_; ++b)
    for(int32_t q = start[b]; q < start[b + 1]; ++q) local[perm[q]] = q - start[b];

  std::vector<Step> steps;
  std::vector<int32_t> stepStart(1, 0), pos, dpos, slotDiag, level(n, 0);
  std::vector<int32_t> row;
  std::vector<uint4> col;
  std::vector<int32_t> cnt, ord;
  for(int64_t b = 0; b < nBlocks_; ++b) {
    const int32_t p0 = start[b], p1 = start[b + 1];
    for(int lower = 1; lower >= 0; --lower) {
      // levels (the block's rows ascend in perm)
      int32_t nl = 0;
      for(int32_t k = 0; k < p1 - p0; ++k) {
        const int32_t i = perm[lower ? p0 + k : p1 - 1 - k];
        const int32_t kb = lower ? lia[i] : ldiag[i] + 1, ke = lower ? ldiag[i] : lia[i + 1];
        int32_t m = 0;
        for(int32_t e = kb; e < ke; ++e) m = std::max(m, level[lja[e]] + 1);
        level[i] = m;
        nl = std::max(nl, m + 1);
      }
      cnt.assign(nl + 1, 0);
      for(int32_t q = p0; q < p1; ++q) cnt[level[perm[q]] + 1]++;
      for(int32_t l = 0; l < nl; ++l) cnt[l + 1] += cnt[l];
      ord.resize(p1 - p0);
      {
        std::vector<int32_t> fill(cnt.begin(), cnt.end() - 1);
        for(int32_t q = p0; q < p1; ++q) ord[fill[level[perm[q]]]++] = perm[q];
      }
      for(int32_t l = 0; l < nl; ++l) {
        // rows of similar length together
        auto len = [&](int32_t i) { return lower ? ldiag[i] - lia[i] : lia[i + 1] - ldiag[i] - 1; };
        std::stable_sort(ord.begin() + cnt[l], ord.begin() + cnt[l + 1],
                         [&](int32_t x, int32_t y) { return len(x) > len(y); });
        for(int32_t r0 = cnt[l]; r0 < cnt[l + 1]; r0 += WORKERS / 2) {
          const int32_t nr = std::min<int32_t>(WORKERS / 2, cnt[l + 1] - r0);
          const int per = (len(ord[r0]) + 1) / 2;  // entries per slot of the longest row
          const int chunks = std::max(1, (per + E - 1) / E);
          for(int c = 0; c < chunks; ++c) {
            Step st = {};
            st.entry = (int32_t)pos.size();
            st.slot = (int32_t)row.size();
            st.n = (uint16_t)(2 * nr);
            st.flags = (uint8_t)((c == 0 ? STEP_FIRST : 0) | (c + 1 == chunks ? STEP_LAST : 0));
            for(int k = 0; k < E; ++k) {
              // slots that hold an entry k: the leading ones, in whole warps
              int32_t m = 0;
              while(m < nr && len(ord[r0 + m]) > 2 * (c * E + k)) ++m;
              st.groups[k] = (uint8_t)((2 * m + 31) / 32);
              for(int32_t t = 0; t < 32 * st.groups[k]; ++t) {
                const int32_t q = t / 2;
                const int32_t i = q < nr ? ord[r0 + q] : -1;
                const int32_t e = i < 0 ? 0 : (lower ? lia[i] : ldiag[i] + 1) + 2 * (c * E + k) + (t & 1);
                const bool ok = i >= 0 && e < (lower ? ldiag[i] : lia[i + 1]);
                pos.push_back(ok ? e : -1);
                dpos.push_back(ok && !lower ? ldiag[i] : -1);
              }
            }
            for(int32_t q = 0; q < nr; ++q)
              for(int h = 0; h < 2; ++h) {
                const int32_t i = ord[r0 + q];
                row.push_back(local[i]);
                slotDiag.push_back(!lower && h == 0 ? ldiag[i] : -1);
                uint32_t w[4] = {0, 0, 0, 0};
                for(int k = 0; k < E; ++k) {
                  const int32_t e = (lower ? lia[i] : ldiag[i] + 1) + 2 * (c * E + k) + h;
                  // padding (value 0) reads the row's own entry of the vector
                  const int32_t j = e < (lower ? ldiag[i] : lia[i + 1]) ? local[lja[e]] : local[i];
                  w[k >> 1] |= (uint32_t)j << (16 * (k & 1));
                }
                col.push_back(make_uint4(w[0], w[1], w[2], w[3]));
              }
            steps.push_back(st);
          }
        }
      }
    }
    stepStart.push_back((int32_t)steps.size());
    const int32_t own = stepStart[b + 1] - stepStart[b];
    const size_t need = stages + (((size_t)(p1 - p0) * vs + 15) & ~(size_t)15) + (size_t)own * sizeof(Step);
    if(own > MAX_STEPS || need > MAX_SMEM || pos.size() > (size_t)INT32_MAX / 2) return FE_OK;
    smem_ = std::max(smem_, need);
  }
  nEntries_ = (int64_t)pos.size();
  nSlots_ = (int64_t)row.size();
  FE_TRY(to_device(&steps_, steps));
  FE_TRY(to_device(&stepStart_, stepStart));
  FE_TRY(to_device(&start_, start));
  FE_TRY(to_device(&perm_, perm));
  FE_TRY(to_device(&col_, col));
  FE_TRY(to_device(&pos_, pos));
  FE_TRY(to_device(&dpos_, dpos));
  FE_TRY(to_device(&row_, row));
  FE_TRY(to_device(&slotDiag_, slotDiag));
  CKI(cudaMalloc(&val_, vs * std::max<int64_t>(1, nEntries_)));
  CKI(cudaMalloc(&scale_, vs * std::max<int64_t>(1, nSlots_)));
  // the copies ran on the legacy stream, with which s is not ordered
  CKI(cudaStreamSynchronize(cudaStreamLegacy));
  if(fp32) CKI(cudaFuncSetAttribute(k_ilu_stream<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
  else CKI(cudaFuncSetAttribute(k_ilu_stream<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM));
  usable_ = true;
  return FE_OK;
}

void IluStream::gather(const void *f)
{
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((nEntries_ + 255) / 256, 4096));
  if(fp32_)
    ::feng::launch_k(k_ilu_pack<float>, g, 256, 0, s_, nEntries_, pos_, dpos_, (const float *)f, (float *)val_, nSlots_,
                     slotDiag_, (float *)scale_);
  else
    ::feng::launch_k(k_ilu_pack<double>, g, 256, 0, s_, nEntries_, pos_, dpos_, (const double *)f, (double *)val_,
                     nSlots_, slotDiag_, (double *)scale_);
}

template <typename V>
void IluStream::launch(const V *r, V *z, const int *done) const
{
  ::feng::launch_k(k_ilu_stream<V>, (int)nBlocks_, THREADS, smem_, s_, steps_, stepStart_, start_, perm_, col_,
                   (const V *)val_, row_, (const V *)scale_, r, z, done);
}

void IluStream::solve(const float *r, float *z, const int *done) const { launch<float>(r, z, done); }
void IluStream::solve(const double *r, double *z, const int *done) const { launch<double>(r, z, done); }

}  // namespace feng
