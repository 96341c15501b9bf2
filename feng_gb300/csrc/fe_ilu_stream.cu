// Triangular solves with the vector in shared memory (see fe_ilu_stream.h).
#include "fe_ilu_stream.h"

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdlib>

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
constexpr int WORKERS = 256;       // threads that solve
constexpr int THREADS = WORKERS + 32;  // the last warp copies the coming steps' operands
constexpr int STAGES = 3;
constexpr int WARPS = WORKERS / 32;
constexpr int LONG_ROW = 8;        // rows with more entries take LONG_SLOTS slots, the others two
constexpr int LONG_SLOTS = 4;
constexpr unsigned NO_ROW = 0xffffu;  // above every block's rows
constexpr int MAX_STEPS = 4096;    // of one block (shared memory)
constexpr size_t MAX_SMEM = 226 * 1024;
enum : uint8_t { STEP_FIRST = 1, STEP_LAST = 2, STEP_SCALE = 4 };

// A step's operands in shared memory.
template <typename V>
struct Stage {
  uint4 col[WORKERS];  // 16 bits each: the E entries' local columns, then the row
  V val[E][WORKERS];
};

// A stage's barrier: one arrival and the bytes of its copies.
__device__ __forceinline__ void bar_init(uint64_t *b)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"((unsigned)__cvta_generic_to_shared(b)) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t *b, unsigned bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"((unsigned)__cvta_generic_to_shared(b)),
               "r"(bytes)
               : "memory");
}
// False when the copies have not come (a few microseconds are usual).
__device__ __forceinline__ bool bar_wait(uint64_t *b, unsigned parity)
{
  const unsigned a = (unsigned)__cvta_generic_to_shared(b);
  for(int t = 0; t < 1 << 14; ++t) {
    unsigned ok;
    asm volatile(
      "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(a), "r"(parity)
      : "memory");
    if(ok) return true;
  }
  return false;
}
// Multiples of 16 bytes from and to 16-byte boundaries.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, unsigned bytes, uint64_t *b)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                 (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(bytes), "r"((unsigned)__cvta_generic_to_shared(b))
               : "memory");
}

// *p (shared memory) when on, without a branch (a conditional load in C++ is one, and branches
// keep loads from overlapping).
__device__ __forceinline__ void load_if(bool on, const float *p, float &v)
{
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p ld.shared.f32 %0, [%2];\n\t}"
               : "+f"(v)
               : "r"((unsigned)on), "r"((unsigned)__cvta_generic_to_shared(p)));
}
__device__ __forceinline__ void load_if(bool on, const double *p, double &v)
{
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p ld.shared.f64 %0, [%2];\n\t}"
               : "+d"(v)
               : "r"((unsigned)on), "r"((unsigned)__cvta_generic_to_shared(p)));
}

// z = U^-1 L^-1 r on one diagonal block, z in shared memory.  A row's entries
// are dealt to two or four slots (neighbouring lanes; a warp holds rows of one
// kind, of similar length), and the last slot starts from the row's right-hand
// side.  The FP64 pipe takes 64 cycles per warp instruction and a dependent one
// waits 110: two slots end rows of up to four products each soonest, four the
// longer ones, more only queue (eight: 0.46 ms where four took 0.37, all rows
// in four likewise).  Between the triangles the vector is scaled by U's inverse
// diagonal, as U's entries are beforehand, so a row ends with additions.
// One warp brings the operands of the steps ahead by bulk copies and waits for
// them; the others take the next step's into registers before the barrier that
// ends a step, with the right-hand sides, which no step but the row's own
// writes.
// Bound: the chain of levels (FP64 products and exchanges, about 700 cycles;
// gathers, the next step's operands and the barrier, as many).  64 x 64 P2
// diffusion (16 k rows, 254 levels per triangle): 0.34 ms per application; six
// products in a chain and copies by half of the threads 0.42, a warp per row
// and the vector in global memory 3.75.
template <typename V>
__global__ void __launch_bounds__(THREADS) k_ilu_stream(const IluStream::Step *__restrict__ steps,
                                                        const int32_t *__restrict__ stepStart,
                                                        const int32_t *__restrict__ start,
                                                        const int32_t *__restrict__ perm,
                                                        const uint4 *__restrict__ col, const V *__restrict__ val,
                                                        const V *__restrict__ scale, const V *__restrict__ r,
                                                        V *__restrict__ z,
                                                        const int *__restrict__ done, int lateStep)
{
  FE_PDL_ENTRY();
  if(done && *done) return;
  extern __shared__ __align__(16) unsigned char smem[];
  const int b = blockIdx.x, tid = threadIdx.x;
  const int32_t p0 = start[b];
  const unsigned n = start[b + 1] - p0;
  const int32_t s0 = stepStart[b], ns = stepStart[b + 1] - s0;
  Stage<V> *stage = reinterpret_cast<Stage<V> *>(smem);
  V *x = reinterpret_cast<V *>(smem + STAGES * sizeof(Stage<V>));
  IluStream::Step *st = reinterpret_cast<IluStream::Step *>(
      smem + STAGES * sizeof(Stage<V>) + (((size_t)n * sizeof(V) + 15) & ~(size_t)15));
  __shared__ uint64_t full[STAGES];
  __shared__ int late;  // a copy did not come
  if(tid == 0) {
    late = 0;
    for(int k = 0; k < STAGES; ++k) bar_init(full + k);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
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
  const int warp = tid >> 5, lane = tid & 31;
  // the copying warp: lane k < E brings the warps' entries k, lane E the columns
  auto copy = [&](int q) {
    if(q >= ns) return;
    const IluStream::Step s = st[q];
    Stage<V> &g = stage[q % STAGES];
    const int pre = lane <= E ? lane : E;
    int before = 0, own = 0;  // warps with an entry j < pre, with entry lane
#pragma unroll
    for(int w = 0; w < WARPS; ++w) {
      const int chain = (s.chains >> (4 * w)) & 15;
      before += min(chain, pre);
      own += chain > lane;
    }
    const void *src = val + s.entry + 32 * before;
    void *dst = &g.val[lane < E ? lane : 0][0];
    unsigned bytes = lane < E ? 32u * own * (unsigned)sizeof(V) : 0u;
    if(lane == E) {
      src = col + s.slot;
      dst = &g.col[0];
      bytes = 32u * s.warps * 16u;
    }
    const unsigned all = __reduce_add_sync(0xffffffffu, bytes);
    if(lane == 0) bar_expect(full + q % STAGES, all);
    __syncwarp();
    if(bytes) bulk_copy(dst, src, bytes, full + q % STAGES);
  };
  auto phase = [](int q) { return (unsigned)(q / STAGES) & 1u; };
  // until step q's operands are there; the barrier that follows tells the others.
  // When they do not come (lateStep: a step that counts as late, to test this),
  // the copying warp asks for nothing more, and there is no result at the end.
  int missing = INT_MAX;  // the first step that has not come
  auto arrived = [&](int q) {
    const bool here = q >= ns || (q != lateStep && bar_wait(full + q % STAGES, phase(q)));
    if(__all_sync(0xffffffffu, here) || missing != INT_MAX) return;
    missing = q;
    if(lane == 0) late = 1;
  };
  // The solving threads run on without asking whether a step's operands came
  // (that costs 4 to 9% of an application, as a flag or in the barrier): the
  // indices that they take from a stage are bounded by the vector's length, so
  // what lies in a stage that was not filled reads and writes entries of it.
  const unsigned top = (unsigned)(n - 1) | (unsigned)(n - 1) << 16;
  // the solving threads: the next step's operands, and what the slot starts from
  uint4 c4 = make_uint4(0, 0, 0, 0);
  V v[E], acc = 0, rhs = 0;
  IluStream::Step s = {}, ahead = st[0];
  auto fetch = [&](int q) {
    s = ahead;
    if(q >= ns) s.warps = s.flags = 0;
    if(q + 1 < ns) ahead = st[q + 1];
    if(warp >= s.warps) return;
    const Stage<V> &g = stage[q % STAGES];
    c4 = g.col[tid];
    c4.x = __vminu2(c4.x, top);
    c4.y = __vminu2(c4.y, top);
    c4.z = __vminu2(c4.z, top);
#pragma unroll
    for(int k = 0; k < E; ++k) load_if(k < (int)((s.chains >> (4 * warp)) & 15), &g.val[k][tid], v[k]);
    const unsigned row = c4.w >> 16;
    const int last = (s.wide >> warp) & 1 ? LONG_SLOTS - 1 : 1;
    const V own = x[row < n ? row : 0];
    rhs = (tid & last) == last ? own : (V)0;
  };
  if(warp == WARPS) {
#pragma unroll
    for(int q = 0; q < STAGES; ++q) copy(q);
    arrived(0);
    arrived(1);
  }
  __syncthreads();
  if(warp < WARPS) fetch(0);
  __syncthreads();
  int asked = STAGES;
  for(int q = 0; q < ns; ++q) {
    if(warp == WARPS) {
      if(missing == INT_MAX) {
        copy(q + STAGES);  // into the stage of this step, whose operands are in registers
        asked = q + STAGES + 1;
        arrived(q + 2);
      }
    } else if(warp < s.warps) {
      const unsigned cw[4] = {c4.x, c4.y, c4.z, c4.w};
      const unsigned row = c4.w >> 16;
      const int chain = (s.chains >> (4 * warp)) & 15;
      const bool wide = (s.wide >> warp) & 1, end = s.flags & STEP_LAST;
      V xv[E];
#pragma unroll
      for(int k = 0; k < E; ++k) load_if(k < chain, x + ((cw[k >> 1] >> (16 * (k & 1))) & 0xffffu), xv[k]);
      if(s.flags & STEP_FIRST) acc = rhs;
#pragma unroll
      for(int k = 0; k < E; ++k)
        if(k < chain) acc -= v[k] * xv[k];
      fetch(q + 1);
      if(end) {
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        if(wide)
#pragma unroll
          for(int o = 2; o < LONG_SLOTS; o <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if(row < n && !(tid & (wide ? LONG_SLOTS - 1 : 1))) x[row] = acc;
      }
    } else {
      if(s.flags & STEP_SCALE) {
#pragma unroll 8
        for(int i = tid; i < n; i += WORKERS) x[i] *= scale[p0 + i];
        // the next step takes right-hand sides that others have scaled
        asm volatile("bar.sync 1, %0;" ::"n"(WORKERS) : "memory");
      }
      fetch(q + 1);
    }
    __syncthreads();
  }
  if(late) {  // no result: the caller sees that it is not finite
    for(int i = tid; i < n; i += THREADS) z[perm[p0 + i]] = (V)NAN;
    if(warp == WARPS)  // the copies in flight
      for(int k = missing; k < min(ns, asked); ++k) bar_wait(full + k % STAGES, phase(k));
    return;
  }
  for(int i = tid; i < n; i += THREADS) z[perm[p0 + i]] = x[i];
}

// The packed values: L as it is, U divided by its row's diagonal, and the
// inverse diagonal by row.
template <typename V>
__global__ void k_ilu_pack(int64_t ne, const int32_t *__restrict__ pos, const int32_t *__restrict__ dpos,
                           const V *__restrict__ f, V *__restrict__ val, int64_t nrows,
                           const int32_t *__restrict__ rowDiag, V *__restrict__ scale)
{
  FE_PDL_ENTRY();
  for(int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < ne; e += (int64_t)gridDim.x * blockDim.x) {
    V v = pos[e] >= 0 ? f[pos[e]] : (V)0;
    if(pos[e] >= 0 && dpos[e] >= 0) v /= f[dpos[e]];
    val[e] = v;
  }
  for(int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nrows; q += (int64_t)gridDim.x * blockDim.x)
    scale[q] = (V)1 / f[rowDiag[q]];
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
  cudaFree(rowDiag_); cudaFree(scale_);
}

int IluStream::build(const std::vector<int32_t> &lia, const std::vector<int32_t> &lja,
                     const std::vector<int32_t> &ldiag, const std::vector<int32_t> &perm,
                     const std::vector<int32_t> &start, bool fp32, cudaStream_t s)
{
  s_ = s;
  fp32_ = fp32;
  // FENG_ILU_LATE_STEP=k: the copies of every block's step k count as late
  if(const char *e = std::getenv("FENG_ILU_LATE_STEP")) lateStep_ = std::atoi(e);
  nBlocks_ = (int64_t)start.size() - 1;
  const size_t vs = fp32 ? sizeof(float) : sizeof(double);
  const size_t stages = STAGES * (fp32 ? sizeof(Stage<float>) : sizeof(Stage<double>));
  const int64_t n = (int64_t)perm.size();
  for(int64_t b = 0; b < nBlocks_; ++b) {
    const int64_t rows = start[b + 1] - start[b];
    if(rows >= (int64_t)NO_ROW || stages + rows * vs > MAX_SMEM) return FE_OK;  // the level kernels
  }
  // the vector's order: a block's rows by levels of L, so that the rows of a
  // warp read neighbouring entries (fewer bank conflicts)
  std::vector<int32_t> local(n), order(n);
  std::vector<Step> steps;
  std::vector<int32_t> stepStart(1, 0), pos, dpos, rowDiag(n), level(n, 0);
  std::vector<uint4> col;
  pos.reserve(2 * lja.size());
  dpos.reserve(2 * lja.size());
  col.reserve(6 * (size_t)n);
  std::vector<int32_t> cnt, ord;
  // a warp of a level: rows ord[first] .. ord[first + rows - 1], `slots` each
  struct Warp {
    int32_t first, rows, slots, chain;
  };
  std::vector<Warp> warps;
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
      auto len = [&](int32_t i) { return lower ? ldiag[i] - lia[i] : lia[i + 1] - ldiag[i] - 1; };
      for(int32_t l = 0; l < nl; ++l)  // rows of similar length together
        std::stable_sort(ord.begin() + cnt[l], ord.begin() + cnt[l + 1],
                         [&](int32_t x, int32_t y) { return len(x) > len(y); });
      if(lower)
        for(int32_t q = 0; q < p1 - p0; ++q) {
          order[p0 + q] = ord[q];
          local[ord[q]] = q;
          rowDiag[p0 + q] = ldiag[ord[q]];
        }
      for(int32_t l = 0; l < nl; ++l) {
        warps.clear();
        for(int32_t r0 = cnt[l]; r0 < cnt[l + 1];) {
          const int slots = len(ord[r0]) > LONG_ROW ? LONG_SLOTS : 2;
          int32_t r1 = r0 + 1;
          while(r1 < cnt[l + 1] && r1 - r0 < 32 / slots && (slots == 2 || len(ord[r1]) > LONG_ROW)) ++r1;
          warps.push_back({r0, r1 - r0, slots, (len(ord[r0]) + slots - 1) / slots});
          r0 = r1;
        }
        std::stable_sort(warps.begin(), warps.end(), [](const Warp &x, const Warp &y) { return x.chain > y.chain; });
        for(size_t w0 = 0; w0 < warps.size(); w0 += WARPS) {
          const int nw = (int)std::min<size_t>(WARPS, warps.size() - w0);
          const int chunks = std::max(1, (warps[w0].chain + E - 1) / E);
          for(int c = 0; c < chunks; ++c) {
            Step st = {};
            st.entry = (int32_t)pos.size();
            st.slot = (int32_t)col.size();
            st.warps = (uint8_t)nw;
            st.flags = (uint8_t)((c == 0 ? STEP_FIRST : 0) | (c + 1 == chunks ? STEP_LAST : 0));
            for(int w = 0; w < nw; ++w)
              if(warps[w0 + w].slots != 2) st.wide |= (uint8_t)(1u << w);
            // row, first entry and end of lane t of warp w (row -1: none)
            auto lane = [&](int w, int t, int32_t &i, int32_t &e, int32_t &end, int &slots) {
              const Warp &W = warps[w0 + w];
              slots = W.slots;
              i = t / slots < W.rows ? ord[W.first + t / slots] : -1;
              e = i < 0 ? 0 : (lower ? lia[i] : ldiag[i] + 1) + slots * c * E + t % slots;
              end = i < 0 ? 0 : (lower ? ldiag[i] : lia[i + 1]);
            };
            for(int w = 0; w < nw; ++w)
              st.chains |= (uint32_t)std::max(0, std::min<int>(E, warps[w0 + w].chain - c * E)) << (4 * w);
            for(int k = 0; k < E; ++k) {
              int g = 0;
              while(g < nw && warps[w0 + g].chain > c * E + k) ++g;
              for(int t = 0; t < 32 * g; ++t) {
                int32_t i, e, end;
                int slots;
                lane(t / 32, t % 32, i, e, end, slots);
                const bool ok = i >= 0 && e + slots * k < end;
                pos.push_back(ok ? e + slots * k : -1);
                dpos.push_back(ok && !lower ? ldiag[i] : -1);
              }
            }
            for(int t = 0; t < 32 * nw; ++t) {
              int32_t i, e, end;
              int slots;
              lane(t / 32, t % 32, i, e, end, slots);
              uint32_t w[4] = {0, 0, 0, (i >= 0 ? (uint32_t)local[i] : NO_ROW) << 16};
              for(int k = 0; k < E && i >= 0; ++k) {
                // padding (value 0) reads the row's own entry of the vector
                const int32_t j = e + slots * k < end ? local[lja[e + slots * k]] : local[i];
                w[k >> 1] |= (uint32_t)j << (16 * (k & 1));
              }
              col.push_back(make_uint4(w[0], w[1], w[2], w[3]));
            }
            steps.push_back(st);
          }
        }
      }
      // between the triangles a step without rows, which scales the vector
      if(lower) {
        steps.push_back(Step{});
        steps.back().flags = STEP_SCALE;
      }
    }
    stepStart.push_back((int32_t)steps.size());
    const int32_t own = stepStart[b + 1] - stepStart[b];
    const size_t need = stages + (((size_t)(p1 - p0) * vs + 15) & ~(size_t)15) + (size_t)own * sizeof(Step);
    if(own > MAX_STEPS || need > MAX_SMEM || pos.size() > (size_t)INT32_MAX / 2) return FE_OK;
    smem_ = std::max(smem_, need);
  }
  nEntries_ = (int64_t)pos.size();
  nRows_ = n;
  FE_TRY(to_device(&steps_, steps));
  FE_TRY(to_device(&stepStart_, stepStart));
  FE_TRY(to_device(&start_, start));
  FE_TRY(to_device(&perm_, order));
  FE_TRY(to_device(&col_, col));
  FE_TRY(to_device(&pos_, pos));
  FE_TRY(to_device(&dpos_, dpos));
  FE_TRY(to_device(&rowDiag_, rowDiag));
  CKI(cudaMalloc(&val_, vs * std::max<int64_t>(1, nEntries_)));
  CKI(cudaMalloc(&scale_, vs * std::max<int64_t>(1, nRows_)));
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
    ::feng::launch_k(k_ilu_pack<float>, g, 256, 0, s_, nEntries_, pos_, dpos_, (const float *)f, (float *)val_, nRows_,
                     rowDiag_, (float *)scale_);
  else
    ::feng::launch_k(k_ilu_pack<double>, g, 256, 0, s_, nEntries_, pos_, dpos_, (const double *)f, (double *)val_,
                     nRows_, rowDiag_, (double *)scale_);
}

template <typename V>
void IluStream::launch(const V *r, V *z, const int *done) const
{
  ::feng::launch_k(k_ilu_stream<V>, (int)nBlocks_, THREADS, smem_, s_, steps_, stepStart_, start_, perm_, col_,
                   (const V *)val_, (const V *)scale_, r, z, done, lateStep_);
}

void IluStream::solve(const float *r, float *z, const int *done) const { launch<float>(r, z, done); }
void IluStream::solve(const double *r, double *z, const int *done) const { launch<double>(r, z, done); }

}  // namespace feng
