// Triangular solves with the vector in shared memory (see fe_ilu_stream.h).
#include "fe_ilu_stream.h"

#include <algorithm>
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
constexpr unsigned NO_ROW = 0xffffu;
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
// diffusion (16 k rows, 254 levels per triangle): 0.33 ms per application; six
// products in a chain and copies by half of the threads 0.42, a warp per row
// and the vector in global memory 3.75.
// MANY: more than one block.  The copying warp's lanes then meet after their
// wait: apart they take issue slots from the SM's other blocks (256 x 256
// Kovasznay, blocks of 256 rows, FP64 434 -> 360 us, FP32 357 -> 307); alone on
// its SM a block is faster without (329 against 335, 243 against 257).
template <typename V, bool MANY>
__global__ void __launch_bounds__(THREADS) k_ilu_stream(const IluStream::Step *__restrict__ steps,
                                                        const int32_t *__restrict__ stepStart,
                                                        const int32_t *__restrict__ start,
                                                        const int32_t *__restrict__ perm,
                                                        const uint4 *__restrict__ col, const V *__restrict__ val,
                                                        const V *__restrict__ scale, const V *r,
                                                        V *__restrict__ z,
                                                        const int *done, int lateStep)
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
  __shared__ uint64_t full[STAGES];
  // A copy did not come.  The solving threads run on (to ask at each step costs 4
  // to 9% of an application, as a flag or in the barrier): a stage's columns hold
  // indices of the block at any time, those set here or an earlier step's.
  __shared__ volatile int late;
  if(tid == 0) {
    late = 0;
    for(int k = 0; k < STAGES; ++k) bar_init(full + k);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for(int i = tid; i < STAGES * WORKERS; i += THREADS)
    stage[i / WORKERS].col[i % WORKERS] = make_uint4(0, 0, 0, NO_ROW << 16);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the copies come after
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
  // the copying warp: lane k < E brings the warps' entries k, lane E the columns.
  // Steps below `asked` have been asked for; a copy that did not come ends that.
  int asked = 0;
  auto copy = [&](int q) {
    if(q >= ns) return;
    const IluStream::Step s = st[q];
    if(late) return;
    asked = q + 1;
    Stage<V> &g = stage[q % STAGES];
    const int pre = lane <= E ? lane : E;
    int before = 0, own = 0;  // warps with an entry j < pre, with entry lane
    const unsigned lanes = s.lanes;
#pragma unroll
    for(int j = 0; j < E; ++j) {
      // nibbles (at most E) above j
      const int c = __popc((s.chains + (7u - j) * 0x11111111u) & 0x88888888u);
      before += j < pre ? c : 0;
      own = j == lane ? c : own;
    }
    const void *src = val + s.entry + (int)lanes * before;
    void *dst = &g.val[lane < E ? lane : 0][0];
    unsigned bytes = lane < E ? lanes * own * (unsigned)sizeof(V) : 0u;
    if(lane == E) {
      src = col + s.slot;
      dst = &g.col[0];
      bytes = lanes * s.warps * 16u;
      bar_expect(full + q % STAGES, bytes + lanes * before * (unsigned)sizeof(V));
    }
    __syncwarp();
    if(bytes) bulk_copy(dst, src, bytes, full + q % STAGES);
  };
  auto phase = [](int q) { return (unsigned)(q / STAGES) & 1u; };
  // until step q's operands are there; the barrier that follows tells the others
  // (lateStep: a step that counts as late, to test what follows)
  auto arrived = [&](int q) {
    if(q < asked && (q == lateStep || !bar_wait(full + q % STAGES, phase(q)))) late = 1;
    if constexpr(MANY) __syncwarp();
  };
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
#pragma unroll
    for(int k = 0; k < E; ++k) load_if(k < (int)((s.chains >> (4 * warp)) & 15), &g.val[k][tid], v[k]);
    const unsigned row = c4.w >> 16;
    const int last = (s.wide >> warp) & 1 ? LONG_SLOTS - 1 : 1;
    const V own = x[row != NO_ROW ? row : 0];
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
  for(int q = 0; q < ns; ++q) {
    if(warp == WARPS) {
      copy(q + STAGES);  // into the stage of this step, whose operands are in registers
      arrived(q + 2);
    } else if(warp < s.warps) {
      const unsigned cw[4] = {c4.x, c4.y, c4.z, c4.w};
      const unsigned row = c4.w >> 16;
      const int chain = (s.chains >> (4 * warp)) & 15;
      const bool wide = (s.wide >> warp) & 1, end = s.flags & STEP_LAST, stored = lane < s.lanes;
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
        if(stored && row != NO_ROW && !(tid & (wide ? LONG_SLOTS - 1 : 1))) x[row] = acc;
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
      for(int k = max(0, asked - STAGES); k < asked; ++k) bar_wait(full + k % STAGES, phase(k));
    return;
  }
  for(int i = tid; i < n; i += THREADS) z[perm[p0 + i]] = x[i];
}

// The packed values: L as it is, U divided by its row's diagonal, and the
// inverse diagonal by row.  A warp per step (and warp of the step, grid y),
// which finds the factor's entries from the rows of its slots.
template <typename V>
__global__ void __launch_bounds__(256) k_ilu_pack(int64_t nSteps, const IluStream::Step *__restrict__ steps,
                                                  const int2 *__restrict__ from, const uint4 *__restrict__ col,
                                                  const int32_t *__restrict__ perm, const int32_t *__restrict__ lia,
                                                  const int32_t *__restrict__ ldiag, const V *f,
                                                  V *__restrict__ val, int64_t nRows, V *__restrict__ scale)
{
  FE_PDL_ENTRY();
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(blockIdx.y == 0)
    for(int64_t q = t; q < nRows; q += (int64_t)gridDim.x * blockDim.x) scale[q] = (V)1 / f[ldiag[perm[q]]];
  const int64_t q = t >> 5;
  if(q >= nSteps) return;
  const IluStream::Step s = steps[q];
  const int w = blockIdx.y, lane = (int)(t & 31);
  if(w >= s.warps || lane >= s.lanes) return;
  const int2 at = from[q];  // the block's first row, the step's chunk of its rows (odd: of L)
  const bool lower = at.y & 1;
  const int slots = (s.wide >> w) & 1 ? LONG_SLOTS : 2;
  const unsigned row = col[s.slot + 32 * w + lane].w >> 16;
  int32_t e = 0, end = 0;
  V inv = 1;
  if(row != NO_ROW) {
    const int32_t i = perm[at.x + (int)row], d = ldiag[i];
    e = (lower ? lia[i] : d + 1) + slots * (at.y >> 1) * E + lane % slots;
    end = lower ? d : lia[i + 1];
    if(!lower) inv = f[d];
  }
  int64_t dst = s.entry + 32 * w + lane;
  for(int k = 0; k < (int)((s.chains >> (4 * w)) & 15); ++k, e += slots) {
    V v = e < end ? f[e] : (V)0;
    if(e < end && !lower) v /= inv;
    val[dst] = v;
    for(int u = 0; u < WARPS; ++u) dst += ((s.chains >> (4 * u)) & 15) > k ? s.lanes : 0;
  }
}

template <typename T>
int to_device(T **dst, const std::vector<T> &v)
{
  CKI(cudaMalloc(dst, sizeof(T) * std::max<size_t>(1, v.size())));
  CKI(cudaMemcpy(*dst, v.data(), sizeof(T) * v.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

// The steps of some consecutive blocks.
struct Packed {
  std::vector<IluStream::Step> steps;
  std::vector<int2> from;          // k_ilu_pack
  std::vector<uint4> col;
  std::vector<int32_t> count;      // steps of each block
  int64_t entries = 0;
  size_t smem = 0;
  bool fits = true;
};

}  // namespace

IluStream::~IluStream()
{
  cudaFree(steps_); cudaFree(from_); cudaFree(stepStart_); cudaFree(start_); cudaFree(perm_);
  cudaFree(col_); cudaFree(val_); cudaFree(scale_);
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
  std::vector<int32_t> local(n), order(n), level(n, 0);
  auto pack = [&](int64_t b0, int64_t b1, Packed &P) {
    std::vector<int32_t> cnt, ord;
    // a warp of a level: rows ord[first] .. ord[first + rows - 1], `slots` each
    struct Warp {
      int32_t first, rows, slots, chain;
    };
    std::vector<Warp> warps;
    for(int64_t b = b0; b < b1 && P.fits; ++b) {
      const int32_t p0 = start[b], p1 = start[b + 1];
      const size_t first = P.steps.size();
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
            // a warp alone keeps the lanes that it uses (copies of 16 bytes)
            const int pad = 16 / (int)vs - 1, lanes = nw > 1 ? 32 : (warps[w0].rows * warps[w0].slots + pad) & ~pad;
            for(int c = 0; c < chunks; ++c) {
              Step st = {};
              st.entry = (int32_t)P.entries;
              st.slot = (int32_t)P.col.size();
              st.warps = (uint8_t)nw;
              st.lanes = (uint8_t)lanes;
              st.flags = (uint8_t)((c == 0 ? STEP_FIRST : 0) | (c + 1 == chunks ? STEP_LAST : 0));
              for(int w = 0; w < nw; ++w) {
                const Warp &W = warps[w0 + w];
                const int chain = std::max(0, std::min<int>(E, W.chain - c * E));
                if(W.slots != 2) st.wide |= (uint8_t)(1u << w);
                st.chains |= (uint32_t)chain << (4 * w);
                P.entries += chain * lanes;
                for(int t = 0; t < lanes; ++t) {
                  // row, first entry and end of the lane (row -1: none)
                  const int32_t i = t / W.slots < W.rows ? ord[W.first + t / W.slots] : -1;
                  const int32_t e = i < 0 ? 0 : (lower ? lia[i] : ldiag[i] + 1) + W.slots * c * E + t % W.slots;
                  const int32_t end = i < 0 ? 0 : (lower ? ldiag[i] : lia[i + 1]);
                  uint32_t x[4] = {0, 0, 0, (i >= 0 ? (uint32_t)local[i] : NO_ROW) << 16};
                  for(int k = 0; k < E && i >= 0; ++k) {
                    // padding (value 0) reads the row's own entry of the vector
                    const int32_t j = e + W.slots * k < end ? local[lja[e + W.slots * k]] : local[i];
                    x[k >> 1] |= (uint32_t)j << (16 * (k & 1));
                  }
                  P.col.push_back(make_uint4(x[0], x[1], x[2], x[3]));
                }
              }
              P.steps.push_back(st);
              P.from.push_back(make_int2(p0, 2 * c + lower));
            }
          }
        }
        // between the triangles a step without rows, which scales the vector
        if(lower) {
          P.steps.push_back(Step{});
          P.steps.back().flags = STEP_SCALE;
          P.from.push_back(make_int2(p0, 0));
        }
      }
      const size_t own = P.steps.size() - first;
      const size_t need = stages + (((size_t)(p1 - p0) * vs + 15) & ~(size_t)15) + own * sizeof(Step);
      P.count.push_back((int32_t)own);
      P.smem = std::max(P.smem, need);
      P.fits = own <= MAX_STEPS && need <= MAX_SMEM && P.entries <= INT32_MAX / 2;
    }
  };
  // blocks are independent: packed by ranges, side by side
  const int64_t parts = std::max<int64_t>(1, std::min<int64_t>(nBlocks_, 64));
  std::vector<Packed> P(parts);
  parallel_for(parts, [&](int64_t q0, int64_t q1) {
    for(int64_t q = q0; q < q1; ++q) pack(nBlocks_ * q / parts, nBlocks_ * (q + 1) / parts, P[q]);
  }, 1);
  size_t nCol = 0;
  nSteps_ = nEntries_ = 0;
  maxWarps_ = 1;
  std::vector<int32_t> stepStart(1, 0);
  for(Packed &p : P) {
    for(Step &st : p.steps) {
      st.entry += (int32_t)nEntries_;
      st.slot += (int32_t)nCol;
      maxWarps_ = std::max<int>(maxWarps_, st.warps);
    }
    for(int32_t c : p.count) stepStart.push_back(stepStart.back() + c);
    nSteps_ += (int64_t)p.steps.size();
    nEntries_ += p.entries;
    nCol += p.col.size();
    smem_ = std::max(smem_, p.smem);
    if(!p.fits || nEntries_ > INT32_MAX / 2) return FE_OK;
  }
  nRows_ = n;
  CKI(cudaMalloc(&steps_, sizeof(Step) * std::max<int64_t>(1, nSteps_)));
  CKI(cudaMalloc(&from_, sizeof(int2) * std::max<int64_t>(1, nSteps_)));
  CKI(cudaMalloc(&col_, sizeof(uint4) * std::max<size_t>(1, nCol)));
  size_t s0 = 0, c0 = 0;
  for(const Packed &p : P) {
    CKI(cudaMemcpy(steps_ + s0, p.steps.data(), sizeof(Step) * p.steps.size(), cudaMemcpyHostToDevice));
    CKI(cudaMemcpy(from_ + s0, p.from.data(), sizeof(int2) * p.from.size(), cudaMemcpyHostToDevice));
    CKI(cudaMemcpy(col_ + c0, p.col.data(), sizeof(uint4) * p.col.size(), cudaMemcpyHostToDevice));
    s0 += p.steps.size();
    c0 += p.col.size();
  }
  FE_TRY(to_device(&stepStart_, stepStart));
  FE_TRY(to_device(&start_, start));
  FE_TRY(to_device(&perm_, order));
  CKI(cudaMalloc(&val_, vs * std::max<int64_t>(1, nEntries_)));
  CKI(cudaMalloc(&scale_, vs * std::max<int64_t>(1, nRows_)));
  // the copies ran on the legacy stream, with which s is not ordered
  CKI(cudaStreamSynchronize(cudaStreamLegacy));
  const auto opt_in = [](auto kernel) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)MAX_SMEM);
  };
  if(fp32) CKI(nBlocks_ > 1 ? opt_in(k_ilu_stream<float, true>) : opt_in(k_ilu_stream<float, false>));
  else CKI(nBlocks_ > 1 ? opt_in(k_ilu_stream<double, true>) : opt_in(k_ilu_stream<double, false>));
  usable_ = true;
  return FE_OK;
}

void IluStream::gather(const void *f, const int32_t *lia, const int32_t *ldiag)
{
  const dim3 g((unsigned)std::max<int64_t>(1, (nSteps_ + 7) / 8), (unsigned)maxWarps_);
  auto go = [&](auto kernel, auto *v, auto *scale, auto *fv) {
    ::feng::launch_k(kernel, g, 256, 0, s_, nSteps_, steps_, from_, col_, perm_, lia, ldiag, fv, v, nRows_, scale);
  };
  if(fp32_) go(k_ilu_pack<float>, (float *)val_, (float *)scale_, (const float *)f);
  else go(k_ilu_pack<double>, (double *)val_, (double *)scale_, (const double *)f);
}

template <typename V>
void IluStream::launch(const V *r, V *z, const int *done) const
{
  auto kernel = nBlocks_ > 1 ? k_ilu_stream<V, true> : k_ilu_stream<V, false>;
  ::feng::launch_k(kernel, (int)nBlocks_, THREADS, smem_, s_, steps_, stepStart_, start_, perm_, col_,
                   (const V *)val_, (const V *)scale_, r, z, done, lateStep_);
}

void IluStream::solve(const float *r, float *z, const int *done) const { launch<float>(r, z, done); }
void IluStream::solve(const double *r, double *z, const int *done) const { launch<double>(r, z, done); }

}  // namespace feng
