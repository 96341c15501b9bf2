// Block-column sliced-ELL products (see fe_bsell.h).
#include "fe_bsell.h"

#include <algorithm>
#include <type_traits>
#include <vector>

#include "fe_common.h"
#include "fe_df.h"
#include "fe_launch.h"

namespace feng {

#define CKB(x)                                                                         \
  do {                                                                                 \
    cudaError_t _e = (x);                                                              \
    if(_e != cudaSuccess) {                                                            \
      set_error("CUDA error %s at %s:%d", cudaGetErrorString(_e), __FILE__, __LINE__); \
      return FE_CUDA_FAIL;                                                             \
    }                                                                                  \
  } while(0)

namespace {

enum Mode { MUL32 = 0, RESID32 = 1, RESID32_DF = 2, MUL64 = 3, RESID64 = 4 };

// Values per vector load of an entry of NV values: the widest of 16 bytes
// that divides it.
template <typename VA, int NV>
constexpr int vec_width()
{
  constexpr int most = 16 / (int)sizeof(VA);
  return NV % most == 0 ? most : NV % 2 == 0 ? 2 : 1;
}

template <typename VA, int W>
__device__ __forceinline__ void load_vec(const VA *p, VA *v)
{
  if constexpr(W == 1) {
    v[0] = __ldcs(p);
  } else if constexpr(sizeof(VA) == 4 && W == 4) {
    const float4 t = __ldcs(reinterpret_cast<const float4 *>(p));
    v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
  } else if constexpr(sizeof(VA) == 4) {
    const float2 t = __ldcs(reinterpret_cast<const float2 *>(p));
    v[0] = t.x; v[1] = t.y;
  } else {
    const double2 t = __ldcs(reinterpret_cast<const double2 *>(p));
    v[0] = t.x; v[1] = t.y;
  }
}

// NC consecutive entries of x from column c; VEC: c is even, one load for two.
template <int NC, bool VEC, typename X>
__device__ __forceinline__ void load_x(const X *__restrict__ x, int32_t c, X (&v)[NC])
{
  if constexpr(NC == 2 && VEC) {
    if constexpr(sizeof(X) == 4) {
      const float2 t = *reinterpret_cast<const float2 *>(x + c);
      v[0] = t.x; v[1] = t.y;
    } else if constexpr(std::is_same_v<X, float2>) {
      const float4 t = *reinterpret_cast<const float4 *>(x + c);
      v[0] = make_float2(t.x, t.y); v[1] = make_float2(t.z, t.w);
    } else {
      const double2 t = *reinterpret_cast<const double2 *>(x + c);
      v[0] = t.x; v[1] = t.y;
    }
  } else {
#pragma unroll
    for(int j = 0; j < NC; ++j) v[j] = x[c + j];
  }
}

__device__ __forceinline__ void madd(float &s, float a, float x) { s = fmaf(a, x, s); }
__device__ __forceinline__ void madd(double &s, double a, double x) { s = fma(a, x, s); }
__device__ __forceinline__ void madd(double &s, float a, double x) { s = fma((double)a, x, s); }
// a (x_hi + x_lo) exact in its leading part, added in double-float
__device__ __forceinline__ void madd(dfl &s, float a, float2 x)
{
  const float p = __fmul_rn(a, x.x);
  float e = __fmaf_rn(a, x.x, -p);
  e = __fmaf_rn(a, x.y, e);
  s = df_add(s, df_fast2(p, e));
}

// Adds the entries k0, k0 + st, ... below k1 of one lane (NR rows, NC columns
// each) to acc, UNR entries at a time, the next ones' columns and values
// loaded before the gathers of x of these (one memory latency per UNR).
// enter: called once the first entries are on their way; true ends the walk.
template <int NR, int NC, int UNR, bool VEC, typename VA, typename X, typename S, typename R>
__device__ __forceinline__ bool walk(const int32_t *__restrict__ col, const VA *__restrict__ val, int32_t k0,
                                     int32_t k1, int st, int lane, const X *x, S (&acc)[NR], R &&enter)
{
  constexpr int NV = NR * NC, W = vec_width<VA, NV>(), PL = NV / W;
  int32_t c[UNR];
  VA v[UNR][NV];
  auto load = [&](int32_t k) {
#pragma unroll
    for(int u = 0; u < UNR; ++u) {
      c[u] = -1;
      if(k + u * st < k1) {
        c[u] = __ldcs(col + ((int64_t)(k + u * st) << 5) + lane);
#pragma unroll
        for(int p = 0; p < PL; ++p)
          load_vec<VA, W>(val + ((((int64_t)(k + u * st) * PL + p) << 5) + lane) * W, &v[u][p * W]);
      }
    }
  };
  load(k0);
  if(enter()) return false;
  for(int32_t k = k0; k < k1; k += UNR * st) {
    int32_t cc[UNR];
    VA vc[UNR][NV];
#pragma unroll
    for(int u = 0; u < UNR; ++u) {
      cc[u] = c[u];
#pragma unroll
      for(int q = 0; q < NV; ++q) vc[u][q] = v[u][q];
    }
    load(k + UNR * st);
#pragma unroll
    for(int u = 0; u < UNR; ++u)
      if(cc[u] >= 0) {
        X xv[NC];
        load_x<NC, VEC, X>(x, cc[u], xv);
#pragma unroll
        for(int i = 0; i < NR; ++i)
#pragma unroll
          for(int j = 0; j < NC; ++j) madd(acc[i], vc[u][i * NC + j], xv[j]);
      }
  }
  return true;
}

__device__ __forceinline__ float add(float a, float b) { return a + b; }
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ dfl add(dfl a, dfl b) { return df_add(a, b); }
__device__ __forceinline__ float from_lane(float a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ double from_lane(double a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
__device__ __forceinline__ dfl from_lane(dfl a, int o)
{
  dfl r;
  r.hi = __shfl_xor_sync(0xffffffffu, a.hi, o);
  r.lo = __shfl_xor_sync(0xffffffffu, a.lo, o);
  return r;
}

// Entries in flight per thread: about 20 registers of them.
template <typename VA, int NV>
constexpr int unroll()
{
  constexpr int words = NV * (int)sizeof(VA) / 4 + 1;
  return words <= 2 ? 8 : words <= 5 ? 4 : words <= 10 ? 2 : 1;
}

template <int NR, int D, bool VEC, typename VA, typename X, typename S, typename R>
__device__ __forceinline__ bool group_sum(const BlockSell::Part &P, int64_t g, int sub, int lanes, const X *x,
                                          S (&acc)[NR], R &&enter)
{
  const int64_t sl = g >> 5;
  const int lane = (int)(g & 31);
  auto entered = [] { return false; };
  if constexpr(D > 1) {
    if(!walk<NR, D, unroll<VA, NR * D>(), VEC, VA, X, S>(P.pCol, (const VA *)P.pVal, P.pPtr[sl] + sub, P.pPtr[sl + 1],
                                                         lanes, lane, x, acc, enter))
      return false;
    walk<NR, 1, unroll<VA, NR>(), false, VA, X, S>(P.sCol, (const VA *)P.sVal, P.sPtr[sl] + sub, P.sPtr[sl + 1], lanes,
                                                   lane, x, acc, entered);
  } else {
    if(!walk<NR, 1, unroll<VA, NR>(), false, VA, X, S>(P.sCol, (const VA *)P.sVal, P.sPtr[sl] + sub, P.sPtr[sl + 1],
                                                       lanes, lane, x, acc, enter))
      return false;
  }
  for(int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
    for(int i = 0; i < NR; ++i) acc[i] = add(acc[i], from_lane(acc[i], o));
  return true;
}

template <typename S>
__device__ __forceinline__ S zero_of()
{
  if constexpr(std::is_same_v<S, dfl>) return df_zero();
  else return (S)0;
}

// y = A x or b - A x, `lanes` (a power of two) threads per row group, each
// taking every lanes-th entry; the single rows' blocks come
// first (pressure rows, whose groups are as long as a vertex node's).
// Bound: HBM, the layout's bytes (88 MB for the FP32 Jacobian of the 256 x
// 256 Kovasznay case against 143 MB with a column per entry, 21.8 us cold
// against 26.3 us; 32^3 cube 65 us against 116 us); in FP64 the FP64 pipe (one
// product per entry, no lane sums) and the bytes about equally: 41 us against
// 82 us with eight lanes per CSR row.
template <int MODE, int D, bool VEC, typename VA, typename X, typename Y>
__global__ void __launch_bounds__(256) k_bsell(BlockSell::Part grp, BlockSell::Part one, int lanes,
                                               const X *x, const double *b, Y *__restrict__ y, const int *done)
{
  // within an iteration (done non-null: the kernel before has not written the
  // matrix) the first entries are read before the entry
  if(!done) FE_PDL_ENTRY();
  auto enter = [&] {
    if(!done) return false;
    FE_PDL_ENTRY();
    return *done != 0;
  };
  using S = std::conditional_t<MODE == MUL32, float, std::conditional_t<MODE == RESID32_DF, dfl, double>>;
  auto put = [&](int64_t row, S s) {
    if constexpr(MODE == MUL32 || MODE == MUL64) y[row] = s;
    else if constexpr(MODE == RESID32_DF) y[row] = b[row] - df_to(s);
    else y[row] = b[row] - s;
  };
  const int64_t ob = (one.n * lanes + 255) >> 8;
  const int sub = threadIdx.x & (lanes - 1);
  // groups past the end repeat the last one, so that the lane sums run with
  // full warps
  if((int64_t)blockIdx.x < ob) {
    const int64_t t = ((int64_t)blockIdx.x * 256 + threadIdx.x) / lanes, g = t < one.n ? t : one.n - 1;
    S acc[1] = {zero_of<S>()};
    if(!group_sum<1, D, VEC, VA, X, S>(one, g, sub, lanes, x, acc, enter)) return;
    if(t == g && sub == 0) put(one.row[g], acc[0]);
    return;
  }
  if constexpr(D > 1) {
    const int64_t t = (((int64_t)blockIdx.x - ob) * 256 + threadIdx.x) / lanes, g = t < grp.n ? t : grp.n - 1;
    S acc[D];
#pragma unroll
    for(int i = 0; i < D; ++i) acc[i] = zero_of<S>();
    if(!group_sum<D, D, VEC, VA, X, S>(grp, g, sub, lanes, x, acc, enter)) return;
    if(t != g || sub != 0) return;
    const int64_t row = grp.row[g];
#pragma unroll
    for(int i = 0; i < D; ++i) put(row + i, acc[i]);
  }
}

// same[r] = 1 when rows r and r + 1 have the same columns
__global__ void k_same_next(int64_t n, const int32_t *__restrict__ ia, const int32_t *__restrict__ ja,
                            uint8_t *__restrict__ same)
{
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(r >= n) return;
  uint8_t eq = 0;
  if(r + 1 < n) {
    const int32_t a = ia[r], b = ia[r + 1], len = b - a;
    eq = ia[r + 2] - b == len;
    for(int32_t k = 0; eq && k < len; ++k) eq = ja[a + k] == ja[b + k];
  }
  same[r] = eq;
}

// Whether the entry at k of a row ending at `end` starts a block of D columns.
__device__ __forceinline__ bool block_at(const int32_t *__restrict__ ja, const uint8_t *__restrict__ start, int D,
                                         int32_t k, int32_t end)
{
  return D > 1 && start[ja[k]] && k + D <= end && ja[k + D - 1] == ja[k] + D - 1;
}

// Entries of each group: block entries and single columns.
__global__ void k_count(int64_t n, const int32_t *__restrict__ row, const int32_t *__restrict__ ia,
                        const int32_t *__restrict__ ja, const uint8_t *__restrict__ start, int D, int2 *__restrict__ cnt)
{
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(g >= n) return;
  const int32_t end = ia[row[g] + 1];
  int2 c = make_int2(0, 0);
  for(int32_t k = ia[row[g]]; k < end;) {
    if(block_at(ja, start, D, k, end)) { ++c.x; k += D; }
    else { ++c.y; ++k; }
  }
  cnt[g] = c;
}

// Columns and row offsets of each group's entries; padding: offset -1 on the
// group's last column of that kind (any existing column).
__global__ void k_fill(BlockSell::Part P, const int32_t *__restrict__ ia, const int32_t *__restrict__ ja,
                       const uint8_t *__restrict__ start, int D)
{
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(g >= ((P.n + 31) & ~(int64_t)31)) return;
  const int64_t sl = g >> 5;
  const int lane = (int)(g & 31);
  int32_t kp = P.pPtr[sl], ks = P.sPtr[sl], cp = 0, cs = 0;
  if(g < P.n) {
    const int32_t beg = ia[P.row[g]], end = ia[P.row[g] + 1];
    for(int32_t k = beg; k < end;) {
      if(block_at(ja, start, D, k, end)) {
        const int64_t e = ((int64_t)kp++ << 5) + lane;
        P.pCol[e] = cp = ja[k];
        P.pOff[e] = k - beg;
        k += D;
      } else {
        const int64_t e = ((int64_t)ks++ << 5) + lane;
        P.sCol[e] = cs = ja[k];
        P.sOff[e] = k - beg;
        ++k;
      }
    }
  }
  for(; kp < P.pPtr[sl + 1]; ++kp) {
    P.pCol[((int64_t)kp << 5) + lane] = cp;
    P.pOff[((int64_t)kp << 5) + lane] = -1;
  }
  for(; ks < P.sPtr[sl + 1]; ++ks) {
    P.sCol[((int64_t)ks << 5) + lane] = cs;
    P.sOff[((int64_t)ks << 5) + lane] = -1;
  }
}

// The values of every entry from the CSR rows (padding: 0), one thread per
// group, the loads of four entries ahead of their stores (32^3 cube, two time
// steps with an entry at a time 40.2 ms, two 39.1, four 38.9).
template <int NR, int NC, typename VA>
__device__ __forceinline__ void gather_steps(const int32_t *__restrict__ off, VA *__restrict__ val, int32_t k0,
                                             int32_t k1, int lane, const VA *a, const int32_t (&beg)[NR])
{
  constexpr int NV = NR * NC, W = vec_width<VA, NV>(), PL = NV / W, U = 4;
  for(int32_t k = k0; k < k1; k += U) {
    int32_t o[U];
    VA v[U][NV];
#pragma unroll
    for(int u = 0; u < U; ++u) o[u] = k + u < k1 ? off[((int64_t)(k + u) << 5) + lane] : -1;
#pragma unroll
    for(int u = 0; u < U; ++u)
#pragma unroll
      for(int q = 0; q < NV; ++q) v[u][q] = o[u] >= 0 ? a[beg[q / NC] + o[u] + q % NC] : (VA)0;
#pragma unroll
    for(int u = 0; u < U; ++u)
      if(k + u < k1)
#pragma unroll
        for(int q = 0; q < NV; ++q) val[((((int64_t)(k + u) * PL + q / W) << 5) + lane) * W + q % W] = v[u][q];
  }
}

template <int NR, int D, typename VA>
__global__ void __launch_bounds__(256) k_bgather(BlockSell::Part P, const int32_t *__restrict__ ia,
                                                 const VA *a)
{
  FE_PDL_ENTRY();
  const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(g >= ((P.n + 31) & ~(int64_t)31)) return;
  const int64_t sl = g >> 5;
  const int lane = (int)(g & 31);
  int32_t beg[NR];
#pragma unroll
  for(int i = 0; i < NR; ++i) beg[i] = g < P.n ? ia[P.row[g] + i] : 0;
  if constexpr(D > 1)
    gather_steps<NR, D, VA>(P.pOff, (VA *)P.pVal, P.pPtr[sl], P.pPtr[sl + 1], lane, a, beg);
  gather_steps<NR, 1, VA>(P.sOff, (VA *)P.sVal, P.sPtr[sl], P.sPtr[sl + 1], lane, a, beg);
}

unsigned blocks_of(int64_t n) { return (unsigned)std::max<int64_t>(1, (n + 255) / 256); }

}  // namespace

BlockSell::~BlockSell()
{
  for(Part *P : {&grp_, &one_}) {
    cudaFree(P->row);
    cudaFree(P->pPtr); cudaFree(P->sPtr); cudaFree(P->pCol); cudaFree(P->sCol);
    cudaFree(P->pOff); cudaFree(P->sOff); cudaFree(P->pVal); cudaFree(P->sVal);
  }
}

// The slices of a set of row groups: entry counts on the device, the slices'
// lengths on the host (groups sorted by length within windows of a few
// thousand, so that a slice holds groups of one length and the gathers stay
// local), columns and offsets on the device.
int BlockSell::fill(Part &P, const std::vector<int32_t> &rows, const uint8_t *dStart)
{
  P.n = (int64_t)rows.size();
  const int64_t ns = (P.n + 31) / 32;
  CKB(cudaMalloc(&P.row, sizeof(int32_t) * std::max<int64_t>(1, P.n)));
  std::vector<int32_t> pp(ns + 1, 0), sp(ns + 1, 0);
  if(P.n > 0) {
    CKB(cudaMemcpyAsync(P.row, rows.data(), sizeof(int32_t) * P.n, cudaMemcpyHostToDevice, s_));
    int2 *dc = nullptr;
    CKB(cudaMalloc(&dc, sizeof(int2) * P.n));
    (k_count<<<blocks_of(P.n), 256, 0, s_>>>(P.n, P.row, A_.ia, A_.ja, dStart, D_, dc), ::feng::count_launch());
    std::vector<int2> cnt(P.n);
    cudaError_t e = cudaMemcpyAsync(cnt.data(), dc, sizeof(int2) * P.n, cudaMemcpyDeviceToHost, s_);
    if(e == cudaSuccess) e = cudaStreamSynchronize(s_);
    cudaFree(dc);
    CKB(e);
    constexpr int64_t WINDOW = 4096;
    std::vector<int32_t> ord(P.n), sorted(P.n);
    for(int64_t g = 0; g < P.n; ++g) ord[g] = (int32_t)g;
    parallel_for((P.n + WINDOW - 1) / WINDOW, [&](int64_t w0, int64_t w1) {
      for(int64_t w = w0; w < w1; ++w)
        std::stable_sort(ord.begin() + w * WINDOW, ord.begin() + std::min(P.n, (w + 1) * WINDOW),
                         [&](int32_t x, int32_t y) {
                           return cnt[x].x != cnt[y].x ? cnt[x].x > cnt[y].x : cnt[x].y > cnt[y].y;
                         });
    }, 4);
    int64_t ps = 0, ss = 0;
    for(int64_t sl = 0; sl < ns; ++sl) {
      int mp = 0, ms = 0;
      for(int64_t g = sl * 32; g < std::min(P.n, sl * 32 + 32); ++g) {
        mp = std::max(mp, cnt[ord[g]].x);
        ms = std::max(ms, cnt[ord[g]].y);
        sorted[g] = rows[ord[g]];
      }
      ps += mp;
      ss += ms;
      pp[sl + 1] = (int32_t)ps;
      sp[sl + 1] = (int32_t)ss;
    }
    P.pSteps = ps;
    P.sSteps = ss;
    CKB(cudaMemcpyAsync(P.row, sorted.data(), sizeof(int32_t) * P.n, cudaMemcpyHostToDevice, s_));
    CKB(cudaStreamSynchronize(s_));
  }
  const bool group = &P == &grp_;
  const size_t vs = (fp32_ ? sizeof(float) : sizeof(double)) * (group ? D_ : 1);
  const size_t pe = 32 * (size_t)std::max<int64_t>(1, P.pSteps), se = 32 * (size_t)std::max<int64_t>(1, P.sSteps);
  CKB(cudaMalloc(&P.pPtr, sizeof(int32_t) * (ns + 1)));
  CKB(cudaMalloc(&P.sPtr, sizeof(int32_t) * (ns + 1)));
  CKB(cudaMemcpyAsync(P.pPtr, pp.data(), sizeof(int32_t) * (ns + 1), cudaMemcpyHostToDevice, s_));
  CKB(cudaMemcpyAsync(P.sPtr, sp.data(), sizeof(int32_t) * (ns + 1), cudaMemcpyHostToDevice, s_));
  CKB(cudaMalloc(&P.pCol, sizeof(int32_t) * pe));
  CKB(cudaMalloc(&P.pOff, sizeof(int32_t) * pe));
  CKB(cudaMalloc(&P.sCol, sizeof(int32_t) * se));
  CKB(cudaMalloc(&P.sOff, sizeof(int32_t) * se));
  CKB(cudaMalloc(&P.pVal, vs * D_ * pe));
  CKB(cudaMalloc(&P.sVal, vs * se));
  if(P.n > 0)
    (k_fill<<<blocks_of((P.n + 31) / 32 * 32), 256, 0, s_>>>(P, A_.ia, A_.ja, dStart, D_), ::feng::count_launch());
  CKB(cudaGetLastError());
  CKB(cudaStreamSynchronize(s_));  // the host arrays of the copies go out of scope
  return FE_OK;
}

int BlockSell::build(const DeviceCSR &A, bool fp32, cudaStream_t s)
{
  A_ = A;
  s_ = s;
  fp32_ = fp32;
  const int64_t n = A.n;
  // the pattern was copied on the legacy stream, with which s (non-blocking)
  // is not ordered, and such a copy may return before it has reached the device
  CKB(cudaStreamSynchronize(cudaStreamLegacy));
  uint8_t *d = nullptr;
  CKB(cudaMalloc(&d, (size_t)std::max<int64_t>(1, n)));
  struct Free { uint8_t *p; ~Free() { cudaFree(p); } } guard{d};
  if(n > 0) (k_same_next<<<blocks_of(n), 256, 0, s>>>(n, A.ia, A.ja, d), ::feng::count_launch());
  std::vector<uint8_t> same(n);
  CKB(cudaMemcpyAsync(same.data(), d, (size_t)n, cudaMemcpyDeviceToHost, s));
  CKB(cudaStreamSynchronize(s));
  // D consecutive rows with equal columns form a group: the largest D that
  // groups at least half of the rows
  auto group = [&](int D, std::vector<int32_t> *grp, std::vector<int32_t> *one) {
    int64_t in = 0;
    for(int64_t r = 0; r < n;) {
      bool ok = D > 1 && r + D <= n;
      for(int i = 0; ok && i + 1 < D; ++i) ok = same[r + i];
      if(ok) {
        if(grp) grp->push_back((int32_t)r);
        r += D;
        in += D;
      } else {
        if(one) one->push_back((int32_t)r);
        ++r;
      }
    }
    return in;
  };
  D_ = 2 * group(3, nullptr, nullptr) >= n ? 3 : 2 * group(2, nullptr, nullptr) >= n ? 2 : 1;
  if(n == 0) D_ = 1;
  std::vector<int32_t> grp, one;
  group(D_, &grp, &one);
  std::vector<uint8_t> start(n, 0);
  even_ = D_ == 2;
  for(int32_t r : grp) {
    start[r] = 1;
    if(r & 1) even_ = false;
  }
  CKB(cudaMemcpyAsync(d, start.data(), (size_t)n, cudaMemcpyHostToDevice, s));
  FE_TRY(fill(grp_, grp, d));
  FE_TRY(fill(one_, one, d));
  // threads per group: at least a quarter of the 311 k resident threads of
  // the GPU (20^3 cube, 69 k groups: 27.0 ms per two time steps with two
  // threads against 28.1 ms with one; four times as many threads are no
  // faster)
  const int64_t groups = (int64_t)(grp.size() + one.size());
  lanes_ = 1;
  while(lanes_ < (fp32 ? 8 : 4) && groups * lanes_ < 75000) lanes_ *= 2;
  built_ = true;
  return FE_OK;
}

void BlockSell::gather(const void *vals)
{
  auto go = [&](auto kernel, const Part &P, auto *a) {
    if(P.n > 0) ::feng::launch_k(kernel, blocks_of((P.n + 31) / 32 * 32), 256, 0, s_, P, A_.ia, a);
  };
  if(fp32_) {
    const float *a = (const float *)vals;
    if(D_ == 3) { go(k_bgather<3, 3, float>, grp_, a); go(k_bgather<1, 3, float>, one_, a); }
    else if(D_ == 2) { go(k_bgather<2, 2, float>, grp_, a); go(k_bgather<1, 2, float>, one_, a); }
    else go(k_bgather<1, 1, float>, one_, a);
  } else {
    const double *a = (const double *)vals;
    if(D_ == 3) { go(k_bgather<3, 3, double>, grp_, a); go(k_bgather<1, 3, double>, one_, a); }
    else if(D_ == 2) { go(k_bgather<2, 2, double>, grp_, a); go(k_bgather<1, 2, double>, one_, a); }
    else go(k_bgather<1, 1, double>, one_, a);
  }
}

template <int MODE, typename VA, typename X, typename Y>
void BlockSell::launch(const X *x, const double *b, Y *y, const int *done) const
{
  const unsigned g = (unsigned)((one_.n * lanes_ + 255) / 256 + (grp_.n * lanes_ + 255) / 256);
  auto k = D_ == 3   ? k_bsell<MODE, 3, false, VA, X, Y>
           : D_ == 1 ? k_bsell<MODE, 1, false, VA, X, Y>
           : even_   ? k_bsell<MODE, 2, true, VA, X, Y>
                     : k_bsell<MODE, 2, false, VA, X, Y>;
  if(g > 0) ::feng::launch_k(k, g, 256, 0, s_, grp_, one_, lanes_, x, b, y, done);
}

void BlockSell::mul32(const float *x, float *y, const int *done) const
{
  launch<MUL32, float, float, float>(x, nullptr, y, done);
}

void BlockSell::resid32(const double *x, const double *b, double *r) const
{
  launch<RESID32, float, double, double>(x, b, r, nullptr);
}

void BlockSell::resid32_df(const float2 *xs, const double *b, double *r) const
{
  launch<RESID32_DF, float, float2, double>(xs, b, r, nullptr);
}

void BlockSell::mul64(const double *x, double *y, const int *done) const
{
  launch<MUL64, double, double, double>(x, nullptr, y, done);
}

void BlockSell::resid64(const double *x, const double *b, double *r) const
{
  launch<RESID64, double, double, double>(x, b, r, nullptr);
}

int64_t BlockSell::bytes() const
{
  const int64_t vs = fp32_ ? 4 : 8;
  auto of = [&](const Part &P, int64_t rows) {
    return 32 * (P.pSteps * (4 + rows * D_ * vs) + P.sSteps * (4 + rows * vs)) + (P.n + 31) / 32 * 8 + P.n * 4;
  };
  return of(grp_, D_) + of(one_, 1);
}

}  // namespace feng
