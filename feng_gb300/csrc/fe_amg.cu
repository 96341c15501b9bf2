// Device V-cycle of the smoothed-aggregation hierarchy (see fe_amg.h).
// Smoother degree 1 (damped Jacobi, the default): two kernels per level on
// the level's combined operators (AMGDevice::Lev: T, Q, Q^T).  Degree 2 to 6:
// Chebyshev smoothing on D^-1 A (polynomial, SpMV-only), residual,
// restriction, coarse correction, prolongation, Chebyshev again.  The
// coarsest level is a dense inverse applied as a mat-vec.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fe_amg.h"
#include "fe_common.h"
#include "fe_launch.h"

namespace feng {

#define CKA(x)                                                                         \
  do {                                                                                 \
    cudaError_t _e = (x);                                                              \
    if(_e != cudaSuccess) {                                                            \
      set_error("CUDA error %s at %s:%d", cudaGetErrorString(_e), __FILE__, __LINE__); \
      return FE_CUDA_FAIL;                                                             \
    }                                                                                  \
  } while(0)

namespace {

int grid(int64_t n, int per = 256) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + per - 1) / per, 1 << 20)); }

// Vectors hold NV interleaved components per row (NV = 2: both velocity
// components of a node share one pass over the matrix).
template <typename V, int NV>
struct Vals {
  V v[NV];
};

template <typename V, int NV>
__device__ __forceinline__ Vals<V, NV> ldv(const V *__restrict__ p, int64_t i)
{
  Vals<V, NV> r;
  if constexpr(NV == 2 && sizeof(V) == 4) {
    const float2 t = *reinterpret_cast<const float2 *>(p + 2 * i);
    r.v[0] = t.x;
    r.v[1] = t.y;
  } else if constexpr(NV == 2 && sizeof(V) == 8) {
    const double2 t = *reinterpret_cast<const double2 *>(p + 2 * i);
    r.v[0] = t.x;
    r.v[1] = t.y;
  } else {
#pragma unroll
    for(int c = 0; c < NV; ++c) r.v[c] = p[i * NV + c];
  }
  return r;
}

// Row dot products acc[c] = sum_k a[k] x[ja[k]][c] over LANES lanes per row
// (butterfly reduction: the sums are valid in every lane of the row).  The
// row is walked UNR segments of LANES entries at a time: the column indices
// and values of all UNR segments are loaded first (streaming: each matrix
// entry is used once per product), then the gathers of x.
template <typename V, int LANES, int NV>
__device__ __forceinline__ void row_dot(int32_t beg, int32_t end, int sub, const int32_t *__restrict__ ja,
                                        const V *__restrict__ a, const V *x, V (&acc)[NV])
{
  constexpr int UNR = LANES >= 8 ? 4 : 2;
#pragma unroll
  for(int c = 0; c < NV; ++c) acc[c] = 0;
  for(int32_t k0 = beg + sub; k0 < end; k0 += LANES * UNR) {
    int32_t j[UNR];
    V av[UNR];
#pragma unroll
    for(int u = 0; u < UNR; ++u) {
      const int32_t k = k0 + u * LANES;
      const bool ok = k < end;
      j[u] = ok ? __ldcs(ja + k) : -1;
      av[u] = ok ? __ldcs(a + k) : (V)0;
    }
#pragma unroll
    for(int u = 0; u < UNR; ++u)
      if(j[u] >= 0) {
        const Vals<V, NV> xv = ldv<V, NV>(x, j[u]);
#pragma unroll
        for(int c = 0; c < NV; ++c) acc[c] += av[u] * xv.v[c];
      }
  }
#pragma unroll
  for(int c = 0; c < NV; ++c)
#pragma unroll
    for(int o = LANES / 2; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o, LANES);
}

// Lane sums acc[c] = sum_k (a[k] w[ja[k]]) x[ja[k]][c] over the entries
// k = beg + sub, beg + sub + LANES, ... of a row (in that order; no
// reduction across the lanes), walked as row_dot: the column indices and
// values of UNR segments first, then their gathers.
template <typename V, int LANES, int NV>
__device__ __forceinline__ void row_dot_w(int32_t beg, int32_t end, int sub, const int32_t *__restrict__ ja,
                                          const V *__restrict__ a, const V *__restrict__ w,
                                          const V *x, V (&acc)[NV])
{
  constexpr int UNR = LANES >= 8 ? 4 : 2;
#pragma unroll
  for(int c = 0; c < NV; ++c) acc[c] = 0;
  for(int32_t k0 = beg + sub; k0 < end; k0 += LANES * UNR) {
    int32_t j[UNR];
    V av[UNR];
#pragma unroll
    for(int u = 0; u < UNR; ++u) {
      const int32_t k = k0 + u * LANES;
      const bool ok = k < end;
      j[u] = ok ? __ldcs(ja + k) : -1;
      av[u] = ok ? __ldcs(a + k) : (V)0;
    }
#pragma unroll
    for(int u = 0; u < UNR; ++u)
      if(j[u] >= 0) {
        const V ak = av[u] * w[j[u]];
        const Vals<V, NV> xv = ldv<V, NV>(x, j[u]);
#pragma unroll
        for(int c = 0; c < NV; ++c) acc[c] += ak * xv.v[c];
      }
  }
}

// y = A x (MODE 0), y += A x (MODE 2), y = A (b .* x) with b a per-row scale
// of x (MODE 3);
// csr_row: the LANES lanes of virtual thread t's row (row t / LANES).
template <typename V, int LANES, int MODE, int NV>
__device__ __forceinline__ void csr_row(int64_t t, int64_t n, const int32_t *__restrict__ ia,
                                        const int32_t *__restrict__ ja, const V *__restrict__ a,
                                        const V *x, const V *b, V *y)
{
  const int64_t row = t / LANES;
  const int sub = (int)(t % LANES);
  const bool live = row < n;
  const int32_t beg = live ? ia[row] : 0, end = live ? ia[row + 1] : 0;
  V acc[NV];
  if(MODE == 3) {
    row_dot_w<V, LANES, NV>(beg, end, sub, ja, a, b, x, acc);
#pragma unroll
    for(int c = 0; c < NV; ++c)
#pragma unroll
      for(int o = LANES / 2; o > 0; o >>= 1) acc[c] += __shfl_down_sync(0xffffffffu, acc[c], o, LANES);
  } else {
    row_dot<V, LANES, NV>(beg, end, sub, ja, a, x, acc);
  }
  if(live && sub == 0) {
#pragma unroll
    for(int c = 0; c < NV; ++c) {
      const int64_t o = row * NV + c;
      if(MODE == 0 || MODE == 3) y[o] = acc[c];
      else y[o] += acc[c];
    }
  }
}

template <typename V, int LANES, int MODE, int NV>
__global__ void __launch_bounds__(256) k_csr(int64_t n, const int32_t *__restrict__ ia,
                                             const int32_t *__restrict__ ja, const V *__restrict__ a,
                                             const V *x, const V *b,
                                             V *y, const int *skip)
{
  FE_PDL_ENTRY();
  if(skip && *skip) return;
  csr_row<V, LANES, MODE, NV>((int64_t)blockIdx.x * blockDim.x + threadIdx.x, n, ia, ja, a, x, b, y);
}

template <typename V, int MODE, int NV>
void csr(int lanes, int64_t n, const int32_t *ia, const int32_t *ja, const V *a, const V *x, const V *b,
         V *y, cudaStream_t s, const int *skip)
{
  const int g = grid(n * lanes);
  if(lanes == 8) ::feng::launch_k(k_csr<V, 8, MODE, NV>, g, 256, 0, s, n, ia, ja, a, x, b, y, skip);
  else if(lanes == 16) ::feng::launch_k(k_csr<V, 16, MODE, NV>, g, 256, 0, s, n, ia, ja, a, x, b, y, skip);
  else ::feng::launch_k(k_csr<V, 4, MODE, NV>, g, 256, 0, s, n, ia, ja, a, x, b, y, skip);
}

// Chebyshev start from a nonzero x: r = D^-1 (b - A x), d = r / theta.
template <typename V, int LANES, int NV>
__global__ void __launch_bounds__(256) k_cheb_restart(int64_t n, const int32_t *__restrict__ ia,
                                                      const int32_t *__restrict__ ja, const V *__restrict__ a,
                                                      const V *__restrict__ dinv, const V *b,
                                                      const V *x, V *__restrict__ r,
                                                      V *__restrict__ d, V inv_theta, const int *skip)
{
  FE_PDL_ENTRY();
  if(skip && *skip) return;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
  const int sub = threadIdx.x % LANES;
  const bool live = row < n;
  const int32_t beg = live ? ia[row] : 0, end = live ? ia[row + 1] : 0;
  V acc[NV];
  row_dot<V, LANES, NV>(beg, end, sub, ja, a, x, acc);
  if(live && sub == 0) {
    const V di = dinv[row];
#pragma unroll
    for(int c = 0; c < NV; ++c) {
      const int64_t o = row * NV + c;
      const V ri = di * (b[o] - acc[c]);
      r[o] = ri;
      d[o] = ri * inv_theta;
    }
  }
}

// One Chebyshev step: x += d; r -= D^-1 A d; dn = c1 d + c2 r.
template <typename V, int LANES, int NV>
__global__ void __launch_bounds__(256) k_cheb_step(int64_t n, const int32_t *__restrict__ ia,
                                                   const int32_t *__restrict__ ja, const V *__restrict__ a,
                                                   const V *__restrict__ dinv, const V *d,
                                                   V *__restrict__ dn, V *r,
                                                   V *x, V c1, V c2, const int *skip)
{
  FE_PDL_ENTRY();
  if(skip && *skip) return;
  const int64_t row = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / LANES;
  const int sub = threadIdx.x % LANES;
  const bool live = row < n;
  const int32_t beg = live ? ia[row] : 0, end = live ? ia[row + 1] : 0;
  V acc[NV];
  row_dot<V, LANES, NV>(beg, end, sub, ja, a, d, acc);
  if(live && sub < NV) {
    // lane c of the row updates component c
    const V dv = dinv[row];
    V ac = acc[0];
#pragma unroll
    for(int c = 1; c < NV; ++c)
      if(sub == c) ac = acc[c];
    const int64_t o = row * NV + sub;
    const V di = d[o];
    x[o] += di;
    const V ri = r[o] - dv * ac;
    r[o] = ri;
    dn[o] = c1 * di + c2 * ri;
  }
}

// Start from x = 0 fused with the first step: with d = D^-1 b / theta
// (formed on the fly for the neighbours), x = d, r = D^-1 b - D^-1 A d,
// dn = c1 d + c2 r.
template <typename V, int LANES, int NV>
__device__ __forceinline__ void cheb_first_row(int64_t t, int64_t n, const int32_t *__restrict__ ia,
                                               const int32_t *__restrict__ ja, const V *__restrict__ a,
                                               const V *__restrict__ dinv, const V *b,
                                               V *__restrict__ dn, V *r, V *x,
                                               V inv_theta, V c1, V c2)
{
  const int64_t row = t / LANES;
  const int sub = (int)(t % LANES);
  const bool live = row < n;
  const int32_t beg = live ? ia[row] : 0, end = live ? ia[row + 1] : 0;
  V acc[NV];
  row_dot_w<V, LANES, NV>(beg, end, sub, ja, a, dinv, b, acc);
#pragma unroll
  for(int c = 0; c < NV; ++c)
#pragma unroll
    for(int o = LANES / 2; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o, LANES);
  if(live && sub < NV) {
    const V dv = dinv[row];
    V ac = acc[0];
#pragma unroll
    for(int c = 1; c < NV; ++c)
      if(sub == c) ac = acc[c];
    const int64_t o = row * NV + sub;
    const V r0 = dv * b[o];
    const V di = r0 * inv_theta;
    x[o] = di;
    const V ri = r0 - dv * ac * inv_theta;
    r[o] = ri;
    dn[o] = c1 * di + c2 * ri;
  }
}

template <typename V, int LANES, int NV>
__global__ void __launch_bounds__(256) k_cheb_first(int64_t n, const int32_t *__restrict__ ia,
                                                    const int32_t *__restrict__ ja, const V *__restrict__ a,
                                                    const V *__restrict__ dinv, const V *b,
                                                    V *__restrict__ dn, V *__restrict__ r, V *__restrict__ x,
                                                    V inv_theta, V c1, V c2, const int *skip)
{
  FE_PDL_ENTRY();
  if(skip && *skip) return;
  cheb_first_row<V, LANES, NV>((int64_t)blockIdx.x * blockDim.x + threadIdx.x, n, ia, ja, a, dinv, b, dn, r, x,
                               inv_theta, c1, c2);
}

// Walks the len entries of row lane of a sliced-ELL slice (entry k at
// base + 32 k + lane) in order, calling f(column, value) for each, in steps
// of UNR entries, software-pipelined: the next step's columns and values are
// loaded before this step's gathers, so a step waits for one memory latency
// instead of two.
// enter: called once the first step's columns and values are on their way
// (early_entry); true ends the walk.
template <int UNR, typename V, typename F, typename R>
__device__ __forceinline__ bool sell_walk(int32_t base, int32_t len, int lane, const int32_t *__restrict__ sc,
                                          const V *__restrict__ sv, F &&f, R &&enter)
{
  int32_t c[UNR];
  V a[UNR];
#pragma unroll
  for(int u = 0; u < UNR; ++u) {
    const bool ok = u < len;
    const int32_t e = base + (u << 5) + lane;
    c[u] = ok ? __ldcs(sc + e) : -1;
    a[u] = ok ? __ldcs(sv + e) : (V)0;
  }
  if(enter()) return false;
  for(int32_t k = 0; k < len; k += UNR) {
    int32_t cn[UNR];
    V an[UNR];
#pragma unroll
    for(int u = 0; u < UNR; ++u) {
      const bool ok = k + UNR + u < len;
      const int32_t e = base + ((k + UNR + u) << 5) + lane;
      cn[u] = ok ? __ldcs(sc + e) : -1;
      an[u] = ok ? __ldcs(sv + e) : (V)0;
    }
#pragma unroll
    for(int u = 0; u < UNR; ++u)
      if(c[u] >= 0) f(c[u], a[u]);
#pragma unroll
    for(int u = 0; u < UNR; ++u) {
      c[u] = cn[u];
      a[u] = an[u];
    }
  }
  return true;
}
template <int UNR, typename V, typename F>
__device__ __forceinline__ void sell_walk(int32_t base, int32_t len, int lane, const int32_t *__restrict__ sc,
                                          const V *__restrict__ sv, F &&f)
{
  sell_walk<UNR, V>(base, len, lane, sc, sv, f, [] { return false; });
}

// A kernel of an iteration (skip non-null: the kernel before it has not
// written the operator) enters after its first operator loads, others at once.
// True: the iteration has ended.
__device__ __forceinline__ bool early_entry(const int *skip)
{
  if(!skip) return false;
  FE_PDL_ENTRY();
  return *skip != 0;
}

// k_cheb_first on the sliced-ELL copy of A: thread = row, both components.
template <typename V, int NV>
__global__ void __launch_bounds__(256) k_cheb_first_sell(int64_t n, const int32_t *__restrict__ sp,
                                                         const int32_t *__restrict__ sc, const V *__restrict__ sv,
                                                         const V *__restrict__ dinv, const V *b,
                                                         V *__restrict__ dn, V *__restrict__ r, V *__restrict__ x,
                                                         V inv_theta, V c1, V c2, const int *skip)
{
  FE_PDL_ENTRY();
  if(skip && *skip) return;
  const int64_t row = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(row >= n) return;
  const int64_t sl = row >> 5;
  const int lane = (int)(row & 31);
  const int32_t base = sp[sl], len = (sp[sl + 1] - base) >> 5;
  V acc[NV];
#pragma unroll
  for(int c = 0; c < NV; ++c) acc[c] = 0;
  sell_walk<8, V>(base, len, lane, sc, sv, [&](int32_t j, V a) {
    const V ak = a * dinv[j];
    const Vals<V, NV> bv = ldv<V, NV>(b, j);
#pragma unroll
    for(int c = 0; c < NV; ++c) acc[c] += ak * bv.v[c];
  });
  const V dv = dinv[row];
#pragma unroll
  for(int c = 0; c < NV; ++c) {
    const int64_t o = row * NV + c;
    const V r0 = dv * b[o];
    const V di = r0 * inv_theta;
    x[o] = di;
    const V ri = r0 - dv * acc[c] * inv_theta;
    r[o] = ri;
    dn[o] = c1 * di + c2 * ri;
  }
}

// Sum over the `lanes` lanes of a row (a power of two, 4 to 32) of
// acc[0..NV): on return every lane of the row holds the total of component
// (sub % 2) in acc[0] for NV = 2 (the even and odd lanes take one component
// each in the first exchange: half the additions of two butterflies, which on
// the FP64 pipe cost as much as the products), of every component for NV = 1
// and 3.
template <typename V, int NV>
__device__ __forceinline__ void lane_sum(int sub, int lanes, V (&acc)[NV])
{
  if constexpr(NV == 2) {
    const bool odd = sub & 1;
    const V give = odd ? acc[0] : acc[1];
    V keep = odd ? acc[1] : acc[0];
    keep += __shfl_xor_sync(0xffffffffu, give, 1);
    for(int o = lanes / 2; o > 1; o >>= 1) keep += __shfl_xor_sync(0xffffffffu, keep, o);
    acc[0] = keep;
  } else {
    for(int o = lanes / 2; o > 0; o >>= 1)
#pragma unroll
      for(int c = 0; c < NV; ++c) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
  }
}

// Lane sums of a CSR row over its lanes (no reduction) in steps of four
// segments, the columns and values of a step loaded before its gathers.
// FINE (the finest level): streaming loads, and the next step's columns and
// values loaded before this step's gathers; otherwise plain loads (a few MB
// read again by every cycle stay in the L2) and no such prefetch (most rows
// take one step: 5.2 us against 5.8 us per pass over 28.6 k rows).
template <typename V, int NV, bool FINE>
__device__ __forceinline__ bool row_part(int32_t beg, int32_t end, int sub, int lanes,
                                         const int32_t *__restrict__ ja, const V *__restrict__ a,
                                         const V *x, V (&acc)[NV], const int *skip)
{
  constexpr int UNR = 4;
  int32_t j[UNR];
  V av[UNR];
  auto load = [&](int32_t k0) {
#pragma unroll
    for(int u = 0; u < UNR; ++u) {
      const int32_t k = k0 + u * lanes;
      const bool ok = k < end;
      j[u] = ok ? (FINE ? __ldcs(ja + k) : __ldg(ja + k)) : -1;
      av[u] = ok ? (FINE ? __ldcs(a + k) : __ldg(a + k)) : (V)0;
    }
  };
  auto use = [&](const int32_t (&jc)[UNR], const V (&ac)[UNR]) {
#pragma unroll
    for(int u = 0; u < UNR; ++u)
      if(jc[u] >= 0) {
        const Vals<V, NV> xv = ldv<V, NV>(x, jc[u]);
#pragma unroll
        for(int c = 0; c < NV; ++c) acc[c] += ac[u] * xv.v[c];
      }
  };
#pragma unroll
  for(int c = 0; c < NV; ++c) acc[c] = 0;
  int32_t k0 = beg + sub;
  load(k0);
  if(early_entry(skip)) return false;
  if constexpr(FINE) {
    for(; k0 < end; k0 += lanes * UNR) {
      int32_t jc[UNR];
      V ac[UNR];
#pragma unroll
      for(int u = 0; u < UNR; ++u) {
        jc[u] = j[u];
        ac[u] = av[u];
      }
      load(k0 + lanes * UNR);
      use(jc, ac);
    }
  } else {
    while(k0 < end) {
      use(j, av);
      k0 += lanes * UNR;
      if(k0 < end) load(k0);
    }
  }
  return true;
}

// The component a lane writes after lane_sum, and its total; -1: none.
template <typename V, int NV>
__device__ __forceinline__ int lane_out(int sub, const V (&acc)[NV], V &v)
{
  if(sub >= NV) return -1;
  v = acc[0];
  if constexpr(NV == 3) v = sub == 0 ? acc[0] : sub == 1 ? acc[1] : acc[2];
  return sub;
}

// One level of the degree-1 V-cycle on the way down, both of its products
// with the level's right-hand side b in one launch: the leading blocks form
// the next right-hand side bc = Q^T b (lr lanes per coarse row: its rows
// hold 30 to 250 entries), the others s = T b, the smoothed part of the
// result that does not depend on the coarse levels (sliced ELL, thread =
// row, on a large finest level; lt lanes per row otherwise).
// Bound: the operators' bytes on the finest level (24 MB of T and 19 MB of
// Q^T at 256^2, FP32, two components: 18 us cold), launch latency on the
// coarse ones (5 to 8 us cold).  Against the four kernels per level of
// pre-smoothing, restriction, prolongation and post-smoothing (13 + 7 + 9 +
// 15 us on the finest level, four times 5 to 8 us on the next ones):
// Kovasznay 256^2 74.2 -> 65.0 ms mixed and 654 -> 560 ms FP64 per Newton
// solve, P2 diffusion 320^2 36.3 -> 26.3 ms, cavity 384^2 55.1 -> 50.6 ms and
// 32^3 cube 62.7 -> 58.0 ms per two steps.
template <typename V, int NV, bool SELL>
__global__ void __launch_bounds__(256) k_down(int lr, int lt, int64_t nc, const int32_t *__restrict__ ria,
                                              const int32_t *__restrict__ rja, const V *__restrict__ ra, int64_t n,
                                              const int32_t *__restrict__ tia, const int32_t *__restrict__ tja,
                                              const V *__restrict__ ta, const int32_t *__restrict__ trow,
                                              const V *b, V *__restrict__ bc, V *__restrict__ s, const int *skip)
{
  if(!skip) FE_PDL_ENTRY();
  const int64_t rBlocks = (nc * lr + 255) / 256;
  if((int64_t)blockIdx.x < rBlocks) {
    const int64_t row = ((int64_t)blockIdx.x * 256 + threadIdx.x) / lr;
    const int sub = threadIdx.x & (lr - 1);
    const bool live = row < nc;
    V acc[NV], v;
    if(!row_part<V, NV, SELL>(live ? ria[row] : 0, live ? ria[row + 1] : 0, sub, lr, rja, ra, b, acc, skip)) return;
    lane_sum<V, NV>(sub, lr, acc);
    const int c = lane_out<V, NV>(sub, acc, v);
    if(live && c >= 0) bc[row * NV + c] = v;
    return;
  }
  const int64_t t = ((int64_t)blockIdx.x - rBlocks) * 256 + threadIdx.x;
  if constexpr(SELL) {
    if(t >= n) return;
    const int64_t sl = t >> 5;
    const int32_t base = tia[sl], len = (tia[sl + 1] - base) >> 5;
    V acc[NV];
#pragma unroll
    for(int c = 0; c < NV; ++c) acc[c] = 0;
    if(!sell_walk<8, V>(
         base, len, (int)(t & 31), tja, ta,
         [&](int32_t j, V a) {
           const Vals<V, NV> bv = ldv<V, NV>(b, j);
#pragma unroll
           for(int c = 0; c < NV; ++c) acc[c] += a * bv.v[c];
         },
         [&] { return early_entry(skip); }))
      return;
#pragma unroll
    for(int c = 0; c < NV; ++c) s[(int64_t)trow[t] * NV + c] = acc[c];
  } else {
    const int64_t row = t / lt;
    const int sub = threadIdx.x & (lt - 1);
    const bool live = row < n;
    V acc[NV], v;
    if(!row_part<V, NV, false>(live ? tia[row] : 0, live ? tia[row + 1] : 0, sub, lt, tja, ta, b, acc, skip)) return;
    lane_sum<V, NV>(sub, lt, acc);
    const int c = lane_out<V, NV>(sub, acc, v);
    if(live && c >= 0) s[row * NV + c] = v;
  }
}

// The same level on the way up: x = s + Q xc.  OUT (the finest level of a
// cycle whose result goes straight to the caller's vector): component c of
// row i is written, times *scale, to z[om.dof(i, c)], and with the pressure
// fold the pressure rows come from the leading blocks (scheduled first,
// overlapping the rows).
template <typename V, int NV, bool SELL, bool OUT>
__global__ void __launch_bounds__(256) k_up(int lu, int64_t n, const int32_t *__restrict__ qia,
                                            const int32_t *__restrict__ qja, const V *__restrict__ qa,
                                            const int32_t *__restrict__ qrow, const V *xc, const V *s, V *x,
                                            const int *skip, AMGDevice::OutMap om)
{
  if(!skip) FE_PDL_ENTRY();
  int64_t blk = blockIdx.x;
  if constexpr(OUT) {
    const int64_t pBlocks = om.bgu ? (om.nP + 255) / 256 : 0;
    if(blk < pBlocks) {
      const int64_t k = blk * 256 + threadIdx.x;
      if(early_entry(skip) || k >= om.nP) return;
      const double c = *om.cr, cSc = om.consts[1], cMc = om.consts[2];
      const double shift = cMc > 0 ? c / cMc : 0., lift = cSc != 0. ? c / cSc : 0.;
      const int32_t i = om.pRows[k];
      const double rp = (double)((const V *)om.r)[i] - shift * om.pMass[k];
      ((V *)om.z)[i] = (V)((double)((const V *)om.pScale)[k] * rp + lift);
      return;
    }
    blk -= pBlocks;
  }
  const int64_t t = blk * 256 + threadIdx.x;
  // component c of row `row`, v = (Q xc)_row,c
  auto put = [&](int64_t row, int c, V v) {
    const int64_t o = row * NV + c;
    const V xo = s[o] + v;
    if constexpr(OUT) {
      const V xf = om.bgu ? xo - (V)*om.cr * ((const V *)om.bgu)[o] : xo;
      const int32_t d = om.dofC ? om.dofC[o] : c == 0 ? om.dofX[row] : om.dofY[row];
      ((V *)om.z)[d] = xf * (V)*om.scale;
    } else {
      x[o] = xo;
    }
  };
  if constexpr(SELL) {
    if(t >= n) return;
    const int64_t sl = t >> 5;
    const int32_t base = qia[sl], len = (qia[sl + 1] - base) >> 5;
    V acc[NV];
#pragma unroll
    for(int c = 0; c < NV; ++c) acc[c] = 0;
    if(!sell_walk<8, V>(
         base, len, (int)(t & 31), qja, qa,
         [&](int32_t j, V a) {
           const Vals<V, NV> xv = ldv<V, NV>(xc, j);
#pragma unroll
           for(int c = 0; c < NV; ++c) acc[c] += a * xv.v[c];
         },
         [&] { return early_entry(skip); }))
      return;
#pragma unroll
    for(int c = 0; c < NV; ++c) put(qrow[t], c, acc[c]);
  } else {
    const int64_t row = t / lu;
    const int sub = threadIdx.x & (lu - 1);
    const bool live = row < n;
    V acc[NV], v;
    if(!row_part<V, NV, false>(live ? qia[row] : 0, live ? qia[row + 1] : 0, sub, lu, qja, qa, xc, acc, skip)) return;
    lane_sum<V, NV>(sub, lu, acc);
    const int c = lane_out<V, NV>(sub, acc, v);
    if(live && c >= 0) put(row, c, v);
  }
}

// Last step of a smoothing whose residual is not needed afterwards: x += d
// only (the step's product with A would be discarded).
template <typename V>
__global__ void k_cheb_last(int64_t m, const V *d, V *x, const int *skip)
{
  FE_PDL_ENTRY();
  if(skip && *skip) return;
  for(int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    x[i] += d[i];
}

// x = Minv b for the coarsest level (dense, row-major): one block of
// DENSE_T threads per row, so that every load of the row is in flight at
// once; warp sums, then the warps' sums in order (deterministic).
constexpr int DENSE_T = 128;
template <typename V, int NV>
__global__ void __launch_bounds__(DENSE_T) k_dense(int64_t n, const V *__restrict__ M, const V *b,
                                                   V *__restrict__ x, const int *skip)
{
  if(!skip) FE_PDL_ENTRY();
  __shared__ V red[DENSE_T / 32][NV];
  const int64_t row = blockIdx.x;
  V acc[NV];
#pragma unroll
  for(int c = 0; c < NV; ++c) acc[c] = 0;
  constexpr int UNR = 4;
  V m[UNR];
  auto load = [&](int64_t k0) {
#pragma unroll
    for(int u = 0; u < UNR; ++u) m[u] = k0 + u * DENSE_T < n ? M[row * n + k0 + u * DENSE_T] : (V)0;
  };
  int64_t k0 = threadIdx.x;
  load(k0);
  if(early_entry(skip)) return;
  while(k0 < n) {
#pragma unroll
    for(int u = 0; u < UNR; ++u)
      if(k0 + u * DENSE_T < n)
#pragma unroll
        for(int c = 0; c < NV; ++c) acc[c] += m[u] * b[(k0 + u * DENSE_T) * NV + c];
    k0 += UNR * DENSE_T;
    if(k0 < n) load(k0);
  }
#pragma unroll
  for(int c = 0; c < NV; ++c) {
    for(int o = 16; o > 0; o >>= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][c] = acc[c];
  }
  __syncthreads();
  if(threadIdx.x < NV) {
    V t = red[0][threadIdx.x];
#pragma unroll
    for(int w = 1; w < DENSE_T / 32; ++w) t += red[w][threadIdx.x];
    x[row * NV + threadIdx.x] = t;
  }
}

template <typename V>
int upload_vec(void **dst, const std::vector<double> &src)
{
  std::vector<V> tmp(src.begin(), src.end());
  CKA(cudaMalloc(dst, sizeof(V) * std::max<size_t>(1, tmp.size())));
  CKA(cudaMemcpy(*dst, tmp.data(), sizeof(V) * tmp.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

int upload_idx(int32_t **dst, const std::vector<int64_t> &src)
{
  std::vector<int32_t> tmp(src.begin(), src.end());
  CKA(cudaMalloc(dst, sizeof(int32_t) * std::max<size_t>(1, tmp.size())));
  CKA(cudaMemcpy(*dst, tmp.data(), sizeof(int32_t) * tmp.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

int upload_idx(int32_t **dst, const std::vector<int32_t> &src)
{
  CKA(cudaMalloc(dst, sizeof(int32_t) * std::max<size_t>(1, src.size())));
  CKA(cudaMemcpy(*dst, src.data(), sizeof(int32_t) * src.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

// Row order of a sliced-ELL copy: the rows of every window of SORT_WINDOW
// rows by descending length (stable).  The nodes come in the order of their
// first element, so a slice of 32 mixes P2 vertex rows (19 entries) with edge
// rows (9) and would be padded to 19 throughout (11.4 entries on average);
// within a window of a few thousand rows the gathers stay local.
constexpr int64_t SORT_WINDOW = 4096;
std::vector<int32_t> sell_order(const HostCSR &A)
{
  std::vector<int32_t> o(A.n);
  for(int64_t i = 0; i < A.n; ++i) o[i] = (int32_t)i;
  parallel_for((A.n + SORT_WINDOW - 1) / SORT_WINDOW, [&](int64_t w0, int64_t w1) {
    for(int64_t w = w0; w < w1; ++w)
      std::stable_sort(o.begin() + w * SORT_WINDOW, o.begin() + std::min(A.n, (w + 1) * SORT_WINDOW),
                       [&](int32_t x, int32_t y) { return A.ia[x + 1] - A.ia[x] > A.ia[y + 1] - A.ia[y]; });
  }, 4);
  return o;
}

// A sliced-ELL copy of A (AMGDevice::Lev::sellPtr), its rows in the given
// order (null: ascending).
template <typename V>
int upload_sell(const HostCSR &A, const int32_t *order, int32_t **sellPtr, int32_t **sellCol, void **sellVal)
{
  const int64_t n = A.n, ns = (n + 31) / 32;
  const int64_t mcols = A.m > 0 ? A.m : n;
  auto row = [&](int64_t q) { return order && q < n ? (int64_t)order[q] : q; };
  std::vector<int32_t> ptr(ns + 1, 0);
  for(int64_t sl = 0; sl < ns; ++sl) {
    int64_t len = 0;
    for(int64_t q = sl * 32; q < std::min<int64_t>(n, sl * 32 + 32); ++q) {
      const int64_t r = row(q);
      len = std::max<int64_t>(len, A.ia[r + 1] - A.ia[r]);
    }
    if(ptr[sl] + 32 * len >= (int64_t)INT32_MAX) return FE_OK;  // keep the CSR kernels
    ptr[sl + 1] = (int32_t)(ptr[sl] + 32 * len);
  }
  std::vector<int32_t> col(std::max<int32_t>(ptr[ns], 1));
  std::vector<V> val(col.size(), (V)0);
  parallel_for(ns, [&](int64_t s0, int64_t s1) {
    for(int64_t sl = s0; sl < s1; ++sl) {
      const int32_t len = (ptr[sl + 1] - ptr[sl]) / 32;
      for(int lane = 0; lane < 32; ++lane) {
        const int64_t q = sl * 32 + lane, r = row(q);
        const int64_t own = q < n ? A.ia[r + 1] - A.ia[r] : 0;
        for(int32_t k = 0; k < len; ++k) {
          const int64_t e = ptr[sl] + (int64_t)k * 32 + lane;
          if(k < own) {
            col[e] = (int32_t)A.ja[A.ia[r] + k];
            val[e] = (V)A.a[A.ia[r] + k];
          } else {
            // padding: value 0 on an existing column
            col[e] = own > 0 ? A.ja[A.ia[r + 1] - 1] : (int32_t)std::min<int64_t>(q, mcols - 1);
            val[e] = (V)0;
          }
        }
      }
    }
  }, 256);
  CKA(cudaMalloc(sellPtr, sizeof(int32_t) * ptr.size()));
  CKA(cudaMalloc(sellCol, sizeof(int32_t) * col.size()));
  CKA(cudaMalloc(sellVal, sizeof(V) * val.size()));
  CKA(cudaMemcpy(*sellPtr, ptr.data(), sizeof(int32_t) * ptr.size(), cudaMemcpyHostToDevice));
  CKA(cudaMemcpy(*sellCol, col.data(), sizeof(int32_t) * col.size(), cudaMemcpyHostToDevice));
  CKA(cudaMemcpy(*sellVal, val.data(), sizeof(V) * val.size(), cudaMemcpyHostToDevice));
  return FE_OK;
}

int lanes_for(const HostCSR &M)
{
  const double avg = M.n ? (double)M.nnz() / M.n : 0;
  // 4 lanes per row on the P2 stiffness (~11 entries per row): 21 us per
  // finest smoother step against 27 us with 8 lanes
  return avg > 24 ? 16 : avg > 12 ? 8 : 4;
}

}  // namespace

AMGDevice::~AMGDevice()
{
  for(Lev &L : lv_) {
    cudaFree(L.Aia); cudaFree(L.Aja); cudaFree(L.Pia); cudaFree(L.Pja); cudaFree(L.Ria); cudaFree(L.Rja);
    cudaFree(L.Aa); cudaFree(L.Pa); cudaFree(L.Ra); cudaFree(L.dinv); cudaFree(L.diag);
    cudaFree(L.x); cudaFree(L.b); cudaFree(L.r); cudaFree(L.d0); cudaFree(L.d1);
    cudaFree(L.sellPtr); cudaFree(L.sellCol); cudaFree(L.sellVal);
    cudaFree(L.tPtr); cudaFree(L.tCol); cudaFree(L.tVal);
    cudaFree(L.qPtr); cudaFree(L.qCol); cudaFree(L.qVal);
    cudaFree(L.rPtr); cudaFree(L.rCol); cudaFree(L.rVal);
    cudaFree(L.tRow); cudaFree(L.qRow);
  }
  cudaFree(coarseInv_);
}

// The combined operators of a level (AMGDevice::Lev: T, Q, Q^T): with w = D^-1 / theta,
//   T = 2 w - w A w    (A's pattern),
//   Q = P - w (A P)    (the pattern of A P, which holds P's: A has a diagonal),
// so that the damped-Jacobi V-cycle of the level is b_c = Q^T b and
// x = T b + Q x_c: pre-smoothing x0 = w b, restriction P^T (b - A x0) =
// Q^T b (A symmetric), prolongation y = x0 + P x_c and post-smoothing
// y + w (b - A y) = T b + Q x_c.
int AMGDevice::upload_combined(const AMGLevel &h, Lev &L, bool fine, double theta)
{
  const int64_t n = h.A.n;
  std::vector<double> w(n);
  for(int64_t i = 0; i < n; ++i) w[i] = h.dinv[i] / theta;
  HostCSR T, Q;
  T.n = T.m = n;
  T.ia = h.A.ia;
  T.ja = h.A.ja;
  T.a.resize(h.A.a.size());
  Q.n = n;
  Q.m = h.P.m;
  Q.ia = h.AP.ia;
  Q.ja = h.AP.ja;
  Q.a.resize(h.AP.a.size());
  parallel_for(n, [&](int64_t r0, int64_t r1) {
    for(int64_t i = r0; i < r1; ++i) {
      for(int64_t k = h.A.ia[i]; k < h.A.ia[i + 1]; ++k) {
        const int32_t j = h.A.ja[k];
        T.a[k] = (j == i ? 2. * w[i] : 0.) - w[i] * h.A.a[k] * w[j];
      }
      // the columns of both rows ascend
      int64_t kp = h.P.ia[i];
      for(int64_t k = h.AP.ia[i]; k < h.AP.ia[i + 1]; ++k) {
        double v = -w[i] * h.AP.a[k];
        if(kp < h.P.ia[i + 1] && h.P.ja[kp] == h.AP.ja[k]) v += h.P.a[kp++];
        Q.a[k] = v;
      }
    }
  }, 4096);
  const HostCSR R = amg_transpose(Q);
  // Lanes per CSR row: enough threads to hide the latency of the loads (about
  // one wave of 2,048 threads on 152 SMs for the finest level's long rows,
  // two on the coarse levels, whose chains are shorter the more lanes share a
  // row; fewer in FP64, where the lane sums share the FP64 pipe with the
  // products), at most a lane for every two entries, 4 to 32.
  const int64_t room = !fp32_ ? 100000 : fine ? 300000 : 600000;
  auto lanes_of = [&](const HostCSR &M) {
    int l = 4;
    while(l < 32 && M.n * l * 2 <= room && M.nnz() >= M.n * l * 4) l *= 2;
    return l;
  };
  L.lanesR = lanes_of(R);
  L.lanesT = lanes_of(T);
  L.lanesQ = lanes_of(Q);
  auto csr_up = [&](const HostCSR &M, int32_t **ia, int32_t **ja, void **a) {
    FE_TRY(upload_idx(ia, M.ia));
    FE_TRY(upload_idx(ja, M.ja));
    return fp32_ ? upload_vec<float>(a, M.a) : upload_vec<double>(a, M.a);
  };
  FE_TRY(csr_up(R, &L.rPtr, &L.rCol, &L.rVal));
  L.nnzT = T.nnz();
  L.nnzR = R.nnz();
  if(fine && n >= 32 * 152) {
    const std::vector<int32_t> ot = sell_order(T), oq = sell_order(Q);
    FE_TRY(fp32_ ? upload_sell<float>(T, ot.data(), &L.tPtr, &L.tCol, &L.tVal)
                 : upload_sell<double>(T, ot.data(), &L.tPtr, &L.tCol, &L.tVal));
    if(L.tPtr)
      FE_TRY(fp32_ ? upload_sell<float>(Q, oq.data(), &L.qPtr, &L.qCol, &L.qVal)
                   : upload_sell<double>(Q, oq.data(), &L.qPtr, &L.qCol, &L.qVal));
    if(L.qPtr) {
      FE_TRY(upload_idx(&L.tRow, ot));
      FE_TRY(upload_idx(&L.qRow, oq));
      L.sellTQ = true;
      return FE_OK;
    }
    cudaFree(L.tPtr); cudaFree(L.tCol); cudaFree(L.tVal);
    L.tPtr = L.tCol = nullptr;
    L.tVal = nullptr;
  }
  FE_TRY(csr_up(T, &L.tPtr, &L.tCol, &L.tVal));
  return csr_up(Q, &L.qPtr, &L.qCol, &L.qVal);
}

int AMGDevice::upload(const AMGHierarchy &H, const AMGParams &p, int fp32, cudaStream_t s, bool keepA)
{
  p_ = p;
  fp32_ = fp32;
  s_ = s;
  const size_t vs = fp32 ? sizeof(float) : sizeof(double);
  const bool combined = p.chebyDegree == 1;
  lv_.resize(H.levels.size());
  n0_ = H.levels.empty() ? 0 : H.levels[0].A.n;
  diagSum_ = 0;
  for(int64_t i = 0; i < n0_; ++i) diagSum_ += 1.0 / H.levels[0].dinv[i];
  for(size_t l = 0; l < H.levels.size(); ++l) {
    const AMGLevel &h = H.levels[l];
    Lev &L = lv_[l];
    const bool coarsest = l + 1 == H.levels.size();
    L.n = h.A.n;
    L.lmax = h.lmax;
    L.lanesA = lanes_for(h.A);
    // the operator itself: the Chebyshev path, and products with the finest
    // one (spmv64 / spmv32)
    if(!combined || (l == 0 && keepA)) {
      FE_TRY(upload_idx(&L.Aia, h.A.ia));
      FE_TRY(upload_idx(&L.Aja, h.A.ja));
      FE_TRY(fp32 ? upload_vec<float>(&L.Aa, h.A.a) : upload_vec<double>(&L.Aa, h.A.a));
    }
    // room for up to three interleaved components per row
    for(void **v : {&L.x, &L.b, &L.r}) CKA(cudaMalloc(v, 3 * vs * std::max<int64_t>(1, L.n)));
    if(combined) {
      if(!coarsest) {
        L.nc = h.P.m;
        // damped Jacobi: theta = (low + high) / 2 of the smoothing interval
        FE_TRY(upload_combined(h, L, l == 0, 0.5 * (p.chebyLow * h.lmax + p.chebyHigh * h.lmax)));
      }
      continue;
    }
    for(void **v : {&L.d0, &L.d1}) CKA(cudaMalloc(v, 3 * vs * std::max<int64_t>(1, L.n)));
    if(l == 0 && h.A.n >= 32 * 152)
      FE_TRY(fp32 ? upload_sell<float>(h.A, nullptr, &L.sellPtr, &L.sellCol, &L.sellVal)
                  : upload_sell<double>(h.A, nullptr, &L.sellPtr, &L.sellCol, &L.sellVal));
    FE_TRY(fp32 ? upload_vec<float>(&L.dinv, h.dinv) : upload_vec<double>(&L.dinv, h.dinv));
    std::vector<double> dg(h.dinv.size());
    for(size_t i = 0; i < dg.size(); ++i) dg[i] = 1.0 / h.dinv[i];
    FE_TRY(fp32 ? upload_vec<float>(&L.diag, dg) : upload_vec<double>(&L.diag, dg));
    if(!coarsest) {
      L.nc = h.P.m;
      L.lanesP = lanes_for(h.P);
      L.lanesR = lanes_for(h.R);
      FE_TRY(upload_idx(&L.Pia, h.P.ia));
      FE_TRY(upload_idx(&L.Pja, h.P.ja));
      FE_TRY(fp32 ? upload_vec<float>(&L.Pa, h.P.a) : upload_vec<double>(&L.Pa, h.P.a));
      FE_TRY(upload_idx(&L.Ria, h.R.ia));
      FE_TRY(upload_idx(&L.Rja, h.R.ja));
      FE_TRY(fp32 ? upload_vec<float>(&L.Ra, h.R.a) : upload_vec<double>(&L.Ra, h.R.a));
    }
  }
  nCoarse_ = lv_.empty() ? 0 : lv_.back().n;
  nnz0_ = H.levels.empty() ? 0 : H.levels[0].A.nnz();
  FE_TRY(fp32 ? upload_vec<float>(&coarseInv_, H.coarseInv) : upload_vec<double>(&coarseInv_, H.coarseInv));
  // the copies ran on the legacy stream, with which s (non-blocking) is not
  // ordered, and one may return before it has reached the device
  CKA(cudaStreamSynchronize(cudaStreamLegacy));
  return FE_OK;
}

// needResidual: r = D^-1 (b - A x) must hold for the final x (the
// pre-smoothing, whose residual is restricted); otherwise the last step only
// moves x.
template <typename V, int NV>
static void chebyshev(int lanes, int64_t n, const int32_t *ia, const int32_t *ja, const V *a, const int32_t *sp,
                      const int32_t *sc, const V *sv, const V *dinv, const V *b, V *x, V *r, V *d0, V *d1,
                      double lmax, const AMGParams &p, bool zeroStart, bool needResidual, cudaStream_t s,
                      const int *skip)
{
  // Chebyshev iteration on D^-1 A over [low, high] * lmax (Saad, Alg. 12.1).
  const double lo = p.chebyLow * lmax, hi = p.chebyHigh * lmax;
  const double theta = 0.5 * (hi + lo), delta = 0.5 * (hi - lo), sigma = theta / delta;
  double rho = 1.0 / sigma;
  const int g = grid(n * lanes);
  int k0 = 0;
  V *d = d0, *dn = d1;
  if(zeroStart) {
    // start + first step in one pass
    const double rhoN = 1.0 / (2.0 * sigma - rho);
    const V c1 = (V)(rhoN * rho), c2 = (V)(2.0 * rhoN / delta);
    const V it = (V)(1.0 / theta);
    if(sp) ::feng::launch_k(k_cheb_first_sell<V, NV>, grid(n), 256, 0, s, n, sp, sc, sv, dinv, b, dn, r, x, it, c1, c2, skip);
    else if(lanes == 16) ::feng::launch_k(k_cheb_first<V, 16, NV>, g, 256, 0, s, n, ia, ja, a, dinv, b, dn, r, x, it, c1, c2, skip);
    else if(lanes == 8) ::feng::launch_k(k_cheb_first<V, 8, NV>, g, 256, 0, s, n, ia, ja, a, dinv, b, dn, r, x, it, c1, c2, skip);
    else ::feng::launch_k(k_cheb_first<V, 4, NV>, g, 256, 0, s, n, ia, ja, a, dinv, b, dn, r, x, it, c1, c2, skip);
    rho = rhoN;
    std::swap(d, dn);
    k0 = 1;
  } else {
    if(lanes == 16) ::feng::launch_k(k_cheb_restart<V, 16, NV>, g, 256, 0, s, n, ia, ja, a, dinv, b, x, r, d0, (V)(1.0 / theta), skip);
    else if(lanes == 8) ::feng::launch_k(k_cheb_restart<V, 8, NV>, g, 256, 0, s, n, ia, ja, a, dinv, b, x, r, d0, (V)(1.0 / theta), skip);
    else ::feng::launch_k(k_cheb_restart<V, 4, NV>, g, 256, 0, s, n, ia, ja, a, dinv, b, x, r, d0, (V)(1.0 / theta), skip);
  }
  for(int k = k0; k < p.chebyDegree; ++k) {
    if(!needResidual && k == p.chebyDegree - 1) {
      ::feng::launch_k(k_cheb_last<V>, grid(n * NV), 256, 0, s, n * NV, d, x, skip);
      break;
    }
    const double rhoN = 1.0 / (2.0 * sigma - rho);
    const V c1 = (V)(rhoN * rho), c2 = (V)(2.0 * rhoN / delta);
    if(lanes == 16) ::feng::launch_k(k_cheb_step<V, 16, NV>, g, 256, 0, s, n, ia, ja, a, dinv, d, dn, r, x, c1, c2, skip);
    else if(lanes == 8) ::feng::launch_k(k_cheb_step<V, 8, NV>, g, 256, 0, s, n, ia, ja, a, dinv, d, dn, r, x, c1, c2, skip);
    else ::feng::launch_k(k_cheb_step<V, 4, NV>, g, 256, 0, s, n, ia, ja, a, dinv, d, dn, r, x, c1, c2, skip);
    rho = rhoN;
    std::swap(d, dn);
  }
}

template <typename V, int NV>
void AMGDevice::down(const Lev &L, const V *b, V *bc, V *s)
{
  const int64_t tThreads = L.sellTQ ? L.n : L.n * L.lanesT;
  const int g = (int)((L.nc * L.lanesR + 255) / 256 + (tThreads + 255) / 256);
  ::feng::launch_k(L.sellTQ ? k_down<V, NV, true> : k_down<V, NV, false>, g, 256, 0, s_, L.lanesR, L.lanesT, L.nc,
                   L.rPtr, L.rCol, (const V *)L.rVal, L.n, L.tPtr, L.tCol, (const V *)L.tVal, L.tRow, b, bc, s, skip_);
}

template <typename V, int NV>
void AMGDevice::up(const Lev &L, const V *xc, const V *s, V *x, bool out)
{
  const int64_t threads = L.sellTQ ? L.n : L.n * L.lanesQ;
  const int extra = out && out_.bgu ? (int)((out_.nP + 255) / 256) : 0;
  auto kernel = L.sellTQ ? (out ? k_up<V, NV, true, true> : k_up<V, NV, true, false>)
                         : (out ? k_up<V, NV, false, true> : k_up<V, NV, false, false>);
  ::feng::launch_k(kernel, (int)((threads + 255) / 256) + extra, 256, 0, s_, L.lanesQ, L.n, L.qPtr, L.qCol,
                   (const V *)L.qVal, L.qRow, xc, s, x, skip_, out ? out_ : OutMap());
}

template <typename V, int NV>
void AMGDevice::vcycle_t(int l, const V *b, V *x)
{
  Lev &L = lv_[l];
  if(l == (int)lv_.size() - 1) {
    if(L.n > 0) ::feng::launch_k(k_dense<V, NV>, (int)L.n, DENSE_T, 0, s_, L.n, (const V *)coarseInv_, b, x, skip_);
    return;
  }
  Lev &C = lv_[l + 1];
  if(p_.chebyDegree == 1) {
    down<V, NV>(L, b, (V *)C.b, (V *)L.r);
    vcycle_t<V, NV>(l + 1, (const V *)C.b, (V *)C.x);
    const bool out = l == 0 && out_.z;
    up<V, NV>(L, (const V *)C.x, (const V *)L.r, x, out);
    if(out) outWritten_ = true;
    return;
  }
  const V *A = (const V *)L.Aa;
  chebyshev<V, NV>(L.lanesA, L.n, L.Aia, L.Aja, A, L.sellPtr, L.sellCol, (const V *)L.sellVal, (const V *)L.dinv, b,
                   x, (V *)L.r, (V *)L.d0, (V *)L.d1, L.lmax, p_, true, true, s_, skip_);
  // Chebyshev keeps r = D^-1 (b - A x): restrict the residual D r directly
  // (no extra pass over A).
  csr<V, 3, NV>(L.lanesR, C.n, L.Ria, L.Rja, (const V *)L.Ra, (const V *)L.r, (const V *)L.diag, (V *)C.b, s_,
                skip_);
  vcycle_t<V, NV>(l + 1, (const V *)C.b, (V *)C.x);
  csr<V, 2, NV>(L.lanesP, L.n, L.Pia, L.Pja, (const V *)L.Pa, (const V *)C.x, nullptr, x, s_, skip_);
  chebyshev<V, NV>(L.lanesA, L.n, L.Aia, L.Aja, A, L.sellPtr, L.sellCol, (const V *)L.sellVal, (const V *)L.dinv, b,
                   x, (V *)L.r, (V *)L.d0, (V *)L.d1, L.lmax, p_, false, false, s_, skip_);
}

void AMGDevice::vcycle64(const double *b, double *x) { vcycle_t<double, 1>(0, b, x); }
void AMGDevice::vcycle32(const float *b, float *x) { vcycle_t<float, 1>(0, b, x); }
bool AMGDevice::vcycle2_64(const double *b, double *x, const OutMap *om)
{
  out_ = om ? *om : OutMap();
  outWritten_ = false;
  vcycle_t<double, 2>(0, b, x);
  out_ = OutMap();
  return outWritten_;
}

bool AMGDevice::vcycle2_32(const float *b, float *x, const OutMap *om)
{
  out_ = om ? *om : OutMap();
  outWritten_ = false;
  vcycle_t<float, 2>(0, b, x);
  out_ = OutMap();
  return outWritten_;
}

bool AMGDevice::vcycle3_64(const double *b, double *x, const OutMap *om)
{
  out_ = om ? *om : OutMap();
  outWritten_ = false;
  vcycle_t<double, 3>(0, b, x);
  out_ = OutMap();
  return outWritten_;
}

bool AMGDevice::vcycle3_32(const float *b, float *x, const OutMap *om)
{
  out_ = om ? *om : OutMap();
  outWritten_ = false;
  vcycle_t<float, 3>(0, b, x);
  out_ = OutMap();
  return outWritten_;
}

void AMGDevice::fineStep2()
{
  // The finest-level pass of a V-cycle on the way down, on the level's own
  // vectors: b = the level's b (finite values of its allocation or of
  // earlier cycles), s and the next level's b written; degree 2 and up: the
  // pre-smoothing pass; a single level: the dense solve.
  const Lev &L = lv_[0];
  const int g = grid(L.n * L.lanesA);
  auto go = [&](auto tag) {
    using V = decltype(tag);
    const V *b = (const V *)L.b;
    V *r = (V *)L.r, *x = (V *)L.x;
    if(lv_.size() == 1) {
      if(L.n > 0) ::feng::launch_k(k_dense<V, 2>, (int)L.n, DENSE_T, 0, s_, L.n, (const V *)coarseInv_, b, x, skip_);
      return;
    }
    if(p_.chebyDegree == 1) {
      down<V, 2>(L, b, (V *)lv_[1].b, r);
      return;
    }
    const V *a = (const V *)L.Aa, *dinv = (const V *)L.dinv;
    V *dn = (V *)L.d1;
    const V it = (V)0.5, c1 = (V)0.5, c2 = (V)0.5;
    if(L.sellPtr)
      ::feng::launch_k(k_cheb_first_sell<V, 2>, grid(L.n), 256, 0, s_, L.n, L.sellPtr, L.sellCol, (const V *)L.sellVal, dinv, b, dn,
                                                          r, x, it, c1, c2, skip_);
    else if(L.lanesA == 16) ::feng::launch_k(k_cheb_first<V, 16, 2>, g, 256, 0, s_, L.n, L.Aia, L.Aja, a, dinv, b, dn, r, x, it, c1, c2, skip_);
    else if(L.lanesA == 8) ::feng::launch_k(k_cheb_first<V, 8, 2>, g, 256, 0, s_, L.n, L.Aia, L.Aja, a, dinv, b, dn, r, x, it, c1, c2, skip_);
    else ::feng::launch_k(k_cheb_first<V, 4, 2>, g, 256, 0, s_, L.n, L.Aia, L.Aja, a, dinv, b, dn, r, x, it, c1, c2, skip_);
  };
  if(fp32_) go(float());
  else go(double());
}

int64_t AMGDevice::fineStep2Bytes() const
{
  if(lv_.empty()) return 0;
  const Lev &L = lv_[0];
  const int64_t vs = fp32_ ? 4 : 8;
  if(lv_.size() == 1) return L.n * L.n * vs + 2 * 2 * L.n * vs;
  // both operators (values + columns, row pointers), and per component: b
  // read, s and the next b written
  if(p_.chebyDegree == 1)
    return (L.nnzT + L.nnzR) * (vs + 4) + (L.n + L.nc + 2) * 4 + 2 * (2 * L.n + L.nc) * vs;
  // values + columns, row pointers, dinv, and per component: b read, x, r,
  // dn written
  return nnz0_ * (vs + 4) + (L.n + 1) * 4 + L.n * vs + 2 * L.n * vs * 4;
}

void AMGDevice::spmv64(const double *x, double *y)
{
  const Lev &L = lv_[0];
  csr<double, 0, 1>(L.lanesA, L.n, L.Aia, L.Aja, (const double *)L.Aa, x, nullptr, y, s_, skip_);
}

void AMGDevice::spmv32(const float *x, float *y)
{
  const Lev &L = lv_[0];
  csr<float, 0, 1>(L.lanesA, L.n, L.Aia, L.Aja, (const float *)L.Aa, x, nullptr, y, s_, skip_);
}

}  // namespace feng
