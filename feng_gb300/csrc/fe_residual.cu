// Taylor-Hood residuals, one thread per element and velocity component (see
// fe_residual.h).
#include "fe_residual.h"

#include <algorithm>
#include <type_traits>
#include <vector>

#include "fe_common.h"
#include "fe_df.h"
#include "fe_setup.h"
#include "fe_sources.h"

namespace feng {

#define CKR(x)                                                                         \
  do {                                                                                 \
    cudaError_t _e = (x);                                                              \
    if(_e != cudaSuccess) {                                                            \
      set_error("CUDA error %s at %s:%d", cudaGetErrorString(_e), __FILE__, __LINE__); \
      return FE_CUDA_FAIL;                                                             \
    }                                                                                  \
  } while(0)

namespace {

// Local node of edge (i, j): after the vertices, in the element's edge order.
template <int D>
__host__ __device__ constexpr int edge_node(int i, int j)
{
  const int a = i < j ? i : j, b = i < j ? j : i;
  if(D == 2) return a == 0 ? (b == 1 ? 3 : 5) : 4;            // (0,1) (1,2) (2,0)
  if(a == 0) return b == 2 ? 4 : b == 1 ? 6 : 8;              // (0,2) (2,1) (1,0) (1,3) (3,0) (3,2)
  return a == 1 ? (b == 2 ? 5 : 7) : 9;
}

// Arithmetic of an element: FP64, or double-float on the FP32 pipes.
struct F64 {
  using T = double;
  using In = double;
  static __device__ __forceinline__ T zero() { return 0.; }
  static __device__ __forceinline__ T load(const double *p, int64_t i) { return p[i]; }
  static __device__ __forceinline__ T add(T a, T b) { return a + b; }
  static __device__ __forceinline__ T sub(T a, T b) { return a - b; }
  static __device__ __forceinline__ T mul(T a, T b) { return a * b; }
  static __device__ __forceinline__ T fma(T a, T b, T c) { return ::fma(a, b, c); }
  static __device__ __forceinline__ T scale(T a, float f) { return a * (double)f; }
  static __device__ __forceinline__ T neg(T a) { return -a; }
  static __device__ __forceinline__ double to(T a) { return a; }
};
struct DF {
  using T = dfl;
  using In = float2;
  static __device__ __forceinline__ T zero() { return df_zero(); }
  static __device__ __forceinline__ T load(const float2 *p, int64_t i)
  {
    const float2 v = p[i];
    return {v.x, v.y};
  }
  static __device__ __forceinline__ T add(T a, T b) { return df_add(a, b); }
  static __device__ __forceinline__ T sub(T a, T b) { return df_sub(a, b); }
  static __device__ __forceinline__ T mul(T a, T b) { return df_mul(a, b); }
  static __device__ __forceinline__ T fma(T a, T b, T c) { return df_fma(a, b, c); }
  // f a power of two or a small integer with few bits: exact up to one rounding
  static __device__ __forceinline__ T scale(T a, float f) { return df_mul(a, {f, 0.f}); }
  static __device__ __forceinline__ T neg(T a) { return df_neg(a); }
  static __device__ __forceinline__ double to(T a) { return df_to(a); }
};

// The forms' coefficients in an arithmetic, formed on the host: conversions
// from FP64 in every thread would be FP64 work.
template <typename T>
struct Coeffs {
  T conv, mass, sigma, sigmaMu, divu;  // -conv, -mass, -sigma, sigma mu, -divu
};
template <typename T>
Coeffs<T> coeffs(const FormCoeffs &fc)
{
  auto t = [](double x) {
    if constexpr(std::is_same_v<T, double>) return x;
    else return dfl{(float)x, (float)(x - (double)(float)x)};
  };
  return {t(-fc.conv), t(-fc.mass), t(-fc.sigma), t(fc.sigma * fc.mu), t(-fc.divu)};
}

// Index of lambda_i lambda_j lambda_k among the cubic products, i <= j <= k
// in lexicographic order: a closed form, so that unrolled loops index
// registers.
template <int D>
__host__ __device__ constexpr int cubic(int i, int j, int k)
{
  const int x = i < j ? (i < k ? i : k) : (j < k ? j : k), z = i > j ? (i > k ? i : k) : (j > k ? j : k),
            y = i + j + k - x - z;
  // products before (x, ., .), before (x, y, .) and before (x, y, z)
  const int m = D + 1 - x, n = D + 1 - y, all = (D + 1) * (D + 2) * (D + 3) / 6;
  return all - m * (m + 1) * (m + 2) / 6 + (m * (m + 1) - n * (n + 1)) / 2 + z - y;
}
static_assert(cubic<3>(0, 0, 0) == 0 && cubic<3>(2, 1, 0) == 5 && cubic<3>(1, 1, 1) == 10 && cubic<3>(3, 3, 3) == 19 &&
                  cubic<2>(0, 2, 1) == 4 && cubic<2>(1, 2, 2) == 8,
              "lexicographic order");
// Slot of lambda_i lambda_j among the quadratic products: the P2 node there.
template <int D>
__host__ __device__ constexpr int quadr(int i, int j)
{
  return i == j ? i : edge_node<D>(i, j);
}

// 8-byte words of shared memory: the rule's tables, the own rule's, an element.
constexpr int n2_of(int D) { return D == 2 ? 6 : 10; }
constexpr int n3_of(int D) { return D == 2 ? 10 : 20; }
constexpr int table_words(int D) { return n2_of(D) * n3_of(D) + 3 * (D + 1) * (D + 1); }
constexpr int own_words(int D, int nqs) { return nqs * (n2_of(D) + D + 1); }
constexpr int elem_words(int D) { return 2 * D * n2_of(D) + (D + 1) * D * D; }

// The element's residual vector be[local row][element]: thread (e, c) of a
// block holds velocity component c of element e (one warp, one component).
//
// A P2 function is a homogeneous quadratic in the barycentric coordinates l:
// sum_i u_i l_i^2 + sum_(i<j) (4 u_ij - u_i - u_j) l_i l_j.  Its gradient at
// the vertices is differences of those coefficients.  With p and the gradient
// affine (straight-sided elements) no term needs a quadrature node: the
// stress is formed at the vertices, and its moments and those of the
// divergence go through the rule's P1 mass matrix; u . grad u is a cubic
// whose 20 (triangles: 10) coefficients are products of the quadratic's and
// the gradient's, u-dot joins them times sum l = 1, and the rule's moments of
// the cubic products with the P2 functions give the rows.  All are the rule's
// own sums regrouped, whatever its degree.  Tetrahedra: about 2,000 products
// per element against 23,000 for the contraction of the reference tensors
// with a warp per P2 function and 2,600 with the convective term at a rule's
// 14 nodes.
// Bound: the FP64 pipe (196,608 tetrahedra with a source, FP64: about 3,300
// products, 1040 us of the pipe, 1064 measured; 1300 with node sums).  In
// double-float the FP32 issue rate and, with a source, the FP64 pipe too: 675
// us, of which the sources hold the FP64 pipe for 410; one thread for all
// components held 255 registers, 8 warps an SM, and took 1113.  294,912
// triangles in double-float: 95 us, 120 with node sums.
template <int D, typename A>
__global__ void __launch_bounds__(D == 3 ? 96 : 128, D == 3 ? 5 : 4) k_residual_elem(int64_t nE, const int32_t *__restrict__ adr,
                                                         const double *__restrict__ geo,
                                                         const float2 *__restrict__ geoPair,
                                                         const double *__restrict__ xy,
                                                         const typename A::In *__restrict__ tab,
                                                         const double *__restrict__ own, FormCoeffs fc,
                                                         Coeffs<typename A::T> cf,
                                                         const typename A::In *__restrict__ u,
                                                         const typename A::In *__restrict__ ud, int nqs,
                                                         double *__restrict__ be)
{
  using T = typename A::T;
  constexpr int NV = D + 1, N2 = n2_of(D), N3 = n3_of(D);
  extern __shared__ __align__(16) unsigned char smem[];
  T *sW = reinterpret_cast<T *>(smem), *sm = sW + N2 * N3, *sm4 = sm + NV * NV, *smv = sm4 + NV * NV;
  double *sSw = reinterpret_cast<double *>(smv + NV * NV), *sSl = sSw + nqs * N2;
  const int lane = threadIdx.x, c = threadIdx.y, EB = blockDim.x;
  T *sU = reinterpret_cast<T *>(sSl + nqs * NV);  // [N2][D][EB] quadratic coefficients of u_c
  T *sG = sU + N2 * D * EB;                       // [NV][D][D][EB]  d_k u_c at vertex v
  T *sB = sG + NV * D * D * EB;                   // [N2][D][EB] rows of the convective term and u-dot
  for(int i = c * EB + lane; i < table_words(D); i += EB * D) sW[i] = A::load(tab, i);
  for(int i = c * EB + lane; i < own_words(D, nqs); i += EB * D) sSw[i] = own[i];
  const int64_t p0 = (int64_t)blockIdx.x * EB + lane;
  const bool live = p0 < nE;
  const int64_t p = live ? p0 : nE - 1;
  auto geom = [&](int k) {
    if constexpr(std::is_same_v<T, double>) return geo[(int64_t)k * nE + p];
    else return DF::load(geoPair, (int64_t)k * nE + p);
  };
  // quadratic coefficients of a P2 function from its nodal values
  auto quadratic = [&](const typename A::In *v, T *h) {
#pragma unroll
    for(int a = 0; a < N2; ++a) h[a] = A::load(v, adr[(int64_t)(D * a + c) * nE + p]);
#pragma unroll
    for(int i = 0; i < NV; ++i)
#pragma unroll
      for(int j = i + 1; j < NV; ++j)
        h[quadr<D>(i, j)] = A::sub(A::scale(h[quadr<D>(i, j)], 4.f), A::add(h[i], h[j]));
  };
  T G[D][D];
#pragma unroll
  for(int r = 0; r < D; ++r)
#pragma unroll
    for(int k = 0; k < D; ++k) G[r][k] = geom(D * r + k);
  T g[NV][D];  // d_k u_c at vertex v
  {
    T h[N2];
    quadratic(u, h);
#pragma unroll
    for(int a = 0; a < N2; ++a) sU[(a * D + c) * EB + lane] = h[a];
#pragma unroll
    for(int v = 0; v < NV; ++v) {
      T d[NV];
#pragma unroll
      for(int i = 0; i < NV; ++i) d[i] = i == v ? A::add(h[v], h[v]) : h[quadr<D>(v, i)];
#pragma unroll
      for(int r = 1; r < NV; ++r) d[r] = A::sub(d[r], d[0]);
#pragma unroll
      for(int k = 0; k < D; ++k) {
        T s = A::mul(G[0][k], d[1]);
#pragma unroll
        for(int r = 1; r < D; ++r) s = A::fma(G[r][k], d[r + 1], s);
        g[v][k] = s;
        sG[((v * D + k) * D + c) * EB + lane] = s;
      }
    }
  }
  __syncthreads();

  // Be_(a,c) -= int phi_a (conv u . grad u + mass udot)_c
  T b[N2];
  if(fc.hasConv || fc.hasMass) {
    T f[N3];
#pragma unroll
    for(int j = 0; j < N3; ++j) f[j] = A::zero();
    if(fc.hasMass) {
      T h[N2];
      quadratic(ud, h);
#pragma unroll
      for(int a = 0; a < N2; ++a) h[a] = A::mul(cf.mass, h[a]);
#pragma unroll
      for(int i = 0; i < NV; ++i)
#pragma unroll
        for(int j = i; j < NV; ++j)
#pragma unroll
          for(int v = 0; v < NV; ++v) f[cubic<D>(i, j, v)] = A::add(f[cubic<D>(i, j, v)], h[quadr<D>(i, j)]);
    }
    if(fc.hasConv) {
#pragma unroll 1
      for(int k = 0; k < D; ++k) {
        T x[NV];
#pragma unroll
        for(int v = 0; v < NV; ++v) x[v] = A::mul(cf.conv, sG[((v * D + k) * D + c) * EB + lane]);
#pragma unroll
        for(int i = 0; i < NV; ++i)
#pragma unroll
          for(int j = i; j < NV; ++j) {
            const T y = sU[(quadr<D>(i, j) * D + k) * EB + lane];
#pragma unroll
            for(int v = 0; v < NV; ++v) f[cubic<D>(i, j, v)] = A::fma(y, x[v], f[cubic<D>(i, j, v)]);
          }
      }
    }
#pragma unroll 1
    for(int a = 0; a < N2; a += 2) {
      T s0 = A::zero(), s1 = A::zero();
#pragma unroll
      for(int j = 0; j < N3; ++j) {
        s0 = A::fma(sW[a * N3 + j], f[j], s0);
        s1 = A::fma(sW[(a + 1) * N3 + j], f[j], s1);
      }
      sB[(a * D + c) * EB + lane] = s0;
      sB[((a + 1) * D + c) * EB + lane] = s1;
    }
#pragma unroll
    for(int a = 0; a < N2; ++a) b[a] = sB[(a * D + c) * EB + lane];
  } else {
#pragma unroll
    for(int a = 0; a < N2; ++a) b[a] = A::zero();
  }

  // Be_(a,c) += sigma (mu sum_m (d_m u_c + d_c u_m) d_m phi_a - p d_c phi_a)
  if(fc.hasSigma) {
    T S[NV][D];  // sum_m G[r][m] stress_mc at the vertices
#pragma unroll
    for(int v = 0; v < NV; ++v) {
      const T P = A::mul(cf.sigma, A::load(u, adr[(int64_t)(D * N2 + v) * nE + p]));
      T st[D];
#pragma unroll
      for(int m = 0; m < D; ++m) {
        st[m] = A::mul(cf.sigmaMu, A::add(g[v][m], sG[((v * D + c) * D + m) * EB + lane]));
        if(m == c) st[m] = A::add(st[m], P);
      }
#pragma unroll
      for(int r = 0; r < D; ++r) {
        T s = A::mul(G[r][0], st[0]);
#pragma unroll
        for(int m = 1; m < D; ++m) s = A::fma(G[r][m], st[m], s);
        S[v][r] = s;
      }
    }
    // edge (w, i): 4 (int lambda_w S_i + int lambda_i S_w), S_0 = -sum_r S_r;
    // vertex w: int (4 lambda_w - 1) S_w
#pragma unroll
    for(int w = 0; w < NV; ++w) {
      T e0 = A::zero();
#pragma unroll
      for(int r = 0; r < D; ++r) {
        T h = A::mul(sm4[w * NV], S[0][r]);
#pragma unroll
        for(int v = 1; v < NV; ++v) h = A::fma(sm4[w * NV + v], S[v][r], h);
        if(r + 1 != w) {
          const int q = edge_node<D>(w, r + 1 == w ? (w + 1) % NV : r + 1);
          b[q] = A::add(b[q], h);
        }
        e0 = A::sub(e0, h);
      }
      if(w) {
        const int q = edge_node<D>(w == 0 ? 1 : w, 0);
        b[q] = A::add(b[q], e0);
      }
      T x[NV];
#pragma unroll
      for(int v = 0; v < NV; ++v) {
        if(w) x[v] = S[v][w ? w - 1 : 0];
        else {
          x[v] = S[v][0];
#pragma unroll
          for(int r = 1; r < D; ++r) x[v] = A::add(x[v], S[v][r]);
          x[v] = A::neg(x[v]);
        }
      }
#pragma unroll
      for(int v = 0; v < NV; ++v) b[w] = A::fma(smv[w * NV + v], x[v], b[w]);
    }
  }
  // Be_pj -= divu int (div u) psi_j
  {
    T dv[NV];
#pragma unroll
    for(int v = 0; v < NV; ++v) {
      T s = sG[v * D * D * EB + lane];
#pragma unroll
      for(int k = 1; k < D; ++k) s = A::add(s, sG[((v * D + k) * D + k) * EB + lane]);
      dv[v] = s;
    }
    const T f = fc.hasDivu ? A::mul(cf.divu, geom(D * D)) : A::zero();
    for(int j = c; j < NV; j += D) {
      T s = A::mul(sm[j * NV], dv[0]);
#pragma unroll
      for(int v = 1; v < NV; ++v) s = A::fma(sm[j * NV + v], dv[v], s);
      if(live) be[(int64_t)(D * N2 + j) * nE + p] = fc.hasDivu ? A::to(A::mul(f, s)) : 0.;
    }
  }
  const T J = geom(D * D);
  double o[N2];
#pragma unroll
  for(int a = 0; a < N2; ++a) o[a] = A::to(A::mul(J, b[a]));
  // Be_(a,c) -= int f_c phi_a with the form's own rule, in FP64: the
  // component threads share the nodes and add their sums
  if(nqs > 0) {
    const double sj = -fc.srcCoeff * geo[(int64_t)(D * D) * nE + p];
    if(D == 3 && fc.srcKind == SRC_CONST_VEC) {
      const double f = sj * (c == 0 ? fc.srcParam[0] : c == 1 ? fc.srcParam[1] : fc.srcParam[2]);
#pragma unroll 1
      for(int q = 0; q < nqs; ++q)
#pragma unroll
        for(int a = 0; a < N2; ++a) o[a] += sSw[q * N2 + a] * f;
    } else {
      constexpr int NC = D == 2 ? 2 : 1;  // tetrahedral sources: the first component
      double acc[N2][NC];
#pragma unroll
      for(int a = 0; a < N2; ++a)
#pragma unroll
        for(int k = 0; k < NC; ++k) acc[a][k] = 0.;
#pragma unroll 1
      for(int q = c; q < nqs; q += D) {
        double x[D], f[2];
#pragma unroll
        for(int k = 0; k < D; ++k) {
          x[k] = sSl[q * NV] * xy[(int64_t)k * nE + p];
#pragma unroll
          for(int v = 1; v < NV; ++v) x[k] += sSl[q * NV + v] * xy[(int64_t)(D * v + k) * nE + p];
        }
        if constexpr(D == 2) source_value(fc.srcKind, fc.srcParam, x[0], x[1], f);
        else f[0] = source_x(fc.srcKind, fc.srcParam, x[0], x[1], x[D - 1]);
#pragma unroll
        for(int a = 0; a < N2; ++a)
#pragma unroll
          for(int k = 0; k < NC; ++k) acc[a][k] += sSw[q * N2 + a] * f[k];
      }
      static_assert(D * N2 * NC <= elem_words(D), "the sums fit where the element was");
      double *sX = reinterpret_cast<double *>(sU);  // [D][N2][NC][EB]
      __syncthreads();
#pragma unroll
      for(int a = 0; a < N2; ++a)
#pragma unroll
        for(int k = 0; k < NC; ++k) sX[((c * N2 + a) * NC + k) * EB + lane] = acc[a][k];
      __syncthreads();
      if(c < NC)
#pragma unroll
        for(int a = 0; a < N2; ++a) {
          double s = sX[(a * NC + c) * EB + lane];
#pragma unroll
          for(int t = 1; t < D; ++t) s += sX[((t * N2 + a) * NC + c) * EB + lane];
          o[a] += sj * s;
        }
    }
  }
  if(!live) return;
#pragma unroll
  for(int a = 0; a < N2; ++a) be[(int64_t)(D * a + c) * nE + p] = o[a];
}

// rhs[r] += its elements' terms in color order (the colored scatter's sums).
__global__ void __launch_bounds__(256) k_residual_rows(int64_t n, const int32_t *__restrict__ ptr,
                                                      const int32_t *__restrict__ ent, const double *__restrict__ be,
                                                      double *__restrict__ rhs)
{
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(r >= n) return;
  const int32_t k1 = ptr[r + 1];
  double s = rhs[r];
  for(int32_t k = ptr[r]; k < k1; k += 8) {
    double v[8];
#pragma unroll
    for(int q = 0; q < 8; ++q) v[q] = k + q < k1 ? be[ent[k + q]] : 0.;
#pragma unroll
    for(int q = 0; q < 8; ++q)
      if(k + q < k1) s += v[q];
  }
  rhs[r] = s;
}

__global__ void k_row_counts(int64_t m, int64_t n, const int32_t *__restrict__ adr, int32_t *__restrict__ cnt)
{
  for(int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    if(adr[i] < n) atomicAdd(cnt + adr[i], 1);
}

__global__ void k_row_entries(int64_t m, int64_t n, const int32_t *__restrict__ adr, int32_t *__restrict__ next,
                              int32_t *__restrict__ ent)
{
  for(int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    if(adr[i] < n) ent[atomicAdd(next + adr[i], 1)] = (int32_t)i;
}

// Entries of each row by element (entry = local row * nE + element).
__global__ void k_row_sort(int64_t n, int32_t nE, const int32_t *__restrict__ ptr, int32_t *__restrict__ ent)
{
  const int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(r >= n) return;
  for(int32_t k = ptr[r] + 1; k < ptr[r + 1]; ++k) {
    const int32_t e = ent[k], key = e % nE;
    int32_t j = k;
    for(; j > ptr[r] && ent[j - 1] % nE > key; --j) ent[j] = ent[j - 1];
    ent[j] = e;
  }
}

}  // namespace

void build_residual_tables(const QuadRule &rule, int dim, ResidualTables &T)
{
  const int nv = dim + 1, n2 = dim == 2 ? 6 : 10;
  auto basis = [&](const QuadRule &q, int k, double *lam, double *phi) {
    lam[1] = q.r[k];
    lam[2] = q.s[k];
    if(dim == 3) lam[3] = q.t[k];
    lam[0] = 1.;
    for(int i = 1; i < nv; ++i) lam[0] -= lam[i];
    for(int i = 0; i < nv; ++i) phi[i] = lam[i] * (2. * lam[i] - 1.);
    for(int i = 0; i < nv; ++i)
      for(int j = i + 1; j < nv; ++j) phi[dim == 2 ? edge_node<2>(i, j) : edge_node<3>(i, j)] = 4. * lam[i] * lam[j];
  };
  const int n3 = n3_of(dim), nq = T.nq = rule.n();
  T.rule.assign(table_words(dim), 0.);
  T.own.assign(own_words(dim, nq), 0.);
  double *W = T.rule.data(), *m = W + n2 * n3, *m4 = m + nv * nv, *mv = m4 + nv * nv;
  for(int q = 0; q < nq; ++q) {
    double *l = T.own.data() + nq * n2 + q * nv, f[10];
    basis(rule, q, l, f);
    const double w = rule.w[q];
    for(int a = 0; a < n2; ++a) T.own[q * n2 + a] = w * f[a];
    for(int i = 0; i < nv; ++i)
      for(int j = 0; j < nv; ++j) {
        m[i * nv + j] += w * l[i] * l[j];
        m4[i * nv + j] += 4. * w * l[i] * l[j];
        mv[i * nv + j] += w * (4. * l[i] - 1.) * l[j];
        for(int k = j; k < nv; ++k)
          if(i <= j)
            for(int a = 0; a < n2; ++a)
              W[a * n3 + (dim == 2 ? cubic<2>(i, j, k) : cubic<3>(i, j, k))] += w * f[a] * l[i] * l[j] * l[k];
      }
  }
}

ResidualTH::~ResidualTH()
{
  cudaFree(tab_);
  cudaFree(pairs_);
  cudaFree(own_);
  cudaFree(be_);
  cudaFree(rowPtr_);
  cudaFree(rowEnt_);
}

int ResidualTH::build(const DeviceMesh &dm, int dim, int64_t nInc, const ResidualTables &T, cudaStream_t s)
{
  dm_ = dm;
  dim_ = dim;
  nq_ = T.nq;
  nInc_ = nInc;
  s_ = s;
  const int64_t m = dm.nElm * dm.nloc;
  if(m >= (int64_t)INT32_MAX) {
    set_error("too many element DOFs for the residual's row tables");
    return FE_INVALID_ARG;
  }
  std::vector<float2> pairs(T.rule.size());
  for(size_t i = 0; i < pairs.size(); ++i) {
    const float h = (float)T.rule[i];
    pairs[i] = make_float2(h, (float)(T.rule[i] - (double)h));
  }
  CKR(cudaMalloc(&tab_, sizeof(double) * T.rule.size()));
  CKR(cudaMalloc(&pairs_, sizeof(float2) * pairs.size()));
  CKR(cudaMalloc(&own_, sizeof(double) * T.own.size()));
  CKR(cudaMemcpy(tab_, T.rule.data(), sizeof(double) * T.rule.size(), cudaMemcpyHostToDevice));
  CKR(cudaMemcpy(pairs_, pairs.data(), sizeof(float2) * pairs.size(), cudaMemcpyHostToDevice));
  CKR(cudaMemcpy(own_, T.own.data(), sizeof(double) * T.own.size(), cudaMemcpyHostToDevice));
  CKR(cudaMalloc(&be_, sizeof(double) * std::max<int64_t>(1, m)));
  CKR(cudaMalloc(&rowPtr_, sizeof(int32_t) * (nInc + 1)));
  // the mesh was copied on the legacy stream, with which s is not ordered
  CKR(cudaStreamSynchronize(cudaStreamLegacy));
  CKR(cudaMemsetAsync(rowPtr_, 0, sizeof(int32_t) * (nInc + 1), s));
  const unsigned g = (unsigned)std::max<int64_t>(1, std::min<int64_t>((m + 255) / 256, 1 << 16));
  (k_row_counts<<<g, 256, 0, s>>>(m, nInc, dm.adr, rowPtr_), ::feng::count_launch());
  std::vector<int32_t> ptr(nInc + 1);
  CKR(cudaMemcpyAsync(ptr.data(), rowPtr_, sizeof(int32_t) * (nInc + 1), cudaMemcpyDeviceToHost, s));
  CKR(cudaStreamSynchronize(s));
  int32_t sum = 0;
  for(int64_t r = 0; r <= nInc; ++r) {
    const int32_t c = ptr[r];
    ptr[r] = sum;
    if(r < nInc) sum += c;
  }
  int32_t *next = nullptr;
  CKR(cudaMalloc(&next, sizeof(int32_t) * (nInc + 1)));
  struct Free { int32_t *p; ~Free() { cudaFree(p); } } guard{next};
  CKR(cudaMalloc(&rowEnt_, sizeof(int32_t) * std::max<int32_t>(1, sum)));
  CKR(cudaMemcpyAsync(rowPtr_, ptr.data(), sizeof(int32_t) * (nInc + 1), cudaMemcpyHostToDevice, s));
  CKR(cudaMemcpyAsync(next, rowPtr_, sizeof(int32_t) * (nInc + 1), cudaMemcpyDeviceToDevice, s));
  (k_row_entries<<<g, 256, 0, s>>>(m, nInc, dm.adr, next, rowEnt_), ::feng::count_launch());
  if(nInc > 0)
    (k_row_sort<<<(unsigned)((nInc + 255) / 256), 256, 0, s>>>(nInc, (int32_t)dm.nElm, rowPtr_, rowEnt_),
     ::feng::count_launch());
  CKR(cudaGetLastError());
  CKR(cudaStreamSynchronize(s));
  return FE_OK;
}

template <int D, typename A, typename In>
void ResidualTH::run(const FormCoeffs &fc, const In *tab, const In *u, const In *ud, double *rhs) const
{
  const int64_t nE = dm_.nElm;
  if(nE <= 0 || nInc_ <= 0) return;
  // SRC_SIN3 is a scalar source: no vector form has it
  const int nqs = fc.srcKind == SRC_NONE || fc.srcKind == SRC_SIN3 ? 0 : nq_;
  // tetrahedra: 3 warps a block, 15 an SM within 128 registers; triangles: 4,
  // or 2 while the elements do not give every SM one block
  const int eb = D == 2 && nE >= 152 * 64 ? 64 : 32;
  // (at most 34 KB: 64 nodes of a tetrahedral rule)
  auto bytes = [](int ns, int e) { return 8 * (size_t)(table_words(D) + own_words(D, ns) + elem_words(D) * e); };
  (k_residual_elem<D, A><<<(unsigned)((nE + eb - 1) / eb), dim3(eb, D), bytes(nqs, eb), s_>>>(
       nE, dm_.adr, dm_.geo, dm_.geoPair, dm_.xy, tab, own_, fc, coeffs<typename A::T>(fc), u, ud, nqs, be_),
   ::feng::count_launch());
  (k_residual_rows<<<(unsigned)((nInc_ + 255) / 256), 256, 0, s_>>>(nInc_, rowPtr_, rowEnt_, be_, rhs),
   ::feng::count_launch());
}

void ResidualTH::add64(const FormCoeffs &fc, const double *u, const double *udot, double *rhs) const
{
  if(dim_ == 2) run<2, F64>(fc, tab_, u, udot, rhs);
  else run<3, F64>(fc, tab_, u, udot, rhs);
}

void ResidualTH::add_df(const FormCoeffs &fc, const float2 *up, const float2 *udp, double *rhs) const
{
  if(dim_ == 2) run<2, DF>(fc, pairs_, up, udp, rhs);
  else run<3, DF>(fc, pairs_, up, udp, rhs);
}

}  // namespace feng
