// Taylor-Hood residuals, one thread per element (see fe_residual.h).
#include "fe_residual.h"

#include <algorithm>
#include <cstring>
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
  static __device__ __forceinline__ T from(double x) { return x; }
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
  static __device__ __forceinline__ T from(double x) { return df_from(x); }
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

template <typename A, int D>
__host__ __device__ constexpr size_t table_bytes(int nq, int nqs)
{
  constexpr int NV = D + 1, N2 = D == 2 ? 6 : 10;
  return sizeof(typename A::T) * (size_t)(nq * (2 * N2 + NV) + NV * NV + N2 * N2) +
         sizeof(double) * (size_t)(nqs * (N2 + NV));
}

// The element's residual vector be[local row][element].
//
// With p and the velocity gradient affine in the element (P1, P2 velocity on
// a straight-sided element) the stress and divergence terms need no
// quadrature nodes: the gradient is formed at the vertices (one
// multiplication per vertex and function), the stress there, and its moments
// with the P1 functions through the rule's P1 mass matrix, whose adjoint of
// the same sparse map gives the rows.  Only the convective term runs over
// the rule's nodes; the time derivative goes through the rule's P2 mass
// matrix.  All are the rule's own sums regrouped.  Tetrahedra: about 2,400
// products per element against 23,000 for the contraction of the reference
// tensors with a warp per P2 function and 4,900 with every term at the
// rule's 14 nodes.
// Bound: the FP64 pipe, or the FP32 issue rate in double-float.  Residual
// call with its host copies, before (colored scatter, one launch per color)
// and now: 196,608 tetrahedra in FP64 7.29 -> 1.78 ms; 294,912 triangles in
// double-float 534 -> 457 us.
template <int D, typename A>
__global__ void __launch_bounds__(128, 2) k_residual_elem(int64_t nE, const int32_t *__restrict__ adr,
                                                         const double *__restrict__ geo,
                                                         const float2 *__restrict__ geoPair,
                                                         const double *__restrict__ xy,
                                                         const ResidualTables *__restrict__ tab, FormCoeffs fc,
                                                         const typename A::In *__restrict__ u,
                                                         const typename A::In *__restrict__ ud, int nq, int nqs,
                                                         double *__restrict__ be)
{
  using T = typename A::T;
  constexpr int NV = D + 1, N2 = D == 2 ? 6 : 10;
  extern __shared__ __align__(16) unsigned char smem[];
  T *sPhi = reinterpret_cast<T *>(smem), *sWphi = sPhi + nq * N2, *sLam = sWphi + nq * N2, *sm = sLam + nq * NV,
    *sM = sm + NV * NV;
  double *sSw = reinterpret_cast<double *>(sM + N2 * N2), *sSl = sSw + nqs * N2;
  T *sU = reinterpret_cast<T *>(sSl + nqs * NV);  // [D N2][threads]
  const int tid = threadIdx.x, nt = blockDim.x;
  for(int i = tid; i < nq * N2; i += nt) {
    sPhi[i] = A::from(tab->phi[i / N2][i % N2]);
    sWphi[i] = A::from(tab->wphi[i / N2][i % N2]);
  }
  for(int i = tid; i < nq * NV; i += nt) sLam[i] = A::from(tab->lam[i / NV][i % NV]);
  for(int i = tid; i < NV * NV; i += nt) sm[i] = A::from(tab->m[i / NV][i % NV]);
  for(int i = tid; i < N2 * N2; i += nt) sM[i] = A::from(tab->M[i / N2][i % N2]);
  for(int i = tid; i < nqs * N2; i += nt) sSw[i] = tab->swphi[i / N2][i % N2];
  for(int i = tid; i < nqs * NV; i += nt) sSl[i] = tab->slam[i / NV][i % NV];
  const int64_t p = (int64_t)blockIdx.x * nt + tid;
  const bool live = p < nE;
  if(live) {
#pragma unroll
    for(int i = 0; i < D * N2; ++i) sU[i * nt + tid] = A::load(u, adr[(int64_t)i * nE + p]);
  }
  __syncthreads();
  if(!live) return;
  auto U = [&](int b, int c) { return sU[(D * b + c) * nt + tid]; };
  auto geom = [&](int k) {
    if constexpr(std::is_same_v<T, double>) return geo[(int64_t)k * nE + p];
    else return DF::load(geoPair, (int64_t)k * nE + p);
  };
  T G[D][D];
#pragma unroll
  for(int r = 0; r < D; ++r)
#pragma unroll
    for(int k = 0; k < D; ++k) G[r][k] = geom(D * r + k);
  const T J = geom(D * D);

  // g[v][k][c] = d_k u_c at vertex v: the reference gradient there is
  // sum_i grad lambda_i d_i with d_v = 3 u_v, d_i = 4 u_(v,i) - u_i
  T g[NV][D][D];
#pragma unroll
  for(int c = 0; c < D; ++c)
#pragma unroll
    for(int v = 0; v < NV; ++v) {
      T d[NV];
#pragma unroll
      for(int i = 0; i < NV; ++i)
        d[i] = i == v ? A::scale(U(v, c), 3.f) : A::sub(A::scale(U(edge_node<D>(v, i == v ? (v + 1) % NV : i), c), 4.f), U(i, c));
#pragma unroll
      for(int r = 1; r < NV; ++r) d[r] = A::sub(d[r], d[0]);
#pragma unroll
      for(int k = 0; k < D; ++k) {
        T s = A::mul(G[0][k], d[1]);
#pragma unroll
        for(int r = 1; r < D; ++r) s = A::fma(G[r][k], d[r + 1], s);
        g[v][k][c] = s;
      }
    }

  T b[N2][D];
#pragma unroll
  for(int a = 0; a < N2; ++a)
#pragma unroll
    for(int c = 0; c < D; ++c) b[a][c] = A::zero();

  // Be_(a,c) += sigma (mu sum_m (d_m u_c + d_c u_m) d_m phi_a - p d_c phi_a)
  if(fc.hasSigma) {
    const T sp = A::from(-fc.sigma), smu = A::mul(A::from(fc.sigma), A::from(fc.mu));
    T P[NV];
#pragma unroll
    for(int j = 0; j < NV; ++j) P[j] = A::mul(sp, A::load(u, adr[(int64_t)(D * N2 + j) * nE + p]));
#pragma unroll
    for(int c = 0; c < D; ++c) {
      T S[NV][D];  // sum_m G[r][m] stress_mc at the vertices
#pragma unroll
      for(int v = 0; v < NV; ++v) {
        T st[D];
#pragma unroll
        for(int m = 0; m < D; ++m) {
          st[m] = A::mul(smu, A::add(g[v][m][c], g[v][c][m]));
          if(m == c) st[m] = A::add(st[m], P[v]);
        }
#pragma unroll
        for(int r = 0; r < D; ++r) {
          T s = A::mul(G[r][0], st[0]);
#pragma unroll
          for(int m = 1; m < D; ++m) s = A::fma(G[r][m], st[m], s);
          S[v][r] = s;
        }
      }
      T tot[NV];  // sum over the vertices w of e_i(w), e_0 = -sum_r H_r, e_r = H_r
#pragma unroll
      for(int i = 0; i < NV; ++i) tot[i] = A::zero();
#pragma unroll
      for(int w = 0; w < NV; ++w) {
        T e[NV];
        e[0] = A::zero();
#pragma unroll
        for(int r = 0; r < D; ++r) {
          T h = A::mul(sm[w * NV], S[0][r]);
#pragma unroll
          for(int v = 1; v < NV; ++v) h = A::fma(sm[w * NV + v], S[v][r], h);
          e[r + 1] = h;
          e[0] = A::sub(e[0], h);
        }
#pragma unroll
        for(int i = 0; i < NV; ++i) {
          tot[i] = A::add(tot[i], e[i]);
          if(i == w) b[w][c] = A::add(b[w][c], A::scale(e[w], 4.f));
          else {
            const int q = edge_node<D>(w, i == w ? (w + 1) % NV : i);
            b[q][c] = A::add(b[q][c], A::scale(e[i], 4.f));
          }
        }
      }
#pragma unroll
      for(int i = 0; i < NV; ++i) b[i][c] = A::sub(b[i][c], tot[i]);
    }
  }
  // Be_pj -= divu int (div u) psi_j
  {
    T dv[NV];
#pragma unroll
    for(int v = 0; v < NV; ++v) {
      T s = g[v][0][0];
#pragma unroll
      for(int k = 1; k < D; ++k) s = A::add(s, g[v][k][k]);
      dv[v] = s;
    }
    const T f = fc.hasDivu ? A::mul(A::from(-fc.divu), J) : A::zero();
#pragma unroll
    for(int j = 0; j < NV; ++j) {
      T s = A::mul(sm[j * NV], dv[0]);
#pragma unroll
      for(int v = 1; v < NV; ++v) s = A::fma(sm[j * NV + v], dv[v], s);
      be[(int64_t)(D * N2 + j) * nE + p] = fc.hasDivu ? A::to(A::mul(f, s)) : 0.;
    }
  }
  // Be_(a,c) -= conv int phi_a (u . grad u)_c
  if(fc.hasConv) {
    const T cf = A::from(-fc.conv);
#pragma unroll 1
    for(int q = 0; q < nq; ++q) {
      T uq[D], f[D];
#pragma unroll
      for(int c = 0; c < D; ++c) {
        T s = A::mul(sPhi[q * N2], U(0, c));
#pragma unroll
        for(int a = 1; a < N2; ++a) s = A::fma(sPhi[q * N2 + a], U(a, c), s);
        uq[c] = s;
      }
#pragma unroll
      for(int c = 0; c < D; ++c) {
        f[c] = A::zero();
#pragma unroll
        for(int k = 0; k < D; ++k) {
          T s = A::mul(sLam[q * NV], g[0][k][c]);
#pragma unroll
          for(int v = 1; v < NV; ++v) s = A::fma(sLam[q * NV + v], g[v][k][c], s);
          f[c] = A::fma(uq[k], s, f[c]);
        }
        f[c] = A::mul(cf, f[c]);
      }
#pragma unroll
      for(int a = 0; a < N2; ++a) {
        const T w = sWphi[q * N2 + a];
#pragma unroll
        for(int c = 0; c < D; ++c) b[a][c] = A::fma(w, f[c], b[a][c]);
      }
    }
  }
  // Be_(a,c) -= mass int udot_c phi_a
  if(fc.hasMass && ud) {
    const T mf = A::from(-fc.mass);
#pragma unroll 1
    for(int d = 0; d < N2; ++d) {
      T x[D];
#pragma unroll
      for(int c = 0; c < D; ++c) x[c] = A::mul(mf, A::load(ud, adr[(int64_t)(D * d + c) * nE + p]));
#pragma unroll
      for(int a = 0; a < N2; ++a) {
        const T m = sM[d * N2 + a];
#pragma unroll
        for(int c = 0; c < D; ++c) b[a][c] = A::fma(m, x[c], b[a][c]);
      }
    }
  }
  double o[N2][D];
#pragma unroll
  for(int a = 0; a < N2; ++a)
#pragma unroll
    for(int c = 0; c < D; ++c) o[a][c] = A::to(A::mul(J, b[a][c]));
  // Be_(a,c) -= int f_c phi_a with the form's own rule, in FP64
  if(nqs > 0) {
    const double sj = -fc.srcCoeff * geo[(int64_t)(D * D) * nE + p];
    double X[NV][D];
#pragma unroll
    for(int v = 0; v < NV; ++v)
#pragma unroll
      for(int k = 0; k < D; ++k) X[v][k] = xy[(int64_t)(D * v + k) * nE + p];
#pragma unroll 1
    for(int q = 0; q < nqs; ++q) {
      double x[D], f[D];
#pragma unroll
      for(int k = 0; k < D; ++k) {
        x[k] = sSl[q * NV] * X[0][k];
#pragma unroll
        for(int v = 1; v < NV; ++v) x[k] += sSl[q * NV + v] * X[v][k];
        f[k] = 0.;
      }
      if constexpr(D == 2) source_value(fc.srcKind, fc.srcParam, x[0], x[1], f);
      else if(fc.srcKind == SRC_CONST_VEC) {
        for(int k = 0; k < D; ++k) f[k] = fc.srcParam[k];
      } else f[0] = source_x(fc.srcKind, fc.srcParam, x[0], x[1], x[D - 1]);
#pragma unroll
      for(int c = 0; c < D; ++c) f[c] *= sj;
      const bool one = D == 3 && fc.srcKind != SRC_CONST_VEC;  // only the first component
#pragma unroll
      for(int a = 0; a < N2; ++a) {
        const double w = sSw[q * N2 + a];
        o[a][0] += w * f[0];
        if(!one)
#pragma unroll
          for(int c = 1; c < D; ++c) o[a][c] += w * f[c];
      }
    }
  }
#pragma unroll
  for(int a = 0; a < N2; ++a)
#pragma unroll
    for(int c = 0; c < D; ++c) be[(int64_t)(D * a + c) * nE + p] = o[a][c];
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

void build_residual_tables(const QuadRule &rule, const QuadRule *own, int dim, ResidualTables &T)
{
  std::memset(&T, 0, sizeof(T));
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
  T.nq = rule.n();
  for(int k = 0; k < T.nq; ++k) {
    basis(rule, k, T.lam[k], T.phi[k]);
    const double w = rule.w[k];
    for(int a = 0; a < n2; ++a) {
      T.wphi[k][a] = w * T.phi[k][a];
      for(int b = 0; b < n2; ++b) T.M[a][b] += w * T.phi[k][a] * T.phi[k][b];
    }
    for(int i = 0; i < nv; ++i)
      for(int j = 0; j < nv; ++j) T.m[i][j] += w * T.lam[k][i] * T.lam[k][j];
  }
  if(!own) return;
  T.nqs = own->n();
  for(int k = 0; k < T.nqs; ++k) {
    double phi[10];
    basis(*own, k, T.slam[k], phi);
    for(int a = 0; a < n2; ++a) T.swphi[k][a] = own->w[k] * phi[a];
  }
}

ResidualTH::~ResidualTH()
{
  cudaFree(tab_);
  cudaFree(be_);
  cudaFree(rowPtr_);
  cudaFree(rowEnt_);
}

int ResidualTH::build(const DeviceMesh &dm, int dim, int64_t nInc, const ResidualTables &T, cudaStream_t s)
{
  dm_ = dm;
  dim_ = dim;
  nq_ = T.nq;
  nqs_ = T.nqs;
  nInc_ = nInc;
  s_ = s;
  const int64_t m = dm.nElm * dm.nloc;
  if(m >= (int64_t)INT32_MAX) {
    set_error("too many element DOFs for the residual's row tables");
    return FE_INVALID_ARG;
  }
  CKR(cudaMalloc(&tab_, sizeof(ResidualTables)));
  CKR(cudaMemcpy(tab_, &T, sizeof(ResidualTables), cudaMemcpyHostToDevice));
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
void ResidualTH::run(const FormCoeffs &fc, const In *u, const In *ud, double *rhs) const
{
  constexpr int N2 = D == 2 ? 6 : 10;
  const int64_t nE = dm_.nElm;
  if(nE <= 0 || nInc_ <= 0) return;
  // SRC_SIN3 is a scalar source: no vector form has it
  const int nqs = fc.srcKind == SRC_NONE || fc.srcKind == SRC_SIN3 ? 0 : nqs_;
  // smaller blocks while the elements do not give every SM one of 128
  const int tb = nE >= 152 * 128 ? 128 : nE >= 152 * 64 ? 64 : 32;
  const size_t sm = table_bytes<A, D>(nq_, nqs) + sizeof(typename A::T) * (size_t)(D * N2 * tb);
  static bool set = false;
  if(!set) {
    cudaFuncSetAttribute(k_residual_elem<D, A>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)(table_bytes<A, D>(RES_MAXQ, RES_MAXQ) + sizeof(typename A::T) * D * N2 * 128));
    set = true;
  }
  (k_residual_elem<D, A><<<(unsigned)((nE + tb - 1) / tb), tb, sm, s_>>>(nE, dm_.adr, dm_.geo, dm_.geoPair, dm_.xy, tab_,
                                                                        fc, u, ud, nq_, nqs, be_),
   ::feng::count_launch());
  (k_residual_rows<<<(unsigned)((nInc_ + 255) / 256), 256, 0, s_>>>(nInc_, rowPtr_, rowEnt_, be_, rhs),
   ::feng::count_launch());
}

void ResidualTH::add64(const FormCoeffs &fc, const double *u, const double *udot, double *rhs) const
{
  if(dim_ == 2) run<2, F64>(fc, u, udot, rhs);
  else run<3, F64>(fc, u, udot, rhs);
}

void ResidualTH::add_df(const FormCoeffs &fc, const float2 *up, const float2 *udp, double *rhs) const
{
  if(dim_ == 2) run<2, DF>(fc, up, udp, rhs);
  else run<3, DF>(fc, up, udp, rhs);
}

}  // namespace feng
