// Element assembly kernels: residual (FP64) and Jacobian (FP64 or FP32) of
// the fused weak forms.
//
// Colored kernels (scalar P2 residual and Jacobian; Taylor-Hood residuals:
// fe_residual.cu): one launch per element color, entries scattered into CSR
// through the element-to-nonzero map as L2 reductions; no two elements of a color share a DOF, so every entry
// receives one contribution per color and the sums are the colored
// read-modify-write's, in color order.
//
// Taylor-Hood Jacobian in FP64: the element matrices of all elements to a
// buffer, then the scatter a color at a time (k_jac_th, k_jac_scatter).
//
// Row-owned kernel (Taylor-Hood FP32 Jacobian, k_matrix_th_rows): one thread per
// CSR row sums the element-matrix rows of the elements holding that DOF, in
// color order, in shared memory; each block writes its contiguous range of
// CSR values once (no atomics, no map, no separate zeroing pass).
//
// Mapping: a block holds 32 elements (lane = element) x 6 warps (warp = P2
// function a of the element).  Thread (e, a) produces the element-matrix rows
// of the DOFs attached to function a -- one row for a scalar field, the two
// component rows (a,x) (a,y) for the Taylor-Hood velocity -- plus, for a < 3,
// the pressure row of P1 function a.  All lanes of a warp read the same
// reference tensor entries (shared-memory broadcast) and their own element's
// data (shared-memory columns), so the contraction has no divergence.
//
// Arithmetic: for affine (P1) geometry the physical gradients are
// grad phi = G^T dphi/dr with G[r][k] = d r_r / d x_k constant per element,
// so every quadrature sum of the reference weak forms factors into constant
// reference tensors contracted with G, |J| and the element DOF values:
//   int dphi_a/dx_k dphi_b/dx_l     = |J| sum_rs G[r][k] G[s][l] K[r][s][a][b]
//   int phi_a phi_c dphi_b/dx_k     = |J| sum_r  G[r][k] T[r][a][c][b]
//   int psi_j dphi_a/dx_k           = |J| sum_r  G[r][k] D[r][j][a]
//   int phi_a phi_b                 = |J| M[a][b]
// The tensors are sums over the same quadrature nodes and weights the
// reference loops over (feSysElm.cpp:530-583, feVectorSysElm.cpp:112-130,
// 390-427, 685-747, 1171-1240, 1454-1530), so the results are the same sums
// regrouped: they agree to rounding.
#include <cuda_runtime.h>

#include <algorithm>

#include "fe_common.h"
#include "fe_device.h"
#include "fe_sources.h"

namespace feng {

namespace {

constexpr int EPB = 32;  // elements per block (one per lane)
template <typename V>
struct SharedTensors {
  V K[2][2][6][6];
  V T[2][6][6][6];
  V D[2][3][6];
  V M[6][6];
};

template <typename V>
__device__ void load_tensors(SharedTensors<V> &s, const RefTensors *g)
{
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
  const double *K = &g->K[0][0][0][0], *T = &g->T[0][0][0][0], *D = &g->D[0][0][0], *M = &g->M[0][0];
  V *sK = &s.K[0][0][0][0], *sT = &s.T[0][0][0][0], *sD = &s.D[0][0][0], *sM = &s.M[0][0];
  for(int i = tid; i < 144; i += nt) sK[i] = (V)K[i];
  for(int i = tid; i < 432; i += nt) sT[i] = (V)T[i];
  for(int i = tid; i < 36; i += nt) sD[i] = (V)D[i];
  for(int i = tid; i < 36; i += nt) sM[i] = (V)M[i];
}

// ---------------------------------------------------------------------------
// Residual, scalar P2 (DIFFUSION + SOURCE).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(EPB * 6) k_residual_p2(DeviceMesh dm, FormCoeffs fc,
                                                        const RefTensors *__restrict__ gT,
                                                        const double *__restrict__ u, double t,
                                                        int64_t nInc, double *__restrict__ rhs,
                                                        int64_t begin, int64_t end)
{
  __shared__ SharedTensors<double> sT;
  __shared__ double sU[6][EPB];
  __shared__ double sG[5][EPB];
  __shared__ double sF[16][EPB];
  __shared__ int32_t sA[6][EPB];
  const int lane = threadIdx.x, a = threadIdx.y;
  const int64_t p = begin + (int64_t)blockIdx.x * EPB + lane;
  const bool live = p < end;
  const int64_t nE = dm.nElm;
  load_tensors(sT, gT);
  if(live) {
    int32_t d = dm.adr[(int64_t)a * nE + p];
    sA[a][lane] = d;
    sU[a][lane] = u[d];
    if(a < 5) sG[a][lane] = dm.geo[(int64_t)a * nE + p];
  }
  const int nq = gT->nq;
  if(fc.srcKind != SRC_NONE && live) {
    const double x0 = dm.xy[0 * nE + p], y0 = dm.xy[1 * nE + p], x1 = dm.xy[2 * nE + p],
                 y1 = dm.xy[3 * nE + p], x2 = dm.xy[4 * nE + p], y2 = dm.xy[5 * nE + p];
    for(int q = a; q < nq; q += 6) {
      const double r = gT->qr[q], s = gT->qs[q];
      const double x = x0 * (1. - r - s) + x1 * r + x2 * s;
      const double y = y0 * (1. - r - s) + y1 * r + y2 * s;
      double f[2];
      source_value(fc.srcKind, fc.srcParam, x, y, f);
      sF[q][lane] = f[0];
    }
  }
  __syncthreads();
  if(!live) return;
  const double G[2][2] = {{sG[0][lane], sG[1][lane]}, {sG[2][lane], sG[3][lane]}};
  const double J = sG[4][lane];
  double be = 0.;
  if(fc.hasDiff) {
    // Be_a -= k grad phi_a . grad u  (feSysElm.cpp:560-583)
    double GG[2][2];
    for(int r = 0; r < 2; ++r)
      for(int s2 = 0; s2 < 2; ++s2) GG[r][s2] = G[r][0] * G[s2][0] + G[r][1] * G[s2][1];
    double acc = 0.;
    for(int b = 0; b < 6; ++b) {
      double L = 0.;
      for(int r = 0; r < 2; ++r)
        for(int s2 = 0; s2 < 2; ++s2) L += GG[r][s2] * sT.K[r][s2][a][b];
      acc += L * sU[b][lane];
    }
    be -= fc.diff * acc * J;
  }
  if(fc.srcKind != SRC_NONE) {
    // Be_a -= phi_a S jac w  (feSysElm.cpp:16-27)
    double acc = 0.;
    for(int q = 0; q < nq; ++q) acc += gT->phi[q][a] * sF[q][lane] * gT->qw[q];
    be -= fc.srcCoeff * acc * J;
  }
  const int32_t d = sA[a][lane];
  if(d < nInc) atomicAdd(rhs + d, be);  // one contribution per DOF and color
}

// ---------------------------------------------------------------------------
// Jacobian, scalar P2 (DIFFUSION).
// ---------------------------------------------------------------------------
template <typename V>
__global__ void __launch_bounds__(EPB * 6) k_matrix_p2(DeviceMesh dm, FormCoeffs fc,
                                                      const RefTensors *__restrict__ gT,
                                                      V *__restrict__ values, int64_t begin,
                                                      int64_t end)
{
  __shared__ SharedTensors<V> sT;
  __shared__ V sG[5][EPB];
  const int lane = threadIdx.x, a = threadIdx.y;
  const int64_t p = begin + (int64_t)blockIdx.x * EPB + lane;
  const bool live = p < end;
  const int64_t nE = dm.nElm;
  load_tensors(sT, gT);
  if(live && a < 5) sG[a][lane] = (V)dm.geo[(int64_t)a * nE + p];
  __syncthreads();
  if(!live || !fc.hasDiff) return;
  const V G[2][2] = {{sG[0][lane], sG[1][lane]}, {sG[2][lane], sG[3][lane]}};
  const V cJ = (V)fc.diff * sG[4][lane];
  V GG[2][2];
  for(int r = 0; r < 2; ++r)
    for(int s2 = 0; s2 < 2; ++s2) GG[r][s2] = G[r][0] * G[s2][0] + G[r][1] * G[s2][1];
  for(int b = 0; b < 6; ++b) {
    V L = 0;
    for(int r = 0; r < 2; ++r)
      for(int s2 = 0; s2 < 2; ++s2) L += GG[r][s2] * sT.K[r][s2][a][b];
    const int32_t pos = dm.map[(int64_t)(a * 6 + b) * nE + p];
    if(pos >= 0) atomicAdd(values + pos, cJ * L);  // one contribution per entry and color
  }
}

__global__ void k_split_pairs(int64_t n, const double *__restrict__ x, float2 *__restrict__ out)
{
  for(int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double v = x[i];
    const float h = __double2float_rn(v);
    out[i] = make_float2(h, __double2float_rn(v - (double)h));
  }
}

// Local entry k = a*18 + j of the staged rows (2a+m) of a Taylor-Hood
// element matrix -> index of the element-to-nonzero map (i = 2a+m; j < 12
// velocity column j, 12 <= j < 15 pressure column j-12, 15 <= j < 18 the
// entry of pressure row j-15 in column i).
__device__ __forceinline__ int th_map_index(int k, int m)
{
  const int a = k / 18, j = k % 18, i = 2 * a + m;
  return j < 15 ? i * 15 + j : (12 + j - 15) * 15 + i;
}

// ---------------------------------------------------------------------------
// Jacobian, Taylor-Hood P2-P1: element matrices, then the colored scatter.
// ---------------------------------------------------------------------------
constexpr int TH_ENT = 216;  // structurally nonzero entries: entry m * 108 + k (th_map_index)

// Entries of the elements [p0, end) to buf[entry][p - p0] (leading dimension
// ld).  Thread (e, a), as above.
//
// A P2 function's gradient is affine, so u . grad u and its derivative need no
// tensor over three P2 functions: with S[a][b][j] = int phi_a phi_b psi_j
//   int phi_a phi_b d_n u_m     = J sum_v (d_n u_m)(vertex v) S[a][b][v],
//   int phi_a psi_j u . grad l_i = J sum_c (u_c . grad l_i) S[a][c][j],
// and grad phi_b is 4 l_i grad l_i - grad l_i or 4 (l_i grad l_j + l_j grad
// l_i): the rule's own sums regrouped, 1,700 products an element for 3,300.
// Bound: the FP64 pipe (32,768 elements: 91 us of it, 114 measured).  A color
// at a time, with the scatter inside, the 128 x 128 Jacobian was six launches
// of 170 blocks (the chip holds 600), 72 us each; now 114 us and the colors'
// scatters of 12 (cold).  Call with its 28 MB copy to the host: 732 -> 455 us.
template <typename V>
__global__ void __launch_bounds__(EPB * 6) k_jac_th(DeviceMesh dm, FormCoeffs fc, const RefTensors *__restrict__ gT,
                                                   const double *__restrict__ u, double c0, V *__restrict__ buf,
                                                   int64_t ld, int64_t p0, int64_t end)
{
  __shared__ V sK[2][2][6][6], sS[6][6][3], sD[2][3][6], sM[6][6];
  __shared__ V sU[12][EPB], sA[2][6][EPB], sG[3][2][2][EPB];
  const int lane = threadIdx.x, a = threadIdx.y, tid = a * EPB + lane;
  for(int i = tid; i < 144; i += EPB * 6) (&sK[0][0][0][0])[i] = (V)(&gT->K[0][0][0][0])[i];
  for(int i = tid; i < 108; i += EPB * 6) (&sS[0][0][0])[i] = (V)(&gT->S[0][0][0])[i];
  for(int i = tid; i < 36; i += EPB * 6) {
    (&sD[0][0][0])[i] = (V)(&gT->D[0][0][0])[i];
    (&sM[0][0])[i] = (V)(&gT->M[0][0])[i];
  }
  const int64_t nE = dm.nElm, q = p0 + (int64_t)blockIdx.x * EPB + lane, p = q < end ? q : end - 1;
  V G[2][2];
#pragma unroll
  for(int r = 0; r < 2; ++r)
#pragma unroll
    for(int k = 0; k < 2; ++k) G[r][k] = (V)dm.geo[(int64_t)(2 * r + k) * nE + p];
  const V J = (V)dm.geo[4 * nE + p], cc = (V)fc.conv * J;
  if(fc.hasConv) {
    const V x = (V)u[dm.adr[(int64_t)(2 * a) * nE + p]], y = (V)u[dm.adr[(int64_t)(2 * a + 1) * nE + p]];
    sU[2 * a][lane] = x;
    sU[2 * a + 1][lane] = y;
#pragma unroll
    for(int r = 0; r < 2; ++r) sA[r][a][lane] = cc * (G[r][0] * x + G[r][1] * y);
    __syncthreads();
    // cc d_n u_m at vertex v: differences of the quadratic's coefficients
    // 2 u_v and 4 u_(v,i) - u_v - u_i
    const int v = a % 3, m = a / 3;
    V h[3];
#pragma unroll
    for(int i = 0; i < 3; ++i) {
      const int e = v + i == 1 ? 3 : (v + i == 3 ? 4 : 5);  // edges (0,1) (1,2) (2,0)
      const V uv = sU[2 * v + m][lane];
      h[i] = i == v ? uv + uv : (V)4 * sU[2 * e + m][lane] - (uv + sU[2 * i + m][lane]);
    }
    const V d0 = cc * (h[1] - h[0]), d1 = cc * (h[2] - h[0]);
#pragma unroll
    for(int n = 0; n < 2; ++n) sG[v][n][m][lane] = G[0][n] * d0 + G[1][n] * d1;
  }
  __syncthreads();
  if(q >= end) return;
  V *out = buf + (q - p0) + (int64_t)(a * 18) * ld;
  const int64_t ldm = 108 * ld;  // from row component 0 to 1

  V W[6] = {0, 0, 0, 0, 0, 0};  // cc int phi_a u . grad phi_b
  V g[3][2][2];
  if(fc.hasConv) {
    V R[3][3];  // [i][j]: cc int phi_a psi_j u . grad l_i
#pragma unroll
    for(int r = 0; r < 2; ++r)
#pragma unroll
      for(int j = 0; j < 3; ++j) {
        V s = sA[r][0][lane] * sS[a][0][j];
#pragma unroll
        for(int c = 1; c < 6; ++c) s += sA[r][c][lane] * sS[a][c][j];
        R[r + 1][j] = s;
      }
#pragma unroll
    for(int j = 0; j < 3; ++j) R[0][j] = -(R[1][j] + R[2][j]);
#pragma unroll
    for(int i = 0; i < 3; ++i) {
      W[i] = (V)4 * R[i][i] - (R[i][0] + R[i][1] + R[i][2]);
      W[3 + i] = (V)4 * (R[(i + 1) % 3][i] + R[i][(i + 1) % 3]);
    }
#pragma unroll
    for(int v = 0; v < 3; ++v)
#pragma unroll
      for(int n = 0; n < 2; ++n)
#pragma unroll
        for(int m = 0; m < 2; ++m) g[v][n][m] = sG[v][n][m][lane];
  }
  const V cs = fc.hasSigma ? -(V)fc.sigma * (V)fc.mu * J : (V)0, cm = fc.hasMass ? (V)fc.mass * (V)c0 * J : (V)0;
  V H[2][2];
#pragma unroll
  for(int r = 0; r < 2; ++r)
#pragma unroll
    for(int k = 0; k < 2; ++k) H[r][k] = cs * G[r][k];
#pragma unroll
  for(int b = 0; b < 6; ++b) {
    // A_(a,m),(b,n) += -c mu [ delta_mn grad phi_a . grad phi_b + d_n phi_a d_m phi_b ]
    // (feVectorSysElm.cpp:1454-1492)
    V A[2][2] = {{0, 0}, {0, 0}}, d = W[b];  // A[m][n]; d: the delta_mn terms
    if(fc.hasSigma) {
#pragma unroll
      for(int m = 0; m < 2; ++m) {
        const V P0 = sK[0][0][a][b] * G[0][m] + sK[0][1][a][b] * G[1][m],
                P1 = sK[1][0][a][b] * G[0][m] + sK[1][1][a][b] * G[1][m];
#pragma unroll
        for(int n = 0; n < 2; ++n) A[m][n] = H[0][n] * P0 + H[1][n] * P1;
      }
      d += A[0][0] + A[1][1];
    }
    // (feVectorSysElm.cpp:390-408)
    if(fc.hasMass) d += cm * sM[a][b];
    // A_(a,m),(b,n) += c [ delta_mn phi_a (u0 . grad phi_b) + phi_a phi_b d_n u0_m ]
    // (vectorDotGradShapeDotShape + shapeDotTensorDotShape, feVectorSpace.cpp:202-290)
    if(fc.hasConv)
#pragma unroll
      for(int v = 0; v < 3; ++v)
#pragma unroll
        for(int m = 0; m < 2; ++m)
#pragma unroll
          for(int n = 0; n < 2; ++n) A[m][n] += g[v][n][m] * sS[a][b][v];
    A[0][0] += d;
    A[1][1] += d;
#pragma unroll
    for(int m = 0; m < 2; ++m)
#pragma unroll
      for(int n = 0; n < 2; ++n) out[m * ldm + (int64_t)(2 * b + n) * ld] = A[m][n];
  }
  // Pressure columns of rows (a,m) and the column (a,m) of the pressure rows:
  // both are int psi_j d_m phi_a.
  const V sj = (V)fc.sigma * J, dj = (V)fc.divu * J;
#pragma unroll
  for(int m = 0; m < 2; ++m)
#pragma unroll
    for(int j = 0; j < 3; ++j) {
      const V bp = G[0][m] * sD[0][j][a] + G[1][m] * sD[1][j][a];
      if(fc.hasSigma) out[m * ldm + (int64_t)(12 + j) * ld] = sj * bp;
      if(fc.hasDivu) out[m * ldm + (int64_t)(15 + j) * ld] = dj * bp;
    }
}

// values += the entries of the elements [begin, end) of one color.  Within a
// color every CSR entry receives at most one contribution, so the reduction
// in L2 (no round trip to the SM) gives the bits of a read-modify-write.
constexpr int JAC_BATCH = 6;
template <typename V>
__global__ void __launch_bounds__(256) k_jac_scatter(int64_t nE, const int32_t *__restrict__ map, int hasSigma,
                                                    int hasDivu, const V *__restrict__ buf, int64_t ld, int64_t p0,
                                                    int64_t begin, int64_t end, V *__restrict__ values)
{
  const int64_t p = begin + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if(p >= end) return;
  int32_t pos[JAC_BATCH];
  V add[JAC_BATCH];
#pragma unroll
  for(int t = 0; t < JAC_BATCH; ++t) {
    const int e = (int)blockIdx.y * JAC_BATCH + t, m = e >= 108, k = m ? e - 108 : e, j = k % 18;
    const bool on = j < 12 || (j < 15 ? hasSigma : hasDivu);
    pos[t] = on ? __ldg(map + (int64_t)th_map_index(k, m) * nE + p) : -1;
    add[t] = on ? buf[(int64_t)e * ld + p - p0] : (V)0;
  }
#pragma unroll
  for(int t = 0; t < JAC_BATCH; ++t)
    if(pos[t] >= 0) atomicAdd(values + pos[t], add[t]);
}

int64_t nblocks(int64_t begin, int64_t end) { return (end - begin + EPB - 1) / EPB; }

// ---------------------------------------------------------------------------
// Row-owned Jacobian, Taylor-Hood.
// ---------------------------------------------------------------------------
template <typename V>
__global__ void k_pack_th(DeviceMesh dm, int hasConv, const double *__restrict__ u, V *__restrict__ pack)
{
  const int64_t nE = dm.nElm;
  for(int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < nE; p += (int64_t)gridDim.x * blockDim.x) {
    V *o = pack + p * ROWASM_PACK;
#pragma unroll
    for(int i = 0; i < 12; ++i) o[i] = hasConv ? (V)u[dm.adr[(int64_t)i * nE + p]] : (V)0;
#pragma unroll
    for(int k = 0; k < 5; ++k) o[12 + k] = (V)dm.geo[(int64_t)k * nE + p];
  }
}

// Both component rows (a, 0) and (a, 1) of velocity function a of an
// element, from its packed data e (u, G, J): A[m][12] velocity columns and
// the pressure-column factors Bp[m][3], by the contraction described above for
// one (element, a) (k_jac_th regroups it: the two agree to rounding).
template <typename V>
__device__ __forceinline__ void th_rows_pair(const SharedTensors<V> &sT, const FormCoeffs &fc, double c0,
                                             const V *e, int a, V (&A)[2][12], V (&Bp)[2][3])
{
  const V G[2][2] = {{e[12], e[13]}, {e[14], e[15]}};
  const V J = e[16];
#pragma unroll
  for(int m = 0; m < 2; ++m)
#pragma unroll
    for(int j = 0; j < 12; ++j) A[m][j] = 0;
  if(fc.hasConv) {
    V U[12];
#pragma unroll
    for(int i = 0; i < 12; ++i) U[i] = e[i];
    V V0[2][6];
#pragma unroll
    for(int c = 0; c < 6; ++c)
#pragma unroll
      for(int q = 0; q < 2; ++q) V0[q][c] = U[2 * c] * G[q][0] + U[2 * c + 1] * G[q][1];
    const V cc = (V)fc.conv * J;
#pragma unroll
    for(int b = 0; b < 6; ++b) {
      V W = 0, Z[2][2] = {{0, 0}, {0, 0}};
#pragma unroll
      for(int c = 0; c < 6; ++c) {
        W += V0[0][c] * sT.T[0][a][c][b] + V0[1][c] * sT.T[1][a][c][b];
        const V t0 = sT.T[0][a][b][c], t1 = sT.T[1][a][b][c];
        const V uc0 = U[2 * c], uc1 = U[2 * c + 1];
        Z[0][0] += uc0 * t0; Z[0][1] += uc1 * t0;
        Z[1][0] += uc0 * t1; Z[1][1] += uc1 * t1;
      }
#pragma unroll
      for(int m = 0; m < 2; ++m)
#pragma unroll
        for(int n = 0; n < 2; ++n) {
          V v = G[0][n] * Z[0][m] + G[1][n] * Z[1][m];
          if(m == n) v += W;
          A[m][2 * b + n] += cc * v;
        }
    }
  }
  if(fc.hasSigma) {
    const V cs = -(V)fc.sigma * (V)fc.mu * J;
    V GG[2][2][2][2];
#pragma unroll
    for(int k = 0; k < 2; ++k)
#pragma unroll
      for(int l = 0; l < 2; ++l)
#pragma unroll
        for(int q = 0; q < 2; ++q)
#pragma unroll
          for(int s2 = 0; s2 < 2; ++s2) GG[k][l][q][s2] = G[q][k] * G[s2][l];
#pragma unroll
    for(int b = 0; b < 6; ++b) {
      V S[2][2];
#pragma unroll
      for(int k = 0; k < 2; ++k)
#pragma unroll
        for(int l = 0; l < 2; ++l) {
          V v = 0;
#pragma unroll
          for(int q = 0; q < 2; ++q)
#pragma unroll
            for(int s2 = 0; s2 < 2; ++s2) v += GG[k][l][q][s2] * sT.K[q][s2][a][b];
          S[k][l] = v;
        }
      const V tr = S[0][0] + S[1][1];
#pragma unroll
      for(int m = 0; m < 2; ++m)
#pragma unroll
        for(int n = 0; n < 2; ++n) A[m][2 * b + n] += cs * ((m == n ? tr : (V)0) + S[n][m]);
    }
  }
  if(fc.hasMass) {
    const V cm = (V)fc.mass * (V)c0 * J;
#pragma unroll
    for(int b = 0; b < 6; ++b) {
      A[0][2 * b] += cm * sT.M[a][b];
      A[1][2 * b + 1] += cm * sT.M[a][b];
    }
  }
#pragma unroll
  for(int m = 0; m < 2; ++m)
#pragma unroll
    for(int j = 0; j < 3; ++j) Bp[m][j] = (G[0][m] * sT.D[0][j][a] + G[1][m] * sT.D[1][j][a]) * J;
}

// Thread = unit (RowAsm): a pair of component rows of one velocity node, or
// one row.  Entry (p, li): li < 12 is velocity row (a = li / 2, component
// m = li % 2) of element p, whose 12 velocity and 3 pressure columns are the
// element matrix's row; li >= 12 is pressure row j = li - 12,
// whose 12 velocity columns are divu * int psi_j d_m phi_a.  A pair takes
// the entries of its component-0 row and builds both rows (same columns,
// same offsets); th_rows_pair.
template <typename V>
__global__ void __launch_bounds__(256) k_matrix_th_rows(RowAsm ra, FormCoeffs fc, const RefTensors *__restrict__ gT,
                                                        double c0, V *__restrict__ values, int accumulate)
{
  extern __shared__ __align__(16) unsigned char rowsmem[];
  V *sv = reinterpret_cast<V *>(rowsmem);
  __shared__ SharedTensors<V> sT;
  load_tensors(sT, gT);
  const int32_t uA = ra.blockUnits[blockIdx.x], uB = ra.blockUnits[blockIdx.x + 1];
  const int32_t base = ra.ia[ra.unitRow[uA]], L = ra.ia[ra.unitRow[uB]] - base;
  for(int i = threadIdx.x; i < L; i += blockDim.x) sv[i] = accumulate ? values[base + i] : (V)0;
  __syncthreads();
  const int32_t u = uA + (int32_t)threadIdx.x;
  if(u < uB && ra.unitTwo[u]) {
    const int32_t r = ra.unitRow[u];
    V *row0 = sv + (ra.ia[r] - base), *row1 = sv + (ra.ia[r + 1] - base);
    const V *pk = reinterpret_cast<const V *>(ra.pack);
    for(int32_t k = ra.rowPtr[r]; k < ra.rowPtr[r + 1]; ++k) {
      const int32_t ent = ra.rowEnt[k];
      const int64_t p = ent >> 4;
      const int a = (ent & 15) >> 1;
      uint8_t off[16];
      *reinterpret_cast<uint4 *>(off) = reinterpret_cast<const uint4 *>(ra.offs)[k];
      V A[2][12], Bp[2][3];
      th_rows_pair<V>(sT, fc, c0, pk + p * ROWASM_PACK, a, A, Bp);
#pragma unroll
      for(int j = 0; j < 12; ++j)
        if(off[j] != 255) {
          row0[off[j]] += A[0][j];
          row1[off[j]] += A[1][j];
        }
#pragma unroll
      for(int j = 0; j < 3; ++j)
        if(off[12 + j] != 255) {
          row0[off[12 + j]] += fc.hasSigma ? (V)fc.sigma * Bp[0][j] : (V)0;
          row1[off[12 + j]] += fc.hasSigma ? (V)fc.sigma * Bp[1][j] : (V)0;
        }
    }
  } else if(u < uB) {
    const int32_t r = ra.unitRow[u];
    V *row = sv + (ra.ia[r] - base);
    const V *pk = reinterpret_cast<const V *>(ra.pack);
    for(int32_t k = ra.rowPtr[r]; k < ra.rowPtr[r + 1]; ++k) {
      const int32_t ent = ra.rowEnt[k];
      const int64_t p = ent >> 4;
      const int li = ent & 15;
      uint8_t off[16];
      *reinterpret_cast<uint4 *>(off) = reinterpret_cast<const uint4 *>(ra.offs)[k];
      const V *e = pk + p * ROWASM_PACK;
      const V G[2][2] = {{e[12], e[13]}, {e[14], e[15]}};
      const V J = e[16];
      if(li < 12) {
        const int a = li >> 1, m = li & 1;
        V A[12];
#pragma unroll
        for(int j = 0; j < 12; ++j) A[j] = 0;
        if(fc.hasConv) {
          V U[12];
#pragma unroll
          for(int i = 0; i < 12; ++i) U[i] = e[i];
          V V0[2][6];
#pragma unroll
          for(int c = 0; c < 6; ++c)
#pragma unroll
            for(int q = 0; q < 2; ++q) V0[q][c] = U[2 * c] * G[q][0] + U[2 * c + 1] * G[q][1];
          const V cc = (V)fc.conv * J;
#pragma unroll
          for(int b = 0; b < 6; ++b) {
            V W = 0, Z0 = 0, Z1 = 0;  // Z_q = sum_c U_cm T[q][a][b][c]
#pragma unroll
            for(int c = 0; c < 6; ++c) {
              W += V0[0][c] * sT.T[0][a][c][b] + V0[1][c] * sT.T[1][a][c][b];
              const V t0 = sT.T[0][a][b][c], t1 = sT.T[1][a][b][c];
              const V ucm = U[2 * c + m];
              Z0 += ucm * t0;
              Z1 += ucm * t1;
            }
#pragma unroll
            for(int n = 0; n < 2; ++n) {
              V v = G[0][n] * Z0 + G[1][n] * Z1;
              if(m == n) v += W;
              A[2 * b + n] += cc * v;
            }
          }
        }
        if(fc.hasSigma) {
          const V cs = -(V)fc.sigma * (V)fc.mu * J;
          V GG[2][2][2][2];
#pragma unroll
          for(int kk = 0; kk < 2; ++kk)
#pragma unroll
            for(int l = 0; l < 2; ++l)
#pragma unroll
              for(int q = 0; q < 2; ++q)
#pragma unroll
                for(int s2 = 0; s2 < 2; ++s2) GG[kk][l][q][s2] = G[q][kk] * G[s2][l];
#pragma unroll
          for(int b = 0; b < 6; ++b) {
            V S[2][2];
#pragma unroll
            for(int kk = 0; kk < 2; ++kk)
#pragma unroll
              for(int l = 0; l < 2; ++l) {
                V v = 0;
#pragma unroll
                for(int q = 0; q < 2; ++q)
#pragma unroll
                  for(int s2 = 0; s2 < 2; ++s2) v += GG[kk][l][q][s2] * sT.K[q][s2][a][b];
                S[kk][l] = v;
              }
            const V tr = S[0][0] + S[1][1];
#pragma unroll
            for(int n = 0; n < 2; ++n) A[2 * b + n] += cs * ((m == n ? tr : (V)0) + S[n][m]);
          }
        }
        if(fc.hasMass) {
          const V cm = (V)fc.mass * (V)c0 * J;
#pragma unroll
          for(int b = 0; b < 6; ++b) A[2 * b + m] += cm * sT.M[a][b];
        }
#pragma unroll
        for(int j = 0; j < 12; ++j)
          if(off[j] != 255) row[off[j]] += A[j];
#pragma unroll
        for(int j = 0; j < 3; ++j) {
          const V bp = (G[0][m] * sT.D[0][j][a] + G[1][m] * sT.D[1][j][a]) * J;
          if(off[12 + j] != 255) row[off[12 + j]] += fc.hasSigma ? (V)fc.sigma * bp : (V)0;
        }
      } else {
        const int j = li - 12;
#pragma unroll
        for(int a = 0; a < 6; ++a)
#pragma unroll
          for(int m = 0; m < 2; ++m) {
            const V bp = (G[0][m] * sT.D[0][j][a] + G[1][m] * sT.D[1][j][a]) * J;
            if(off[2 * a + m] != 255) row[off[2 * a + m]] += fc.hasDivu ? (V)fc.divu * bp : (V)0;
          }
      }
    }
  }
  __syncthreads();
  for(int i = threadIdx.x; i < L; i += blockDim.x) values[base + i] = sv[i];
}

int pack_grid(int64_t n) { return (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 8192)); }

}  // namespace

void launch_pack_th_f32(const DeviceMesh &dm, const FormCoeffs &fc, const double *u, float *pack, cudaStream_t s)
{
  (k_pack_th<float><<<pack_grid(dm.nElm), 256, 0, s>>>(dm, fc.hasConv, u, pack), ::feng::count_launch());
}

void launch_matrix_th_rows_f32(const RowAsm &ra, const FormCoeffs &fc, const RefTensors *dT, double c0,
                               float *values, int accumulate, cudaStream_t s)
{
  if(ra.nBlocks < 1) return;
  (k_matrix_th_rows<float><<<ra.nBlocks, 256, ra.capBytes, s>>>(ra, fc, dT, c0, values, accumulate),
   ::feng::count_launch());
}

void launch_split_pairs(int64_t n, const double *x, float2 *out, cudaStream_t s)
{
  const int g = (int)std::max<int64_t>(1, std::min<int64_t>((n + 255) / 256, 4096));
  (k_split_pairs<<<g, 256, 0, s>>>(n, x, out), ::feng::count_launch());
}

void launch_assemble_residual(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensors *dT,
                              const double *u, double t, int64_t nInc, double *rhs, int64_t begin, int64_t end,
                              cudaStream_t s)
{
  if(end <= begin) return;
  dim3 block(EPB, 6);
  (k_residual_p2<<<nblocks(begin, end), block, 0, s>>>(dm, fc, dT, u, t, nInc, rhs, begin, end), ::feng::count_launch());
}

void launch_assemble_matrix_p2_f64(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensors *dT, double *values,
                                   int64_t begin, int64_t end, cudaStream_t s)
{
  if(end <= begin) return;
  (k_matrix_p2<double><<<nblocks(begin, end), dim3(EPB, 6), 0, s>>>(dm, fc, dT, values, begin, end),
   ::feng::count_launch());
}

void launch_assemble_matrix_p2_f32(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensors *dT, float *values,
                                   int64_t begin, int64_t end, cudaStream_t s)
{
  if(end <= begin) return;
  (k_matrix_p2<float><<<nblocks(begin, end), dim3(EPB, 6), 0, s>>>(dm, fc, dT, values, begin, end),
   ::feng::count_launch());
}

int64_t matrix_th_chunk(int64_t nElm) { return std::min<int64_t>(nElm, 1 << 18); }
size_t matrix_th_buffer_bytes(int64_t nElm, int valueBytes)
{
  return (size_t)TH_ENT * (size_t)matrix_th_chunk(nElm) * valueBytes;
}

template <typename V>
static void matrix_th(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensors *dT, const double *u, double c0,
                      V *buf, V *values, cudaStream_t s)
{
  const int64_t ch = matrix_th_chunk(dm.nElm);
  int c = 0;
  for(int64_t p0 = 0; p0 < dm.nElm; p0 += ch) {
    const int64_t p1 = std::min(dm.nElm, p0 + ch);
    (k_jac_th<V><<<(unsigned)nblocks(p0, p1), dim3(EPB, 6), 0, s>>>(dm, fc, dT, u, c0, buf, ch, p0, p1),
     ::feng::count_launch());
    for(int64_t b = p0; b < p1;) {
      while(dm.colorOff[c + 1] <= b) ++c;
      const int64_t e = std::min(p1, dm.colorOff[c + 1]);
      (k_jac_scatter<V><<<dim3((unsigned)((e - b + 255) / 256), TH_ENT / JAC_BATCH), 256, 0, s>>>(
           dm.nElm, dm.map, fc.hasSigma, fc.hasDivu, buf, ch, p0, b, e, values),
       ::feng::count_launch());
      b = e;
    }
  }
}

void launch_matrix_th_f64(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensors *dT, const double *u, double c0,
                          double *buf, double *values, cudaStream_t s)
{
  matrix_th<double>(dm, fc, dT, u, c0, buf, values, s);
}

void launch_matrix_th_f32(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensors *dT, const double *u, double c0,
                          float *buf, float *values, cudaStream_t s)
{
  matrix_th<float>(dm, fc, dT, u, c0, buf, values, s);
}

}  // namespace feng
