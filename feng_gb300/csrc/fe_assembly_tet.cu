// Element assembly on tetrahedra: scalar P2 (DIFFUSION + SOURCE, the
// reference's feSysElm_Diffusion<3> and feSysElm_Source on feSpaceTetPn(2),
// src/feSysElm.cpp:16-27, 520-589) and Taylor-Hood P2-P1 (the vector forms
// of src/feVectorSysElm.cpp in three dimensions, which the reference
// instantiates only in two).
//
// Colored kernels: one launch per element color; a block holds 32 elements
// (lane = element) x 10 warps (warp = P2 function a).  Thread (e, a) forms
// the element-matrix rows of the DOFs of function a (one scalar row, or the
// three velocity component rows), and threads a < 4 the pressure row of P1
// function a.  Entries go to the CSR values through the element-to-nonzero
// map as L2 reductions (one contribution per entry and color: the sums of a
// colored read-modify-write, in color order).
//
// Arithmetic: affine (P1) geometry, so grad phi = G^T dphi/d(r,s,t) with
// G[r][k] = d r_r / d x_k constant per element and every quadrature sum of
// the weak forms is a reference tensor (RefTensorsTet, built from the same
// rule's nodes and weights) contracted with G, J and the element's DOF values:
//   int dphi_a/dx_k dphi_b/dx_l = J sum_rs G[r][k] G[s][l] K[r][s][a][b]
//   int phi_a phi_c dphi_b/dx_k = J sum_r  G[r][k] T[r][a][c][b]
//   int psi_j dphi_a/dx_k       = J sum_r  G[r][k] D[r][j][a]
//   int phi_a phi_b             = J M[a][b]
// Source terms are summed over the rule's nodes (non-polynomial integrands).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fe_common.h"
#include "fe_device.h"
#include "fe_mesh3d.h"
#include "fe_setup.h"
#include "fe_sources.h"

namespace feng {

namespace {

constexpr int EPB = 32;
constexpr int TPB = 10;  // warps per block: one per P2 function
constexpr int NTEN = 900 + 3000 + 120 + 100;  // K, T, D, M

template <typename V>
struct TetTensors {
  const V *K, *T, *D, *M;
  __device__ V k(int r, int s, int a, int b) const { return K[((r * 3 + s) * 10 + a) * 10 + b]; }
  __device__ V t(int r, int a, int c, int b) const { return T[((r * 10 + a) * 10 + c) * 10 + b]; }
  __device__ V d(int r, int j, int a) const { return D[(r * 4 + j) * 10 + a]; }
  __device__ V m(int a, int b) const { return M[a * 10 + b]; }
};

template <typename V>
__device__ TetTensors<V> load_tet_tensors(V *sh, const RefTensorsTet *g)
{
  const int tid = threadIdx.y * blockDim.x + threadIdx.x, nt = blockDim.x * blockDim.y;
  const double *src[4] = {&g->K[0][0][0][0], &g->T[0][0][0][0], &g->D[0][0][0], &g->M[0][0]};
  const int len[4] = {900, 3000, 120, 100};
  int off = 0;
  for(int k = 0; k < 4; ++k) {
    for(int i = tid; i < len[k]; i += nt) sh[off + i] = (V)src[k][i];
    off += len[k];
  }
  return TetTensors<V>{sh, sh + 900, sh + 3900, sh + 4020};
}

// ---------------------------------------------------------------------------
// Residual, scalar P2, FP64 (Taylor-Hood: fe_residual.cu).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(EPB *TPB) k_residual_tet(DeviceMesh dm, FormCoeffs fc, const RefTensorsTet *__restrict__ gT,
                                                           const double *__restrict__ u, int64_t nInc,
                                                           double *__restrict__ rhs, int64_t begin, int64_t end)
{
  extern __shared__ __align__(16) double smem[];
  const int nq = gT->nq;
  double *sTen = smem;
  double *sU = sTen + NTEN;           // [10][EPB]
  double *sG = sU + 10 * EPB;         // [10][EPB]
  double *sF = sG + 10 * EPB;         // [nq][EPB]
  const int lane = threadIdx.x, a = threadIdx.y;
  const int64_t p = begin + (int64_t)blockIdx.x * EPB + lane;
  const bool live = p < end;
  const int64_t nE = dm.nElm;
  const TetTensors<double> Tt = load_tet_tensors(sTen, gT);
  if(live) {
    sU[a * EPB + lane] = u[dm.adr[(int64_t)a * nE + p]];
    sG[a * EPB + lane] = dm.geo[(int64_t)a * nE + p];
    if(fc.srcKind == SRC_SIN3) {
      double X[4][3];
      for(int v = 0; v < 4; ++v)
        for(int k = 0; k < 3; ++k) X[v][k] = dm.xy[(int64_t)(3 * v + k) * nE + p];
      for(int q = a; q < nq; q += TPB) {
        const double r = gT->qr[q], s = gT->qs[q], t = gT->qt[q], l0 = 1. - r - s - t;
        double x[3];
        for(int k = 0; k < 3; ++k) x[k] = l0 * X[0][k] + r * X[1][k] + s * X[2][k] + t * X[3][k];
        sF[q * EPB + lane] = source_x(fc.srcKind, fc.srcParam, x[0], x[1], x[2]);
      }
    }
  }
  __syncthreads();
  if(!live) return;
  double G[3][3];
  for(int r = 0; r < 3; ++r)
    for(int k = 0; k < 3; ++k) G[r][k] = sG[(3 * r + k) * EPB + lane];
  const double J = sG[9 * EPB + lane];
  // Be_a -= k grad phi_a . grad u   (feSysElm.cpp:558-583),  Be_a -= phi_a f   (feSysElm.cpp:16-27)
  double GG[3][3];
  for(int r = 0; r < 3; ++r)
    for(int s = 0; s < 3; ++s) GG[r][s] = G[r][0] * G[s][0] + G[r][1] * G[s][1] + G[r][2] * G[s][2];
  double acc = 0.;
  for(int b = 0; b < 10; ++b) {
    double L = 0.;
    for(int r = 0; r < 3; ++r)
      for(int s = 0; s < 3; ++s) L += GG[r][s] * Tt.k(r, s, a, b);
    acc += L * sU[b * EPB + lane];
  }
  double be = fc.hasDiff ? -fc.diff * acc * J : 0.;
  if(fc.srcKind == SRC_SIN3) {
    // source integral of phi_a: sum_q w phi_a(q) f(q)
    double srcA = 0.;
    for(int q = 0; q < nq; ++q) srcA += gT->phi[q][a] * sF[q * EPB + lane] * gT->qw[q];
    be -= fc.srcCoeff * srcA * J;
  }
  const int32_t d = dm.adr[(int64_t)a * nE + p];
  if(d < nInc) atomicAdd(rhs + d, be);
}

// ---------------------------------------------------------------------------
// Jacobian, scalar P2 and Taylor-Hood, in V = double or float.
// ---------------------------------------------------------------------------
template <typename V>
__global__ void __launch_bounds__(EPB *TPB) k_matrix_tet(DeviceMesh dm, FormCoeffs fc, const RefTensorsTet *__restrict__ gT,
                                                         const double *__restrict__ u, double c0, V *__restrict__ values,
                                                         int64_t begin, int64_t end)
{
  extern __shared__ __align__(16) unsigned char smemRaw[];
  V *smem = (V *)smemRaw;
  const bool th = fc.elemType == 4;
  V *sTen = smem;
  V *sU = sTen + NTEN;       // [30][EPB]
  V *sG = sU + 30 * EPB;     // [10][EPB]
  V *sV0 = sG + 10 * EPB;    // [3][10][EPB]  V0[r][c] = sum_k G[r][k] u_(c,k)
  const int lane = threadIdx.x, a = threadIdx.y;
  const int64_t p0 = begin + (int64_t)blockIdx.x * EPB;
  const int64_t p = p0 + lane;
  const bool live = p < end;
  const int64_t nE = dm.nElm;
  const int nloc = th ? 34 : 10;
  const TetTensors<V> Tt = load_tet_tensors(sTen, gT);
  if(live) {
    sG[a * EPB + lane] = (V)dm.geo[(int64_t)a * nE + p];
    if(th && fc.hasConv)
      for(int m = 0; m < 3; ++m) sU[(3 * a + m) * EPB + lane] = (V)u[dm.adr[(int64_t)(3 * a + m) * nE + p]];
  } else {
    sG[a * EPB + lane] = 0;
    for(int m = 0; m < 3; ++m) sU[(3 * a + m) * EPB + lane] = 0;
  }
  __syncthreads();
  V G[3][3];
  for(int r = 0; r < 3; ++r)
    for(int k = 0; k < 3; ++k) G[r][k] = sG[(3 * r + k) * EPB + lane];
  const V J = sG[9 * EPB + lane];
  if(!th) {
    // A_ab += k J sum_rs (G G^T)[r][s] K[r][s][a][b]   (feSysElm.cpp:531-556)
    V GG[3][3];
    for(int r = 0; r < 3; ++r)
      for(int s = 0; s < 3; ++s) GG[r][s] = G[r][0] * G[s][0] + G[r][1] * G[s][1] + G[r][2] * G[s][2];
    const V cd = (V)fc.diff * J;
    for(int b = 0; b < 10; ++b) {
      V L = 0;
      for(int r = 0; r < 3; ++r)
        for(int s = 0; s < 3; ++s) L += GG[r][s] * Tt.k(r, s, a, b);
      const int32_t pos = live ? __ldg(dm.map + (int64_t)(a * 10 + b) * nE + p) : -1;
      if(pos >= 0) atomicAdd(values + pos, cd * L);
    }
    return;
  }
  if(fc.hasConv) {
    for(int r = 0; r < 3; ++r)
      sV0[(r * 10 + a) * EPB + lane] =
          G[r][0] * sU[(3 * a) * EPB + lane] + G[r][1] * sU[(3 * a + 1) * EPB + lane] + G[r][2] * sU[(3 * a + 2) * EPB + lane];
  }
  __syncthreads();
  // W_b = sum_c sum_r V0[r][c] T[r][a][c][b] (the u . grad phi_b term), all m
  V W[10];
  for(int b = 0; b < 10; ++b) {
    V w = 0;
    if(fc.hasConv)
      for(int c = 0; c < 10; ++c)
        for(int r = 0; r < 3; ++r) w += sV0[(r * 10 + c) * EPB + lane] * Tt.t(r, a, c, b);
    W[b] = w;
  }
  const V cc = (V)fc.conv * J, cs = -(V)fc.sigma * (V)fc.mu * J, cm = (V)fc.mass * (V)c0 * J;
  for(int m = 0; m < 3; ++m) {
    V A[30];
    for(int j = 0; j < 30; ++j) A[j] = 0;
    for(int b = 0; b < 10; ++b) {
      if(fc.hasConv) {
        // A_(a,m),(b,n) += c [delta_mn phi_a (u . grad phi_b) + phi_a phi_b d_n u_m]
        // (feVectorSysElm.cpp:1171-1240)
        V Z[3];
        for(int r = 0; r < 3; ++r) {
          V z = 0;
          for(int c = 0; c < 10; ++c) z += sU[(3 * c + m) * EPB + lane] * Tt.t(r, a, b, c);
          Z[r] = z;
        }
        for(int n = 0; n < 3; ++n) {
          V v = G[0][n] * Z[0] + G[1][n] * Z[1] + G[2][n] * Z[2];
          if(n == m) v += W[b];
          A[3 * b + n] += cc * v;
        }
      }
      if(fc.hasSigma) {
        // A_(a,m),(b,n) += -c mu [delta_mn grad phi_a . grad phi_b + d_n phi_a d_m phi_b]
        // (feVectorSysElm.cpp:1454-1492); S[k][l] = int d_k phi_a d_l phi_b / J
        V P[3][3];
        for(int r = 0; r < 3; ++r)
          for(int l = 0; l < 3; ++l) P[r][l] = Tt.k(r, 0, a, b) * G[0][l] + Tt.k(r, 1, a, b) * G[1][l] + Tt.k(r, 2, a, b) * G[2][l];
        V tr = 0;
        for(int k = 0; k < 3; ++k) tr += G[0][k] * P[0][k] + G[1][k] * P[1][k] + G[2][k] * P[2][k];
        for(int n = 0; n < 3; ++n) {
          const V snm = G[0][n] * P[0][m] + G[1][n] * P[1][m] + G[2][n] * P[2][m];
          A[3 * b + n] += cs * ((n == m ? tr : (V)0) + snm);
        }
      }
      if(fc.hasMass) A[3 * b + m] += cm * Tt.m(a, b);   // (feVectorSysElm.cpp:390-408)
    }
    if(!live) continue;
    const int row = 3 * a + m;
    for(int j = 0; j < 30; ++j) {
      const int32_t pos = __ldg(dm.map + (int64_t)(row * nloc + j) * nE + p);
      if(pos >= 0) atomicAdd(values + pos, A[j]);
    }
    // pressure columns of row (a,m) (sigma int psi_j d_m phi_a) and the
    // column (a,m) of the pressure rows (divu int psi_j d_m phi_a)
    for(int j = 0; j < 4; ++j) {
      const V bp = (G[0][m] * Tt.d(0, j, a) + G[1][m] * Tt.d(1, j, a) + G[2][m] * Tt.d(2, j, a)) * J;
      if(fc.hasSigma) {
        const int32_t pos = __ldg(dm.map + (int64_t)(row * nloc + 30 + j) * nE + p);
        if(pos >= 0) atomicAdd(values + pos, (V)fc.sigma * bp);
      }
      if(fc.hasDivu) {
        const int32_t pos = __ldg(dm.map + (int64_t)((30 + j) * nloc + row) * nE + p);
        if(pos >= 0) atomicAdd(values + pos, (V)fc.divu * bp);
      }
    }
  }
}

__global__ void k_build_map(const int32_t *__restrict__ adr, int64_t nE, int nloc, const uint8_t *__restrict__ mask,
                            const int32_t *__restrict__ ia, const int32_t *__restrict__ ja, int64_t nInc,
                            int32_t *__restrict__ map, unsigned long long *missing)
{
  const int64_t total = (int64_t)nloc * nloc * nE;
  for(int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t p = t % nE, ij = t / nE;
    const int i = (int)(ij / nloc), j = (int)(ij % nloc);
    int32_t pos = -1;
    if(mask[ij]) {
      const int32_t row = adr[(int64_t)i * nE + p], col = adr[(int64_t)j * nE + p];
      if(row < nInc && col < nInc) {
        int32_t lo = ia[row], hi = ia[row + 1] - 1;
        while(lo <= hi) {
          const int32_t mid = (lo + hi) >> 1, c = ja[mid];
          if(c == col) { pos = mid; break; }
          if(c < col) lo = mid + 1;
          else hi = mid - 1;
        }
        if(pos < 0) atomicAdd(missing, 1ull);
      }
    }
    map[t] = pos;
  }
}

// ---------------------------------------------------------------------------
// Row-owned FP32 Taylor-Hood Jacobian (RowAsmTet).
// ---------------------------------------------------------------------------
constexpr int RT_WARPS = 8;

// Per element, in FP32: G (9), J, two unused, V0[c][q] = sum_k G[q][k] u_(c,k)
// (10 x 4, the fourth unused) and g[m][n][v] = d_n u_m at vertex v (3 x 3 x 4,
// from the differences of the quadratic's coefficients 2 u_v and
// 4 u_(v,i) - u_v - u_i).  32 elements per block, read per local DOF (coalesced
// over elements), written per element (coalesced) through shared memory.
constexpr int PK_V0 = 12, PK_G = 52;
static_assert(PK_G + 36 == ROWTET_PACK, "the packed element");

// Local node of edge (i, j).
__device__ __forceinline__ int tet_edge(int i, int j)
{
  const int a = min(i, j), b = max(i, j);  // (0,2) (2,1) (1,0) (1,3) (3,0) (3,2)
  return a == 0 ? (b == 2 ? 4 : b == 1 ? 6 : 8) : a == 1 ? (b == 2 ? 5 : 7) : 9;
}

__global__ void __launch_bounds__(256) k_pack_tet(DeviceMesh dm, int hasConv, const double *__restrict__ u,
                                                  float *__restrict__ pack)
{
  __shared__ float sh[32][41];  // u at the 30 velocity DOFs (3 c + k), G, J
  __shared__ float out[32][ROWTET_PACK + 1];
  const int64_t nE = dm.nElm;
  for(int64_t p0 = (int64_t)blockIdx.x * 32; p0 < nE; p0 += (int64_t)gridDim.x * 32) {
    const int cnt = (int)(nE - p0 < 32 ? nE - p0 : 32);
    for(int idx = threadIdx.x; idx < 32 * 40; idx += blockDim.x) {
      const int i = idx >> 5, l = idx & 31;
      const int64_t p = p0 + (l < cnt ? l : 0);
      float v;
      if(i < 30) v = hasConv ? (float)u[dm.adr[(int64_t)i * nE + p]] : 0.f;
      else v = (float)dm.geo[(int64_t)(i - 30) * nE + p];
      sh[l][i] = v;
      if(i >= 30) out[l][i - 30] = v;
    }
    __syncthreads();
    // 40 values of V0 and two unused words, 12 pairs (vertex, component)
    for(int idx = threadIdx.x; idx < 32 * 54; idx += blockDim.x) {
      const int i = idx >> 5, l = idx & 31;
      const float *E = sh[l], *G = E + 30;
      if(i < 40) {
        const int c = i >> 2, q = i & 3;
        out[l][PK_V0 + i] = q < 3 ? G[3 * q] * E[3 * c] + G[3 * q + 1] * E[3 * c + 1] + G[3 * q + 2] * E[3 * c + 2] : 0.f;
      } else if(i < 42) {
        out[l][10 + i - 40] = 0.f;
      } else {
        const int v = (i - 42) & 3, m = (i - 42) >> 2;
        float h[4];
#pragma unroll
        for(int r = 0; r < 4; ++r)
          h[r] = r == v ? 2.f * E[3 * v + m] : 4.f * E[3 * tet_edge(v, r) + m] - (E[3 * v + m] + E[3 * r + m]);
#pragma unroll
        for(int n = 0; n < 3; ++n)
          out[l][PK_G + (3 * m + n) * 4 + v] = G[n] * (h[1] - h[0]) + G[3 + n] * (h[2] - h[0]) + G[6 + n] * (h[3] - h[0]);
      }
    }
    __syncthreads();
    for(int idx = threadIdx.x; idx < cnt * ROWTET_PACK; idx += blockDim.x)
      pack[p0 * ROWTET_PACK + idx] = out[idx / ROWTET_PACK][idx % ROWTET_PACK];
    __syncthreads();
  }
}

__global__ void k_rowtet_offsets(int64_t nEnt, const int32_t *__restrict__ ent, const int32_t *__restrict__ entRow,
                                 const int32_t *__restrict__ map, int64_t nE, const int32_t *__restrict__ ia,
                                 uint8_t *__restrict__ offs)
{
  const int64_t total = nEnt * ROWTET_OFFS;
  for(int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = t / ROWTET_OFFS;
    const int j = (int)(t % ROWTET_OFFS);
    uint8_t o = 255;
    if(j < 34) {
      const int32_t e = ent[k];
      const int64_t p = e >> 6;
      const int li = e & 63;
      const int32_t pos = map[(int64_t)(li * 34 + j) * nE + p];
      if(pos >= 0) o = (uint8_t)(pos - ia[entRow[k]]);
    }
    offs[t] = o;
  }
}

// One lane's share of entry k: pack words lane, 32 + lane and 64 + lane (a
// pressure row's entries: the first), offset word lane, and the entry's local
// DOF.
struct RowTetFetch {
  float pa, pb, pc;
  uint32_t po;
  int li;
};

__device__ __forceinline__ RowTetFetch rowtet_fetch(const int32_t *__restrict__ ent, const float *__restrict__ pack,
                                                    const uint8_t *__restrict__ offs, int32_t k, int lane, bool vel)
{
  RowTetFetch f{0.f, 0.f, 0.f, 0u, 0};
  const int32_t e = ent[k];
  const float *pk = pack + (int64_t)(e >> 6) * ROWTET_PACK;
  f.pa = pk[lane];
  if(vel) {
    f.pb = pk[32 + lane];
    if(lane < ROWTET_PACK - 64) f.pc = pk[64 + lane];
  }
  if(lane < ROWTET_OFFS / 4) f.po = reinterpret_cast<const uint32_t *>(offs + (int64_t)k * ROWTET_OFFS)[lane];
  f.li = e & 63;
  return f;
}

// Tensors of the row-owned kernel in shared memory: K[a][b][q s] (9 of 12) and
// S[a][b][j] for float4 reads, T, D, M as in TetTensors.
constexpr int RT_K = 0, RT_S = 1200, RT_T = 1600, RT_D = 4600, RT_M = 4720, RT_TEN = 4820;

// A persistent grid walks the row blocks; per block the CSR values of its
// units live in shared memory.  Warp w takes units uA + w, uA + w + 8, ...
// and, for each of a unit's entries in order, the element's terms:
//   velocity unit, lane (m, b) = (lane / 10, lane % 10), lane < 30: the
//   columns (b, n) of row (a, m) -- k_matrix_tet's convection, stress and
//   mass terms; lanes (m, j) = (lane / 4, lane % 4), lane < 12: the pressure
//   columns sigma J sum_r G[r][m] D[r][j][a];
//   pressure unit (row of P1 function j), lane (a, m) = (lane / 3, lane % 3),
//   lane < 30: divu J sum_r G[r][m] D[r][j][a].
// Every value gets one contribution per element, in the entries' (color)
// order: the colored scatter's sum.
// Bound: shared-memory reads.  int phi_a phi_b d_n u_m comes from the gradient
// at the vertices (four products and two float4 reads a column, where the
// tensor over three P2 functions took thirty of each) and the stress from nine
// entries of K in three reads instead of shuffles: 196,608 tetrahedra
// 1.17 -> 0.87 ms; cube 32^3 42.9 -> 41.9 ms per two steps.
__global__ void __launch_bounds__(RT_WARPS * 32) k_matrix_tet_rows(RowAsmTet ra, FormCoeffs fc,
                                                                   const RefTensorsTet *__restrict__ gT, double c0,
                                                                   float *__restrict__ values, int accumulate)
{
  extern __shared__ __align__(16) unsigned char rtsm[];
  float *sTen = reinterpret_cast<float *>(rtsm);
  float *sv = sTen + RT_TEN;
  __shared__ __align__(16) float sE[RT_WARPS][ROWTET_PACK];
  __shared__ __align__(16) uint8_t sOff[RT_WARPS][ROWTET_OFFS];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for(int i = tid; i < 1200; i += blockDim.x) {
    const int ab = i / 12, qs = i % 12;
    sTen[RT_K + i] = qs < 9 ? (float)(&gT->K[0][0][0][0])[qs * 100 + ab] : 0.f;
  }
  for(int i = tid; i < 400; i += blockDim.x) sTen[RT_S + i] = (float)(&gT->S[0][0][0])[i];
  for(int i = tid; i < 3000; i += blockDim.x) sTen[RT_T + i] = (float)(&gT->T[0][0][0][0])[i];
  for(int i = tid; i < 120; i += blockDim.x) sTen[RT_D + i] = (float)(&gT->D[0][0][0])[i];
  for(int i = tid; i < 100; i += blockDim.x) sTen[RT_M + i] = (float)(&gT->M[0][0])[i];
  const TetTensors<float> Tt{nullptr, sTen + RT_T, sTen + RT_D, sTen + RT_M};
  const float4 *sK4 = reinterpret_cast<const float4 *>(sTen + RT_K), *sS4 = reinterpret_cast<const float4 *>(sTen + RT_S);
  const float fconv = (float)fc.conv, fcs = -(float)fc.sigma * (float)fc.mu, fcm = (float)fc.mass * (float)c0;
  const float fsig = (float)fc.sigma, fdiv = (float)fc.divu;
  for(int blk = blockIdx.x; blk < ra.nBlocks; blk += gridDim.x) {
    const int32_t uA = ra.blockUnits[blk], uB = ra.blockUnits[blk + 1];
    const int32_t base = ra.ia[ra.unitRow[uA]], L = ra.ia[ra.unitRow[uB]] - base;
    __syncthreads();  // the previous block's values are written out (and the tensors loaded)
    for(int i = tid; i < L; i += blockDim.x) sv[i] = accumulate ? values[base + i] : 0.f;
    __syncthreads();
    for(int32_t un = uA + warp; un < uB; un += RT_WARPS) {
      const int32_t r = ra.unitRow[un];
      const bool vel = ra.unitKind[un] == 3;
      float *row0 = sv + (ra.ia[r] - base);
      const int32_t rl = ra.ia[r + 1] - ra.ia[r];
      const int32_t kb = ra.unitPtr[un], ke = ra.unitPtr[un + 1];
      // the next entry's packed element data and column offsets are loaded
      // into registers while the current one is computed
      RowTetFetch nx = kb < ke ? rowtet_fetch(ra.ent, ra.pack, ra.offs, kb, lane, vel) : RowTetFetch{0.f, 0.f, 0.f, 0u, 0};
      for(int32_t k = kb; k < ke; ++k) {
        const int li = nx.li;
        sE[warp][lane] = nx.pa;
        if(vel) {
          sE[warp][32 + lane] = nx.pb;
          if(lane < ROWTET_PACK - 64) sE[warp][64 + lane] = nx.pc;
        }
        if(lane < ROWTET_OFFS / 4) reinterpret_cast<uint32_t *>(sOff[warp])[lane] = nx.po;
        __syncwarp();
        if(k + 1 < ke) nx = rowtet_fetch(ra.ent, ra.pack, ra.offs, k + 1, lane, vel);
        const float *E = sE[warp];
        const float4 *E4 = reinterpret_cast<const float4 *>(E);
        const float J = E[9];
        if(vel) {
          const int a = li / 3;
          if(lane < 30) {
            const int m = lane / 10, b = lane % 10;
            // lanes b, b + 10, b + 20 hold the same column b: the term that
            // does not depend on m is split among them and exchanged by shuffles
            constexpr unsigned L30 = 0x3fffffffu;
            float A[3] = {0.f, 0.f, 0.f};
            if(fc.hasConv) {
              // W = sum_c sum_r V0[c][r] T[r][a][c][b] (lane m sums c = m, m + 3, ...)
              float Wp = 0.f;
#pragma unroll
              for(int cc = 0; cc < 4; ++cc) {
                const int c = m + 3 * cc;
                if(c < 10) {
                  const float4 v0 = E4[PK_V0 / 4 + c];
                  Wp += v0.x * Tt.t(0, a, c, b) + v0.y * Tt.t(1, a, c, b) + v0.z * Tt.t(2, a, c, b);
                }
              }
              const float W = __shfl_sync(L30, Wp, b) + __shfl_sync(L30, Wp, b + 10) + __shfl_sync(L30, Wp, b + 20);
              const float cc = fconv * J;
              const float4 s4 = sS4[a * 10 + b];
#pragma unroll
              for(int n = 0; n < 3; ++n) {
                const float4 g = E4[PK_G / 4 + 3 * m + n];
                float v = g.x * s4.x + g.y * s4.y + g.z * s4.z + g.w * s4.w;
                if(n == m) v += W;
                A[n] += cc * v;
              }
            }
            if(fc.hasSigma) {
              const float4 k0 = sK4[(a * 10 + b) * 3], k1 = sK4[(a * 10 + b) * 3 + 1], k2 = sK4[(a * 10 + b) * 3 + 2];
              const float4 e0 = E4[0], e1 = E4[1];
              const float G[3][3] = {{e0.x, e0.y, e0.z}, {e0.w, e1.x, e1.y}, {e1.z, e1.w, E[8]}};
              // column m of P = K G
              const float x0 = E[m], x1 = E[3 + m], x2 = E[6 + m];
              const float P0 = k0.x * x0 + k0.y * x1 + k0.z * x2, P1 = k0.w * x0 + k1.x * x1 + k1.y * x2,
                          P2 = k1.z * x0 + k1.w * x1 + k2.x * x2;
              // S[n][m] of grad phi_a (x) grad phi_b; the trace from the three lanes' m = n
              float sn[3];
#pragma unroll
              for(int n = 0; n < 3; ++n) sn[n] = G[0][n] * P0 + G[1][n] * P1 + G[2][n] * P2;
              const float own = m == 0 ? sn[0] : m == 1 ? sn[1] : sn[2];
              const float tr = __shfl_sync(L30, own, b) + __shfl_sync(L30, own, b + 10) + __shfl_sync(L30, own, b + 20);
              const float cs = fcs * J;
#pragma unroll
              for(int n = 0; n < 3; ++n) A[n] += cs * ((n == m ? tr : 0.f) + sn[n]);
            }
            if(fc.hasMass) {
              const float mv = fcm * J * Tt.m(a, b);
#pragma unroll
              for(int n = 0; n < 3; ++n)
                if(n == m) A[n] += mv;
            }
            float *row = row0 + m * rl;
#pragma unroll
            for(int n = 0; n < 3; ++n) {
              const uint8_t o = sOff[warp][3 * b + n];
              if(o != 255) row[o] += A[n];
            }
          }
          if(fc.hasSigma && lane < 12) {
            const int m = lane >> 2, j = lane & 3;
            const uint8_t o = sOff[warp][30 + j];
            if(o != 255) {
              const float bp = (E[m] * Tt.d(0, j, a) + E[3 + m] * Tt.d(1, j, a) + E[6 + m] * Tt.d(2, j, a)) * J;
              row0[m * rl + o] += fsig * bp;
            }
          }
        } else if(fc.hasDivu && lane < 30) {
          const int j = li - 30, a = lane / 3, m = lane % 3;
          const uint8_t o = sOff[warp][lane];
          if(o != 255) {
            const float bp = (E[m] * Tt.d(0, j, a) + E[3 + m] * Tt.d(1, j, a) + E[6 + m] * Tt.d(2, j, a)) * J;
            row0[o] += fdiv * bp;
          }
        }
        __syncwarp();
      }
    }
    __syncthreads();
    for(int i = tid; i < L; i += blockDim.x) values[base + i] = sv[i];
  }
}

size_t residual_smem(int nq) { return sizeof(double) * (NTEN + (30 + 30 + 10 + 4 + nq) * EPB); }
template <typename V>
size_t matrix_smem() { return sizeof(V) * (NTEN + (30 + 10 + 30) * EPB); }

int64_t nblk(int64_t begin, int64_t end) { return (end - begin + EPB - 1) / EPB; }

}  // namespace

void build_ref_tensors_tet(const QuadRule &q, RefTensorsTet &T)
{
  T = RefTensorsTet();
  T.nq = std::min(q.n(), TET_MAXQ);
  for(int k = 0; k < T.nq; ++k) {
    const double r = q.r[k], s = q.s[k], t = q.t[k], w = q.w[k];
    const double l[4] = {1. - r - s - t, r, s, t};
    const double dl[4][3] = {{-1, -1, -1}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}};
    double phi[10], dphi[10][3];
    for(int v = 0; v < 4; ++v) {
      phi[v] = l[v] * (2. * l[v] - 1.);
      for(int d = 0; d < 3; ++d) dphi[v][d] = (4. * l[v] - 1.) * dl[v][d];
    }
    for(int e = 0; e < 6; ++e) {
      const int va = TET_EDGES[e][0], vb = TET_EDGES[e][1];
      phi[4 + e] = 4. * l[va] * l[vb];
      for(int d = 0; d < 3; ++d) dphi[4 + e][d] = 4. * (l[vb] * dl[va][d] + l[va] * dl[vb][d]);
    }
    T.qw[k] = w; T.qr[k] = r; T.qs[k] = s; T.qt[k] = t;
    for(int a = 0; a < 10; ++a) T.phi[k][a] = phi[a];
    for(int rr = 0; rr < 3; ++rr)
      for(int ss = 0; ss < 3; ++ss)
        for(int a = 0; a < 10; ++a)
          for(int b = 0; b < 10; ++b) T.K[rr][ss][a][b] += w * dphi[a][rr] * dphi[b][ss];
    for(int rr = 0; rr < 3; ++rr)
      for(int a = 0; a < 10; ++a)
        for(int c = 0; c < 10; ++c)
          for(int b = 0; b < 10; ++b) T.T[rr][a][c][b] += w * phi[a] * phi[c] * dphi[b][rr];
    for(int rr = 0; rr < 3; ++rr)
      for(int j = 0; j < 4; ++j)
        for(int a = 0; a < 10; ++a) T.D[rr][j][a] += w * l[j] * dphi[a][rr];
    for(int a = 0; a < 10; ++a)
      for(int b = 0; b < 10; ++b) {
        T.M[a][b] += w * phi[a] * phi[b];
        for(int j = 0; j < 4; ++j) T.S[a][b][j] += w * phi[a] * phi[b] * l[j];
      }
  }
}

void launch_assemble_residual_tet(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensorsTet *dT,
                                  const double *u, int64_t nInc, double *rhs, int64_t begin, int64_t end,
                                  cudaStream_t s)
{
  if(end <= begin) return;
  const size_t sm = residual_smem(TET_MAXQ);
  static bool set = false;
  if(!set) {
    cudaFuncSetAttribute(k_residual_tet, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    set = true;
  }
  (k_residual_tet<<<(unsigned)nblk(begin, end), dim3(EPB, TPB), sm, s>>>(dm, fc, dT, u, nInc, rhs, begin, end),
   ::feng::count_launch());
}

template <typename V>
static void launch_matrix_tet(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensorsTet *dT, const double *u,
                              double c0, V *values, int64_t begin, int64_t end, cudaStream_t s)
{
  if(end <= begin) return;
  const size_t sm = matrix_smem<V>();
  static bool set = false;
  if(!set) {
    cudaFuncSetAttribute(k_matrix_tet<V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    set = true;
  }
  (k_matrix_tet<V><<<(unsigned)nblk(begin, end), dim3(EPB, TPB), sm, s>>>(dm, fc, dT, u, c0, values, begin, end),
   ::feng::count_launch());
}

void launch_assemble_matrix_tet_f64(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensorsTet *dT,
                                    const double *u, double c0, double *values, int64_t begin, int64_t end,
                                    cudaStream_t s)
{
  launch_matrix_tet<double>(dm, fc, dT, u, c0, values, begin, end, s);
}

void launch_assemble_matrix_tet_f32(const DeviceMesh &dm, const FormCoeffs &fc, const RefTensorsTet *dT,
                                    const double *u, double c0, float *values, int64_t begin, int64_t end,
                                    cudaStream_t s)
{
  launch_matrix_tet<float>(dm, fc, dT, u, c0, values, begin, end, s);
}

void launch_pack_tet_f32(const DeviceMesh &dm, const FormCoeffs &fc, const double *u, float *pack, cudaStream_t s)
{
  const int64_t blocks = std::min<int64_t>((dm.nElm + 31) / 32, 152 * 16);
  (k_pack_tet<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, s>>>(dm, fc.hasConv, u, pack), ::feng::count_launch());
}

void launch_rowtet_offsets(int64_t nEnt, const int32_t *ent, const int32_t *entRow, const int32_t *map,
                           int64_t nElm, const int32_t *ia, uint8_t *offs, cudaStream_t s)
{
  const int64_t blocks = std::min<int64_t>((nEnt * ROWTET_OFFS + 255) / 256, 152 * 32);
  (k_rowtet_offsets<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, s>>>(nEnt, ent, entRow, map, nElm, ia, offs),
   ::feng::count_launch());
}

void launch_matrix_tet_rows_f32(const RowAsmTet &ra, const FormCoeffs &fc, const RefTensorsTet *dT, double c0,
                                float *values, int accumulate, cudaStream_t s)
{
  if(ra.nBlocks <= 0) return;
  const size_t sm = sizeof(float) * RT_TEN + (size_t)ra.capBytes;
  static size_t set = 0;
  if(set != sm) {
    cudaFuncSetAttribute(k_matrix_tet_rows, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    set = sm;
  }
  int dev = 0, nsm = 152, perSM = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSM, k_matrix_tet_rows, RT_WARPS * 32, sm);
  const int grid = (int)std::min<int64_t>(ra.nBlocks, (int64_t)nsm * std::max(perSM, 1));
  (k_matrix_tet_rows<<<grid, RT_WARPS * 32, sm, s>>>(ra, fc, dT, c0, values, accumulate), ::feng::count_launch());
}

void launch_build_map(const int32_t *adr, int64_t nElm, int nloc, const uint8_t *mask, const int32_t *ia,
                      const int32_t *ja, int64_t nInc, int32_t *map, unsigned long long *missing, cudaStream_t s)
{
  const int64_t total = (int64_t)nloc * nloc * nElm;
  const int64_t blocks = std::min<int64_t>((total + 255) / 256, 152 * 32);
  (k_build_map<<<(unsigned)std::max<int64_t>(blocks, 1), 256, 0, s>>>(adr, nElm, nloc, mask, ia, ja, nInc, map, missing),
   ::feng::count_launch());
}

}  // namespace feng
