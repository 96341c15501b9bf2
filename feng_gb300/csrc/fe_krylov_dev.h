// Device state of a GMRES cycle, its rotations and the scale pass of an
// Arnoldi step, shared by the Krylov kernels and the preconditioner kernels
// that carry the pass.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace feng {

constexpr int MAXM = 128;      // maximum restart length

struct RedState {
  unsigned int counter;
  float finv;   // 1 / ||w|| of the last FP32 Gram-Schmidt norm pass
  int reorth;   // the last Gram-Schmidt pass asks for a second one
  unsigned int slices[MAXM / 8];  // blocks done of each column slice (k_gs64)
  double result[4];
};

// Givens rotations on Hessenberg column j (device, one thread).  H is stored
// column-major with leading dimension MAXM+1.
struct GmresHead {
  int done;       // set once the estimate reaches tol or on breakdown
  int k;          // number of basis vectors in use
  double est;     // |g[k]|: residual norm estimate
  double tol;
  double beta;    // ||r|| at the start of the cycle
};
struct GmresState : GmresHead {
  double H[MAXM * (MAXM + 1)];
  double cs[MAXM], sn[MAXM], g[MAXM + 1], y[MAXM];
  double hcur[MAXM + 1], hcur2[MAXM + 1];
};

// One warp: the column and the previous rotations are staged in shared
// memory, the rotation chain runs as a scan over the lanes, and the column is
// written back by the warp.
// Applies the previous rotations to Hessenberg column j, forms rotation j,
// updates g and the residual estimate, sets done (one warp; sh, scs, ssn:
// shared arrays of MAXM + 1, MAXM, MAXM doubles).
__device__ __forceinline__ void givens_warp(GmresState *gs, int j, int lane, double *sh, double *scs, double *ssn)
{
  double *h = gs->H + (int64_t)j * (MAXM + 1);
  for(int i = lane; i <= j + 1; i += 32) sh[i] = h[i];
  for(int i = lane; i < j; i += 32) {
    scs[i] = gs->cs[i];
    ssn[i] = gs->sn[i];
  }
  __syncwarp();
  // The chain t_0 = h_0, t_{i+1} = -s_i t_i + c_i h_{i+1}, h_i <- c_i t_i +
  // s_i h_{i+1}, h_j <- t_j is an affine recurrence: lane l composes the
  // maps t -> -s_i t + c_i h_{i+1} of its GCH consecutive rotations, a warp
  // scan composes the lanes' maps (Hillis-Steele, five shuffle rounds), and
  // each lane replays its rotations from its start value: ~25 dependent FP64
  // operations instead of two per rotation in sequence.
  {
    constexpr int GCH = (MAXM + 31) / 32;
    const int i0 = lane * GCH;
    const double h0 = sh[0];
    double cv[GCH], sv[GCH], hv[GCH];
    double A = 1., B = 0.;  // the lane's map t -> A t + B
#pragma unroll
    for(int u = 0; u < GCH; ++u) {
      const bool ok = i0 + u < j;
      cv[u] = ok ? scs[i0 + u] : 1.;
      sv[u] = ok ? ssn[i0 + u] : 0.;
      hv[u] = ok ? sh[i0 + u + 1] : 0.;
      if(ok) {
        const double al = -sv[u], be = cv[u] * hv[u];
        A = al * A;
        B = al * B + be;
      }
    }
    // inclusive scan: (A, B) <- (A, B) o (lane - off's map)
#pragma unroll
    for(int off = 1; off < 32; off <<= 1) {
      const double Ap = __shfl_up_sync(0xffffffffu, A, off), Bp = __shfl_up_sync(0xffffffffu, B, off);
      if(lane >= off) {
        B = A * Bp + B;
        A = A * Ap;
      }
    }
    // exclusive: the composition of the lanes before this one
    double Ae = __shfl_up_sync(0xffffffffu, A, 1), Be = __shfl_up_sync(0xffffffffu, B, 1);
    if(lane == 0) {
      Ae = 1.;
      Be = 0.;
    }
    __syncwarp();  // every read of sh before the writes below
    double t = Ae * h0 + Be;
#pragma unroll
    for(int u = 0; u < GCH; ++u)
      if(i0 + u < j) {
        sh[i0 + u] = cv[u] * t + sv[u] * hv[u];
        t = -sv[u] * t + cv[u] * hv[u];
        if(i0 + u == j - 1) sh[j] = t;
      }
  }
  __syncwarp();
  for(int i = lane; i < j; i += 32) h[i] = sh[i];
  if(lane != 0) return;
  const double a = sh[j], b = sh[j + 1];
  // one reciprocal root instead of hypot and two divisions (dependent FP64
  // operations take about 110 cycles each); hypot where a^2 + b^2 leaves the
  // normal range
  double r, c = 1., s = 0.;
  const double ss = a * a + b * b;
  if(ss > 1e-280 && ss < 1e280) {
    const double inv = rsqrt(ss);
    r = ss * inv;
    c = a * inv;
    s = b * inv;
  } else {
    r = hypot(a, b);
    if(r != 0) { c = a / r; s = b / r; }  // not finite: so is the estimate
  }
  gs->cs[j] = c;
  gs->sn[j] = s;
  h[j] = r;
  h[j + 1] = 0.;
  gs->g[j + 1] = -s * gs->g[j];
  gs->g[j] = c * gs->g[j];
  gs->k = j + 1;
  gs->est = fabs(gs->g[j + 1]);
  if(!(gs->est > gs->tol) || b == 0.0 || !isfinite(gs->est)) gs->done = 1;
}

// The FP32 Arnoldi basis of the mixed path is stored in row blocks of VBLK
// rows: column c of row block k at V + (k m1 + c) VBLK (m1 = restart + 1
// columns per block), so that a block of threads streaming several columns
// over the same rows reads one contiguous region.  vidx4: the float4 index
// of float4 row g (rows 4g..4g+3) of column c.
constexpr int VBLK = 1024;
__host__ __device__ __forceinline__ int64_t vidx4(int64_t g, int c, int m1)
{
  return ((g >> 8) * m1 + c) * (VBLK / 4) + (g & (VBLK / 4 - 1));
}

// The end of Arnoldi step j: basis vector j + 1 = w / ||w|| and the Givens
// rotation of column j.  ||w|| comes from the last update + norm pass.
// FP32: n counts rows of four; the vector goes to column `col` of the
// row-blocked basis blk (m1 columns) and to its contiguous copy v.  FP64: v.
template <typename V>
struct ScaleStep {
  const V *w;
  const RedState *st;
  V *v, *blk;
  int64_t n;
  int m1, col;
  const int *done;
  GmresState *gs;  // null: no rotation
  int j, blocks;   // blocks: that scale, besides the one that rotates
};
__device__ __forceinline__ float scale_of(const ScaleStep<float> &s) { return s.st->finv; }
__device__ __forceinline__ double scale_of(const ScaleStep<double> &s) { return s.st->result[1]; }

// Block vb: 0 applies the rotation (with gs), the others scale.  A block that
// starts after the rotation converged skips its share of the vector, which
// the cycle no longer reads.
template <typename V>
__device__ __forceinline__ void scale_blocks(const ScaleStep<V> &s, int vb)
{
  __shared__ double sh[MAXM + 1], scs[MAXM], ssn[MAXM];
  if(*s.done) return;
  if(s.gs && vb == 0) {
    if(threadIdx.x < 32) givens_warp(s.gs, s.j, threadIdx.x, sh, scs, ssn);
    return;
  }
  const V inv = scale_of(s);
  const int64_t i0 = (int64_t)(vb - (s.gs ? 1 : 0)) * blockDim.x + threadIdx.x, step = (int64_t)s.blocks * blockDim.x;
  if constexpr(sizeof(V) == 4) {
    const float4 *w4 = reinterpret_cast<const float4 *>(s.w);
    float4 *V4 = reinterpret_cast<float4 *>(s.blk), *c4 = reinterpret_cast<float4 *>(s.v);
    for(int64_t g = i0; g < s.n; g += step) {
      float4 t = w4[g];
      t.x *= inv;
      t.y *= inv;
      t.z *= inv;
      t.w *= inv;
      V4[vidx4(g, s.col, s.m1)] = t;
      c4[g] = t;
    }
  } else {
    for(int64_t i = i0; i < s.n; i += step) s.v[i] = s.w[i] * inv;
  }
}

}  // namespace feng
