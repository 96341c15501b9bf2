// Taylor-Hood P2-P1 residuals on triangles and tetrahedra: one thread per
// element, element vectors in a buffer, one thread per row adding its
// elements' terms in color order.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "fe_device.h"

namespace feng {

constexpr int RES_MAXQ = 64;  // nodes of a rule

// Tables of a rule on the reference element (D = 2: 3 + 3 functions, D = 3:
// 4 + 6): nodes of the polynomial terms (phi, w phi, barycentric coordinates)
// with the P1 and P2 mass matrices that the same nodes give, and the form's
// own nodes for the sources.
struct ResidualTables {
  int nq = 0, nqs = 0;
  double phi[RES_MAXQ][10], wphi[RES_MAXQ][10], lam[RES_MAXQ][4];
  double m[4][4], M[10][10];
  double swphi[RES_MAXQ][10], slam[RES_MAXQ][4];
};
// rule: the polynomial terms' rule; own: the form's rule, for the sources
// (nqs = 0 without one).  Both on triangles (t empty) or tetrahedra.
void build_residual_tables(const QuadRule &rule, const QuadRule *own, int dim, ResidualTables &T);

class ResidualTH {
 public:
  ResidualTH() = default;
  ResidualTH(const ResidualTH &) = delete;
  ResidualTH &operator=(const ResidualTH &) = delete;
  ~ResidualTH();
  int build(const DeviceMesh &dm, int dim, int64_t nInc, const ResidualTables &T, cudaStream_t s);
  // rhs += the residual of the forms at u, udot: in FP64, or in double-float
  // from float pairs of u and udot and dm.geoPair.
  void add64(const FormCoeffs &fc, const double *u, const double *udot, double *rhs) const;
  void add_df(const FormCoeffs &fc, const float2 *up, const float2 *udp, double *rhs) const;

 private:
  template <int D, typename A, typename In>
  void run(const FormCoeffs &fc, const In *u, const In *ud, double *rhs) const;
  DeviceMesh dm_;
  int dim_ = 0, nq_ = 0, nqs_ = 0;
  int64_t nInc_ = 0;
  cudaStream_t s_ = 0;
  ResidualTables *tab_ = nullptr;
  double *be_ = nullptr;        // [nloc][nElm] element vectors
  int32_t *rowPtr_ = nullptr;   // [nInc + 1]
  int32_t *rowEnt_ = nullptr;   // local row * nElm + element, elements ascending (color order)
};

}  // namespace feng
