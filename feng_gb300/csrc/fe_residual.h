// Taylor-Hood P2-P1 residuals on triangles and tetrahedra: one thread per
// element and velocity component, element vectors in a buffer, one thread per
// row adding its elements' terms in color order.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "fe_device.h"

namespace feng {

// Tables of a rule on the reference element (D = 2: 3 + 3 functions, D = 3:
// 4 + 6), in the order in which a block keeps them; l: the barycentric
// coordinates.
struct ResidualTables {
  int nq = 0;
  // sums over the nodes: w phi_a l_i l_j l_k (i <= j <= k), w l_i l_j, 4 times
  // that, w (4 l_i - 1) l_j
  std::vector<double> rule;
  std::vector<double> own;  // per node, for the sources: w phi, l
};
// rule: on triangles (t empty) or tetrahedra.
void build_residual_tables(const QuadRule &rule, int dim, ResidualTables &T);

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
  void run(const FormCoeffs &fc, const In *tab, const In *u, const In *ud, double *rhs) const;
  DeviceMesh dm_;
  int dim_ = 0, nq_ = 0;
  int64_t nInc_ = 0;
  cudaStream_t s_ = 0;
  double *tab_ = nullptr;       // rule tables
  float2 *pairs_ = nullptr;     // the same as float pairs
  double *own_ = nullptr;
  double *be_ = nullptr;        // [nloc][nElm] element vectors
  int32_t *rowPtr_ = nullptr;   // [nInc + 1]
  int32_t *rowEnt_ = nullptr;   // local row * nElm + element, elements ascending (color order)
};

}  // namespace feng
