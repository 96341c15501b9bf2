// Device-evaluated source functions (SourceKind in fe_device.h).
#pragma once

#include <cuda_runtime.h>

#include "fe_device.h"

namespace feng {

// Value on triangles (scalar sources: f[0]).
__device__ __forceinline__ void source_value(int kind, const double *p, double x, double y,
                                             double f[2])
{
  switch(kind) {
    case SRC_SIN_SIN:
      f[0] = p[0] * sinpi(x) * sinpi(y);
      f[1] = 0.;
      break;
    case SRC_NS_MMS_POLY: {
      // f = -( -u.grad u - grad p + lap u ) for u=(x^4 y^4, -4/5 x^3 y^5), p = x^2 y^2
      const double mdpdx0 = -2. * x * y * y, mdpdx1 = -2. * x * x * y;
      const double lap0 = 12. * (x * x * y * y * y * y + x * x * x * x * y * y);
      const double lap1 = -4. / 5. * (6. * x * y * y * y * y * y + 20. * x * x * x * y * y * y);
      const double u0 = x * x * x * x * y * y * y * y, u1 = -4. / 5. * x * x * x * y * y * y * y * y;
      const double g00 = 4. * x * x * x * y * y * y * y, g01 = -12. * x * x * y * y * y * y * y / 5.;
      const double g10 = 4. * x * x * x * x * y * y * y, g11 = -4. * x * x * x * y * y * y * y;
      const double c0 = u0 * g00 + u1 * g10, c1 = u0 * g01 + u1 * g11;
      f[0] = -(-c0 + mdpdx0 + lap0);
      f[1] = -(-c1 + mdpdx1 + lap1);
      break;
    }
    case SRC_CONST_VEC:
      f[0] = p[0];
      f[1] = p[1];
      break;
    case SRC_SIN_BODY:
      f[0] = p[0] * sinpi(x) * sinpi(y);
      f[1] = 0.;
      break;
    default:
      f[0] = f[1] = 0.;
  }
}

// x component (scalar sources: the value) on tetrahedra.
__device__ __forceinline__ double source_x(int kind, const double *p, double x, double y, double z)
{
  if(kind == SRC_SIN3 || kind == SRC_SIN3_BODY) return p[0] * sinpi(x) * sinpi(y) * sinpi(z);
  return 0.;
}

}  // namespace feng
