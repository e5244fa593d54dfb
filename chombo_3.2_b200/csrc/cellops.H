// The cell arithmetic shared by the device kernels: one GSRB update, one
// operator or residual value and the operator's scalars, each in the
// reference's expression order.
#ifndef CMG_CELLOPS_H
#define CMG_CELLOPS_H

#include <cuda_runtime.h>

namespace cmg {

struct Scal {
  double dxinv, lambda, alpha, beta;
  int laplacian;
};

// One GSRB update (k_gsrb's arithmetic) from loaded values: v the six
// neighbours (+x, -x, +y, -y, +z, -z), f the face coefficients
// (b0[+x], b0[c], b1[+y], b1[c], b2[+z], b2[c]) of a VC operator.
template <class T, int VC>
__device__ __forceinline__ T gsrbValue(const Scal& sc, T pc, T rh, const T* v, T av, T lv, const T* f) {
  const T dxinv = T(sc.dxinv);
  if (VC) {
    T div = f[0] * (v[0] - pc) - f[1] * (pc - v[1]) + f[2] * (v[2] - pc) - f[3] * (pc - v[3]) + f[4] * (v[4] - pc) -
            f[5] * (pc - v[5]);
    T lofphi = T(sc.alpha) * av * pc - T(sc.beta) * div * dxinv;
    return pc - lv * (lofphi - rh);
  } else if (sc.laplacian) {
    T lphi = (v[0] + v[1] + v[2] + v[3] + v[4] + v[5]) * dxinv;
    return T(sc.lambda) * (rh - lphi);
  } else {
    T lphi = ((v[0] + v[1] + v[2] + v[3] + v[4] + v[5]) - T(2.0) * T(3) * pc) * dxinv;
    T helmop = T(sc.alpha) * pc + T(sc.beta) * lphi;
    return pc + T(sc.lambda) * (helmop - rh);
  }
}

// OPERATORLAPRES / OPERATORLAP (AMRPoissonOpF.ChF:287-377) and
// VCCOMPUTERES3D / VCCOMPUTEOP3D (VCAMRPoissonOpF.ChF:148-312) value of one
// cell from loaded values (v and f as in gsrbValue).  MODE 0: r = rhs - L(phi)
// (residual form), MODE 1: r = L(phi).
template <class T, int VC, int MODE>
__device__ __forceinline__ T opValue(const Scal& sc, T pc, T rh, const T* v, T av, const T* f) {
  const T dxinv = T(sc.dxinv);
  if (VC) {
    T div = f[0] * (v[0] - pc) - f[1] * (pc - v[1]) + f[2] * (v[2] - pc) - f[3] * (pc - v[3]) + f[4] * (v[4] - pc) -
            f[5] * (pc - v[5]);
    T lofphi = T(sc.alpha) * av * pc - T(sc.beta) * div * dxinv;
    return MODE == 0 ? rh - lofphi : lofphi;
  } else {
    T lap = ((v[0] + v[1] + v[2] + v[3] + v[4] + v[5]) - T(6) * pc) * dxinv;
    return MODE == 0 ? -(T(sc.alpha) * pc) - T(sc.beta) * lap + rh : T(sc.alpha) * pc + T(sc.beta) * lap;
  }
}

// max(a, b) that keeps a NaN from either side (fmax drops it).
__device__ __forceinline__ double nanMax(double a, double b) { return (b > a || b != b) ? b : a; }

// The scalars of a level's operator.
inline Scal scalars(double dx, double alpha, double beta, int vc) {
  Scal s;
  s.dxinv = 1.0 / (dx * dx);
  double sum_b = 0.0;
  for (int d = 0; d < 3; ++d) sum_b = sum_b + 2.0 * s.dxinv;
  s.alpha = alpha;
  s.beta = beta;
  s.laplacian = (!vc && alpha == 0.0 && beta == 1.0) ? 1 : 0;
  s.lambda = s.laplacian ? -1.0 / sum_b : -1.0 / (alpha - beta * sum_b);
  return s;
}

}  // namespace cmg

#endif
