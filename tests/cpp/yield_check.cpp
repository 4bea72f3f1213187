// Host build of the yield policy that the engine generates for its step kernels
// (dl_yield_source), included as "yield_policy.inc": prep, f and grad of it, as the
// kernels call them.
#include <cmath>

#include "rodkin.cuh"

#define __device__
#define __forceinline__ inline

namespace dl {
template <class T>
struct DevModel {};
#include "yield_policy.inc"
}  // namespace dl

extern "C" void yc_eval(const double *args, double *f, double *grad) {
  using Y = dl::YieldJit;
  dl::DevModel<double> m;
  double inv[Y::kInv > 0 ? Y::kInv : 1], ginv[Y::kGradInv > 0 ? Y::kGradInv : 1], regs[1];
  Y::prep(args, inv);
  Y::prep_grad(args, ginv);
  *f = Y::f(m, args, inv, regs);
  Y::grad(m, args, ginv, grad, regs);
}
