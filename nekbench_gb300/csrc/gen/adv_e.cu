// Instantiations of the adv operator for (Nq, cubNq) = (10, 15).
#include "adv_impl.cuh"

namespace nekb {
namespace adv {
// split = false: native FP64; true: double-float on the FP32 pipes
int launch_10_15(bool split, int64_t E, const double* vgeo, const double* cubvgeo, const double* cubD,
                 const double* cubInterpT, int64_t offset, const double* U, double* NU, cudaStream_t s)
{
  return split ? launch_p<10, 15, DF>(E, vgeo, cubvgeo, cubD, cubInterpT, offset, U, NU, s)
               : launch_p<10, 15, F64>(E, vgeo, cubvgeo, cubD, cubInterpT, offset, U, NU, s);
}
}  // namespace adv
}  // namespace nekb
