// C entry of the adv benchmark's advection operator (advCubatureHex3D_v0,
// adv/kernel/VOLTA/adv.okl:27-261): argument checks and the dispatch to the
// kernel built for the (Nq, cubNq) pair; the kernels are adv_fx.cuh and
// adv_impl.cuh, their instantiations csrc/gen/adv_*.cu.
#include "internal.h"

namespace nekb {
// NEKB_FP64 and NEKB_FP64_SPLIT alike: the fixed-point operator keeps FP64's digits and is
// faster than the double-float one at nearly every size measured (0.92 to 2.7 times)
namespace adv_fx {
template <int NQ, int CQ>
int launch(int64_t E, const double* vgeo, const double* cubvgeo, const double* cubD,
           const double* cubInterpT, int64_t offset, const double* U, double* NU, cudaStream_t s);
}  // namespace adv_fx
namespace adv {
int launch_10_15(bool split, int64_t E, const double* vgeo, const double* cubvgeo, const double* cubD,
                 const double* cubInterpT, int64_t offset, const double* U, double* NU, cudaStream_t s);
}  // namespace adv

namespace {

using Launcher = int (*)(int64_t, const double*, const double*, const double*, const double*, int64_t,
                         const double*, double*, cudaStream_t);

// cubNq = Nq (Nq = 2..12) and the 3/2 rule cubNq = ceil(3 Nq / 2) (Nq = 2..9; 10 apart)
Launcher find_launcher(int Nq, int cubNq)
{
#define NEKB_ADV(nq, cq) \
  if (Nq == nq && cubNq == cq) return adv_fx::launch<nq, cq>;
  NEKB_ADV(2, 2) NEKB_ADV(3, 3) NEKB_ADV(4, 4) NEKB_ADV(5, 5) NEKB_ADV(6, 6) NEKB_ADV(7, 7)
  NEKB_ADV(8, 8) NEKB_ADV(9, 9) NEKB_ADV(10, 10) NEKB_ADV(11, 11) NEKB_ADV(12, 12)
  NEKB_ADV(2, 3) NEKB_ADV(3, 5) NEKB_ADV(4, 6) NEKB_ADV(5, 8) NEKB_ADV(6, 9) NEKB_ADV(7, 11)
  NEKB_ADV(8, 12) NEKB_ADV(9, 14)
#undef NEKB_ADV
  return nullptr;
}

}  // namespace
}  // namespace nekb

extern "C" int nekb_adv_cubature(int Nq, int cubNq, int precision, int64_t Nelements,
                                 const double* vgeo,
                                 const double* cubvgeo, const double* cubD, const double* cubInterpT,
                                 int64_t offset, const double* U, double* NU, void* stream)
{
  using namespace nekb;
  const auto fn = find_launcher(Nq, cubNq);
  const bool large = Nq == 10 && cubNq == 15;
  if (!fn && !large)
    return fail(NEKB_ERR_UNSUPPORTED,
                "adv: Nq=%d cubNq=%d not built (cubNq = Nq for Nq 2..12, cubNq = ceil(3 Nq/2) "
                "for Nq 2..10)", Nq, cubNq);
  if (precision != NEKB_FP64 && precision != NEKB_FP64_SPLIT)
    return fail(NEKB_ERR_UNSUPPORTED, "adv: precision %d (NEKB_FP64 or NEKB_FP64_SPLIT)", precision);
  const int64_t Np = (int64_t)Nq * Nq * Nq;
  if (Nelements < 0 || Nelements > INT32_MAX || offset < Nelements * Np)
    return fail(NEKB_ERR_INVALID, "adv: Nelements=%lld offset=%lld (offset >= Nelements*Np)",
                (long long)Nelements, (long long)offset);
  if (Nelements == 0) return NEKB_OK;
  if (!vgeo || !cubvgeo || !cubD || !cubInterpT || !U || !NU)
    return fail(NEKB_ERR_INVALID, "adv: NULL argument");
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (large)
    return adv::launch_10_15(precision == NEKB_FP64_SPLIT, Nelements, vgeo, cubvgeo, cubD, cubInterpT, offset, U, NU, s);
  return fn(Nelements, vgeo, cubvgeo, cubD, cubInterpT, offset, U, NU, s);
}
