// Instantiations of the adv operator for (Nq, cubNq) = (8, 8), (9, 9), (5, 8), (6, 9).
#include "adv_fx.cuh"

namespace nekb {
namespace adv_fx {
template int launch<8, 8>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<9, 9>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<5, 8>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<6, 9>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
}  // namespace adv_fx
}  // namespace nekb
