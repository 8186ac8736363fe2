// Instantiations of the adv operator for (Nq, cubNq) = (11, 11), (12, 12), (9, 14).
#include "adv_fx.cuh"

namespace nekb {
namespace adv_fx {
template int launch<11, 11>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<12, 12>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<9, 14>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
}  // namespace adv_fx
}  // namespace nekb
