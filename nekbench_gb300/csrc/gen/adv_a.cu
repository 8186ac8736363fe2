// Instantiations of the adv operator for (Nq, cubNq) = (2, 2), (3, 3), (4, 4), (5, 5), (6, 6), (7, 7), (2, 3), (3, 5), (4, 6).
#include "adv_fx.cuh"

namespace nekb {
namespace adv_fx {
template int launch<2, 2>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<3, 3>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<4, 4>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<5, 5>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<6, 6>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<7, 7>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<2, 3>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<3, 5>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
template int launch<4, 6>(int64_t, const double*, const double*, const double*, const double*, int64_t,
                           const double*, double*, cudaStream_t);
}  // namespace adv_fx
}  // namespace nekb
