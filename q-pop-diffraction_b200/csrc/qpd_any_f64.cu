// float64 instantiations of the runtime-length passes.
#include "qpd_any.cuh"

namespace qpd {
QPD_ANY_INSTANTIATE(double)
}  // namespace qpd
