// Part 3 of the compile-time y and x passes.
#include "qpd_axisct_part.cuh"

namespace qpd {
QPD_AXIS_CT_PART(launch_axis_ct_3, QPD_AXIS_CT_3)
}  // namespace qpd
