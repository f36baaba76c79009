// Part 4 of the compile-time y and x passes.
#include "qpd_axisct_part.cuh"

namespace qpd {
QPD_AXIS_CT_PART(launch_axis_ct_4, QPD_AXIS_CT_4)
}  // namespace qpd
