// Run-time-plan kernels, complex128.
#include "ses_line_inst.cuh"

namespace sesk {
template <>
LineXKernel<double> line_x<double>(int mode, int rmax, bool kick) {
    return rmax <= 10 ? line_x_of<double, 10>(mode, kick) : line_x_of<double, 16>(mode, kick);
}
template <>
LineSKernel<double> line_s<double>(int mode, int rmax) {
    return rmax <= 10 ? line_s_of<double, 10>(mode) : line_s_of<double, 16>(mode);
}
}  // namespace sesk
