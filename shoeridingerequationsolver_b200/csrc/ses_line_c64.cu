// Run-time-plan kernels, complex64.
#include "ses_line_inst.cuh"

namespace sesk {
template <>
LineXKernel<float> line_x<float>(int mode, int rmax, bool kick) {
    return rmax <= 10 ? line_x_of<float, 10>(mode, kick) : line_x_of<float, 16>(mode, kick);
}
template <>
LineSKernel<float> line_s<float>(int mode, int rmax) {
    return rmax <= 10 ? line_s_of<float, 10>(mode) : line_s_of<float, 16>(mode);
}
}  // namespace sesk
