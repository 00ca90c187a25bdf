// Instances of the run-time-plan kernels of one precision.
#pragma once

#include "ses_line.cuh"

namespace sesk {

template <typename T, int RM>
LineXKernel<T> line_x_of(int mode, bool kick) {
    if (kick) switch (mode) {
            case XM_START: return line_x_kernel<T, XM_START, RM, true>;
            case XM_MID: return line_x_kernel<T, XM_MID, RM, true>;
            case XM_END: return line_x_kernel<T, XM_END, RM, true>;
            default: return nullptr;
        }
    switch (mode) {
        case XM_FWD: return line_x_kernel<T, XM_FWD, RM, false>;
        case XM_INV: return line_x_kernel<T, XM_INV, RM, false>;
        case XM_START: return line_x_kernel<T, XM_START, RM, false>;
        case XM_MID: return line_x_kernel<T, XM_MID, RM, false>;
        case XM_END: return line_x_kernel<T, XM_END, RM, false>;
        case XM_1D: return line_x_kernel<T, XM_1D, RM, false>;
        case XM_REDUCE: return line_x_kernel<T, XM_REDUCE, RM, false>;
        default: return nullptr;
    }
}

template <typename T, int RM>
LineSKernel<T> line_s_of(int mode) {
    switch (mode) {
        case SM_FWD: return line_s_kernel<T, SM_FWD, RM>;
        case SM_INV: return line_s_kernel<T, SM_INV, RM>;
        case SM_FUSED: return line_s_kernel<T, SM_FUSED, RM>;
        case SM_REDUCE: return line_s_kernel<T, SM_REDUCE, RM>;
        default: return nullptr;
    }
}

}  // namespace sesk
