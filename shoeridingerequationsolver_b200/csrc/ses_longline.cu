// Long-line kernels of the power-of-two lines 8192 .. 131072 (complex128: .. 65536, the
// longest whose rows and columns fit the shared memory of 16 CTAs).  Arguments:
// <type, N1, x E, x radices, N2, y E, y radices, CTAs of the cluster>; the plans are
// those the axis passes of the factors use.
#include "ses_longline.cuh"

namespace sesk {
void register_long_lines(std::vector<LongEntry<float>>& f, std::vector<LongEntry<double>>& d) {
    f.push_back(make_long_entry<float, 128, 16, 16, 8, 1, 64, 8, 8, 8, 1, 8>());
    f.push_back(make_long_entry<float, 128, 16, 16, 8, 1, 128, 16, 16, 8, 1, 8>());
    f.push_back(make_long_entry<float, 256, 16, 16, 16, 1, 128, 16, 16, 8, 1, 16>());
    f.push_back(make_long_entry<float, 256, 16, 16, 16, 1, 128, 16, 16, 8, 1, 8>());
    f.push_back(make_long_entry<float, 256, 16, 16, 16, 1, 256, 16, 16, 16, 1, 16>());
    f.push_back(make_long_entry<float, 256, 16, 16, 16, 1, 256, 16, 16, 16, 1, 8>());
    f.push_back(make_long_entry<float, 512, 16, 8, 8, 8, 256, 16, 16, 16, 1, 16>());
    d.push_back(make_long_entry<double, 128, 16, 16, 8, 1, 64, 8, 8, 8, 1, 8>());
    d.push_back(make_long_entry<double, 128, 16, 16, 8, 1, 128, 16, 16, 8, 1, 8>());
    d.push_back(make_long_entry<double, 256, 16, 16, 16, 1, 128, 16, 16, 8, 1, 16>());
    d.push_back(make_long_entry<double, 256, 16, 16, 16, 1, 128, 16, 16, 8, 1, 8>());
    d.push_back(make_long_entry<double, 256, 16, 16, 16, 1, 256, 16, 16, 16, 1, 16>());
}
}  // namespace sesk
