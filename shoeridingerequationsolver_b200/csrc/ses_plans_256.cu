// Compiled plan 256 = 16 x 16 with its pipelined variants.
#include "ses_plans.cuh"

namespace sesk {
void register_plans_256(std::vector<PlanEntry<float>>& f, std::vector<PlanEntry<double>>& d) {
    f.push_back(make_plan_entry<float, 256, 16, 16, 16, 1, 32>());
    add_x_variant<float, 256, 16, 16, 16, 1, 4, 2, 1>(f.back());
    add_x_variant<float, 256, 16, 16, 16, 1, 4, 2, 3>(f.back());
    add_x_variant<float, 256, 16, 16, 16, 1, 8, 2, 2>(f.back());
    add_x_variant<float, 256, 16, 16, 16, 1, 4, 2, 4>(f.back());
    add_x_variant<float, 256, 16, 16, 16, 1, 2, 2, 6>(f.back());
    add_s_variant<float, 256, 16, 16, 16, 1, 32, 2, 1>(f.back());
    add_s_variant<float, 256, 16, 16, 16, 1, 16, 2, 2>(f.back());
    add_s_variant<float, 256, 16, 16, 16, 1, 16, 3, 2>(f.back());
    add_s_variant<float, 256, 16, 16, 16, 1, 8, 2, 4>(f.back());
    add_s4_variant<float, 256, 16, 16, 16, 64, 4, 12>(f.back());
    set_defaults(f.back(), kXStaged, 4, 4, 4, 4);
    set_few(f.back(), 4096, 3, 3);  // fused: 1024 lines 15.8 / 16.4, 8192 60.9 / 59.2; y: 13.2 / 14.0, 44.6 / 41.8
    d.push_back(make_plan_entry<double, 256, 16, 16, 16, 1, 16>());
    add_x_variant<double, 256, 16, 16, 16, 1, 2, 2, 1>(d.back());
    add_x_variant<double, 256, 16, 16, 16, 1, 4, 2, 2>(d.back());
    add_x_variant<double, 256, 16, 16, 16, 1, 1, 2, 8>(d.back());
    add_s_variant<double, 256, 16, 16, 16, 1, 16, 2, 1>(d.back());
    add_s_variant<double, 256, 16, 16, 16, 1, 8, 2, 2>(d.back());
    add_s_variant<double, 256, 16, 16, 16, 1, 4, 2, 4>(d.back());
    add_s4_variant<double, 256, 16, 16, 16, 64, 6, 12>(d.back());
    set_defaults(d.back(), kXStaged, 3, 3, 3, 3);
    set_few(d.back(), 2048, 2, 2);  // fused: 512 lines 15.6 / 16.7, 8192 89.3 / 85.7; y: 12.5 / 13.8, 66.5 / 63.4
    set_few_x(d.back(), 512, 0);    // with an absorber: 256 lines 11.1 / 12.0, 2048 19.6 / 18.7
}
}  // namespace sesk
