// Compiled plans: 16, 32, 64, 128 (pipelined variants for 32, 64, 128).
#include "ses_plans.cuh"

namespace sesk {
void register_plans_small(std::vector<PlanEntry<float>>& f, std::vector<PlanEntry<double>>& d) {
    f.push_back(make_plan_entry<float, 16, 16, 16, 1, 1, 32>());
    d.push_back(make_plan_entry<double, 16, 16, 16, 1, 1, 16>());
    f.push_back(make_plan_entry<float, 32, 8, 8, 4, 1, 32>());
    add_x_variant<float, 32, 8, 8, 4, 1, 4, 2, 4>(f.back());
    add_x_variant<float, 32, 8, 8, 4, 1, 8, 2, 2>(f.back());
    add_s_variant<float, 32, 8, 8, 4, 1, 32, 2, 4>(f.back());
    add_s_variant<float, 32, 8, 8, 4, 1, 32, 3, 3>(f.back());
    set_defaults(f.back(), -1, 0, 0, 0, 0);
    set_rest(f.back(), -1, 0);  // 65536 lines, one step: TMA-fed 70.0, register path 64.5; equal below 4096
    d.push_back(make_plan_entry<double, 32, 8, 8, 4, 1, 16>());
    d.back().xdef = -1;  // staged rows 7.00 against 6.49 at 128 lines, 20.3 against 19.2 at 16384
    f.push_back(make_plan_entry<float, 64, 8, 8, 8, 1, 32>());
    add_x_variant<float, 64, 8, 8, 8, 1, 4, 2, 2>(f.back());
    add_s_variant<float, 64, 8, 8, 8, 1, 32, 2, 2>(f.back());
    add_s4_variant<float, 64, 8, 8, 8, 128, 4, 16>(f.back());
    set_defaults(f.back(), kXStaged, -1, 0, 0, 1);
    d.push_back(make_plan_entry<double, 64, 8, 8, 8, 1, 16>());
    add_x_variant<double, 64, 8, 8, 8, 1, 4, 2, 2>(d.back());
    add_s_variant<double, 64, 8, 8, 8, 1, 16, 2, 2>(d.back());
    add_s4_variant<double, 64, 8, 8, 8, 128, 6, 18>(d.back());
    set_defaults(d.back(), kXStaged, -1, 0, -1, -1);
    f.push_back(make_plan_entry<float, 128, 16, 16, 8, 1, 32>());
    add_x_variant<float, 128, 16, 16, 8, 1, 4, 2, 3>(f.back());
    add_x_variant<float, 128, 16, 16, 8, 1, 2, 2, 6>(f.back());
    add_s_variant<float, 128, 16, 16, 8, 1, 32, 2, 1>(f.back());
    add_s_variant<float, 128, 16, 16, 8, 1, 16, 2, 2>(f.back());
    add_s_variant<float, 128, 16, 16, 8, 1, 8, 2, 4>(f.back());
    add_s4_variant<float, 128, 16, 16, 8, 128, 4, 12>(f.back());
    set_defaults(f.back(), kXStaged, -1, 3, 3, 3);
    set_few(f.back(), 8192, -1, 2);  // fused: 4096 lines 24.1 / 24.9, 16384 66.1 / 64.1
    d.push_back(make_plan_entry<double, 128, 16, 16, 8, 1, 16>());
    add_s4_variant<double, 128, 16, 16, 8, 128, 6, 12>(d.back());
    set_defaults(d.back(), kXStaged, 0, 0, 0, 0);
    set_few(d.back(), 8192, -1, -1);  // fused: 4096 lines 25.5 / 26.0, 65536 570 / 564; y: 19.5 / 21.7, 386 / 373
}
}  // namespace sesk
