// What the host decides for an axial-column scan, without a GPU: reads view
// tables and volumes, writes rows and window of the line projector (rows 0: the
// slab projector) and whether the backprojector's lines form in runs.
#include <cstdio>
#include <iostream>

#include "ykb_internal.hpp"

int main()
{
    int n, nu, nv;
    ykb_volume v{};
    while (std::cin >> n >> nu >> nv >> v.nx >> v.ny >> v.nz >> v.vox_x >> v.vox_y >> v.vox_z >> v.center_x >>
           v.center_y >> v.center_z) {
        std::vector<ykb_cone_view> views(n);
        for (ykb_cone_view& w : views) {
            float* const f = reinterpret_cast<float*>(&w);
            for (size_t i = 0; i < sizeof w / sizeof(float); ++i) std::cin >> f[i];
        }
        std::vector<ykb::JosephView> joseph;
        std::string why;
        if (!ykb::build_joseph_views(views.data(), n, nu, nv, v, joseph, why)) return 1;
        const ykb::JosephFpLines l = ykb::joseph_fp_lines_shape(joseph, nv);
        std::printf("%d %d %d\n", l.rows, l.window, ykb::joseph_bp_runs(joseph, nv) ? 1 : 0);
    }
    return 0;
}
