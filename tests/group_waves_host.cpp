// Host test shim: the grouped search's cut of groups into waves and of waves into launches
// (simple3.0_b200/csrc/group_waves.h, the same source the library compiles).
#include "group_waves.h"

extern "C" int group_waves_run(const int *geom /* P, ns, dlen, J, row tile, column tile */, int ngroups,
                               const int *groups /* r_lo, r_end, c_lo, c_hi each */, size_t z_wave, size_t z_max, size_t d_max,
                               int max_waves, int *waves /* 8 a wave */, int *set_of, size_t *sums /* z, d, y a set */)
{
    const pftcc::WaveGeom g{geom[0], geom[1], geom[2], geom[3], geom[4], geom[5]};
    std::vector<pftcc::WavePlan> plan;
    for (int q = 0; q < ngroups; ++q)
        pftcc::plan_waves(plan, g, groups[4 * q], groups[4 * q + 1], groups[4 * q + 2], groups[4 * q + 3], z_wave);
    if ((int)plan.size() > max_waves) return -1;
    int set = 0;
    for (size_t w0 = 0; w0 < plan.size(); ++set) {
        pftcc::WaveBytes sum;
        const size_t w1 = pftcc::wave_set_end(plan, w0, g, z_max, d_max, &sum);
        if (w1 <= w0) return -2;
        sums[3 * set] = sum.z; sums[3 * set + 1] = sum.d; sums[3 * set + 2] = sum.y;
        for (size_t i = w0; i < w1; ++i) {
            const pftcc::WavePlan &p = plan[i];
            const int v[8] = {p.r_lo, p.r_hi, p.a_lo, p.a_hi, p.c_lo, p.c_hi, p.t_lo, p.t_hi};
            for (int e = 0; e < 8; ++e) waves[8 * i + e] = v[e];
            set_of[i] = set;
        }
        w0 = w1;
    }
    return (int)plan.size();
}
