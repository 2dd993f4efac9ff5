// group_waves.h -- how the grouped search cuts its groups into waves and puts waves into launches
// (search_mdomain_groups in k_search.cu).  Host code only, so that it is tested without a GPU.
#pragma once

#include <algorithm>
#include <cstddef>
#include <vector>

namespace pftcc {

// one wave: the rows [r_lo, r_hi) against the columns [c_lo, c_hi), in stage 1 the aligned rows
// [a_lo, a_hi) and column tiles [t_lo, t_hi)
struct WavePlan { int r_lo, r_hi, a_lo, a_hi, c_lo, c_hi, t_lo, t_hi; };

// the geometry that the sizes follow from: planes of Z, shifts, stage 2's factors and Y's values per
// (reference, column), the row and column tiles of stage 1
struct WaveGeom { int P, ns, dlen, J, row_tile, col_tile; };

// bytes of a wave's packed spectrum Z (complex FP32), its factors and its Y
struct WaveBytes { size_t z, d, y; };

inline WaveBytes wave_bytes(const WaveGeom &g, const WavePlan &p)
{
    const size_t nrefs = (size_t)((p.r_hi - 1) / g.ns - p.r_lo / g.ns + 1), pairs = nrefs * (size_t)(p.c_hi - p.c_lo);
    return {(size_t)g.P * (p.a_hi - p.a_lo) * (size_t)(p.t_hi - p.t_lo) * g.col_tile * 8, pairs * g.dlen * 4, pairs * g.J * 8};
}

// the waves of one group, rows [r_lo, r_end) and columns [c_lo, c_hi): cut by rows where its Z would
// pass z_wave_max
inline void plan_waves(std::vector<WavePlan> &plan, const WaveGeom &g, int r_lo, int r_end, int c_lo, int c_hi, size_t z_wave_max)
{
    const int t_lo = c_lo / g.col_tile, t_hi = (c_hi + g.col_tile - 1) / g.col_tile;
    const size_t zrow = (size_t)(t_hi - t_lo) * g.col_tile * g.P * 8;   // Z bytes per row
    const int rows_max = (int)std::max<size_t>(g.row_tile, z_wave_max / zrow / g.row_tile * g.row_tile);
    while (r_lo < r_end) {
        const int a_lo = r_lo / g.row_tile * g.row_tile, r_hi = std::min(r_end, a_lo + rows_max);
        const int a_hi = (r_hi + g.row_tile - 1) / g.row_tile * g.row_tile;
        plan.push_back(WavePlan{r_lo, r_hi, a_lo, a_hi, c_lo, c_hi, t_lo, t_hi});
        r_lo = r_hi;
    }
}

// The end of the set of waves from w0 that share one stage-1 and one stage-2 launch: as many as keep
// within z_max bytes of Z and d_max of factors, and no two with a column in common.  Each block of stage 2
// reads, merges and writes its column's top 8 without any order between blocks, so the row waves of a
// cut group follow one another in launches of their own (the plan is in column order, a group's waves
// next to each other).  sum: the set's Z and factors, and its largest Y.
inline size_t wave_set_end(const std::vector<WavePlan> &plan, size_t w0, const WaveGeom &g, size_t z_max, size_t d_max,
                           WaveBytes *sum)
{
    size_t w1 = w0;
    *sum = WaveBytes{0, 0, 0};
    for (; w1 < plan.size(); ++w1) {
        const WaveBytes b = wave_bytes(g, plan[w1]);
        if (w1 > w0 && (sum->z + b.z > z_max || sum->d + b.d > d_max || plan[w1].c_lo < plan[w1 - 1].c_hi)) break;
        *sum = WaveBytes{sum->z + b.z, sum->d + b.d, std::max(sum->y, b.y)};
    }
    return w1;
}

}  // namespace pftcc
