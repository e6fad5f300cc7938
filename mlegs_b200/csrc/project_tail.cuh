// The passes after a right-hand side's fold products (ProjectTail), one warp per axial
// mode: a launch of its own or further blocks of the solve that follows (solve.cu).  As
// separate VEL2PLN and far-field launches they were two of the nine of a right-hand
// side, each as long as a launch's latency: CALC_BOUSSI_FORCE at 64x32x32 43.8 ->
// 34.5 us, ten AB2-CN steps there 335 -> 309 us.
#pragma once

#include "mlegs_internal.h"

namespace mlegs {

__device__ __forceinline__ void project_tail_warp(const DevGrid& g, const ProjectTail& t, int k, int lane) {
    if (k >= g.NXCHOPDIM) return;
    const size_t st = g.NXCHOPDIM;
    double pln = 0.0;
    if (k == 0) {
        for (int j = lane; j < g.NR; j += 32) pln += t.Lpff[j] * t.line[(size_t)j * st].x;
        for (int o = 16; o > 0; o >>= 1) pln += __shfl_xor_sync(0xffffffffu, pln, o);
    }
    double2* a = t.psi + k;
    double sx = 0.0, sy = 0.0;
    for (int n = lane; n < g.NRCHOP; n += 32) {
        double2 v = a[(size_t)n * st];
        if (k == 0) {
            v.x += pln * t.dvec[n];
            a[(size_t)n * st] = v;
        }
        sx += g.at1[n] * v.x;
        sy += g.at1[n] * v.y;
    }
    for (int o = 16; o > 0; o >>= 1) {
        sx += __shfl_xor_sync(0xffffffffu, sx, o);
        sy += __shfl_xor_sync(0xffffffffu, sy, o);
    }
    if (lane == 0) {  // this lane wrote row 0 above, if anyone did
        const double2 v = a[0];
        a[0] = make_double2(v.x - sx / g.at1[0], v.y - sy / g.at1[0]);
        for (int j = 0; j < 3 && k == 0; ++j) *t.zero_ln[j] = 0.0;
    }
}

}  // namespace mlegs
