// Planes per z-march of a step launch (host).
#pragma once

namespace pe {

// How the time of a pair launch (two blocks per SM) depends on its blocks, in
// waves: `lone` while every SM has at most one, `one` up to a full wave,
// beyond it `whole` times the whole waves plus the rest times the fraction,
// plus `tail`; each wave takes a march's planes and `startup` planes more.
struct MarchModel {
    double startup, lone, one, whole, tail;
};
// Fitted to the profiled times of 62 grids from 20x24x28 to 160x256x256 at 6 to
// 20 march lengths each. The stress kernel's blocks drift apart (interior tiles
// are faster), so much of its last wave counts by its fraction; the velocity
// kernel's waves run nearly in step. Against whole waves with at least four
// planes no choice on those grids is slower by more than 1.3 % (stress) and 0.4
// % (velocity), and the means over the grids are 2.2 and 1.9 % above the best
// length's time, where whole waves are 7.1 and 7.8 % above it. In us: velocity
// 96x160x160 53.2 -> 47.5 (20 -> 9 planes), 20x24x28 14.7 -> 10.3 (4 -> 1);
// stress 30x200x200 54.2 -> 48.4 (15 -> 6), 87x223x223 134 -> 129 (44 -> 22).
constexpr MarchModel STRESS_PAIR_MARCH{2.0, 0.85, 1.2, 0.25, 0.4};
constexpr MarchModel VELOCITY_PAIR_MARCH{1.0, 0.9, 1.1, 0.75, 0.05};

// The split of nz into chunks that minimises the modelled time of a launch of
// `tiles` columns. Without a model (kernels that run their waves in step, one
// block per slot, and the untiled ones, which on 15 grids come within 3 % of
// their best length so) a wave counts whole and the least cost wins; with one a
// shorter march must be worth 2 %, since longer ones re-read less of the halo.
inline int pick_zchunk(int nz, long long tiles, int slots, int nsm, double startup, const MarchModel *m = nullptr)
{
    int best_zc = nz;
    double best = 1e300;
    for (int nch = 1; nch <= nz; ++nch) {
        const int zc = (nz + nch - 1) / nch;
        const long long blocks = tiles * ((nz + zc - 1) / zc);
        const double whole = (double)((blocks + slots - 1) / slots);
        double waves = whole;
        if (m) {
            if (blocks <= nsm) waves = m->lone;
            else if (blocks <= slots) waves = m->one;
            else waves = m->whole * whole + (1.0 - m->whole) * blocks / slots + m->tail;
        }
        const double cost = waves * (zc + (m ? m->startup : startup));
        if (cost < (m ? 0.98 * best : best - 1e-9)) {
            best = cost;
            best_zc = zc;
        }
    }
    return best_zc;
}

}  // namespace pe
