// step_plan.h -- how the step kernel cuts a lattice (host code, no CUDA).
#pragma once
#include <algorithm>

namespace tslb {

constexpr int LXV = 30;       // target columns of a warp: lanes 1 .. 30 (lanes 0 and 31 are sources only)
// Warps of a block, W: 16 (one block on an SM) or 8 (two, for lattices whose
// rows or planes do not fill 16).
constexpr int BIGW = 16, SMALLW = 8;

// Warps of a block, target rows of a tile, target planes of a block (0: `grid`
// blocks share the tiles' planes equally).
struct StepPlan { int warps, th, zchunk, grid; };

inline int even_rows(int ny, int most) {   // tiles of equal height, at most `most` rows (any positive number)
    most = std::min(most, ny);
    const int tiles = (int)(((long long)ny + most - 1) / most);
    return (int)(((long long)ny + tiles - 1) / tiles);
}

// What a plan's time is estimated from, about microseconds on a B200.  A source
// plane takes a block of 16 warps 2, one of 8 warps `one` or, beside a second on its
// SM, `two`.  Equal shares of the planes have no last wave, but their blocks are at
// different planes and share less of what they read: `share` as long.  Where some
// planes or tiles take several times longer than others, the last blocks to finish
// are those, by their length: `tail` a plane, and chunks only.
struct PlanCosts { double one, two, share, tail; };
// Measured on the 384 x 192 x 128 colour channel: 16-warp blocks in 32 / 16 / 8
// plane chunks 0.333 / 0.355 / 0.404 ms, 8-warp blocks in 64 / 32 / 16 plane
// chunks 0.331 / 0.340 / 0.352 ms: 3 planes a block outside its targets (two more
// source planes, its start), and a plane of two 8-warp blocks on an SM takes 0.85
// of one of 16 warps, with fewer rows (6 of 8 are targets, against 14 of 16).
// Equal shares: 48 against 51 us in the best chunks on a 173 x 59 x 91 Couette cell.
constexpr PlanCosts kEvenCosts{1.25, 1.72, 1.08, 0.0};
// 16-bit storage converts and stores more slowly, so rim rows cost more: BF16 colour
// of 64 x 64 x 256 / 96^3 / 384 x 192 x 128 nodes with the costs above 68.8 / 54.6 /
// 361 us, with these 64.7 / 50.5 / 345.
constexpr PlanCosts kEven16Costs{1.35, 1.84, 1.12, 0.0};
// Phase field: planes with interface nodes are slower.  18 lattices, FP32: 5.2% above
// the best cut on average, with a tail of 1 / 3 a plane 6.4% / 7.4% (96^3 80.3 / 80.3 /
// 82.3 us, 192 x 96 x 64 channel 89.5 / 89.5 / 97.2, 64^3 40.9 / 44.6 / 40.9).
constexpr PlanCosts kPhaseCosts{1.25, 1.72, 1.08, 1.5};
// Interior solids, and slow boundary nodes at x or y faces: their tiles are slower.
constexpr PlanCosts kUnevenCosts{1.25, 1.72, 1.08, 3.0};

// The plan with the least estimated time; blocks run in waves.
// A number of waves is used best by as many chunks as fit it, so only those are
// weighed, up to 16 waves (more only add planes outside the chunks) and the next
// shorter chunk: some 35 estimates, 0.3 us (all chunk lengths of a 16 x 16 x 4096
// lattice took 28 us a call of the step on device buffers).
inline StepPlan step_plan(int nx, int ny, int nz, bool xper, const PlanCosts& costs, int sms) {
    StepPlan best{BIGW, 1, nz, 0};
    double least = 1e300;
    const long long tx = (xper && nx <= 32) ? 1 : (nx + LXV - 1LL) / LXV;
    constexpr double extra = 3.0;
    constexpr int waves = 16;
    for (int w : {BIGW, SMALLW}) {
        const int th = even_rows(ny, w - 2), bps = BIGW / w;
        const long long ty = (ny + th - 1LL) / th, cols = tx * ty, slots = (long long)bps * sms;
        auto plane = [&](long long blocks) { return w == BIGW ? 2.0 : blocks <= sms ? costs.one : costs.two; };
        auto weigh = [&](long long chunks) {
            const int zc = (int)((nz + chunks - 1) / chunks);
            const long long blocks = cols * ((nz + zc - 1LL) / zc);
            const double cost = (double)((blocks + slots - 1) / slots) * (zc + extra) * plane(blocks) + costs.tail * zc;
            if (cost < least) { least = cost; best = StepPlan{w, th, zc, 0}; }
        };
        weigh(1);
        if (w == SMALLW && cols <= sms) weigh(std::min<long long>(sms / cols, nz));   // one block an SM
        long long most = 0;
        for (int k = 1; k <= waves && most < nz; ++k) {
            most = std::min<long long>(k * slots / cols, nz);
            if (most > 1) weigh(most);
        }
        const int shorter = most > 0 ? (int)((nz + most - 1) / most) - 1 : (nz + 1) / 2;   // planes
        if (most < nz && shorter > 0) weigh((nz + shorter - 1LL) / shorter);
        const long long parts = std::min(slots / tx, ty * nz);
        if (costs.tail == 0.0 && parts > 0 && ty * nz < (1LL << 31)) {
            const double share = (double)(ty * nz) / parts;
            const double cost = costs.share * (share + extra * (share / nz + 1.0)) * plane(parts * tx);
            if (cost < least) { least = cost; best = StepPlan{w, th, 0, (int)(parts * tx)}; }
        }
    }
    return best;
}

}  // namespace tslb
