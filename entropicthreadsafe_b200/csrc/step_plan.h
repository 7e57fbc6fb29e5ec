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

// The plan with the least estimated time, about microseconds on a B200.  A block
// takes `plane` per source plane and about `extra` planes' time outside its
// target planes (two more source planes, its start); blocks run in waves.
// Measured on the 384 x 192 x 128 colour channel: 16-warp blocks in 32 / 16 / 8
// plane chunks 0.333 / 0.355 / 0.404 ms, 8-warp blocks in 64 / 32 / 16 plane
// chunks 0.331 / 0.340 / 0.352 ms: 3 planes extra, and a plane of two 8-warp
// blocks on an SM takes 0.85 of one of 16 warps, with fewer rows (6 of 8 are
// targets, against 14 of 16).  Equal shares have no last wave, but their blocks
// are at different planes and share less of what they read: 8% slower a plane
// (48 against 51 us in the best chunks on a 173 x 59 x 91 Couette cell).
// uneven: some planes or tiles take several times longer than others, so the
// last blocks to finish are those, by their length: chunks only, and short ones.
// So for the phase field, whose planes with interface nodes are about three times
// slower (96^3 with one droplet: 130 us in 24-plane chunks), interior solids, and
// slow boundary nodes at x or y faces.
// A number of waves is used best by as many chunks as fit it, so only those are
// weighed, up to 16 waves (more only add planes outside the chunks) and the next
// shorter chunk: some 35 estimates, 0.3 us (all chunk lengths of a 16 x 16 x 4096
// lattice took 28 us a call of the step on device buffers).
inline StepPlan step_plan(int nx, int ny, int nz, bool xper, bool uneven, int sms) {
    StepPlan best{BIGW, 1, nz, 0};
    double least = 1e300;
    const long long tx = (xper && nx <= 32) ? 1 : (nx + LXV - 1LL) / LXV;
    constexpr double extra = 3.0;
    constexpr int waves = 16;
    for (int w : {BIGW, SMALLW}) {
        const int th = even_rows(ny, w - 2), bps = BIGW / w;
        const long long ty = (ny + th - 1LL) / th, cols = tx * ty, slots = (long long)bps * sms;
        auto plane = [&](long long blocks) { return w == BIGW ? 2.0 : blocks <= sms ? 1.25 : 1.72; };
        auto weigh = [&](long long chunks) {
            const int zc = (int)((nz + chunks - 1) / chunks);
            const long long blocks = cols * ((nz + zc - 1LL) / zc);
            const double cost = (double)((blocks + slots - 1) / slots) * (zc + extra) * plane(blocks) + (uneven ? 3.0 * zc : 0.0);
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
        if (!uneven && parts > 0 && ty * nz < (1LL << 31)) {
            const double share = (double)(ty * nz) / parts;
            const double cost = 1.08 * (share + extra * (share / nz + 1.0)) * plane(parts * tx);
            if (cost < least) { least = cost; best = StepPlan{w, th, 0, (int)(parts * tx)}; }
        }
    }
    return best;
}

}  // namespace tslb
