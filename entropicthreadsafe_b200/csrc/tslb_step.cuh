// tslb_step.cuh -- the fused pull step kernel.
//
// A block owns a tile of (x, y) columns and a chunk of `zchunk` target
// planes, and marches through the source planes s = z0-1 .. z1 of the chunk.
// A warp is one row of 32 source nodes, one per thread.  The outermost lanes
// and rows of a tile are sources only: 30 x (W - 2) targets per block of W
// warps.
//
// The populations that land on a node are never formed one by one.  A
// post-collision population is f_c = w_c (1 + P'(c)) with P' a polynomial of
// 17 coefficients in cx, cy, cz, and w_c = w(cx) w(cy) w(cz) is a product, so
// the moments of the 27 pulled populations,
//   M_abc(x) = sum_c cx^a cy^b cz^c w_c P'_{x-c}(c),
// factor into three one-dimensional sums, one axis after the other:
//   x  every monomial cy^j cz^k of P' is evaluated at cx = -1, 0, 1 and pulled
//      from the two neighbouring lanes (shuffles), summed with cx^a;
//   y  the results, polynomials in cy, are evaluated at cy = -1, 0, 1 and
//      exchanged with the neighbouring warps through shared memory;
//   z  the results, polynomials in cz, are added to the targets s-1, s, s+1,
//      whose partial sums stay in registers.
// Three sums of three terms instead of one of 27: about 265 FP32 operations per
// node with the coefficients, against about 560 for a pull of the 27
// populations from a tile of coefficients.
//
// Per source plane s:
//   0. phi of a plane ahead is read for the block's ring of phi planes;
//   1. every thread forms the coefficients of its node, the x sums and the y
//      values it sends;
//   2. one CTA barrier publishes the y values and the phi plane;
//   3. the moments of plane s+1 are read ahead, the y and z sums completed,
//      populations whose source lies behind a non-periodic face or in an
//      interior solid added, and target plane s-1 written out.
// Reading moments and writing moments is all the HBM traffic there is:
// the populations f, g of the reference (recursive_2c_TSLB3D.f90:54) never
// exist in memory.
//
// What bounds it: the latency of the chain through a plane, not HBM.  On the
// 384 x 192 x 128 colour channel (FP32, 8-warp blocks) a step takes 0.326 ms on a
// B200, where the kernel that pulled 27 populations took 0.45 ms (1109 thread
// instructions a node, issue active 62%) and 88 B a node at the measured copy rate
// take 0.129 ms.  It executes 794 thread instructions a node, rims included
// (30 of 32 lanes and 6 of 8 rows are targets), issue is active 62% of the cycles;
// the stalls are spread over shared-memory and shuffle latency, fixed instruction
// latency and the plane barrier.  So registers buy more than instructions: 16
// warps of 128 registers an SM, without a spill in every kernel of a lattice whose
// boundary nodes have closed sums (a spilled word comes back from L2, as shared
// memory leaves little L1: 24 bytes of spills in the plane loop cost 12%; the
// kernels with the other boundary paths, GEN > 0, have up to 90 bytes in some
// storage forms); two rows a thread on paired FP32 instructions needs 5/7 of the
// instructions a row but 255 registers, and 8 warps an SM were slower (0.51 ms),
// 12 with spills slower still (0.66 ms).
#pragma once

#include "step_plan.h"
#include "tslb_device.cuh"

namespace tslb {

// Slot of the monomial cx^i cy^j cz^k of P'
__host__ __device__ constexpr int kslot(int i, int j, int k) {
    return i + j + k == 0 ? K_0
         : i + j + k == 1 ? (i ? K_X : j ? K_Y : K_Z)
         : i + j + k == 2 ? (i == 2 ? K_XX : j == 2 ? K_YY : k == 2 ? K_ZZ : !k ? K_XY : !j ? K_XZ : K_YZ)
         : i == 1 && j == 1 ? K_XYZ : i == 2 ? (j ? K_XXY : K_XXZ) : j == 2 ? (i ? K_XYY : K_YYZ) : (i ? K_XZZ : K_YZZ);
}
// the same with exponents along a face's normal axis AX and the two axes after it (cyclic)
template <int AX>
__host__ __device__ constexpr int kslot_ax(int n, int p, int q) {
    return AX == 0 ? kslot(n, p, q) : AX == 1 ? kslot(q, n, p) : kslot(p, q, n);
}
__host__ __device__ constexpr int aslot(int p, int q) {   // second-order accumulator of axes p, q
    return p == q ? (p == 0 ? A_XX : p == 1 ? A_YY : A_ZZ) : p + q == 1 ? A_XY : p + q == 2 ? A_XZ : A_YZ;
}
// Moments of the nine populations w_c P(r c) with c = s along the normal axis
// AX (s, r = +-1): P is a polynomial and the weights are products, so the sums
// over the two other axes are closed (sum w = 1, sum w c^2 = sum w c^4 = 1/3).
template <int AX, class Acc>
__device__ __forceinline__ void face_sum(const float* K, float s, float r, const Acc& acc) {
    constexpr int P = (AX + 1) % 3, Q = (AX + 2) % 3;
    constexpr float t = 1.f / 3.f;
    auto k = [&](int n, int p, int q) { return K[kslot_ax<AX>(n, p, q)]; };
    const float rs = r * s;
    const float q00 = k(0, 0, 0) + k(2, 0, 0) + rs * k(1, 0, 0);
    const float q10 = r * (k(0, 1, 0) + k(2, 1, 0)) + s * k(1, 1, 0), q01 = r * (k(0, 0, 1) + k(2, 0, 1)) + s * k(1, 0, 1);
    const float q20 = k(0, 2, 0) + rs * k(1, 2, 0), q02 = k(0, 0, 2) + rs * k(1, 0, 2);
    const float q11 = k(0, 1, 1) + rs * k(1, 1, 1), q21 = r * k(0, 2, 1), q12 = r * k(0, 1, 2);
    constexpr float w = 1.f / 6.f;
    const float s00 = w * (q00 + t * (q20 + q02)), s10 = w * t * (q10 + t * q12), s01 = w * t * (q01 + t * q21);
    acc[A_RHO] += s00;
    acc[A_JX + AX] += s * s00;
    acc[A_JX + P] += s10;
    acc[A_JX + Q] += s01;
    acc[aslot(AX, AX)] += s00;
    acc[aslot(P, P)] += w * t * (q00 + q20 + t * q02);
    acc[aslot(Q, Q)] += w * t * (q00 + q02 + t * q20);
    acc[aslot(AX, P)] += s * s10;
    acc[aslot(AX, Q)] += s * s01;
    acc[aslot(P, Q)] += (w / 9.f) * q11;
}

// The same of the three populations with c = s along axis AX and c = t along
// axis BX, taken away (they belong to two faces).
template <int AX, int BX, class Acc>
__device__ __forceinline__ void edge_sub(const float* K, float s, float t, float r, const Acc& acc) {
    constexpr int CX = 3 - AX - BX;
    constexpr float w = -1.f / 36.f, th = 1.f / 3.f;
    auto k = [&](int i, int j, int n) {
        return K[kslot(AX == 0 ? i : BX == 0 ? j : n, AX == 1 ? i : BX == 1 ? j : n, AX == 2 ? i : BX == 2 ? j : n)];
    };
    const float rs = r * s, rt = r * t;
    const float q0 = k(0, 0, 0) + k(2, 0, 0) + k(0, 2, 0) + rs * (k(1, 0, 0) + k(1, 2, 0)) + rt * (k(0, 1, 0) + k(2, 1, 0)) + rs * rt * k(1, 1, 0);
    const float q1 = r * (k(0, 0, 1) + k(2, 0, 1) + k(0, 2, 1) + rs * k(1, 0, 1) + rt * k(0, 1, 1) + rs * rt * k(1, 1, 1));
    const float q2 = k(0, 0, 2) + rs * k(1, 0, 2) + rt * k(0, 1, 2);
    const float e0 = w * (q0 + th * q2), e1 = w * th * q1;
    acc[A_RHO] += e0;
    acc[A_JX + AX] += s * e0;
    acc[A_JX + BX] += t * e0;
    acc[A_JX + CX] += e1;
    acc[aslot(AX, AX)] += e0;
    acc[aslot(BX, BX)] += e0;
    acc[aslot(CX, CX)] += w * th * (q0 + q2);
    acc[aslot(AX, BX)] += s * t * e0;
    acc[aslot(AX, CX)] += s * e1;
    acc[aslot(BX, CX)] += t * e1;
}

// Half-way bounce-back f_c(x) = f^post_{-c}(x) at a node with several
// bounce-back faces (bits mask): the faces' populations, less those of their
// edges, counted twice, and with three faces the corner's again.
template <int MODE, class Acc>
__device__ __forceinline__ void bounce_target(const float* K, unsigned mask, const Acc& acc) {
    const float sx = mask & 1u ? 1.f : -1.f, sy = mask & 4u ? 1.f : -1.f, sz = mask & 16u ? 1.f : -1.f;
    const bool fx = mask & 3u, fy = mask & 12u, fz = mask & 48u;
    const float bx = sx * K[K_C1], by = sy * K[K_C2], bz = sz * K[K_C3];
    if (fx) face_sum<0>(K, sx, -1.f, acc);
    if (fy) face_sum<1>(K, sy, -1.f, acc);
    if (fz) face_sum<2>(K, sz, -1.f, acc);
    if (fx && fy) edge_sub<0, 1>(K, sx, sy, -1.f, acc);
    if (fx && fz) edge_sub<0, 2>(K, sx, sz, -1.f, acc);
    if (fy && fz) edge_sub<1, 2>(K, sy, sz, -1.f, acc);
    if (fx && fy && fz)
        acc_dir_rt(acc, (int)sx, (int)sy, (int)sz, (1.f / 216.f) * eval_P(K, 1, -(int)sx, -(int)sy, -(int)sz));
    if (MODE == TSLB_MODE_COLOUR) {
        // the reflected populations carry the target's own colour: only the recolouring terms
        constexpr float r2 = 0.70710678118654752f, r3 = 0.57735026918962576f;
        constexpr float wf = (16.f + 16.f * r2 + 4.f * r3) / 216.f, we = (4.f * r2 + 2.f * r3) / 216.f;
        float v = (fx ? wf * bx : 0.f) + (fy ? wf * by : 0.f) + (fz ? wf * bz : 0.f);
        if (fx && fy) v -= we * (bx + by);
        if (fx && fz) v -= we * (bx + bz);
        if (fy && fz) v -= we * (by + bz);
        if (fx && fy && fz) v += (r3 / 216.f) * (bx + by + bz);
        // sources behind an x or y face were visited as nodes of phi 0
        const float u = (fx && fy ? 11.f / 36.f : fx || fy ? 1.f / 6.f : 0.f) * (fz ? 5.f / 6.f : 1.f);
        acc[A_COL] += u * K[K_C0] - v;
    }
    // phase field: the axis directions
    if (MODE == TSLB_MODE_PHASEFIELD) {
        if (fx) acc[A_COL] += K[K_C0] - bx;
        if (fy) acc[A_COL] += K[K_C0] - by;
        if (fz) acc[A_COL] += K[K_C0] - bz;
    }
}

// Populations entering a node from behind one velocity or pressure face f: all
// nine at once.  K: the node's coefficients, m its
// moments.
template <int MODE, class Acc>
__device__ __forceinline__ void face_target(const StepArgs& a, const float* K, const float* m, float dt, int f, const Acc& acc) {
    const FaceBC& fb = a.face[f];
    const int ax = f >> 1;
    const float s = f & 1 ? -1.f : 1.f, pht = K[K_C0];
    // colour mode: a source behind an x or y face was visited as a node of phi 0
    if (MODE == TSLB_MODE_COLOUR && ax < 2) acc[A_COL] += (1.f / 6.f) * pht;
    // f^eq(rho, Ub) + (1 - omega) w a^neq(Pi, u): density 1 and the node's velocity
    // and phi at a pressure outlet
    const bool pressure = fb.kind == TSLB_BC_PRESSURE;
    const float phib = pressure || fb.phi < -2.f ? m[F_PHI] : fb.phi;
    float omega = a.omega_pf;
    if (MODE == TSLB_MODE_COLOUR) {
        const float ca = 0.5f * (1.f + m[F_PHI]), cb = 0.5f * (1.f - m[F_PHI]);
        const float nu = 1.f / (ca * a.inv_nu_a + cb * a.inv_nu_b);
        omega = 2.f / (6.f * nu + 1.f + 2.f * dt);
    }
    const float U = pressure ? m[F_U] : fb.u[0], V = pressure ? m[F_V] : fb.u[1], W = pressure ? m[F_W] : fb.u[2];
    float Kb[K_XYZ + 1];
    coefs_moments(pressure ? 0.f : m[F_D], m, U, V, W, 1.f - omega, Kb);
    const float r0 = acc[A_RHO];
    if (ax == 0) face_sum<0>(Kb, s, 1.f, acc);
    else if (ax == 1) face_sum<1>(Kb, s, 1.f, acc);
    else face_sum<2>(Kb, s, 1.f, acc);
    if (MODE == TSLB_MODE_COLOUR) {
        const float dphi = phib - pht;
        acc[A_COL] += dphi * (1.f / 6.f + (acc[A_RHO] - r0));
    } else if (MODE == TSLB_MODE_PHASEFIELD) {
        // g entering from the face (:984-986, :1044-1045)
        acc[A_COL] += 0.125f * phib * (1.f + 3.f * s * fb.u[ax]);
    }
}

// accumulators in shared memory, S apart (registers are short where they are used)
template <int S>
struct Strided {
    float* p;
    __device__ __forceinline__ float& operator[](int i) const { return p[i * S]; }
};

// The populations of one node from behind non-periodic faces or from interior
// solids, the general path: edges of faces of different kinds, inlets, outlets,
// and face nodes beside interior solids.  Single walls, bounce-back edges and
// nodes beside solids only have closed or shorter sums of their own.
// A node's 26 directions are a chain of about 26,000 cycles when one thread takes
// them in turn, and its block waits at the plane barrier for it.  So the nodes are
// listed, and the block's warps share them, half a warp a node and a lane a
// direction (9 at a face, 15 at an edge, 19 at a corner): 160 x 128 x 96
// colour steps with outlets normal to x / edges of bounce-back and moving walls took
// 941 / 821 us in turn and take 191 / 177 us.

// The directions, as bits of a 3 x 3 x 3 index, whose source lies behind one of the
// faces of mask.
__device__ __forceinline__ unsigned directions_behind(unsigned mask) {
    constexpr unsigned xm = 0x1249249u, ym = 0x1c0e07u, zm = 0x1ffu;   // c = -1 along x, y, z
    return (mask & 1u ? xm << 2 : 0u) | (mask & 2u ? xm : 0u) | (mask & 4u ? ym << 6 : 0u) | (mask & 8u ? ym : 0u) |
           (mask & 16u ? zm << 18 : 0u) | (mask & 32u ? zm : 0u);
}
// position of set bit k (from 0) of b
__device__ __forceinline__ int nth_bit(unsigned b, int k) {
    int pos = 0;
#pragma unroll
    for (int w = 16; w > 0; w >>= 1) {
        const int c = __popc(b >> pos & ((1u << w) - 1u));
        if (k >= c) { k -= c; pos += w; }
    }
    return pos;
}
// Direction q of them (a 3 x 3 x 3 index): the population's value f and what it
// adds to the colour sum.  Kp, stride: the node's coefficients; mom(f): its moments;
// dt: its correction of the relaxation time.
struct Incoming {
    float f, col;
};
template <int MODE, class T, bool SOLID, class Mom>
__device__ __forceinline__ Incoming direction_from_behind(const StepArgs& a, const float* Kp, int stride, unsigned mask, int x,
                                                          int y, int z, int q, const Mom& mom, float dt) {
    Incoming r{0.f, 0.f};
    // colour mode accumulates colour increments over the target's own phi
    const float pht = Kp[K_C0 * stride];
    const int dx = (q % 3) - 1, dy = ((q / 3) % 3) - 1, dz = (q / 9) - 1;
    const int c[3] = {dx, dy, dz};
    // face through which the source x - c lies: axis a, side (c>0 -> minus face)
    int vface = -1;
    bool solid = false;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        if (c[ax] == 0) continue;
        const int f = 2 * ax + (c[ax] > 0 ? 0 : 1);
        if (mask & (1u << f)) {
            solid = true;
            const int k = a.face[f].kind;
            // a later velocity face wins, as the oracle's face loop overwrites in face order
            if (k == TSLB_BC_VELOCITY || k == TSLB_BC_INLET || k == TSLB_BC_OUTLET || k == TSLB_BC_PRESSURE) vface = f;
        }
    }
    // an interior solid source node (the lattice's solid mask), periodic axes wrapped
    bool msolid = false;
    if (SOLID && !solid) {
        const int sx = x - dx, sy = y - dy, sz = z - dz;
        msolid = bit_at(a.solid, nidx(a, sx < 0 ? sx + a.nx : (sx >= a.nx ? sx - a.nx : sx),
                                      sy < 0 ? sy + a.ny : (sy >= a.ny ? sy - a.ny : sy),
                                      sz < 0 ? sz + a.nz : (sz >= a.nz ? sz - a.nz : sz)));
    }
    if (!solid && !msolid) return r;
    const int c2 = dx * dx + dy * dy + dz * dz;
    const float wq = wclass(c2);
    // The pull skips whole solid z planes, but a source behind an x or y
    // face, or an interior solid node, is a zero-coefficient node it visited.
    const bool xy_solid = (dx && (mask & (1u << (dx > 0 ? 0 : 1)))) || (dy && (mask & (1u << (dy > 0 ? 2 : 3))));
    const bool zplane_solid = a.face[4].kind != TSLB_BC_PERIODIC && (z - dz < 0 || z - dz >= a.nz);
    const bool visited = (xy_solid && !zplane_solid) || msolid;
    // colour mode: the visited zero node added w (0 - phi_t): undo it
    if (MODE == TSLB_MODE_COLOUR && visited) r.col += wq * pht;
    if (vface < 0) {
        // half-way bounce-back: f_c(x) = f^post_{-c}(x)
        r.f = wq * eval_P(Kp, stride, -dx, -dy, -dz);
        if (MODE == TSLB_MODE_COLOUR) {
            // the reflected population carries the target's own colour: only the recolouring term
            const float bc = -(dx * Kp[K_C1 * stride] + dy * Kp[K_C2 * stride] + dz * Kp[K_C3 * stride]);
            r.col += wq * invlen(c2) * bc;
        } else if (MODE == TSLB_MODE_PHASEFIELD && c2 == 1) {
            const float ge = -(dx * Kp[K_C1 * stride] + dy * Kp[K_C2 * stride] + dz * Kp[K_C3 * stride]);
            r.col += pht + ge;
        }
    } else {
        float m[NF];
#pragma unroll
        for (int f = 0; f < NF; ++f) m[f] = mom(f);
        const FaceBC& fb = a.face[vface];
        const int ax = vface >> 1;
        float Ub[3] = {fb.u[0], fb.u[1], fb.u[2]};
        float phib = fb.phi < -2.f ? m[F_PHI] : fb.phi;
        // in-plane position of the ghost node the population leaves, x - c
        // (periodic axes wrap, a non-periodic axis clamps), in the target's layer
        int g[3] = {x, y, z};
        {
            const int cc[3] = {dx, dy, dz};
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                if (b == ax) continue;
                const int n = dimn(a, b), v = g[b] - cc[b];
                g[b] = (v >= 0 && v < n) ? v : (a.face[2 * b].kind == TSLB_BC_PERIODIC ? wrapi(v, n) : (v < 0 ? 0 : n - 1));
            }
        }
        if (fb.kind == TSLB_BC_INLET) {
            // the inlet plane at the ghost node (boundary_cds_3D_module.f90:934-986:
            // u, v, w of node (i, j, 1) feed the populations it sends)
            const long long pa = plane_area(a, vface), pi = plane_index(a, vface, g[0], g[1], g[2]);
            Ub[0] = fb.plane[pi];
            Ub[1] = fb.plane[pa + pi];
            Ub[2] = fb.plane[2 * pa + pi];
            phib = fb.plane[3 * pa + pi];
        } else if (fb.kind == TSLB_BC_OUTLET || fb.kind == TSLB_BC_PRESSURE) {
            phib = m[F_PHI];
        }
        float Uf[3] = {Ub[0], Ub[1], Ub[2]};  // velocity of the f equilibrium
        if (fb.kind == TSLB_BC_OUTLET) {
            // outlet: the normal velocity of the fluid node next to the ghost
            // node (zero gradient, :992 w(i,j,nz) = w(i,j,nz-1))
            Uf[ax] = ld_field<T>(a, F_U + ax, nidx(a, g[0], g[1], g[2]));
        } else if (fb.kind == TSLB_BC_PRESSURE) {
            // pressure outlet: the fluid node's velocity at density 1
            Uf[0] = m[F_U]; Uf[1] = m[F_V]; Uf[2] = m[F_W];
        }
        const float d = fb.kind == TSLB_BC_PRESSURE ? 0.f : m[F_D], rho = 1.f + d;
        float omega;
        if (MODE == TSLB_MODE_COLOUR) {
            const float ca = 0.5f * (1.f + m[F_PHI]), cb = 0.5f * (1.f - m[F_PHI]);
            const float nu = 1.f / (ca * a.inv_nu_a + cb * a.inv_nu_b);
            omega = 2.f / (6.f * nu + 1.f + 2.f * dt);
        } else {
            omega = a.omega_pf;
        }
        // f^eq(rho, Ub)/w - 1 (boundary_cds_3D_module.f90:461-507)
        const float cu = dx * Uf[0] + dy * Uf[1] + dz * Uf[2];
        const float uu = Uf[0] * Uf[0] + Uf[1] * Uf[1] + Uf[2] * Uf[2];
        const float t3 = 1.f / 3.f;
        const float hxxy = (dx * dx - t3) * dy, hxxz = (dx * dx - t3) * dz, hxyy = (dy * dy - t3) * dx;
        const float hyyz = (dy * dy - t3) * dz, hxzz = (dz * dz - t3) * dx, hyzz = (dz * dz - t3) * dy;
        const float hxyz = (float)(dx * dy * dz);
        const float U = Uf[0], V = Uf[1], W = Uf[2];
        const float h3e = 13.5f * (hxxy * U * U * V + hxxz * U * U * W + hxyy * U * V * V + hyyz * V * V * W +
                                   hxzz * U * W * W + hyzz * V * W * W) + 27.f * hxyz * U * V * W;
        const float feqm1 = d + rho * (3.f * cu + 4.5f * cu * cu - 1.5f * uu + h3e);
        // a^neq(Pi, u) of the fluid node
        const float u = m[F_U], v = m[F_V], w = m[F_W];
        const float pxx = m[F_XX], pxy = m[F_XY], pxz = m[F_XZ], pyy = m[F_YY], pyz = m[F_YZ], pzz = m[F_ZZ];
        const float h2 = (dx * dx - t3) * pxx + (dy * dy - t3) * pyy + (dz * dz - t3) * pzz +
                         2.f * (dx * dy * pxy + dx * dz * pxz + dy * dz * pyz);
        const float an = 4.5f * h2 +
                         13.5f * (hxxy * (2.f * u * pxy + v * pxx) + hxxz * (2.f * u * pxz + w * pxx) +
                                  hxyy * (u * pyy + 2.f * v * pxy) + hyyz * (2.f * v * pyz + w * pyy) +
                                  hxzz * (u * pzz + 2.f * w * pxz) + hyzz * (v * pzz + 2.f * w * pyz)) +
                         27.f * hxyz * (u * pyz + v * pxz + w * pxy);
        const float P = feqm1 + (1.f - omega) * an;
        r.f = wq * P;
        if (MODE == TSLB_MODE_COLOUR) {
            const float dphi = phib - pht;
            r.col += wq * fmaf(dphi, P, dphi);
        } else if (MODE == TSLB_MODE_PHASEFIELD && c2 == 1) {
            // g entering from the face (:984-986, :1044-1045)
            const float eu = dx * Ub[0] + dy * Ub[1] + dz * Ub[2];
            r.col += 0.125f * phib * (1.f + 3.f * eu);
        }
    }
    return r;
}

// Half-way bounce-back off interior solid nodes, and off the faces of mask, all of
// them bounce-back: first which of the 26 sources are solid (loads that wait on
// nothing), then their reflected populations, added to acc.  As part of the general
// path, direction by direction, a step of a 160 x 128 x 96 colour lattice with one
// sphere / a packing of 300 took 373 / 1083 us and takes 179 / 466 us.
template <int MODE, class Acc>
__device__ __forceinline__ void bounce_solids(const StepArgs& a, const float* K, unsigned mask, int x, int y, int z, const Acc& acc) {
    const int xm = x > 0 ? x - 1 : a.nx - 1, xp = x < a.nx - 1 ? x + 1 : 0;
    unsigned from = 0;   // bit q: the source x - c of direction q is solid
#pragma unroll 3
    for (int r = 0; r < 9; ++r) {
        int sy = y - (r % 3 - 1), sz = z - (r / 3 - 1);
        sy = sy < 0 ? sy + a.ny : sy >= a.ny ? sy - a.ny : sy;
        sz = sz < 0 ? sz + a.nz : sz >= a.nz ? sz - a.nz : sz;
        const unsigned row = (unsigned)sz * a.plane + (unsigned)sy * a.nx;
        const unsigned b = (bit_at(a.solid, row + xp) ? 1u : 0u) | (bit_at(a.solid, row + x) ? 2u : 0u) |
                           (bit_at(a.solid, row + xm) ? 4u : 0u);
        from |= b << 3 * r;
    }
    const unsigned behind = directions_behind(mask), zface = directions_behind(mask & 48u);
    from |= behind;
    float r[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) r[i] = 0.f;
#pragma unroll 1
    for (int q = 0; q < 27; ++q) {
        if (!(from >> q & 1u)) continue;
        const int dx = q % 3 - 1, dy = q / 3 % 3 - 1, dz = q / 9 - 1, c2 = dx * dx + dy * dy + dz * dz;
        const float wq = wclass(c2);
        acc_dir_rt(r, dx, dy, dz, wq * eval_P(K, 1, -dx, -dy, -dz));
        const float b = -(dx * K[K_C1] + dy * K[K_C2] + dz * K[K_C3]);
        // (colour: the reflected population carries the target's own colour; the pull
        // visited a solid source as a node of phi 0, but no plane behind a z face)
        if (MODE == TSLB_MODE_COLOUR) r[A_COL] += wq * ((zface >> q & 1u ? 0.f : K[K_C0]) + invlen(c2) * b);
        if (MODE == TSLB_MODE_PHASEFIELD && c2 == 1) r[A_COL] += K[K_C0] + b;
    }
#pragma unroll
    for (int i = 0; i < NACC; ++i) acc[i] = r[i];
}

// ---- tile geometry (LXV, BIGW, SMALLW: step_plan.h) ----
constexpr int NMOM = NF - 1;  // moments read per node (phi comes from the phi ring)

// Phi rows and columns held beyond the block's source nodes: colour mode
// reads the gradient at the source nodes, 1; the phase field also the normals
// of their neighbours for the curvature, 2.  The phi planes held ahead of the
// source plane are one more.
__host__ __device__ constexpr int phi_rim(int mode) { return mode == TSLB_MODE_PHASEFIELD ? 2 : 1; }
// Ring slots: plane z sits in slot z & (RING - 1).  While the slowest warp
// still reads planes s-1 .. s+1 (colour; the phase field from s-2 on) the
// fastest may already write plane s+3 (phase field s+4).
constexpr int RING = 8;
// A row of 32 source nodes is read as the 16-byte chunks that cover it: ROWE
// elements from its start rounded down to a chunk.
constexpr int ROWE = 40, MROW = ROWE * 4;   // elements, and bytes kept for a row of moments
// Shared memory of a block: y values exchanged between warps, quads
// [parity][direction][k][row][lane]; moments read ahead, [parity][field][row]
// of MROW bytes, and the tau correction, [parity][thread]; the phi ring's rim
// nodes, [2][thread] (place, offset); the moments of populations from behind
// faces, [NACC][thread]; sources of the chunk reads, [2][thread]; the phi ring;
// phase field: the curvature work list (the candidate nodes' tile indices for
// two planes, their curvatures, two counts); the count of listed boundary nodes.
// What is used once a plane is kept here rather than in registers.
template <int MODE, int W>
struct Smem {
    static constexpr int NT = 32 * W;
    // (a plane of the ring is 12 banks past the one before: the curvature's lanes
    // read three planes at once)
    static constexpr int RAREA = (ROWE * (W + 2 * phi_rim(MODE)) + 31) / 32 * 32 + 12;
    static_assert(RAREA % 4 == 0, "16-byte rows");
    static constexpr int exch = 0;
    static constexpr int mom = exch + 2 * 2 * 3 * NT * 16;
    static constexpr int dt = mom + 2 * NMOM * W * MROW;
    static constexpr int rim = dt + 2 * NT * 4;
    static constexpr int bnd = rim + (MODE != TSLB_MODE_SINGLE ? 2 * NT * 8 : 0);
    static constexpr int src = bnd + NACC * NT * 4;
    static constexpr int ring = src + 2 * NT * 8;
    static constexpr int curv = ring + (MODE != TSLB_MODE_SINGLE ? RING * RAREA * 4 : 0);
    static constexpr int list = curv + (MODE == TSLB_MODE_PHASEFIELD ? NT * 4 : 0);
    static constexpr int count = list + (MODE == TSLB_MODE_PHASEFIELD ? 2 * NT * 2 : 0);
    static constexpr int gcount = count + (MODE == TSLB_MODE_PHASEFIELD ? 16 : 0);
    static constexpr int bytes = gcount + 16;
};

// gradient 3 sum_i p_i c_i phi(x+c_i) of one node (Ar1) or two (Ar2) from
// phi planes held in shared memory: P(dz, dx, dy) returns phi at offset
// (dx, dy, dz) of the node(s).  Every operation is explicit (see Ar1).
template <class Ar, class LD>
__device__ __forceinline__ void grad_v(LD P, typename Ar::V g[3]) {
    using V = typename Ar::V;
    auto S4 = [](V a, V b, V c, V d) { return Ar::add(Ar::add(Ar::add(a, b), c), d); };
    const V x1 = Ar::sub(P(0, 1, 0), P(0, -1, 0));
    const V x2 = Ar::sub(S4(P(0, 1, 1), P(0, 1, -1), P(1, 1, 0), P(-1, 1, 0)),
                         S4(P(0, -1, 1), P(0, -1, -1), P(1, -1, 0), P(-1, -1, 0)));
    const V x3 = Ar::sub(S4(P(1, 1, 1), P(1, 1, -1), P(-1, 1, 1), P(-1, 1, -1)),
                         S4(P(1, -1, 1), P(1, -1, -1), P(-1, -1, 1), P(-1, -1, -1)));
    const V y1 = Ar::sub(P(0, 0, 1), P(0, 0, -1));
    const V y2 = Ar::sub(S4(P(0, 1, 1), P(0, -1, 1), P(1, 0, 1), P(-1, 0, 1)),
                         S4(P(0, 1, -1), P(0, -1, -1), P(1, 0, -1), P(-1, 0, -1)));
    const V y3 = Ar::sub(S4(P(1, 1, 1), P(1, -1, 1), P(-1, 1, 1), P(-1, -1, 1)),
                         S4(P(1, 1, -1), P(1, -1, -1), P(-1, 1, -1), P(-1, -1, -1)));
    const V z1 = Ar::sub(P(1, 0, 0), P(-1, 0, 0));
    const V z2 = Ar::sub(S4(P(1, 1, 0), P(1, -1, 0), P(1, 0, 1), P(1, 0, -1)),
                         S4(P(-1, 1, 0), P(-1, -1, 0), P(-1, 0, 1), P(-1, 0, -1)));
    const V z3 = Ar::sub(S4(P(1, 1, 1), P(1, 1, -1), P(1, -1, 1), P(1, -1, -1)),
                         S4(P(-1, 1, 1), P(-1, 1, -1), P(-1, -1, 1), P(-1, -1, -1)));
    const V c1 = Ar::c(3.f * wclass(1)), c2 = Ar::c(3.f * wclass(2)), c3 = Ar::c(3.f * wclass(3));
    g[0] = Ar::fma(c3, x3, Ar::fma(c2, x2, Ar::mul(c1, x1)));
    g[1] = Ar::fma(c3, y3, Ar::fma(c2, y2, Ar::mul(c1, y1)));
    g[2] = Ar::fma(c3, z3, Ar::fma(c2, z2, Ar::mul(c1, z1)));
}
// Phase-field interface normal (recursive_2c_TSLB3D.f90:555-571)
// n = g / (|g| + 1e-9) of one node (Ar1) or two (Ar2), operation by operation
template <class Ar>
__device__ __forceinline__ void normalize_v(typename Ar::V n[3]) {
    const typename Ar::V m2 = Ar::fma(n[2], n[2], Ar::fma(n[1], n[1], Ar::mul(n[0], n[0])));
    const typename Ar::V inv = Ar::map(m2, [](float x) { return __frcp_rn(__fadd_rn(sqrtf(x), 1e-9f)); });
    n[0] = Ar::mul(n[0], inv); n[1] = Ar::mul(n[1], inv); n[2] = Ar::mul(n[2], inv);
}
// the phase field's interface indicator phi (1 - phi) |n|^2 (recursive_2c_TSLB3D.f90:614)
template <class Ar>
__device__ __forceinline__ typename Ar::V pf_indicator(typename Ar::V phi, const typename Ar::V n[3]) {
    const typename Ar::V nn = Ar::fma(n[2], n[2], Ar::fma(n[1], n[1], Ar::mul(n[0], n[0])));
    return Ar::mul(Ar::mul(phi, Ar::sub(Ar::c(1.f), phi)), nn);
}

struct XYNode {
    int off;      // gx + nx * gy (wrapped/clamped)
    int gx, gy;   // raw coordinates (may be out of range)
    bool out;     // behind a non-periodic x or y face
};

__device__ __forceinline__ XYNode xy_node(const StepArgs& a, int gx, int gy, bool xper, bool yper) {
    XYNode n;
    n.gx = gx; n.gy = gy; n.out = false;
    int cx = gx, cy = gy;
    if (cx < 0 || cx >= a.nx) { if (xper) cx = wrapi(cx, a.nx); else { n.out = true; cx = cx < 0 ? 0 : a.nx - 1; } }
    if (cy < 0 || cy >= a.ny) { if (yper) cy = wrapi(cy, a.ny); else { n.out = true; cy = cy < 0 ? 0 : a.ny - 1; } }
    n.off = cx + a.nx * cy;
    return n;
}

using V2 = Ar2::V;

// Phase-field curvature -div n of two coefficient nodes (one per lane of the
// pairs), computed by a whole warp: the isotropic stencil over the nodes' 26
// neighbours (recursive_2c_TSLB3D.f90:617-627), each neighbour's normal
// recomputed from the staged phi; a neighbour behind a non-periodic face, or an
// interior solid one, has n = 0.  Lane j < 26 computes neighbour j of both
// and a butterfly sums the 26 terms; every lane returns the sums.  z is the
// source plane (ring index), gz its lattice plane, pi the nodes' staged offsets
// and (gx, gy) their lattice coordinates (may lie beyond a periodic face).
// What bounds it is the latency of one node's chain (loads, square root,
// reciprocal, butterfly), so two nodes go through it together.
template <int SWv, bool SOLID>
__device__ __forceinline__ V2 node_curvature(const float* ring, int parea, int z, const int pi[2], const int gx[2],
                                             const int gy[2], int gz, const StepArgs& a, bool xper, bool yper, bool zper) {
    using A = Ar2;
    const int lane = threadIdx.x;
    const int j = lane < 13 ? lane : min(lane + 1, 26);   // 3 x 3 x 3 index of the neighbour, the centre (13) skipped
    const int dx = j % 3 - 1, dy = (j / 3) % 3 - 1, dz = j / 9 - 1;
    bool ok[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int xn = gx[k] + dx, yn = gy[k] + dy, zn = gz + dz;
        ok[k] = lane < 26 && (zper || (zn >= 0 && zn < a.nz)) && (xper || (xn >= 0 && xn < a.nx)) &&
                (yper || (yn >= 0 && yn < a.ny));
        if (SOLID && ok[k]) ok[k] = !bit_at(a.solid, nidx(a, wrapi(xn, a.nx), wrapi(yn, a.ny), wrapi(zn, a.nz)));
    }
    const int o = dy * SWv + dx;
    const float *p0 = ring + ((z + dz) & (RING - 1)) * parea + o, *pm = ring + ((z + dz - 1) & (RING - 1)) * parea + o,
                *pp = ring + ((z + dz + 1) & (RING - 1)) * parea + o;
    V2 n[3];
    grad_v<A>([&](int ez, int ex, int ey) {
        const float* p = (ez < 0 ? pm : ez > 0 ? pp : p0) + ey * SWv + ex;
        return make_float2(p[pi[0]], p[pi[1]]);
    }, n);
    normalize_v<A>(n);
    V2 t = A::mul(A::c(wclass(dx * dx + dy * dy + dz * dz)),
                  A::fma(A::c((float)dz), n[2], A::fma(A::c((float)dy), n[1], A::mul(A::c((float)dx), n[0]))));
    if (!ok[0]) t.x = 0.f;
    if (!ok[1]) t.y = 0.f;
#pragma unroll
    for (int h = 16; h > 0; h >>= 1)
        t = A::add(t, make_float2(__shfl_xor_sync(0xffffffffu, t.x, h), __shfl_xor_sync(0xffffffffu, t.y, h)));
    return A::mul(A::c(-3.f), t);
}

// The value of the node at x - 1 (lo) and x + 1 (hi): the neighbouring lanes', or
// with the whole periodic axis in a warp any two lanes'.
struct ShflNext {
    __device__ __forceinline__ float lo(float v) const { return __shfl_up_sync(0xffffffffu, v, 1); }
    __device__ __forceinline__ float hi(float v) const { return __shfl_down_sync(0xffffffffu, v, 1); }
};
struct ShflWrap {
    int lm, lp;
    __device__ __forceinline__ float lo(float v) const { return __shfl_sync(0xffffffffu, v, lm); }
    __device__ __forceinline__ float hi(float v) const { return __shfl_sync(0xffffffffu, v, lp); }
};

// x sums of one monomial cy^j cz^k of P': the polynomial q0 + q1 cx + q2 cx^2
// (NI coefficients) of the nodes at x - cx, weighted 1, 4, 1 and by cx^a:
// T, D, S for a = 0, 1, 2; C (colour) as T with the factor phi(x - cx) - phi(x).
// Held in pairs, as the y and z sums treat all four alike.
struct XSum {
    V2 td, sc;
};
template <int NI, bool COL, bool ONE, class SH>
__device__ __forceinline__ XSum xsum(float q0, float q1, float q2, float dm, float dp, const SH& sh) {
    using A = Ar1;
    float Pp = q0, Pm = q0;
    if (NI == 2) { Pp = A::add(q0, q1); Pm = A::sub(q0, q1); }
    if (NI == 3) { const float t = A::add(q0, q2); Pp = A::add(t, q1); Pm = A::sub(t, q1); }
    const float a = sh.lo(Pp), b = sh.hi(Pm);
    XSum r;
    const float S = A::add(a, b);
    r.td = make_float2(A::fma(4.f, q0, S), A::sub(a, b));
    // ONE: the constant 1 of 1 + P' belongs to this monomial
    const float C = !COL ? 0.f : ONE ? A::add(A::fma(dm, a, dm), A::fma(dp, b, dp)) : A::fma(dp, b, A::mul(dm, a));
    r.sc = make_float2(S, C);
    return r;
}

// A pair of polynomials in cy, q0 + q1 cy + q2 cy^2, at cy = 1 and -1
struct YVal {
    V2 p, m;
};
template <int NJ>
__device__ __forceinline__ YVal yval(V2 q0, V2 q1, V2 q2) {
    using A = Ar2;
    const V2 t = NJ == 3 ? A::add(q0, q2) : q0;
    return YVal{A::add(t, q1), A::sub(t, q1)};
}

// Write the 11 moments of one target node; chk is their sum.
template <int MODE, class T, bool SOLID>
__device__ __forceinline__ void store_target(const StepArgs& a, unsigned int id, long long plane, unsigned int sr_step,
                                             const float* o, float chk) {
    // single-component mode does not step phi (held at 1 in both buffers)
    constexpr int nout = MODE == TSLB_MODE_SINGLE ? F_PHI : NF;
    if (SOLID && bit_at(a.solid, id)) {
        // interior solid nodes keep their moments
#pragma unroll
        for (int f = 0; f < NF; ++f) static_cast<T*>(a.fo[f])[id] = static_cast<const T*>(a.fi[f])[id];
        return;
    }
    bool bad;
    if constexpr (sizeof(T) == 2) {
        // 16-bit storage: two fields per conversion (store_pair16), stochastic
        // rounding seeded by the node (its index in the whole lattice) and the step
        const unsigned int hnode = sr_node((unsigned int)(id + a.zoff * plane), sr_step);
        float vmax = 0.f;
#pragma unroll
        for (int f = 0; f < nout; f += 2) {
            const int g = f + 1 < nout ? f + 1 : f;
            vmax = max_nan(vmax, store_pair16<T>(a, id, f, g, o[f], o[g], a.sr, sr_field(hnode, f)));
        }
        // non-finite, or beyond the storage's range (NaN fails the comparison)
        bad = !(vmax <= Stor16Max<T>::value);
    } else {
#pragma unroll
        for (int f = 0; f < nout; ++f) static_cast<T*>(a.fo[f])[id] = o[f];
        bad = !isfinite(chk);
    }
    if (bad) atomicOr(a.flags, 1u);
}

__device__ __forceinline__ void cp_async4(void* sdst, const void* gsrc) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"((unsigned)__cvta_generic_to_shared(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(sdst)), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Coefficients, [coefficient][thread], and list of the nodes of plane s that take
// the general boundary path, where the y values of plane s-1 were.
template <int W>
__device__ __forceinline__ float* listed_coefs(float4* exch, int s) {
    return reinterpret_cast<float*>(exch + ((s + 1) & 1) * (2 * 3 * 32 * W));
}
template <int W>
__device__ __forceinline__ int* listed(float* coefs) {
    static_assert((NCOEF + 1) * 4 <= 2 * 3 * 16, "list and coefficients fit a plane's y values");
    return reinterpret_cast<int*>(coefs + NCOEF * 32 * W);
}
// Moments of a node of the plane held in shared memory.
template <int MODE, class T, int W>
struct NodeMoments {
    const StepArgs& a;
    const char* m;
    const float* phi;
    // X0, y0, rx, mcol: the tile's first source column, first target row, ring column of
    // its first phi column, byte of its first column in a row of moments (-1: node by node)
    __device__ __forceinline__ NodeMoments(const StepArgs& a_, const char* sm, int row, int ln, int X0, int y0, int s, int rx, int mcol)
        : a(a_) {
        using SM = Smem<MODE, W>;
        m = sm + SM::mom + (s & 1) * NMOM * W * MROW + row * MROW + (mcol >= 0 ? mcol + ln * (int)sizeof(T) : ln * 4);
        if (sizeof(T) == 2 && mcol < 0) m += (((unsigned)s * a.plane + (unsigned)((y0 - 1 + row) * a.nx + X0 + ln)) & 1) * 2;
        phi = reinterpret_cast<const float*>(sm + SM::ring) + (s & (RING - 1)) * SM::RAREA + (row + phi_rim(MODE)) * ROWE + rx + ln + phi_rim(MODE);
    }
    __device__ __forceinline__ float operator()(int f) const {
        if (f == F_PHI) return MODE != TSLB_MODE_SINGLE ? *phi : 0.f;
        return cvt_in<T>(*reinterpret_cast<const T*>(m + f * W * MROW), a, f);
    }
};

// The listed nodes of plane s, half a warp a node, warp w taking entries 2 w,
// 2 w + 2 W, ...; their sums go to the moments from behind faces.
template <int MODE, class T, int W, bool TAU, bool SOLID>
__device__ __forceinline__ void listed_nodes(const StepArgs& a, int X0, int y0, int s, int rx, int mcol, int cnt) {
    using SM = Smem<MODE, W>;
    constexpr int NT = 32 * W;
    extern __shared__ float4 smem4[];
    char* sm = reinterpret_cast<char*>(smem4);
    float* coefs = listed_coefs<W>(reinterpret_cast<float4*>(sm + SM::exch), s);
    const int* list = listed<W>(coefs);
    const int lane = threadIdx.x, half = lane >> 4, hl = lane & 15;
    const bool xper = a.face[0].kind == TSLB_BC_PERIODIC, yper = a.face[2].kind == TSLB_BC_PERIODIC, zper = a.face[4].kind == TSLB_BC_PERIODIC;
    for (int e = 2 * threadIdx.y; e < cnt; e += 2 * W) {
        const int tn = list[min(e + half, cnt - 1)], row = tn >> 5, ln = tn & 31, x = X0 + ln, y = y0 - 1 + row;
        const unsigned mask = (xper ? 0u : (x == 0 ? 1u : 0u) | (x == a.nx - 1 ? 2u : 0u)) |
                              (yper ? 0u : (y == 0 ? 4u : 0u) | (y == a.ny - 1 ? 8u : 0u)) |
                              (zper ? 0u : (s == 0 ? 16u : 0u) | (s == a.nz - 1 ? 32u : 0u));
        const NodeMoments<MODE, T, W> mom(a, sm, row, ln, X0, y0, s, rx, mcol);
        const float dt = TAU ? reinterpret_cast<const float*>(sm + SM::dt)[(s & 1) * NT + tn] : 0.f;
        // (beside interior solids any source may be one)
        const unsigned dirs = SOLID ? 0x7ffffffu & ~(1u << 13) : directions_behind(mask);
        const int nd = __popc(dirs);
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = 0.f;
#pragma unroll 1
        for (int k = hl; k < nd; k += 16) {
            const int q = nth_bit(dirs, k);
            const Incoming in = direction_from_behind<MODE, T, SOLID>(a, coefs + tn, NT, mask, x, y, s, q, mom, dt);
            acc_dir_rt(v, q % 3 - 1, q / 3 % 3 - 1, q / 9 - 1, in.f);
            v[A_COL] += in.col;
        }
        __syncwarp();
        // sums over the half warp: lanes that differ in bit h send each other the
        // half of the values that the other keeps; lane hl is left with value hl
#pragma unroll
        for (int h = 8; h > 0; h >>= 1) {
            const bool up = lane & h;
#pragma unroll
            for (int i = 0; i < h; ++i) {
                const float keep = up ? v[i + h] : v[i], send = up ? v[i] : v[i + h];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
            }
        }
        if (hl < NACC && e + half < cnt) reinterpret_cast<float*>(sm + SM::bnd)[hl * NT + tn] = v[0];
    }
}

// The populations entering this thread's node from behind one inlet or outlet
// face f normal to y or z, where whole rows have one: the nine of them in turn, all
// of a row at once.  160 x 128 x 96 colour steps with outlets normal to y / an inlet and
// an outlet normal to z: 159 / 107 us (all 26 directions in turn 721 / 111).
constexpr int IOFACE0 = 2;
template <int MODE, class T, int W, bool TAU>
__device__ __forceinline__ void io_face(const StepArgs& a, int X0, int y0, int s, int rx, int mcol, int f) {
    using SM = Smem<MODE, W>;
    constexpr int NT = 32 * W;
    extern __shared__ float4 smem4[];
    char* sm = reinterpret_cast<char*>(smem4);
    const int lane = threadIdx.x, row = threadIdx.y, tid = row * 32 + lane, X = X0 + lane, Y = y0 - 1 + row;
    const NodeMoments<MODE, T, W> mom(a, sm, row, lane, X0, y0, s, rx, mcol);
    const float dt = TAU ? reinterpret_cast<const float*>(sm + SM::dt)[(s & 1) * NT + tid] : 0.f;
    const FaceBC& fb = a.face[f];
    const int ax = f >> 1, c = f & 1 ? -1 : 1;
    const bool inlet = fb.kind == TSLB_BC_INLET, xper = a.face[0].kind == TSLB_BC_PERIODIC;
    const bool pper = ax == 1 ? a.face[4].kind == TSLB_BC_PERIODIC : a.face[2].kind == TSLB_BC_PERIODIC;
    float m[NF];
#pragma unroll
    for (int i = 0; i < NF; ++i) m[i] = mom(i);
    float omega = a.omega_pf;
    if (MODE == TSLB_MODE_COLOUR) {
        const float ca = 0.5f * (1.f + m[F_PHI]), cb = 0.5f * (1.f - m[F_PHI]);
        const float nu = 1.f / (ca * a.inv_nu_a + cb * a.inv_nu_b);
        omega = 2.f / (6.f * nu + 1.f + 2.f * dt);
    }
    // rho at rest and (1 - omega) w a^neq(Pi, u); the moving part of f^eq is the ghost node's
    float K[K_XYZ + 1];
    coefs_moments(m[F_D], m, 0.f, 0.f, 0.f, 1.f - omega, K);
    const float rho = 1.f + m[F_D], pht = m[F_PHI];
    float v[NACC];
#pragma unroll
    for (int i = 0; i < NACC; ++i) v[i] = 0.f;
    // (colour mode: a source behind a y face was visited as a node of phi 0)
    if (MODE == TSLB_MODE_COLOUR && ax < 2) v[A_COL] = (1.f / 6.f) * pht;
    for (int q = 0; q < 9; ++q) {
        // c along the face's normal, dx and dp (z of a y face, y of a z face) in its plane
        const int dx = q % 3 - 1, dp = q / 3 - 1, dy = ax == 1 ? c : dp, dz = ax == 1 ? dp : c;
        // the ghost node it leaves: periodic axes wrap, others clamp
        const int np = ax == 1 ? a.nz : a.ny;
        int gx = X - dx, gp = (ax == 1 ? s : Y) - dp;
        gx = (unsigned)gx < (unsigned)a.nx ? gx : xper ? wrapi(gx, a.nx) : gx < 0 ? 0 : a.nx - 1;
        gp = (unsigned)gp < (unsigned)np ? gp : pper ? wrapi(gp, np) : gp < 0 ? 0 : np - 1;
        float U = fb.u[0], V = fb.u[1], Wv = fb.u[2], phib = m[F_PHI];
        if (inlet) {
            // the inlet plane's u, v, w, phi (boundary_cds_3D_module.f90:934-986)
            const long long pa = plane_area(a, f), pi = (long long)gx + (long long)a.nx * gp;
            U = fb.plane[pi]; V = fb.plane[pa + pi]; Wv = fb.plane[2 * pa + pi]; phib = fb.plane[3 * pa + pi];
        }
        const float eu = dx * U + dy * V + dz * Wv;   // (g enters with the face's velocity)
        if (!inlet) {
            // zero gradient of the normal velocity (:992)
            const float n = ld_field<T>(a, F_U + ax, ax == 1 ? nidx(a, gx, Y, gp) : nidx(a, gx, gp, s));
            if (ax == 1) V = n;
            else Wv = n;
        }
        const float t3 = 1.f / 3.f;
        const float cu = dx * U + dy * V + dz * Wv, uu = U * U + V * V + Wv * Wv;
        const float h3e = 13.5f * (U * V * ((dx * dx - t3) * dy * U + (dy * dy - t3) * dx * V) +
                                   U * Wv * ((dx * dx - t3) * dz * U + (dz * dz - t3) * dx * Wv) +
                                   V * Wv * ((dy * dy - t3) * dz * V + (dz * dz - t3) * dy * Wv)) +
                          27.f * (float)(dx * dy * dz) * U * V * Wv;
        const int c2 = 1 + dx * dx + dp * dp;
        const float wq = wclass(c2), P = eval_P(K, 1, dx, dy, dz) + rho * (3.f * cu + 4.5f * cu * cu - 1.5f * uu + h3e);
        acc_dir_rt(v, dx, dy, dz, wq * P);
        if (MODE == TSLB_MODE_COLOUR) {
            const float dphi = phib - pht;
            v[A_COL] += wq * fmaf(dphi, P, dphi);
        } else if (MODE == TSLB_MODE_PHASEFIELD && c2 == 1) {
            v[A_COL] += 0.125f * phib * (1.f + 3.f * eu);
        }
    }
    float* bnd = reinterpret_cast<float*>(sm + SM::bnd);
#pragma unroll
    for (int i = 0; i < NACC; ++i) bnd[i * NT + tid] = v[i];
}

// T: storage type of the moment state (float, __nv_bfloat16, __half).
// One block's work: target planes z0 .. z1 - 1 of tile (bx, by) of lattice a.
// TAU: the lattice has a per-node correction of the relaxation time (a.dtau).
// SOLID: the lattice has interior solid nodes (bit masks a.solid, a.near).
// GEN (a.general): 0 no node takes io_face or the general boundary path, 1 nodes take
// io_face, 2 both; the plane loop of kernels without them is faster, as they cost it
// registers (160 x 128 x 96 colour, 0 / 2: 93 / 98 us).
template <int MODE, class T, int W, bool TAU, bool SOLID, int GEN>
__device__ __forceinline__ void step_block(const StepArgs& a, int bx, int by, int z0, int z1) {
    using A = Ar2;
    using F = Ar1;
    constexpr bool ASYNC = sizeof(T) == 4;   // phi copied by cp.async (16-bit phi is converted on the way)
    constexpr bool COL = MODE == TSLB_MODE_COLOUR, PF = MODE == TSLB_MODE_PHASEFIELD, PHI = MODE != TSLB_MODE_SINGLE;
    using SM = Smem<MODE, W>;
    constexpr int RIM = phi_rim(MODE), RW = ROWE, RAREA = SM::RAREA, NEX = PF ? 2 : 1, NT = 32 * W;
    // the row is the same for the whole warp: the shuffle tells the compiler
    const int lane = threadIdx.x, wy = __shfl_sync(0xffffffffu, threadIdx.y, 0), tid = wy * 32 + lane;
    extern __shared__ float4 smem4[];
    char* sm = reinterpret_cast<char*>(smem4);
    float4* exch = reinterpret_cast<float4*>(sm + SM::exch);
    char* mst = sm + SM::mom;
    float* dts = reinterpret_cast<float*>(sm + SM::dt);
    int2* exts = reinterpret_cast<int2*>(sm + SM::rim);
    float* bnd = reinterpret_cast<float*>(sm + SM::bnd);
    float* ring = reinterpret_cast<float*>(sm + SM::ring);
    float* cq_curv = reinterpret_cast<float*>(sm + SM::curv);
    unsigned short* cq_list = reinterpret_cast<unsigned short*>(sm + SM::list);
    int* cq_n = reinterpret_cast<int*>(sm + SM::count);
    int* gen_n = reinterpret_cast<int*>(sm + SM::gcount);
    const bool xper = a.face[0].kind == TSLB_BC_PERIODIC;
    const bool yper = a.face[2].kind == TSLB_BC_PERIODIC;
    const bool zper = a.face[4].kind == TSLB_BC_PERIODIC;
    const unsigned plane = a.plane;
    // the step that seeds the stochastic rounding of 16-bit stores (an ensemble
    // advances a device counter after each step: its graph replays fixed arguments)
    const unsigned int sr_step = a.sr_counter ? *a.sr_counter : a.sr_step;

    // this thread's node: column X, row Y
    const int y0 = by * a.th, X = a.xwrap ? lane : bx * LXV - 1 + lane, Y = y0 - 1 + wy;
    const int yend = min(y0 + a.th, a.ny);
    const bool wact = Y <= yend;                // the row holds targets or sources of the tile
    const bool wtgt = Y >= y0 && Y < yend;      // targets (the rim rows only send)
    const bool valid = (a.xwrap ? lane < a.nx : (lane >= 1 && lane <= LXV && X < a.nx)) && wtgt;
    const XYNode n0 = xy_node(a, X, Y, xper, yper);
    // rows below and above, for the colour differences
    const XYNode nd = xy_node(a, X, Y - 1, xper, yper), nu = xy_node(a, X, Y + 1, xper, yper);
    // flags of the node: bits 0..3 the faces it touches (z faces are added per
    // plane), then: it, its lower, its upper neighbour lies behind an x or y
    // face; any node of the warp does
    constexpr unsigned OUT0 = 64u, OUTD = 128u, OUTU = 256u, ANYOUT = 512u, GENXY = 1024u;
    unsigned fl = (n0.out ? OUT0 : 0u) | (nd.out ? OUTD : 0u) | (nu.out ? OUTU : 0u);
    if (!xper) fl |= (X == 0 ? 1u : 0u) | (X == a.nx - 1 ? 2u : 0u);
    if (!yper) fl |= (Y == 0 ? 4u : 0u) | (Y == a.ny - 1 ? 8u : 0u);
    if (__any_sync(0xffffffffu, n0.out)) fl |= ANYOUT;
    // a plane's place in the lattice: wrapped, or the nearest plane behind a face
    auto zclamp = [&](int z) {
        if ((unsigned)z < (unsigned)a.nz) return z;
        if (!zper) return z < 0 ? 0 : a.nz - 1;
        while (z < 0) z += a.nz;
        while (z >= a.nz) z -= a.nz;
        return z;
    };
    auto zbehind = [&](int z) { return !zper && (unsigned)z >= (unsigned)a.nz; };
    auto solid_bit = [&](unsigned out, int off, int gz) {
        return (fl & out) || (SOLID && bit_at(a.solid, (unsigned)gz * plane + off));
    };

    // ---- rows read as 16-byte chunks: FP32 or 16-bit rows of whole chunks (nx a
    // multiple of EPC), x periodic (every chunk is wrapped whole) or the tile's
    // columns (with the phi rim) inside a row ----
    constexpr int EPC = 16 / (int)sizeof(T), CPR = ROWE / EPC;   // elements of a chunk, chunks of a row
    const int X0 = X - lane;
    const int Xm = X0 & ~(EPC - 1), Xp = (X0 - RIM) & ~3;        // first columns read (moments, phi)
    const bool chunks = a.nx % EPC == 0 && (xper || (X0 - RIM >= 0 && max(Xm, Xp) + ROWE <= a.nx));
    const bool yin = yper || (y0 - 1 - RIM >= 0 && y0 - 1 + W + RIM <= a.ny);   // no row behind a y face
    // (a tile with computed ghost rows reads phi node by node in every warp: a rim
    // node belongs to another warp than the row it ends, so a block reads in one way)
    const bool pchunks = PHI && ASYNC && chunks && (a.phi_mirror || yin);
    // inner: no node of the tile or its rim lies behind a face; then the planes
    // whose neighbours and reads ahead are planes of the lattice as they stand
    // take the iteration without those cases
    const bool inner = !SOLID && !a.xwrap && (xper || (X0 - RIM >= 0 && X0 + 32 + RIM <= a.nx)) && yin;

    // the tile has nodes at an x or y face, which may take the general path (direction_from_behind)
    if (GEN == 2 && ((!xper && (X0 <= 0 || X0 + 31 >= a.nx - 1)) || (!yper && (y0 == 0 || yend == a.ny)))) fl |= GENXY;

    // ---- phi ring: this thread fills its own node and up to NEX rim nodes ----
    const int rx = pchunks ? X0 - RIM - Xp : 0;   // ring column of the tile's first phi column
    const int ri = (wy + RIM) * RW + rx + lane + RIM;
    // a mirrored wall repeats the nearest node, to which the offsets are clamped;
    // other ghost values are computed
    bool slow = n0.out;
#pragma unroll
    for (int k = 0; k < NEX; ++k) {
        int2 ex = make_int2(-1, n0.off);
        constexpr int PW = 32 + 2 * RIM, side = 2 * RIM * PW;   // rim rows below and above, then side columns
        const int e = tid + k * NT;
        if (PHI && e < side + 2 * W * RIM) {
            int r, c;
            if (e < side) { r = e / PW; c = e % PW; if (r >= RIM) r += W; }
            else { r = RIM + (e - side) / (2 * RIM); c = (e - side) % (2 * RIM); if (c >= RIM) c += 32; }
            const XYNode n = xy_node(a, X0 + c - RIM, y0 - 1 + r - RIM, xper, yper);
            ex = make_int2(r * RW + rx + c, n.off);
            slow |= n.out;
        }
        if (PHI) exts[k * NT + tid] = ex;
    }
    slow = PHI && !a.phi_mirror && __any_sync(0xffffffffu, slow);
    const T* phin = static_cast<const T*>(a.fi[F_PHI]);
    // phi of a plane on its way: values, or (16-bit storage, a plane read from
    // memory) the stored bits, which are converted only when they are put in the
    // ring: a conversion at the load waits for it there and then (12% of the BF16
    // channel step)
    struct PhiRow { float own, ex[NEX]; };
    auto computed = [&](int z) { return slow || (!a.phi_mirror && zbehind(z)); };
    auto phi_raw = [&](unsigned off) {
        return __uint_as_float(sizeof(T) == 2 ? (unsigned)reinterpret_cast<const unsigned short*>(phin)[off] : 0u);
    };
    auto phi_store = [&](auto fast, int z, const PhiRow& p) {
        constexpr bool FAST = decltype(fast)::value;
        const bool raw = !ASYNC && (FAST || !computed(z));
        auto value = [&](float v) {
            if constexpr (!ASYNC) return raw ? cvt_in<T>(bits_as<T>((unsigned short)__float_as_uint(v)), a, F_PHI) : v;
            else return v;
        };
        float* slot = ring + (z & (RING - 1)) * RAREA;
        slot[ri] = value(p.own);
#pragma unroll
        for (int k = 0; k < NEX; ++k) {
            const int d = exts[k * NT + tid].x;
            if (d >= 0) slot[d] = value(p.ex[k]);
        }
    };
    // node by node
    auto phi_load = [&](int z, PhiRow& p) {
        const unsigned zoff = (unsigned)zclamp(z) * plane;
        if (computed(z)) {
            p.own = phi_at<T>(a, X, Y, z);
#pragma unroll
            for (int k = 0; k < NEX; ++k) {
                const int d = exts[k * NT + tid].x;
                p.ex[k] = d < 0 ? 0.f : phi_at<T>(a, X0 + d % RW - rx - RIM, y0 - 1 + d / RW - RIM, z);
            }
            if (ASYNC) phi_store(std::false_type{}, z, p);
        } else if (ASYNC) {
            float* slot = ring + (z & (RING - 1)) * RAREA;
            cp_async4(slot + ri, phin + (zoff + n0.off));
#pragma unroll
            for (int k = 0; k < NEX; ++k) {
                const int2 e = exts[k * NT + tid];
                if (e.x >= 0) cp_async4(slot + e.x, phin + (zoff + e.y));
            }
        } else {
            p.own = phi_raw(zoff + n0.off);
#pragma unroll
            for (int k = 0; k < NEX; ++k) p.ex[k] = phi_raw(zoff + exts[k * NT + tid].y);
        }
    };
    // A warp's chunk reads of a plane: lanes below 30 read chunk lane % CPR of
    // field lane / CPR + FPI i, i < NCHK, of their row of moments (cps: the
    // source in plane 0); lanes 10 .. 29 the phi row and, in the warps that have
    // one, a rim row (cpp).
    constexpr int FPI = 30 / CPR, NCHK = (NMOM + FPI - 1) / FPI, mlast = CPR * (NMOM - FPI * (NCHK - 1));
    const T** srcs = reinterpret_cast<const T**>(sm + SM::src) + tid;   // kept in shared memory: moments, phi
    srcs[0] = static_cast<const T*>(a.in) + (lane / CPR) * a.N + (xy_node(a, 0, Y, xper, yper).off + wrapi(Xm + (lane % CPR) * EPC, a.nx));
    char* cpd = mst + (lane / CPR) * W * MROW + wy * MROW + (lane % CPR) * 16;
    const T* cpp = nullptr;
    int cpr = 0;
    if (pchunks && lane >= 10 && lane < 30) {
        int r = wy + RIM;
        bool has = true;
        if (lane >= 20) {   // rim rows: below in the first warps, above in the last
            has = wy < RIM || wy >= W - RIM;
            r = wy < RIM ? wy : wy + 2 * RIM;
        }
        if (has) {
            const XYNode n = xy_node(a, 0, y0 - 1 + r - RIM, xper, yper);
            cpp = phin + (n.off + wrapi(Xp + (lane % 10) * 4, a.nx));
            cpr = r * RW + (lane % 10) * 4;
        }
    }
    srcs[NT] = cpp;
    // two-dimensional parts of the gradient of one phi plane at the node: the x
    // and y derivatives smoothed across, phi (c) and the smoothed phi less 36 c.
    // Differences of phi come first, sums after: near a uniform phi the
    // differences are exact, and the gradient's error is that of phi itself.
    struct Sten { float dx, dy, ss, c; };
    auto stencil = [&](int z) {
        const float* r = ring + (z & (RING - 1)) * RAREA + ri - RW;
        float d[3], s[3], c[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            c[k] = r[k * RW];
            const float l = F::sub(r[k * RW - 1], c[k]), h = F::sub(r[k * RW + 1], c[k]);
            d[k] = F::sub(h, l);
            s[k] = F::add(h, l);
        }
        const float lo = F::sub(c[0], c[1]), hi = F::sub(c[2], c[1]);
        Sten q;
        q.dx = F::fma(4.f, d[1], F::add(d[0], d[2]));
        q.dy = F::fma(6.f, F::sub(hi, lo), F::sub(s[2], s[0]));
        q.ss = F::fma(6.f, F::add(hi, lo), F::fma(4.f, s[1], F::add(s[0], s[2])));
        q.c = c[1];
        return q;
    };

    // ---- reads ahead: phi of plane zp, then (mom) the moments and tau correction
    // of plane z, as two groups of copies ----
    auto load_ahead = [&](auto fast, int z, int zp, bool mom, PhiRow& p) {
        constexpr bool FAST = decltype(fast)::value;
        if (PHI && FAST) {
            const unsigned zoff = (unsigned)zp * plane;
            if (pchunks) {
                const T* cpp = srcs[NT];
                if (cpp) cp_async16(ring + cpr + (zp & (RING - 1)) * RAREA, cpp + zoff);
            } else if (ASYNC) {
                float* slot = ring + (zp & (RING - 1)) * RAREA;
                cp_async4(slot + ri, phin + (zoff + n0.off));
#pragma unroll
                for (int k = 0; k < NEX; ++k) {
                    const int2 e = exts[k * NT + tid];
                    if (e.x >= 0) cp_async4(slot + e.x, phin + (zoff + e.y));
                }
            } else {
                p.own = phi_raw(zoff + n0.off);
#pragma unroll
                for (int k = 0; k < NEX; ++k) p.ex[k] = phi_raw(zoff + exts[k * NT + tid].y);
            }
        } else if (PHI) {
            if (pchunks && (a.phi_mirror || !zbehind(zp))) {   // (no ghost columns or rows: never `slow`)
                const T* cpp = srcs[NT];
                if (cpp) cp_async16(ring + cpr + (zp & (RING - 1)) * RAREA, cpp + (unsigned)zclamp(zp) * plane);
            } else {
                phi_load(zp, p);
            }
        }
        cp_async_commit();
        if (mom) {
            const unsigned zoff = (unsigned)(FAST ? z : zclamp(z)) * plane;
            const int par = (z & 1) * NMOM * W * MROW;
            if (TAU) cp_async4(dts + (z & 1) * NT + tid, a.dtau + (zoff + n0.off));
            if (chunks) {
                const T* src = srcs[0] + zoff;
                if (lane < 30) {
#pragma unroll
                    for (int i = 0; i < NCHK; ++i) {
                        if (i < NCHK - 1 || lane < mlast) cp_async16(cpd + par + i * FPI * W * MROW, src);
                        src += FPI * a.N;
                    }
                }
            } else {
                // node by node: the 4-byte word that holds it
                const unsigned id = zoff + n0.off;
                char* st = mst + par + wy * MROW + lane * 4;
#pragma unroll
                for (int f = 0; f < NMOM; ++f)
                    cp_async4(st + f * W * MROW, static_cast<const unsigned*>(a.fi[f]) + (sizeof(T) == 4 ? id : id >> 1));
            }
        }
        cp_async_commit();
    };
    // the node's moments from a plane read ahead (after the warp's copies have landed)
    float m[NF], dt = 0.f;
    const char* mrd = mst + wy * MROW + (chunks ? (X - Xm) * (int)sizeof(T) : lane * 4);
    auto mom_take = [&](int z) {
        const char* e = mrd + (z & 1) * NMOM * W * MROW;
        if (sizeof(T) == 2 && !chunks) e += (((unsigned)zclamp(z) * plane + n0.off) & 1) * 2;
#pragma unroll
        for (int f = 0; f < NMOM; ++f) m[f] = cvt_in<T>(*reinterpret_cast<const T*>(e + f * W * MROW), a, f);
        if (TAU) dt = dts[(z & 1) * NT + tid];
    };

    // Phase field: the curvature of a plane's interface nodes is shared by all
    // warps of the block.  The coefficient phase of plane s lists the nodes of
    // plane s+1 that may need it (candidates: phi (1 - phi) above the
    // indicator's threshold, a superset of the nodes where phi (1 - phi) |n|^2
    // exceeds it); the next coefficient phase, after the plane barrier, first
    // computes their curvatures warp by warp, then (one more barrier) the
    // coefficients.  cslot: the node's position in its plane's list.
    int cslot = -1;
    auto list_candidates = [&](int z) {
        cslot = -1;
        if (zbehind(z) || !wact || solid_bit(OUT0, n0.off, zclamp(z))) return;
        const float ph = ring[(z & (RING - 1)) * RAREA + ri];
        if (!(ph * (1.f - ph) > 0.2f * (1.f - 1e-5f))) return;
        cslot = atomicAdd(&cq_n[z & 1], 1);
        cq_list[(z & 1) * NT + cslot] = (unsigned short)tid;
    };

    // The step may have been launched while the kernel before it still runs: the
    // indices above are its own, all that follows reads what that kernel wrote.
    cudaGridDependencySynchronize();

    // prologue: the phi planes the first source plane reads, its moments
    for (int z = z0 - 1 - RIM; z <= z0 - 1 + RIM; ++z) {
        PhiRow p;
        if (PHI || z == z0 - 1 + RIM) load_ahead(std::false_type{}, z0 - 1, z, wact && z == z0 - 1 + RIM, p);
        if (PHI && !ASYNC) phi_store(std::false_type{}, z, p);
    }
    if (PF && tid == 0) cq_n[0] = cq_n[1] = 0;
    if (GEN == 2 && tid == 0) *gen_n = 0;
    cp_async_wait<0>();
    __syncthreads();
    // gradient so far at planes s (x, y: planes s-1 and s; z: their difference) and
    // s+1 (plane s; z: its smoothed phi gs, phi itself being in the ring)
    float gx = 0.f, gy = 0.f, gz_ = 0.f, gx1 = 0.f, gy1 = 0.f, gs = 0.f;
    // own phi (0 at nodes that send nothing) of one plane of the ring;
    // of a plane behind a z face: the nearest plane's, so that it has no phi difference
    auto own_phi = [&](int z) {
        const int zc = zclamp(z);
        float p = ring[((zbehind(z) ? zc : z) & (RING - 1)) * RAREA + ri];
        if (SOLID || (fl & ANYOUT)) {
            if (solid_bit(OUT0, n0.off, zc)) p = 0.f;
        }
        return p;
    };
    if (PHI) {
        const Sten a1 = stencil(z0 - 2), a2 = stencil(z0 - 1);
        gx = F::fma(4.f, a2.dx, a1.dx); gy = F::fma(4.f, a2.dy, a1.dy);
        gx1 = a2.dx; gy1 = a2.dy;
        gz_ = F::fma(36.f, F::sub(a2.c, a1.c), F::sub(a2.ss, a1.ss)); gs = a2.ss;
    }
    if (PF) {
        list_candidates(z0 - 1);
        __syncthreads();
    }

    // partial sums of the targets, in units of 1/216.  Moments (a, b, c) in
    // pairs: A = (00, 10), B = (20, colour), M = (01, 11) and 02 of a, b.
    // Target s: M0* (c = 0), M1* (c = 1: 00 10 01), M2 (c = 2: 00);
    // target s+1: U* (the same for every c).
    const V2 zero2 = make_float2(0.f, 0.f);
    V2 M0A = zero2, M0B = zero2, M0M = zero2, M1A = zero2, UA = zero2, UB = zero2, UM = zero2;
    float M02 = 0.f, M1b = 0.f, M2 = 0.f, U02 = 0.f;

    // source plane s.  FAST: an inner tile and plane (see `inner`)
    auto iterate = [&](auto fast, const int s) {
        constexpr bool FAST = decltype(fast)::value;
        const bool more = s < z1;
        auto neighbours = [&]() {
            if constexpr (FAST) return ShflNext{};
            else return ShflWrap{a.xwrap ? (lane == 0 ? a.nx - 1 : lane - 1) : max(lane - 1, 0),
                                 a.xwrap && lane == a.nx - 1 ? 0 : min(lane + 1, 31)};
        };
        const auto sh = neighbours();
        const bool zsolid = !FAST && zbehind(s);   // a solid source plane sends nothing
        const int gz = FAST ? s : zclamp(s);
        auto phi_of = [&](int z) { return FAST ? ring[(z & (RING - 1)) * RAREA + ri] : own_phi(z); };
        float4* ex = exch + (s & 1) * (2 * 3 * NT);
        // ---- 0. moments of the next plane, phi of the plane after the ring's last ----
        cp_async_wait<0>();
        __syncwarp();   // the warp's copies of the moments of plane s have landed
        // The listed nodes' coefficients, [coefficient][thread], and the list are kept
        // where the y values of plane s-1 were, once every warp has read those.
        const bool gen = GEN == 2 && !FAST && s >= z0 && s < z1 && ((fl & GENXY) || (!zper && (s == 0 || s == a.nz - 1)));
        if (gen) __syncthreads();
        PhiRow ph;
        if (more) load_ahead(fast, s + 1, s + 1 + RIM, wact, ph);
        // ---- curvatures of this plane's candidates, warp w taking entries w, w + nw, ...
        // (the count is the same for every thread: the list was completed before
        // the previous plane's barrier)
        if (PF) {
            const int cnt = cq_n[s & 1];
            if (cnt > 0) {
                for (int e = wy; e < cnt; e += 2 * W) {
                    int pi[2], gx2[2], gy2[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {   // (an odd last entry twice)
                        const int ci = cq_list[(s & 1) * NT + (e + k * W < cnt ? e + k * W : e)];
                        gx2[k] = X0 + (ci & 31);
                        gy2[k] = y0 - 1 + (ci >> 5);
                        pi[k] = ((ci >> 5) + RIM) * RW + rx + (ci & 31) + RIM;
                    }
                    const V2 k2 = node_curvature<RW, SOLID>(ring, RAREA, s, pi, gx2, gy2, gz, a, xper, yper, zper);
                    if (lane == 0) {
                        cq_curv[e] = k2.x;
                        if (e + W < cnt) cq_curv[e + W] = k2.y;
                    }
                }
                __syncthreads();
                // every thread has read cnt; the next entries of this parity come after the plane barrier
                if (tid == 0) cq_n[s & 1] = 0;
            }
        }
        // kept across the barrier: the sums at cy = 0 per k, own phi of plane s+1
        V2 ktd[3], ksc[3];
        float pc = 0.f, rest = 0.f, gzf = 0.f;
        bool near = false;   // the target has populations from behind a face or from interior solids
        if (wact) {
            // ---- 1. coefficients ----
            float g[3], K[NCOEF];
            mom_take(s);
            if (PHI) {
                const Sten q = stencil(s + 1);
                constexpr float k72 = 1.f / 72.f;
                g[0] = F::mul(F::add(gx, q.dx), k72);
                g[1] = F::mul(F::add(gy, q.dy), k72);
                const float dz = F::fma(36.f, F::sub(q.c, ring[(s & (RING - 1)) * RAREA + ri]), F::sub(q.ss, gs));
                g[2] = F::mul(F::add(gz_, dz), k72);
                gz_ = dz; gs = q.ss;
                gx = F::fma(4.f, q.dx, gx1); gx1 = q.dx;
                gy = F::fma(4.f, q.dy, gy1); gy1 = q.dy;
            }
            bool iface = false;
            if (COL) {
                m[F_PHI] = pc = phi_of(s);
                iface = coefs_colour<TAU>(a, m, g, dt, K);
            } else if (PF) {
                m[F_PHI] = ring[(s & (RING - 1)) * RAREA + ri];
                normalize_v<F>(g);
                // a node that needs the curvature was listed as a candidate
                const float curv = pf_indicator<F>(m[F_PHI], g) > 0.2f && cslot >= 0 ? cq_curv[cslot] : 0.f;
                coefs_shifted<true>(a, m, g, curv, K);
            } else {
                coefs_shifted<false>(a, m, g, 0.f, K);
            }
            // solid nodes (behind a face, or interior solids) send nothing
            if (!FAST && (SOLID || (fl & ANYOUT) || zsolid)) {
                if (zsolid || solid_bit(OUT0, n0.off, gz)) {
#pragma unroll
                    for (int c = 0; c < NCOEF; ++c) K[c] = 0.f;
                }
            }
            // ---- populations from behind non-periodic faces, target plane s ----
            bool io = false;   // from behind one inlet or outlet face normal to y or z
            if (!FAST && s >= z0 && s < z1) {
                const unsigned mask = (fl & 15u) | (zper ? 0u : (s == 0 ? 16u : 0u) | (s == a.nz - 1 ? 32u : 0u));
                near = valid && (mask || (SOLID && bit_at(a.near, (unsigned)s * plane + n0.off)));
                if (near) {
                    const Strided<NT> acc{bnd + tid};
                    bool allbounce = true;
#pragma unroll
                    for (int f = 0; f < 6; ++f)
                        if (mask >> f & 1u) allbounce = allbounce && a.face[f].kind == TSLB_BC_BOUNCEBACK;
                    const bool bounce = allbounce && (mask & mask >> 1 & 0x15u) == 0;   // (one face of each axis)
                    const int f = __ffs(mask) - 1, kind = f >= 0 ? a.face[f].kind : TSLB_BC_PERIODIC;
                    const bool solids = SOLID && bit_at(a.near, (unsigned)s * plane + n0.off);
                    if (SOLID && solids && allbounce) {
                        bounce_solids<MODE>(a, K, mask, X, Y, s, acc);
                    } else if (!solids && (bounce || ((mask & (mask - 1)) == 0 && (kind == TSLB_BC_VELOCITY || kind == TSLB_BC_PRESSURE)))) {
#pragma unroll
                        for (int i = 0; i < NACC; ++i) acc[i] = 0.f;
                        if (bounce) {
                            bounce_target<MODE>(K, mask, acc);
                        } else {
                            mom_take(s);
                            face_target<MODE>(a, K, m, dt, f, acc);
                        }
                    } else if (GEN && !solids && (mask & (mask - 1)) == 0 && f >= IOFACE0) {
                        io = true;   // (taken when the coefficients' registers are free)
                    } else if (GEN == 2) {
                        float* gen_k = listed_coefs<W>(exch, s);
                        listed<W>(gen_k)[atomicAdd(gen_n, 1)] = tid;
#pragma unroll
                        for (int c = 0; c < NCOEF; ++c) gen_k[c * NT + tid] = K[c];
                    }
                }
            }
            // ---- x sums, y values ----
            float dm = 0.f, dp = 0.f, upd = 0.f, dnd = 0.f;
            if (COL && !zsolid) {
                // phi differences along x and y (0 for a node that sends nothing)
                dm = F::sub(sh.lo(pc), pc);
                dp = F::sub(sh.hi(pc), pc);
                const float* r = ring + (s & (RING - 1)) * RAREA + ri;
                float pd = r[-RW], pu = r[RW];
                if (!FAST && solid_bit(OUTD, nd.off, gz)) pd = 0.f;
                if (!FAST && solid_bit(OUTU, nu.off, gz)) pu = 0.f;
                upd = F::sub(pc, pu);
                dnd = F::sub(pc, pd);
            }
            // recolouring sum_c (w_c / |c|) c.B over the neighbours, by class of |c|
            float rB = 0.f, rE1 = 0.f, rE2 = 0.f, rZc = 0.f, rZs = 0.f;
            constexpr float w1 = 16.f, w2 = 4.f * 0.70710678118654752f, w3 = 0.57735026918962576f;
            if (COL && iface) {
                auto sum = [&](float v) { return F::add(sh.lo(v), sh.hi(v)); };
                rB = F::sub(sh.lo(K[K_C1]), sh.hi(K[K_C1]));
                const float sy = sum(K[K_C2]), sz = sum(K[K_C3]);
                rE1 = F::fma(0.25f * w2, sy, F::mul(0.25f * w1, K[K_C2]));
                rE2 = F::fma(w3, sy, F::mul(w2, K[K_C2]));
                rZc = F::fma(0.25f * w2, sz, F::mul(0.25f * w1, K[K_C3]));
                rZs = F::fma(w3, sz, F::mul(w2, K[K_C3]));
            }
            if (COL) rest = K[K_C4];
            // y values of one k: the sums at cy = 1 and -1 go to the rows above and below
            auto send = [&](int k, V2 td, V2 sc, const YVal& ytd, const YVal& ysc) {
                ktd[k] = td;
                ksc[k] = sc;
                ex[(0 * 3 + k) * NT + tid] = make_float4(ytd.p.x, ytd.p.y, ysc.p.x, ysc.p.y);
                ex[(1 * 3 + k) * NT + tid] = make_float4(ytd.m.x, ytd.m.y, ysc.m.x, ysc.m.y);
            };
            {   // k = 0
                const XSum j0 = xsum<3, COL, true>(K[K_0], K[K_X], K[K_XX], dm, dp, sh);
                const XSum j1 = xsum<3, COL, false>(K[K_Y], K[K_XY], K[K_XXY], dm, dp, sh);
                const XSum j2 = xsum<2, COL, false>(K[K_YY], K[K_XYY], 0.f, dm, dp, sh);
                const YVal t = yval<3>(j0.td, j1.td, j2.td);
                YVal c = yval<3>(j0.sc, j1.sc, j2.sc);
                V2 cc = j0.sc;
                if (COL) {
                    // the receiver's phi difference; the x weights of the constant 1 sum to 6
                    c.p.y = F::fma(upd, F::add(t.p.x, 6.f), c.p.y);
                    c.m.y = F::fma(dnd, F::add(t.m.x, 6.f), c.m.y);
                    if (iface) {
                        const float h = F::mul(0.25f * w2, rB);
                        cc.y = F::add(cc.y, rB);
                        c.p.y = F::add(c.p.y, F::add(h, rE1));
                        c.m.y = F::add(c.m.y, F::sub(h, rE1));
                    }
                }
                if (PF) {
                    // phase field g (D3Q7): axis directions and the rest population (q = 0:
                    // p0g phi = 2 G0), in units of 1/4 and 1/16 like the sums beside them
                    const float g0 = K[K_C0];
                    const float sx = F::add(sh.lo(F::add(g0, K[K_C1])), sh.hi(F::sub(g0, K[K_C1])));
                    cc.y = F::mul(0.0625f, F::fma(2.f, g0, sx));
                    c.p.y = F::mul(0.25f, F::add(g0, K[K_C2]));
                    c.m.y = F::mul(0.25f, F::sub(g0, K[K_C2]));
                    rest = g0;
                    gzf = K[K_C3];
                }
                send(0, j0.td, cc, t, c);
            }
            {   // k = 1
                const XSum j0 = xsum<3, COL, false>(K[K_Z], K[K_XZ], K[K_XXZ], dm, dp, sh);
                const XSum j1 = xsum<2, COL, false>(K[K_YZ], K[K_XYZ], 0.f, dm, dp, sh);
                const XSum j2 = xsum<1, COL, false>(K[K_YYZ], 0.f, 0.f, dm, dp, sh);
                const YVal t = yval<3>(j0.td, j1.td, j2.td);
                YVal c = yval<3>(j0.sc, j1.sc, j2.sc);
                V2 cc = j0.sc;
                if (COL) {
                    c.p.y = F::fma(upd, t.p.x, c.p.y);
                    c.m.y = F::fma(dnd, t.m.x, c.m.y);
                    if (iface) {
                        cc.y = F::add(cc.y, rZc);
                        c.p.y = F::add(c.p.y, rZs);
                        c.m.y = F::add(c.m.y, rZs);
                    }
                }
                send(1, j0.td, cc, t, c);
            }
            {   // k = 2
                const XSum j0 = xsum<2, COL, false>(K[K_ZZ], K[K_XZZ], 0.f, dm, dp, sh);
                const XSum j1 = xsum<1, COL, false>(K[K_YZZ], 0.f, 0.f, dm, dp, sh);
                const YVal t = yval<2>(j0.td, j1.td, zero2);
                YVal c = yval<2>(j0.sc, j1.sc, zero2);
                V2 cc = j0.sc;
                if (COL) {
                    c.p.y = F::fma(upd, t.p.x, c.p.y);
                    c.m.y = F::fma(dnd, t.m.x, c.m.y);
                    if (iface) {
                        // what k = 0 put into the planes s+-1 is taken out again
                        const float h = F::mul(w3 - 0.25f * w2, rB), e = F::sub(rE2, rE1);
                        cc.y = F::fma(0.25f * w2 - 1.f, rB, cc.y);
                        c.p.y = F::add(c.p.y, F::add(h, e));
                        c.m.y = F::add(c.m.y, F::sub(h, e));
                    }
                }
                send(2, j0.td, cc, t, c);
            }
            if (GEN && !FAST && io) {
                const int f = (fl & 15u) ? __ffs(fl & 15u) - 1 : s == 0 ? 4 : 5;
                io_face<MODE, T, W, TAU>(a, X0, y0, s, rx, chunks ? (X0 - Xm) * (int)sizeof(T) : -1, f);
            }
        }
        // phase field: candidates of the next source plane (its phi is staged)
        if (PF) {
            if (more) list_candidates(s + 1);
            else cslot = -1;
        }
        if (PHI && !ASYNC && more) phi_store(fast, s + 1 + RIM, ph);
        cp_async_wait<1>();   // this thread's phi copies have landed
        __syncthreads();
        if (gen) {   // the listed nodes
            const int cnt = *gen_n;
            if (cnt > 0) {
                listed_nodes<MODE, T, W, TAU, SOLID>(a, X0, y0, s, rx, chunks ? (X0 - Xm) * (int)sizeof(T) : -1, cnt);
                __syncthreads();
                // (the next entries come after a barrier that follows this)
                if (tid == 0) *gen_n = 0;
            }
        }
        if (!wtgt) return;
        // ---- 3. y and z sums ----
        V2 HA[3], HB[3], HM[3];
        float H2[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            // from the row below (cy = 1) and above (cy = -1)
            const float4 lo = ex[(0 * 3 + k) * NT + max(tid - 32, lane)];
            const float4 hi = ex[(1 * 3 + k) * NT + min(tid + 32, NT - 32 + lane)];
            const V2 ltd = make_float2(lo.x, lo.y), htd = make_float2(hi.x, hi.y);
            const V2 std_ = A::add(ltd, htd), ssc = A::add(make_float2(lo.z, lo.w), make_float2(hi.z, hi.w));
            HA[k] = A::fma(A::c(4.f), ktd[k], std_);
            HB[k] = A::fma(A::c(4.f), ksc[k], ssc);
            HM[k] = A::sub(ltd, htd);
            H2[k] = std_.x;
        }
        const V2 tA = A::add(HA[0], HA[2]), tB = A::add(HB[0], HB[2]), tM = A::add(HM[0], HM[2]);
        const float t2 = F::add(H2[0], H2[2]);
        const V2 pA = A::add(tA, HA[1]), mA = A::sub(tA, HA[1]), pM = A::add(tM, HM[1]), mM = A::sub(tM, HM[1]);
        V2 pB = A::add(tB, HB[1]), mB = A::sub(tB, HB[1]);
        const float p2 = F::add(t2, H2[1]), m2 = F::sub(t2, H2[1]);
        const float pm_ = COL ? phi_of(s - 1) : 0.f;
        if (COL) {
            const float pn = phi_of(s + 1);
            // the receiver's phi difference; the x and y weights of the constant 1 sum to 36
            pB.y = F::fma(F::sub(pc, pn), F::add(pA.x, 36.f), pB.y);
            mB.y = F::fma(F::sub(pc, pm_), F::add(mA.x, 36.f), mB.y);
        }
        if (PF) {
            pB.y = F::add(rest, gzf);
            mB.y = F::sub(rest, gzf);
        }
        // ---- target plane s-1 is complete ----
        M0A = A::add(M0A, mA); M0B = A::add(M0B, mB); M0M = A::add(M0M, mM);
        M02 = F::add(M02, m2);
        M1A = A::sub(M1A, mA);
        M1b = F::sub(M1b, mM.x);
        M2 = F::add(M2, mA.x);
        const int t = s - 1;
        if (valid && t >= z0) {
            constexpr float c216 = 1.f / 216.f;
            const float d = F::mul(M0A.x, c216), rho = F::add(d, 1.f), inv = F::mul(__frcp_rn(rho), c216);
            float o[NF];
            o[F_D] = d;
            const float u = o[F_U] = F::mul(M0A.y, inv), v = o[F_V] = F::mul(M0M.x, inv), w = o[F_W] = F::mul(M1A.x, inv);
            const float ru = F::mul(-rho, u), rv = F::mul(-rho, v), rw = F::mul(-rho, w), d3 = F::mul(d, -1.f / 3.f);
            o[F_XX] = F::fma(ru, u, F::fma(M0B.x, c216, d3));
            o[F_YY] = F::fma(rv, v, F::fma(M02, c216, d3));
            o[F_ZZ] = F::fma(rw, w, F::fma(M2, c216, d3));
            o[F_XY] = F::fma(ru, v, F::mul(M0M.y, c216));
            o[F_XZ] = F::fma(ru, w, F::mul(M1A.y, c216));
            o[F_YZ] = F::fma(rv, w, F::mul(M1b, c216));
            // colour mode: phi_t + (colour increment) / rho
            o[F_PHI] = COL ? F::fma(M0B.y, inv, pm_) : M0B.y;
            float chk = 0.f;
            if (sizeof(T) == 4) {
#pragma unroll
                for (int f = 0; f < (PHI ? NF : F_PHI); ++f) chk = F::add(chk, o[f]);
            }
            store_target<MODE, T, SOLID>(a, (unsigned)t * plane + n0.off, plane, sr_step, o, chk);
        }
        // ---- rotate: target s becomes the one to complete, s+1 opens ----
        M1A = UA; M1b = UM.x; M2 = UA.x;
        M0A = A::fma(A::c(4.f), HA[0], UA);
        M0B = A::fma(A::c(4.f), HB[0], UB);
        M0M = A::fma(A::c(4.f), HM[0], UM);
        M02 = F::fma(4.f, H2[0], U02);
        UA = pA; UB = pB; UM = pM; U02 = p2;
        if (COL) M0A.x = F::fma(216.f, rest, M0A.x);   // rest population: f_0 += delta0
        if (!FAST && near) {
            auto add = [&](float& v, int i) { v = F::fma(216.f, bnd[i * NT + tid], v); };
            add(M0A.x, A_RHO); add(M0A.y, A_JX); add(M0B.x, A_XX); add(M0M.x, A_JY); add(M0M.y, A_XY); add(M02, A_YY);
            add(M1A.x, A_JZ); add(M1A.y, A_XZ); add(M1b, A_YZ); add(M2, A_ZZ);
            if (COL) add(M0B.y, A_COL);
            if (PF) M0B.y = F::add(M0B.y, bnd[A_COL * NT + tid]);
        }
    };
    const int f0 = max(z0 - 1, 1), f1 = min(z1, a.nz - 2 - RIM);
    for (int s = z0 - 1; s <= z1;) {
        if (inner && s >= f0 && s <= f1) {
#pragma unroll 1
            for (; s <= f1; ++s) iterate(std::true_type{}, s);
        } else {
            iterate(std::false_type{}, s);
            ++s;
        }
    }
    cp_async_wait<0>();
}

// Blocks of consecutive index work on tiles next to each other in x, at the
// same planes, so that the rows and memory sectors they share are read from
// DRAM once.  zchunk > 0: every block takes one chunk of zchunk planes of a
// tile.  zchunk = 0: the tiles of one x position, each with all its target
// planes, are a sequence of planes; grid / tx blocks take equal shares of it,
// in one piece or, across the end of a tile, in several.
template <int MODE, class T, int W, bool TAU, bool SOLID, int GEN>
__global__ void __launch_bounds__(32 * W, BIGW / W) step_kernel(const __grid_constant__ StepArgs a) {
    cudaTriggerProgrammaticLaunchCompletion();   // the next step may start; it waits as this one does
    const int planes = a.zt1 - a.zt0, tx = a.xwrap ? 1 : (a.nx + LXV - 1) / LXV, ty = (a.ny + a.th - 1) / a.th;
    const int bx = blockIdx.x % tx, b = blockIdx.x / tx;
    int p, end;   // the block's part of the sequence
    if (a.zchunk > 0) {
        const int first = b % ty * planes, z = b / ty * a.zchunk;
        p = first + z;
        end = first + min(z + a.zchunk, planes);
    } else {
        const long long total = (long long)ty * planes, n = gridDim.x / tx;
        p = (int)(total * b / n);
        end = (int)(total * (b + 1) / n);
    }
    while (p < end) {
        const int by = p / planes, z = p % planes, n = min(end - p, planes - z);
        step_block<MODE, T, W, TAU, SOLID, GEN>(a, bx, by, a.zt0 + z, a.zt0 + z + n);
        p += n;
        if (p < end) __syncthreads();
    }
}

// Work item of the ensemble kernel: lattice, tile column, z chunk.
struct WorkItem {
    int dom, bx, by, bz;
};

// Ensemble step: blocks walk a list of work items over many independent
// lattices; each item is one tile column and z chunk of one lattice.  Block
// b starts with item b; later items go, in list order (longest first), to
// whichever block asks next (a work counter), so a grid smaller than the
// list balances items of uneven length.  The lattice's arguments are staged
// in shared memory when the block moves to a new lattice.  All lattices
// share MODE and T.  step[0] is the step counter that seeds the
// stochastic rounding (every member's arguments point at it), step[1] a
// ticket and step[2] the work counter: the last block of the launch to
// finish, after every block has read the step and taken its last item,
// advances the step and clears the other two for the next launch.
template <int MODE, class T, int GEN>
__global__ void __launch_bounds__(32 * SMALLW, BIGW / SMALLW) ensemble_kernel(const StepArgs* __restrict__ args,
                                                          const WorkItem* __restrict__ work, int nwork,
                                                          unsigned int* step) {
    __shared__ StepArgs sa;
    __shared__ int next;
    int cur = -1;
    for (int it = blockIdx.x; it < nwork;) {
        const WorkItem w = work[it];
        if (w.dom != cur) {
            __syncthreads();
            const int words = (int)(sizeof(StepArgs) / sizeof(int));
            const int* src = reinterpret_cast<const int*>(args + w.dom);
            int* dst = reinterpret_cast<int*>(&sa);
            for (int i = threadIdx.y * 32 + threadIdx.x; i < words; i += 32 * SMALLW) dst[i] = src[i];
            __syncthreads();
            cur = w.dom;
        }
        step_block<MODE, T, SMALLW, false, false, GEN>(sa, w.bx, w.by, sa.zt0 + w.bz * sa.zchunk, min(sa.zt0 + (w.bz + 1) * sa.zchunk, sa.zt1));
        __syncthreads();
        // every thread has read `next` (it was read before this item's barriers)
        if (step) {
            if (threadIdx.x == 0 && threadIdx.y == 0) next = (int)gridDim.x + (int)atomicAdd(step + 2, 1u);
            __syncthreads();
            it = next;
        } else {
            it += gridDim.x;
        }
    }
    if (step && threadIdx.x == 0 && threadIdx.y == 0) {
        __threadfence();
        if (atomicAdd(step + 1, 1u) == gridDim.x - 1) {
            step[1] = 0;
            step[2] = 0;
            step[0] += 1;
            __threadfence();
        }
    }
}

}  // namespace tslb
