// tslb_device.cuh -- device-side building blocks of the fused TSLB step.
//
// State layout in HBM: 11 SoA fields of nx*ny*nz floats (x fastest, field
// stride N padded to 32 floats):
//   0 d = rho - 1   1 u   2 v   3 w   4 pxx 5 pxy 6 pxz 7 pyy 8 pyz 9 pzz  10 phi
// p** is the non-equilibrium second moment Pi^neq.  Storing rho - 1 keeps
// the density's small deviations exact to FP32 round-off of the deviation.
//
// Post-collision populations are written as f_c = w_c (1 + P'(c)) where
// P'(c) is a polynomial in the components of c with 17 per-node
// coefficients (the monomials 1, cx, cy, cz, cx^2, ..., cx cy cz that
// survive on D3Q27 because c_a^3 = c_a).  The coefficients fold:
//   f^eq(rho, u_s) in third-order Hermite form
//     (recursive_2c_TSLB3D.f90:639-804 "feqs")
//   (1 - omega) w a^neq(Pi, u), the recursive regularized non-equilibrium
//     (recursive_2c_TSLB3D.f90:640-805 "fneq1")
//   colour mode: the perturbation operator and the force source of
//     turbulent_benchmark/couette/recursive_colorTSLB3D.f90:765-959
// so that every pulled population costs a handful of FMAs.
#pragma once

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdint>
#include <type_traits>

#include "../../include/tslb.h"

namespace tslb {

constexpr int NF = 11;
enum { F_D = 0, F_U, F_V, F_W, F_XX, F_XY, F_XZ, F_YY, F_YZ, F_ZZ, F_PHI };

// Coefficient slots of a node: the 17 monomials of P' and the colour terms
// c0..c4: phi, Bx, By, Bz, delta0 | phase field: G0, G1x, G1y, G1z, -.
enum {
    K_0 = 0, K_X, K_Y, K_Z, K_XX, K_YY, K_ZZ, K_XY, K_XZ, K_YZ,
    K_XXY, K_XXZ, K_XYY, K_YYZ, K_XZZ, K_YZZ, K_XYZ,
    K_C0, K_C1, K_C2, K_C3, K_C4,
    NCOEF
};

// accumulator slots of a target node
enum { A_RHO = 0, A_JX, A_JY, A_JZ, A_XX, A_XY, A_XZ, A_YY, A_YZ, A_ZZ, A_COL, NACC };

// lattice weights by |c|^2 (recursive_2c_TSLB3D.f90:71-74)
__host__ __device__ constexpr float wclass(int c2) {
    return c2 == 0 ? 8.0f / 27.0f : c2 == 1 ? 2.0f / 27.0f : c2 == 2 ? 1.0f / 54.0f : 1.0f / 216.0f;
}
// 1/|c| by |c|^2 for the recolouring cos(theta)
__host__ __device__ constexpr float invlen(int c2) {
    return c2 == 1 ? 1.0f : c2 == 2 ? 0.70710678118654752f : c2 == 3 ? 0.57735026918962576f : 0.0f;
}

struct FaceBC {
    int kind;          // TSLB_BC_*
    float u[3];        // wall velocity
    float phi;         // colour of incoming populations (< -2: own phi); ghost phi on solid faces
    const float* plane;  // TSLB_BC_INLET: u, v, w, phi planes of the face
};

struct StepArgs {
    int nx, ny, nz;
    unsigned plane;         // nx ny
    long long N;            // field stride (elements)
    const void* in;         // 11 fields of the storage type
    void* out;              // 11 fields of the storage type
    float scale[NF];        // stored = value * scale (fp16 storage; 1 otherwise)
    float iscale[NF];       // value = stored * iscale
    const void* fi[NF];     // the fields of `in` and `out`
    void* fo[NF];
    const float* nrm;       // phase field: interface normals (3 fields of stride N)
    int zchunk;             // target planes per block; 0: `grid` blocks share the tiles' planes equally
    int grid;
    int warps;              // warps of a block (tslb_step.cuh: BIGW, SMALLW)
    int th;                 // target rows of a tile, at most warps - 2
    int xwrap;              // a warp holds the whole periodic x axis (nx <= 32)
    int phi_mirror;         // ghost phi is the nearest node's on every face that is not periodic
    int general;            // nodes without closed boundary sums: 0 none, 1 at single inlet or outlet faces
                            // normal to y or z (io_face), 2 others too (direction_from_behind)
    int mode;
    float omega_pf;         // 1/tau (phase field)
    float inv_nu_a, inv_nu_b;  // colour: 1/nu of each component
    float sigma, beta, sharp, thr, acoef;
    float force[3];
    int wall_phi_mode;
    FaceBC face[6];
    unsigned int* flags;    // bit 0: non-finite moment produced
    const float* dtau;      // colour: per-node correction of tau (stride N), or null
    const unsigned int* solid;  // interior solid nodes, one bit per node (bit i & 31 of word i >> 5), or null
    const unsigned int* near;   // fluid nodes with a solid one among their 26 neighbours, same layout
    int zt0, zt1;           // target planes [zt0, zt1) a step updates (a z slab: its own planes;
                            // the planes outside them are halo copies of the neighbours')
    int zoff;               // global index of local plane 0 (a z slab's offset; seeds the rounding)
    int sr;                 // 16-bit storage: store the moments with stochastic rounding
    unsigned int sr_step;   // step counter that seeds the rounding (with the node and the field)
    const unsigned int* sr_counter;  // ensembles: device step counter read instead of sr_step, or null
};

// Counter-based uniform in [0, 1) of four integers: the reference's
// rand_noseeded (TSLB_2C-mpi/vars_single_3D_module.f90:150-215), which seeds
// the two lagged generators of the Marsaglia-Zaman "universal" method from
// (i, j, k, l) in 24 rounds each and returns one output.  Every FP32 value
// is a multiple of 2^-24 in [-1, 2), so the arithmetic is exact and equal
// on the host, on the device and in the Fortran original.
__host__ __device__ inline float rand_noseeded(int i, int j, int k, int l) {
    int isub = i % 178 + 1, jsub = j % 178 + 1, ksub = k % 178 + 1, lsub = l % 169;
    float u[2];
    for (int g = 0; g < 2; ++g) {
        float s = 0.f, t = 0.5f;
        for (int jj = 0; jj < 24; ++jj) {
            const int msub = ((isub * jsub) % 179) * ksub % 179;
            isub = jsub;
            jsub = ksub;
            ksub = msub;
            lsub = (53 * lsub + 1) % 169;
            if ((lsub * msub) % 64 >= 32) s += t;
            t *= 0.5f;
        }
        u[g] = s;   // u97, then u33
    }
    float uni = u[0] - u[1];
    if (uni < 0.f) uni += 1.f;
    const float c = 362436.0f / 16777216.0f, cd = 7654321.0f / 16777216.0f, cm = 16777213.0f / 16777216.0f;
    float csub = c - cd;
    if (csub < 0.f) csub += cm;
    uni -= csub;
    if (uni < 0.f) uni += 1.f;
    return uni;
}

// bit i of a mask (set before any step that reads it is launched, so the read-only
// path is open to it, as to nothing else that a step reads)
__device__ __forceinline__ bool bit_at(const unsigned int* b, long long i) {
    return (__ldg(b + (i >> 5)) >> (i & 31)) & 1u;
}

// Storage types of the moment state: FP32, BF16 or FP16 (scaled).  All
// arithmetic is FP32; conversion happens on load and store.
template <class T>
struct Stor;
template <>
struct Stor<float> {
    static __device__ __forceinline__ float ld(float v) { return v; }
    static __device__ __forceinline__ float st(float v) { return v; }
};
template <>
struct Stor<__nv_bfloat16> {
    static __device__ __forceinline__ float ld(__nv_bfloat16 v) { return __bfloat162float(v); }
    static __device__ __forceinline__ __nv_bfloat16 st(float v) { return __float2bfloat16_rn(v); }
};
template <>
struct Stor<__half> {
    static __device__ __forceinline__ float ld(__half v) { return __half2float(v); }
    static __device__ __forceinline__ __half st(float v) { return __float2half_rn(v); }
};

__device__ __forceinline__ long long nidx(const StepArgs& a, int x, int y, int z) {
    return (long long)x + (long long)a.nx * ((long long)y + (long long)a.ny * z);
}
// periodic wrap of any coordinate into [0, n) (tiles may reach several periods out on tiny lattices)
__device__ __forceinline__ int wrapi(int c, int n) {
    if ((unsigned)c < (unsigned)n) return c;
    c %= n;
    return c < 0 ? c + n : c;
}
__device__ __forceinline__ int dimn(const StepArgs& a, int ax) { return ax == 0 ? a.nx : ax == 1 ? a.ny : a.nz; }

__device__ __forceinline__ long long plane_index(const StepArgs& a, int face, int x, int y, int z) {
    int ax = face >> 1;
    if (ax == 0) return (long long)y + (long long)a.ny * z;
    if (ax == 1) return (long long)x + (long long)a.nx * z;
    return (long long)x + (long long)a.nx * y;
}
__device__ __forceinline__ long long plane_area(const StepArgs& a, int face) {
    int ax = face >> 1;
    return ax == 0 ? (long long)a.ny * a.nz : ax == 1 ? (long long)a.nx * a.nz : (long long)a.nx * a.ny;
}

// phi at any node of the halo'd lattice: periodic axes wrap; on solid faces
// the inlet plane's phi (inlet faces), bc phi (wall_phi_mode 0) or the
// nearest fluid value (mirror).  The first out-of-range non-periodic axis in
// x, y, z order names the face.
// stored value -> FP32 value of field f (fp16 storage carries a per-field scale)
template <class T>
__device__ __forceinline__ float cvt_in(T v, const StepArgs& a, int f) {
    if constexpr (std::is_same<T, __half>::value) return Stor<T>::ld(v) * a.iscale[f];
    else return Stor<T>::ld(v);
}
template <class T>
__device__ __forceinline__ T cvt_out(float v, const StepArgs& a, int f) {
    if constexpr (std::is_same<T, __half>::value) return Stor<T>::st(v * a.scale[f]);
    else return Stor<T>::st(v);
}

// largest finite value of a 16-bit storage type (bf16: FP32's range)
template <class T>
struct Stor16Max;
template <>
struct Stor16Max<__half> {
    static constexpr float value = 65504.0f;
};
template <>
struct Stor16Max<__nv_bfloat16> {
    static constexpr float value = 3.3895313892515355e38f;
};
template <class T>
__device__ __forceinline__ T bits_as(unsigned short u);
template <>
__device__ __forceinline__ __half bits_as<__half>(unsigned short u) { return __ushort_as_half(u); }
template <>
__device__ __forceinline__ __nv_bfloat16 bits_as<__nv_bfloat16>(unsigned short u) { return __ushort_as_bfloat16(u); }

// Stochastic rounding of the 16-bit stored moments: a value rounds away from
// zero with the probability of its distance from the value toward zero, so
// the expected stored value is the FP32 one.  Rounding to nearest drops every
// change smaller than half a unit in the last place at every step - the body
// force of the channel adds about 2.5e-6 to u per step, 1/200 of a BF16 unit
// at u = 0.07 - and the stored flow stops following the forcing.  The step
// stores two fields with one stochastically rounded hardware conversion
// (cvt.rs.bf16x2.f32 / cvt.rs.f16x2.f32, sm_100a) whose random bits hash the
// node, the pair's first field and the step counter, so a run (and its
// restart from a checkpoint) is reproducible.
__device__ __forceinline__ unsigned int sr_node(unsigned int node, unsigned int step) {
    unsigned int h = node * 0x9E3779B1u ^ (step * 0x85EBCA77u + 0x165667B1u);
    h ^= h >> 15;
    h *= 0x2C1B3C6Du;
    h ^= h >> 12;
    return h;
}
__device__ __forceinline__ unsigned int sr_field(unsigned int hnode, int f) {
    unsigned int h = (hnode + (unsigned int)f * 0x9E3779B9u) * 0x85EBCA6Bu;
    return h ^ (h >> 16);
}
// the larger of two numbers, NaN if either is one (fmaxf drops a NaN)
__device__ __forceinline__ float max_nan(float x, float y) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
    return r;
}
// Store fields f and g (g == f: f alone) of node id in 16-bit storage with
// one paired conversion: cvt.rn / cvt.rs (stochastic, random bits r) to
// f16x2 or bf16x2 of the stored values (fp16: value * per-field scale).
// Returns the largest stored magnitude before rounding (NaN if either is), for
// the range check.
template <class T>
__device__ __forceinline__ float store_pair16(const StepArgs& a, unsigned int id, int f, int g, float vf, float vg, int sr,
                                              unsigned int r) {
    constexpr bool H = std::is_same<T, __half>::value;
    const float xf = H ? vf * a.scale[f] : vf, xg = H ? vg * a.scale[g] : vg;
    unsigned int d;
    if (sr) {
        if (H) asm("cvt.rs.f16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(xg), "f"(xf), "r"(r));
        else asm("cvt.rs.bf16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(xg), "f"(xf), "r"(r));
    } else {
        if (H) asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(xg), "f"(xf));
        else asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(xg), "f"(xf));
    }
    // the low half holds field f, the high half field g
    static_cast<T*>(a.fo[f])[id] = bits_as<T>((unsigned short)(d & 0xFFFFu));
    if (g != f) static_cast<T*>(a.fo[g])[id] = bits_as<T>((unsigned short)(d >> 16));
    return max_nan(fabsf(xf), fabsf(xg));
}

template <class T>
__device__ __forceinline__ float ld_field(const StepArgs& a, int f, long long idx) {
    return cvt_in<T>(reinterpret_cast<const T*>(a.in)[f * a.N + idx], a, f);
}

template <class T>
__device__ float phi_at(const StepArgs& a, int x, int y, int z) {
    int c[3] = {x, y, z};
    int face = -1;
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
        int n = dimn(a, ax);
        if (c[ax] < 0 || c[ax] >= n) {
            if (a.face[2 * ax].kind == TSLB_BC_PERIODIC) {
                c[ax] = wrapi(c[ax], n);
            } else {
                if (face < 0) face = 2 * ax + (c[ax] >= n ? 1 : 0);
                c[ax] = c[ax] < 0 ? 0 : n - 1;
            }
        }
    }
    if (face < 0) return ld_field<T>(a, F_PHI, nidx(a, c[0], c[1], c[2]));
    const FaceBC& fb = a.face[face];
    if (fb.kind == TSLB_BC_INLET) return fb.plane[3 * plane_area(a, face) + plane_index(a, face, c[0], c[1], c[2])];
    if (a.wall_phi_mode == 0) return fb.phi;
    return ld_field<T>(a, F_PHI, nidx(a, c[0], c[1], c[2]));
}

__device__ __forceinline__ bool interior1(const StepArgs& a, int x, int y, int z) {
    return x >= 1 && x < a.nx - 1 && y >= 1 && y < a.ny - 1 && z >= 1 && z < a.nz - 1;
}

// isotropic gradient 3 sum_i p_i c_i s(x+c_i) of phi
// (recursive_2c_TSLB3D.f90:555-565; recursive_colorTSLB3D.f90:726-744)
template <class T>
__device__ void grad_phi(const StepArgs& a, int x, int y, int z, float g[3]) {
    float gx = 0.f, gy = 0.f, gz = 0.f;
    const bool fast = interior1(a, x, y, z);
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                if (dx == 0 && dy == 0 && dz == 0) continue;
                const float wv = wclass(dx * dx + dy * dy + dz * dz);
                float s = fast ? ld_field<T>(a, F_PHI, nidx(a, x + dx, y + dy, z + dz)) : phi_at<T>(a, x + dx, y + dy, z + dz);
                s *= wv;
                if (dx) gx += dx > 0 ? s : -s;
                if (dy) gy += dy > 0 ? s : -s;
                if (dz) gz += dz > 0 ? s : -s;
            }
    g[0] = 3.f * gx;
    g[1] = 3.f * gy;
    g[2] = 3.f * gz;
}

// Arithmetic of the step, one operation at a time.  The step computes a
// node's coefficients in every tile that holds it, as a target node of one
// tile and as a source on the rim of its neighbours.  The populations it
// sends into different tiles must be the same numbers, or mass is not
// conserved exactly, so no operation is left for the compiler to contract:
// Ar1 evaluates one number in FP32, Ar2 two at once on the paired FP32
// instructions of sm_100.
struct Ar1 {
    using V = float;
    static __device__ __forceinline__ V c(float x) { return x; }
    static __device__ __forceinline__ V add(V x, V y) { return __fadd_rn(x, y); }
    static __device__ __forceinline__ V sub(V x, V y) { return __fsub_rn(x, y); }
    static __device__ __forceinline__ V mul(V x, V y) { return __fmul_rn(x, y); }
    static __device__ __forceinline__ V fma(V x, V y, V z) { return __fmaf_rn(x, y, z); }
    // lane-wise functions (square root, division, selection)
    template <class F>
    static __device__ __forceinline__ V map(V x, F f) { return f(x); }
    template <class F>
    static __device__ __forceinline__ V map2(V x, V y, F f) { return f(x, y); }
};
struct Ar2 {
    using V = float2;
    static __device__ __forceinline__ V c(float x) { return make_float2(x, x); }
    static __device__ __forceinline__ V add(V x, V y) { return __fadd2_rn(x, y); }
    static __device__ __forceinline__ V sub(V x, V y) { return __fadd2_rn(x, make_float2(-y.x, -y.y)); }
    static __device__ __forceinline__ V mul(V x, V y) { return __fmul2_rn(x, y); }
    static __device__ __forceinline__ V fma(V x, V y, V z) { return __ffma2_rn(x, y, z); }
    template <class F>
    static __device__ __forceinline__ V map(V x, F f) { return make_float2(f(x.x), f(x.y)); }
    template <class F>
    static __device__ __forceinline__ V map2(V x, V y, F f) { return make_float2(f(x.x, y.x), f(x.y, y.y)); }
};

// Coefficients of P'(c) = f_c / w_c - 1 of a node.  With r = 4.5 rho
// and o = 4.5 (1 - omega) the second-order coefficients are
//   K_ab = (2 - delta_ab) (r u_a u_b + o Pi_ab),
// and the third-order ones, 13.5 (rho u_a u_a u_b + (1 - omega) a3_aab) with
// the recursive a3_aab = u_b Pi_aa + 2 u_a Pi_ab, come from them:
//   K_aab = 3 u_b K_aa + 3 u_a (2 o Pi_ab).
// m[] are the node's moments (m[F_D] = rho - 1).

// Colour mode: g is the gradient of phi, m[F_PHI] phi; TAU: the relaxation
// time is tau(phi) + dt (a local eddy-viscosity correction; the
// surface-tension coefficient follows the corrected omega).  Returns whether
// any node of the warp lies on the interface; if none does, the recolouring
// terms K_C1..K_C3 are 0 in the whole warp.
template <bool TAU>
__device__ __forceinline__ bool coefs_colour(const StepArgs& a, const float* m, const float* g, float dt, float* K) {
    using A = Ar1;
    using V = A::V;
    auto c = [](float x) { return A::c(x); };
    const V d = m[F_D], u = m[F_U], v = m[F_V], w = m[F_W], phi = m[F_PHI];
    // 1/nu = (rhoA/rho)/nu_a + (rhoB/rho)/nu_b ; omega = 2/(6 nu + 1) = 2q/(6 + q)
    const float qa = 0.5f * (a.inv_nu_a + a.inv_nu_b), qd = 0.5f * (a.inv_nu_a - a.inv_nu_b);
    const V q = A::fma(phi, c(qd), c(qa)), q2 = A::add(q, q);
    // TAU: 1/omega = (6 + q)/(2q) + dtau
    const V den = TAU ? A::fma(q2, dt, A::add(q, c(6.f))) : A::add(q, c(6.f));
    const V omega = A::map2(q2, den, [](float n, float e) { return __fdividef(n, e); });
    const V rho = A::add(c(1.f), d), om1 = A::sub(c(1.f), omega);
    const V o = A::mul(om1, c(4.5f)), o2 = A::add(o, o), r = A::mul(rho, c(4.5f));
    const V ru = A::mul(r, u), rv = A::mul(r, v), rw = A::mul(r, w), ru2 = A::add(ru, ru), rv2 = A::add(rv, rv);
    const V xx = A::fma(o, m[F_XX], A::mul(ru, u)), yy = A::fma(o, m[F_YY], A::mul(rv, v)), zz = A::fma(o, m[F_ZZ], A::mul(rw, w));
    const V pxy = A::mul(o2, m[F_XY]), pxz = A::mul(o2, m[F_XZ]), pyz = A::mul(o2, m[F_YZ]);
    const V xy = A::fma(ru2, v, pxy), xz = A::fma(ru2, w, pxz), yz = A::fma(rv2, w, pyz);
    const V u3 = A::mul(u, c(3.f)), v3 = A::mul(v, c(3.f)), w3 = A::mul(w, c(3.f));
    K[K_XXY] = A::fma(v3, xx, A::mul(u3, pxy));
    K[K_XXZ] = A::fma(w3, xx, A::mul(u3, pxz));
    K[K_XYY] = A::fma(u3, yy, A::mul(v3, pxy));
    K[K_YYZ] = A::fma(w3, yy, A::mul(v3, pyz));
    K[K_XZZ] = A::fma(u3, zz, A::mul(w3, pxz));
    K[K_YZZ] = A::fma(v3, zz, A::mul(w3, pyz));
    K[K_XYZ] = A::fma(u3, yz, A::fma(v3, pxz, A::mul(w3, pxy)));
    // K_a = 3 rho u_a - (K_abb + K_acc)/3, with the force as population source
    // 3 w c.F (recursive_colorTSLB3D.f90:776)
    const V mt = c(-1.f / 3.f), tt = c(2.f / 3.f);
    K[K_X] = A::fma(mt, A::add(K[K_XYY], K[K_XZZ]), A::fma(tt, ru, c(3.f * a.force[0])));
    K[K_Y] = A::fma(mt, A::add(K[K_XXY], K[K_YZZ]), A::fma(tt, rv, c(3.f * a.force[1])));
    K[K_Z] = A::fma(mt, A::add(K[K_XXZ], K[K_YYZ]), A::fma(tt, rw, c(3.f * a.force[2])));
    K[K_0] = A::fma(mt, A::add(A::add(xx, yy), zz), d);
    K[K_XX] = xx; K[K_YY] = yy; K[K_ZZ] = zz; K[K_XY] = xy; K[K_XZ] = xz; K[K_YZ] = yz;
    K[K_C0] = phi; K[K_C1] = K[K_C2] = K[K_C3] = K[K_C4] = c(0.f);
    const V m2 = A::fma(g[2], g[2], A::fma(g[1], g[1], A::mul(g[0], g[0])));
    const float thr2 = a.thr * a.thr;
    const bool iface = __any_sync(0xffffffffu, m2 > thr2);
    if (iface) {
        const V rs = A::map(m2, [](float x) { return rsqrtf(x); });
        // outside the interface (|g|^2 <= thr^2) |g| and n are 0
        const V mg = A::map2(m2, rs, [thr2](float x, float y) { return x > thr2 ? __fmul_rn(x, y) : 0.f; });
        const V inv = A::map2(m2, rs, [thr2](float x, float y) { return x > thr2 ? y : 0.f; });
        const V nx = A::mul(g[0], inv), ny = A::mul(g[1], inv), nz = A::mul(g[2], inv);
        // perturbation (A/2)|g| [w (c.n)^2 - B_i], B_i = w_i for i >= 1
        const V Am = A::mul(A::mul(c(a.acoef * a.sigma), omega), mg);
        const V h = A::mul(c(0.5f), Am), h2 = Am;
        const V hx = A::mul(h, nx), hy = A::mul(h, ny), hz = A::mul(h, nz), hx2 = A::mul(h2, nx), hy2 = A::mul(h2, ny);
        K[K_0] = A::sub(K[K_0], h);
        K[K_XX] = A::fma(hx, nx, xx);
        K[K_YY] = A::fma(hy, ny, yy);
        K[K_ZZ] = A::fma(hz, nz, zz);
        K[K_XY] = A::fma(hx2, ny, xy);
        K[K_XZ] = A::fma(hx2, nz, xz);
        K[K_YZ] = A::fma(hy2, nz, yz);
        // rest population: B_0 = -10/27 instead of w_0
        K[K_C4] = A::mul(Am, c(1.f / 3.f));
        // recolouring 2 beta (rhoA rhoB / rho) n  (published form, cos theta)
        const V bb = A::mul(A::mul(c(0.5f * a.beta), rho), A::fma(A::mul(c(-1.f), phi), phi, c(1.f)));
        K[K_C1] = A::mul(bb, nx); K[K_C2] = A::mul(bb, ny); K[K_C3] = A::mul(bb, nz);
    }
    return iface;
}

// Coefficients K_0 .. K_XYZ with the equilibrium at (1 + d, U) and the
// non-equilibrium part of the node's u and Pi: f^eq(1 + d, U) + om1 w a^neq(Pi, u).
__device__ __forceinline__ void coefs_moments(float d, const float* m, float U, float Vv, float W, float om1, float* K) {
    using A = Ar1;
    using V = float;
    auto c = [](float x) { return A::c(x); };
    const V u = m[F_U], v = m[F_V], w = m[F_W];
    const V rho = A::add(c(1.f), d);
    const V o = A::mul(c(4.5f), om1), o2 = A::add(o, o), r = A::mul(rho, c(4.5f));
    const V ru = A::mul(r, U), rv = A::mul(r, Vv), rw = A::mul(r, W), ru2 = A::add(ru, ru), rv2 = A::add(rv, rv);
    // equilibrium (e) and non-equilibrium (p) parts of the second order
    const V exx = A::mul(ru, U), eyy = A::mul(rv, Vv), ezz = A::mul(rw, W);
    const V pxx = A::mul(o, m[F_XX]), pyy = A::mul(o, m[F_YY]), pzz = A::mul(o, m[F_ZZ]);
    const V pxy = A::mul(o2, m[F_XY]), pxz = A::mul(o2, m[F_XZ]), pyz = A::mul(o2, m[F_YZ]);
    const V eyz = A::mul(rv2, W);
    K[K_XX] = A::add(exx, pxx); K[K_YY] = A::add(eyy, pyy); K[K_ZZ] = A::add(ezz, pzz);
    K[K_XY] = A::fma(ru2, Vv, pxy); K[K_XZ] = A::fma(ru2, W, pxz); K[K_YZ] = A::add(eyz, pyz);
    const V u3 = A::mul(u, c(3.f)), v3 = A::mul(v, c(3.f)), w3 = A::mul(w, c(3.f));
    const V U3 = A::mul(U, c(3.f)), V3 = A::mul(Vv, c(3.f)), W3 = A::mul(W, c(3.f));
    K[K_XXY] = A::fma(V3, exx, A::fma(v3, pxx, A::mul(u3, pxy)));
    K[K_XXZ] = A::fma(W3, exx, A::fma(w3, pxx, A::mul(u3, pxz)));
    K[K_XYY] = A::fma(U3, eyy, A::fma(u3, pyy, A::mul(v3, pxy)));
    K[K_YYZ] = A::fma(W3, eyy, A::fma(w3, pyy, A::mul(v3, pyz)));
    K[K_XZZ] = A::fma(U3, ezz, A::fma(u3, pzz, A::mul(w3, pxz)));
    K[K_YZZ] = A::fma(V3, ezz, A::fma(v3, pzz, A::mul(w3, pyz)));
    K[K_XYZ] = A::fma(U3, eyz, A::fma(u3, pyz, A::fma(v3, pxz, A::mul(w3, pxy))));
    const V mt = c(-1.f / 3.f), tt = c(2.f / 3.f);
    K[K_X] = A::fma(mt, A::add(K[K_XYY], K[K_XZZ]), A::mul(tt, ru));
    K[K_Y] = A::fma(mt, A::add(K[K_XXY], K[K_YZZ]), A::mul(tt, rv));
    K[K_Z] = A::fma(mt, A::add(K[K_XXZ], K[K_YYZ]), A::mul(tt, rw));
    K[K_0] = A::fma(mt, A::add(A::add(K[K_XX], K[K_YY]), K[K_ZZ]), d);
}

// Phase field (PHASE: the equilibrium at the CSF-shifted velocity
// u + sigma kappa n (+ F), recursive_2c_TSLB3D.f90:630-636,
// lb_kernels_module.f90:769; n the interface normal, curv the curvature
// -div n where the interface indicator exceeds 0.2, else 0) and single
// component (fused_TSLB_force_1c: at u + F).
template <bool PHASE>
__device__ __forceinline__ void coefs_shifted(const StepArgs& a, const float* m, const float* n, float curv, float* K) {
    using A = Ar1;
    using V = float;
    auto c = [](float x) { return A::c(x); };
    const V u = m[F_U], v = m[F_V], w = m[F_W];
    V U = A::add(u, c(a.force[0])), Vv = A::add(v, c(a.force[1])), W = A::add(w, c(a.force[2]));
    if (PHASE) {
        const V sk = A::mul(c(a.sigma), curv);
        U = A::fma(sk, n[0], U); Vv = A::fma(sk, n[1], Vv); W = A::fma(sk, n[2], W);
    }
    coefs_moments(m[F_D], m, U, Vv, W, 1.f - a.omega_pf, K);
    K[K_C0] = K[K_C1] = K[K_C2] = K[K_C3] = K[K_C4] = c(0.f);
    if (PHASE) {
        // D3Q7 phase field: g_q = G0 + e_q.G1 (recursive_2c_TSLB3D.f90:808-831)
        const V phi = m[F_PHI];
        const V sh = A::mul(A::mul(c(0.125f * a.sharp), phi), A::sub(c(1.f), phi)), p3 = A::mul(c(0.375f), phi);
        K[K_C0] = A::mul(c(0.125f), phi);
        K[K_C1] = A::fma(sh, n[0], A::mul(p3, u));
        K[K_C2] = A::fma(sh, n[1], A::mul(p3, v));
        K[K_C3] = A::fma(sh, n[2], A::mul(p3, w));
    }
}

// P'(c) for a runtime direction (boundary paths)
__device__ __forceinline__ float eval_P(const float* K, long long stride, int cx, int cy, int cz) {
    const float fx = (float)cx, fy = (float)cy, fz = (float)cz;
    const float ax = (float)(cx * cx), ay = (float)(cy * cy), az = (float)(cz * cz);
    return K[K_0 * stride] + fx * K[K_X * stride] + fy * K[K_Y * stride] + fz * K[K_Z * stride] +
           ax * K[K_XX * stride] + ay * K[K_YY * stride] + az * K[K_ZZ * stride] +
           fx * fy * K[K_XY * stride] + fx * fz * K[K_XZ * stride] + fy * fz * K[K_YZ * stride] +
           ax * fy * K[K_XXY * stride] + ax * fz * K[K_XXZ * stride] + fx * ay * K[K_XYY * stride] +
           ay * fz * K[K_YYZ * stride] + fx * az * K[K_XZZ * stride] + fy * az * K[K_YZZ * stride] +
           fx * fy * fz * K[K_XYZ * stride];
}

// accumulate population value f (already weighted) of direction c into acc
template <class Acc>
__device__ __forceinline__ void acc_dir_rt(Acc&& acc, int cx, int cy, int cz, float f) {
    acc[A_RHO] += f;
    acc[A_JX] += cx * f; acc[A_JY] += cy * f; acc[A_JZ] += cz * f;
    acc[A_XX] += (cx * cx) * f; acc[A_YY] += (cy * cy) * f; acc[A_ZZ] += (cz * cz) * f;
    acc[A_XY] += (cx * cy) * f; acc[A_XZ] += (cx * cz) * f; acc[A_YZ] += (cy * cz) * f;
}

}  // namespace tslb
