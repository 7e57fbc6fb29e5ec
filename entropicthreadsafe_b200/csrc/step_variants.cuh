// step_variants.cuh -- the step kernel (tslb_step.cuh) in every variant: storage
// type, warps of a block, per-node tau correction, interior solid mask; and its
// ensemble form, for one value of GEN (a translation unit each, to compile side by
// side: k_scalar.cu, k_inlet.cu, k_general.cu).
#pragma once
#include "step_launch.h"

namespace tslb_launch {

namespace {
template <class Fn>
void with_storage(int prec, Fn&& fn) {
    if (prec == TSLB_PREC_BF16) fn(__nv_bfloat16{});
    else if (prec == TSLB_PREC_FP16S) fn(__half{});
    else fn(float{});
}
}  // namespace

template <int GEN>
cudaError_t step_variants(const tslb::StepArgs& a, int mode, int prec, cudaStream_t st, bool launch, bool early) {
    using namespace tslb;
    const unsigned grid = a.zchunk > 0 ? (unsigned)(tiles_x(a) * tiles_y(a) * ((a.zt1 - a.zt0 + a.zchunk - 1) / a.zchunk)) : (unsigned)a.grid;
    cudaError_t err = cudaSuccess;
    auto with_warps = [&](auto warps) {
        constexpr int W = decltype(warps)::value;
        auto go = [&](void (*kernel)(const StepArgs), int sm) {
            err = ensure_smem_attr((const void*)kernel, sm);
            if (err == cudaSuccess && launch) launch_after(kernel, grid, dim3(32, W, 1), sm, st, early, a);
        };
        constexpr int C = TSLB_MODE_COLOUR, P = TSLB_MODE_PHASEFIELD, S = TSLB_MODE_SINGLE;
        with_storage(prec, [&](auto tag) {
            using T = decltype(tag);
            if (a.solid && std::is_same<T, float>::value) {
                // interior solid nodes (FP32 storage, no tau correction; checked by tslb_set_solid_mask)
                if (mode == C) go(step_kernel<C, float, W, false, true, GEN>, Smem<C, W>::bytes);
                else if (mode == S) go(step_kernel<S, float, W, false, true, GEN>, Smem<S, W>::bytes);
                else go(step_kernel<P, float, W, false, true, GEN>, Smem<P, W>::bytes);
            } else if (mode == C && a.dtau && std::is_same<T, float>::value) {
                // per-node tau correction (FP32 storage only; checked by the callers)
                go(step_kernel<C, float, W, true, false, GEN>, Smem<C, W>::bytes);
            } else if (mode == C) {
                go(step_kernel<C, T, W, false, false, GEN>, Smem<C, W>::bytes);
            } else if (mode == S) {
                go(step_kernel<S, T, W, false, false, GEN>, Smem<S, W>::bytes);
            } else {
                go(step_kernel<P, T, W, false, false, GEN>, Smem<P, W>::bytes);
            }
        });
    };
    if (a.warps == SMALLW) with_warps(std::integral_constant<int, SMALLW>{});
    else with_warps(std::integral_constant<int, BIGW>{});
    return err;
}

template <int GEN>
cudaError_t ensemble_variants(const tslb::StepArgs* args, const tslb::WorkItem* work, int nwork, int grid, int mode,
                              int prec, unsigned int* step, cudaStream_t st, bool launch) {
    using namespace tslb;
    cudaError_t err = cudaSuccess;
    with_storage(prec, [&](auto tag) {
        using T = decltype(tag);
        auto go = [&](void (*kernel)(const StepArgs*, const WorkItem*, int, unsigned int*), int sm) {
            err = ensure_smem_attr((const void*)kernel, sm);
            if (err == cudaSuccess && launch) kernel<<<grid, dim3(32, SMALLW, 1), sm, st>>>(args, work, nwork, step);
        };
        if (mode == TSLB_MODE_COLOUR) go(ensemble_kernel<TSLB_MODE_COLOUR, T, GEN>, Smem<TSLB_MODE_COLOUR, SMALLW>::bytes);
        else go(ensemble_kernel<TSLB_MODE_PHASEFIELD, T, GEN>, Smem<TSLB_MODE_PHASEFIELD, SMALLW>::bytes);
    });
    return err;
}

}  // namespace tslb_launch
