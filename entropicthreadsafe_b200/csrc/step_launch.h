// step_launch.h -- host-side launchers of the step and ensemble kernels,
// whose instantiations live in translation units of their own (k_scalar.cu,
// k_inlet.cu, k_general.cu) that compile in parallel with the rest.  Every launcher with launch =
// false only sets the kernel's shared-memory attribute (before a stream
// capture, for instance).
#pragma once
#include <cuda_runtime.h>

#include <type_traits>

#include "tslb_step.cuh"

namespace tslb_launch {

// tiles of a lattice
inline int tiles_x(const tslb::StepArgs& a) { return a.xwrap ? 1 : (a.nx + tslb::LXV - 1) / tslb::LXV; }
inline int tiles_y(const tslb::StepArgs& a) { return (a.ny + a.th - 1) / a.th; }

// set the dynamic shared-memory limit of kernel fn once per device (tslb.cu)
cudaError_t ensure_smem_attr(const void* fn, size_t bytes);

// One kernel launch; its error is left to cudaGetLastError.
// early: the kernel may be launched while the one before it on the stream
// runs, for which it waits on the device (its launch and index set-up then
// cost nothing: colour steps of 24^3 nodes 10.2 us apart without and 8.5 with,
// of 64^3 24.2 and 20.7, of 173 x 59 x 91 49.6 and 46.9, of the 384 x 192 x 128
// channel 333 and 331; 20 phase-field steps of 101 x 64 x 47 with diagnostics and a
// print stamp 2116 us before the diagnostics did so too, 2047 since).
// Never in a stream capture, where the graph keeps the plain order.
template <class... P, class... A>
void launch_after(void (*kernel)(P...), unsigned grid, dim3 block, size_t smem, cudaStream_t st, bool early, A... args) {
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (early && cudaStreamIsCapturing(st, &cap) != cudaSuccess) cudaGetLastError();   // the launch reports it
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = early && cap == cudaStreamCaptureStatusNone ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

// step kernel (tslb_step.cuh): every storage type, tau correction and
// interior solid mask (early: see launch_after)
cudaError_t scalar_step(const tslb::StepArgs& a, int mode, int prec, cudaStream_t st, bool launch, bool early = false);
// general: the largest StepArgs::general of the members
cudaError_t scalar_ensemble(const tslb::StepArgs* args, const tslb::WorkItem* work, int nwork, int grid, int mode, int prec,
                            int general, unsigned int* step, cudaStream_t st, bool launch);

}  // namespace tslb_launch
