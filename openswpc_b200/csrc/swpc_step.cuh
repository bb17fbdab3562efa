// swpc_step.cuh -- what a staged stress or velocity launch also does inside a
// time step: the point sources of its cells, the recorder, the step counter,
// and programmatic dependent launch.
//
// A step of a small grid is bound by its launches: source injection, the
// recorder and the counter took 2.4, 2.8 and 1.5 us a step beside 10.7 us of
// the two updates on a 40 x 36 x 32 grid (2.0, 3.2 and 1.6 us beside 9.6 us on
// a 256 x 128 P-SV model).  Here the thread that updates a cell adds the
// sources of that cell, the recorder takes a few CTAs of the stress launch
// (it reads the velocity, which that launch leaves alone), and the counter
// moves with the velocity launch.
#pragma once

#include <cuda_runtime.h>

#include <utility>

#include "swpc_kernels.cuh"

namespace swpc {

// Dependent launches: wait for the launch before this one to complete and its
// stores to be visible; let the next one start its prologue.  The trigger
// comes after the wait, so a prologue may read what launches before its
// predecessor wrote (setup data), and only when every CTA of the predecessor
// is resident.
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void pdl_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

template <typename... P, typename... A>
cudaError_t launch_pdl(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// The sources of cell `cell`, whose column's entries start at n: the
// expressions and the list order of inject_kernel (the thread has just stored
// the cell's values and reads them back).  The entries of a column stand in
// the order of their cells, and the thread looks its cell up by halving: a
// column of a finite fault holds hundreds of entries, and walking them one
// after another held its tiles back (96 x 96 x 160 cells with 40 subfaults in
// a column 171 us a step, by halving 88, and 89 with the subfaults apart; P-SV
// 512 x 256 with 60 in a column 59.8 and 11.0 us).
static __device__ __noinline__ void inject_cell(const StepInj &s, int it, int n, long long cell) {
    if (it < 1 || it > s.nt) return;
    const int end = n + s.list[n].rest;
    for (int hi = end; n < hi;) {
        const int mid = (n + hi) >> 1;
        if (s.list[mid].cell < cell) n = mid + 1;
        else hi = mid;
    }
    for (; n < end; n++) {
        const InjCell en = s.list[n];
        if (en.cell != cell) return;
        const float st = s.stime[(long long)(it - 1) * s.nsrc + en.src];
        const float f = *en.p;
        switch (en.mode) {
        case INJ_GLUT: *en.p = f - en.coef * (s.mo[en.src] * st * s.dt_dxyz); break;
        case INJ_GLUT4: *en.p = f - en.coef * (s.mo[en.src] * st * s.dt_dxyz) / 4; break;
        case INJ_GLUT2: *en.p = f - en.coef * (s.mo[en.src] * st * s.dt_dxyz) / 2; break;
        case INJ_BF3: *en.p = f + *en.b * en.coef * st * s.dt_dxyz / 2; break;
        case INJ_GREEN: *en.p = f + *en.b * (en.coef * s.dt_dxyz * st) / 2; break;
        default: break;
        }
    }
}

}  // namespace swpc
