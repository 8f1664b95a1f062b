// finalize.cuh -- the end of a step: by the last CTA of stage 3 (step_end), by
// the ensemble's kernel for all members, or after a standalone CFL pass.
#pragma once
#include "../../include/mhd3d.h"
#include "mhd3d_dev.cuh"

namespace mhd3d {

// End of a step (advance=1: NIT, TIMC, TIMT of STEP 3dmhdsub.f:1171-1173 and
// the driver's DT check 3dmhd.f:924) and DT/UMACH of the next step from the
// CFL accumulators (DT=SF*MIN(...), 3dmhdsub.f:866-873; UMACH=SQRT(...), 761).
// The accumulators are read past L1 (other CTAs' atomics wrote them).
__device__ __forceinline__ void finalize_one(Control* ctl, Accum* acc, double sf, double dtmin, int lmag, int advance,
                                             unsigned long long w4key)
{
    if (advance) {
        if (ctl->stop) return;
        ctl->timc = ctl->timc + ctl->dt;
        ctl->timt = ctl->timi + ctl->timc;
        ctl->nit += 1;
        ctl->last_dt = ctl->dt;
        ctl->last_umach = ctl->umach;
        if (!(ctl->dt >= dtmin)) {
            ctl->stop = 1;
            ctl->status = isfinite(ctl->dt) ? MHD3D_ERR_DT_SMALL : MHD3D_ERR_NONFINITE;
        }
    }
    double w = of_key(__ldcg(&acc->wmin[0]));
    const double w2 = of_key(__ldcg(&acc->wmin[1])), w3 = of_key(__ldcg(&acc->wmin[2]));
    const double w4 = of_key(__ldcg(&acc->wmin[3]));
    w = w2 < w ? w2 : w;
    w = w3 < w ? w3 : w;
    if (lmag) w = w4 < w ? w4 : w;
    ctl->dt = sf * w;
    ctl->umach = sqrt(of_key(__ldcg(&acc->umax)));
    if (__ldcg(&acc->bad) && !ctl->stop) {
        ctl->stop = 1;
        ctl->status = MHD3D_ERR_NONFINITE;
    }
    for (int i = 0; i < 3; ++i) acc->wmin[i] = ~0ull;
    acc->wmin[3] = w4key;
    acc->umax = 0ull;
    acc->bad = 0u;
    acc->done = 0u;
}

// Called by one thread of every stage-3 CTA after its atomics: the last CTA
// ends the step, so no kernel of one thread has to be launched behind stage 3
// (3 us a step).  CTAs that return early (stop flag, a wait that gave up) are
// not counted, and the step is then not ended.
template <typename Args>
__device__ __forceinline__ void step_end(const Args& a)
{
    if (!a.end_step) return;
    __threadfence();
    if (atomicAdd(&a.acc->done, 1u) == gridDim.x * gridDim.y - 1u) {
        __threadfence();
        finalize_one(a.ctl, a.acc, a.s.sf, a.s.dtmin, a.s.lmag, 1, a.w4key);
    }
}

// Programmatic dependent launch: a stage is launched while the one before it
// drains and waits here for all of its memory.  The stage before does not ask
// for it early (launch_dependents): CTAs that came in beside a running stage
// made a step at 96x96x64 (reference rounding) 191 us long, without them it
// takes 168 us, with plain launches 175; 64x64x48 61 us against 67, 66 early;
// in FP32 51 against 57.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// launch of a stage kernel that calls grid_wait
template <typename K, typename A>
inline cudaError_t launch_chained(K kernel, dim3 grid, int threads, size_t smem, cudaStream_t st, const A& a)
{
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, a);
}

}  // namespace mhd3d
