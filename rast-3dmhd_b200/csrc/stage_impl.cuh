// stage_impl.cuh -- the fused FP64 RK3 stage kernel (RHS + update + BCON +
// ghost-plane toggle + CFL reduction) and the standalone CFL/BCON kernels.
//
// Included twice: by stage_exact.cu (compiled with -fmad=false, so every
// product and sum is rounded separately, as gfortran -O2 evaluates the
// reference; the stage kernel of stage_exact.cuh) and by stage_fast.cu (FMA
// contraction allowed; the column march of stage_march.cuh).  MHD3D_NS names
// the namespace of each copy.
//
// Work decomposition of both: a CTA owns a TX x TY tile of (x,y) columns and
// a chunk of z planes and marches down the chunk.  The raw fields of each
// plane arrive by TMA (cp.async.bulk.tensor, one 4-D box per plane: x with
// the periodic halo, y with the halo, one plane, all fields) into a ring of four
// slots (five in the march's stages without Z); 1/RO of the planes in use sits
// in a ring next to it.  Velocities and
// pressure are formed where they are used, from the same two operands
// FLUXES multiplies (3dmhdsub.f:1386-1425).  The Z tile of the plane (stages
// 2, 3) arrives by its own TMA box a plane ahead.  The wall planes take BCON
// (2751-2955) in the same pass: the thread owning a column finalises them
// from values it wrote itself.  No TMA load uses cluster multicast.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <cfloat>

#include "../../include/mhd3d.h"
#include "mhd3d_dev.cuh"
#include "smem_attr.cuh"
#include "cfl_cell.cuh"
#include "finalize.cuh"
#include "ring.cuh"
#if MHD3D_FAST_BODY
#include "march.cuh"
#endif

namespace mhd3d {
namespace MHD3D_NS {

#ifndef MHD3D_NRAW
#define MHD3D_NRAW 4
#endif
// raw-plane ring slots
constexpr int NRAW = MHD3D_NRAW;
static_assert(NRAW >= 3 && NRAW <= 6, "three to six ring slots");

// store a cell of U and the periodic halo copies COMMUNICATE would make of it
__device__ __forceinline__ void store_u(double* __restrict__ u, size_t fofs, const StageArgs& a, int gi, int gj,
                                        int kz, double v)
{
    const int npx = a.s.npx, npy = a.s.npy;
    const size_t base = fofs + (size_t)kz * a.uz;
    const int ix = gi + 1, jy = gj + 1;
    u[base + (size_t)jy * a.upitch + ix] = v;
    const int hx = (gi == 0) ? npx + 1 : (gi == npx - 1) ? 0 : -1;
    const int hy = (gj == 0) ? npy + 1 : (gj == npy - 1) ? 0 : -1;
    if (hx >= 0) u[base + (size_t)jy * a.upitch + hx] = v;
    if (hy >= 0) u[base + (size_t)hy * a.upitch + ix] = v;
    if (hx >= 0 && hy >= 0) u[base + (size_t)hy * a.upitch + hx] = v;
}

#include "cfl_acc.cuh"

// Block-wide reduction of the CFL parts into the global accumulators.
__device__ __forceinline__ void cfl_commit(Accum* acc, unsigned long long k1, unsigned long long k2,
                                           unsigned long long k3, unsigned long long k4, unsigned long long km,
                                           unsigned int bad, unsigned long long* red)
{
    for (int o = 16; o > 0; o >>= 1) {
        k1 = min(k1, __shfl_xor_sync(0xffffffffu, k1, o));
        k2 = min(k2, __shfl_xor_sync(0xffffffffu, k2, o));
        k3 = min(k3, __shfl_xor_sync(0xffffffffu, k3, o));
        k4 = min(k4, __shfl_xor_sync(0xffffffffu, k4, o));
        km = max(km, __shfl_xor_sync(0xffffffffu, km, o));
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) {
        red[w * 6 + 0] = k1;
        red[w * 6 + 1] = k2;
        red[w * 6 + 2] = k3;
        red[w * 6 + 3] = k4;
        red[w * 6 + 4] = km;
        red[w * 6 + 5] = bad;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < NT / 32; ++i) {
            k1 = min(k1, red[i * 6 + 0]);
            k2 = min(k2, red[i * 6 + 1]);
            k3 = min(k3, red[i * 6 + 2]);
            k4 = min(k4, red[i * 6 + 3]);
            km = max(km, red[i * 6 + 4]);
            bad |= (unsigned int)red[i * 6 + 5];
        }
        atomicMin(&acc->wmin[0], k1);
        atomicMin(&acc->wmin[1], k2);
        atomicMin(&acc->wmin[2], k3);
        atomicMin(&acc->wmin[3], k4);
        atomicMax(&acc->umax, km);
        if (bad) atomicOr(&acc->bad, 1u);
    }
}

#if MHD3D_FAST_BODY
#include "stage_march.cuh"
#else
#include "stage_exact.cuh"
#endif

// Standalone CFL reduction over the current state (STEP 3dmhdsub.f:741-873),
// used before the first step and after a state change.
template <bool MAG>
__global__ void __launch_bounds__(NT) k_cfl(const __grid_constant__ StageArgs a)
{
    const Scalars& s = a.s;
    const int npx = s.npx, npy = s.npy, npz = s.npz;
    const size_t ncell = (size_t)npx * npy * npz;
    unsigned long long kw1 = ~0ull, kw2 = ~0ull, kw3 = ~0ull, kw4 = ~0ull, kmu = 0ull;
    unsigned int bad = 0;
    for (size_t q = (size_t)blockIdx.x * NT + threadIdx.x; q < ncell; q += (size_t)gridDim.x * NT) {
        const int gi = (int)(q % npx);
        const int gj = (int)((q / npx) % npy);
        const int k = (int)(q / ((size_t)npx * npy));
        const double* u = a.u_in + (size_t)(k + 1) * a.uz + (size_t)(gj + 1) * a.upitch + (gi + 1);
        CflPart cp;
        cfl_cell<MAG>(s, u[F_RU * a.uf], u[F_RV * a.uf], u[F_RW * a.uf], u[F_RO * a.uf], u[F_TT * a.uf],
                      MAG ? u[F_BX * a.uf] : 0.0, MAG ? u[F_BY * a.uf] : 0.0, MAG ? u[F_BZ * a.uf] : 0.0,
                      cell_dd(a.m, gi, gj, k), a.m.rkapa[k + 1], cp);
        kw1 = min(kw1, key_of(cp.w1)); kw2 = min(kw2, key_of(cp.w2));
        kw3 = min(kw3, key_of(cp.w3)); kw4 = min(kw4, key_of(cp.w4));
        kmu = max(kmu, key_of(cp.mach2)); bad |= cp.bad;
    }
    __shared__ unsigned long long red[(NT / 32) * 6];
    cfl_commit(a.acc, kw1, kw2, kw3, kw4, kmu, bad, red);
}

// Standalone BCON on the current state, in place (test entry point).
template <bool MAG>
__global__ void __launch_bounds__(NT) k_bcon(const __grid_constant__ StageArgs a)
{
    const Scalars& s = a.s;
    const int npx = s.npx, npy = s.npy, npz = s.npz;
    const int q = blockIdx.x * NT + threadIdx.x;
    if (q >= npx * npy) return;
    const int gi = q % npx, gj = q / npx;
    double* u = const_cast<double*>(a.u_in);
    const size_t col = (size_t)(gj + 1) * a.upitch + (gi + 1);
    auto at = [&](int f, int k) -> double { return u[(size_t)f * a.uf + (size_t)(k + 1) * a.uz + col]; };
    auto put = [&](int f, int k, double v) { store_u(u, (size_t)f * a.uf, a, gi, gj, k + 1, v); };
    const double C13 = s.c13, C23 = s.c23, C43 = s.c43;
    // top
    {
        const double ro0 = at(F_RO, 0), ro1 = at(F_RO, 1), ro2 = at(F_RO, 2);
        const double ru_w = ro0 * (C43 * at(F_RU, 1) / ro1 - C13 * at(F_RU, 2) / ro2);
        const double rv_w = ro0 * (C43 * at(F_RV, 1) / ro1 - C13 * at(F_RV, 2) / ro2);
        double tt_w = at(F_TT, 0);
        const double t1 = at(F_TT, 1), t2 = at(F_TT, 2);
        if (s.plume) {
            const double tpr = (s.tc != 0.0) ? s.tp + (1.0 - s.tp) * exp(-a.ctl->timt / s.tc) : s.tp;
            const double gx = a.m.plume_gx[gi + 1], gy = a.m.plume_gy[gj + 1];
            if (s.itcon == 0) tt_w = 1.0 - (1.0 - tpr) * gx / s.hh * gy / s.hh;
            else tt_w = C43 * t1 - C13 * t2 - C23 * s.top_dz * (s.theta - (s.theta - tpr) * gx / s.hh * gy / s.hh);
        } else if (s.itcon == 0 || s.itcon == 2 || s.itcon == 4) {
            tt_w = 1.0;
            if (s.itcon == 4 && gi + 2 <= (npx + 2) / 2) tt_w = 1.0 - s.tp;
        } else if (s.itcon == 1) {
            tt_w = C43 * t1 - C13 * t2 - s.top_flux;
        }
        put(F_RU, 0, ru_w);
        put(F_RV, 0, rv_w);
        put(F_RW, 0, 0.0);
        put(F_TT, 0, tt_w);
        if (MAG && s.ibcon == 0) put(F_BZ, 0, 0.0);
    }
    // bottom
    {
        const int kb = npz - 1;
        const double ro0 = at(F_RO, kb), ro1 = at(F_RO, kb - 1), ro2 = at(F_RO, kb - 2);
        const double ru_w = ro0 * (C43 * at(F_RU, kb - 1) / ro1 - C13 * at(F_RU, kb - 2) / ro2);
        const double rv_w = ro0 * (C43 * at(F_RV, kb - 1) / ro1 - C13 * at(F_RV, kb - 2) / ro2);
        const double tt_w = (s.izcon == 0) ? s.tb : C43 * at(F_TT, kb - 1) - C13 * at(F_TT, kb - 2) + s.bot_flux;
        put(F_RU, kb, ru_w);
        put(F_RV, kb, rv_w);
        put(F_RW, kb, 0.0);
        put(F_TT, kb, tt_w);
        if (MAG && s.ibcon == 0) put(F_BZ, kb, 0.0);
    }
}

template <bool MAG, bool ROT>
static cudaError_t launch_stage_t(int stage, const StageArgs& a, cudaStream_t st)
{
    const int nty = (a.s.npy + TY - 1) / TY;
    dim3 grid(a.ntx * nty, a.nchunks);
#define L_(S, ...)                                                                                         \
    case S: {                                                                                              \
        constexpr size_t smem = Lay<MAG, S>::BYTES;                                                        \
        static std::atomic<unsigned long long> attr_set{0};                                                \
        cudaError_t ae = smem_attr_once(attr_set, reinterpret_cast<const void*>(k_stage<MAG, ROT, __VA_ARGS__>), smem); \
        if (ae != cudaSuccess) return ae;                                                                  \
        return launch_chained(k_stage<MAG, ROT, __VA_ARGS__>, grid, NT, smem, st, a);                      \
    }
#if MHD3D_FAST_BODY
    if (a.general) switch (stage) { L_(1, 1, true) L_(2, 2, true) L_(3, 3, true) }
#endif
    switch (stage) {
        L_(0, 0) L_(1, 1) L_(2, 2) L_(3, 3)
    default:
        return cudaErrorInvalidValue;
    }
#undef L_
}

cudaError_t launch_stage(int stage, const StageArgs& a, cudaStream_t st)
{
    if (a.s.lmag) return a.s.lrot ? launch_stage_t<true, true>(stage, a, st) : launch_stage_t<true, false>(stage, a, st);
    return a.s.lrot ? launch_stage_t<false, true>(stage, a, st) : launch_stage_t<false, false>(stage, a, st);
}

cudaError_t launch_cfl(const StageArgs& a, cudaStream_t st)
{
    const size_t ncell = (size_t)a.s.npx * a.s.npy * a.s.npz;
    size_t nb = (ncell + NT - 1) / NT;
    if (nb > 148 * 8) nb = 148 * 8;
    if (a.s.lmag) k_cfl<true><<<(unsigned)nb, NT, 0, st>>>(a);
    else k_cfl<false><<<(unsigned)nb, NT, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_bcon(const StageArgs& a, cudaStream_t st)
{
    const int n = a.s.npx * a.s.npy;
    const int nb = (n + NT - 1) / NT;
    if (a.s.lmag) k_bcon<true><<<nb, NT, 0, st>>>(a);
    else k_bcon<false><<<nb, NT, 0, st>>>(a);
    return cudaGetLastError();
}

}  // namespace MHD3D_NS
}  // namespace mhd3d
