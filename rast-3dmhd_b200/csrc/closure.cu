// closure.cu -- kernels of the learned subgrid closure (no counterpart in the
// reference): a 3-layer 3-D convolutional network on the coarse grid, BF16
// weights and activations, FP32 accumulation.
//
// Activations are channels-last BF16 arrays [z][y][x][C] over the coarse
// interior, periodic in x and y, zero outside in z.  A 3x3x3 convolution is an
// implicit GEMM: D[m][n] = sum_k A[m][k] B[n][k], m = 128 consecutive x points
// of one (y, z) row, n = output channel, k = tap*CIN + input channel.
//
//  - k_conv3d (forward, and the input gradient with transposed, flipped
//    weights): tcgen05.mma (kind::f16, BF16 in, FP32 accumulators in TMEM,
//    M=128, K=16 per instruction) issued by one thread.  Input rows (130 x
//    3 z planes) sit in a shared-memory ring, so the A operand of tap
//    (dx, dz) is one descriptor moved by whole voxel rows: with 32 input
//    channels, 64-byte voxel rows in the copy engine's 64-byte swizzle (one
//    TMA box per plane); with 16, [8-channel chunk][voxel] 16-byte rows, the
//    canonical K-major no-swizzle layout with 8-row groups 128 bytes apart.
//    Any nx: the boxes of a row's last segment end with the row, and only its
//    own outputs are stored.  One MMA serves three output rows (N = 3*COUT,
//    the y taps stacked in the B operand), see k_conv3d.  Warp roles: a
//    loader, one MMA thread and four epilogue warps, handing off through
//    mbarriers.  The epilogue adds the bias, applies ReLU or the ReLU mask of
//    the layer below, and writes BF16 (and FP32) outputs.
//  - k_conv3d_wgrad_tc: dW[n][tap*CIN+ci] = sum over voxels of dY[v][n] *
//    X[v+tap][ci] on tcgen05 as well, with K running over voxels: per x
//    segment a dY row read at the three x shifts forms A and the input rows
//    of the y taps form B (the z taps), both MN-major as they lie in memory;
//    per-CTA partials are added in CTA order by k_wgrad_reduce.
//
// Every wait is bounded; a CTA that gives up records an error and releases
// its tensor memory.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "../../include/mhd3d.h"
#include "ring.cuh"
#include "smem_attr.cuh"

namespace mhd3d {
namespace clo {

constexpr int CT = 32 * (4 + 1 + 1);     // threads: 4 epilogue warps (TMEM lanes 0..127), loader, MMA
constexpr int RING = 4;            // input rows held in the ring: the loaders run up to three steps ahead
constexpr int MT = 128;            // output voxels per tile: one 128-point x segment

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor, no swizzle: start address, leading
// (K-direction) and stride (8-row group) byte offsets, SM100 version 1
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFFu) << 32;
    d |= (uint64_t)1 << 46;
    return d;
}

// instruction descriptor: BF16 x BF16 -> FP32, both K-major, M x N
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t acc)
{
    const uint32_t z = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
        ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"(acc), "r"(z), "r"(z), "r"(z), "r"(z)
        : "memory");
}

__device__ __forceinline__ void umma_commit(unsigned long long* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

template <int N>
__device__ __forceinline__ void tmem_ld(uint32_t taddr, float (&v)[N]);

template <>
__device__ __forceinline__ void tmem_ld<16>(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

template <>
__device__ __forceinline__ void tmem_ld<32>(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Ring of input rows for the convolution: [chunk][slot 0..RING-1][z plane 0..2]
// [BXP] of 16-byte rows (or, in the swizzled form, [slot][z plane][BXP] of
// 64-byte rows), voxel xi (x0-1+xi) at row XR0+xi, so that the 128 interior
// voxels start on a 128-byte (512-byte) boundary, a TMA destination; step s
// of a CTA keeps its input row in slot s % RING.
constexpr int XR0 = 7;
constexpr int BXP = 144;              // XR0 + MT + 2 rounded up to 8 rows
constexpr int RSEG = RING * 3 * BXP;  // voxel rows of one chunk of the ring
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The input row of a step by TMA (w <= 128 voxels from x0, the width of map's
// boxes): one 5-D box (8 channels, 1 chunk, w x, 1 y, 1 z) per chunk and z
// plane into the ring's interior rows, zeros outside z (out-of-range box);
// the two periodic x halo voxels by cp.async from the calling warp.  What a
// short row leaves behind its halo feeds only outputs that are not stored.  The
// TMA bytes complete on bar (after the caller's expect_tx); each lane's
// copies are signalled by the caller's cp.async.mbarrier.arrive.
template <int CIN>
__device__ __forceinline__ void load_row_tma(unsigned char* ring, const CUtensorMap* map, unsigned long long* bar,
                                             const __nv_bfloat16* __restrict__ x, int x0, int w, int yr, int z,
                                             int nx, int ny, int nz, int lane, int slot)
{
    constexpr int NC = CIN / 8;
    int gy = yr % ny;
    gy = gy < 0 ? gy + ny : gy;
    const uint32_t sbase = smem_u32(ring);
    if (lane == 0) {
        for (int c = 0; c < NC; ++c)
            for (int zi = 0; zi < 3; ++zi) {
                const uint32_t dst = sbase + (uint32_t)((c * RSEG + (slot * 3 + zi) * BXP + XR0 + 1) * 16);
                asm volatile(
                    "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                    "%3, %4, %5, %6}], [%7];" ::"r"(dst),
                    "l"(reinterpret_cast<unsigned long long>(map)), "r"(0), "r"(c), "r"(x0), "r"(gy), "r"(z - 1 + zi),
                    "r"(smem_u32(bar))
                    : "memory");
            }
    }
    for (int q = lane; q < 2 * NC * 3; q += 32) {
        const int side = q & 1, c = (q >> 1) % NC, zi = (q >> 1) / NC;
        const int xi = side ? w + 1 : 0;
        int gx = x0 - 1 + xi;
        gx = gx < 0 ? gx + nx : (gx >= nx ? gx - nx : gx);
        int gz = z - 1 + zi;
        const uint32_t nbytes = (gz >= 0 && gz < nz) ? 16u : 0u;
        gz = gz < 0 ? 0 : (gz >= nz ? nz - 1 : gz);
        const __nv_bfloat16* src = x + (((size_t)gz * ny + gy) * nx + gx) * CIN + c * 8;
        const uint32_t dst = sbase + (uint32_t)((c * RSEG + (slot * 3 + zi) * BXP + XR0 + xi) * 16);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(nbytes) : "memory");
    }
}

// The input row of a step by TMA for 32 input channels, in the 64-byte
// swizzled K-major layout: plane p = slot*3 + zi of the ring is BXP voxel
// rows of 64 bytes (all 32 channels) from byte p*BXP*64, and the 16-byte
// chunk j (channels 8j..8j+7) of row R sits at chunk position j ^ ((R >> 1) & 3)
// -- the copy engine's SWIZZLE_64B pattern (address bits 4-5 XOR bits 7-8,
// planes 512-byte aligned), which SWIZZLE_64B matrix descriptors read back.
// One 4-D box (32 channels, w x, 1 y, 1 z) per plane lands the interior at
// row XR0+1; the two periodic halo voxels come by cp.async, placed by the
// same rule.
__device__ __forceinline__ void load_row_tma_sw64(unsigned char* ring, const CUtensorMap* map,
                                                  unsigned long long* bar, const __nv_bfloat16* __restrict__ x,
                                                  int x0, int w, int yr, int z, int nx, int ny, int nz, int lane,
                                                  int slot)
{
    constexpr int CIN = 32;
    int gy = yr % ny;
    gy = gy < 0 ? gy + ny : gy;
    const uint32_t sbase = smem_u32(ring);
    if (lane == 0) {
        for (int zi = 0; zi < 3; ++zi) {
            const uint32_t dst = sbase + (uint32_t)(((slot * 3 + zi) * BXP + XR0 + 1) * 64);
            asm volatile(
                "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, "
                "%3, %4, %5}], [%6];" ::"r"(dst),
                "l"(reinterpret_cast<unsigned long long>(map)), "r"(0), "r"(x0), "r"(gy), "r"(z - 1 + zi),
                "r"(smem_u32(bar))
                : "memory");
        }
    }
    if (lane < 24) {
        const int side = lane & 1, j = (lane >> 1) & 3, zi = lane >> 3;
        const int xi = side ? w + 1 : 0;
        int gx = x0 - 1 + xi;
        gx = gx < 0 ? gx + nx : (gx >= nx ? gx - nx : gx);
        int gz = z - 1 + zi;
        const uint32_t nbytes = (gz >= 0 && gz < nz) ? 16u : 0u;
        gz = gz < 0 ? 0 : (gz >= nz ? nz - 1 : gz);
        const __nv_bfloat16* src = x + (((size_t)gz * ny + gy) * nx + gx) * CIN + j * 8;
        const int R = XR0 + xi;
        const uint32_t dst = sbase + (uint32_t)(((slot * 3 + zi) * BXP + R) * 64 + ((j ^ ((R >> 1) & 3)) * 16));
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(nbytes) : "memory");
    }
}

// shared-memory matrix descriptor of a K-major operand in the 64-byte swizzled
// layout: 64-byte rows, 8-row groups 512 bytes apart (the leading offset is
// unused when the K of one MMA lies inside a row), SM100 version 1, base
// offset 0.  The pattern follows the absolute address bits, so a start moved
// by whole rows (an x tap) or by 32 bytes inside a row (the second K half)
// reads the rows the copy engine wrote there (checked against the numpy
// convolution by the GPU parity tests).
__device__ __forceinline__ uint64_t smem_desc_sw64(uint32_t saddr)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;
    return d;
}

__device__ __forceinline__ void mbar_arrive(unsigned long long* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// bounded wait without sleeping between polls: mbarrier.try_wait itself
// suspends the thread for a while, and the pipeline's hand-offs between warp
// roles are on the critical path; false when it gave up
__device__ __forceinline__ bool mbar_wait_fast(unsigned long long* bar, unsigned parity)
{
    for (long it = 0; it < WAIT_LIMIT; ++it)
        if (mbar_test(bar, parity)) return true;
    return false;
}

template <int N>
__device__ __forceinline__ void tmem_st_zero(uint32_t taddr);

template <>
__device__ __forceinline__ void tmem_st_zero<16>(uint32_t taddr)
{
    const uint32_t z = 0;
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr),
        "r"(z)
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

template <>
__device__ __forceinline__ void tmem_st_zero<32>(uint32_t taddr)
{
    const uint32_t z = 0;
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,"
        "%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};\n" ::"r"(taddr),
        "r"(z)
        : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// The steps of a CTA: its range of output rows forms runs along y within one
// (x segment, z) column; a run of output rows ya..yb takes input rows
// ya-1..yb+1, one step each.  f(s, x0, z, r, first, emit) for every step s in
// order: r the unwrapped input row, first the run's first step, emit whether
// output row r-1 is in the run; f returns false to stop.
template <class F>
__device__ __forceinline__ void for_steps(int t_begin, int t_end, int ny, int nz, F f)
{
    int s = 0;
    for (int t = t_begin; t < t_end;) {
        const int ya = t % ny, z = (t / ny) % nz, x0 = (t / (ny * nz)) * MT;
        const int run = (t_end - t) < (ny - ya) ? (t_end - t) : (ny - ya);
        const int yb = ya + run - 1;
        for (int r = ya - 1; r <= yb + 1; ++r, ++s)
            if (!f(s, x0, z, r, r == ya - 1, r - 1 >= ya && r - 1 <= yb)) return;
        t += run;
    }
}

template <int CIN, int COUT>
struct ConvLay {
    static constexpr int K = 27 * CIN;
    static constexpr int KB = 9 * CIN;          // K of one y-tap block: (dz, dx, ci)
    static constexpr int NW = 3 * COUT;         // N of an MMA: three output rows
    static constexpr uint32_t NCOL = NW <= 32 ? 32 : NW <= 64 ? 64 : 128;   // TMEM: three accumulator slots
    static constexpr size_t W_B = (size_t)5 * COUT * KB * 2;   // y-tap blocks 2, 1, 0, 2, 1
    static constexpr size_t X_OFF = (W_B + 1023) / 1024 * 1024;   // the ring's planes 512-byte aligned
    static constexpr size_t X_B = ((size_t)CIN * RSEG * 2 + 127) / 128 * 128;  // ring of RING input rows
    static constexpr size_t BAR_OFF = X_OFF + X_B;
    // barriers: ready[4], mmadone[4], accfull, accempty; then the TMEM
    // address, the abort flag and the last committed step
    static constexpr size_t BYTES = BAR_OFF + 10 * 8 + 16 + 1024;   // + alignment of the base to 1024 bytes
};

// Y = act(conv(X, W) + bias) [* (mask > 0)], persistent over (x segment, y, z) tiles.
// w: [COUT][27*CIN] BF16, k = tap*CIN + ci with tap = dx+1 + 3*(dy+1) + 9*(dz+1).
//
// One MMA serves three output rows: an input row r (one of the CTA's steps)
// contributes to output rows r+1, r, r-1 through the weights of y-taps 0, 1,
// 2.  Three accumulators of COUT columns sit side by side in TMEM, output row
// y in slot y mod 3, and the B operand stacks the y-tap blocks in the slot
// order, which rotates with r mod 3: the weights are kept as the y-tap blocks
// 2, 1, 0, 2, 1 and each step reads the window of three starting at
// (1 - r) mod 3.  Per input row the MMAs are 9 * CIN/16 of N = 3*COUT
// (instead of 27 * CIN/16 of N = COUT per output row), so each input tile
// is read from shared memory a third as often.  After step r, output row r-1
// is complete: the epilogue reads its slot, zeroes it for output row r+2 and
// stores.  The first MMA of a run starts all three slots from zero.
//
// Warp roles, pipelined over the CTA's steps s (ready and mmadone by s & 3):
//   loader (warp 4): the step's input row (three z planes, periodic in x and y,
//     zeros outside z) into ring slot s % RING: one TMA box per z plane of 32
//     channels x 128 voxels (fewer at the row's end) in 64-byte swizzled rows
//     (CIN = 32), or of 8 channels x 128 voxels per chunk and plane (CIN = 16),
//     complete_tx on ready(s), and the two x-halo voxels by cp.async, which
//     arrive on ready(s) as they land (cp.async.mbarrier.arrive); a slot is
//     reused once the MMAs of step s - RING have completed (mmadone).
//   warp 5, lane 0 (MMA): waits ready(s) and the release of step s-1's
//     finished slot (accempty), issues the step's MMAs, commits to accfull
//     and to mmadone(s).
//   warps 0-3 (epilogue): wait accfull(s), read and zero the finished slot
//     (TMEM lanes 32*warp..), release it (accempty) and store while the next
//     step's MMAs run.
//
// A row's last segment has boxes of its own width rather than voxels copied
// one by one with the wrap computed for each: us at nx x 128 x 64, 16->32,
// 32->32, 32->16, before and now: nx = 55: 105, 169, 157 / 63, 81, 71;
// 250 (one full segment, one of 122): 154, 234, 211 / 112, 142, 124; 128
// (full segments only): 65, 83, 72.  The epilogue reads the mask as 16-byte
// vectors: input gradient at 128x128x64, 16->32 and 32->32: 112, 130 us with
// one load a value, 91, 102 now.
template <int CIN, int COUT>
__global__ void __launch_bounds__(CT, 1) k_conv3d(const __grid_constant__ CUtensorMap xmap,
                                                  const __grid_constant__ CUtensorMap xtail,
                                                  const __nv_bfloat16* __restrict__ x,
                                                  const __nv_bfloat16* __restrict__ w, const float* __restrict__ bias,
                                                  const __nv_bfloat16* __restrict__ mask, int relu,
                                                  __nv_bfloat16* __restrict__ y, float* __restrict__ yf, int nx, int ny,
                                                  int nz, int* err)
{
    using L = ConvLay<CIN, COUT>;
    constexpr int K = L::K, KB = L::KB;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* const sb = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    unsigned char* const sw = sb;
    unsigned char* const sx = sb + L::X_OFF;
    unsigned long long* const bars = reinterpret_cast<unsigned long long*>(sb + L::BAR_OFF);
    unsigned long long* const ready = bars;
    unsigned long long* const mmadone = bars + 4;
    unsigned long long* const accfull = bars + 8;
    unsigned long long* const accempty = bars + 9;
    uint32_t* const tslot = reinterpret_cast<uint32_t*>(sb + L::BAR_OFF + 80);
    volatile int* const abort_flag = reinterpret_cast<volatile int*>(sb + L::BAR_OFF + 84);
    volatile int* const last_commit = reinterpret_cast<volatile int*>(sb + L::BAR_OFF + 88);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // weights -> y-tap blocks 2,1,0,2,1 of [COUT][KB], k' = (dz*3 + dx)*CIN + ci, in
    // the canonical K-major layout: row n', k' at ((n'/8)*(KB/8) + k'/8)*128 + (n'%8)*16 + (k'%8)*2
    {
        // eight loads in flight per thread before their stores
        constexpr int NQ = 5 * COUT * (KB / 8), BATCH = 8;
        for (int q0 = tid; q0 < NQ; q0 += CT * BATCH) {
            uint4 v[BATCH];
            int dst[BATCH];
#pragma unroll
            for (int u = 0; u < BATCH; ++u) {
                const int q = q0 + u * CT;
                dst[u] = -1;
                if (q < NQ) {
                    const int blk = q / (COUT * (KB / 8)), rem = q % (COUT * (KB / 8));
                    const int n = rem / (KB / 8), kc = rem % (KB / 8);
                    const int dyi = blk == 2 ? 0 : (blk == 1 || blk == 4) ? 1 : 2;
                    const int dzdx = (kc * 8) / CIN, ci = (kc * 8) % CIN, dzi = dzdx / 3, dxi = dzdx % 3;
                    const int tap = dxi + 3 * dyi + 9 * dzi;
                    v[u] = __ldg(reinterpret_cast<const uint4*>(w + (size_t)n * K + tap * CIN + ci));
                    const int nr = blk * COUT + n;
                    dst[u] = (int)(((nr >> 3) * (KB / 8) + kc) * 128 + (nr & 7) * 16);
                }
            }
#pragma unroll
            for (int u = 0; u < BATCH; ++u)
                if (dst[u] >= 0) *reinterpret_cast<uint4*>(sw + dst[u]) = v[u];
        }
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(L::NCOL)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int b = 0; b < 4; ++b) {
            // the expect_tx arrival and one completion arrival per lane of the loader warp
            mbar_init(ready + b, 1 + 32);
            mbar_init(mmadone + b, 1);
        }
        mbar_init(accfull, 1);
        mbar_init(accempty, 4);
        *abort_flag = 0;
        *last_commit = -1;
        fence_mbar_init();
    }
    fence_proxy_async();   // the weights, written by plain stores, are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    // output rows in (segment, z, y) order with y fastest; each CTA takes one
    // contiguous range, walked as runs along y
    const int nseg = (nx + MT - 1) / MT;
    const int ntile = nseg * ny * nz;
    const int t_begin = (int)(((long)ntile * blockIdx.x) / gridDim.x);
    const int t_end = (int)(((long)ntile * (blockIdx.x + 1)) / gridDim.x);
    auto give_up = [&]() {
        *abort_flag = 1;
        atomicExch(err, 1);
    };

    if (warp == 4) {
        // one warp: the TMA boxes of the step's row and its two halo voxels
        for_steps(t_begin, t_end, ny, nz, [&](int s, int x0, int zz, int r, bool, bool) {
            if (*abort_flag) return false;
            const int jw = s - RING;   // slot s % RING was last read by step s - RING
            if (jw >= 0 && !mbar_wait_fast(mmadone + (jw & 3), (unsigned)(jw >> 2) & 1u)) {
                give_up();
                return false;
            }
            unsigned long long* const bar = ready + (s & 3);
            const int w = nx - x0 < MT ? nx - x0 : MT;
            const CUtensorMap* const map = w < MT ? &xtail : &xmap;
            if (lane == 0) mbar_expect_tx(bar, (unsigned)(CIN / 8 * 3 * w * 16));
            if constexpr (CIN == 32) load_row_tma_sw64(sx, map, bar, x, x0, w, r, zz, nx, ny, nz, lane, s % RING);
            else load_row_tma<CIN>(sx, map, bar, x, x0, w, r, zz, nx, ny, nz, lane, s % RING);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
            return true;
        });
        cp_async_wait<0>();
    } else if (warp == 5) {
        if (lane == 0) {
            constexpr uint32_t IDESC = idesc_bf16(MT, L::NW);
            const uint64_t da0 = smem_desc(smem_u32(sx), RSEG * 16, 128);
            const uint64_t da0s = smem_desc_sw64(smem_u32(sx));
            const uint64_t db0 = smem_desc(smem_u32(sw), 128, (KB / 8) * 128);
            for_steps(t_begin, t_end, ny, nz, [&](int s, int, int, int r, bool first, bool) {
                if (*abort_flag) return false;
                if (!mbar_wait_fast(ready + (s & 3), (unsigned)(s >> 2) & 1u) ||
                    (s > 0 && !mbar_wait_fast(accempty, (unsigned)(s - 1) & 1u))) {
                    give_up();
                    return false;
                }
                fence_proxy_async();   // the ring row, written by cp.async, is read by the tensor cores
                tc_fence_after();
                // window of y-tap blocks for slots 0, 1, 2: starts at (1 - r) mod 3
                const uint32_t st = (uint32_t)(((1 - r) % 3 + 3) % 3);
                const uint32_t as = (uint32_t)((s % RING) * 3 * BXP + XR0);
                // the step's descriptors first (their low words: the start
                // addresses; the high words are fixed), then its MMAs back to
                // back.  Tap (dz, dx) moves the A start by whole voxel rows:
                // 64-byte rows in the swizzled form (the second K half 32
                // bytes into the row), 16-byte rows otherwise (the second K
                // half one chunk of the ring further)
                constexpr int NM = 9 * CIN / 16, KH = CIN / 16;
                constexpr bool swz = CIN == 32;
                const uint64_t dab = swz ? da0s : da0;
                const uint32_t a0 = (uint32_t)dab + (swz ? as * 4 : as);
                const uint32_t b0 = (uint32_t)db0 + st * (COUT / 8) * (KB / 8) * 8;
                uint32_t alo[NM], blo[NM];
#pragma unroll
                for (int j = 0; j < NM; ++j) {
                    const int dz = j / (3 * KH), dx = (j / KH) % 3, kk = j % KH;
                    alo[j] = a0 + (swz ? (uint32_t)((dz * BXP + dx) * 4 + 2 * kk)
                                       : (uint32_t)(2 * kk * RSEG + dz * BXP + dx));
                    blo[j] = b0 + (uint32_t)((((dz * 3 + dx) * CIN + kk * 16) >> 3) * 8);
                }
                const uint64_t ahi = dab & 0xFFFFFFFF00000000ull, bhi = db0 & 0xFFFFFFFF00000000ull;
#pragma unroll
                for (int j = 0; j < NM; ++j)
                    umma_bf16(tmem, ahi | alo[j], bhi | blo[j], IDESC, (first && j == 0) ? 0u : 1u);
                umma_commit(accfull);
                umma_commit(mmadone + (s & 3));
                *last_commit = s;
                return true;
            });
        }
        __syncwarp();
    } else {
        for_steps(t_begin, t_end, ny, nz, [&](int s, int x0, int zz, int r, bool, bool emit) {
            if (*abort_flag) return false;
            if (!mbar_wait_fast(accfull, (unsigned)s & 1u)) {
                give_up();
                return false;
            }
            tc_fence_after();
            const int yo = r - 1;   // the output row this step completes
            const uint32_t col = (uint32_t)((((yo % 3) + 3) % 3) * COUT);
            const uint32_t ta = tmem + ((uint32_t)(warp * 32) << 16) + col;
            float acc[COUT];
            if (emit) tmem_ld<COUT>(ta, acc);
            tmem_st_zero<COUT>(ta);
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(accempty);
            if (!emit) return true;
            const int m = warp * 32 + lane;
            const bool own = x0 + m < nx;   // lanes beyond the row's end store nothing
            const size_t vox = ((size_t)zz * ny + yo) * nx + (own ? x0 + m : 0);
#pragma unroll
            for (int n = 0; n < COUT; ++n) {
                const float o = acc[n] + (bias ? bias[n] : 0.f);
                acc[n] = relu ? (o > 0.f ? o : 0.f) : o;
            }
            if (mask) {
#pragma unroll
                for (int n = 0; n < COUT; n += 8) {
                    const uint4 q = __ldg(reinterpret_cast<const uint4*>(mask + vox * COUT + n));
                    const __nv_bfloat16* const h = reinterpret_cast<const __nv_bfloat16*>(&q);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        if (!(__bfloat162float(h[i]) > 0.f)) acc[n + i] = 0.f;
                }
            }
            if (y && own) {
#pragma unroll
                for (int n = 0; n < COUT; n += 8) {
                    __align__(16) __nv_bfloat16 h[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) h[i] = __float2bfloat16_rn(acc[n + i]);
                    *reinterpret_cast<uint4*>(y + vox * COUT + n) = *reinterpret_cast<const uint4*>(h);
                }
            }
            if (yf && own) {
#pragma unroll
                for (int n = 0; n < COUT; n += 4)
                    *reinterpret_cast<float4*>(yf + vox * COUT + n) =
                        make_float4(acc[n], acc[n + 1], acc[n + 2], acc[n + 3]);
            }
            return true;
        });
    }
    // every MMA has completed once the epilogue has seen its last accumulator;
    // after an abort, wait (bounded) for the last issued step's MMAs before
    // freeing TMEM
    __syncthreads();
    if (*abort_flag && tid == 0 && *last_commit >= 0) {
        const int jl = *last_commit;
        mbar_wait_fast(mmadone + (jl & 3), (unsigned)(jl >> 2) & 1u);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::NCOL));
}

// ---------------------------------------------------------------------------
// Weight gradient on the tensor cores.
//
// dW[n][tap(dx,dy,dz)*CIN+ci] = sum_v dY[v][n] X[v + (dx-1, dy-1, dz-1)][ci]
// is a GEMM whose K runs over voxels.  For an x segment of WT=64 voxels
// (x0..x0+63) of one (y, z) row, with u = 0..KT-1 indexing x0-1+u:
//
//   A[(dx, n)][u]   = dY[x0 + u - dx][n]  (zero outside the segment's own
//                     voxels)                              M = 128
//   B_dy[(dz,ci)][u] = X[x0-1+u, y+dy-1, z+dz-1][ci] (periodic in x, y; zero
//                     outside z and for u >= WT+2)             N = 3*CIN
//   D_dy[(dx,n)][(dz,ci)] += sum_u A B_dy                      K = KT = 80
//
// so one segment is 3 (y taps) x 5 (K steps of 16) MMAs of M=128, N=3*CIN.
// Channels-last rows are MN-major operands as they lie in memory: a voxel is
// one row of K, its channels one row of M or N (64- or 32-byte rows in the
// swizzle of that width, which the matrix descriptors read back), so TMA boxes
// (and cp.async for the two halo voxels) fill both operands and nothing is
// transposed.  The x taps are blocks of one staged dY row that start a voxel
// apart (block j holds dx = 2-j; the leading offset of A is one voxel; blocks
// beyond the third are unused lanes), the z taps the three planes of an input
// row.  A row's last segment has boxes of its own width and only the K steps
// that its voxels reach.  The loader warp runs up to WST segments ahead of
// the MMA thread.  The three accumulators (3*3*CIN columns) stay in TMEM over
// all of a CTA's segments (a fixed set, in a fixed order); each CTA writes
// its partial sums to a workspace row and a second kernel adds the rows to dW
// in CTA order, so the result does not depend on timing.
//
// No unit is full: 32->32 at 128x128x64, a segment takes 2050 cycles of its SM,
// 720 of them with the tensor pipe active (48 an MMA of N = 96); L2 is at 37 %
// (42 KB a segment), DRAM at 12 %, issue at 12 %.  What is left is the chain of a
// segment, boxes and halo copies, hand-off, 15 MMAs, hand-off, of which three
// are in flight.  128x128x64, us: 16->32 117, 32->32 143, 32->16 129.  The
// form that transposed both operands through registers took 463, 657 and 605,
// this one with every voxel by cp.async 151, 241 and 231.  Marching along y with
// 128-voxel segments and the roles of the operands exchanged took 137, 146 and
// 114, but sums in another order; this one's bits are those of the first form.
constexpr int WT = 64;               // voxels of an x segment
constexpr int KT = 80;               // K of a segment: WT + 2 halo voxels, padded to 16
constexpr int WG_LD = 1;             // loader warp
constexpr int WG_SUM = 256;          // threads that sum dY (the first four warps are the epilogue)
constexpr int WG_NTH = WG_SUM + 32 * (WG_LD + 1);
// Rows of the staged operands: voxel x0 of an input row or of dY sits at row 8,
// a TMA destination (512 or 256 bytes); u = 0 is row WXR0 of an input row and
// row WYR0 of dY with dx = 2.
constexpr int WXR0 = 7, WYR0 = 6;
constexpr int WXR = 88;              // rows of an input row: WXR0 + KT rounded up to 8
constexpr int WYR = 96;              // of dY: WYR0 + KT and what the unused blocks read
constexpr int WST = 3;               // stages

template <int CIN, int COUT>
struct WgLay {
    static constexpr int XB = CIN * 2, YB = COUT * 2;         // bytes of a voxel
    static constexpr int N = 3 * CIN;                         // columns of one y-tap accumulator
    static constexpr uint32_t NCOL = 3 * N <= 256 ? 256 : 512;
    static constexpr int X_ROW = WXR * XB;                    // one input row (y, z)
    static constexpr int Y_OFF = (9 * X_ROW + 511) / 512 * 512;   // dY behind the nine input rows of a stage
    static constexpr int STAGE_B = (Y_OFF + WYR * YB + 1023) / 1024 * 1024;
    static constexpr int RED_OFF = WST * STAGE_B;
    static constexpr int BAR_OFF = RED_OFF + WG_SUM * 8 * 4;
    // barriers: ready[WST], mmadone[WST], sumdone[WST]; the TMEM address, the
    // abort flag and the last committed segment
    static constexpr size_t BYTES = BAR_OFF + 3 * WST * 8 + 16 + 1024;   // + alignment of the base to 1024 bytes
};

// matrix descriptor of an MN-major operand: rows of ROWB bytes (64: 64-byte
// swizzle, 32: 32-byte swizzle) along K, 8-row groups ROWB*8 bytes apart,
// blocks of ROWB bytes along MN lbo bytes apart
template <int ROWB>
__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t saddr, uint32_t lbo)
{
    uint64_t d = (uint64_t)((saddr >> 4) & 0x3FFFu);
    d |= (uint64_t)((lbo >> 4) & 0x3FFFu) << 16;
    d |= (uint64_t)(ROWB * 8 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)(ROWB == 64 ? 4 : 6) << 61;
    return d;
}

// 16-byte chunk c of row r of an operand whose rows have ROWB bytes
template <int ROWB>
__device__ __forceinline__ uint32_t swz_chunk(int r, int c)
{
    return (uint32_t)(r * ROWB + ((ROWB == 64 ? c ^ ((r >> 1) & 3) : c ^ ((r >> 2) & 1)) * 16));
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool on)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(on ? 16u : 0u) : "memory");
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(WG_NTH, 1) k_conv3d_wgrad_tc(const __grid_constant__ CUtensorMap xmap,
                                                               const __grid_constant__ CUtensorMap xtail,
                                                               const __grid_constant__ CUtensorMap ymap,
                                                               const __nv_bfloat16* __restrict__ x,
                                                               const __nv_bfloat16* __restrict__ dy,
                                                               float* __restrict__ ws, int nx, int ny, int nz,
                                                               int* __restrict__ err)
{
    using L = WgLay<CIN, COUT>;
    constexpr int N = L::N, K = 27 * CIN, NCX = CIN / 8, NCY = COUT / 8;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* const sb = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const uint32_t sa = smem_u32(sb);
    float* const red = reinterpret_cast<float*>(sb + L::RED_OFF);
    unsigned long long* const ready = reinterpret_cast<unsigned long long*>(sb + L::BAR_OFF);
    unsigned long long* const mmadone = ready + WST;
    unsigned long long* const sumdone = ready + 2 * WST;
    uint32_t* const tslot = reinterpret_cast<uint32_t*>(sb + L::BAR_OFF + 3 * WST * 8);
    volatile int* const abort_flag = reinterpret_cast<volatile int*>(tslot + 1);
    volatile int* const last_commit = reinterpret_cast<volatile int*>(tslot + 2);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    // what no copy writes stays zero: input rows u >= WT+2, dY outside the segment
    for (int q = tid; q < WST * L::STAGE_B / 16; q += WG_NTH)
        *reinterpret_cast<uint4*>(sb + (size_t)q * 16) = make_uint4(0, 0, 0, 0);
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)),
                     "r"(L::NCOL)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    if (tid == 0) {
        for (int b = 0; b < WST; ++b) {
            mbar_init(ready + b, 1 + 32);
            mbar_init(mmadone + b, 1);
            mbar_init(sumdone + b, WG_SUM / 32);
        }
        *abort_flag = 0;
        *last_commit = -1;
        fence_mbar_init();
    }
    fence_proxy_async();   // the zeros, written by plain stores, are read by the tensor cores
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    const int nseg = (nx + WT - 1) / WT;
    const int ntile = nseg * ny * nz;
    // segments blockIdx.x, blockIdx.x + gridDim.x, ..: the i-th in stage i % WST;
    // f(i, t, stage, parity) returns false to stop
    auto segments = [&](auto f) {
        int i = 0, st = 0;
        unsigned ph = 0;
        for (int t = blockIdx.x; t < ntile; t += gridDim.x, ++i) {
            if (*abort_flag || !f(i, t, st, ph)) return;
            if (++st == WST) {
                st = 0;
                ph ^= 1u;
            }
        }
    };
    auto give_up = [&]() {
        *abort_flag = 1;
        atomicExch(err, 1);
        return false;
    };

    // K steps of a segment of w voxels: u = 0..w+1 can meet a dY of its own
    auto ksteps = [](int w) { return (w + 2 + 15) / 16; };

    float dbacc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // dY sums of this thread's 8 channels
    if (warp == WG_SUM / 32) {
        // one warp: ten TMA boxes (dY zeros beyond the row's end) and the input
        // rows' halo voxels; what a short row leaves behind its halo meets zeros
        segments([&](int i, int t, int st, unsigned ph) {
            if (i >= WST && (!mbar_wait_fast(mmadone + st, ph ^ 1u) || !mbar_wait_fast(sumdone + st, ph ^ 1u)))
                return give_up();
            const int x0 = (t % nseg) * WT, yy = (t / nseg) % ny, zz = t / (nseg * ny);
            const uint32_t sx = sa + (uint32_t)(st * L::STAGE_B);
            const int w = nx - x0 < WT ? nx - x0 : WT;   // the segment's own voxels
            const CUtensorMap* const map = w < WT ? &xtail : &xmap;
            if (lane == 0) {
                mbar_expect_tx(ready + st, (unsigned)(9 * w * L::XB + WT * L::YB));
                for (int rz = 0; rz < 9; ++rz) {
                    int gy = yy + rz / 3 - 1;
                    gy = gy < 0 ? gy + ny : (gy >= ny ? gy - ny : gy);
                    tma_load4(sb + (size_t)st * L::STAGE_B + rz * L::X_ROW + 8 * L::XB, map, ready + st, 0, x0, gy,
                              zz + rz % 3 - 1);   // zeros outside z
                }
                tma_load4(sb + (size_t)st * L::STAGE_B + L::Y_OFF + 8 * L::YB, &ymap, ready + st, 0, x0, yy, zz);
            }
            for (int q = lane; q < 9 * 2 * NCX; q += 32) {
                const int c = q % NCX, side = q / NCX % 2, rz = q / (2 * NCX);
                int gy = yy + rz / 3 - 1;
                gy = gy < 0 ? gy + ny : (gy >= ny ? gy - ny : gy);
                const int gz = zz + rz % 3 - 1;
                const bool on = gz >= 0 && gz < nz;
                int gx = side ? x0 + w : x0 - 1;
                gx = gx < 0 ? gx + nx : (gx >= nx ? gx - nx : gx);
                cp_async16(sx + (uint32_t)(rz * L::X_ROW) + swz_chunk<L::XB>(side ? 8 + w : 7, c),
                           x + (((size_t)(on ? gz : zz) * ny + gy) * nx + gx) * CIN + c * 8, on);
            }
            // a short segment: zeros up to the end of its last K step
            const int nzr = ksteps(w) * 16 - (w + 2);
            if (w < WT)
                for (int q = lane; q < 9 * nzr * NCX; q += 32) {
                    const int c = q % NCX, u = q / NCX % nzr, rz = q / (nzr * NCX);
                    cp_async16(sx + (uint32_t)(rz * L::X_ROW) + swz_chunk<L::XB>(9 + w + u, c), x, false);
                }
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(ready + st)) : "memory");
            return true;
        });
        cp_async_wait<0>();
    } else if (warp == WG_SUM / 32 + WG_LD) {
        if (lane == 0) {
            constexpr uint32_t IDESC = idesc_bf16(128, N) | (1u << 15) | (1u << 16);   // both operands MN-major
            segments([&](int i, int t, int st, unsigned ph) {
                if (!mbar_wait_fast(ready + st, ph)) return give_up();
                const int x0 = (t % nseg) * WT, ks = ksteps(nx - x0 < WT ? nx - x0 : WT);
                fence_proxy_async();   // rows written by cp.async are read by the tensor cores
                tc_fence_after();
                const uint32_t sx = sa + (uint32_t)(st * L::STAGE_B);
                const uint64_t da = smem_desc_mn<L::YB>(sx + L::Y_OFF + WYR0 * L::YB, L::YB);
                const uint64_t db = smem_desc_mn<L::XB>(sx + WXR0 * L::XB, L::X_ROW);
#pragma unroll
                for (int d = 0; d < 3; ++d)
#pragma unroll
                    for (int k2 = 0; k2 < KT / 16; ++k2) {
                        if (k2 >= ks) break;
                        umma_bf16(tmem + (uint32_t)(d * N), da + (uint64_t)(k2 * L::YB),
                                  db + (uint64_t)((d * 3 * L::X_ROW >> 4) + k2 * L::XB), IDESC,
                                  (i == 0 && k2 == 0) ? 0u : 1u);
                    }
                umma_commit(mmadone + st);
                *last_commit = i;
                return true;
            });
        }
        __syncwarp();
    } else if (tid < WG_SUM) {
        // bias gradient from the staged dY (zeros beyond the segment's own voxels)
        segments([&](int, int, int st, unsigned ph) {
            if (!mbar_wait_fast(ready + st, ph)) return give_up();
            const unsigned char* const sy = sb + (size_t)st * L::STAGE_B + L::Y_OFF;
            for (int q = tid; q < WT * NCY; q += WG_SUM) {
                const uint4 v = *reinterpret_cast<const uint4*>(sy + swz_chunk<L::YB>(q / NCY + 8, q % NCY));
                const __nv_bfloat16* h = reinterpret_cast<const __nv_bfloat16*>(&v);
#pragma unroll
                for (int e = 0; e < 8; ++e) dbacc[e] += __bfloat162float(h[e]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(sumdone + st);
            return true;
        });
    }
    __syncthreads();
    // the accumulators are complete (after an abort: the MMAs issued have
    // completed, bounded) once the last commit has
    if (tid == 0 && *last_commit >= 0) {
        const int jl = *last_commit;
        if (!mbar_wait_fast(mmadone + jl % WST, (unsigned)(jl / WST) & 1u)) give_up();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    float* const wrow = ws + (size_t)blockIdx.x * ((size_t)COUT * K + COUT);
    if (!*abort_flag && warp < 4) {
        // accumulator lane m = (2-dx, n); columns (dz, ci) of y tap d
        const int dxs = 2 - tid / COUT, n = tid % COUT;
#pragma unroll
        for (int d = 0; d < 3; ++d)
#pragma unroll
            for (int c0 = 0; c0 < N; c0 += 16) {
                float v[16];
                tmem_ld<16>(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)(d * N + c0), v);
                if (dxs >= 0) {
                    float* const o = wrow + (size_t)n * K + (dxs + 3 * d + 9 * (c0 / CIN)) * CIN + c0 % CIN;
#pragma unroll
                    for (int e = 0; e < 16; ++e) o[e] = v[e];
                }
            }
    }
    // bias gradient: this thread's 8 channel sums, added up over the threads
    // that hold the same channels, in thread order
    if (tid < WG_SUM)
#pragma unroll
        for (int e = 0; e < 8; ++e) red[tid * 8 + e] = dbacc[e];
    __syncthreads();
    if (tid < COUT) {
        float sacc = 0.f;
        for (int t2 = tid / 8; t2 < WG_SUM; t2 += NCY) sacc += red[t2 * 8 + tid % 8];
        wrow[(size_t)COUT * K + tid] = sacc;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(L::NCOL));
}

// dW += sum over CTAs of their rows of the workspace, in CTA order (and db);
// NaN everywhere when a CTA of the gradient kernel gave up a wait
__global__ void k_wgrad_reduce(const float* __restrict__ ws, int rows, int nw, int nb, float* __restrict__ dw,
                               float* __restrict__ db, const int* __restrict__ err)
{
    const int stride = nw + nb;
    const bool bad = *err != 0;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < stride; q += gridDim.x * blockDim.x) {
        // in row order, 32 loads in flight
        float acc = 0.f;
        int r = 0;
        for (; r + 32 <= rows; r += 32) {
            float v[32];
#pragma unroll
            for (int t = 0; t < 32; ++t) v[t] = ws[(size_t)(r + t) * stride + q];
#pragma unroll
            for (int t = 0; t < 32; ++t) acc += v[t];
        }
        for (; r < rows; ++r) acc += ws[(size_t)r * stride + q];
        if (bad) acc = __int_as_float(0x7fc00000);
        if (q < nw) dw[q] += acc;
        else if (db) db[q - nw] += acc;
    }
}

// W[n][tap*CIN+ci] -> Wt[ci][(26-tap)*COUT+n]: the input-gradient convolution
__global__ void k_wtranspose(const __nv_bfloat16* __restrict__ w, __nv_bfloat16* __restrict__ wt, int cin, int cout)
{
    const int K = 27 * cin;
    for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < cout * K; q += gridDim.x * blockDim.x) {
        const int n = q / K, k = q % K, tap = k / cin, ci = k % cin;
        wt[(size_t)ci * (27 * cout) + (26 - tap) * cout + n] = w[q];
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// tiled TMA map of a BF16 array of the given rank, zeros outside
cudaError_t encode_bf16(CUtensorMap* map, int rank, void* base, const cuuint64_t* dims, const cuuint64_t* strides,
                        const cuuint32_t* box, CUtensorMapSwizzle swz)
{
    static EncodeTiledFn enc = nullptr;
    if (!enc) {
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || !fn)
            return cudaErrorInvalidValue;
        enc = reinterpret_cast<EncodeTiledFn>(fn);
    }
    const cuuint32_t estr[5] = {1, 1, 1, 1, 1};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, (cuuint32_t)rank, base, dims, strides, box, estr,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, swz, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

template <int CIN, int COUT>
cudaError_t launch_conv_t(const void* x, const void* w, const float* bias, const void* mask, int relu, void* y,
                          float* yf, int nx, int ny, int nz, int* err, cudaStream_t st)
{
    using L = ConvLay<CIN, COUT>;
    static std::atomic<unsigned long long> attr{0};
    cudaError_t ae = smem_attr_once(attr, reinterpret_cast<const void*>(k_conv3d<CIN, COUT>), L::BYTES);
    if (ae != cudaSuccess) return ae;
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int ntile = ((nx + MT - 1) / MT) * ny * nz;
    const int grid = ntile < sms ? ntile : sms;
    // boxes of 128 voxels, and of what the row's last segment holds
    CUtensorMap maps[2];
    std::memset(maps, 0, sizeof(maps));
    for (int o = 0; o < 2; ++o) {
        const int w = o ? nx % MT : MT;
        if (!w || (!o && nx < MT)) continue;
        cudaError_t e;
        if (CIN == 32) {
            // (channel, x, y, z) boxes of 32 channels, 64-byte swizzled rows
            const cuuint64_t dims[4] = {(cuuint64_t)CIN, (cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
            const cuuint64_t strides[3] = {(cuuint64_t)CIN * 2, (cuuint64_t)nx * CIN * 2, (cuuint64_t)nx * ny * CIN * 2};
            const cuuint32_t box[4] = {(cuuint32_t)CIN, (cuuint32_t)w, 1, 1};
            e = encode_bf16(&maps[o], 4, const_cast<void*>(x), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_64B);
        } else {
            // (8 channels, chunk, x, y, z) boxes, 16-byte rows
            const cuuint64_t dims[5] = {8, (cuuint64_t)CIN / 8, (cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
            const cuuint64_t strides[4] = {16, (cuuint64_t)CIN * 2, (cuuint64_t)nx * CIN * 2,
                                           (cuuint64_t)nx * ny * CIN * 2};
            const cuuint32_t box[5] = {8, 1, (cuuint32_t)w, 1, 1};
            e = encode_bf16(&maps[o], 5, const_cast<void*>(x), dims, strides, box, CU_TENSOR_MAP_SWIZZLE_NONE);
        }
        if (e != cudaSuccess) return e;
    }
    k_conv3d<CIN, COUT><<<grid, CT, L::BYTES, st>>>(
        maps[0], maps[1], static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(w), bias,
        static_cast<const __nv_bfloat16*>(mask), relu, static_cast<__nv_bfloat16*>(y), yf, nx, ny, nz, err);
    return cudaGetLastError();
}

// CTAs of the weight gradient: one per SM, at most one per segment
int wgrad_grid(int ntile)
{
    int sms = 148, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return ntile < sms ? ntile : sms;
}

// a partial row a CTA, and the error flag
size_t wgrad_bytes(int cin, int cout, int grid)
{
    return (size_t)grid * ((size_t)cout * 27 * cin + cout) * sizeof(float) + 16;
}

// the tensor-core weight gradient: a fixed grid over the segments, its partial
// rows in the workspace, then the ordered reduction into dw, db
template <int CIN, int COUT>
cudaError_t launch_wgrad_tc_t(const void* x, const void* dy, float* dw, float* db, int nx, int ny, int nz, void* buf,
                              cudaStream_t st)
{
    using L = WgLay<CIN, COUT>;
    static std::atomic<unsigned long long> attr{0};
    cudaError_t e = smem_attr_once(attr, reinterpret_cast<const void*>(k_conv3d_wgrad_tc<CIN, COUT>), L::BYTES);
    if (e != cudaSuccess) return e;
    const int grid = wgrad_grid(((nx + WT - 1) / WT) * ny * nz);
    const size_t stride = (size_t)COUT * 27 * CIN + COUT;
    int* err = reinterpret_cast<int*>(static_cast<char*>(buf) + wgrad_bytes(CIN, COUT, grid) - 16);
    e = cudaMemsetAsync(err, 0, sizeof(int), st);
    // (channel, x, y, z) boxes: 64 voxels of x and dy, and of x what the row's last segment holds
    CUtensorMap maps[3];
    std::memset(maps, 0, sizeof(maps));
    for (int o = 0; o < 3 && e == cudaSuccess; ++o) {
        const int w = o == 1 ? nx % WT : WT;
        if (!w || (o == 0 && nx < WT)) continue;
        const cuuint64_t c = o == 2 ? COUT : CIN;
        const cuuint64_t dims[4] = {c, (cuuint64_t)nx, (cuuint64_t)ny, (cuuint64_t)nz};
        const cuuint64_t strides[3] = {c * 2, (cuuint64_t)nx * c * 2, (cuuint64_t)nx * ny * c * 2};
        const cuuint32_t box[4] = {(cuuint32_t)c, (cuuint32_t)w, 1, 1};
        e = encode_bf16(&maps[o], 4, const_cast<void*>(o == 2 ? dy : x), dims, strides, box,
                        c == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B);
    }
    if (e == cudaSuccess) {
        k_conv3d_wgrad_tc<CIN, COUT><<<grid, WG_NTH, L::BYTES, st>>>(
            maps[0], maps[1], maps[2], static_cast<const __nv_bfloat16*>(x), static_cast<const __nv_bfloat16*>(dy),
            static_cast<float*>(buf), nx, ny, nz, err);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) {
        const int nw = COUT * 27 * CIN;
        k_wgrad_reduce<<<(int)((stride + 63) / 64), 64, 0, st>>>(static_cast<const float*>(buf), grid, nw, COUT,
                                                                    dw, db, err);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_wgrad(int cin, int cout, const void* x, const void* dy, float* dw, float* db, int nx, int ny,
                         int nz, void* buf, cudaStream_t st)
{
    if (cin == 16) return launch_wgrad_tc_t<16, 32>(x, dy, dw, db, nx, ny, nz, buf, st);
    if (cout == 32) return launch_wgrad_tc_t<32, 32>(x, dy, dw, db, nx, ny, nz, buf, st);
    return launch_wgrad_tc_t<32, 16>(x, dy, dw, db, nx, ny, nz, buf, st);
}

bool wgrad_shape(int cin, int cout)
{
    return (cin == 16 && cout == 32) || (cin == 32 && (cout == 32 || cout == 16));
}

}  // namespace clo
}  // namespace mhd3d

using namespace mhd3d::clo;

// activations and weights move as 16-byte vectors
static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

extern "C" {

int mhd3d_conv3d(int32_t cin, int32_t cout, const void* x, const void* w, const float* bias, const void* mask,
                 int32_t relu, void* y, float* yf, int32_t nx, int32_t ny, int32_t nz, int32_t* err, void* stream)
{
    if (!x || !w || !err || nx <= 0 || ny <= 0 || nz <= 0 || (!y && !yf))
        return MHD3D_ERR_ARG;
    if (!aligned16(x) || !aligned16(w) || !aligned16(mask) || !aligned16(y) || !aligned16(yf)) return MHD3D_ERR_ARG;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    cudaError_t e;
    if (cin == 16 && cout == 32) e = launch_conv_t<16, 32>(x, w, bias, mask, relu, y, yf, nx, ny, nz, err, st);
    else if (cin == 32 && cout == 32) e = launch_conv_t<32, 32>(x, w, bias, mask, relu, y, yf, nx, ny, nz, err, st);
    else if (cin == 32 && cout == 16) e = launch_conv_t<32, 16>(x, w, bias, mask, relu, y, yf, nx, ny, nz, err, st);
    else return MHD3D_ERR_ARG;
    return e == cudaSuccess ? MHD3D_OK : MHD3D_ERR_CUDA;
}

int64_t mhd3d_conv3d_wgrad_workspace(int32_t cin, int32_t cout)
{
    return wgrad_shape(cin, cout) ? (int64_t)wgrad_bytes(cin, cout, wgrad_grid(INT32_MAX)) : -1;
}

// With no workspace given one is taken from the stream's allocator, whose
// default pool returns its memory to the system at every synchronisation: the
// first call after one then took 220 us of host time for a 24x16x8 layer, 15
// with memory at hand.
int mhd3d_conv3d_wgrad_ws(int32_t cin, int32_t cout, const void* x, const void* dy, float* dw, float* db, int32_t nx,
                          int32_t ny, int32_t nz, void* ws, int64_t ws_bytes, void* stream)
{
    if (!x || !dy || !dw || nx <= 0 || ny <= 0 || nz <= 0) return MHD3D_ERR_ARG;
    if (!aligned16(x) || !aligned16(dy) || !aligned16(ws) || !wgrad_shape(cin, cout)) return MHD3D_ERR_ARG;
    const int grid = wgrad_grid(((nx + WT - 1) / WT) * ny * nz);
    if (grid <= 0) return MHD3D_ERR_ARG;
    const size_t bytes = wgrad_bytes(cin, cout, grid);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    void* own = nullptr;
    if (ws && (ws_bytes < 0 || (size_t)ws_bytes < bytes)) return MHD3D_ERR_ARG;
    if (!ws && cudaMallocAsync(&own, bytes, st) != cudaSuccess) return MHD3D_ERR_CUDA;
    const cudaError_t e = launch_wgrad(cin, cout, x, dy, dw, db, nx, ny, nz, ws ? ws : own, st);
    const cudaError_t f = own ? cudaFreeAsync(own, st) : cudaSuccess;
    return e == cudaSuccess && f == cudaSuccess ? MHD3D_OK : MHD3D_ERR_CUDA;
}

int mhd3d_conv3d_wgrad(int32_t cin, int32_t cout, const void* x, const void* dy, float* dw, float* db, int32_t nx,
                       int32_t ny, int32_t nz, void* stream)
{
    return mhd3d_conv3d_wgrad_ws(cin, cout, x, dy, dw, db, nx, ny, nz, nullptr, 0, stream);
}

int mhd3d_conv3d_wtranspose(int32_t cin, int32_t cout, const void* w, void* wt, void* stream)
{
    if (!w || !wt || cin <= 0 || cout <= 0) return MHD3D_ERR_ARG;
    k_wtranspose<<<64, 256, 0, static_cast<cudaStream_t>(stream)>>>(static_cast<const __nv_bfloat16*>(w),
                                                                  static_cast<__nv_bfloat16*>(wt), cin, cout);
    return cudaGetLastError() == cudaSuccess ? MHD3D_OK : MHD3D_ERR_CUDA;
}

}  // extern "C"
