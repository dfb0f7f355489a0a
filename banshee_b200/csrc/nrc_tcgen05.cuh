// Radiance-cache MLP inference on the 5th-generation tensor cores (tcgen05).
//
// Persistent CTAs; each group of 128 threads works on one tile of 128 query
// rows at a time (the inference kernel's layout is described above it):
//   * the six weight matrices live in shared memory for the whole kernel, in
//     the K-major no-swizzle canonical layout of the UMMA shared-memory
//     descriptors: 8x8 bf16 core matrices of 128 contiguous bytes, core
//     matrices adjacent in K 128 bytes apart (LBO), 8-row groups K/8 * 128
//     bytes apart (SBO);
//   * the activation tile (A operand, 128 x K bf16) is in the same layout;
//   * the fp32 accumulator (128 lanes x 64 columns) is in tensor memory;
//   * thread 0 issues tcgen05.mma (M = 128, N = 64 or 16, K = 16 per
//     instruction) and commits to an mbarrier; every thread then reads its own
//     accumulator row (TMEM lane = tile row) with tcgen05.ld, applies ReLU,
//     rounds to bf16 and writes the next layer's A row.
// Waits on the mbarrier are bounded (NrcDev::wait_polls polls, 0 = the
// default of 2^24): on timeout the kernel raises BG_FLAG_TIMEOUT, stops, gives
// its outstanding MMA group one more wait with the default bound, releases
// its tensor memory and returns.
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

#include "cache.h"
#include "nrc_encode.cuh"

namespace bg {

constexpr int kTcRows = 128;                               // rows per tile (UMMA M)
constexpr int kTcW0 = 0;                                   // [64 x 128]
constexpr int kTcW1 = kTcW0 + 64 * 128 * 2;                // 4 x [64 x 64]
constexpr int kTcW5 = kTcW1 + 4 * 64 * 64 * 2;             // [16 x 64]
constexpr int kTcA0 = kTcW5 + 16 * 64 * 2;                 // end of the weights, first tile
constexpr uint32_t kTcWaitLimit = 1u << 24;                // mbarrier polls before giving up

// byte offset of core-matrix row `r`, 16-byte chunk `kc` in a K-major tile with KC chunks per row
__host__ __device__ constexpr uint32_t tc_off(int r, int kc, int KC) {
    return uint32_t((r >> 3) * (KC * 128) + kc * 128 + (r & 7) * 16);
}

__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return uint64_t((saddr >> 4) & 0x3FFFu) | (uint64_t((lbo >> 4) & 0x3FFFu) << 16) |
           (uint64_t((sbo >> 4) & 0x3FFFu) << 32) | (uint64_t(1) << 46);   // version 1, no swizzle
}

// kind::f16 instruction descriptor: bf16 x bf16 -> f32, A K-major, B K-major
// (b_mn = false) or MN-major (b_mn = true), M = 128
__host__ __device__ constexpr uint32_t tc_idesc(int N, bool b_mn = false) {
    return (1u << 4) | (1u << 7) | (1u << 10) | (b_mn ? (1u << 16) : 0u) | (uint32_t(N >> 3) << 17) |
           (uint32_t(kTcRows >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n"
        :: "r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}

__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(bar) : "memory");
}

__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// true once the phase of parity `phase` of the mbarrier has completed; false
// after `polls` polls (0 = kTcWaitLimit).  The first poll is a non-blocking
// test_wait, the rest are try_wait (which may suspend the thread briefly), so
// a budget of one poll gives up at once unless the phase is already complete.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t phase, uint32_t polls = 0) {
    const uint32_t limit = polls ? polls : kTcWaitLimit;
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done) : "r"(bar), "r"(phase) : "memory");
    if (done) return true;
    for (uint32_t it = 1; it < limit; ++it) {
        asm volatile(
            "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
            : "=r"(done) : "r"(bar), "r"(phase) : "memory");
        if (done) return true;
    }
    return false;
}

// 16 consecutive fp32 columns of this thread's TMEM lane
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// 8 of them
__device__ __forceinline__ void tc_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ uint32_t tc_pack(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

// weight matrix [N][K] (row-major bf16 in global memory) -> canonical K-major smem tile
__device__ __forceinline__ void tc_load_weights(const __nv_bfloat16* __restrict__ w, int N, int K, unsigned char* dst) {
    const int KC = K / 8;
    for (int i = threadIdx.x; i < N * KC; i += blockDim.x) {
        const int n = i / KC, kc = i % KC;
        *reinterpret_cast<uint4*>(dst + tc_off(n, kc, KC)) = *reinterpret_cast<const uint4*>(w + size_t(n) * K + kc * 8);
    }
}

// Inference from raw query records (16 floats each).  CTAs of kTiGroups groups
// of 256 threads; each group runs its own 128-row tiles with its own mbarrier,
// its own 64 TMEM columns and its own 32 KB activation slot: the 128-wide input
// tile, whose first 16 KB the 64-wide hidden tiles reuse once the layer-0 MMA
// has completed.  Groups synchronise on named barriers (ids 1..kTiGroups), the
// CTA only at start and end.
//   encode   a pair of lanes per row (encode_pair), straight into the A tile:
//            no encoded row goes through global memory
//   layers   warps w and w + 4 of a group share TMEM lanes 32 (w % 4) .. + 31
//            and split the columns
// The kernel is bound by the encoding's gathers through L1 and L2; encode_pair
// says how they are paired.  Two groups per SM overlap one group's MMA chain
// with the other's gathers.  Measured for 200,003 / 1,000,000 / 5,000 rows
// (tables of 2^19 entries): one lane per row, 128 threads per tile, 109 / 500 /
// 18.5 us; pairs of lanes, 256 threads, two CTAs of one group 85 / 382 / 16.5;
// one CTA of two groups 94 / 430 / 16.5, of three 90 / 410 / 16.5 (their tiles
// spread over the SMs), one group per SM some 120 / 565.
constexpr int kTiGroups = 1;
constexpr int kTiCtasPerSm = 2;                            // CTAs per SM in the grid
constexpr int kTiGroupThreads = 256;
constexpr int kTiThreads = kTiGroupThreads * kTiGroups;
constexpr int kTiSlot0 = kTcA0;                            // group g's slot at kTiSlot0 + g * kTiSlotBytes
constexpr int kTiSlotBytes = kTcRows * 128 * 2;            // 32 KB: the [128 x 128] input tile
constexpr int kTiBar = kTiSlot0 + kTiGroups * kTiSlotBytes;   // kTiGroups mbarriers + TMEM base
constexpr int kTiSmem = kTiBar + 8 * kTiGroups + 16;
constexpr uint32_t kTiCols = kTiGroups == 1 ? 64 : kTiGroups == 2 ? 128 : 256;   // TMEM columns (a power of two)
// words 51-63 of an encoded row are 0: the layer-0 product stops at K = 112
constexpr int kTiK0 = 112;
static_assert(kTiSmem <= 227 * 1024, "inference shared memory");
static_assert(kTiGroups * 64 <= int(kTiCols), "TMEM allocation");

__device__ __forceinline__ void group_sync(int g) {
    asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(kTiGroupThreads) : "memory");
}

__global__ void __launch_bounds__(kTiThreads, kTiCtasPerSm) k_nrc_infer_tc(NrcDev C, const int* n_dev, int64_t n_static,
                                                                float4* __restrict__ out,
                                                                unsigned* __restrict__ errflags,
                                                                const float* __restrict__ feat) {
    extern __shared__ __align__(1024) unsigned char tc_smem[];
    unsigned char* smem = tc_smem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int g = tid / kTiGroupThreads;  // tile group
    const int gw = warp & 7;              // warp within the group
    const int row = (gw & 3) * 32 + lane; // TMEM lane = tile row of this thread in the layers
    const int half = gw >> 2;             // its half of the columns
    const uint32_t sbase = uint32_t(__cvta_generic_to_shared(smem));
    const uint32_t bar = sbase + kTiBar + 8 * g;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kTiBar + 8 * kTiGroups);
    // set by a wait that gave up, one flag per mbarrier parity: a thread already in the
    // next layer must not change the flag that its group still reads for this one
    __shared__ int abort_flag[kTiGroups][2];
    unsigned char* slot = smem + kTiSlot0 + g * kTiSlotBytes;
    const uint32_t sslot = sbase + kTiSlot0 + g * kTiSlotBytes;

    tc_load_weights(C.wb + kNrcW0, 64, 128, smem + kTcW0);
    for (int l = 0; l < 4; ++l) tc_load_weights(C.wb + kNrcW1 + l * 4096, 64, 64, smem + kTcW1 + l * 8192);
    tc_load_weights(C.wb + kNrcW5, 16, 64, smem + kTcW5);
    if (tid < kTiGroups) {
        abort_flag[tid][0] = abort_flag[tid][1] = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sbase + kTiBar + 8 * tid) : "memory");
    }
    if (tid == 0) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(sbase + kTiBar + 8 * kTiGroups), "r"(kTiCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot + uint32_t(64 * g);           // this group's accumulator columns
    const uint32_t trow = tmem + (uint32_t((gw & 3) * 32) << 16);  // this warp's 32 lanes

    const int64_t n = n_dev ? int64_t(*n_dev) : n_static;
    const int64_t ntiles = (n + kTcRows - 1) / kTcRows;
    uint32_t phase = 0;
    bool gave_up = false;
    for (int64_t tile = int64_t(blockIdx.x) * kTiGroups + g; tile < ntiles && !gave_up; tile += int64_t(gridDim.x) * kTiGroups) {
        const int64_t row0 = tile * kTcRows;
        {
            // lanes 2r, 2r + 1 of a warp encode row r of its 16; rows past n repeat the last one (not written out)
            const int r = gw * 16 + (lane >> 1), h = lane & 1;
            const int64_t gr = row0 + r < n ? row0 + r : n - 1;
            uint32_t wg[8], wb[16], wt[4];
            encode_pair(C, feat + size_t(gr) * kNrcFeatFloats, h, wg, wb, wt);
#pragma unroll
            for (int k = 0; k < 2; ++k)
                *reinterpret_cast<uint4*>(slot + tc_off(r, 2 * h + k, 16)) =
                    make_uint4(wg[4 * k], wg[4 * k + 1], wg[4 * k + 2], wg[4 * k + 3]);
#pragma unroll
            for (int k = 0; k < 4; ++k)
                *reinterpret_cast<uint4*>(slot + tc_off(r, 4 + 4 * h + k, 16)) =
                    make_uint4(wb[4 * k], wb[4 * k + 1], wb[4 * k + 2], wb[4 * k + 3]);
            *reinterpret_cast<uint4*>(slot + tc_off(r, 12 + h, 16)) =
                h ? make_uint4(0u, 0u, 0u, 0u) : make_uint4(wt[0], wt[1], wt[2], wt[3]);
        }
        tc_fence_async_smem();
        tc_fence_before();
        group_sync(g);
        for (int layer = 0; layer < 6; ++layer) {
            if (tid % kTiGroupThreads == 0) {
                tc_fence_after();
                const int KC = layer == 0 ? 16 : 8, steps = layer == 0 ? kTiK0 / 16 : 4;
                const uint32_t b = sbase + (layer == 0 ? kTcW0 : layer < 5 ? kTcW1 + (layer - 1) * 8192 : kTcW5);
                const uint32_t idesc = tc_idesc(layer < 5 ? 64 : 16);
                for (int s = 0; s < steps; ++s)
                    tc_mma(tmem, tc_desc(sslot + s * 256, 128, KC * 128), tc_desc(b + s * 256, 128, KC * 128), idesc,
                           s > 0 ? 1u : 0u);
                tc_commit(bar);
            }
            const bool done = __all_sync(0xffffffffu, tc_wait(bar, phase, C.wait_polls));
            if (!done) {
                atomicOr(errflags, BG_FLAG_TIMEOUT);
                abort_flag[g][phase] = 1;
            }
            tc_fence_after();
            if (done && layer < 5) {
                // ReLU, bf16, into the hidden tile (the slot's first 16 KB: the MMA that read them is done)
#pragma unroll
                for (int c2 = 0; c2 < 2; ++c2) {
                    const int c4 = 2 * half + c2;
                    float v[16];
                    tc_ld16(trow + uint32_t(c4 * 16), v);
                    uint4 p0, p1;
                    p0.x = tc_pack(fmaxf(v[0], 0.f), fmaxf(v[1], 0.f));
                    p0.y = tc_pack(fmaxf(v[2], 0.f), fmaxf(v[3], 0.f));
                    p0.z = tc_pack(fmaxf(v[4], 0.f), fmaxf(v[5], 0.f));
                    p0.w = tc_pack(fmaxf(v[6], 0.f), fmaxf(v[7], 0.f));
                    p1.x = tc_pack(fmaxf(v[8], 0.f), fmaxf(v[9], 0.f));
                    p1.y = tc_pack(fmaxf(v[10], 0.f), fmaxf(v[11], 0.f));
                    p1.z = tc_pack(fmaxf(v[12], 0.f), fmaxf(v[13], 0.f));
                    p1.w = tc_pack(fmaxf(v[14], 0.f), fmaxf(v[15], 0.f));
                    *reinterpret_cast<uint4*>(slot + tc_off(row, 2 * c4, 8)) = p0;
                    *reinterpret_cast<uint4*>(slot + tc_off(row, 2 * c4 + 1, 8)) = p1;
                }
                tc_fence_async_smem();
            } else if (done && half == 0) {
                float v[16];
                tc_ld16(trow, v);
                if (row0 + row < n) out[row0 + row] = make_float4(v[0], v[1], v[2], 0.f);
            }
            tc_fence_before();
            group_sync(g);
            gave_up = abort_flag[g][phase] != 0;   // the same in every thread of the group
            if (gave_up) break;
            phase ^= 1u;
        }
    }
    // after a timeout, give the group's outstanding MMA one more bounded wait before the TMEM is freed
    if (gave_up && tid % kTiGroupThreads == 0) tc_wait(bar, phase);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(*tmem_slot), "r"(kTiCols) : "memory");
    }
}


// ------------------------------------------------------------- training
// The gradients of one Adam step's encoded rows in one kernel: forward, loss,
// backward, the six weight gradients and the hash grid's.  One CTA per SM; a
// tile of 128 rows stays on the chip from its inputs to its gradients:
//   X            the encoded rows (k_nrc_encode), K-major, 16 chunks per row
//   P1, P2, P3   the hidden activations [H0 | H1], [H2 | H3], [H4 | 0], laid out as X
//   dZ           two buffers for the layer-output gradients, by the layer's parity
//   dZ5          the output layer's
// Forward: H_l = relu(A_l W_l) with A_0 = X, A_l = H_{l-1}.  Backward products
// dH = dZ W need B = W with the layer's inputs as N: the forward weight tiles hold
// W[out][in] in 8x8 core matrices of 8 rows (out) x 16 contiguous bytes (in), which
// is exactly an MN-major B core matrix (8 K-rows x 8 contiguous N elements), so
// the backward reads them through MN-major descriptors (SBO = 128 bytes between
// groups of 8 inputs, LBO = KC * 128 bytes between groups of 8 outputs).
// Weight gradients dW_l[o][i] = sum_s A_l[s][i] dZ_l[s][o] have the rows as K:
// both tiles read as MN-major operands (LBO = the stride between groups of 8
// rows, SBO = 128 bytes between groups of 8 features).  Every product has M =
// 128: the two layers of a P tile are multiplied by each one's dZ in turn, and
// the half of the lanes that belongs to the other layer is not used.  They are
// issued behind the backward product that the chain waits for, accumulate in
// TMEM over the CTA's tiles (cols 64 + 64 l for layer l, transposed, D[i][o]),
// and are added to global memory once per CTA.
// Threads: warp w reads TMEM lanes 32 (w % 4) .. + 31 (lane = tile row), 16
// columns (w / 4) .. of the 64; each keeps its ReLU masks in registers.  A step of
// 16,384 rows is one tile per SM and a chain of twelve dependent products, so
// it is bound by latency: 4 us of weights and TMEM, 9 of the chain, 11 of the
// scatter's atomics (L2), 4 of the weight gradients' atomics.
// Forward and backward, weight gradients and scatter as kernels of their own,
// with the activations and gradients through global memory, took 25 + 19 + 17
// us at 16,384 rows and 2^19 entries per level; this one takes 35.
constexpr int kTtThreads = 512;
constexpr int kTtX = kTcA0;                                // X, P1, P2, P3
constexpr int kTtTile = kTcRows * 128 * 2;
constexpr int kTtDz = kTtX + 4 * kTtTile;                  // two of [128 x 64]
constexpr int kTtDzB = kTcRows * 64 * 2;
constexpr int kTtDz5 = kTtDz + 2 * kTtDzB;                 // [128 x 16]
constexpr int kTtBar = kTtDz5 + kTcRows * 16 * 2;          // mbarrier (8 B) + TMEM base (4 B)
constexpr int kTtSmem = kTtBar + 16;
constexpr uint32_t kTtCols = 512;                          // TMEM columns: accumulator 0-63, weight gradients 64-399
static_assert(kTtSmem <= 227 * 1024, "training shared memory");

struct TcTrainArgs {
    const float* feat;           // raw records of the whole set; this step's rows start at `offset`
    const __nv_bfloat16* X;      // encoded rows of this step [B][128]
    const float4* target;        // targets of the whole set
    float* dW;                   // [kNrcParams], accumulated
    float* loss;
    int* step;                   // Adam's step count, advanced for the update that follows (null: none follows)
    int B;
};

__global__ void __launch_bounds__(kTtThreads, 1) k_nrc_train_tc(NrcDev C, TcTrainArgs T, const int* n_dev, int offset,
                                                                int limit, unsigned* __restrict__ errflags) {
    extern __shared__ __align__(1024) unsigned char tt_smem[];
    unsigned char* smem = tt_smem;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int row = (warp & 3) * 32 + lane, cg = warp >> 2;   // TMEM lane, group of 16 columns
    const uint32_t sbase = uint32_t(__cvta_generic_to_shared(smem));
    const uint32_t bar = sbase + kTtBar;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kTtBar + 8);
    // set by a wait that gave up, one flag per mbarrier parity: a thread already in the
    // next wait must not change the flag that others still read for this one
    __shared__ int abort_flag[2];

    if (T.step && blockIdx.x == 0 && tid == 0) *T.step += 1;
    int n = n_dev ? *n_dev - offset : T.B;
    if (limit > 0 && n > limit) n = limit;
    if (n < 0) n = 0;
    const int ntiles = (n + kTcRows - 1) / kTcRows;
    if (int(blockIdx.x) >= ntiles) return;   // (uniform per CTA, before any TMEM allocation)
    const float invn = 1.f / (3.f * float(n));

    tc_load_weights(C.wb + kNrcW0, 64, 128, smem + kTcW0);
    for (int l = 0; l < 4; ++l) tc_load_weights(C.wb + kNrcW1 + l * 4096, 64, 64, smem + kTcW1 + l * 8192);
    tc_load_weights(C.wb + kNrcW5, 16, 64, smem + kTcW5);
    for (int v = tid; v < kTcRows * 8; v += kTtThreads)      // the zero half of P3, once
        *reinterpret_cast<uint4*>(smem + kTtX + 3 * kTtTile + tc_off(v & 127, 8 + (v >> 7), 16)) = make_uint4(0u, 0u, 0u, 0u);
    if (tid == 0) {
        abort_flag[0] = abort_flag[1] = 0;
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     :: "r"(sbase + kTtBar + 8), "r"(kTtCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    const uint32_t trow = tmem + (uint32_t((warp & 3) * 32) << 16);
    uint32_t phase = 0;
    float lsum = 0.f;
    bool first = true, gave_up = false;

    // the chain's next product into columns 0 .. N - 1: the tile at `a` (K-major, a_sbo bytes
    // between its 8-row groups, K / 16 = steps) by the weights at `b`; thread 0 only
    auto product = [&](uint32_t a, uint32_t a_sbo, int steps, uint32_t b, uint32_t b_lbo, uint32_t b_sbo, uint32_t b_kstep,
                       uint32_t idesc) {
        tc_fence_after();
        for (int s = 0; s < steps; ++s)
            tc_mma(tmem, tc_desc(a + s * 256, 128, a_sbo), tc_desc(b + s * b_kstep, b_lbo, b_sbo), idesc, s > 0 ? 1u : 0u);
        tc_commit(bar);
    };
    // a weight gradient into the accumulator at `col`: activations at `a`, dZ at `b` (b_lbo
    // bytes between its 8-row groups); thread 0 only
    auto wgrad = [&](uint32_t a, uint32_t b, uint32_t b_lbo, int N, uint32_t col) {
        const uint32_t idesc = tc_idesc(N, true) | (1u << 15);   // A and B MN-major
        for (int k = 0; k < kTcRows / 16; ++k)
            tc_mma(tmem + col, tc_desc(a + k * 2 * 2048, 2048, 128), tc_desc(b + k * 2 * b_lbo, b_lbo, 128), idesc,
                   (first && k == 0) ? 0u : 1u);
    };
    // every thread waits for the last commit; false (in all of them) after a timeout
    auto wait = [&]() {
        if (!tc_wait(bar, phase, C.wait_polls)) {
            atomicOr(errflags, BG_FLAG_TIMEOUT);
            abort_flag[phase] = 1;
        }
        tc_fence_after();
        __syncthreads();
        gave_up = abort_flag[phase] != 0;
        phase ^= 1u;
        return !gave_up;
    };
    // shared memory written, TMEM read: thread 0 may issue the next product
    auto ready = [&]() {
        tc_fence_async_smem();
        tc_fence_before();
        __syncthreads();
    };
    auto pack16 = [&](const float (&v)[16], uint4& p0, uint4& p1) {
        p0 = make_uint4(tc_pack(v[0], v[1]), tc_pack(v[2], v[3]), tc_pack(v[4], v[5]), tc_pack(v[6], v[7]));
        p1 = make_uint4(tc_pack(v[8], v[9]), tc_pack(v[10], v[11]), tc_pack(v[12], v[13]), tc_pack(v[14], v[15]));
    };
    const uint32_t sX = sbase + kTtX, sP = sX + kTtTile, sDz = sbase + kTtDz, sDz5 = sbase + kTtDz5;

    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int row0 = tile * kTcRows;
        const bool live = row0 + row < n;
        // ---- the encoded rows; those past n repeat the last one (their dZ is zero)
        for (int j = 0; j < 4; ++j) {                        // eight lanes load one core matrix: no bank conflicts
            const int r = warp * 8 + (lane & 7), kc = j * 4 + (lane >> 3);
            *reinterpret_cast<uint4*>(smem + kTtX + tc_off(r, kc, 16)) =
                *reinterpret_cast<const uint4*>(T.X + size_t(min(row0 + r, n - 1)) * kNrcIn + kc * 8);
        }
        ready();
        uint32_t mask[5];
        // ---- forward: hidden layers
#pragma unroll
        for (int l = 0; l < 5; ++l) {
            if (tid == 0) {
                if (l == 0) product(sX, 2048, 8, sbase + kTcW0, 128, 16 * 128, 256, tc_idesc(64));
                else product(sP + ((l - 1) >> 1) * kTtTile + ((l - 1) & 1) * 1024, 2048, 4, sbase + kTcW1 + (l - 1) * 8192, 128,
                             8 * 128, 256, tc_idesc(64));
            }
            if (!wait()) break;
            float v[16];
            tc_ld16(trow + uint32_t(cg * 16), v);
            mask[l] = 0u;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                if (v[j] > 0.f) mask[l] |= 1u << j;
                v[j] = fmaxf(v[j], 0.f);
            }
            uint4 p0, p1;
            pack16(v, p0, p1);
            unsigned char* dst = smem + kTtX + (1 + (l >> 1)) * kTtTile;
            *reinterpret_cast<uint4*>(dst + tc_off(row, 8 * (l & 1) + 2 * cg, 16)) = p0;
            *reinterpret_cast<uint4*>(dst + tc_off(row, 8 * (l & 1) + 2 * cg + 1, 16)) = p1;
            ready();
        }
        if (gave_up) break;
        // ---- output layer and the loss gradient (columns 0..2 of 16)
        if (tid == 0) product(sP + 2 * kTtTile, 2048, 4, sbase + kTcW5, 128, 8 * 128, 256, tc_idesc(16));
        if (!wait()) break;
        if (cg == 0) {
            float v[16], g[16];
            tc_ld16(trow, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) g[j] = 0.f;
            if (live) {
                const float* y = reinterpret_cast<const float*>(T.target + size_t(offset) + size_t(row0 + row));
#pragma unroll
                for (int j = 0; j < 3; ++j) {
                    const float p = v[j], den = p * p + 0.01f, d = p - y[j];
                    lsum += d * d / den;
                    g[j] = 2.f * d / den * invn;
                }
            }
            uint4 z0, z1;
            pack16(g, z0, z1);
            *reinterpret_cast<uint4*>(smem + kTtDz5 + tc_off(row, 0, 2)) = z0;
            *reinterpret_cast<uint4*>(smem + kTtDz5 + tc_off(row, 1, 2)) = z1;
        }
        ready();
        // ---- backward: dH_{l-1} = dZ_l W_l; each dW_l behind the product the chain waits for.
        // A dZ buffer is written again two layers on, when the wait for the layer between
        // has covered the weight gradient that read it.
        if (tid == 0) {
            product(sDz5, 256, 1, sbase + kTcW5, 8 * 128, 128, 2 * 8 * 128, tc_idesc(64, true));
            wgrad(sP + 2 * kTtTile, sDz5, 256, 16, 384);
        }
#pragma unroll
        for (int l = 4; l >= 0; --l) {
            if (!wait()) break;
            float v[16];
            tc_ld16(trow + uint32_t(cg * 16), v);
#pragma unroll
            for (int j = 0; j < 16; ++j)
                if (!((mask[l] >> j) & 1u)) v[j] = 0.f;              // dZ_l = dH_l masked by ReLU'(z_l)
            uint4 p0, p1;
            pack16(v, p0, p1);
            unsigned char* dst = smem + kTtDz + (l & 1) * kTtDzB;
            *reinterpret_cast<uint4*>(dst + tc_off(row, 2 * cg, 8)) = p0;
            *reinterpret_cast<uint4*>(dst + tc_off(row, 2 * cg + 1, 8)) = p1;
            ready();
            if (tid == 0) {
                const uint32_t z = sDz + (l & 1) * kTtDzB;
                if (l > 0) {
                    product(z, 1024, 4, sbase + kTcW1 + (l - 1) * 8192, 8 * 128, 128, 2 * 8 * 128, tc_idesc(64, true));
                    wgrad(sP + ((l - 1) >> 1) * kTtTile, z, 1024, 64, 64 + 64 * l);
                } else {   // dX = dZ0 W0, hash-grid columns 0..31 only
                    product(z, 1024, 4, sbase + kTcW0, 16 * 128, 128, 2 * 16 * 128, tc_idesc(32, true));
                    wgrad(sX, z, 1024, 64, 64);
                }
            }
        }
        if (gave_up || !wait()) break;
        first = false;
        // ---- the tile's last weight gradients complete behind the scatter of dX
        if (tid == 0) tc_commit(bar);
        {
            float d[8], u[3];
            tc_ld8(trow + uint32_t(cg * 8), d);              // levels 4 cg .. 4 cg + 3 of this row
            const float* f = T.feat + (size_t(offset) + size_t(min(row0 + row, n - 1))) * kNrcFeatFloats;
            const float fr[3] = {f[0], f[1], f[2]};
            norm_pos(C, fr, u);
            for (int k = 0; k < 2; ++k) {                    // the pair of lanes scatters its two rows in turn
                const int src = (lane & ~1) | k;
                const float uk[3] = {__shfl_sync(0xffffffffu, u[0], src), __shfl_sync(0xffffffffu, u[1], src),
                                     __shfl_sync(0xffffffffu, u[2], src)};
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float dx = __shfl_sync(0xffffffffu, d[2 * j], src), dy = __shfl_sync(0xffffffffu, d[2 * j + 1], src);
                    if (dx != 0.f || dy != 0.f) scatter_level(C, 4 * cg + j, uk, lane & 1, dx, dy);
                }
            }
        }
        tc_fence_before();
        if (!wait()) break;
    }
    if (!gave_up) {
        const int i = row;                                   // TMEM lane = input feature
        auto out = [&](uint32_t col0, float* dst, int ld, int ioff) {
            float v[16];
            tc_ld16(trow + col0, v);
#pragma unroll
            for (int j = 0; j < 16; ++j) atomicAdd(dst + size_t(j) * ld + (i - ioff), v[j]);
        };
        const uint32_t c = uint32_t(cg * 16);                // this warp's 16 outputs o
        out(64 + c, T.dW + kNrcW0 + size_t(c) * 128, 128, 0);                          // dW0[o][i], i = 0..127
        const int up = i >= 64 ? 1 : 0;                                                // (uniform per warp)
        out(128 + 64 * up + c, T.dW + kNrcW1 + up * 4096 + size_t(c) * 64, 64, 64 * up);         // dW1, dW2
        out(256 + 64 * up + c, T.dW + kNrcW1 + (2 + up) * 4096 + size_t(c) * 64, 64, 64 * up);   // dW3, dW4
        if (cg == 0 && !up) out(384, T.dW + kNrcW5, 64, 0);                            // dW5
    }
    for (int off = 16; off > 0; off >>= 1) lsum += __shfl_down_sync(0xffffffffu, lsum, off);
    if (lane == 0 && lsum != 0.f) atomicAdd(T.loss, lsum);
    // after a timeout, give the outstanding products, the weight gradients issued behind the
    // last commit among them, one more bounded wait each before their TMEM is freed
    if (gave_up && tid == 0) {
        tc_commit(bar);
        tc_wait(bar, phase ^ 1u);
        tc_wait(bar, phase);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(tmem), "r"(kTtCols) : "memory");
    }
}

}  // namespace bg
