// Radiance-cache input encoding (shared by the encode kernel and the fused
// tcgen05 inference kernel): multiresolution hash grid of the normalised
// position (16 levels x 2 features, trilinear; Mueller et al., "Instant Neural
// Graphics Primitives", 2022) and one-blob encodings of the direction and
// normal in spherical coordinates (Mueller et al., "Neural Importance
// Sampling", 2019), packed as 128 bf16 values (64 words).
#pragma once

#include <cuda_bf16.h>
#include <cstdint>

#include "cache.h"
#include "device_common.cuh"

namespace bg {

// two floats -> bf16 pair (round to nearest even), low half first
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// ------------------------------------------------------------- encoding
__device__ __forceinline__ uint32_t grid_index(const NrcDev& C, int level, int x, int y, int z) {
    const uint32_t T = 1u << C.log2_T;
    const uint32_t n1 = uint32_t(C.res[level]) + 1u;
    if (uint64_t(n1) * n1 * n1 <= T) return uint32_t(x) + n1 * (uint32_t(y) + n1 * uint32_t(z));
    return (uint32_t(x) * 1u ^ uint32_t(y) * 2654435761u ^ uint32_t(z) * 805459861u) & (T - 1u);
}

struct GridCorner {
    int x0, y0, z0;
    float fx, fy, fz;
};
__device__ __forceinline__ GridCorner grid_cell(const NrcDev& C, int level, const float* u) {
    GridCorner g;
    const float N = float(C.res[level]);
    // (every rounding that reaches an encoded value is spelled out here and below: which
    // product the compiler would fuse into an add depends on the code around it)
    float x = __fmul_rn(u[0], N), y = __fmul_rn(u[1], N), z = __fmul_rn(u[2], N);
    float fx0 = fminf(floorf(x), N - 1.f), fy0 = fminf(floorf(y), N - 1.f), fz0 = fminf(floorf(z), N - 1.f);
    g.x0 = int(fx0); g.y0 = int(fy0); g.z0 = int(fz0);
    g.fx = __fsub_rn(x, fx0); g.fy = __fsub_rn(y, fy0); g.fz = __fsub_rn(z, fz0);
    return g;
}

__device__ __forceinline__ void norm_pos(const NrcDev& C, const float* f, float* u) {
#pragma unroll
    for (int k = 0; k < 3; ++k) u[k] = fminf(fmaxf((f[k] - C.bmin[k]) * C.bscale[k], 0.f), 1.f);
}

// one-blob encoding of v = a * m in [0,1] into 16 bf16 values, packed two per word:
// values first .. first + N - 1 of them
template <int N = 16>
__device__ __forceinline__ void one_blob(float a, float m, uint32_t* w, int first = 0) {
#pragma unroll
    for (int k = 0; k < N; k += 2) {
        const int b = first + k;
        const float d0 = __fmaf_rn(a, m, -((b + 0.5f) * (1.f / 16.f))), d1 = __fmaf_rn(a, m, -((b + 1.5f) * (1.f / 16.f)));
        w[k / 2] = pack_bf16(__expf(-d0 * d0 * 128.f), __expf(-d1 * d1 * 128.f));
    }
}

// polar angle (radians) and azimuth in [0,1]
__device__ __forceinline__ void sph(float x, float y, float z, float& th, float& ph) {
    th = acosf(fminf(fmaxf(z, -1.f), 1.f));
    ph = __fmaf_rn(atan2f(y, x), 0.5f / BG_PI, 0.5f);
}
constexpr float kPolar = 1.f / BG_PI;   // polar angle to [0,1]

// The encoded row of one raw query record (16 floats: position, outgoing
// direction, shading normal, roughness, albedo) is 64 words: 0-15 the grid
// features, 16-47 the four one-blobs, 48-49 roughness and albedo, 50 a constant
// 1, the rest 0.  It is built by a pair of adjacent lanes, h = lane & 1:
//   g  words 8h .. 8h + 7 (levels 8h .. 8h + 7)
//   b  words 16 + 16h .. 31 + 16h (h = 0: the direction's one-blobs, 1: the normal's)
//   t  words 48-51, the same in both lanes
// What bounds the encoding is the 128 table entries a row gathers: the L1
// looks up about one distinct 128-byte line per cycle, and one lane per row
// touches 32 lines per load.  The two corners of a cell that differ in x lie
// in one line (adjacent entries in a dense level; indices that differ in a few
// low bits in a hashed one, whose x factor is 1), so lane h of a pair loads
// the four corners of x offset h and a load touches 16 lines.  The lanes then
// exchange their corners so that lane h sums feature h of every level over the
// corners in the order x, y, z of one lane alone: the same sums, bit for bit.
// Both lanes of a pair must call it, with all 32 lanes of the warp converged.
// Measured: queries as k_nrc_infer_tc says, training rows as k_nrc_encode does.
// The loads are plain ones, of two levels before either's sums: with __ldg and one
// level at a time the compiler kept their order and 128 registers, and queries
// of 200,003 / 1,000,000 / 5,000 rows took 92 / 409 / 17.4 us instead of 85 / 382 / 16.5.
__device__ __forceinline__ void gather_level(const NrcDev& C, int l, const float* u, int h, float2 (&v)[4]) {
    const GridCorner g = grid_cell(C, l, u);
    const float2* table = reinterpret_cast<const float2*>(C.grid) + (size_t(l) << C.log2_T);
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = table[grid_index(C, l, g.x0 + h, g.y0 + (k & 1), g.z0 + (k >> 1))];
}
__device__ __forceinline__ float sum_level(const NrcDev& C, int l, const float* u, int h, const float2 (&v)[4]) {
    const GridCorner g = grid_cell(C, l, u);
    float a = 0.f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float wy = (k & 1) ? g.fy : 1.f - g.fy, wz = (k >> 1) ? g.fz : 1.f - g.fz;
        const float got = __shfl_xor_sync(0xffffffffu, h ? v[k].x : v[k].y, 1);   // the partner's feature of this corner
        const float own = h ? v[k].y : v[k].x;
        a = fmaf((1.f - g.fx) * wy * wz, h ? got : own, a);
        a = fmaf(g.fx * wy * wz, h ? own : got, a);
    }
    return a;
}
// two levels: lane 0 keeps the features of level lo (its own feature 0, the partner's 1), lane 1 those of hi
__device__ __forceinline__ uint32_t encode_levels(const NrcDev& C, int lo, int hi, const float* u, int h) {
    float2 v0[4], v1[4];
    gather_level(C, lo, u, h, v0);
    gather_level(C, hi, u, h, v1);
    const float a = sum_level(C, lo, u, h, v0), b = sum_level(C, hi, u, h, v1);
    const float got = __shfl_xor_sync(0xffffffffu, h ? a : b, 1);
    return h ? pack_bf16(got, b) : pack_bf16(a, got);
}

__device__ __forceinline__ void encode_pair(const NrcDev& C, const float* __restrict__ f, int h, uint32_t (&g)[8],
                                            uint32_t (&b)[16], uint32_t (&t)[4]) {
    const float4* f4 = reinterpret_cast<const float4*>(f);
    const float4 q0 = __ldg(f4), q1 = __ldg(f4 + 1), q2 = __ldg(f4 + 2), q3 = __ldg(f4 + 3);
    const float pos[3] = {q0.x, q0.y, q0.z};
    float u[3];
    norm_pos(C, pos, u);
#pragma unroll
    for (int l = 0; l < kNrcLevels / 2; ++l) g[l] = encode_levels(C, l, l + kNrcLevels / 2, u, h);
    float th, ph;
    sph(h ? q1.z : q0.w, h ? q1.w : q1.x, h ? q2.x : q1.y, th, ph);
    one_blob(th, kPolar, b);
    one_blob(ph, 1.f, b + 8);
    t[0] = pack_bf16(q2.y, q2.z);
    t[1] = pack_bf16(q2.w, q3.x);
    t[2] = pack_bf16(1.f, 0.f);
    t[3] = 0u;
}

// Scatters a row's gradient (dx, dy) of level l's features over the table: the
// four corners of x offset h, so that a pair of lanes covers the cell and meets
// in one sector (see gather_level).
__device__ __forceinline__ void scatter_level(const NrcDev& C, int l, const float* u, int h, float dx, float dy) {
    const GridCorner g = grid_cell(C, l, u);
    float* table = C.grid_grad + (size_t(l) << C.log2_T) * 2;
    const float wx = h ? g.fx : 1.f - g.fx;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const float w = wx * ((k & 1) ? g.fy : 1.f - g.fy) * ((k >> 1) ? g.fz : 1.f - g.fz);
        const uint32_t idx = grid_index(C, l, g.x0 + h, g.y0 + (k & 1), g.z0 + (k >> 1));
        atomicAdd(reinterpret_cast<float2*>(table + size_t(idx) * 2), make_float2(w * dx, w * dy));   // both features, one vector atomic
    }
}

}  // namespace bg
