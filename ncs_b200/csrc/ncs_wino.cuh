// ncs_wino.cuh -- the warm-start network's 32 -> 32 channel 3x3 convolutions by
// Winograd's minimal filtering F(2x2, 3x3) (S. Winograd, "Arithmetic Complexity
// of Computations", SIAM 1980; A. Lavin, S. Gray, "Fast Algorithms for
// Convolutional Neural Networks", CVPR 2016), FP32 throughout:
//   Y = A' [ (G g G') . (B' d B) ] A
// per 4x4 input patch d and 2x2 output patch Y.  A 16x16 tile is 64 patches; at
// each of the 16 points the products are a 64 x 32 x 32 GEMM, 2.25 times fewer
// multiply-adds than the direct form.  Sums run over 32 channels instead of 288
// products, so the rounding error is below the direct sum's (one layer against
// FP64: 1.2e-7 relative, direct 2.0e-7).
//
// A CTA owns a tile and takes it in chunks of CP patches (16 CP threads): a
// thread transforms two patches of a channel, a quarter-warp runs 8 patches x 32
// output channels of one point's GEMM, and a thread transforms two output
// patches back, which it keeps in registers until the whole tile is done, so a
// layer can run in place.
//
// What bounds it: the FMA pipe and shared memory together.  A warp's 128-bit
// shared load takes 4 cycles of the SM's 128-byte path (2 where each
// quarter-warp reads one address), so a lane's 8 x 4 products per channel need 8
// cycles of it for 32 of its scheduler's FMA cycles, i.e. as many for the SM's
// four schedulers.  A 4 x 4 block per lane needed 6 for 16 and ran 1.5 times
// slower.
#pragma once

#include "ncs_warp_common.cuh"

namespace ncsb {
namespace wino {

using warp::fma2;
using warp::splat;

constexpr int kC = 32;  // channels in and out
// Zero-bordered planes: rows 24 floats apart and planes 434, so that the 64-bit
// patch reads are free of bank conflicts with the lanes over patches (two patch
// rows fall on different half-banks) and with the lanes over channels (434 = 18
// mod 32).
constexpr int kRow = 24;
constexpr int kPlane = 434;
constexpr int kPlanes = kC * kPlane;
// U[point][ci][co], V[point][ci][patch] and M[point][patch][co] (in V's place)
constexpr int kU = 16 * kC * kC;
constexpr int kV(int cp) { return 16 * kC * cp; }

// U = G g G' of wt[ci][tap][co] (flip: of the input gradient's filter, whose
// channels are exchanged and whose taps are reversed), in FP64, rounded once.
__device__ __forceinline__ void weights(float* U, const float* __restrict__ wt, bool flip) {
    for (int idx = threadIdx.x; idx < kC * kC; idx += blockDim.x) {
        const int ci = idx >> 5, co = idx & 31;
        double g[3][3], t[4][3];
#pragma unroll
        for (int k = 0; k < 9; ++k)
            g[k / 3][k % 3] = flip ? wt[(co * 9 + 8 - k) * kC + ci] : wt[(ci * 9 + k) * kC + co];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            t[0][x] = g[0][x];
            t[1][x] = 0.5 * (g[0][x] + g[1][x] + g[2][x]);
            t[2][x] = 0.5 * (g[0][x] - g[1][x] + g[2][x]);
            t[3][x] = g[2][x];
        }
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            const double u[4] = {t[y][0], 0.5 * (t[y][0] + t[y][1] + t[y][2]),
                                 0.5 * (t[y][0] - t[y][1] + t[y][2]), t[y][2]};
#pragma unroll
            for (int x = 0; x < 4; ++x) U[(4 * y + x) * kC * kC + idx] = (float)u[x];
        }
    }
}

// V = B' d B of the 4x4 patch at p (top left, zero-bordered coordinates).
__device__ __forceinline__ void patch_in(const float* p, float (&V)[16]) {
    float2 d[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        d[r][0] = *reinterpret_cast<const float2*>(p + r * kRow);
        d[r][1] = *reinterpret_cast<const float2*>(p + r * kRow + 2);
    }
    float t[4][4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        const float d0 = x & 1 ? d[0][x >> 1].y : d[0][x >> 1].x;
        const float d1 = x & 1 ? d[1][x >> 1].y : d[1][x >> 1].x;
        const float d2 = x & 1 ? d[2][x >> 1].y : d[2][x >> 1].x;
        const float d3 = x & 1 ? d[3][x >> 1].y : d[3][x >> 1].x;
        t[0][x] = d0 - d2;
        t[1][x] = d1 + d2;
        t[2][x] = d2 - d1;
        t[3][x] = d1 - d3;
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) {
        V[4 * y + 0] = t[y][0] - t[y][2];
        V[4 * y + 1] = t[y][1] + t[y][2];
        V[4 * y + 2] = t[y][2] - t[y][1];
        V[4 * y + 3] = t[y][1] - t[y][3];
    }
}

// One layer on the CTA's tile: planes (zero-bordered, kC channels) in; the
// thread's outputs in out (see store_planes).  Every thread of the CTA (16 CP)
// calls it; planes may be overwritten when it returns.
template <int CP>
__device__ __forceinline__ void layer(const float* planes, const float* U, float* vm, float bias,
                                      float (&out)[512 / CP]) {
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    constexpr int kT = 16 * CP;
    // GEMM: unit = point and 16 patches; a quarter-warp has 8 of the patches, a
    // lane 4 output channels
    const int unit = 2 * w + (lane >> 4), point = unit / (CP / 16);
    const int p0 = 16 * (unit % (CP / 16)) + (lane & 8), co = 4 * (lane & 7);
    const float* vp = vm + point * kC * CP + p0;
    const float* up = U + point * kC * kC + co;
    float* mp = vm + (point * CP + p0) * kC + co;
#pragma unroll
    for (int c = 0; c < 64 / CP; ++c) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int item = e * kT + t, ci = item / CP, pos = c * CP + item % CP;
            float V[16];
            patch_in(planes + ci * kPlane + 2 * (pos >> 3) * kRow + 2 * (pos & 7), V);
#pragma unroll
            for (int k = 0; k < 16; ++k) vm[k * kC * CP + item] = V[k];
        }
        __syncthreads();
        float2 acc[8][2];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = make_float2(0.0f, 0.0f);
#pragma unroll 8
        for (int k = 0; k < kC; ++k) {
            const float4 v0 = *reinterpret_cast<const float4*>(vp + k * CP);
            const float4 v1 = *reinterpret_cast<const float4*>(vp + k * CP + 4);
            const float4 u = *reinterpret_cast<const float4*>(up + k * kC);
            const float2 u0 = make_float2(u.x, u.y), u1 = make_float2(u.z, u.w);
            const float vi[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[i][0] = fma2(splat(vi[i]), u0, acc[i][0]);
                acc[i][1] = fma2(splat(vi[i]), u1, acc[i][1]);
            }
        }
        __syncthreads();  // V is no longer read
#pragma unroll
        for (int i = 0; i < 8; ++i)
            *reinterpret_cast<float4*>(mp + i * kC) =
                make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
        __syncthreads();
#pragma unroll
        for (int e = 0; e < 2; ++e) {  // patch (e kT + t) / 32, channel lane
            float m[4][4], r[2][4];
#pragma unroll
            for (int k = 0; k < 16; ++k) m[k >> 2][k & 3] = vm[k * kC * CP + e * kT + t];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                r[0][x] = m[0][x] + m[1][x] + m[2][x];
                r[1][x] = m[1][x] - m[2][x] - m[3][x];
            }
            float* o = out + 8 * c + 4 * e;
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                o[2 * y] = r[y][0] + r[y][1] + r[y][2] + bias;
                o[2 * y + 1] = r[y][1] - r[y][2] - r[y][3] + bias;
            }
        }
        __syncthreads();  // M is no longer read
    }
}

// The thread's outputs of layer() into the planes: patch c CP + e CP / 2 + w of
// channel lane, 2 x 2 values each.
template <int CP>
__device__ __forceinline__ void store_planes(float* planes, const float (&out)[512 / CP]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 128 / CP; ++q) {
        const int pos = q * (CP / 2) + w;
        float* p = planes + lane * kPlane + (2 * (pos >> 3) + 1) * kRow + 2 * (pos & 7) + 1;
#pragma unroll
        for (int e = 0; e < 4; ++e) p[(e >> 1) * kRow + (e & 1)] = out[4 * q + e];
    }
}

}  // namespace wino
}  // namespace ncsb
