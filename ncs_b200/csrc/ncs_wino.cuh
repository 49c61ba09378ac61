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
__host__ __device__ constexpr int kV(int cp) { return 16 * kC * cp; }

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

// Of the convolution kernels (a layer at a time): CP = 32, 16 warps
constexpr int kCp = 32, kThreads = 16 * kCp;

// The thread's 16 values of a [kC][16][16] tile, as four float4s: channel and
// row of each from load_at().
__device__ __forceinline__ int tile_at(int q) { return q * kThreads + threadIdx.x; }  // float4 index
__device__ __forceinline__ void load_tile(const float* __restrict__ x, float4 (&v)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = __ldg(reinterpret_cast<const float4*>(x) + tile_at(q));
}
__device__ __forceinline__ void tile_to_planes(const float4 (&v)[4], float* planes) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int i = tile_at(q), ch = i >> 6, r = (i >> 2) & 15, c4 = 4 * (i & 3);
        float* p = planes + ch * kPlane + (r + 1) * kRow + c4 + 1;
        p[0] = v[q].x;
        p[1] = v[q].y;
        p[2] = v[q].z;
        p[3] = v[q].w;
    }
}

// The transforms add up to four inputs, so an infinity turns every output of its
// patches into NaN, where the direct form has infinities at the neighbours alone, and
// large values may overflow.  conv and wgrad watch their results for either and, rarely,
// take those tiles again in the direct form: tiles or weights with a value past kWild
// (NaN included), below which nothing overflows.
constexpr float kWild = 1.0e15f;
// |x| as bits: ordered as |x|, NaN above all
__device__ __forceinline__ int abs_bits(float x) { return __float_as_int(x) & 0x7fffffff; }
constexpr int kInfBits = 0x7f800000;
__device__ __noinline__ bool wild(const float* __restrict__ x, int n) {  // for the CTA
    bool w = false;
#pragma unroll 1
    for (int i = threadIdx.x; i < n; i += kThreads) w = w || !(fabsf(x[i]) <= kWild);
    return __syncthreads_or(w) != 0;
}

// The layer of one tile (pointers to its kC x 256 values) in the direct form.
__device__ __noinline__ void direct_conv(const float* __restrict__ x, const float* __restrict__ wt,
                                         const float* __restrict__ b, const float* __restrict__ act,
                                         float* __restrict__ y, bool relu, bool flip) {
#pragma unroll 1
    for (int i = threadIdx.x; i < kC * 256; i += kThreads) {
        const int co = i >> 8, r = (i >> 4) & 15, c = i & 15;
        float acc = b ? b[co] : 0.0f;
#pragma unroll 1
        for (int ci = 0; ci < kC; ++ci)
#pragma unroll 1
            for (int k = 0; k < 9; ++k) {
                const int yy = r + k / 3 - 1, xx = c + k % 3 - 1;
                const float v = (unsigned)yy < 16u && (unsigned)xx < 16u
                                    ? x[ci * 256 + yy * 16 + xx] : 0.0f;
                acc = fmaf(flip ? wt[(co * 9 + 8 - k) * kC + ci] : wt[(ci * 9 + k) * kC + co], v, acc);
            }
        if (relu) acc = fmaxf(acc, 0.0f);
        y[i] = act && !(act[i] > 0.0f) ? 0.0f : acc;
    }
}

// The weight gradient of one tile, added to dwt.
__device__ __noinline__ void direct_wgrad(const float* __restrict__ x, const float* __restrict__ dy,
                                          float* __restrict__ dwt) {
#pragma unroll 1
    for (int i = threadIdx.x; i < 9 * kC * kC; i += kThreads) {
        const int co = i & 31, k = (i >> 5) % 9, ci = i / (9 * kC);
        double s = 0.0;
#pragma unroll 1
        for (int p = 0; p < 256; ++p) {
            const int yy = (p >> 4) + k / 3 - 1, xx = (p & 15) + k % 3 - 1;
            const float v = (unsigned)yy < 16u && (unsigned)xx < 16u ? x[ci * 256 + yy * 16 + xx] : 0.0f;
            s = fma((double)v, (double)dy[co * 256 + p], s);
        }
        atomicAdd(dwt + i, (float)s);
    }
}

// The kernels of a training step.  2048 tiles take 0.14 ms a layer here and 0.13
// ms in wgrad (direct kernels: 0.38 and 0.32 ms); a step 2.91 -> 0.95 ms, its
// gradient's error against FP64 6.7e-7 -> 3.5e-7.
//
// y = conv(x, wt) + b per tile (b may be null), then ReLU (RELU), or the gradient
// mask of a ReLU whose output is act (act non-null: y = 0 where act <= 0).  FLIP:
// the convolution is the input gradient's, with wt the forward weights.  FIRST:
// y is the output gradient of the first layer, whose two input channels are f:
// it is not stored but reduced to that layer's weight gradient in dw [2][9][32]
// and db (128 MB less traffic per step of 2048 tiles than a pass of its own).
template <bool RELU, bool FLIP, bool FIRST>
__global__ void __launch_bounds__(kThreads) conv(const float* __restrict__ x,
                                                 const float* __restrict__ wt,
                                                 const float* __restrict__ b,
                                                 const float* __restrict__ act,
                                                 float* __restrict__ y, int n,
                                                 const float* __restrict__ f,
                                                 float* __restrict__ dw, float* __restrict__ db) {
    extern __shared__ __align__(16) float sm[];
    float* U = sm;
    float* planes = U + kU;
    float* vm = planes + kPlanes;
    float* fp = vm + kV(kCp);  // FIRST: the feature planes, 18 rows of kRow, 2 channels
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int i = t; i < kPlanes; i += kThreads) planes[i] = 0.0f;
    if (FIRST)
        for (int i = t; i < 2 * kPlane; i += kThreads) fp[i] = 0.0f;
    weights(U, wt, FLIP);
    const float bias = b ? b[lane] : 0.0f;
    __shared__ int odd;  // an output of this CTA is not finite
    if (t == 0) odd = 0;
    float tot[FIRST ? 19 : 1] = {};  // FIRST: this lane's channel: 18 weights and the bias
    float4 next[4];
    int tile = blockIdx.x;
    if (tile < n) load_tile(x + (size_t)tile * kC * 256, next);
    for (; tile < n; tile += gridDim.x) {
        __syncthreads();  // weights and borders written; the last tile's planes read
        tile_to_planes(next, planes);
        if (FIRST)
            fp[(t >> 8) * kPlane + (((t >> 4) & 15) + 1) * kRow + (t & 15) + 1] =
                __ldg(f + (size_t)tile * 512 + t);
        if (tile + gridDim.x < n) load_tile(x + (size_t)(tile + gridDim.x) * kC * 256, next);
        __syncthreads();
        float out[16];
        layer<kCp>(planes, U, vm, bias, out);
        if (!FIRST) {
            int top = 0;
#pragma unroll
            for (int k = 0; k < 16; ++k) top = max(top, abs_bits(out[k]));
            if (top >= kInfBits) odd = 1;
        }
        if (RELU) {
#pragma unroll
            for (int k = 0; k < 16; ++k) out[k] = fmaxf(out[k], 0.0f);
        }
        store_planes<kCp>(planes, out);
        __syncthreads();
        float4* yt = FIRST ? nullptr : reinterpret_cast<float4*>(y + (size_t)tile * kC * 256);
        const float4* at =
            act ? reinterpret_cast<const float4*>(act + (size_t)tile * kC * 256) : nullptr;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = tile_at(q), ch = i >> 6, r = (i >> 2) & 15, c4 = 4 * (i & 3);
            float* p = planes + ch * kPlane + (r + 1) * kRow + c4 + 1;
            float4 o = make_float4(p[0], p[1], p[2], p[3]);
            if (act) {
                const float4 a = __ldg(at + i);
                o.x = a.x > 0.0f ? o.x : 0.0f;
                o.y = a.y > 0.0f ? o.y : 0.0f;
                o.z = a.z > 0.0f ? o.z : 0.0f;
                o.w = a.w > 0.0f ? o.w : 0.0f;
            }
            if (FIRST) {
                p[0] = o.x;
                p[1] = o.y;
                p[2] = o.z;
                p[3] = o.w;
            } else {
                yt[i] = o;
            }
        }
        if (FIRST) {  // lane = output channel, warp = row
            __syncthreads();
            float g[16], acc[18];
            const float* p = planes + lane * kPlane + (w + 1) * kRow + 1;
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                g[c] = p[c];
                tot[18] += g[c];
            }
#pragma unroll
            for (int k = 0; k < 18; ++k) acc[k] = 0.0f;
#pragma unroll
            for (int k = 0; k < 6; ++k) {  // input channel and window row
                const float* xr = fp + (k / 3) * kPlane + (w + k % 3) * kRow;
                float v[20];
#pragma unroll
                for (int q = 0; q < 5; ++q) {
                    const float2 a = *reinterpret_cast<const float2*>(xr + 4 * q);
                    const float2 c = *reinterpret_cast<const float2*>(xr + 4 * q + 2);
                    v[4 * q] = a.x;
                    v[4 * q + 1] = a.y;
                    v[4 * q + 2] = c.x;
                    v[4 * q + 3] = c.y;
                }
#pragma unroll
                for (int kx = 0; kx < 3; ++kx)
#pragma unroll
                    for (int c = 0; c < 16; ++c)
                        acc[3 * k + kx] = fmaf(g[c], v[c + kx], acc[3 * k + kx]);
            }
#pragma unroll
            for (int k = 0; k < 18; ++k) tot[k] += acc[k];
        }
    }
    if (!FIRST) {
        __syncthreads();
        if (odd) {
            const bool all = wild(wt, 9 * kC * kC);
            for (tile = blockIdx.x; tile < n; tile += gridDim.x) {
                const size_t at = (size_t)tile * kC * 256;
                if (wild(x + at, kC * 256) || all)
                    direct_conv(x + at, wt, b, act ? act + at : nullptr, y + at, RELU, FLIP);
            }
        }
    }
    if (FIRST) {
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 19; ++k) vm[(w * 19 + k) * kC + lane] = tot[k];
        __syncthreads();
        for (int i = t; i < 19 * kC; i += kThreads) {
            double s = 0.0;
            for (int k = 0; k < 16; ++k) s += vm[k * 19 * kC + i];
            atomicAdd(i < 18 * kC ? dw + i : db + (i - 18 * kC), (float)s);
        }
    }
}

constexpr size_t kConvSmem = (size_t)(kU + kPlanes + kV(kCp)) * sizeof(float);
constexpr size_t kFirstSmem = kConvSmem + 2 * kPlane * sizeof(float);

// Weight gradient: dL/dg = G' [ sum (A dy A') . (B' d B) ] G, db = sum dy.  Warp
// w accumulates point w's 32 x 32 products over all patches of the CTA's tiles
// in registers; one atomic per weight and CTA at the end.
constexpr int kG = 258;  // dy plane stride: 64-bit reads over channels hit distinct banks
constexpr int kP = 512;  // V and dY: [point][patch][channel]
constexpr size_t kWgradSmem =
    (size_t)(kPlanes + kC * kG + 2 * 16 * kP) * sizeof(float);

__global__ void __launch_bounds__(kThreads) wgrad(const float* __restrict__ x,
                                                  const float* __restrict__ dy,
                                                  float* __restrict__ dwt, float* __restrict__ db,
                                                  int n) {
    extern __shared__ __align__(16) float sm[];
    float* planes = sm;
    float* gs = planes + kPlanes;
    float* V = gs + kC * kG;
    float* Y = V + 16 * kP;
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int i = t; i < kPlanes; i += kThreads) planes[i] = 0.0f;
    const int ig = lane >> 3, og = lane & 7;  // 8 input and 4 output channels
    float2 acc[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = make_float2(0.0f, 0.0f);
    double bsum = 0.0;
    float4 nx[4], ng[4];
    int tile = blockIdx.x;
    if (tile < n) {
        load_tile(x + (size_t)tile * kC * 256, nx);
        load_tile(dy + (size_t)tile * kC * 256, ng);
    }
    for (; tile < n; tile += gridDim.x) {
        __syncthreads();  // the last tile's planes are read, the borders written
        tile_to_planes(nx, planes);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int i = tile_at(q);
            float* p = gs + (i >> 6) * kG + 4 * (i & 63);
            *reinterpret_cast<float2*>(p) = make_float2(ng[q].x, ng[q].y);
            *reinterpret_cast<float2*>(p + 2) = make_float2(ng[q].z, ng[q].w);
        }
        if (tile + gridDim.x < n) {
            load_tile(x + (size_t)(tile + gridDim.x) * kC * 256, nx);
            load_tile(dy + (size_t)(tile + gridDim.x) * kC * 256, ng);
        }
        __syncthreads();
#pragma unroll 1
        for (int c = 0; c < 4; ++c) {
            const int tr = 2 * c + (w >> 3), tj = w & 7;  // this warp's patch
            {
                float v[16];
                patch_in(planes + lane * kPlane + 2 * tr * kRow + 2 * tj, v);
#pragma unroll
                for (int k = 0; k < 16; ++k) V[k * kP + t] = v[k];
            }
            {
                const float* p = gs + lane * kG + 32 * tr + 2 * tj;
                const float2 a = *reinterpret_cast<const float2*>(p);
                const float2 b = *reinterpret_cast<const float2*>(p + 16);
                bsum += (double)((a.x + a.y) + (b.x + b.y));
                const float2 rows[4] = {a, make_float2(a.x + b.x, a.y + b.y),
                                        make_float2(a.x - b.x, a.y - b.y), make_float2(-b.x, -b.y)};
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    Y[(4 * y + 0) * kP + t] = rows[y].x;
                    Y[(4 * y + 1) * kP + t] = rows[y].x + rows[y].y;
                    Y[(4 * y + 2) * kP + t] = rows[y].x - rows[y].y;
                    Y[(4 * y + 3) * kP + t] = -rows[y].y;
                }
            }
            __syncthreads();
            const float* vp = V + w * kP + 8 * ig;
            const float* yp = Y + w * kP + 4 * og;
#pragma unroll 4
            for (int k = 0; k < 16; ++k) {
                const float4 v0 = *reinterpret_cast<const float4*>(vp + k * kC);
                const float4 v1 = *reinterpret_cast<const float4*>(vp + k * kC + 4);
                const float4 g = *reinterpret_cast<const float4*>(yp + k * kC);
                const float2 g0 = make_float2(g.x, g.y), g1 = make_float2(g.z, g.w);
                const float vi[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    acc[i][0] = fma2(splat(vi[i]), g0, acc[i][0]);
                    acc[i][1] = fma2(splat(vi[i]), g1, acc[i][1]);
                }
            }
            __syncthreads();
        }
    }
    int top = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        top = max(top, max(max(abs_bits(acc[i][0].x), abs_bits(acc[i][0].y)),
                           max(abs_bits(acc[i][1].x), abs_bits(acc[i][1].y))));
    const bool odd = __syncthreads_or(top >= kInfBits) != 0;
    if (odd)
        for (tile = blockIdx.x; tile < n; tile += gridDim.x)
            direct_wgrad(x + (size_t)tile * kC * 256, dy + (size_t)tile * kC * 256, dwt);
    // M[point][ci][co] through shared memory (V and dY's 16 x 1024 floats)
    float* M = V;
#pragma unroll
    for (int i = 0; i < 8; ++i)
        *reinterpret_cast<float4*>(M + w * 1024 + (8 * ig + i) * kC + 4 * og) =
            make_float4(acc[i][0].x, acc[i][0].y, acc[i][1].x, acc[i][1].y);
    reinterpret_cast<double*>(gs)[t] = bsum;  // [warp][channel]
    __syncthreads();
    for (int idx = odd ? kC * kC : t; idx < kC * kC; idx += kThreads) {
        const int ci = idx >> 5, co = idx & 31;
        float m[4][4], r[3][4];
#pragma unroll
        for (int k = 0; k < 16; ++k) m[k >> 2][k & 3] = M[k * 1024 + idx];
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const float p = 0.5f * (m[1][c] + m[2][c]), q = 0.5f * (m[1][c] - m[2][c]);
            r[0][c] = m[0][c] + p;
            r[1][c] = q;
            r[2][c] = p + m[3][c];
        }
#pragma unroll
        for (int y = 0; y < 3; ++y) {
            const float p = 0.5f * (r[y][1] + r[y][2]), q = 0.5f * (r[y][1] - r[y][2]);
            float* o = dwt + (ci * 9 + 3 * y) * kC + co;
            atomicAdd(o, r[y][0] + p);
            atomicAdd(o + kC, q);
            atomicAdd(o + 2 * kC, p + r[y][3]);
        }
    }
    if (t < kC) {
        double s = 0.0;
        for (int k = 0; k < 16; ++k) s += reinterpret_cast<const double*>(gs)[k * kC + t];
        atomicAdd(db + t, (float)s);
    }
}

// The last layer (32 -> 1) of a training step in one pass over its input: output,
// MSE loss against target, weight and bias gradients, and the input gradient g
// masked by the ReLU that made a.  Separate kernels read a three times and ran
// 74 + 7 + 271 + 30 us for 2048 tiles.  Sums over tiles are FP64.
constexpr int kLastPart = 8 * 256;
constexpr size_t kLastSmem = (size_t)(kPlanes + kLastPart + kPlane + 2 + 12 * kC + 64) * sizeof(float);

__global__ void __launch_bounds__(kThreads, 2) last_layer(
    const float* __restrict__ a, const float* __restrict__ wt, const float* __restrict__ b,
    const float* __restrict__ target, float* __restrict__ g, float* __restrict__ dwt,
    float* __restrict__ db, float* __restrict__ loss, int n) {
    extern __shared__ __align__(16) float sm[];
    float* planes = sm;
    float* part = planes + kPlanes;
    float* gp = part + kLastPart;  // dL/dy, zero-bordered
    float* ws = gp + kPlane + 2;   // [ci][12], 16-byte aligned
    double* red = reinterpret_cast<double*>(ws + 12 * kC);
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    for (int i = t; i < kPlanes; i += kThreads) planes[i] = 0.0f;
    for (int i = t; i < kPlane; i += kThreads) gp[i] = 0.0f;
    for (int i = t; i < 9 * kC; i += kThreads) ws[(i / 9) * 12 + i % 9] = wt[i];
    const float bias = b[0];
    const double inv = 1.0 / ((double)n * 256.0);
    const int sr = (t & 63) >> 2, sc = 4 * (t & 3), grp = t >> 6;  // strip, 4 channels
    double wsum[9] = {}, lsum = 0.0, bsum = 0.0;
    for (int tile = blockIdx.x; tile < n; tile += gridDim.x) {
        {
            float4 v[4];
            load_tile(a + (size_t)tile * kC * 256, v);
            __syncthreads();
            tile_to_planes(v, planes);
        }
        __syncthreads();
        {
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float* x = planes + (4 * grp + i) * kPlane + sr * kRow + sc;
                const float* wr = ws + (4 * grp + i) * 12;
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) {
                    float v[6];
#pragma unroll
                    for (int k = 0; k < 3; ++k) {
                        const float2 z = *reinterpret_cast<const float2*>(x + ky * kRow + 2 * k);
                        v[2 * k] = z.x;
                        v[2 * k + 1] = z.y;
                    }
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx)
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            acc[e] = fmaf(wr[3 * ky + kx], v[e + kx], acc[e]);
                }
            }
            *reinterpret_cast<float4*>(part + grp * 256 + sr * 16 + sc) =
                make_float4(acc[0], acc[1], acc[2], acc[3]);
        }
        __syncthreads();
        if (t < 256) {
            float y = bias;
#pragma unroll
            for (int k = 0; k < 8; ++k) y += part[k * 256 + t];
            const float d = y - __ldg(target + (size_t)tile * 256 + t);
            const float gy = (float)(2.0 * inv * (double)d);
            lsum += (double)d * d;
            bsum += (double)gy;
            gp[((t >> 4) + 1) * kRow + (t & 15) + 1] = gy;
        }
        __syncthreads();
        {  // input gradient: strip of 4 pixels, 4 channels
            float v[3][6];
#pragma unroll
            for (int k = 0; k < 9; ++k) {
                const float2 z = *reinterpret_cast<const float2*>(gp + (sr + k / 3) * kRow + sc +
                                                                  2 * (k % 3));
                v[k / 3][2 * (k % 3)] = z.x;
                v[k / 3][2 * (k % 3) + 1] = z.y;
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int ci = 4 * grp + i;
                const float* wr = ws + ci * 12;
                float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int k = 0; k < 9; ++k)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        acc[e] = fmaf(wr[8 - k], v[k / 3][e + k % 3], acc[e]);
                const float* x = planes + ci * kPlane + (sr + 1) * kRow + sc + 1;
                *reinterpret_cast<float4*>(g + (size_t)tile * kC * 256 + ci * 256 + sr * 16 + sc) =
                    make_float4(x[0] > 0.0f ? acc[0] : 0.0f, x[1] > 0.0f ? acc[1] : 0.0f,
                                x[2] > 0.0f ? acc[2] : 0.0f, x[3] > 0.0f ? acc[3] : 0.0f);
            }
        }
        {  // weight gradient: lane = input channel, warp = row
            float gr[16], acc[9];
#pragma unroll
            for (int c = 0; c < 16; ++c) gr[c] = gp[(w + 1) * kRow + c + 1];
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                const float* x = planes + lane * kPlane + (w + ky) * kRow;
                float v[18];
#pragma unroll
                for (int q = 0; q < 9; ++q) {
                    const float2 z = *reinterpret_cast<const float2*>(x + 2 * q);
                    v[2 * q] = z.x;
                    v[2 * q + 1] = z.y;
                }
#pragma unroll
                for (int kx = 0; kx < 3; ++kx) {
                    float s = 0.0f;
#pragma unroll
                    for (int c = 0; c < 16; ++c) s = fmaf(gr[c], v[c + kx], s);
                    acc[3 * ky + kx] = s;
                }
            }
#pragma unroll
            for (int k = 0; k < 9; ++k) wsum[k] += (double)acc[k];
        }
    }
    // one atomic per value and CTA
    __syncthreads();
    double* all = reinterpret_cast<double*>(planes);  // [warp][9][ci]
#pragma unroll
    for (int k = 0; k < 9; ++k) all[(w * 9 + k) * kC + lane] = wsum[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
        bsum += __shfl_xor_sync(0xffffffffu, bsum, o);
    }
    if (lane == 0) {
        red[w] = lsum;
        red[16 + w] = bsum;
    }
    __syncthreads();
    for (int i = t; i < 9 * kC; i += kThreads) {
        double s = 0.0;
        for (int k = 0; k < 16; ++k) s += all[k * 9 * kC + i];
        atomicAdd(dwt + (i % kC) * 9 + i / kC, (float)s);
    }
    if (t == 0) {
        double l = 0.0, s = 0.0;
        for (int k = 0; k < 8; ++k) {
            l += red[k];
            s += red[16 + k];
        }
        atomicAdd(loss, (float)(l * inv));
        atomicAdd(db, (float)s);
    }
}

}  // namespace wino
}  // namespace ncsb
