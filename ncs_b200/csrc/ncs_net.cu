// ncs_net.cu -- kernels of the learned warm start: a 4-layer 3x3 convolutional
// network that maps a tile's photon image and gamma map to a proposed start
// for the L-BFGS solve (include/ncs_b200.h, "learned warm start").  Forward,
// weight gradient, input gradient (forward pass with flipped weights), ReLU
// backward, MSE loss gradient, Adam, and a fused whole-network inference
// kernel that cuts tiles straight from the stack.  FP32 SIMT throughout, the
// 32 -> 32 layers as Winograd convolutions (ncs_wino.cuh); one 16x16 tile is one
// image, zero-padded at its border.
//
// Layouts: activations [n][c][16][16] in global memory; in shared memory one
// channel is an 18x18 zero-bordered plane with a channel stride of kCS = 325
// floats (odd, so 32 lanes reading 32 channels at one pixel hit 32 banks);
// weights wt[ci][tap][co], tap = 3 ky + kx, so the outputs of one pixel read
// consecutive weights (float4 broadcasts).
//
// Input features per tile (mu, s = mean and std + 1 of d):
//   x0 = (d - mu) / s,   x1 = sqrt(max(d, 0) + gamma) / s
// and the proposal is u0 = d + s y, clamped to u0 + gamma >= 0.05 max(d + gamma, 1e-3)
// so that the likelihood stays finite at the start.
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/ncs_b200.h"
#include "ncs_internal.cuh"
#include "ncs_wino.cuh"

namespace ncsb {
namespace net {

constexpr int kPad = 18;  // 16 + 1-px zero border on each side
constexpr int kCS = 325;  // shared-memory channel stride (18 * 18 + 1)
constexpr int kC = 32;    // hidden channels
constexpr int kParams = 2 * 9 * kC + kC + 2 * (kC * 9 * kC + kC) + kC * 9 + 1;
constexpr float kStartFrac = 0.05f;

__host__ __device__ constexpr int round4(int v) { return (v + 3) & ~3; }

// Stage CIN channels of one tile into zero-bordered planes.
template <int CIN>
__device__ __forceinline__ void stage_planes(float* xs, const float* __restrict__ xt) {
    for (int idx = threadIdx.x; idx < CIN * kPad * kPad; idx += blockDim.x) {
        const int ci = idx / (kPad * kPad), rem = idx - ci * (kPad * kPad);
        const int rr = rem / kPad - 1, cc = rem - (rem / kPad) * kPad - 1;
        xs[ci * kCS + rem] =
            (rr >= 0 && rr < 16 && cc >= 0 && cc < 16) ? xt[ci * 256 + rr * 16 + cc] : 0.0f;
    }
}

// acc[co] += sum_ci,tap w[ci][tap][co] x[ci][pixel + tap] for pixel (r, c).
template <int CIN, int COUT>
__device__ __forceinline__ void conv_pixel(const float* xs, const float* ws, int r, int c,
                                           float (&acc)[COUT]) {
    for (int ci = 0; ci < CIN; ++ci) {
        const float* xc = xs + ci * kCS + r * kPad + c;
#pragma unroll
        for (int tap = 0; tap < 9; ++tap) {
            const float xv = xc[(tap / 3) * kPad + tap % 3];
            const float* wr = ws + (ci * 9 + tap) * COUT;
            if constexpr (COUT % 4 == 0) {
#pragma unroll
                for (int q = 0; q < COUT / 4; ++q) {
                    const float4 w4 = reinterpret_cast<const float4*>(wr)[q];
                    acc[4 * q + 0] = fmaf(w4.x, xv, acc[4 * q + 0]);
                    acc[4 * q + 1] = fmaf(w4.y, xv, acc[4 * q + 1]);
                    acc[4 * q + 2] = fmaf(w4.z, xv, acc[4 * q + 2]);
                    acc[4 * q + 3] = fmaf(w4.w, xv, acc[4 * q + 3]);
                }
            } else {
#pragma unroll
                for (int co = 0; co < COUT; ++co) acc[co] = fmaf(wr[co], xv, acc[co]);
            }
        }
    }
}

// y = conv3x3(x) + b (optionally ReLU).  One CTA (256 threads) per tile, one
// thread per pixel.
template <int CIN, int COUT, bool RELU>
__global__ void __launch_bounds__(256) conv3x3_fwd(const float* __restrict__ x,
                                                   const float* __restrict__ wt,
                                                   const float* __restrict__ b,
                                                   float* __restrict__ y, int n) {
    extern __shared__ __align__(16) float sm[];
    float* xs = sm;
    float* ws = sm + round4(CIN * kCS);
    const int tile = blockIdx.x;
    if (tile >= n) return;
    const int p = threadIdx.x, r = p >> 4, c = p & 15;
    stage_planes<CIN>(xs, x + (size_t)tile * CIN * 256);
    for (int idx = threadIdx.x; idx < CIN * 9 * COUT; idx += 256) ws[idx] = wt[idx];
    __syncthreads();
    float acc[COUT];
#pragma unroll
    for (int co = 0; co < COUT; ++co) acc[co] = b ? b[co] : 0.0f;
    conv_pixel<CIN, COUT>(xs, ws, r, c, acc);
    float* yt = y + (size_t)tile * COUT * 256;
#pragma unroll
    for (int co = 0; co < COUT; ++co) yt[co * 256 + p] = RELU ? fmaxf(acc[co], 0.0f) : acc[co];
}

// dwt[ci][tap][co] += sum_tiles,pixels dy[co][p] x[ci][p + tap], db += sum dy.
// Thread (ps, ci, g) owns the 9 x CO_PER weights of input channel ci and
// output channels g*CO_PER.. and walks the rows ps, ps + PS, ... of each tile
// with a sliding 3x3 window: per pixel 3 new x values, CO_PER dy values and
// 9 CO_PER FMAs.  Partial sums go to global memory with one atomicAdd per
// weight per thread at the end.
template <int CIN, int COUT>
__global__ void __launch_bounds__(256) conv3x3_wgrad(const float* __restrict__ x,
                                                     const float* __restrict__ dy,
                                                     float* __restrict__ dwt,
                                                     float* __restrict__ db, int n, int per_cta) {
    constexpr int CO_PER = COUT >= 4 ? 4 : COUT;
    constexpr int NG = COUT / CO_PER;
    constexpr int LANES = CIN * NG;
    constexpr int PS = 256 / LANES;
    static_assert(COUT % CO_PER == 0 && 256 % LANES == 0 && PS >= 1 && PS <= 16, "mapping");
    constexpr int GS = 257;  // dy channel stride in shared memory
    extern __shared__ __align__(16) float sm[];
    float* xs = sm;
    float* gs = sm + round4(CIN * kCS);
    const int t = threadIdx.x;
    const int g = t % NG, ci = (t / NG) % CIN, ps = t / LANES;
    float acc[9][CO_PER], bacc[CO_PER];
#pragma unroll
    for (int k = 0; k < 9; ++k)
#pragma unroll
        for (int j = 0; j < CO_PER; ++j) acc[k][j] = 0.0f;
#pragma unroll
    for (int j = 0; j < CO_PER; ++j) bacc[j] = 0.0f;

    const int t0 = blockIdx.x * per_cta;
    const int t1 = min(t0 + per_cta, n);
    for (int tile = t0; tile < t1; ++tile) {
        __syncthreads();  // the previous tile's planes are no longer read
        stage_planes<CIN>(xs, x + (size_t)tile * CIN * 256);
        const float* gt = dy + (size_t)tile * COUT * 256;
        for (int idx = threadIdx.x; idx < COUT * 256; idx += 256)
            gs[(idx >> 8) * GS + (idx & 255)] = gt[idx];
        __syncthreads();
        const float* xc = xs + ci * kCS;
        for (int r = ps; r < 16; r += PS) {
            float win[3][3];
#pragma unroll
            for (int ky = 0; ky < 3; ++ky) {
                win[ky][0] = xc[(r + ky) * kPad + 0];
                win[ky][1] = xc[(r + ky) * kPad + 1];
            }
#pragma unroll
            for (int c = 0; c < 16; ++c) {
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) win[ky][2] = xc[(r + ky) * kPad + c + 2];
                float dv[CO_PER];
#pragma unroll
                for (int j = 0; j < CO_PER; ++j) dv[j] = gs[(g * CO_PER + j) * GS + r * 16 + c];
#pragma unroll
                for (int ky = 0; ky < 3; ++ky)
#pragma unroll
                    for (int kx = 0; kx < 3; ++kx)
#pragma unroll
                        for (int j = 0; j < CO_PER; ++j)
                            acc[ky * 3 + kx][j] = fmaf(win[ky][kx], dv[j], acc[ky * 3 + kx][j]);
#pragma unroll
                for (int j = 0; j < CO_PER; ++j) bacc[j] += dv[j];
#pragma unroll
                for (int ky = 0; ky < 3; ++ky) {
                    win[ky][0] = win[ky][1];
                    win[ky][1] = win[ky][2];
                }
            }
        }
    }
    if (t1 <= t0) return;
#pragma unroll
    for (int tap = 0; tap < 9; ++tap)
#pragma unroll
        for (int j = 0; j < CO_PER; ++j)
            atomicAdd(dwt + (ci * 9 + tap) * COUT + g * CO_PER + j, acc[tap][j]);
    if (ci == 0) {
#pragma unroll
        for (int j = 0; j < CO_PER; ++j) atomicAdd(db + g * CO_PER + j, bacc[j]);
    }
}

// wf[co][8 - tap][ci] = wt[ci][tap][co]
__global__ void flip_weights(const float* __restrict__ wt, float* __restrict__ wf, int cin,
                             int cout) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= cin * 9 * cout) return;
    const int co = i % cout, tap = (i / cout) % 9, ci = i / (9 * cout);
    wf[(co * 9 + (8 - tap)) * cin + ci] = wt[i];
}

__global__ void relu_bwd(float* __restrict__ g, const float* __restrict__ act, size_t n) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n && !(act[i] > 0.0f)) g[i] = 0.0f;
}

// g = 2 (y - t) / n; loss[0] += sum (y - t)^2 / n, one atomic per CTA.
__global__ void mse_grad(const float* __restrict__ y, const float* __restrict__ t,
                         float* __restrict__ g, float* __restrict__ loss, size_t n) {
    __shared__ float part[8];
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    float e = 0.0f;
    if (i < n) {
        const float d = y[i] - t[i];
        g[i] = 2.0f * d / (float)n;
        e = d * d;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = e;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.0f;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += part[w];
        atomicAdd(loss, s / (float)n);
    }
}

// Adam (Kingma & Ba, 2015) with bias correction factors bc1 = 1 - b1^k,
// bc2 = 1 - b2^k.
__global__ void adam_step(float* __restrict__ w, const float* __restrict__ g, float* __restrict__ m,
                          float* __restrict__ v, size_t n, float lr, float b1, float b2, float eps,
                          float bc1, float bc2) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    w[i] -= lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
}

// Tile mean and (std + 1) of one value per thread of 8 warps: each warp's sums
// into red[16], then (after a barrier) the statistics from them.
__device__ __forceinline__ void tile_sums(float dv, float* red) {
    float s1 = dv, s2 = dv * dv;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s1 += __shfl_xor_sync(0xffffffffu, s1, o);
        s2 += __shfl_xor_sync(0xffffffffu, s2, o);
    }
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5] = s1;
        red[8 + (threadIdx.x >> 5)] = s2;
    }
}
__device__ __forceinline__ float2 tile_stats(const float* red) {
    float a = 0.0f, q = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
        a += red[w];
        q += red[8 + w];
    }
    const float mu = a * (1.0f / 256.0f);
    const float sd = sqrtf(fmaxf(q * (1.0f / 256.0f) - mu * mu, 0.0f)) + 1.0f;
    return make_float2(mu, sd);
}

__global__ void __launch_bounds__(256) features(const float* __restrict__ d,
                                                const float* __restrict__ gam,
                                                float* __restrict__ x, float* __restrict__ scale,
                                                int n) {
    __shared__ float red[16];
    const int t = blockIdx.x;
    if (t >= n) return;
    const float dv = d[(size_t)t * 256 + threadIdx.x], gv = gam[(size_t)t * 256 + threadIdx.x];
    tile_sums(dv, red);
    __syncthreads();
    const float2 ms = tile_stats(red);
    x[(size_t)t * 512 + threadIdx.x] = (dv - ms.x) / ms.y;
    x[(size_t)t * 512 + 256 + threadIdx.x] = sqrtf(fmaxf(dv, 0.0f) + fmaxf(gv, 0.0f)) / ms.y;
    if (threadIdx.x == 0) {
        scale[2 * t] = ms.x;
        scale[2 * t + 1] = ms.y;
    }
}

// ---- fused inference -------------------------------------------------------

struct InferSrc {
    int tile_mode;
    const float* d;      // stack [T][H][W] or tiles [N][256]
    const float* gamma;  // [H][W] / [T][H][W] or tiles [N][256]
    long long gamma_frame_stride;
    int H, W, tiles_x, tiles_y;
    long long n_tiles;
    const StackDesc* stacks;  // batched stacks (stack mode), else null
    int n_stacks;
};

// Shared memory of the fused inference, in floats: both hidden layers'
// transformed weights, the activation planes, the Winograd exchange buffer, then
// the first and last layer's weights and biases, the input planes and the sums
// of the tile scale.  The last layer's weights are [ci][12] (9 taps).
struct InferSmem {
    static constexpr int u2 = 0, u3 = u2 + wino::kU, planes = u3 + wino::kU,
                         vm = planes + wino::kPlanes, w1 = vm + wino::kV(16), b1 = w1 + 2 * 9 * kC,
                         w4 = b1 + kC, b4 = w4 + 12 * kC,
                         xin = b4 + 4, red = xin + 2 * wino::kPlane, end = red + 16;
};
constexpr size_t kInferSmem = InferSmem::end * sizeof(float);
constexpr int kInferThreads = 256;

// Persistent grid, one CTA (8 warps) per SM and one tile per CTA at a time:
// first layer direct, the 32 -> 32 layers by Winograd's F(2x2, 3x3) in place
// (ncs_wino.cuh), last layer direct over strips of four pixels.  The direct form
// of all layers took one float4 weight broadcast per 4 multiply-adds and was
// bound by the shared-memory pipe (96 % busy): 20 x 512^2 frames 9.15 ms, this 3.72
// ms (FMA pipe 51 %, shared memory 79 % of the time); error against FP64 3.1e-7
// direct, 1.5e-7 this.
__global__ void __launch_bounds__(kInferThreads) infer(const InferSrc src,
                                                        const float* __restrict__ params,
                                                        float* __restrict__ u0) {
    using S = InferSmem;
    constexpr int kRow = wino::kRow, kPlane = wino::kPlane;
    extern __shared__ __align__(16) float sm[];
    float* planes = sm + S::planes;
    float* xin = sm + S::xin;
    const int t = threadIdx.x, lane = t & 31;
    constexpr int o2 = 2 * 9 * kC + kC, o3 = o2 + kC * 9 * kC + kC, o4 = o3 + kC * 9 * kC + kC;
    wino::weights(sm + S::u2, params + o2, false);
    wino::weights(sm + S::u3, params + o3, false);
    for (int i = t; i < 2 * 9 * kC + kC; i += kInferThreads) sm[S::w1 + i] = params[i];
    for (int i = t; i < 9 * kC; i += kInferThreads) sm[S::w4 + (i / 9) * 12 + i % 9] = params[o4 + i];
    if (t == 0) sm[S::b4] = params[o4 + 9 * kC];
    for (int i = t; i < wino::kPlanes; i += kInferThreads) planes[i] = 0.0f;
    for (int i = t; i < 2 * kPlane; i += kInferThreads) xin[i] = 0.0f;
    const float bias2 = params[o3 - kC + lane], bias3 = params[o4 - kC + lane];
    // a thread's pixel: a warp holds rows r and r + 2, on distinct banks
    const int r = ((t >> 6) << 2) + ((t >> 5) & 1) + 2 * ((t >> 4) & 1), c = t & 15;
    const long long per_frame = (long long)src.tiles_x * src.tiles_y;
    auto pixel = [&](long long tile, float& dv, float& gv) {
        if (src.tile_mode) {
            dv = src.d[tile * 256 + r * 16 + c];
            gv = src.gamma[tile * 256 + r * 16 + c];
            return;
        }
        const float* sd = src.d;
        const float* sgam = src.gamma;
        long long gstride = src.gamma_frame_stride, lt = tile, pf = per_frame;
        int H = src.H, W = src.W, ty = src.tiles_y;
        if (src.stacks) {  // batched: the last stack whose first tile is <= tile
            int lo = 0, hi = src.n_stacks - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (src.stacks[mid].tile_begin <= tile) lo = mid;
                else hi = mid - 1;
            }
            const StackDesc& st = src.stacks[lo];
            sd = st.data;
            sgam = st.gamma;
            gstride = st.gamma_frame_stride;
            lt = tile - st.tile_begin;
            H = st.H;
            W = st.W;
            ty = st.tiles_y;
            pf = (long long)st.tiles_x * st.tiles_y;
        }
        const int f = (int)(lt / pf);
        const int rem = (int)(lt - (long long)f * pf);
        const int ti = rem / ty, tj = rem - ti * ty;
        const int yy = clampi(tile_origin(ti, H) + r - 1, 0, H - 1);
        const int xx = clampi(tile_origin(tj, W) + c - 1, 0, W - 1);
        dv = sd[(long long)f * H * W + (long long)yy * W + xx];
        gv = sgam[(long long)f * gstride + (long long)yy * W + xx];
    };
    float dn = 0.0f, gn = 0.0f;
    if (blockIdx.x < src.n_tiles) pixel(blockIdx.x, dn, gn);
    for (long long tile = blockIdx.x; tile < src.n_tiles; tile += gridDim.x) {
        const float dv = dn, gv = gn;
        if (tile + gridDim.x < src.n_tiles) pixel(tile + gridDim.x, dn, gn);
        // tile mean and std + 1, then the two feature planes
        tile_sums(dv, sm + S::red);
        __syncthreads();
        const float2 ms = tile_stats(sm + S::red);
        xin[(r + 1) * kRow + c + 1] = (dv - ms.x) / ms.y;
        xin[kPlane + (r + 1) * kRow + c + 1] = sqrtf(fmaxf(dv, 0.0f) + fmaxf(gv, 0.0f)) / ms.y;
        __syncthreads();
        {  // layer 1: thread = pixel, all output channels
            float2 acc[16];
#pragma unroll
            for (int q = 0; q < 16; ++q)
                acc[q] = *reinterpret_cast<const float2*>(sm + S::b1 + 2 * q);
#pragma unroll
            for (int ci = 0; ci < 2; ++ci)
#pragma unroll
                for (int k = 0; k < 9; ++k) {
                    const float2 x2 = warp::splat(xin[ci * kPlane + (r + k / 3) * kRow + c + k % 3]);
                    const float4* wr = reinterpret_cast<const float4*>(sm + S::w1 + (ci * 9 + k) * kC);
#pragma unroll
                    for (int q = 0; q < 8; ++q) {
                        const float4 w = wr[q];
                        acc[2 * q] = warp::fma2(make_float2(w.x, w.y), x2, acc[2 * q]);
                        acc[2 * q + 1] = warp::fma2(make_float2(w.z, w.w), x2, acc[2 * q + 1]);
                    }
                }
            float* o = planes + (r + 1) * kRow + c + 1;
#pragma unroll
            for (int q = 0; q < 16; ++q) {
                o[2 * q * kPlane] = fmaxf(acc[q].x, 0.0f);
                o[(2 * q + 1) * kPlane] = fmaxf(acc[q].y, 0.0f);
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int l = 0; l < 2; ++l) {
            float out[32];
            wino::layer<16>(planes, sm + (l ? S::u3 : S::u2), sm + S::vm, l ? bias3 : bias2, out);
#pragma unroll
            for (int k = 0; k < 32; ++k) out[k] = fmaxf(out[k], 0.0f);
            wino::store_planes<16>(planes, out);
            __syncthreads();
        }
        {  // layer 4: thread = strip of 4 pixels x 8 input channels
            const int sr = (t & 63) >> 2, sc = 4 * (t & 3), g = t >> 6;
            float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll 4
            for (int i = 0; i < 8; ++i) {
                const float* x = planes + (8 * g + i) * kPlane + sr * kRow + sc;
                const float4* w4 = reinterpret_cast<const float4*>(sm + S::w4 + (8 * g + i) * 12);
                const float4 wa = w4[0], wb = w4[1], wc = w4[2];
                const float w[9] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w, wc.x};
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
                        for (int e = 0; e < 4; ++e) acc[e] = fmaf(w[3 * ky + kx], v[e + kx], acc[e]);
                }
            }
            *reinterpret_cast<float4*>(sm + S::vm + g * 256 + sr * 16 + sc) =
                make_float4(acc[0], acc[1], acc[2], acc[3]);
        }
        __syncthreads();
        const float* part = sm + S::vm + r * 16 + c;
        float y = sm[S::b4];
#pragma unroll
        for (int g = 0; g < 4; ++g) y += part[g * 256];
        const float lo = kStartFrac * fmaxf(dv + gv, 1e-3f) - gv;
        u0[tile * 256 + r * 16 + c] = fmaxf(fmaf(ms.y, y, dv), lo);
    }
}

int launch_infer(const InferSrc& src, const float* params, float* u0, cudaStream_t s) {
    if (cudaFuncSetAttribute(infer, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)kInferSmem) != cudaSuccess)
        return NCSB_ECUDA;
    int dev = 0, sms = 1;
    if (cudaGetDevice(&dev) != cudaSuccess) return NCSB_ECUDA;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const long long grid = src.n_tiles < sms ? src.n_tiles : sms;
    infer<<<(unsigned)grid, kInferThreads, kInferSmem, s>>>(src, params, u0);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

template <int CIN, int COUT, bool RELU>
int launch_fwd(const float* x, const float* wt, const float* b, float* y, int n, cudaStream_t s) {
    const size_t smem = ((size_t)round4(CIN * kCS) + (size_t)CIN * 9 * COUT) * sizeof(float);
    if (cudaFuncSetAttribute(conv3x3_fwd<CIN, COUT, RELU>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
        return NCSB_ECUDA;
    conv3x3_fwd<CIN, COUT, RELU><<<n, 256, smem, s>>>(x, wt, b, y, n);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

template <int CIN, int COUT>
int launch_wgrad(const float* x, const float* dy, float* dwt, float* db, int n, cudaStream_t s) {
    const size_t smem = ((size_t)round4(CIN * kCS) + (size_t)COUT * 257) * sizeof(float);
    if (cudaFuncSetAttribute(conv3x3_wgrad<CIN, COUT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)smem) != cudaSuccess)
        return NCSB_ECUDA;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    int grid = 2 * sms;
    if (grid > n) grid = n;
    const int per_cta = (n + grid - 1) / grid;
    grid = (n + per_cta - 1) / per_cta;
    conv3x3_wgrad<CIN, COUT><<<grid, 256, smem, s>>>(x, dy, dwt, db, n, per_cta);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

// The Winograd kernels of the 32 -> 32 layers read and write 16 bytes at a time.
bool aligned16(const void* a, const void* b, const void* c) {
    return (((uintptr_t)a | (uintptr_t)b | (uintptr_t)c) & 15) == 0;
}

int one_per_sm(int n) {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return n < sms ? n : sms;
}

template <bool RELU, bool FLIP, bool FIRST>
int launch_wino(const float* x, const float* wt, const float* b, const float* act, float* y, int n,
                cudaStream_t s, const float* f = nullptr, float* dw = nullptr,
                float* db = nullptr) {
    const auto kernel = wino::conv<RELU, FLIP, FIRST>;
    const size_t smem = FIRST ? wino::kFirstSmem : wino::kConvSmem;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return NCSB_ECUDA;
    kernel<<<one_per_sm(n), wino::kThreads, smem, s>>>(x, wt, b, act, y, n, f, dw, db);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int launch_wino_wgrad(const float* x, const float* dy, float* dwt, float* db, int n,
                      cudaStream_t s) {
    if (cudaFuncSetAttribute(wino::wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)wino::kWgradSmem) != cudaSuccess)
        return NCSB_ECUDA;
    wino::wgrad<<<one_per_sm(n), wino::kThreads, wino::kWgradSmem, s>>>(x, dy, dwt, db, n);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int launch_last(const float* a, const float* wt, const float* b, const float* target, float* g,
                float* dwt, float* db, float* loss, int n, cudaStream_t s) {
    if (cudaFuncSetAttribute(wino::last_layer, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)wino::kLastSmem) != cudaSuccess)
        return NCSB_ECUDA;
    const int grid = 2 * one_per_sm((n + 1) / 2);  // two CTAs per SM
    wino::last_layer<<<grid < n ? grid : n, wino::kThreads, wino::kLastSmem, s>>>(
        a, wt, b, target, g, dwt, db, loss, n);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int launch_infer_batch(const float* params, const StackDesc* stacks, int n_stacks,
                       long long n_tiles, float* u0, cudaStream_t s) {
    if (n_tiles == 0) return NCSB_OK;
    InferSrc src{};
    src.tile_mode = 0;
    src.stacks = stacks;
    src.n_stacks = n_stacks;
    src.tiles_x = 1;
    src.tiles_y = 1;
    src.n_tiles = n_tiles;
    return launch_infer(src, params, u0, s);
}

}  // namespace net
}  // namespace ncsb

using namespace ncsb::net;
using ncsb::tiles_along;

extern "C" {

int ncsb_net_param_count(void) { return kParams; }

int ncsb_net_conv_fwd(const float* x, const float* wt, const float* b, float* y, int n, int cin,
                      int cout, int relu, void* stream) {
    if (!x || !wt || !y || n < 0) return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (cin == 2 && cout == 32)
        return relu ? launch_fwd<2, 32, true>(x, wt, b, y, n, s) : launch_fwd<2, 32, false>(x, wt, b, y, n, s);
    if (cin == 32 && cout == 32 && aligned16(x, y, y) && x != y)
        return relu ? launch_wino<true, false, false>(x, wt, b, nullptr, y, n, s)
                    : launch_wino<false, false, false>(x, wt, b, nullptr, y, n, s);
    if (cin == 32 && cout == 32)
        return relu ? launch_fwd<32, 32, true>(x, wt, b, y, n, s) : launch_fwd<32, 32, false>(x, wt, b, y, n, s);
    if (cin == 32 && cout == 1)
        return relu ? launch_fwd<32, 1, true>(x, wt, b, y, n, s) : launch_fwd<32, 1, false>(x, wt, b, y, n, s);
    if (cin == 1 && cout == 32)
        return relu ? launch_fwd<1, 32, true>(x, wt, b, y, n, s) : launch_fwd<1, 32, false>(x, wt, b, y, n, s);
    return NCSB_EINVAL;
}

int ncsb_net_conv_wgrad(const float* x, const float* dy, float* dwt, float* db, int n, int cin,
                        int cout, void* stream) {
    if (!x || !dy || !dwt || !db || n < 0) return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    cudaStream_t s = (cudaStream_t)stream;
    if (cin == 2 && cout == 32) return launch_wgrad<2, 32>(x, dy, dwt, db, n, s);
    if (cin == 32 && cout == 32 && aligned16(x, dy, dy)) return launch_wino_wgrad(x, dy, dwt, db, n, s);
    if (cin == 32 && cout == 32) return launch_wgrad<32, 32>(x, dy, dwt, db, n, s);
    if (cin == 32 && cout == 1) return launch_wgrad<32, 1>(x, dy, dwt, db, n, s);
    return NCSB_EINVAL;
}

int ncsb_net_conv_xgrad(const float* dy, const float* wt, const float* act, float* dx, int n,
                        void* stream) {
    if (!dy || !wt || !dx || n < 0 || !aligned16(dy, act, dx)) return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    return launch_wino<false, true, false>(dy, wt, nullptr, act, dx, n, (cudaStream_t)stream);
}

int ncsb_net_first_layers_grad(const float* dy, const float* wt, const float* act, const float* x,
                               float* dwt, float* db, int n, void* stream) {
    if (!dy || !wt || !act || !x || !dwt || !db || n < 0 || !aligned16(dy, act, act))
        return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    return launch_wino<false, true, true>(dy, wt, nullptr, act, nullptr, n, (cudaStream_t)stream, x,
                                          dwt, db);
}

int ncsb_net_last_layer(const float* a, const float* wt, const float* b, const float* target,
                        float* g, float* dwt, float* db, float* loss, int n, void* stream) {
    if (!a || !wt || !b || !target || !g || !dwt || !db || !loss || n < 0 || !aligned16(a, g, g))
        return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    return launch_last(a, wt, b, target, g, dwt, db, loss, n, (cudaStream_t)stream);
}

int ncsb_net_flip(const float* wt, float* wf, int cin, int cout, void* stream) {
    if (!wt || !wf || cin < 1 || cout < 1 || cin > 1024 || cout > 1024) return NCSB_EINVAL;
    const int n = cin * 9 * cout;
    flip_weights<<<(n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(wt, wf, cin, cout);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int ncsb_net_relu_bwd(float* g, const float* act, int64_t n, void* stream) {
    if (!g || !act || n < 0) return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    relu_bwd<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(g, act, (size_t)n);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int ncsb_net_mse_grad(const float* y, const float* t, float* g, float* loss, int64_t n,
                      void* stream) {
    if (!y || !t || !g || !loss || n <= 0) return NCSB_EINVAL;
    mse_grad<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(y, t, g, loss, (size_t)n);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int ncsb_net_adam(float* w, const float* g, float* m, float* v, int64_t n, float lr, float b1,
                  float b2, float eps, int step, void* stream) {
    if (!w || !g || !m || !v || n < 0 || step < 1) return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    double p1 = 1.0, p2 = 1.0;
    for (int i = 0; i < step && i < 100000; ++i) {
        p1 *= b1;
        p2 *= b2;
    }
    adam_step<<<(unsigned)((n + 255) / 256), 256, 0, (cudaStream_t)stream>>>(
        w, g, m, v, (size_t)n, lr, b1, b2, eps, (float)(1.0 - p1), (float)(1.0 - p2));
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int ncsb_net_features(const float* d, const float* gamma, float* x, float* scale, int n,
                      void* stream) {
    if (!d || !gamma || !x || !scale || n < 0) return NCSB_EINVAL;
    if (n == 0) return NCSB_OK;
    features<<<n, 256, 0, (cudaStream_t)stream>>>(d, gamma, x, scale, n);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

int ncsb_net_infer_stack(const float* params, const float* images, int n_frames, int height,
                         int width, const float* gamma, int gamma_per_frame, float* u0,
                         void* stream) {
    if (!params || !images || !gamma || !u0 || n_frames < 0 || height <= 0 || width <= 0)
        return NCSB_EINVAL;
    if (height < 14 || width < 14) return NCSB_ESIZE;
    if (n_frames == 0) return NCSB_OK;
    InferSrc src{};
    src.tile_mode = 0;
    src.d = images;
    src.gamma = gamma;
    src.gamma_frame_stride = gamma_per_frame ? (long long)height * width : 0;
    src.H = height;
    src.W = width;
    src.tiles_x = tiles_along(height);
    src.tiles_y = tiles_along(width);
    src.n_tiles = (long long)n_frames * src.tiles_x * src.tiles_y;
    return launch_infer(src, params, u0, (cudaStream_t)stream);
}

int ncsb_net_infer_tiles(const float* params, const float* d, const float* gamma, int64_t n_tiles,
                         float* u0, void* stream) {
    if (!params || !d || !gamma || !u0 || n_tiles < 0) return NCSB_EINVAL;
    if (n_tiles == 0) return NCSB_OK;
    InferSrc src{};
    src.tile_mode = 1;
    src.d = d;
    src.gamma = gamma;
    src.tiles_x = 1;
    src.tiles_y = 1;
    src.H = 16;
    src.W = 16;
    src.n_tiles = n_tiles;
    return launch_infer(src, params, u0, (cudaStream_t)stream);
}

}  // extern "C"
