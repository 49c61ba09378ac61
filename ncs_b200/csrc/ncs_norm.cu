// ncs_norm.cu -- the normalised single-pixel NCS variant
// ("matlab - single pixel with normalization/" in the reference): every pixel
// is its own 3 x 3 segment (the pixel and its 8 neighbours, replicate-padded,
// segpadimg.m with Rs = 1) minimising
//     f(u) = (2/9) sum_i [u_i - c_i log(u_i + gamma_i)] + alpha P(u) / S(u),
//     P(u) = sum_k (|fftshift(fft2(u))_k| / 3 * M_k)^2 = u' Q u,  S(u) = sum_i u_i
// (calcost.m:38-56), from u = d, keeping the segment centre (stitchpadimg.m)
// and setting negative results to 1e-6 (reducenoise.m, optimf).
//
// One thread per pixel: 9 unknowns, FP64 iterate, gradient and costs (the
// cost is a sum of terms of order 100 whose differences near convergence are
// of order 1e-5), BFGS with a dense 9 x 9 inverse-Hessian approximation (45
// packed FP32 entries per thread; the direction and the update in FP32 as the
// main solver's L-BFGS, the update's scalars in FP64),
// backtracking Armijo line search on the FP64 cost change (in difference
// form, see the trial loop) with the fraction-to-barrier rule of the main
// solver.  The
// reference minimises with MATLAB's fminunc quasi-Newton; the stopping rule
// here is fminunc's first-order optimality test, ||g||_inf <= tol *
// max(1, ||g_0||_inf), with its iteration cap.  Q (9 x 9, symmetric) is the
// 3 x 3 circular convolution with the kernel qk = ifft2(M^2) / 9 (block
// circulant with circulant blocks): Q[p][q] = qk[(p1 - q1) mod 3][(p2 - q2)
// mod 3], so the kernel takes 9 values from the host instead of 45.
//
// What bounds it: instruction issue and FP64 latency at 8 warps per SM, and
// divergence -- a warp runs until its slowest pixel, 1.4 times the mean count.
// 20 frames of 512^2 take 3.38 ms: 3.74 with separate FP64 comparisons for the
// step's range, the barrier and the stopping test instead of integer maxima of
// upper words, and s = un - u instead of the FP32 step itself; 4.13 with two
// quadratic instead of one cubic refinement of each reciprocal; 4.82 also with
// Q u as 81 products and two reciprocals per pixel and trial.  Refilling a
// warp's finished lanes with new pixels ran 4.2 ms: first iterations, which
// backtrack, then hold up a warp all the time instead of once.
#include <cuda_runtime.h>
#include <math_constants.h>
#include <stdint.h>

#include "../../include/ncs_b200.h"

namespace ncsb {
namespace norm {

// 64 threads a block: three FP64 vectors (216 B a thread) take 14 KB of static
// shared memory
constexpr int kThreads = 64;
// blocks per SM: 4 (8 warps) with the inverse Hessian and the iterate's vectors
// in registers.  6 blocks (168 registers) with them re-read from shared memory
// ran 4 % slower, and spilled them 30 %.
constexpr int kBlocks = 4;
constexpr int kPacked = 45;  // upper triangle of a symmetric 9 x 9

struct Args {
    const float* data;
    const float* gamma;
    long long gstride;
    float* out;
    int T, H, W;
    double qk[9];  // Q[p][q] = qk[((p/3 - q/3) mod 3) * 3 + (p%3 - q%3) mod 3]
    double alpha, tol, c1, min_step;
    int max_iters;
    int32_t* iters;
    int32_t* status;
    double* cost;
};

__host__ __device__ constexpr int pk(int i, int j) {  // packed index, i <= j
    return i * 9 - i * (i - 1) / 2 + (j - i);
}


// Q u, S = sum u and P = u'Q u at a point (the noise term is alpha P / S).
// Quad: the mask has M(k1, k2) = M(k1, -k2), so qk has four distinct values and
// Q u comes from the segment's row, column and total sums (29 additions and
// multiply-adds instead of 81).
template <bool Quad>
__device__ __forceinline__ void noise_parts(const Args& a, const double (&u)[9], double (&Qu)[9],
                                            double& S, double& P) {
    if constexpr (Quad) {
        const double q0 = a.qk[0], qr = a.qk[1], qc = a.qk[3], qd = a.qk[4];
        double R[3], C[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            R[k] = (u[3 * k] + u[3 * k + 1]) + u[3 * k + 2];
            C[k] = (u[k] + u[k + 3]) + u[k + 6];
        }
        S = (R[0] + R[1]) + R[2];
        const double dS = qd * S, kr = qr - qd, kc = qc - qd, ku = (q0 - qr) - kc;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            R[k] = fma(kr, R[k], dS);
            C[k] = kc * C[k];
        }
#pragma unroll
        for (int i = 0; i < 9; ++i) Qu[i] = fma(ku, u[i], R[i / 3] + C[i % 3]);
    } else {
        S = 0.0;
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            S += u[i];
            double acc = 0.0;
#pragma unroll
            for (int j = 0; j < 9; ++j)
                acc = fma(a.qk[((i / 3 - j / 3 + 3) % 3) * 3 + (i % 3 - j % 3 + 3) % 3], u[j], acc);
            Qu[i] = acc;
        }
    }
    P = 0.0;
#pragma unroll
    for (int i = 0; i < 9; ++i) P = fma(u[i], Qu[i], P);
}

// 1/x for x > 0: the hardware's gross FP64 reciprocal (PTX rcp.approx.ftz.f64,
// from the operand's upper 32 bits, about 20 bits) refined by one third-order
// step r (1 + e + e^2), e = 1 - x r, which cubes the relative error.  No FP32
// round trip: conversions share the pipe with the reciprocal itself.
__device__ __forceinline__ double recip(double x) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}

// log1p(x) for |x| <= 0.3 is 2 atanh(y), y = x / (2 + x), |y| < 0.18;
// 2 atanh(y) / y as a polynomial in y^2, minimax in relative error (4e-14).
constexpr int kSeriesHi = 0x3fd33333;  // upper word of 0.3
__device__ __forceinline__ double atanh2_poly(double y2) {
    double s = fma(y2, 0.19696279890493262, 0.2216823319916572);
    s = fma(y2, s, 0.2857230812738637);
    s = fma(y2, s, 0.3999999354479562);
    s = fma(y2, s, 0.6666666668396458);
    return fma(y2, s, 1.999999999999925);
}

// |x| as its upper 32 bits: ordered as |x| up to 2^-20 relative (NaN above all)
__device__ __forceinline__ int abs_hi(double x) { return __double2hiint(x) & 0x7fffffff; }

// x[i] of a register array at a runtime index
template <typename T>
__device__ __forceinline__ T pick(const T (&x)[9], int i) {
    T v = x[0];
#pragma unroll
    for (int k = 1; k < 9; ++k) v = i == k ? x[k] : v;
    return v;
}

template <bool Quad>
__global__ void __launch_bounds__(kThreads, kBlocks) normalized_kernel(const Args a) {
    __shared__ double Cs[9][kThreads];  // (2/9) (d + gamma)
    __shared__ double Rs[9][kThreads];  // 1 / (u + gamma) at the current iterate
    __shared__ double Gs[9][kThreads];  // the gradient there
    const long long HW = (long long)a.H * a.W;
    const long long idx = (long long)blockIdx.x * kThreads + threadIdx.x;
    if (idx >= (long long)a.T * HW) return;
    const int t = threadIdx.x;
    // the segment's data and gamma (replicate-padded)
    auto segment = [&](double (&d)[9], double (&gm)[9]) {
        const int f = (int)(idx / HW);
        const long long p = idx - (long long)f * HW;
        const int y = (int)(p / a.W), x = (int)(p - (long long)y * a.W);
        const float* img = a.data + (long long)f * HW;
        const float* gmap = a.gamma + (long long)f * a.gstride;
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            const int yy = min(max(y + r - 1, 0), a.H - 1);
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                const int xx = min(max(x + s - 1, 0), a.W - 1);
                d[3 * r + s] = img[(long long)yy * a.W + xx];
                gm[3 * r + s] = gmap[(long long)yy * a.W + xx];
            }
        }
    };
    double u[9], g_stop = 0.0, fq = 0.0, res_f = 0.0;
    float gf[9], H[kPacked];  // gradient, inverse-Hessian approximation
    int status = 0, it = 0, g_hi = 0, stop_hi = 0;
    bool feasible;
    {
        double gm[9], Qu[9], S, P, g0 = 0.0;
        segment(u, gm);
        noise_parts<Quad>(a, u, Qu, S, P);
        feasible = S > 0.0;
#pragma unroll
        for (int i = 0; i < 9; ++i) feasible = feasible && u[i] + gm[i] > 0.0;
        const double is = recip(S);
        fq = feasible ? P * is : 0.0;  // P / S at the current iterate
        // A trial whose cost change is below the cost's FP64 resolution is
        // accepted, as when two full costs compare equal: near the optimum the
        // gradient still steers the steps (its test can need changes far below
        // that resolution), and a step that moves no pixel ends the solve.  The
        // resolution is taken as 2^-52 of a bound on |f|, (2/9) sum (|u| +
        // c |log(u + gamma)|) + alpha |P / S|, from the start (FP32 hardware
        // log2: only its scale matters)
        float bound = 0.0f;
        const double k1 = 2.0 * a.alpha * is, k0 = fma(-a.alpha * P * is, is, 2.0 / 9.0);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const double A = u[i] + gm[i], c = A;  // u = d: c = d + gamma
            const double r = recip(A > 0.0 ? A : 1.0);
            Cs[i][t] = (2.0 / 9.0) * c;
            Rs[i][t] = r;
            const double g = fma(k1, Qu[i], fma(-(2.0 / 9.0) * c, r, k0));
            Gs[i][t] = g;
            gf[i] = (float)g;
            g0 = fmax(g0, fabs(g));
            g_hi = max(g_hi, abs_hi(g));
            float l2;
            asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l2) : "f"((float)A));
            bound += fabsf((float)u[i]) + (float)c * fabsf(l2 * 0.69314718f);
        }
        res_f = 0x1p-52 * ((2.0 / 9.0) * (double)bound + a.alpha * fabs(fq));
#pragma unroll
        for (int i = 0; i < 9; ++i)
#pragma unroll
            for (int j = i; j < 9; ++j) H[pk(i, j)] = i == j ? 1.0f : 0.0f;
        g_stop = a.tol * fmax(1.0, g0);
        stop_hi = abs_hi(g_stop);
    }
    status = feasible ? NCSB_REACHED_MAXITERS : NCSB_INCREASING_GRADIENT;
    while (feasible && it < a.max_iters) {
        // some |g_i| above the stopping threshold, by the upper words unless these
        // leave it open
        bool steep = g_hi > stop_hi && g_hi < 0x7ff00000;
        if (!steep && g_hi >= stop_hi) {
#pragma unroll
            for (int i = 0; i < 9; ++i) steep = steep || fabs(Gs[i][t]) > g_stop;
        }
        if (!steep) {
            status = NCSB_SUCCESS;
            break;
        }
        // direction p = -H g and its slope g'p = -g'H g, both FP32 (a quadratic
        // form: no cancellation; the Armijo threshold needs it to 1e-4 at most)
        float d[9];
        double gd;
        {
            float gdf = 0.0f;
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                float acc = 0.0f;
#pragma unroll
                for (int j = 0; j < 9; ++j)
                    acc = fmaf(H[i <= j ? pk(i, j) : pk(j, i)], gf[j], acc);
                d[i] = -acc;
                gdf = fmaf(gf[i], d[i], gdf);
            }
            gd = (double)gdf;
        }
        if (!(gd < 0.0)) {  // lost positive definiteness: restart from steepest descent
#pragma unroll
            for (int i = 0; i < 9; ++i)
#pragma unroll
                for (int j = i; j < 9; ++j) H[pk(i, j)] = i == j ? 1.0f : 0.0f;
            float gdf = 0.0f;
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                d[i] = -gf[i];
                gdf = fmaf(gf[i], d[i], gdf);
            }
            gd = (double)gdf;
        }
        // backtracking Armijo on the cost change in difference form:
        //   f(un) - f(u) = (2/9) sum_i [s_i - c_i log1p(x_i)]
        //                  + alpha (P(un) / S(un) - P(u) / S(u)),
        // s the step d (FP32 values), x_i = s_i / (u_i + gamma_i), whose log terms
        // are of the order of the step rather than of the costs (about 100), so a
        // polynomial log1p at 4e-14 replaces the FP64 logs of two full costs.  Trials
        // keep u + gamma >= 1% of its value: x >= -0.99.  One reciprocal, of
        // (1 + x)(2 + x), gives y = x / (2 + x) of the log1p and 1 / (un + gamma) =
        // (1 / (u + gamma)) / (1 + x) of the next gradient.
        double step = 1.0, un[9], Qn[9], rn[9], Sn = 0.0, Pn = 0.0, isn = 0.0, fqn = 0.0;
        bool ok = false;
        int x_hi = 0;  // max |x|
        for (int trial = 0; trial < 64; ++trial) {
#pragma unroll
            for (int i = 0; i < 9; ++i) un[i] = u[i] + (double)d[i];
            x_hi = 0;
            double ssum = 0.0, lsum = 0.0;
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                const double s = d[i], r = Rs[i][t], x = s * r;
                x_hi = max(x_hi, abs_hi(x));
                const double x1 = 1.0 + x, x2 = 2.0 + x, q = recip(x1 * x2);
                const double y = x * (q * x1);
                rn[i] = r * (q * x2);
                ssum += s;
                lsum = fma(Cs[i][t], y * atanh2_poly(y * y), lsum);
            }
            noise_parts<Quad>(a, un, Qn, Sn, Pn);
            bool feas = Sn > 0.0;
            if (x_hi >= kSeriesHi) {  // a relative step beyond the series' range
                lsum = 0.0;
#pragma unroll 1
                for (int i = 0; i < 9; ++i) {
                    const double x = (double)pick(d, i) * Rs[i][t];
                    feas = feas && x >= -0.99;
                    lsum = fma(Cs[i][t], log1p(x), lsum);
                }
            }
            if (feas) {
                isn = recip(Sn);
                fqn = Pn * isn;  // the same rounding as fq's
                const double df = fma(2.0 / 9.0, ssum, -lsum) + a.alpha * (fqn - fq);
                if (df <= a.c1 * step * gd || fabs(df) <= res_f) {
                    ok = true;
                    break;
                }
            }
            step *= 0.5;
            if (!(step >= a.min_step)) break;
#pragma unroll
            for (int i = 0; i < 9; ++i) d[i] *= 0.5f;
        }
        if (!ok) {
            status = NCSB_MINIMUM_STEP;
            break;
        }
        // BFGS update of the inverse Hessian with s = d, y = gn - g:
        // H <- H - rho (v s' + s v') + (rho^2 y'Hy + rho) s s', v = H y.  The
        // differences and the scalars in FP64, the 45 entries in FP32 from
        // pre-scaled vectors (no FP32 product of rho or rho^2 alone).
        float yv[9];
        double sy = 0.0, yy = 0.0;
        g_hi = 0;
        if ((it & 15) == 15) {  // against the drift of the products above
            double dat[9], gm[9];
            segment(dat, gm);
#pragma unroll
            for (int i = 0; i < 9; ++i) rn[i] = recip(un[i] + gm[i]);
        }
        // a step above 2^-50 of u + gamma moves u
        bool moved = x_hi >= 0x3cd00000;
        if (!moved) {
#pragma unroll
            for (int i = 0; i < 9; ++i) moved = moved || un[i] != u[i];
        }
        const double k1 = 2.0 * a.alpha * isn, k0 = fma(-a.alpha * fqn, isn, 2.0 / 9.0);
#pragma unroll
        for (int i = 0; i < 9; ++i) {
            const double sd = d[i];
            const double gn = fma(k1, Qn[i], fma(-Cs[i][t], rn[i], k0));
            const double yd = gn - Gs[i][t];
            Gs[i][t] = gn;
            Rs[i][t] = rn[i];
            u[i] = un[i];
            gf[i] = (float)gn;
            g_hi = max(g_hi, abs_hi(gn));
            yv[i] = (float)yd;
            sy = fma(sd, yd, sy);
            if (it == 0) yy = fma(yd, yd, yy);
        }
        if (sy > 1e-30) {  // rho = 1 / sy within FP32 range
            if (it == 0) {  // scale the identity before the first update
                const float sc = (float)(sy / yy);
#pragma unroll
                for (int i = 0; i < 9; ++i) H[pk(i, i)] = sc;
            }
            float v[9], yHyf = 0.0f;
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                float acc = 0.0f;
#pragma unroll
                for (int j = 0; j < 9; ++j)
                    acc = fmaf(H[i <= j ? pk(i, j) : pk(j, i)], yv[j], acc);
                v[i] = acc;
                yHyf = fmaf(yv[i], acc, yHyf);
            }
            const double rho = recip(sy), k2 = rho * rho * (double)yHyf + rho;
            const float rhof = (float)rho;
            float rv[9], ks[9];  // rho v and (rho^2 y'Hy + rho) s (k2 may pass FP32's range)
#pragma unroll
            for (int i = 0; i < 9; ++i) {
                rv[i] = rhof * v[i];
                ks[i] = (float)(k2 * (double)d[i]);
            }
#pragma unroll
            for (int i = 0; i < 9; ++i)
#pragma unroll
                for (int j = i; j < 9; ++j) {
                    const float h = H[pk(i, j)];
                    H[pk(i, j)] =
                        fmaf(ks[i], d[j], fmaf(-rv[i], d[j], fmaf(-d[i], rv[j], h)));
                }
        }
        fq = fqn;
        ++it;
        if (!moved) {
            status = NCSB_REACHED_MAXPRECISION;
            break;
        }
    }
    const float centre = (float)u[4];
    a.out[idx] = centre < 0.0f ? 1.0e-6f : centre;
    if (a.iters) a.iters[idx] = it;
    if (a.status) a.status[idx] = status;
    if (a.cost) {  // with FP64 logs, once
        double cost = CUDART_INF;
        if (feasible) {
            double d[9], gm[9], Qu[9], S, P, ll = 0.0;
            segment(d, gm);
            noise_parts<Quad>(a, u, Qu, S, P);
#pragma unroll
            for (int i = 0; i < 9; ++i) ll += u[i] - (d[i] + gm[i]) * log(u[i] + gm[i]);
            cost = (2.0 / 9.0) * ll + a.alpha * P / S;
        }
        a.cost[idx] = cost;
    }
}

}  // namespace norm
}  // namespace ncsb

using namespace ncsb::norm;

extern "C" {

int ncsb_reduce_noise_normalized(const float* images, int n_frames, int height, int width,
                                 const float* gamma, int gamma_per_frame,
                                 const float* mask3_centred, double alpha, int max_iters,
                                 double tolerance, float* out, int32_t* px_iters,
                                 int32_t* px_status, double* px_cost, void* stream) {
    if (!mask3_centred) return NCSB_EINVAL;
    if (n_frames < 0 || height <= 0 || width <= 0 || max_iters < 0) return NCSB_EINVAL;
    if (!(alpha >= 0.0) || !(tolerance >= 0.0)) return NCSB_EINVAL;
    if (n_frames == 0) return NCSB_OK;  // nothing read or written: buffers may be null
    if (!images || !gamma || !out) return NCSB_EINVAL;
    // Q[a][b] = (1/9) sum_k Mu_k^2 Re(conj(F_a[k]) F_b[k]), Mu = ifftshift(mask) (the mask
    // multiplies fftshift(fft2(u))), symmetrised over k -> -k; F_a = fft2 of unit vector a
    double mu[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) {
            const double m = mask3_centred[((i + 1) % 3) * 3 + (j + 1) % 3];
            if (!(m == m) || m > 1e300 || m < -1e300) return NCSB_EINVAL;
            mu[i][j] = m * m;
        }
    double sym[3][3];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j) sym[i][j] = 0.5 * (mu[i][j] + mu[(3 - i) % 3][(3 - j) % 3]);
    bool quad = true;  // M(k1, k2) = M(k1, -k2)
    for (int i = 0; i < 3; ++i) quad = quad && sym[i][1] == sym[i][2];
    Args a{};
    const double tw = 2.0 * 3.14159265358979323846 / 3.0;
    // qk[d1][d2] = Q[(d1, d2)][(0, 0)]; Re(e^{+i th_p} e^{-i th_q}) = cos(th_p - th_q)
    for (int d1 = 0; d1 < 3; ++d1)
        for (int d2 = 0; d2 < 3; ++d2) {
            double acc = 0.0;
            for (int k1 = 0; k1 < 3; ++k1)
                for (int k2 = 0; k2 < 3; ++k2) acc += sym[k1][k2] * cos(tw * (k1 * d1 + k2 * d2));
            a.qk[d1 * 3 + d2] = acc / 9.0;
        }
    a.data = images;
    a.gamma = gamma;
    a.gstride = gamma_per_frame ? (long long)height * width : 0;
    a.out = out;
    a.T = n_frames;
    a.H = height;
    a.W = width;
    a.alpha = alpha;
    a.tol = tolerance;
    a.c1 = 1e-4;
    a.min_step = 1e-12;
    a.max_iters = max_iters;
    a.iters = px_iters;
    a.status = px_status;
    a.cost = px_cost;
    const long long n = (long long)n_frames * height * width;
    const unsigned grid = (unsigned)((n + kThreads - 1) / kThreads);
    if (quad) normalized_kernel<true><<<grid, kThreads, 0, (cudaStream_t)stream>>>(a);
    else normalized_kernel<false><<<grid, kThreads, 0, (cudaStream_t)stream>>>(a);
    return cudaGetLastError() == cudaSuccess ? NCSB_OK : NCSB_ECUDA;
}

}  // extern "C"
