// ncs_pair.cu -- the spectral form at history size 1 (the default solve): L-BFGS
// with the spectral initial inverse Hessian of ncs_spectral.cu, two tiles per
// warp.
//
// Half-warp h of a warp owns one 16x16 tile; lane c of the half holds column c,
// 16 pixels, as pixel pairs z[j] = (row 2j, row 2j + 1).  The noise term's
// operator F^H diag(w) F needs no complex transform in this layout: w is real
// and w(k) = w(-k), so the real separable Fourier basis (cos k n, sin k n along
// each axis) reduces it to 2 x 2 blocks that mix bin (kr, kc) with bin
// (kr, -kc), and to a diagonal where w(kr, kc) = w(kr, -kc) -- every mask that
// depends on |k| alone.  A pass is
//   16-point real DFT of the lane's column, transpose through shared memory,
//   16-point real DFT of the lane's row of coefficients, weights, and the same
//   steps transposed.
// Each 16-point transform is 58 FP32 operations in the lane's own registers:
// no shuffles and no separation of packed rows, where one tile per warp needs
// a lane to share each row with three others.
//
// What bounds it (stack512, 200 x 512^2): instruction issue and FP32 time in
// turn, 59 % of the issue slots and 46 % of the FMA pipe at 12 warps per SM, with
// waits on fixed latencies and on instruction fetch between; the shared-memory path
// is 56 % busy, mostly with the vectors kept there (160 wavefronts a pass, the
// transposes 64).  A pass takes 1,095
// warp instructions for two tiles, where one tile per warp took 1,004 for one:
// the lane's own transforms replace 47 % of those, and every reduction and
// per-tile decision serves two tiles.  2.01 -> 1.31 ms (sensor2048: 15.75 ->
// 10.22 ms).  Two tiles of a pair rarely differ in iterations (5.04 each, 5.09
// for the slower of two), so they run in lock step and a half that ends first
// idles.
#include "ncs_warp_common.cuh"

namespace ncsb {

using namespace warp;

namespace {

// ---- 16-point real transforms -------------------------------------------------
// Coefficient i of x[0..15]: i = 0..8: sum x cos(2 pi i n / 16), i = 9..15:
// sum x sin(2 pi (16 - i) n / 16).  Scalar FP32: the same steps on packed pairs
// issue fewer instructions but need as many moves to align the pairs (stack512
// 1.41 ms packed, 1.39 ms scalar).
constexpr float kC1 = 0.92387953251128674f;  // cos(pi / 8)
constexpr float kT1 = 0.41421356237309503f;  // tan(pi / 8)

__device__ __forceinline__ void rdft16(const float (&x)[16], float (&X)[16]) {
    float s[8], d[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        s[n] = x[n] + x[n + 8];
        d[n] = x[n] - x[n + 8];
    }
    // even frequencies: the 8-point transform of the sums
    const float a0 = s[0] + s[4], a1 = s[1] + s[5], a2 = s[2] + s[6], a3 = s[3] + s[7];
    const float b0 = s[0] - s[4], b1 = s[1] - s[5], b2 = s[2] - s[6], b3 = s[3] - s[7];
    const float h0 = a0 + a2, h1 = a1 + a3, m = b1 - b3, q = b1 + b3;
    X[0] = h0 + h1;
    X[8] = h0 - h1;
    X[4] = a0 - a2;
    X[12] = a1 - a3;
    X[2] = fmaf(kS2, m, b0);
    X[6] = fmaf(-kS2, m, b0);
    X[14] = fmaf(kS2, q, b2);
    X[10] = fmaf(kS2, q, -b2);
    // odd frequencies: rotations by pi/8 and 3 pi/8 as cos(pi/8) times a shear
    const float m2 = d[2] - d[6], q2 = d[2] + d[6];
    const float Pr = fmaf(kS2, m2, d[0]), Mr = fmaf(-kS2, m2, d[0]);
    const float Pq = fmaf(kS2, q2, d[4]), Mq = fmaf(-kS2, q2, d[4]);
    const float e1 = fmaf(-kT1, d[5], d[1]), f1 = fmaf(kT1, d[1], d[5]);
    const float e3 = fmaf(kT1, d[3], -d[7]), f3 = fmaf(kT1, d[7], d[3]);
    const float Ua = e1 + e3, Da = e1 - e3, Ub = f1 + f3, Db = f1 - f3;
    X[1] = fmaf(kC1, Ua, Pr);
    X[7] = fmaf(-kC1, Ua, Pr);
    X[15] = fmaf(kC1, Ub, Pq);
    X[9] = fmaf(kC1, Ub, -Pq);
    X[5] = fmaf(-kC1, Db, Mr);
    X[3] = fmaf(kC1, Db, Mr);
    X[11] = fmaf(kC1, Da, Mq);
    X[13] = fmaf(kC1, Da, -Mq);
}

// The transposed matrix: z_n = sum_i basis_i(n) Y_i.  With coefficients 1..7
// and 9..15 doubled beforehand, 16 times the inverse of rdft16.
__device__ __forceinline__ void rdft16_t(const float (&Y)[16], float (&z)[16]) {
    const float e = Y[0] + Y[8], f = Y[0] - Y[8];
    const float a0 = e + Y[4], a1 = f + Y[12], a2 = e - Y[4], a3 = f - Y[12];
    const float rp = Y[2] + Y[6], rm = Y[2] - Y[6], sp = Y[14] + Y[10], sm = Y[14] - Y[10];
    const float w1 = rm + sp, w3 = sp - rm;
    const float s[8] = {a0 + rp, fmaf(kS2, w1, a1),  a2 + sm, fmaf(kS2, w3, a3),
                        a0 - rp, fmaf(-kS2, w1, a1), a2 - sm, fmaf(-kS2, w3, a3)};
    const float Pr = Y[1] + Y[7], Ua = Y[1] - Y[7], Pq = Y[15] - Y[9], Ub = Y[15] + Y[9];
    const float Mr = Y[5] + Y[3], Db = Y[3] - Y[5], Mq = Y[11] - Y[13], Da = Y[11] + Y[13];
    const float m = Pr - Mr, q = Pq - Mq;
    const float A1 = Ua + Da, A3 = Ua - Da, B1 = Ub + Db, B3 = Ub - Db;
    const float d[8] = {Pr + Mr, fmaf(kT1, B1, A1),  m + q, fmaf(kT1, A3, B3),
                        Pq + Mq, fmaf(-kT1, A1, B1), q - m, fmaf(kT1, B3, -A3)};
    constexpr float k[8] = {1.0f, kC1, kS2, kC1, 1.0f, kC1, kS2, kC1};
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        z[n] = fmaf(k[n], d[n], s[n]);
        z[n + 8] = fmaf(-k[n], d[n], s[n]);
    }
}

// a - b of a pair in one packed instruction (operator- spends a pair of
// registers on the factor -1)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    unsigned long long x, y, r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(x), "l"(y));
    float2 o;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(o.x), "=f"(o.y) : "l"(r));
    return o;
}

// ---- shared memory ---------------------------------------------------------------
// Transpose buffer of a half-warp: 16 rows of 16 floats, 20 apart, so that the
// lanes' row reads (128 bits) fall on distinct banks; the two halves' buffers
// are 336 floats apart, so that their column writes do too.
constexpr int kRow = 20;
constexpr int kHalfBuf = 336;
constexpr int kBufFloats = 2 * kHalfBuf;
// Weight table: [kr = 0..8][kc = 0..8], rows 12 apart, of -131072 / (fr fc)
// M^2/256 for bins (kr, kc), then the same for (kr, -kc); f is 2 for
// frequencies 1..7 (their inverse basis counts twice) and 1 for 0 and 8.
constexpr int kTabRow = 12;
constexpr int kTab = 9 * kTabRow;
constexpr int kTabFloats = 2 * kTab;

// A vector of the warp's two tiles: [quad][lane] float4s.
__device__ __forceinline__ void load_vec(const float4* p, int lane, float2 (&z)[8]) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float4 v = lds_v4_volatile(p + q * 32 + lane);
        z[2 * q] = make_float2(v.x, v.y);
        z[2 * q + 1] = make_float2(v.z, v.w);
    }
}
__device__ __forceinline__ void store_vec(float4* p, int lane, const float2 (&z)[8]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
        p[q * 32 + lane] = make_float4(z[2 * q].x, z[2 * q].y, z[2 * q + 1].x, z[2 * q + 1].y);
}

constexpr int kVec = 128;  // float4s of one vector of a warp's two tiles
constexpr int kVecs = 5;   // -c, gamma and the history s, y and -Q s

template <bool Batch>
__host__ __device__ constexpr size_t pair_warp_bytes() {
    return kBufFloats * sizeof(float) + kVecs * kVec * sizeof(float4) +
           (Batch ? 2 * kTabFloats * sizeof(float) + 2 * sizeof(StackDesc) : 0);
}
template <bool Batch>
constexpr size_t pair_smem_bytes() {
    return (Batch ? 0 : kTabFloats * sizeof(float)) + kWarps * pair_warp_bytes<Batch>();
}

// ---- sums over a half-warp ----------------------------------------------------------
__device__ __forceinline__ double half_sum_d(double v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}
__device__ __forceinline__ float half_sum_f(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    return v;
}

// Half-warp totals of four FP64 values (warp_sum4_d over 16 lanes).
__device__ __forceinline__ void half_sum4_d(double& a, double& b, double& c, double& d, int lane) {
    const bool up8 = (lane & 8) != 0, up4 = (lane & 4) != 0;
    double v0 = (up8 ? c : a) + __shfl_xor_sync(kFull, up8 ? a : c, 8);
    double v1 = (up8 ? d : b) + __shfl_xor_sync(kFull, up8 ? b : d, 8);
    v0 = (up4 ? v1 : v0) + __shfl_xor_sync(kFull, up4 ? v0 : v1, 4);
    v0 += __shfl_xor_sync(kFull, v0, 2);
    v0 += __shfl_xor_sync(kFull, v0, 1);
    a = __shfl_sync(kFull, v0, 0, 16);
    b = __shfl_sync(kFull, v0, 4, 16);
    c = __shfl_sync(kFull, v0, 8, 16);
    d = __shfl_sync(kFull, v0, 12, 16);
}

// 3-input minimum and maximum (sm_100)
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

struct Geo {
    const float* data;
    const float* gamma;
    float* out;
    long long gstride;
    int H, W, tiles_x, tiles_y;
};

template <bool Batch>
__device__ __forceinline__ Geo geo_of(const SolveArgs& a, const StackDesc& sd) {
    if constexpr (Batch)
        return Geo{sd.data, sd.gamma, sd.out, sd.gamma_frame_stride, sd.H, sd.W, sd.tiles_x,
                   sd.tiles_y};
    else
        return Geo{a.data, a.gamma, a.out, a.gamma_frame_stride, a.H, a.W, a.tiles_x, a.tiles_y};
}

// Entry e of a weight table from M^2/256 of its bin.
__device__ __forceinline__ float tab_scale(int kr, int kc) {
    return -131072.0f * ((kr & 7) ? 0.5f : 1.0f) * ((kc & 7) ? 0.5f : 1.0f);
}

// log1p(x) = 2 atanh(y), y = x / (2 + x).  2 atanh(y) / y as a polynomial in
// y^2, fitted for the relative error: with these FP32 coefficients 8e-9 for
// |y| <= 1/3 (x in -1/2 .. 1) and 2e-8 for |y| <= 0.7 (x in -0.82 .. 4.7), which
// first iterations need; evaluated in FP32 1.3e-7 and 1.4e-7, its own roundings.
constexpr float kNear = 1.0f / 3.0f, kFar = 0.7f;
__device__ constexpr float kNearPoly[5] = {2.0f, 0.666663147f, 0.400249103f, 0.279606027f,
                                           0.281783351f};
__device__ constexpr float kFarPoly[9] = {2.0f,         0.666660494f, 0.400321418f,
                                          0.279324231f, 0.285048438f, -0.158120584f,
                                          1.19674649f,  -1.60518426f, 1.41868061f};

}  // namespace

// Warm: the launch carries proposals (a.u0).  Batch: tiles of several stacks
// share the queue; each half finds its tile's stack by binary search.
// `one_wave`: the grid holds a warp for every pair of tiles, so warps take
// their pair by index and the queue is not touched.  The Late = false instance is
// never launched that way, but its tests stay: without them the compiler schedules
// its pass 0.3 to 2 % slower (stack512 1,303 us with them, 1,307 to 1,334 in seven
// spellings without).
// Late: a warp takes its first pair by index and, for the last two pairs that
// it can expect, draws the next one only when it is free: a pair drawn ahead
// waits for whoever drew it, and just above a full wave that doubled the
// launch (848 x 848, 3,721 tiles: 39.7 -> 30.4 us; 3.7 waves: 77.0 -> 75.7).
// Elsewhere the draw's latency hides behind the solve.  A batch draws late
// throughout (16 stacks: 627 -> 580 us; with the far draws ahead 597).
template <int MinBlocks, bool Warm, bool Batch, bool Late>
__global__ void __launch_bounds__(kWarpCtaThreads, MinBlocks)
ncs_pair_kernel(const SolveArgs a, const int one_wave) {
    extern __shared__ __align__(16) unsigned char dsm[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int h = lane >> 4, c = lane & 15;
    constexpr size_t kCtaTab = Batch ? 0 : kTabFloats * sizeof(float);
    unsigned char* wbase = dsm + kCtaTab + (size_t)wid * pair_warp_bytes<Batch>();
    float* buf = reinterpret_cast<float*>(wbase) + h * kHalfBuf;
    float4* terms = reinterpret_cast<float4*>(wbase + kBufFloats * sizeof(float));
    float4* gterm = terms + kVec;
    float4* hs = terms + 2 * kVec;
    float4* hy = terms + 3 * kVec;
    float4* hq = terms + 4 * kVec;
    // Batch: the halves' weight tables and stack descriptors
    float* btab = reinterpret_cast<float*>(terms + kVecs * kVec);
    StackDesc* sdesc = reinterpret_cast<StackDesc*>(btab + 2 * kTabFloats);

    const float eps2 = a.eps * a.eps;
    const long long n_pairs = (a.n_tiles + 1) >> 1;
    // in the coefficient stage lane c holds row coefficient c: frequency kr
    const int kr = c <= 8 ? c : 16 - c;
    const float fr = (kr & 7) ? 2.0f : 1.0f;
    const float* tab = (Batch ? btab + h * kTabFloats : reinterpret_cast<const float*>(dsm)) +
                       kr * kTabRow;
    bool asym = false;  // any bin with M^2(kr, kc) != M^2(kr, -kc)
    float alpha = a.alpha;
    long long st_begin = 0, st_end = 0;  // Batch: tiles of the half's current stack
    if constexpr (!Batch) {
        float* ct = reinterpret_cast<float*>(dsm);
        bool diff = false;
        for (int idx = threadIdx.x; idx < kTab; idx += blockDim.x) {
            const int r = idx / kTabRow, k = idx - r * kTabRow;
            if (k < 9) {
                const float s = tab_scale(r, k);
                const float A = a.msq[r * 16 + k], B = a.msq[r * 16 + ((16 - k) & 15)];
                ct[idx] = s * A;
                ct[kTab + idx] = s * B;
                diff = diff || A != B;
            }
        }
        asym = __syncthreads_or(diff) != 0;
    }

    long long pair = (long long)wid * gridDim.x + blockIdx.x;
    if (!Late && !one_wave) {
        unsigned long long tk = 0;
        if (lane == 0) tk = atomicAdd(a.queue, 1ull);
        pair = (long long)__shfl_sync(kFull, tk, 0);
    }
    const long long late_from = n_pairs - 8LL * gridDim.x;
    while (pair < n_pairs) {
        // the next pair's index, fetched while this one is solved
        unsigned long long tk = 0;
        const bool ahead = Late ? !Batch && pair < late_from : !one_wave;
        if (ahead && lane == 0) tk = atomicAdd(a.queue, 1ull);
        const long long tile = min(2 * pair + h, a.n_tiles - 1);
        bool act = 2 * pair + h < a.n_tiles;
        long long lt = tile;  // index of the tile within its stack
        if constexpr (Batch) {
            // the half's stack, when this tile is not in the last one's (looking it
            // up for every tile cost 5 %: 16 stacks, 0.66 -> 0.62 ms)
            if (__any_sync(kFull, tile < st_begin || tile >= st_end)) {
                int lo = 0, hi = a.n_stacks - 1;
                while (lo < hi) {  // last stack whose first tile is <= tile
                    const int mid = (lo + hi + 1) >> 1;
                    if (__ldg(&a.stacks[mid].tile_begin) <= tile) lo = mid;
                    else hi = mid - 1;
                }
                st_begin = __ldg(&a.stacks[lo].tile_begin);
                st_end = lo + 1 < a.n_stacks ? __ldg(&a.stacks[lo + 1].tile_begin) : a.n_tiles;
                __syncwarp();
                if (c == 0) sdesc[h] = a.stacks[lo];
                // the half's weight tables from the stack's lane-layout table
                const float* ml = a.mk_lane + (size_t)lo * 256;
                bool diff = false;
                for (int idx = c; idx < kTab; idx += 16) {
                    const int r = idx / kTabRow, k = idx - r * kTabRow;
                    if (k < 9) {
                        const int kn = (16 - k) & 15, i = bitrev3(r >> 1);
                        const float s = tab_scale(r, k);
                        const float A = __ldg(ml + (2 * k + (r & 1)) * 8 + i);
                        const float B = __ldg(ml + (2 * kn + (r & 1)) * 8 + i);
                        btab[h * kTabFloats + idx] = s * A;
                        btab[h * kTabFloats + kTab + idx] = s * B;
                        diff = diff || A != B;
                    }
                }
                asym = __any_sync(kFull, diff);
                __syncwarp();
            }
            lt = tile - sdesc[h].tile_begin;
            alpha = sdesc[h].alpha;
        }

        // ---- gather the tiles (segmentation, ncs.c:66-113) ----------------------
        float2 u[8];
        int f = 0, ox = 0, oy = 0, own_r = 0, own_c = 0;
        if (!a.tile_mode) {
            const Geo sg = geo_of<Batch>(a, sdesc[h]);
            const long long per_frame = (long long)sg.tiles_x * sg.tiles_y;
            f = (int)(lt / per_frame);
            const int rem = (int)(lt - (long long)f * per_frame);
            const int ti = rem / sg.tiles_y, tj = rem - (rem / sg.tiles_y) * sg.tiles_y;
            ox = tile_origin(ti, sg.H);
            oy = tile_origin(tj, sg.W);
            own_r = (ti + 1 < sg.tiles_x ? tile_origin(ti + 1, sg.H) : ox + 14) - ox;
            own_c = (tj + 1 < sg.tiles_y ? tile_origin(tj + 1, sg.W) : oy + 14) - oy;
        }
        // the tile's photon image; also gm, its gamma, when given
        auto load_tile = [&](float2 (&d)[8], float2* gm) {
            if (a.tile_mode) {
                const long long base = tile * kPix + c;
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    (r & 1 ? d[r >> 1].y : d[r >> 1].x) = __ldg(a.data + base + r * kTile);
                    if (gm) (r & 1 ? gm[r >> 1].y : gm[r >> 1].x) = __ldg(a.gamma + base + r * kTile);
                }
            } else {
                const Geo sg = geo_of<Batch>(a, sdesc[h]);
                const int col = clampi(oy + c - 1, 0, sg.W - 1);
                const float* img = sg.data + (long long)f * sg.H * sg.W + col;
                const float* gmap = sg.gamma + (long long)f * sg.gstride + col;
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    const long long row = (long long)clampi(ox + r - 1, 0, sg.H - 1) * sg.W;
                    (r & 1 ? d[r >> 1].y : d[r >> 1].x) = __ldg(img + row);
                    if (gm) (r & 1 ? gm[r >> 1].y : gm[r >> 1].x) = __ldg(gmap + row);
                }
            }
        };
        {
            float2 gm[8], nc[8];
            load_tile(u, gm);
#pragma unroll
            for (int j = 0; j < 8; ++j)
                nc[j] = make_float2(-(u[j].x + gm[j].x), -(u[j].y + gm[j].y));
            store_vec(terms, lane, nc);
            store_vec(gterm, lane, gm);
            // no pair yet: a zero history with rho = 0 leaves every update out
#pragma unroll
            for (int j = 0; j < 8; ++j) nc[j] = make_float2(0.0f, 0.0f);
            store_vec(hy, lane, nc);
            store_vec(hq, lane, nc);
            if constexpr (Warm) {
                // s's place first holds u0 - d, for the start pass
                const float* ut = a.u0 + tile * kPix + c;
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    float& ui = r & 1 ? u[r >> 1].y : u[r >> 1].x;
                    const float di = ui;
                    ui = __ldg(ut + r * kTile);
                    (r & 1 ? nc[r >> 1].y : nc[r >> 1].x) = __fsub_rn(ui, di);
                }
            }
            store_vec(hs, lane, nc);
        }

        // ---- preconditioned L-BFGS, both tiles in lock step -----------------------
        // Names and signs as in ncs_spectral.cu: the transformed vector is nq = -q,
        // wn = -w = -2 alpha Q p, the history keeps wn unscaled with its step tq.
        float2 p[8], wn[8], v[8], g[8], nq[8];
        float rho = 0.0f, al = 0.0f, tq = 0.0f;
        bool sg_fresh = false, have = false;
        int status = kUnstarted, iters = 0, evals = 1;
        float lam = 1.0f;
        bool first = true;
        int start_pass = Warm ? 2 : 0;  // as in ncs_spectral.cu, for the warp
        bool taken = false;             // Warm: this half's proposal passed the bound
        int fell_back = 0;

        for (;;) {
            if (first) {
                if (Warm && start_pass == 1) {
                    load_tile(nq, nullptr);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) nq[j] = u[j];
                }
            } else if (__any_sync(kFull, act && have && !sg_fresh)) {
                // the last step added no pair: the two-loop's first half with the
                // pair kept from before (nq = g here)
                float2 hv[8], acc = make_float2(0.0f, 0.0f);
                load_vec(hs, lane, hv);
#pragma unroll
                for (int j = 0; j < 8; ++j) acc = fma2(hv[j], nq[j], acc);
                const float dot = -half_sum_f(acc.x + acc.y);  // s'q, q = -g
                if (have && !sg_fresh) {
                    al = rho * dot;
                    load_vec(hy, lane, hv);
                    const float2 a2 = splat(al);
#pragma unroll
                    for (int j = 0; j < 8; ++j) nq[j] = fma2(a2, hv[j], nq[j]);
                }
            }

            // ---- p = H0 q (first: 2 alpha Q u) ------------------------------------
            {
                // two real transforms with a transpose between them, each pair as a
                // loop: the pass is about as long as the instruction cache serves
                // well (unrolled it ran 1.5 % slower)
                float X[16], z[16];
                auto transpose = [&](const float (&in)[16], float (&out)[16]) {
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < 16; ++i) buf[i * kRow + c] = in[i];
                    __syncwarp();
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 o = *reinterpret_cast<const float4*>(buf + c * kRow + 4 * q);
                        out[4 * q] = o.x;
                        out[4 * q + 1] = o.y;
                        out[4 * q + 2] = o.z;
                        out[4 * q + 3] = o.w;
                    }
                };
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    z[2 * j] = nq[j].x;
                    z[2 * j + 1] = nq[j].y;
                }
#pragma unroll 1
                for (int stage = 0;; ++stage) {
                    rdft16(z, X);
                    if (stage == 1) break;
                    transpose(X, z);
                }
                // weights: -(fr fc / 256) / (lam + 2 alpha M^2), or 2 alpha M^2 / 256
                // fr fc on the first pass (fr fc: the inverse basis counts
                // frequencies 1..7 twice)
                float tw[9], w[9];
                auto weights = [&](const float* t) {
                    const float4 t0 = *reinterpret_cast<const float4*>(t);
                    const float4 t1 = *reinterpret_cast<const float4*>(t + 4);
                    tw[0] = t0.x; tw[1] = t0.y; tw[2] = t0.z; tw[3] = t0.w;
                    tw[4] = t1.x; tw[5] = t1.y; tw[6] = t1.z; tw[7] = t1.w;
                    tw[8] = t[8];
                    if (first) {
                        const float s = -alpha * fr * fr * (1.0f / 65536.0f);
#pragma unroll
                        for (int k = 0; k < 9; ++k) w[k] = s * tw[k] * ((k & 7) ? 4.0f : 1.0f);
                    } else {
                        const float le = lam * (-256.0f / fr), lm = 0.5f * le;
#pragma unroll
                        for (int k = 0; k < 9; ++k)
                            w[k] = rcp_fast(fmaf(alpha, tw[k], (k & 7) ? lm : le));
                    }
                };
                weights(tab);
                if (asym) {
                    // bins (kr, kc) and (kr, -kc) have weights a and b: the cos-cos
                    // and sin-sin coefficients mix, and so do cos-sin and sin-cos,
                    // with P = (a + b) / 2 and N = (a - b) / 2.  A solve with such a mask
                    // takes a tenth longer (200 x 512 x 512: 990 us radial, 1,087 so; one
                    // tile per warp: 1,510 either way), a batch of 16 stacks 0.1 us more
                    // with one of them, 4 of 56 with all
                    float wa[9];
#pragma unroll
                    for (int k = 0; k < 9; ++k) wa[k] = w[k];
                    weights(tab + kTab);
                    const int partner = (lane & 16) | ((16 - c) & 15);
                    const float sg = c > 8 ? -1.0f : 1.0f;  // this lane holds sines
#pragma unroll
                    for (int k = 1; k < 8; ++k) {
                        const float P = 0.5f * (wa[k] + w[k]), N = 0.5f * (wa[k] - w[k]);
                        const float oc = __shfl_sync(kFull, X[k], partner);
                        const float os = __shfl_sync(kFull, X[16 - k], partner);
                        X[k] = P * X[k] - sg * N * os;
                        X[16 - k] = P * X[16 - k] + sg * N * oc;
                    }
                    X[0] *= wa[0];
                    X[8] *= wa[8];
                } else {
                    X[0] *= w[0];
                    X[8] *= w[8];
#pragma unroll
                    for (int k = 1; k < 8; ++k) {
                        X[k] *= w[k];
                        X[16 - k] *= w[k];
                    }
                }
#pragma unroll 1
                for (int stage = 0;; ++stage) {
                    rdft16_t(X, z);
                    if (stage == 1) break;
                    transpose(z, X);
                }
#pragma unroll
                for (int j = 0; j < 8; ++j) p[j] = make_float2(z[2 * j], z[2 * j + 1]);
            }

            bool fin = false;
            if (first) {
                if (Warm && start_pass == 2) {
                    // the bound of ncs_spectral.cu: accept a proposal with
                    // LL(u0) - LL(d) + (u0 - d)'v0 <= 0 without transforming d
                    float2 de[8], nc[8], gm[8];
                    load_vec(hs, lane, de);
                    load_vec(terms, lane, nc);
                    load_vec(gterm, lane, gm);
                    double bound = 0.0;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {  // FP32 over 8 pixels, then FP64
                        float dl = 0.0f, dq = 0.0f;
#pragma unroll
                        for (int j = 4 * b; j < 4 * b + 4; ++j)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const float ui = e ? u[j].y : u[j].x, di = e ? de[j].y : de[j].x;
                                const float gi = e ? gm[j].y : gm[j].x, ci = e ? nc[j].y : nc[j].x;
                                const float pi = e ? p[j].y : p[j].x;
                                const float lr = __fsub_rn(__logf(fmaxf(ui + gi, kFitMin)),
                                                           __logf(fmaxf(-ci, kFitMin)));
                                dl += fmaf(ci, lr, di);
                                dq += __fmul_rn(di, pi);
                            }
                        bound += (double)dl + (double)dq;
                    }
                    bound = half_sum_d(bound);
                    taken = bound <= 0.0;
                    if (__any_sync(kFull, act && !taken)) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) wn[j] = p[j];
                        start_pass = 1;
                        continue;
                    }
                } else if (Warm && start_pass == 1) {
                    // exact comparison (see ncs_spectral.cu): p = 2 alpha Q d, wn =
                    // 2 alpha Q u0; explicitly rounded, so that u0 = d gives 0
                    float2 dd[8], nc[8], gm[8];
                    load_tile(dd, nullptr);
                    load_vec(terms, lane, nc);
                    load_vec(gterm, lane, gm);
                    double delta = 0.0;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        float dl = 0.0f, dq = 0.0f;
#pragma unroll
                        for (int j = 4 * b; j < 4 * b + 4; ++j)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const float ui = e ? u[j].y : u[j].x, di = e ? dd[j].y : dd[j].x;
                                const float gi = e ? gm[j].y : gm[j].x, ci = e ? nc[j].y : nc[j].x;
                                const float pi = e ? p[j].y : p[j].x, wi = e ? wn[j].y : wn[j].x;
                                const float lr = __fsub_rn(__logf(fmaxf(ui + gi, kFitMin)),
                                                           __logf(fmaxf(di + gi, kFitMin)));
                                dl += fmaf(ci, lr, ui - di);
                                dq += __fsub_rn(__fmul_rn(ui, wi), __fmul_rn(di, pi));
                            }
                        delta += (double)dl + 0.5 * (double)dq;
                    }
                    delta = half_sum_d(delta);
                    if (taken || delta <= 0.0) {
#pragma unroll
                        for (int j = 0; j < 8; ++j) p[j] = wn[j];
                    } else {
                        fell_back = 1;
#pragma unroll
                        for (int j = 0; j < 8; ++j) u[j] = dd[j];
                    }
                }
                if constexpr (Warm) {
                    float2 z[8];
#pragma unroll
                    for (int j = 0; j < 8; ++j) z[j] = make_float2(0.0f, 0.0f);
                    store_vec(hs, lane, z);
                }
                start_pass = 0;
                first = false;
                float2 nc[8], gm[8];
                load_vec(terms, lane, nc);
                load_vec(gterm, lane, gm);
                float2 uu2 = make_float2(0.0f, 0.0f), gg2 = uu2, ll2 = uu2;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float2 A = u[j] + gm[j];
                    const float2 ia = make_float2(rcp_fast(fmaxf(A.x, kFitMin)),
                                                  rcp_fast(fmaxf(A.y, kFitMin)));
                    const float2 r = nc[j] * ia;  // -c / (u + gamma)
                    v[j] = p[j];
                    g[j] = (r + splat(1.0f)) + v[j];
                    nq[j] = g[j];
                    uu2 = fma2(u[j], u[j], uu2);
                    gg2 = fma2(g[j], g[j], gg2);
                    ll2 = fma2(r, ia, ll2);
                }
                const float uu = half_sum_f(uu2.x + uu2.y);
                const float gg = half_sum_f(gg2.x + gg2.y);
                lam = half_sum_f(ll2.x + ll2.y) * (-1.0f / 256.0f);
                if (gg <= eps2 * fmaxf(uu, 1.0f)) { status = kSuccess; fin = act; }
                else if (a.max_iters <= 0) { status = kReachedMaxIters; fin = act; }
            } else {
                // -w = -2 alpha Q H0 q = lambda H0 q - q; then the history's part:
                // p += coef s, wn += coef (-Q s)
                if (alpha > 0.0f) {
                    const float2 l2 = splat(lam);
#pragma unroll
                    for (int j = 0; j < 8; ++j) wn[j] = fma2(l2, p[j], nq[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < 8; ++j) wn[j] = make_float2(0.0f, 0.0f);
                }
                if (__any_sync(kFull, act && have)) {
                    float2 hv[8], acc = make_float2(0.0f, 0.0f);
                    load_vec(hy, lane, hv);
#pragma unroll
                    for (int j = 0; j < 8; ++j) acc = fma2(hv[j], p[j], acc);
                    const float coef = al - rho * half_sum_f(acc.x + acc.y);
                    const float2 cf = splat(coef), cq = splat(coef * tq);
                    load_vec(hs, lane, hv);
#pragma unroll
                    for (int j = 0; j < 8; ++j) p[j] = fma2(cf, hv[j], p[j]);
                    load_vec(hq, lane, hv);
#pragma unroll
                    for (int j = 0; j < 8; ++j) wn[j] = fma2(cq, hv[j], wn[j]);
                }

                // The slopes g'p, p'v, p'w and the cost change of the first trial
                // (t = 1), sum p - c log1p(p / A), A = u + gamma, in one FP64
                // reduction (FP32 over 8 pixels, then FP64).  log1p(p / A) =
                // 2 atanh(y), y = p / (2 A + p): one reciprocal per pixel.  |y| <=
                // kFar keeps the step inside the barrier and, with A above 1e-5,
                // the floor; a half with a pixel outside takes the general form
                // below.  Each half's choice depends on its own pixels only.
                double gd = 0.0, dpv = 0.0, dpw = 0.0, dl0 = 0.0;
                const unsigned half_mask = 0xffffu << (16 * h);
                bool out_any;
                {
                    float2 y[8];
                    float amin = 1.0f, ymax = 0.0f;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float4 gq = lds_v4_volatile(gterm + q * 32 + lane);
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int j = 2 * q + e;
                            const float2 A = u[j] + (e ? make_float2(gq.z, gq.w)
                                                       : make_float2(gq.x, gq.y));
                            const float2 den = (A + p[j]) + A;
                            y[j] = p[j] * make_float2(rcp_fast(den.x), rcp_fast(den.y));
                            amin = min3(amin, A.x, A.y);
                            ymax = max3(ymax, fabsf(y[j].x), fabsf(y[j].y));
                        }
                    }
                    const bool far = (__ballot_sync(kFull, !(ymax <= kNear)) & half_mask) != 0;
                    out_any = (__ballot_sync(kFull, !(amin >= 1.0e-5f && ymax <= kFar)) &
                               half_mask) != 0;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        float2 gp2 = make_float2(0.0f, 0.0f), pv2 = gp2, pw2 = gp2;
#pragma unroll
                        for (int j = 4 * b; j < 4 * b + 4; ++j) {
                            gp2 = fma2(g[j], p[j], gp2);
                            pv2 = fma2(v[j], p[j], pv2);
                            pw2 = fma2(wn[j], p[j], pw2);
                        }
                        gd += (double)(gp2.x + gp2.y);
                        dpv += (double)(pv2.x + pv2.y);
                        dpw += (double)(pw2.x + pw2.y);
                    }
                    // y -> log1p
                    if (__any_sync(kFull, act && far)) {
                        float k[9];
#pragma unroll
                        for (int i = 0; i < 9; ++i)
                            k[i] = far ? kFarPoly[i] : (i < 5 ? kNearPoly[i < 5 ? i : 0] : 0.0f);
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float2 y2 = y[j] * y[j];
                            float2 s = splat(k[8]);
#pragma unroll
                            for (int i = 7; i >= 0; --i) s = fma2(y2, s, splat(k[i]));
                            y[j] = y[j] * s;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const float2 y2 = y[j] * y[j];
                            float2 s = splat(kNearPoly[4]);
#pragma unroll
                            for (int i = 3; i >= 0; --i) s = fma2(y2, s, splat(kNearPoly[i]));
                            y[j] = y[j] * s;
                        }
                    }
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        float2 term = make_float2(0.0f, 0.0f);
#pragma unroll
                        for (int q = 2 * b; q < 2 * b + 2; ++q) {
                            const float4 cq = lds_v4_volatile(terms + q * 32 + lane);
                            term = term + fma2(make_float2(cq.x, cq.y), y[2 * q], p[2 * q]);
                            term = term + fma2(make_float2(cq.z, cq.w), y[2 * q + 1], p[2 * q + 1]);
                        }
                        dl0 += (double)(term.x + term.y);
                    }
                }
                half_sum4_d(gd, dpv, dpw, dl0, lane);
                dpw = -dpw;  // p'w = -p'wn

                // general trial at step t (ncs_spectral.cu): floor, barrier, log2
                auto trial = [&](float t, bool& cross) {
                    float2 nc[8], gm[8];
                    load_vec(terms, lane, nc);
                    load_vec(gterm, lane, gm);
                    const float2 t2 = splat(t);
                    cross = false;
                    double dl = 0.0;
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        float2 term = make_float2(0.0f, 0.0f);
#pragma unroll
                        for (int j = 4 * b; j < 4 * b + 4; ++j) {
                            const float2 ai = u[j] + gm[j];
                            const float2 tp = t2 * p[j];
                            const float2 ni = ai + tp;
                            const float2 bar = splat(kBarrierFrac) * ai;
                            float2 num, rA;
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const float a1 = e ? ai.y : ai.x, n1 = e ? ni.y : ni.x;
                                const bool in_dom = a1 >= kFitMin && n1 >= kFitMin;
                                const float A = fmaxf(a1, kFitMin);
                                const float nm = in_dom ? (e ? tp.y : tp.x) : fmaxf(n1, kFitMin) - A;
                                (e ? num.y : num.x) = nm;
                                (e ? rA.y : rA.x) = rcp_fast(A);
                                cross |= (a1 >= kFitMin) && (n1 < (e ? bar.y : bar.x));
                            }
                            term = term + fma2(nc[j], log1p_ls(num * rA), tp);
                        }
                        dl += (double)(term.x + term.y);
                    }
                    return half_sum_d(dl);
                };
                float t = 1.0f;
                bool ok = false, skip = false;
                if (__any_sync(kFull, act && !(gd < 0.0))) {
                    // not a descent direction: drop the history (H0 alone is positive
                    // definite); fail only if even that does not descend
                    if (!(gd < 0.0)) {
                        if (!have) { status = kIncreasingGradient; fin = act; }
                        have = false;
                        sg_fresh = false;
                        rho = al = tq = 0.0f;
                        skip = true;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            p[j] = wn[j] = make_float2(0.0f, 0.0f);  // u, v and g stay
                        store_vec(hs, lane, p);
                        store_vec(hy, lane, p);
                        store_vec(hq, lane, p);
                    }
                }
                if (!skip && !out_any) {
                    ++evals;
                    ok = dl0 + dpv + 0.5 * dpw <= (double)a.c1 * gd;
                }
                // the general form: from t = 1 where the fast form did not apply,
                // else Armijo backtracking from t = 1/2
                bool search = act && !skip && !ok, at_one = out_any;
                if (__any_sync(kFull, search)) {
                    for (int k = 0; k < 64; ++k) {
                        if (search && !at_one) {
                            t *= 0.5f;
                            if (!(t >= a.min_step)) search = false;  // also stops on NaN
                        }
                        at_one = false;
                        if (!__any_sync(kFull, search)) break;
                        bool cross;
                        const double dl = trial(t, cross);
                        const bool ca = (__ballot_sync(kFull, cross) & half_mask) != 0;
                        if (search) {
                            ++evals;
                            const double td = (double)t;
                            const double delta = ca ? CUDART_INF : dl + td * dpv + 0.5 * td * td * dpw;
                            if (delta <= (double)a.c1 * td * gd) { ok = true; search = false; }
                        }
                    }
                    if (act && !skip && !ok) {
                        status = kMinimumStep;
                        fin = true;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            p[j] = wn[j] = make_float2(0.0f, 0.0f);  // u and v stay
                    }
                }

                // accept; new pair (s, y, -Q s = t wn, stored as wn and t)
                float2 s[8], y[8];
                const float2 z2 = make_float2(0.0f, 0.0f), t2 = splat(t);
                float2 sy2 = z2, uu2 = z2, gg2 = z2, ll2 = z2, mv2 = z2, sg2 = z2;
                {
                    float2 nc[8], gm[8];
                    load_vec(terms, lane, nc);
                    load_vec(gterm, lane, gm);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const float2 un = fma2(t2, p[j], u[j]);
                        v[j] = fma2(splat(-t), wn[j], v[j]);  // v += t w
                        const float2 A = un + gm[j];
                        const float2 ia = make_float2(rcp_fast(fmaxf(A.x, kFitMin)),
                                                      rcp_fast(fmaxf(A.y, kFitMin)));
                        const float2 r = nc[j] * ia;  // -c / (u + gamma)
                        const float2 gn = (r + splat(1.0f)) + v[j];
                        s[j] = sub2(un, u[j]);
                        y[j] = sub2(gn, g[j]);
                        mv2 = fma2(s[j], s[j], mv2);  // zero when no pixel moved
                        u[j] = un;
                        g[j] = gn;
                        sy2 = fma2(s[j], y[j], sy2);
                        sg2 = fma2(s[j], gn, sg2);
                        uu2 = fma2(un, un, uu2);
                        gg2 = fma2(gn, gn, gg2);
                        ll2 = fma2(r, ia, ll2);
                    }
                }
                float vals[8] = {sy2.x + sy2.y, uu2.x + uu2.y, gg2.x + gg2.y,
                                 ll2.x + ll2.y, mv2.x + mv2.y, sg2.x + sg2.y, 0.0f, 0.0f};
#pragma unroll
                for (int o = 4; o >= 1; o >>= 1) {
                    const bool up = (lane & o) != 0;
#pragma unroll
                    for (int i = 0; i < o; ++i) {
                        const float send = up ? vals[i] : vals[i + o];
                        vals[i] = (up ? vals[i + o] : vals[i]) + __shfl_xor_sync(kFull, send, o);
                    }
                }
                const float tot = vals[0] + __shfl_xor_sync(kFull, vals[0], 8);
                const float sy = __shfl_sync(kFull, tot, 0, 16);
                const float uu = __shfl_sync(kFull, tot, 1, 16);
                const float gg = __shfl_sync(kFull, tot, 2, 16);
                const float ll = __shfl_sync(kFull, tot, 3, 16);
                const float mv = __shfl_sync(kFull, tot, 4, 16);
                const float sg = __shfl_sync(kFull, tot, 5, 16);
                float a_new = 0.0f;  // first two-loop coefficient of the new pair
                if (act && !fin && !skip) {
                    ++iters;
                    lam = ll * (-1.0f / 256.0f);
                    sg_fresh = sy > 0.0f;
                    if (gg <= eps2 * fmaxf(uu, 1.0f)) { status = kSuccess; fin = true; }
                    else if (mv == 0.0f) { status = kReachedMaxPrecision; fin = true; }
                    else if (iters >= a.max_iters) { status = kReachedMaxIters; fin = true; }
                    else if (sy > 0.0f) {
                        have = true;
                        rho = rcp_fast(sy);
                        tq = t;
                        al = a_new = -rho * sg;  // rho s'q, q = -g
                        store_vec(hs, lane, s);
                        store_vec(hy, lane, y);
                        store_vec(hq, lane, wn);
                    }
                }
                const float2 a2 = splat(a_new);
#pragma unroll
                for (int j = 0; j < 8; ++j) nq[j] = fma2(a2, y[j], g[j]);
            }

            // ---- outputs of the halves that ended with this pass ---------------------
            if (__any_sync(kFull, fin)) {
                if (a.cost) {
                    if constexpr (Batch) {
                        float2 nc[8], gm[8];
                        load_vec(terms, lane, nc);
                        load_vec(gterm, lane, gm);
                        double e0 = 0.0, e1 = 0.0;
#pragma unroll
                        for (int j = 0; j < 8; ++j)
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                const double ui = e ? u[j].y : u[j].x, gi = e ? gm[j].y : gm[j].x;
                                e0 += ui + (double)(e ? nc[j].y : nc[j].x) * log(fmax(ui + gi, 1.0e-6));
                                e1 += ui * (e ? v[j].y : v[j].x);
                            }
                        e0 = half_sum_d(e0);
                        e1 = half_sum_d(e1);
                        if (fin && c == 0) a.cost[tile] = e0 + 0.5 * e1;  // v = 2 alpha Q u
                    } else {
                        // rolled, with u through shared memory: sixteen inlined FP64 logs
                        // are as much code as the pass and cost the instruction cache
                        // 2.5 % of a solve that does not ask for them (the batched
                        // instance ran 6 % slower rolled)
                        double e0 = 0.0, e1 = 0.0;
                        __syncwarp();
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            buf[(2 * j) * kRow + c] = u[j].x;
                            buf[(2 * j + 1) * kRow + c] = u[j].y;
                            e1 += (double)u[j].x * v[j].x;
                            e1 += (double)u[j].y * v[j].y;
                        }
#pragma unroll 1
                        for (int r = 0; r < 16; ++r) {
                            const int at = (r >> 2) * 128 + lane * 4 + (r & 3);
                            const double ui = buf[r * kRow + c];
                            e0 += ui + (double)reinterpret_cast<const float*>(terms)[at] *
                                           log(fmax(ui + reinterpret_cast<const float*>(gterm)[at], 1.0e-6));
                        }
                        e0 = half_sum_d(e0);
                        e1 = half_sum_d(e1);
                        if (fin && c == 0) a.cost[tile] = e0 + 0.5 * e1;  // v = 2 alpha Q u
                    }
                }
                if (fin) {
                    act = false;
                    if (c == 0) {
                        if (a.iters) a.iters[tile] = iters;
                        if (a.status) a.status[tile] = status;
                        if (a.evals) a.evals[tile] = evals;
                        if (Warm && a.start) a.start[tile] = fell_back;
                    }
                    if (a.tile_mode) {
                        float* o = a.out + tile * kPix + c;
#pragma unroll
                        for (int r = 0; r < 16; ++r)
                            o[r * kTile] = r & 1 ? u[r >> 1].y : u[r >> 1].x;
                    } else if (c >= 1 && c <= own_c) {
                        const Geo sg = geo_of<Batch>(a, sdesc[h]);
                        float* o = sg.out + (long long)f * sg.H * sg.W + (long long)(ox - 1) * sg.W +
                                   oy + c - 1;
#pragma unroll
                        for (int r = 1; r < 15; ++r)
                            if (r <= own_r)
                                o[(long long)r * sg.W] = r & 1 ? u[r >> 1].y : u[r >> 1].x;
                    }
                }
                if (!__any_sync(kFull, act)) break;
            }
        }
        if constexpr (Late) {
            if (one_wave) break;
            if (!ahead && lane == 0) tk = atomicAdd(a.queue, 1ull);
            pair = (long long)__shfl_sync(kFull, tk, 0) + 4LL * gridDim.x;
        } else {
            if (one_wave) pair += 4LL * gridDim.x;
            else pair = (long long)__shfl_sync(kFull, tk, 0);
        }
        __syncwarp();  // every lane is done with this pair's shared memory
    }
}

namespace {

// CTAs per SM: 3 (12 warps, 24 tiles, 168 registers).  On stack512, in an earlier
// state of the kernel, 3 CTAs ran 1.37 ms (1.31 now); 2 (no spills, 8 warps) 1.56
// ms; 4 (128 registers, 200 B spilled) 1.62 ms.
constexpr int kPairBlocks = 3;

using PairFn = void (*)(SolveArgs, int);

// Launches of this many waves draw ahead to the end: the tail is short there
// and the plainer loop compiles to the faster pass (stack512, 77 waves: 1,306
// us against 1,326; at 11 waves, 60 x 411 x 301 raw counts, 226 either way; at
// 3.7 waves 77.0 against 75.7).  Launches with proposals draw late at every size:
// theirs gained at 19 waves too (50 x 512 x 512, inference included: 1,285 ->
// 1,279 us).
constexpr long long kAheadWaves = 4;

PairFn pair_variant(bool warm, bool batch, bool late) {
    if (batch) return warm ? ncs_pair_kernel<kPairBlocks, true, true, true>
                           : ncs_pair_kernel<kPairBlocks, false, true, true>;
    if (warm) return ncs_pair_kernel<kPairBlocks, true, false, true>;
    return late ? ncs_pair_kernel<kPairBlocks, false, false, true>
                : ncs_pair_kernel<kPairBlocks, false, false, false>;
}

}  // namespace

// CTAs of a launch over n_tiles tiles: a warp per pair of tiles up to
// ctas_per_sm (0: kPairBlocks) CTAs on each SM, spread over the SMs first.
long long pair_grid(long long n_tiles, int ctas_per_sm, int num_sms) {
    const int per = ctas_per_sm > 0 && ctas_per_sm < kPairBlocks ? ctas_per_sm : kPairBlocks;
    const long long pairs = (n_tiles + 1) / 2, most = (long long)per * num_sms;
    return pairs < most ? (pairs < 1 ? 1 : pairs) : most;
}

// Whether the launch gives every pair its own warp, so that the work counter
// is not used (and need not be reset: one node less where latency counts).
bool pair_one_wave(long long n_tiles, int ctas_per_sm, int num_sms) {
    return (n_tiles + 1) / 2 <= 4 * pair_grid(n_tiles, ctas_per_sm, num_sms);
}

// Resolves a variant's attributes (before a stream capture, say).
cudaError_t pair_prepare(bool warm, bool batch) {
    const size_t smem = batch ? pair_smem_bytes<true>() : pair_smem_bytes<false>();
    cudaError_t e = cudaSuccess;
    for (int late = warm || batch ? 1 : 0; late <= 1 && e == cudaSuccess; ++late)
        e = cudaFuncSetAttribute(pair_variant(warm, batch, late != 0),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return e;
}

cudaError_t launch_pair(const SolveArgs& args, int ctas_per_sm, int num_sms, cudaStream_t stream) {
    const bool warm = args.u0 != nullptr, batch = args.stacks != nullptr;
    const long long grid = pair_grid(args.n_tiles, ctas_per_sm, num_sms);
    const PairFn fn = pair_variant(warm, batch, (args.n_tiles + 1) / 2 < kAheadWaves * 4 * grid);
    const size_t smem = batch ? pair_smem_bytes<true>() : pair_smem_bytes<false>();
    const cudaError_t e =
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    fn<<<(unsigned)grid, kWarpCtaThreads, smem, stream>>>(
        args, pair_one_wave(args.n_tiles, ctas_per_sm, num_sms) ? 1 : 0);
    return cudaGetLastError();
}

}  // namespace ncsb
