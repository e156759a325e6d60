// sd_poisson.cu -- periodic Poisson solve rho -> phi, all passes hand-written
// (the reference calls cuFFT R2C, kPoissonPeriodic, cuFFT C2R: Sim.cu:3586-3603,
// 528-557).
//
// Spectrum layout: one buffer of 4x4x4 complex "bricks" (512 B each). The kx
// axis holds the H+1 = G/2+1 bins of the real transform padded to H+4 (the last
// brick carries the Nyquist bin and three zero columns). Brick (bx,by,bz) starts
// at (((bz*NBY + by)*NBX + bx) * 64); inside a brick element (kx_l, y_l, z_l)
// sits at z_l*16 + y_l*4 + kx_l.
//
// Passes (CTA = one 4x4 bundle of 16 lines, held interleaved in shared memory):
//   A  x-rows real -> complex (input: float grid or int64 fixed-point grid)
//   B  y-lines forward            (in place)
//   C  z-lines forward, Green's function, z-lines inverse (in place)
//   D  y-lines inverse            (in place)
//   E  x-rows complex -> real, write phi
// Every global access moves whole 512-byte bricks or whole rows, B/C/D stage
// their bricks with cp.async, and each pass reads and writes every element once.
#include <cuda.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <mutex>
#include <vector>

#include "sd_common.cuh"
#include "sd_fft.cuh"
#include "sd_internal.h"

namespace sd {

namespace {

constexpr int kFftThreads = 256;
constexpr int kDepositThreads = 512;

template <int G>
struct Geo {
    static constexpr int H = G / 2;
    static constexpr int NBX = H / 4 + 1;  // kx bricks (last: Nyquist + padding)
    static constexpr int PX = 4 * NBX;     // padded kx positions = H + 4
    static constexpr int NBY = G / 4;
    static constexpr int NBZ = G / 4;
    __device__ __forceinline__ static size_t brick(int bx, int by, int bz) {
        return ((((size_t)bz * NBY + by) * NBX) + bx) * 64;
    }
};

// ---- pass A's x transform at G = 512: one warp per line ---------------------------
// A row of 512 reals is packed as 256 complex z[m] = x[2m] + i x[2m+1]; lane t
// holds z[t + 32k], k = 0..7. The 256-point transform is factored 8 x 32
// (m = t + 32k, f = f1 + 8 f2): a radix-8 DFT over k in registers and the twiddle
// W256^(t f1); then the 32-point DFTs over t, factored 8 x 4 (t = j + 4i,
// f2 = g1 + 8 g2) after a transpose through the warp's own shared scratch: lane
// (f1, j) takes a radix-8 DFT over i and the twiddle W32^(j g1); a second
// transpose hands lane L the output groups gA = L and gB = 64 - L (lane 0: 0 and
// 32), each finished by a radix-4 DFT over j into Z[g + 64 g2]. Both members of
// every pair (k, H - k) of the real-to-complex unpacking then sit in one lane.
// The bins go to a brick-ordered staging buffer, from which the CTA stores whole
// 512-byte bricks (a warp storing its own line would touch 65 bricks per line).
// Only __syncwarp orders the scratch; XOR swizzles keep every 8-byte access of the
// scratch and the staging buffer at two wavefronts.
namespace xl {
constexpr int kTw2 = 3 * 32 + 3 * 4;   // float2 entries of the two twiddle tables
constexpr int kStage = 16 * 4 * 65;     // float2: 65 bricks of 16 lines x 4 bins

// Twiddle tables, lane-contiguous so every load is conflict-free: tw[p*32 + t] =
// W256^(t 2^p) and then tw[96 + p*4 + j] = W32^(j 2^p), p = 0..2, copied from the
// table tw_g[m] = W512^m. Other powers are products of at most two of these.
__device__ __forceinline__ void fill_twiddles(float2* tw2, const float2* __restrict__ tw_g) {
    for (int e = threadIdx.x; e < kTw2; e += blockDim.x)
        tw2[e] = e < 96 ? tw_g[(2 * (e & 31)) << (e >> 5)] : tw_g[(16 * ((e - 96) & 3)) << ((e - 96) >> 2)];
}

// v[q] *= w^q for q = 1..7, given w, w^2, w^4
__device__ __forceinline__ void twiddle8(float2 (&v)[8], float2 w1, float2 w2, float2 w4) {
    const float2 w3 = fft::cmul(w1, w2);
    v[1] = fft::cmul(v[1], w1);
    v[2] = fft::cmul(v[2], w2);
    v[3] = fft::cmul(v[3], w3);
    v[4] = fft::cmul(v[4], w4);
    v[5] = fft::cmul(v[5], fft::cmul(w1, w4));
    v[6] = fft::cmul(v[6], fft::cmul(w2, w4));
    v[7] = fft::cmul(v[7], fft::cmul(w3, w4));
}

// Staging position of bin kx of line l = z_l*4 + y_l: brick kx/4, element
// z_l*16 + y_l*4 + kx%4 (the spectrum's brick layout), bits 2-3 of the element
// XORed with the brick's low bits. 16-byte pairs (kx even, kx + 1) stay adjacent.
__device__ __forceinline__ int stage_pos(int kx, int l) {
    const int b = kx >> 2;
    return b * 64 + ((((l >> 2) << 4) + ((l & 3) << 2) + (kx & 3)) ^ ((b & 3) << 2));
}

// One pair of the unpacking: from Z[k] and Z[H-k], X[k] = E + W512^k O and
// X[H-k] = conj E + W512^(H-k) conj O with E = (Z[k] + conj Z[H-k]) / 2,
// O = (Z[k] - conj Z[H-k]) / (2i); W512^(H-k) = -conj W512^k.
__device__ __forceinline__ void unpack_pair(float2 zk, float2 zc, int k, const float2* tw, float2* st, int l) {
    constexpr int H = 256;
    const float er = 0.5f * (zk.x + zc.x), ei = 0.5f * (zk.y - zc.y);
    const float orr = 0.5f * (zk.y + zc.y), oi = -0.5f * (zk.x - zc.x);
    const float2 w = tw[k];
    st[stage_pos(k, l)] = make_float2(er + (w.x * orr - w.y * oi), ei + (w.x * oi + w.y * orr));
    if (2 * k != H)
        st[stage_pos(H - k, l)] = make_float2(er + (w.y * oi - w.x * orr), -ei + (w.y * orr + w.x * oi));
}

// z: this lane's inputs z[t + 32k] (destroyed); sc: the warp's 256-float2 scratch,
// free on entry and on return; tw: W512^m in shared memory; st: the staging
// buffer, which receives bins 0..259 of line l (257..259 zero).
__device__ __forceinline__ void r2c512(float2 (&z)[8], float2* sc, const float2* tw, const float2* tw2, float2* st,
                                       int l) {
    const int lane = threadIdx.x & 31;
    fft::dft<8, false>(z);
    twiddle8(z, tw2[lane], tw2[32 + lane], tw2[64 + lane]);  // W256^(t f1)
    __syncwarp();
#pragma unroll
    for (int f1 = 0; f1 < 8; ++f1) sc[f1 * 32 + (lane ^ (4 * (f1 & 3)))] = z[f1];
    __syncwarp();
    const int f1 = lane >> 2, j = lane & 3;
#pragma unroll
    for (int i = 0; i < 8; ++i) z[i] = sc[f1 * 32 + ((j + 4 * i) ^ (4 * (f1 & 3)))];
    fft::dft<8, false>(z);
    twiddle8(z, tw2[96 + j], tw2[100 + j], tw2[104 + j]);  // W32^(j g1)
    __syncwarp();
#pragma unroll
    for (int g1 = 0; g1 < 8; ++g1) {
        const int g = f1 + 8 * g1;
        sc[4 * g + (j ^ ((g >> 2) & 3))] = z[g1];
    }
    __syncwarp();
    const int ga = lane, gb = lane ? 64 - lane : 32;
    float2 a[4], b[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        a[q] = sc[4 * ga + (q ^ ((ga >> 2) & 3))];
        b[q] = sc[4 * gb + (q ^ ((gb >> 2) & 3))];
    }
    __syncwarp();  // the scratch is free again
    fft::dft<4, false>(a);  // a[g2] = Z[ga + 64 g2]
    fft::dft<4, false>(b);  // b[g2] = Z[gb + 64 g2]
    if (lane) {
        unpack_pair(a[0], b[3], lane, tw, st, l);
        unpack_pair(a[1], b[2], 64 + lane, tw, st, l);
        unpack_pair(b[1], a[2], 128 - lane, tw, st, l);
        unpack_pair(b[0], a[3], 64 - lane, tw, st, l);
    } else {
        st[stage_pos(0, l)] = make_float2(a[0].x + a[0].y, 0.f);
        st[stage_pos(256, l)] = make_float2(a[0].x - a[0].y, 0.f);
        st[stage_pos(257, l)] = make_float2(0.f, 0.f);
        st[stage_pos(258, l)] = make_float2(0.f, 0.f);
        st[stage_pos(259, l)] = make_float2(0.f, 0.f);
        unpack_pair(a[1], a[3], 64, tw, st, l);
        unpack_pair(a[2], a[2], 128, tw, st, l);
        unpack_pair(b[0], b[3], 32, tw, st, l);
        unpack_pair(b[1], b[2], 96, tw, st, l);
    }
}

// The staged bricks (kx/4 = 0..64) of bundle (by, bz) to the spectrum, 16 bytes
// per thread: each warp instruction writes one whole brick.
template <int G>
__device__ __forceinline__ void store_bricks(const float2* st, float2* __restrict__ spec, int by, int bz) {
    for (int u = threadIdx.x; u < 65 * 32; u += blockDim.x) {
        const int b = u >> 5, c = u & 31;
        const float4 v = *reinterpret_cast<const float4*>(st + b * 64 + ((2 * c) ^ ((b & 3) << 2)));
        *reinterpret_cast<float4*>(spec + Geo<G>::brick(b, by, bz) + 2 * c) = v;
    }
}
}  // namespace xl

// ---- pass A: rows (y = 4by + y_l, z = 4bz + z_l) -> kx bins -----------------
// line l = z_l*4 + y_l; positions m < H hold z[m] = x[2m] + i x[2m+1].
// SRC 0: float grid, 1: int64 fixed-point grid (zeroed after reading). The source
// grid has side src_g <= G: a smaller one (the isolated boundary's density) sits in
// the low corner of the transform box and everything outside it reads as zero.
// At G = 512 a CTA of 512 threads takes a line per warp, its loads issued before the
// twiddle tables are there, and 40 registers keep 48 warps on an SM: with 256 threads and
// two lines a warp, one after the other, 24 warps waited on memory and on each other. A
// sparse int64 grid (2,097,152 particles) 0.556 -> 0.483 ms, 4.97 TB/s.
template <int G>
constexpr int kPassAThreads = G == 512 ? 512 : kFftThreads;

template <int G, int SRC>
__global__ void __launch_bounds__(kPassAThreads<G>, G == 512 ? 3 : 0)
    k_pass_a(const float* __restrict__ rho, long long* __restrict__ acc, float* __restrict__ rho_keep,
             float2* __restrict__ spec, const float2* __restrict__ tw_g, int src_g) {
    wait_previous();
    using T = Geo<G>;
    constexpr int H = T::H, NBX = T::NBX;
    constexpr int ITEMS = 16 * (H / 2);  // (line, pair of positions)
    constexpr int PER = (ITEMS + kFftThreads - 1) / kFftThreads;
    extern __shared__ float2 sm[];
    float2* tw = sm;
    float2* s = sm + G;
    const int by = blockIdx.x, bz = blockIdx.y;
    if constexpr (G == 512) {
        // the fused deposit's transform; shared: tw | twiddle tables | 16 warp scratches | brick staging
        static_assert(kPassAThreads<G> == 16 * 32, "one warp per line");
        float2* tw2 = sm + G;
        const int l = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int y = by * 4 + (l & 3), z = bz * 4 + (l >> 2);
        const size_t row = ((size_t)z * src_g + y) * src_g;
        const bool in_rows = y < src_g && z < src_g;
        // every load of the row is issued before any store: a store that follows the load
        // of the same address in the loop body kept the next load waiting behind it, one
        // memory round trip per 512 bytes (2.46 ms at 512^3)
        float2 v[8];
        longlong2 q[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = lane + 32 * k;
            v[k] = make_float2(0.f, 0.f);
            q[k] = make_longlong2(0, 0);
            if (in_rows && 2 * m < src_g) {
                if (SRC == 0)
                    v[k] = *reinterpret_cast<const float2*>(rho + row + 2 * m);
                else
                    q[k] = *reinterpret_cast<const longlong2*>(acc + row + 2 * m);
            }
        }
        for (int i = threadIdx.x; i < G; i += kPassAThreads<G>) tw[i] = tw_g[i];
        xl::fill_twiddles(tw2, tw_g);
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = lane + 32 * k;
            if (in_rows && 2 * m < src_g) {
                if (SRC == 1) {
                    // cells that hold something are cleared; a sparse grid saves most of the writes
                    v[k] = make_float2(fixed_to_float(q[k].x), fixed_to_float(q[k].y));
                    if (v[k].x != 0.f || v[k].y != 0.f)
                        *reinterpret_cast<longlong2*>(acc + row + 2 * m) = make_longlong2(0, 0);
                }
                if (rho_keep) *reinterpret_cast<float2*>(rho_keep + row + 2 * m) = v[k];
            }
        }
        __syncthreads();
        float2* st = tw2 + xl::kTw2 + 16 * 256;
        xl::r2c512(v, tw2 + xl::kTw2 + l * 256, tw, tw2, st, l);
        __syncthreads();
        xl::store_bricks<G>(st, spec, by, bz);
        return;
    }
    for (int i = threadIdx.x; i < G; i += kFftThreads) tw[i] = tw_g[i];

    float4 v[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * kFftThreads;
        if (ITEMS % kFftThreads == 0 || u < ITEMS) {
            const int l = u & 15, mp = u >> 4;
            const int y = by * 4 + (l & 3), z = bz * 4 + (l >> 2);
            const size_t row = ((size_t)z * src_g + y) * src_g;
            v[p] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (y < src_g && z < src_g && 4 * mp < src_g) {
                if (SRC == 0) {
                    v[p] = *reinterpret_cast<const float4*>(rho + row + 4 * mp);
                } else {
                    const longlong2 q0 = *reinterpret_cast<const longlong2*>(acc + row + 4 * mp);
                    const longlong2 q1 = *reinterpret_cast<const longlong2*>(acc + row + 4 * mp + 2);
                    v[p] = make_float4(fixed_to_float(q0.x), fixed_to_float(q0.y), fixed_to_float(q1.x),
                                       fixed_to_float(q1.y));
                }
            }
        }
    }
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * kFftThreads;
        if (ITEMS % kFftThreads == 0 || u < ITEMS) {
            const int l = u & 15, mp = u >> 4;
            const int y = by * 4 + (l & 3), z = bz * 4 + (l >> 2);
            const size_t row = ((size_t)z * src_g + y) * src_g;
            if (y < src_g && z < src_g && 4 * mp < src_g) {
                if (SRC == 1) {  // a cell that rounds to 0 as a float is 0: its unit is 2^-32
                    if (v[p].x != 0.f || v[p].y != 0.f)
                        *reinterpret_cast<longlong2*>(acc + row + 4 * mp) = make_longlong2(0, 0);
                    if (v[p].z != 0.f || v[p].w != 0.f)
                        *reinterpret_cast<longlong2*>(acc + row + 4 * mp + 2) = make_longlong2(0, 0);
                }
                if (rho_keep) *reinterpret_cast<float4*>(rho_keep + row + 4 * mp) = v[p];
            }
            s[(2 * mp) * 16 + l] = make_float2(v[p].x, v[p].y);
            s[(2 * mp + 1) * 16 + l] = make_float2(v[p].z, v[p].w);
        }
    }
    __syncthreads();
    fft::lines16<H, kFftThreads, 2, false>(s, tw);
    // Z -> X, pairs (k, H-k):  E = (Z[k] + conj Z[H-k])/2,  O = (Z[k] - conj Z[H-k])/(2i),
    // X[k] = E + W^k O,  X[H-k] = conj E + W^(H-k) conj O;  X[0], X[H] from Z[0].
    constexpr int PAIRS = 16 * (H / 2 + 1);
    for (int u = threadIdx.x; u < PAIRS; u += kFftThreads) {
        const int l = u & 15, k = u >> 4;
        if (k == 0) {
            const float2 z0 = s[l];
            s[l] = make_float2(z0.x + z0.y, 0.f);
            s[H * 16 + l] = make_float2(z0.x - z0.y, 0.f);
            s[(H + 1) * 16 + l] = make_float2(0.f, 0.f);
            s[(H + 2) * 16 + l] = make_float2(0.f, 0.f);
            s[(H + 3) * 16 + l] = make_float2(0.f, 0.f);
            continue;
        }
        const float2 zk = s[k * 16 + l], zc = s[(H - k) * 16 + l];
        const float er = 0.5f * (zk.x + zc.x), ei = 0.5f * (zk.y - zc.y);
        const float orr = 0.5f * (zk.y + zc.y), oi = -0.5f * (zk.x - zc.x);
        const float2 w = tw[k];
        s[k * 16 + l] = make_float2(er + (w.x * orr - w.y * oi), ei + (w.x * oi + w.y * orr));
        if (2 * k != H) {
            const float2 w2 = tw[H - k];  // conj E + W^(H-k) conj O
            s[(H - k) * 16 + l] = make_float2(er + (w2.x * orr + w2.y * oi), -ei + (w2.y * orr - w2.x * oi));
        }
    }
    __syncthreads();
    // store bricks (bx, by, bz): brick element e = z_l*16 + y_l*4 + kx_l, two at a time
    for (int u = threadIdx.x; u < NBX * 32; u += kFftThreads) {
        const int bx = u >> 5, c = u & 31;
        const int l = (c >> 3) * 4 + ((c >> 1) & 3), kx = bx * 4 + (c & 1) * 2;
        const float2 a = s[kx * 16 + l], b = s[(kx + 1) * 16 + l];
        *reinterpret_cast<float4*>(spec + T::brick(bx, by, bz) + 2 * c) = make_float4(a.x, a.y, b.x, b.y);
    }
}

// ---- balanced fused deposit ---------------------------------------------------------
// Scratch (DepositWork::ints) of a grid with NB = G^2/16 row bundles, NC = ceil(NB/256):
//   items[NB]    CTAs sharing each bundle (>= 1)
//   xpre[NB]     exclusive prefix of (items - 1) inside each block of 256 bundles
//   arrive[NB]   CTAs of a shared bundle done so far (zero between uses)
//   cta_sum[NC], cta_pre[NC + 1]   per-block totals and their exclusive prefix
//   plan_done    blocks of the plan kernel done (zero between uses)
//   ticket       next work item of the deposit's CTAs, past their first ones
//   use          nonzero: this use deposits from the fixed-point grid (see stray)
//   stray        nonzero: a particle that the bundles' sums would miss (stray_particle; set where
//                keys are made, launch_cell_keys; cleared by the next plan)
template <int G>
struct DepPlan {
    static constexpr int NB = G * G / 16;
    static constexpr int NC = (NB + 255) / 256;
    static constexpr int kItems = 0, kXpre = NB, kArrive = 2 * NB, kCtaSum = 3 * NB, kCtaPre = 3 * NB + NC,
                         kDone = 3 * NB + 2 * NC + 1, kTicket = kDone + 1, kUse = kTicket + 1, kStray = kUse + 1,
                         kInts = kStray + 1;
};

// Where the particles of a bundle's window sit among the sorted ones, as kRanges
// ranges. G is the side of the particles' grid, rs its row table.
//
// Tiled order: the 25 base rows whose CIC stencils reach the 16 rows of bundle
// b = bz*(G/4)+by, as 7 ranges: r = 0 the bundle's own rows (16 consecutive keys);
// r = 1 the rows z_l = 3 of the bundle below in z (4 consecutive keys); r = 2..5 the
// rows y_l = 3, z_l = r - 2 of the bundle below in y; r = 6 the row y_l = z_l = 3 of
// the bundle below in both. Neighbours wrap: in a periodic box the stencils do, in an
// isolated one a base row -1 is stored as row G - 1 (and one that does not reach this
// bundle adds nothing to it).
//
// Row-major order (WIDE): a particle's cell is its base cell or the one above, so the
// window is the 6 x 6 rows of cells around the bundle: for each plane z = 4 bz - 1 ..
// 4 bz + 4 the rows y = 4 by - 1 .. 4 by + 4, one range, and a second one for the row
// that wraps. 36 rows read for 16 against 25, still less than a pass of 64-bit atomics
// over the grid and another to read and clear it (8,000,003 particles on 256^3: 238 us,
// now 190 with the plan; 2,000,000 on 128^3: 78 and 73; 1,000,003 of a galaxy on an
// isolated 128^3: 106 and 78).
template <bool WIDE>
constexpr int kRanges = WIDE ? 12 : 7;

template <int G, bool WIDE, bool ISO>
__device__ __forceinline__ void window_range(int b, int r, const int* __restrict__ rs, int& lo, int& hi) {
    constexpr int TB = G / 4;
    const int by = b & (TB - 1), bz = b / TB;
    int k0, k1;
    if (WIDE) {
        int z = 4 * bz - 1 + (r >> 1);
        const int y0 = 4 * by - 1, y1 = 4 * by + 4;
        int ya = max(y0, 0), yb = min(y1, G - 1);
        bool none = ISO && (unsigned)z >= (unsigned)G;
        if (r & 1) {
            none = none || ISO || (y0 >= 0 && y1 < G);
            ya = yb = (y0 < 0) ? G - 1 : 0;
        }
        z &= G - 1;
        k0 = none ? 0 : z * G + ya;
        k1 = none ? 0 : z * G + yb + 1;
    } else {
        const int bym = (by + TB - 1) & (TB - 1), bzm = (bz + TB - 1) & (TB - 1);
        if (r == 0) {
            k0 = 16 * b;
            k1 = k0 + 16;
        } else if (r == 1) {
            k0 = 16 * (bzm * TB + by) + 12;
            k1 = k0 + 4;
        } else if (r == 6) {
            k0 = 16 * (bzm * TB + bym) + 15;
            k1 = k0 + 1;
        } else {
            k0 = 16 * (bz * TB + bym) + 4 * (r - 2) + 3;
            k1 = k0 + 1;
        }
    }
    lo = rs[k0];
    hi = rs[k1];
}

// Exclusive scan of one int per thread over a block of 256 threads; *total gets the sum.
__device__ __forceinline__ int block_excl_scan256(int v, int* total) {
    __shared__ int wsum[8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) wsum[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        int x = lane < 8 ? wsum[lane] : 0;
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += t;
        }
        if (lane < 8) wsum[lane] = x;
    }
    __syncthreads();
    const int excl = inc - v + (warp ? wsum[warp - 1] : 0);
    *total = wsum[7];
    __syncthreads();  // wsum may be reused by the next call
    return excl;
}

// How many CTAs share each bundle: ceil(window particles / piece) above split, else 1,
// and where each bundle's extra CTAs start. The last block to finish turns the
// block totals into their prefix.
//
// Positions outside the box are accepted. The periodic stencil wraps them and the
// isolated one clamps them, but the row that the row-major key (clamped) or the tiled
// key (wrapped) puts them in is then not the stencil's, so no window finds them. Where
// keys were made from such a position the stray flag is set, and this kernel deposits
// every particle into the fixed-point grid itself, which the bundles read instead of
// particles. Steps leave positions inside the box, so this is at most the first step
// after a load; its speed does not matter, its not costing the others a launch does. A
// position that is no number sets the flag too: its weights are, to the 64-bit sums, one
// large value, and a step takes it as lost.
template <bool WIDE, bool ISO>
constexpr bool kMayStray = WIDE || ISO;
template <int G, bool WIDE, bool ISO>
__global__ void __launch_bounds__(256) k_deposit_plan(const int* __restrict__ rs, int* __restrict__ w, int split,
                                                      int piece, const float4* __restrict__ pos, int n,
                                                      unsigned long long* __restrict__ acc) {
    wait_previous();
    using P = DepPlan<G>;
    const int b = blockIdx.x * 256 + threadIdx.x;
    int extra = 0;
    const int stray = kMayStray<WIDE, ISO> ? w[P::kStray] : 0;
    if (kMayStray<WIDE, ISO> && stray) {
        split = 0x7fffffff;  // no shared bundles
        for (long long i = b; i < n; i += (long long)gridDim.x * 256) deposit_particle(pos[i], G, acc, !ISO);
    }
    if (b < P::NB) {
        int total = 0;
#pragma unroll
        for (int r = 0; r < kRanges<WIDE>; ++r) {
            int lo, hi;
            window_range<G, WIDE, ISO>(b, r, rs, lo, hi);
            total += hi - lo;
        }
        const int items = total > split ? (int)(((long long)total + piece - 1) / piece) : 1;
        w[P::kItems + b] = items;
        extra = items - 1;
    }
    int sum;
    const int excl = block_excl_scan256(extra, &sum);
    if (b < P::NB) w[P::kXpre + b] = excl;
    if constexpr (P::NC == 1) {
        // up to 64^3 one block has it all: 2.4 us, 4.2 with the exchange below
        if (threadIdx.x == 0) {
            w[P::kCtaPre] = 0;
            w[P::kCtaPre + 1] = sum;
            w[P::kTicket] = 0;
            if (kMayStray<WIDE, ISO>) {  // every thread has read the flag
                w[P::kUse] = stray;
                w[P::kStray] = 0;
            }
        }
        return;
    }
    if (threadIdx.x == 0) w[P::kCtaSum + blockIdx.x] = sum;
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(reinterpret_cast<unsigned*>(w + P::kDone), 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    // NC <= 256 blocks (G <= 1024)
    const int v = threadIdx.x < P::NC ? __ldcg(w + P::kCtaSum + threadIdx.x) : 0;
    int all;
    const int pre = block_excl_scan256(v, &all);
    if (threadIdx.x < P::NC) w[P::kCtaPre + threadIdx.x] = pre;
    if (threadIdx.x == 0) {
        w[P::kCtaPre + P::NC] = all;
        w[P::kDone] = 0;
        w[P::kTicket] = 0;
        if (kMayStray<WIDE, ISO>) {  // every block has read the flag
            w[P::kUse] = stray;
            w[P::kStray] = 0;
        }
    }
}

// One CTA's share (slice `slice` of `items`) of bundle b: deposit its particles
// into int64 row sums in shared memory; if the bundle is shared, add the sums into
// the fixed-point grid and let the last CTA continue with the whole bundle; then
// convert, transform the 16 rows along x and store the spectrum bricks.
// ISO: the particles' grid has half the box's side and corners past its edge are
// clamped onto the edge cells (no weight is lost); the upper half of each line is zero.
// (Summing equal corners across a warp's lanes first, with __match_any_sync and
// __reduce_add_sync, made dense scenes slower, not faster: 0.27 against 0.18 ms
// at 4M particles / 256^3.)
template <int G, bool ISO>
struct DepGeo {
    static constexpr int M = ISO ? G / 2 : G;  // side of the particles' grid
    static constexpr int RS = M + 4;           // words between the rows of the sums
    // float2 of the storage that the sums, the line buffer and (512) the warps' scratch share
    static constexpr int kLines = 16 * Geo<G>::PX, kSums = 16 * RS, kWarp = 16 * 256 + xl::kStage;
    static constexpr int kStore = G == 512 ? (kWarp > kSums ? kWarp : kSums) : (kLines > kSums ? kLines : kSums);
};

template <int G>
constexpr bool kDepositLoop = G == 512;
constexpr int kIsoShare = (1 << 14) - 1;  // most particles of an isolated share (deposit_bundle)
template <int G>
constexpr int kDepositPerSm = G >= 128 ? 3 : 2;

template <int G, bool ISO, bool WIDE, bool SHARED>
__device__ __forceinline__ void deposit_bundle(int b, int slice, int items, const float4* __restrict__ pos,
                                               const int* __restrict__ perm, const int* __restrict__ row_start,
                                               float* __restrict__ rho_keep, float2* __restrict__ spec,
                                               const DepositWork& w, unsigned* __restrict__ arrive,
                                               int* __restrict__ ticket, int* s_next, bool reuse, bool from_grid) {
    using T = Geo<G>;
    using D = DepGeo<G, ISO>;
    constexpr int M = D::M, NR = kRanges<WIDE>;
    constexpr int H = T::H, NBX = T::NBX, NT = kDepositThreads, TB = M / 4;
    // The int64 fixed-point sums, as two 32-bit words per cell (lo[16][RS], hi[16][RS]),
    // share their storage with the complex line buffer used after the conversion.
    // Rows are RS = M + 4 words apart, so the row-parallel 16-byte reads of the
    // conversion fall in different banks.
    constexpr int RS = D::RS;
    extern __shared__ float2 sm[];
    const float2* tw = sm;
    unsigned* acc_lo = reinterpret_cast<unsigned*>(sm + G);
    unsigned* acc_hi = acc_lo + 16 * RS;
    float2* s = sm + G;
    __shared__ int r_lo[16], r_off[17];
    __shared__ int s_last;
    const int by = b & (TB - 1), bz = b / TB;
    const int m = M - 1;
    const int j = threadIdx.x;
    int lo = 0, len = 0;
    if (j < NR) {
        int hi;
        window_range<M, WIDE, ISO>(b, j, row_start, lo, hi);
        len = hi - lo;
    }
    if (reuse) __syncthreads();  // the shared buffers of this CTA's previous bundle are free
    for (int i = threadIdx.x; i < 8 * RS; i += NT) reinterpret_cast<uint4*>(acc_lo)[i] = make_uint4(0u, 0u, 0u, 0u);
    if (threadIdx.x < 32) {
        int inc = len;
#pragma unroll
        for (int o = 1; o < (WIDE ? 16 : 8); o <<= 1) {
            const int t = __shfl_up_sync(0xffffffffu, inc, o);
            if (j >= o) inc += t;
        }
        if (j < NR) {
            r_lo[j] = lo;
            r_off[j + 1] = inc;
        }
        if (j == 0) r_off[0] = 0;
    }
    __syncthreads();
    // the CTA's next work item, read after later barriers
    if (kDepositLoop<G> && threadIdx.x == 0) *s_next = atomicAdd(ticket, 1) + (int)gridDim.x;
    const int total = from_grid ? 0 : r_off[NR];  // from_grid: the sums are in the fixed-point grid
    const int f_lo = SHARED ? (int)((long long)total * slice / items) : 0;
    const int f_hi = SHARED ? (int)((long long)total * (slice + 1) / items) : total;
    // A weight q <= 2^32 is added as (q >> kSplit) into the high word and the bits below into
    // the low word: with fewer than 2^kSplit particles in this share neither 32-bit sum can
    // overflow, so plain adds keep the 64-bit total exact. Larger shares add the low 32 bits
    // and carry into the high word instead. Periodic corners are eight cells, so a particle
    // adds to a cell once and the sums stay at or below 2^16 (2^16 - 1). Clamped corners
    // coincide, up to eight in one cell and 2^32 together: the low sums stay at or below
    // 8 (2^14 - 1)^2 < 2^31, the high ones at or below 2^18 (2^14 - 1), and windows are split so
    // that no isolated share is larger (a step of 1,000,000 on 16^3 345 us
    // with the carry, 127 without).
    constexpr int kSplit = ISO ? 14 : 16;
    static_assert(!ISO || kIsoShare < (1 << kSplit), "an isolated share never carries");
    const bool split = ISO || f_hi - f_lo < (1 << kSplit);
    const int lane = threadIdx.x & 31;
    constexpr int kBatch = 4;
    // lane f = base + q * NT + lane
    for (int base = f_lo + (threadIdx.x & ~31); base < f_hi; base += kBatch * NT) {
        int src[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            const int f = base + q * NT + lane;
            src[q] = -1;
            if (f < f_hi) {
                // largest r < NR with r_off[r] <= f
                int r = (WIDE && r_off[8] <= f) ? 8 : 0;
                if (r + 4 < NR && r_off[r + 4] <= f) r += 4;
                if (r + 2 < NR && r_off[r + 2] <= f) r += 2;
                if (r + 1 < NR && r_off[r + 1] <= f) r += 1;
                src[q] = r_lo[r] + (f - r_off[r]);
            }
        }
        if (perm) {
#pragma unroll
            for (int q = 0; q < kBatch; ++q)
                if (src[q] >= 0) src[q] = perm[src[q]];
        }
        float4 pb[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) pb[q] = (src[q] >= 0) ? pos[src[q]] : make_float4(-1.f, -1.f, -1.f, 0.f);
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            if (base + q * NT >= f_hi) break;
            const float4 p = pb[q];
            const bool valid = p.x >= 0.f;  // empty slots sort into row 0
            int ix, iy, iz;
            float fx, fy, fz;
            cic_axis(p.x, M, ix, fx);
            cic_axis(p.y, M, iy, fy);
            cic_axis(p.z, M, iz, fz);
            if (!valid) continue;
            // the weights of cic_weight, scaled by 2^32 with their z factor (exact)
            const float wx[2] = {__fsub_rn(1.f, fx), fx}, wy[2] = {__fsub_rn(1.f, fy), fy};
            const float wz[2] = {__fmul_rn(__fsub_rn(1.f, fz), SD_FIXED_ONE), __fmul_rn(fz, SD_FIXED_ONE)};
            const int x0 = cic_cell(ix, M, !ISO), x1 = cic_corner(ix, 1, M, !ISO);
            // the bundle's rows that the stencil reaches: yl + (0, 1), zl + (0, 1), each in
            // [0, 4) or not this bundle's. In the periodic box they lie at fixed distances
            // from the first one's address, whether that is in the bundle or not.
            int yl[2], zl[2];
            if (ISO) {
#pragma unroll
                for (int o = 0; o < 2; ++o) {
                    yl[o] = cic_corner(iy, o, M, false) - 4 * by;
                    zl[o] = cic_corner(iz, o, M, false) - 4 * bz;
                }
            } else {
                yl[1] = (iy + 1 - 4 * by) & m;
                zl[1] = (iz + 1 - 4 * bz) & m;
                yl[0] = yl[1] - 1;
                zl[0] = zl[1] - 1;
            }
            const int first = (zl[0] * 4 + yl[0]) * RS;
#pragma unroll
            for (int oyz = 0; oyz < 4; ++oyz) {
                const int oy = oyz & 1, oz = oyz >> 1;
                if ((unsigned)yl[oy] >= 4u || (unsigned)zl[oz] >= 4u) continue;
                const int row = ISO ? (zl[oz] * 4 + yl[oy]) * RS : first + (oz * 4 + oy) * RS;
#pragma unroll
                for (int ox = 0; ox < 2; ++ox) {
                    const unsigned long long qv =
                        (unsigned long long)__float2ll_rn(__fmul_rn(__fmul_rn(wx[ox], wy[oy]), wz[oz]));
                    const int c = row + (ox ? x1 : x0);
                    if (split) {
                        atomicAdd(acc_hi + c, (unsigned)(qv >> kSplit));
                        atomicAdd(acc_lo + c, (unsigned)qv & ((1u << kSplit) - 1u));
                    } else {
                        // atomicAdd returns the previous low word, so every wrap is seen by
                        // exactly one add
                        const unsigned lw = (unsigned)qv;
                        const unsigned old = atomicAdd(acc_lo + c, lw);
                        const unsigned up = (unsigned)(qv >> 32) + ((old + lw < old) ? 1u : 0u);
                        if (up) atomicAdd(acc_hi + c, up);
                    }
                }
            }
        }
    }
    __syncthreads();
    int sh = split ? kSplit : 32;  // value of a cell: (hi << sh) + lo
    if (SHARED && (items > 1 || from_grid)) {
        // a shared bundle: every CTA adds its rows into the fixed-point grid; the last
        // to arrive reads the complete sums back (and leaves the grid zero)
        unsigned long long* g = reinterpret_cast<unsigned long long*>(w.acc);
        if (!from_grid) {
#pragma unroll 1
            for (int u = threadIdx.x; u < 16 * M; u += NT) {
                const int l = u / M, x = u & m;
                const unsigned long long v =
                    ((unsigned long long)acc_hi[l * RS + x] << sh) + (unsigned long long)acc_lo[l * RS + x];
                if (v) atomicAdd(g + ((size_t)(4 * bz + (l >> 2)) * M + 4 * by + (l & 3)) * M + x, v);
            }
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) s_last = atomicAdd(arrive + b, 1u) == (unsigned)(items - 1);
            __syncthreads();
            if (!s_last) return;
            __threadfence();
        }
        // all of this thread's loads first, then the shared-memory writes and the zeroing
        // stores (a store behind each load of the same address would serialise them)
        constexpr int RB = 4;  // loads in flight per thread (more spill at the 40-register bound)
#pragma unroll 1
        for (int u0 = threadIdx.x; u0 < 16 * M; u0 += RB * NT) {
            unsigned long long rb[RB];
#pragma unroll
            for (int q = 0; q < RB; ++q) {
                const int u = u0 + q * NT, l = u / M, x = u & m;
                if (u < 16 * M) rb[q] = __ldcg(g + ((size_t)(4 * bz + (l >> 2)) * M + 4 * by + (l & 3)) * M + x);
            }
#pragma unroll
            for (int q = 0; q < RB; ++q) {
                const int u = u0 + q * NT, l = u / M, x = u & m;
                if (u < 16 * M) {
                    acc_lo[l * RS + x] = (unsigned)rb[q];
                    acc_hi[l * RS + x] = (unsigned)(rb[q] >> 32);
                    g[((size_t)(4 * bz + (l >> 2)) * M + 4 * by + (l & 3)) * M + x] = 0ull;
                }
            }
        }
        sh = 32;
        if (threadIdx.x == 0) arrive[b] = 0u;
        __syncthreads();
    }
    if constexpr (G == 512) {
        // warp l converts row l and transforms it (the generic pass A's routine, so
        // both deposit paths give the same bits); its lo row is then its scratch
        static_assert(NT == 16 * 32, "one warp per line");
        const int l = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const unsigned* lo = acc_lo + l * RS;
        const unsigned* hi = acc_hi + l * RS;
        const size_t grow = ((size_t)(bz * 4 + (l >> 2)) * M + by * 4 + (l & 3)) * M;
        float2 v[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const int m = lane + 32 * k;
            if (ISO && k >= 4) {
                v[k] = make_float2(0.f, 0.f);
                continue;
            }
            const uint2 lw = *reinterpret_cast<const uint2*>(lo + 2 * m);
            const uint2 hw = *reinterpret_cast<const uint2*>(hi + 2 * m);
            v[k] = make_float2(fixed_to_float((long long)(((unsigned long long)hw.x << sh) + lw.x)),
                               fixed_to_float((long long)(((unsigned long long)hw.y << sh) + lw.y)));
            if (rho_keep) *reinterpret_cast<float2*>(rho_keep + grow + 2 * m) = v[k];
        }
        // every row is in registers: the sums' storage becomes 16 warp scratches
        // (256 float2 each) and the brick staging
        __syncthreads();
        float2* R = reinterpret_cast<float2*>(acc_lo);
        xl::r2c512(v, R + l * 256, tw, sm + G + D::kStore, R + 16 * 256, l);
        __syncthreads();
        xl::store_bricks<G>(R + 16 * 256, spec, by, bz);
        return;
    }
    // int64 rows -> complex positions z[m] = x[2m] + i x[2m+1] on line l = z_l*4 + y_l,
    // staged through registers because the line buffer overlays the sums.
    constexpr int CITEMS = 16 * (M / 4);
    constexpr int CPER = (CITEMS + NT - 1) / NT;
    float4 cv[CPER];
#pragma unroll
    for (int p = 0; p < CPER; ++p) {
        const int u = threadIdx.x + p * NT;
        if (CITEMS % NT == 0 || u < CITEMS) {
            const int l = u & 15, mp = u >> 4;
            const uint4 lw = *reinterpret_cast<const uint4*>(acc_lo + l * RS + 4 * mp);
            const uint4 hw = *reinterpret_cast<const uint4*>(acc_hi + l * RS + 4 * mp);
            cv[p] = make_float4(fixed_to_float((long long)(((unsigned long long)hw.x << sh) + lw.x)),
                                fixed_to_float((long long)(((unsigned long long)hw.y << sh) + lw.y)),
                                fixed_to_float((long long)(((unsigned long long)hw.z << sh) + lw.z)),
                                fixed_to_float((long long)(((unsigned long long)hw.w << sh) + lw.w)));
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < CPER; ++p) {
        const int u = threadIdx.x + p * NT;
        if (CITEMS % NT == 0 || u < CITEMS) {
            const int l = u & 15, mp = u >> 4;
            if (rho_keep) {
                const size_t grow = ((size_t)(bz * 4 + (l >> 2)) * M + by * 4 + (l & 3)) * M;
                *reinterpret_cast<float4*>(rho_keep + grow + 4 * mp) = cv[p];
            }
            s[(2 * mp) * 16 + l] = make_float2(cv[p].x, cv[p].y);
            s[(2 * mp + 1) * 16 + l] = make_float2(cv[p].z, cv[p].w);
        }
    }
    __syncthreads();
    fft::lines16<H, NT, 2, false, ISO>(s, tw);
    constexpr int PAIRS = 16 * (H / 2 + 1);
    for (int u = threadIdx.x; u < PAIRS; u += NT) {
        const int l = u & 15, k = u >> 4;
        if (k == 0) {
            const float2 z0 = s[l];
            s[l] = make_float2(z0.x + z0.y, 0.f);
            s[H * 16 + l] = make_float2(z0.x - z0.y, 0.f);
            s[(H + 1) * 16 + l] = make_float2(0.f, 0.f);
            s[(H + 2) * 16 + l] = make_float2(0.f, 0.f);
            s[(H + 3) * 16 + l] = make_float2(0.f, 0.f);
            continue;
        }
        const float2 zk = s[k * 16 + l], zc = s[(H - k) * 16 + l];
        const float er = 0.5f * (zk.x + zc.x), ei = 0.5f * (zk.y - zc.y);
        const float orr = 0.5f * (zk.y + zc.y), oi = -0.5f * (zk.x - zc.x);
        const float2 wk = tw[k];
        s[k * 16 + l] = make_float2(er + (wk.x * orr - wk.y * oi), ei + (wk.x * oi + wk.y * orr));
        if (2 * k != H) {
            const float2 w2 = tw[H - k];
            s[(H - k) * 16 + l] = make_float2(er + (w2.x * orr + w2.y * oi), -ei + (w2.y * orr - w2.x * oi));
        }
    }
    __syncthreads();
    for (int u = threadIdx.x; u < NBX * 32; u += NT) {
        const int bx = u >> 5, c = u & 31;
        const int l = (c >> 3) * 4 + ((c >> 1) & 3), kx = bx * 4 + (c & 1) * 2;
        const float2 a = s[kx * 16 + l], c2 = s[(kx + 1) * 16 + l];
        *reinterpret_cast<float4*>(spec + T::brick(bx, by, bz) + 2 * c) = make_float4(a.x, a.y, c2.x, c2.y);
    }
}

// Work items: the extra shares of heavy bundles (first, so they start early), then one
// item per bundle for its first share. At G = 512 as many CTAs as are resident take them by
// ticket: a CTA's twiddles (8 KB with their tables) are loaded once and its next item is
// known while it works (16M particles 0.471 -> 0.445 ms, 2M 0.394 -> 0.360). Smaller grids
// take a CTA per item: the loop's registers are spilled there (4M on 256^3 0.153 against
// 0.181 ms, 2M on 128^3 0.062 against 0.074). 40 registers from 128^3 up keep three CTAs
// per SM; smaller grids need more for their FFT stages.
template <int G, bool ISO, bool WIDE>
__global__ void __launch_bounds__(kDepositThreads, kDepositPerSm<G>)
    k_pass_a_deposit_bal(const float4* __restrict__ pos, const int* __restrict__ perm,
                         const int* __restrict__ row_start, float* __restrict__ rho_keep, float2* __restrict__ spec,
                         const float2* __restrict__ tw_g, DepositWork w) {
    wait_previous();
    using P = DepPlan<DepGeo<G, ISO>::M>;
    extern __shared__ float2 sm[];
    __shared__ int s_next;
    const int* items = w.ints + P::kItems;
    const int* xpre = w.ints + P::kXpre;
    const int* cta_pre = w.ints + P::kCtaPre;
    unsigned* arrive = reinterpret_cast<unsigned*>(w.ints + P::kArrive);
    const bool from_grid = kMayStray<WIDE, ISO> && w.ints[P::kUse] != 0;
    const int extras = cta_pre[P::NC];
    if ((int)blockIdx.x >= extras + P::NB) return;  // fewer extra shares than there can be
    for (int i = threadIdx.x; i < G; i += kDepositThreads) sm[i] = tw_g[i];  // ordered by a later barrier
    if constexpr (G == 512) xl::fill_twiddles(sm + G + DepGeo<G, ISO>::kStore, tw_g);  // the twiddle tables, after the sums
    bool reuse = false;
    for (int e = blockIdx.x; e < extras + P::NB; e = s_next, reuse = true) {
        int b = e - extras, slice = 0;
        if (e < extras) {
            // the bundle of extra share e: the last b whose extras start at or before e
            int lo = 0, hi = P::NB - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if (cta_pre[mid >> 8] + xpre[mid] <= e) lo = mid;
                else hi = mid - 1;
            }
            b = lo;
            slice = 1 + e - (cta_pre[lo >> 8] + xpre[lo]);
        }
        // a bundle that one CTA covers whole takes the instantiation without the
        // shared-bundle code: a path that may run costs registers and time even when
        // it does not (0.513 against 0.479 ms at 16M / 512^3)
        // (at 512^3; smaller grids, whose registers the two copies would spill, keep one)
        const int nb = items[b];
        if (G >= 512 && nb == 1 && !from_grid)
            deposit_bundle<G, ISO, WIDE, false>(b, 0, 1, pos, perm, row_start, rho_keep, spec, w, arrive,
                                                w.ints + P::kTicket, &s_next, reuse, false);
        else
            deposit_bundle<G, ISO, WIDE, true>(b, slice, nb, pos, perm, row_start, rho_keep, spec, w, arrive,
                                               w.ints + P::kTicket, &s_next, reuse, from_grid);
        if (!kDepositLoop<G>) break;
    }
}

// Stage bricks into shared memory with cp.async. DIR 1: y-lines of CTA (bx,bz);
// DIR 2: z-lines of CTA (bx,by). Lines: DIR 1 -> z_l*4 + kx_l, DIR 2 -> y_l*4 + kx_l.
// HALF: only the lower half of each line (load_lines, store_lines).
template <int G, int DIR, bool HALF = false>
__device__ __forceinline__ void load_lines(float2* s, const float2* __restrict__ spec, int b0, int b1) {
    using T = Geo<G>;
    constexpr int NB = ((DIR == 1) ? T::NBY : T::NBZ) / (HALF ? 2 : 1);
    for (int u = threadIdx.x; u < NB * 32; u += kFftThreads) {
        const int b = u >> 5, c = u & 31;
        const int e = 2 * c;
        size_t src;
        int dst;
        if (DIR == 1) {  // b = by
            src = T::brick(b0, b, b1) + e;
            dst = fft::at<true>(b * 4 + ((e >> 2) & 3), (e >> 4) * 4 + (e & 3));
        } else {  // b = bz: the brick lands contiguously
            src = T::brick(b0, b1, b) + e;
            dst = b * 64 + e;
        }
        fft::cp_async16(s + dst, spec + src);
    }
    fft::cp_async_wait_all();
    __syncthreads();
}

template <int G, int DIR, bool HALF = false>
__device__ __forceinline__ void store_lines(const float2* s, float2* __restrict__ spec, int bx, int b1) {
    using T = Geo<G>;
    constexpr int NB = ((DIR == 1) ? T::NBY : T::NBZ) / (HALF ? 2 : 1);
    for (int u = threadIdx.x; u < NB * 32; u += kFftThreads) {
        const int b = u >> 5, c = u & 31;
        const int e = 2 * c;
        size_t dst;
        int src;
        if (DIR == 1) {
            dst = T::brick(bx, b, b1) + e;
            src = fft::at<true>(b * 4 + ((e >> 2) & 3), (e >> 4) * 4 + (e & 3));
        } else {
            dst = T::brick(bx, b1, b) + e;
            src = b * 64 + e;
        }
        *reinterpret_cast<float4*>(spec + dst) = *reinterpret_cast<const float4*>(s + src);
    }
}

// ---- passes B and D: y-lines of CTA (bx, bz), in place -------------------------
// HALF (isolated boundary): the density fills the low corner of the box and the
// potential is read only there, so the forward transform's inputs past half the box
// are zero (never written, not read) and the inverse's outputs past it are not
// stored; the grid covers the lower half of the z slabs. At 512 the
// transforms take 85 to 96 registers left alone, two CTAs an SM (240 us); bounded to
// three 201 (B) and 208 (D), 5.3 TB/s, the pruned one 102.
template <int G, bool INV, bool HALF>
__global__ void __launch_bounds__(kFftThreads, G == 512 ? 3 : 0)
    k_pass_y(float2* __restrict__ spec, const float2* __restrict__ tw_g) {
    wait_previous();
    extern __shared__ float2 sm[];
    float2* tw = sm;
    float2* s = sm + G;
    // pass B runs from the last slab to the first: pass A ended there, and those are in L2
    const int bx = blockIdx.x, bz = blockIdx.y ^ (INV ? 0 : Geo<G>::NBZ / (HALF ? 2 : 1) - 1);
    for (int i = threadIdx.x; i < G; i += kFftThreads) tw[i] = tw_g[i];
    load_lines<G, 1, HALF && !INV>(s, spec, bx, bz);
    fft::lines16<G, kFftThreads, 1, INV, HALF && !INV, true>(s, tw);
    store_lines<G, 1, HALF && INV>(s, spec, bx, bz);
}

// ---- pass C: z-lines of CTA (bx, by): forward, Green's function, inverse ---------
// MODE 0: the periodic Green's function (analytic, Sim.cu:528-557).
// MODE 1: forward transform only (builds the isolated boundary's Green spectrum).
// MODE 2: multiply by a tabulated real Green spectrum table[|ky|][kx / 4][|kz|][kx % 4]
//         (columns past kx = H hold zeros) times table_scale, then inverse (isolated
//         boundary, kMulSpec, Sim.cu:578-584). A CTA's values are 4 contiguous runs.
// HALF: the lines' upper half is zero on input and not needed on output (see k_pass_y).
// Two transforms on one trip through memory, so the instructions count (68 % of the issue
// slots at 512, shared memory 63 %), and the butterflies are in pairs here: 512^3 281 ->
// 244 us (4.4 TB/s), 256^3 35.2 -> 31.6, isolated 256^3 28.6 -> 25.9. (In passes B, D and E, which
// wait for memory and shared memory, pairs gain nothing: D at 512 209 -> 224 us.) 80
// registers keep three CTAs of 512 on an SM; a table takes their shared memory.
template <int G, int MODE, bool HALF>
__global__ void __launch_bounds__(kFftThreads, G == 512 && MODE == 0 ? 3 : 0)
    k_pass_c(float2* __restrict__ spec, const float2* __restrict__ tw_g, const float* __restrict__ gexp_g, float scale,
             const float* __restrict__ table, float table_scale) {
    wait_previous();
    using T = Geo<G>;
    constexpr int H = T::H;
    extern __shared__ float2 sm[];
    float2* tw = sm;
    float* gexp = reinterpret_cast<float*>(sm + G);
    float2* s = sm + G + (H + 2) / 2 + 1;
    const int bx = blockIdx.x, by = blockIdx.y;
    for (int i = threadIdx.x; i < G; i += kFftThreads) tw[i] = tw_g[i];
    if (MODE == 0)
        for (int i = threadIdx.x; i <= H; i += kFftThreads) gexp[i] = gexp_g[i];
    __shared__ float line_g[16];
    __shared__ float line_k2[16];
    if (MODE == 0 && threadIdx.x < 16) {
        const int l = threadIdx.x;
        const int kx = bx * 4 + (l & 3), ky = by * 4 + (l >> 2);
        const int kyf = (ky <= G / 2) ? ky : ky - G;
        line_g[l] = (kx <= H) ? -scale * (gexp_g[kx] * gexp_g[abs(kyf)]) : 0.f;  // the global table: no barrier yet
        line_k2[l] = (float)(kx * kx + kyf * kyf);
    }
    // MODE 2: the table's values of these 16 lines, 4 runs of H + 1 groups of 4 bins, come
    // into shared memory with the lines. Fetched at the multiply, each thread's 16 or 32
    // values came one L2 access after another, a sector for each 16 bytes. The runs are
    // 8 banks apart, so the two kz a warp multiplies by do not conflict.
    constexpr int kRun = 4 * (H + 1) + 4;
    float* line_t = reinterpret_cast<float*>(s + 16 * G);
    if (MODE == 2) {
        const float4* t4 = reinterpret_cast<const float4*>(table);
#pragma unroll
        for (int yl = 0; yl < 4; ++yl) {
            const int ky = by * 4 + yl, kyf = (ky <= G / 2) ? ky : G - ky;
            for (int kz = threadIdx.x; kz <= H; kz += kFftThreads)
                fft::cp_async16(line_t + yl * kRun + 4 * kz, t4 + ((size_t)kyf * T::NBX + bx) * (H + 1) + kz);
        }
    }
    load_lines<G, 2, HALF>(s, spec, bx, by);  // ends with a barrier
    if (MODE == 1) {
        fft::lines16<G, kFftThreads, 1, false>(s, tw);
        store_lines<G, 2>(s, spec, bx, by);
        return;
    }
    // forward, Green's function, inverse; the multiply happens in registers between
    // the forward's last stage and the inverse's first
    auto green = [&](int l, int kz, bool upper, float2 x) {
        const int kzf = upper ? G - kz : kz;  // |frequency|
        float m;
        if (MODE == 0) {
            // Green's function: -scale/k^2 * exp(-k^2 s^2/2), k = 0 -> 0 (Sim.cu:536-556), with
            // the per-line factors of (kx, ky) hoisted; padding columns kx > H are zeroed.
            // k^2 <= 3 * 256^2 is exact in a float.
            const float k2 = fmaf((float)kzf, (float)kzf, line_k2[l]);
            float inv;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(k2));
            m = (kz != 0 || k2 != 0.f) ? line_g[l] * gexp[kzf] * inv : 0.f;
        } else {
            m = line_t[(l >> 2) * kRun + 4 * kzf + (l & 3)] * table_scale;
        }
        return make_float2(x.x * m, x.y * m);
    };
    fft::convolve16<G, kFftThreads, 1, HALF>(s, tw, green);
    store_lines<G, 2, HALF>(s, spec, bx, by);
}

// Real part of a forward spectrum (bricked) into table[|ky|][kx / 4][|kz|][kx % 4].
template <int G>
__global__ void k_green_table(const float2* __restrict__ spec, float* __restrict__ table) {
    using T = Geo<G>;
    constexpr int H = T::H;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t n = (size_t)(H + 1) * T::PX * (H + 1);
    if (i >= n) return;
    const size_t g = i >> 2;
    const int kz = (int)(g % (H + 1)), bx = (int)(g / (H + 1) % T::NBX), ky = (int)(g / ((size_t)(H + 1) * T::NBX));
    const int kx = 4 * bx + (int)(i & 3);
    const size_t e = T::brick(bx, ky >> 2, kz >> 2) + (size_t)((kz & 3) * 16 + (ky & 3) * 4 + (kx & 3));
    table[i] = kx <= H ? spec[e].x : 0.f;
}

// Real-space isolated kernel on the transform box (kGreen, Sim.cu:563-576):
// g = -1 / (r + soft), r the distance in cells to the nearest corner copy.
__global__ void k_green_kernel(float* __restrict__ g, int S, float soft) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)S * S * S) return;
    const int x = (int)(i % S), y = (int)((i / S) % S), z = (int)(i / ((size_t)S * S));
    const int dx = (x <= S / 2) ? x : S - x;
    const int dy = (y <= S / 2) ? y : S - y;
    const int dz = (z <= S / 2) ? z : S - z;
    const float r = sqrtf((float)(dx * dx + dy * dy + dz * dz)) + soft;
    g[i] = -1.0f / r;
}

// ---- pass E: kx bins -> real rows (y = 4by + y_l, z = 4bz + z_l) ----------------
// HALF (isolated boundary): only the lower half of each row is needed and stored;
// the grid covers the rows of the low corner.
template <int G, bool HALF>
__global__ void __launch_bounds__(kFftThreads, 5) k_pass_e(const float2* __restrict__ spec, float* __restrict__ phi,
                                                        const float2* __restrict__ tw_g) {
    wait_previous();
    using T = Geo<G>;
    constexpr int H = T::H, NBX = T::NBX;
    constexpr int ITEMS = NBX * 32;
    constexpr int PER = (ITEMS + kFftThreads - 1) / kFftThreads;
    extern __shared__ float2 sm[];
    float2* tw = sm;
    float2* s = sm + G;
    // CTAs run from the last row bundle to the first: pass D ends on the high-z slabs, still in L2,
    // and the gather starts on the low-z rows of phi written last here (same results, ~8 us less)
    const int by = gridDim.x - 1 - blockIdx.x, bz = gridDim.y - 1 - blockIdx.y;
    for (int i = threadIdx.x; i < G; i += kFftThreads) tw[i] = tw_g[i];
    float4 v[PER];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * kFftThreads;
        if (ITEMS % kFftThreads == 0 || u < ITEMS)
            v[p] = *reinterpret_cast<const float4*>(spec + T::brick(u >> 5, by, bz) + 2 * (u & 31));
    }
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * kFftThreads;
        if (ITEMS % kFftThreads == 0 || u < ITEMS) {
            const int bx = u >> 5, c = u & 31;
            const int l = (c >> 3) * 4 + ((c >> 1) & 3), kx = bx * 4 + (c & 1) * 2;
            s[kx * 16 + l] = make_float2(v[p].x, v[p].y);
            s[(kx + 1) * 16 + l] = make_float2(v[p].z, v[p].w);
        }
    }
    __syncthreads();
    // X -> Z inside the first stage's loads: Z[k] = E + i O with
    //   E = X[k] + conj X[H-k],  O = (X[k] - conj X[H-k]) * exp(+2 pi i k / G)
    // (imaginary parts of the k = 0 and k = H bins are dropped, as a C2R transform
    // does), read from the staged bins, which the stage overwrites only after its
    // barrier. This saves the separate pass over the pairs and its barrier.
    auto c2r_load = [tw](const float2* s, int l, int k) {
        float2 a = s[k * 16 + l], b = s[(H - k) * 16 + l];
        if (k == 0) { a.y = 0.f; b.y = 0.f; }
        const float2 w = tw[k];
        const float er = a.x + b.x, ei = a.y - b.y, dr = a.x - b.x, di = a.y + b.y;
        const float orr = dr * w.x + di * w.y, oi = di * w.x - dr * w.y;
        return make_float2(er - oi, ei + orr);
    };
    // The last stage leaves the lines row-major (stride H + 2 float2, 16-byte
    // aligned), so each warp then writes 512 contiguous bytes of one row instead
    // of 32 bytes of each of 16 rows.
    constexpr int RS = H + 2;
    static_assert(16 * RS <= 16 * T::PX, "row staging fits the line buffer");
    fft::lines16_rows<H, kFftThreads, 2, true, RS>(s, tw, c2r_load);
    constexpr int Q = HALF ? H / 4 : H / 2;  // float4 of a row
    for (int u = threadIdx.x; u < 16 * Q; u += kFftThreads) {
        const int l = u / Q, mp = u % Q;
        const size_t row = ((size_t)(bz * 4 + (l >> 2)) * G + by * 4 + (l & 3)) * G;
        const float4 ab = *reinterpret_cast<const float4*>(s + l * RS + 2 * mp);
        *reinterpret_cast<float4*>(phi + row + 4 * mp) = ab;
    }
}

template <int G>
struct Launcher {
    using T = Geo<G>;
    static size_t smem_ae() { return sizeof(float2) * ((size_t)G + 16 * (size_t)T::PX); }
    // pass A from a grid: at G = 512 the twiddle tables, 16 warp scratches and the brick staging
    static size_t smem_a() {
        return G == 512 ? sizeof(float2) * ((size_t)G + xl::kTw2 + 16 * 256 + xl::kStage) : smem_ae();
    }
    static size_t smem_bd() { return sizeof(float2) * ((size_t)G + 16 * (size_t)G); }
    static size_t smem_c() { return sizeof(float2) * ((size_t)G + (T::H + 2) / 2 + 1 + 16 * (size_t)G); }
    // and the table's values; the lines before them end on a 16-byte boundary
    static size_t smem_ct() { return smem_c() + sizeof(float) * 16 * (size_t)(T::H + 2); }
    // the line buffer overlays the 32-bit sum words (DepGeo); at G = 512 the warp-per-line
    // transform's twiddle tables follow
    template <bool ISO>
    static size_t smem_bal() {
        return sizeof(float2) * ((size_t)G + DepGeo<G, ISO>::kStore + (G == 512 ? xl::kTw2 : 0));
    }
    template <bool ISO, bool WIDE>
    static int deposit(const PoissonPlan& p, const float4* pos, const int* perm, const int* row_start, float* keep,
                       float2* spec, const DepositWork& dw, cudaStream_t s) {
        using P = DepPlan<DepGeo<G, ISO>::M>;
        // an isolated share is one that the plain sums hold (kIsoShare)
        const int split = ISO && dw.split > kIsoShare ? kIsoShare : dw.split;
        const int piece = dw.piece > split ? split : dw.piece;
        launch(k_deposit_plan<DepGeo<G, ISO>::M, WIDE, ISO>, P::NC, 256, 0, s, row_start, dw.ints, split, piece, pos, dw.n,
               reinterpret_cast<unsigned long long*>(dw.acc));
        SD_LAUNCHED(s);
        // a CTA for each extra share that there can be, so none waits for another (a window of
        // w particles has at most w / piece extra shares, and a particle lies in at most four
        // windows); idle ones cost little, 1.5 us for 1,024. Never more than are taken by ticket.
        const long long extra = 4ll * dw.n / piece, wave = 148 * kDepositPerSm<G>;
        const long long ctas = P::NB + (extra < 8 ? 8 : extra);
        launch(k_pass_a_deposit_bal<G, ISO, WIDE>, (unsigned)(kDepositLoop<G> && ctas > wave ? wave : ctas), kDepositThreads,
               smem_bal<ISO>(), s, pos, perm, row_start, keep, spec, p.tw, dw);
        SD_LAUNCHED(s);
        return SD_OK;
    }

    static constexpr bool kIsoBox = G >= 32;  // the transform box of an isolated grid of side G / 2 >= 16

    // The kernels that a plan's use launches, and no others: setting an attribute loads the
    // kernel. All fifteen took a process's first simulation from 11.0 to 13.6 ms (2,000,000
    // on 128^3), an isolated one from 13.3 to 14.9; these take 12.5 and 13.4.
    static int configure(PoissonUse use) {
        int rc = SD_OK;
        // prefer the largest shared-memory carveout so several 70 KB CTAs fit per SM
        auto set = [&rc](auto* kernel, size_t smem) {
            rc |= SD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                               (int)cudaSharedmemCarveoutMaxShared));
            rc |= SD_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        };
        if (use != PoissonUse::kPeriodic) set(k_pass_a<G, 0>, smem_a());
        if (use != PoissonUse::kGrid) set(k_pass_a<G, 1>, smem_a());
        set(k_pass_y<G, false, false>, smem_bd());
        if (use == PoissonUse::kIsolated) {
            if constexpr (kIsoBox) {
                set(k_pass_c<G, 1, false>, smem_c());
                set(k_pass_y<G, false, true>, smem_bd());
                set(k_pass_y<G, true, true>, smem_bd());
                set(k_pass_c<G, 2, true>, smem_ct());
                set(k_pass_e<G, true>, smem_ae());
                set(k_pass_a_deposit_bal<G, true, false>, smem_bal<true>());
                set(k_pass_a_deposit_bal<G, true, true>, smem_bal<true>());
            }
        } else {
            set(k_pass_y<G, true, false>, smem_bd());
            set(k_pass_c<G, 0, false>, smem_c());
            set(k_pass_e<G, false>, smem_ae());
        }
        if (use == PoissonUse::kPeriodic) {
            set(k_pass_a_deposit_bal<G, false, false>, smem_bal<false>());
            set(k_pass_a_deposit_bal<G, false, true>, smem_bal<false>());
        }
        return rc == SD_OK ? SD_OK : SD_E_CUDA;
    }

    static int run(const PoissonPlan& p, const long long* acc, const float* rho, const float4* pos, const int* perm,
                   const int* row_start, float* keep, float2* spec, float* phi, cudaStream_t s, cudaEvent_t* ev,
                   const PoissonIso* iso, const DepositWork* dw) {
        const int src_g = (iso && iso->src_g > 0) ? iso->src_g : G;
        // isolated boundary: the density fills an eighth of the box and the potential is
        // read only there. Pass A runs on the quarter of the rows that hold particles,
        // the y passes on the half of the slabs, every line reads and stores the half
        // that is not zero or wanted, pass E makes a quarter of the rows: a third of the
        // full box's traffic (a 256^3 box: A 39 -> 19 us, B 27 -> 13, C 42 -> 29, D 27 -> 13,
        // E 33 -> 9; a 512^3 box: 266 -> 90, 210 -> 112, 402 -> 253, 210 -> 88, 234 -> 55).
        const bool half = kIsoBox && iso && iso->table && 2 * src_g == G;
        if (iso && iso->table && !half)
            return fail(SD_E_ARG, "poisson: the isolated density has half the box's side");
        const int hy = half ? T::NBY / 2 : T::NBY, hz = half ? T::NBZ / 2 : T::NBZ;
        const dim3 grid_rows(hy, hz), grid_y(T::NBX, hz), grid_z(T::NBX, T::NBY);
        if (pos) {
            if (!dw || !dw->acc || !dw->ints || dw->split <= 0 || dw->piece <= 0)
                return fail(SD_E_ARG, "fused deposit: no work plan");
            int rc = SD_OK;
            if constexpr (kIsoBox) {
                if (half)
                    rc = dw->wide ? deposit<true, true>(p, pos, perm, row_start, keep, spec, *dw, s)
                                  : deposit<true, false>(p, pos, perm, row_start, keep, spec, *dw, s);
            }
            if (!half)
                rc = dw->wide ? deposit<false, true>(p, pos, perm, row_start, keep, spec, *dw, s)
                              : deposit<false, false>(p, pos, perm, row_start, keep, spec, *dw, s);
            if (rc) return rc;
        } else {
            if (acc)
                launch(k_pass_a<G, 1>, grid_rows, kPassAThreads<G>, smem_a(), s, nullptr, const_cast<long long*>(acc), keep,
                       spec, p.tw, src_g);
            else
                launch(k_pass_a<G, 0>, grid_rows, kPassAThreads<G>, smem_a(), s, rho, nullptr, keep, spec, p.tw, src_g);
            SD_LAUNCHED(s);
        }
        if (ev) cudaEventRecord(ev[0], s);
        if constexpr (kIsoBox) {
            if (half) {
                launch(k_pass_y<G, false, true>, grid_y, kFftThreads, smem_bd(), s, spec, p.tw);
                SD_LAUNCHED(s);
                if (ev) cudaEventRecord(ev[1], s);
                launch(k_pass_c<G, 2, true>, grid_z, kFftThreads, smem_ct(), s, spec, p.tw, p.gexp, p.scale, iso->table,
                       iso->table_scale);
                SD_LAUNCHED(s);
                if (ev) cudaEventRecord(ev[2], s);
                launch(k_pass_y<G, true, true>, grid_y, kFftThreads, smem_bd(), s, spec, p.tw);
                SD_LAUNCHED(s);
                if (ev) cudaEventRecord(ev[3], s);
                launch(k_pass_e<G, true>, grid_rows, kFftThreads, smem_ae(), s, spec, phi, p.tw);
                SD_LAUNCHED(s);
                return SD_OK;
            }
        }
        launch(k_pass_y<G, false, false>, grid_y, kFftThreads, smem_bd(), s, spec, p.tw);
        SD_LAUNCHED(s);
        if (ev) cudaEventRecord(ev[1], s);
        if (iso && iso->forward_only) {
            launch(k_pass_c<G, 1, false>, grid_z, kFftThreads, smem_c(), s, spec, p.tw, p.gexp, p.scale, nullptr, 0.f);
            SD_LAUNCHED(s);
            return SD_OK;
        }
        launch(k_pass_c<G, 0, false>, grid_z, kFftThreads, smem_c(), s, spec, p.tw, p.gexp, p.scale, nullptr, 0.f);
        SD_LAUNCHED(s);
        if (ev) cudaEventRecord(ev[2], s);
        launch(k_pass_y<G, true, false>, grid_y, kFftThreads, smem_bd(), s, spec, p.tw);
        SD_LAUNCHED(s);
        if (ev) cudaEventRecord(ev[3], s);
        launch(k_pass_e<G, false>, grid_rows, kFftThreads, smem_ae(), s, spec, phi, p.tw);
        SD_LAUNCHED(s);
        return SD_OK;
    }
};

// The Green's function's exponent table exp(-(2 pi soft / G)^2 k^2 / 2), k = 0..G/2,
// evaluated in FP64 and rounded once (both Poisson entry points build it here).
__global__ void k_fill_gexp(float* __restrict__ gexp, int G, float soft) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > G / 2) return;
    const double s = 6.283185307179586476925286766559 * (double)(soft > 0.f ? soft : 0.f) / (double)G;
    gexp[k] = (float)exp(-0.5 * s * s * (double)k * (double)k);
}

int fill_gexp(float* gexp, int G, float soft, cudaStream_t st) {
    k_fill_gexp<<<(G / 2 + 1 + 127) / 128, 128, 0, st>>>(gexp, G, soft);
    SD_LAUNCHED(st);
    return SD_OK;
}

int poisson_configure(int G, PoissonUse use) {
    switch (G) {
        case 16: return Launcher<16>::configure(use);
        case 32: return Launcher<32>::configure(use);
        case 64: return Launcher<64>::configure(use);
        case 128: return Launcher<128>::configure(use);
        case 256: return Launcher<256>::configure(use);
        case 512: return Launcher<512>::configure(use);
        default: return fail(SD_E_UNSUPPORTED, "poisson: grid size %d not supported", G);
    }
}

}  // namespace

size_t deposit_work_ints(int G) {
    switch (G) {
        case 16: return DepPlan<16>::kInts;
        case 32: return DepPlan<32>::kInts;
        case 64: return DepPlan<64>::kInts;
        case 128: return DepPlan<128>::kInts;
        case 256: return DepPlan<256>::kInts;
        case 512: return DepPlan<512>::kInts;
        default: return 0;
    }
}

int* deposit_stray_flag(int* ints, int G) { return ints + deposit_work_ints(G) - 1; }

int deposit_split(int n, int G, int mult) {
    const long long nb = (long long)G * G / 16;
    const long long t = (long long)mult * (long long)n / (nb > 0 ? nb : 1);
    return (int)(t < 2048 ? 2048 : (t > (1 << 30) ? (1 << 30) : t));
}

void deposit_shares(DepositWork& w, int n, int G) {
    // Three times a window's mean particle count at 256 bundles, which are resident all at
    // once, so the time is the heaviest share's; six times at 1024, ten times above, where
    // shares cost more than they balance (each adds its rows with global atomics); at least
    // 2048. 262,144 particles of a disk on 64^3: 31 us with 5x, 19.5 with 3x, 19.4 with 2x;
    // 1,000,003 on an isolated 128^3 74 us with 10x, 67 with 6x, 64 with 4x, but 2,000,000 of
    // a ball 62, 64 and 69; 4M on 256^3 (two galaxies) 154 with 10x and 6x, 160 with 4x.
    const int nb = G * G / 16;
    w.split = w.piece = deposit_split(n, G, nb <= 256 ? 3 : (nb <= 1024 ? 6 : 10));
    if (nb > 64) return;
    // The 16 or 64 bundles of 16^3 and 32^3 leave most of the chip idle, and a CTA that adds
    // thousands of particles to a few cells alone takes longer than global atomics from the
    // whole chip would. So a window is split into shares that fill the chip once between them,
    // where it holds enough to pay for their atomics: more than an even spread gives up to
    // some 50,000 particles on 16^3 and 170,000 on 32^3, less above. A step on 16^3 in
    // row-major and tiled order, with the rule above and now: 100,000 spread evenly 57 and 39
    // us, 41 and 31; on the edge of an isolated box 130 and 167, 47 and 45 (101 and 88 with
    // global atomics). 1,000,000 on 32^3: 128 and 82 us, 97 and 68; 20,000 there 38 and 28,
    // the same.
    const int most = n / 48 > 6144 ? n / 48 : 6144;
    w.split = n / 24 < 2048 ? 2048 : (n / 24 > most ? most : n / 24);
    w.piece = n / 128 > 512 ? n / 128 : 512;
}

size_t poisson_spectrum_elems(int G) { return (size_t)G * G * (size_t)(G / 2 + 4); }

int poisson_plan_build(PoissonPlan& p, int G, float soft, PoissonUse use) {
    if (p.G == G && p.soft == soft && p.tw) return SD_OK;
    poisson_plan_free(p);
    // kernel attributes are set here, outside any stream capture
    if (int rc = poisson_configure(G, use)) return rc;
    std::vector<float2> tw((size_t)G);
    const double two_pi = 6.283185307179586476925286766559;
    for (int m = 0; m < G; ++m) {
        const double a = -two_pi * (double)m / (double)G;
        tw[m] = make_float2((float)cos(a), (float)sin(a));
    }
    if (SD_CUDA(cudaMalloc(&p.tw, sizeof(float2) * tw.size())) != SD_OK) return SD_E_NOMEM;
    if (SD_CUDA(cudaMalloc(&p.gexp, sizeof(float) * ((size_t)G / 2 + 1))) != SD_OK) return SD_E_NOMEM;
    if (SD_CUDA(cudaMemcpy(p.tw, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice)) != SD_OK)
        return SD_E_CUDA;
    // the same kernel as the allocation-free solve's, so both tables hold the same bits
    if (int rc = fill_gexp(p.gexp, G, soft, nullptr)) return rc;
    if (SD_CUDA(cudaStreamSynchronize(nullptr))) return SD_E_CUDA;
    p.scale = (float)(1.0 / (4.0 * 3.14159265358979323846 * 3.14159265358979323846 * (double)G * G * G));
    p.G = G;
    p.soft = soft;
    return SD_OK;
}

void poisson_plan_free(PoissonPlan& p) {
    if (p.tw) cudaFree(p.tw);
    if (p.gexp) cudaFree(p.gexp);
    p.tw = nullptr;
    p.gexp = nullptr;
    p.G = 0;
}

int launch_poisson(const PoissonPlan& p, const long long* acc, const float* rho, float* keep, float2* spec,
                   float* phi, cudaStream_t s) {
    return launch_poisson_ex(p, acc, rho, nullptr, nullptr, nullptr, keep, spec, phi, s);
}

int launch_poisson_ex(const PoissonPlan& p, const long long* acc, const float* rho, const float4* pos,
                      const int* perm, const int* row_start, float* keep, float2* spec, float* phi, cudaStream_t s,
                      cudaEvent_t* ev, const PoissonIso* iso, const DepositWork* dw) {
    switch (p.G) {
        case 16: return Launcher<16>::run(p, acc, rho, pos, perm, row_start, keep, spec, phi, s, ev, iso, dw);
        case 32: return Launcher<32>::run(p, acc, rho, pos, perm, row_start, keep, spec, phi, s, ev, iso, dw);
        case 64: return Launcher<64>::run(p, acc, rho, pos, perm, row_start, keep, spec, phi, s, ev, iso, dw);
        case 128: return Launcher<128>::run(p, acc, rho, pos, perm, row_start, keep, spec, phi, s, ev, iso, dw);
        case 256: return Launcher<256>::run(p, acc, rho, pos, perm, row_start, keep, spec, phi, s, ev, iso, dw);
        case 512: return Launcher<512>::run(p, acc, rho, pos, perm, row_start, keep, spec, phi, s, ev, iso, dw);
        default: return fail(SD_E_UNSUPPORTED, "poisson: grid size %d not supported", p.G);
    }
}

size_t green_table_elems(int S) {
    const size_t h = (size_t)S / 2 + 1;
    return h * h * (h + 3);
}

int build_green_table(const PoissonPlan& p, float softening_cells, float* kernel_grid, float2* spec, float* table,
                      cudaStream_t s) {
    const int S = p.G;
    const size_t cells = (size_t)S * S * S;
    // the reference floors the isolated softening at half a cell (buildGreen, Sim.cu:3569-3575)
    const float soft = softening_cells > 0.5f ? softening_cells : 0.5f;
    k_green_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, s>>>(kernel_grid, S, soft);
    SD_LAUNCHED(s);
    PoissonIso fwd;
    fwd.forward_only = true;
    if (int rc = launch_poisson_ex(p, nullptr, kernel_grid, nullptr, nullptr, nullptr, nullptr, spec, nullptr, s,
                                   nullptr, &fwd))
        return rc;
    const size_t n = green_table_elems(S);
    switch (S) {
        case 32: k_green_table<32><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(spec, table); break;
        case 64: k_green_table<64><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(spec, table); break;
        case 128: k_green_table<128><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(spec, table); break;
        case 256: k_green_table<256><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(spec, table); break;
        case 512: k_green_table<512><<<(unsigned)((n + 255) / 256), 256, 0, s>>>(spec, table); break;
        default: return fail(SD_E_UNSUPPORTED, "isolated: transform size %d not supported", S);
    }
    SD_LAUNCHED(s);
    return SD_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free Poisson solve (sd_poisson_noalloc).
//
// For callers that must not allocate device memory: code running where
// cudaMalloc is not allowed, such as inside another library's allocator-free
// hot loop, or under a strict memory budget that forbids growth after start-up.
// Its working memory
// is file-scope device storage of fixed size, so grids are limited to
// kNoAllocMaxGrid^3. Every GPU that loads this library holds that storage
// (about 9 MB) until the process exits, and all calls on a device share it:
// calls that overlap on the GPU race on it.
// ---------------------------------------------------------------------------
namespace {

constexpr int kNoAllocMaxGrid = 128;
constexpr size_t kNoAllocSpecElems =
    (size_t)kNoAllocMaxGrid * kNoAllocMaxGrid * (size_t)(kNoAllocMaxGrid / 2 + 4);
constexpr int kNoAllocMaxDevices = 64;

// The bricked spectrum of the largest supported grid, the twiddle tables of
// G = 16, 32, 64, 128 (one row of kNoAllocMaxGrid entries each) and the
// Green's-function exponent table of the current call.
static __device__ __align__(256) float2 g_noalloc_spec[kNoAllocSpecElems];
static __device__ __align__(256) float2 g_noalloc_tw[4 * kNoAllocMaxGrid];
static __device__ __align__(256) float g_noalloc_gexp[kNoAllocMaxGrid / 2 + 1];

struct NoAllocDevice {
    bool ready = false;
    unsigned long long ctx_id = 0;  // the context the addresses and tables belong to
    float2* spec = nullptr;
    float2* tw = nullptr;
    float* gexp = nullptr;
};

// The unique ID of the current context (cuCtxGetId through the runtime's driver
// entry points; 0 if unavailable). A device reset ends the context: its file-scope
// arrays come back zeroed under a new ID, so the cached set-up is redone.
unsigned long long current_ctx_id() {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(f);
        cudaGetLastError();
    });
    CUcontext c = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&c) != CUDA_SUCCESS || !c || get_id(c, &id) != CUDA_SUCCESS) return 0;
    return id;
}
NoAllocDevice g_noalloc[kNoAllocMaxDevices];
std::mutex g_noalloc_mu;

int noalloc_slot(int G) { return G == 16 ? 0 : (G == 32 ? 1 : (G == 64 ? 2 : 3)); }

// Once per device, with that device current: resolve the device addresses of
// the file-scope arrays (their names are host-side stand-ins in host code),
// upload the twiddle tables and set the kernels' shared-memory attributes.
int noalloc_setup(int dev) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    NoAllocDevice& d = g_noalloc[dev];
    void* p = nullptr;
    // resolving a symbol also makes the device's context current, which the ID needs
    if (SD_CUDA(cudaGetSymbolAddress(&p, g_noalloc_spec))) return SD_E_CUDA;
    const unsigned long long ctx = current_ctx_id();
    if (d.ready && ctx == d.ctx_id) return SD_OK;
    d.ready = false;
    d.ctx_id = ctx;
    d.spec = static_cast<float2*>(p);
    if (SD_CUDA(cudaGetSymbolAddress(&p, g_noalloc_tw))) return SD_E_CUDA;
    d.tw = static_cast<float2*>(p);
    if (SD_CUDA(cudaGetSymbolAddress(&p, g_noalloc_gexp))) return SD_E_CUDA;
    d.gexp = static_cast<float*>(p);
    std::vector<float2> tw((size_t)4 * kNoAllocMaxGrid, make_float2(0.f, 0.f));
    const double two_pi = 6.283185307179586476925286766559;
    for (int G = 16; G <= kNoAllocMaxGrid; G *= 2) {
        float2* row = tw.data() + (size_t)noalloc_slot(G) * kNoAllocMaxGrid;
        for (int m = 0; m < G; ++m) {
            const double a = -two_pi * (double)m / (double)G;
            row[m] = make_float2((float)cos(a), (float)sin(a));
        }
        if (int rc = poisson_configure(G, PoissonUse::kGrid)) return rc;
    }
    if (SD_CUDA(cudaMemcpy(d.tw, tw.data(), sizeof(float2) * tw.size(), cudaMemcpyHostToDevice))) return SD_E_CUDA;
    d.ready = true;
    return SD_OK;
}

}  // namespace

}  // namespace sd

extern "C" int sd_poisson_noalloc(const float* rho, int grid_size, float softening_cells, float* phi, void* stream) {
    using namespace sd;
    const int G = grid_size;
    if (!rho || !phi) return fail(SD_E_ARG, "sd_poisson_noalloc: null rho or phi");
    if (G < 16 || G > kNoAllocMaxGrid || (G & (G - 1)))
        return fail(SD_E_ARG,
                    "sd_poisson_noalloc: grid_size %d is not a power of two in [16, %d]; its fixed workspace holds "
                    "the spectrum of a %d^3 grid at most (use sd_poisson with a caller workspace for larger grids)",
                    G, kNoAllocMaxGrid, kNoAllocMaxGrid);
    int dev = 0;
    if (SD_CUDA(cudaGetDevice(&dev))) return SD_E_CUDA;
    if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(SD_E_ARG, "sd_poisson_noalloc: device %d unsupported", dev);
    if (int rc = noalloc_setup(dev)) return rc;
    const NoAllocDevice& d = g_noalloc[dev];
    cudaStream_t st = (cudaStream_t)stream;
    // the exponent table depends on the softening: rebuilt by every call
    if (int rc = fill_gexp(d.gexp, G, softening_cells, st)) return rc;
    PoissonPlan plan;
    plan.G = G;
    plan.soft = softening_cells;
    plan.tw = d.tw + (size_t)noalloc_slot(G) * kNoAllocMaxGrid;
    plan.gexp = d.gexp;
    plan.scale = (float)(1.0 / (4.0 * 3.14159265358979323846 * 3.14159265358979323846 * (double)G * G * G));
    // pass A writes every spectrum element (padding columns as zeros), so the
    // shared workspace needs no clearing between calls
    const int rc = launch_poisson(plan, nullptr, rho, nullptr, d.spec, phi, st);
    plan.tw = nullptr;  // static storage: the plan does not own it
    plan.gexp = nullptr;
    return rc;
}

