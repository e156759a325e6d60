// sd_mlp.cu -- learned sub-grid force correction: features, BF16 tensor-core
// MLP (30 -> 64 -> 64 -> 3, SiLU), its training kernels and the fused inference
// that feeds the kick. No counterpart in the reference; the correction is added
// on top of the plain PM acceleration (kIntegrate's accG sample, Sim.cu:822).
//
// Numerics: weights and activations are BF16, every matrix product accumulates
// in FP32 on the tensor cores (mma.sync m16n8k16), biases and the SiLU are FP32,
// master weights and Adam moments are FP32.
//
// Parameter vector (FP32, kMlpParams floats): W1[32][64] (inputs padded 30->32),
// b1[64], W2[64][64], b2[64], W3[64][8] (outputs padded 3->8), b3[8]; W[k][n]
// maps input k to output n.
//
// Features of a particle at p (grid G, mean count per cell rho_bar):
//   f[(dz+1)*9 + (dy+1)*3 + (dx+1)] = log(1 + rho(c + d) / rho_bar) - log 2,  d in {-1,0,1}^3
//   f[27..29] = p*G - c - 1/2 (sub-cell offset), f[30] = f[31] = 0,
// with c = floor(p*G) the containing cell and rho the CIC density (count units).
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "sd_common.cuh"
#include "sd_internal.h"

namespace sd {
namespace {

constexpr int kIn = 32, kH = 64, kOut = 8;
constexpr int oW1 = 0, oB1 = oW1 + kIn * kH, oW2 = oB1 + kH, oB2 = oW2 + kH * kH, oW3 = oB2 + kH,
              oB3 = oW3 + kH * kOut, kParams = oB3 + kOut;
static_assert(kParams == 6792, "parameter layout");

__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);  // .x = lo (low 16 bits)
    return *reinterpret_cast<const unsigned*>(&v);
}

__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%0,%1,%2,%3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// d = a b + c
__device__ __forceinline__ void mma16816(float (&d)[4], const unsigned (&a)[4], unsigned b0, unsigned b1,
                                         const float4& c) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
        "{%10,%11,%12,%13};\n"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
}

// SiLU through the hardware tanh (one MUFU op): sigmoid(z) = (1 + tanh(z/2)) / 2.
// Its relative error (about 2^-11) is below the BF16 rounding of the activations;
// training and inference use the same function.
__device__ __forceinline__ float tanh_approx(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float sigmoid(float z) { return fmaf(0.5f, tanh_approx(0.5f * z), 0.5f); }

__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
__device__ __forceinline__ float silu_grad(float z) {
    const float s = sigmoid(z);
    return s * fmaf(z, 1.f - s, 1.f);
}

// ---- features -------------------------------------------------------------------
// the density feature of one cell: log(1 + rho / rho_bar) - log 2
// (its argument is at least 1, so flushing subnormals changes nothing)
__device__ __forceinline__ float cell_feature(float r, float inv_mean) {
    float l;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(fmaf(r, inv_mean, 1.f)));
    return fmaf(l, 0.69314718055994531f, -0.69314718055994531f);
}

// The density feature of every cell in BF16, as the network takes it: a step's particles
// read each cell's many times (four cells a thread; the grid's side is a multiple of 16).
__global__ void __launch_bounds__(256) k_feature_table(const float4* __restrict__ rho, size_t quads, float inv_mean,
                                                       uint2* __restrict__ table) {
    wait_previous();
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= quads) return;
    const float4 r = rho[i];
    table[i] = make_uint2(pack_bf16(cell_feature(r.x, inv_mean), cell_feature(r.y, inv_mean)),
                          pack_bf16(cell_feature(r.z, inv_mean), cell_feature(r.w, inv_mean)));
}

__device__ __forceinline__ void particle_features(const float* __restrict__ rho, int G, float inv_mean, float4 p,
                                                  float* f) {
    const int m = G - 1;
    const int cx = min(max((int)(p.x * (float)G), 0), m);
    const int cy = min(max((int)(p.y * (float)G), 0), m);
    const int cz = min(max((int)(p.z * (float)G), 0), m);
#pragma unroll
    for (int dz = -1; dz <= 1; ++dz)
#pragma unroll
        for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
            for (int dx = -1; dx <= 1; ++dx) {
                const float r =
                    __ldg(rho + ((size_t)((cz + dz) & m) * G + ((cy + dy) & m)) * G + ((cx + dx) & m));
                f[(dz + 1) * 9 + (dy + 1) * 3 + (dx + 1)] = cell_feature(r, inv_mean);
            }
    f[27] = p.x * (float)G - (float)cx - 0.5f;
    f[28] = p.y * (float)G - (float)cy - 0.5f;
    f[29] = p.z * (float)G - (float)cz - 0.5f;
    f[30] = 0.f;
    f[31] = 0.f;
}

// The 16 packed feature words of p, from the table: the three cells of a row lie in two
// aligned words (two loads where there were three, no logarithm, no rounding).
__device__ __forceinline__ void table_features(const unsigned* __restrict__ table, int G, float4 p, unsigned (&f)[16]) {
    const int m = G - 1, mw = (G >> 1) - 1;
    const int cx = cell_axis(p.x, G), cy = cell_axis(p.y, G), cz = cell_axis(p.z, G);
    const int w0 = ((cx - 1) >> 1) & mw, w1 = (w0 + 1) & mw;
    const int shift = ((cx - 1) & 1) * 16;
    unsigned lo[9], hi[9];  // the row's words
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        const int y = (cy + r % 3 - 1) & m, z = (cz + r / 3 - 1) & m;
        const unsigned* row = table + ((size_t)z * G + y) * (G >> 1);
        lo[r] = __ldg(row + w0);
        hi[r] = __ldg(row + w1);
    }
#pragma unroll
    for (int r = 0; r < 9; ++r) {  // cells 0 and 1 of the row in lo, cell 2 in the low half of hi
        lo[r] = __funnelshift_r(lo[r], hi[r], shift);
        hi[r] >>= shift;
    }
    // features 3 r, 3 r + 1, 3 r + 2; three words hold two rows
#pragma unroll
    for (int r = 0; r < 8; r += 2) {
        f[3 * r / 2] = lo[r];
        f[3 * r / 2 + 1] = __byte_perm(hi[r], lo[r + 1], 0x5410);
        f[3 * r / 2 + 2] = __byte_perm(lo[r + 1], hi[r + 1], 0x5432);
    }
    f[12] = lo[8];
    const float ox = p.x * (float)G - (float)cx - 0.5f, oy = p.y * (float)G - (float)cy - 0.5f,
                oz = p.z * (float)G - (float)cz - 0.5f;
    f[13] = __byte_perm(hi[8], pack_bf16(0.f, ox), 0x7610);
    f[14] = pack_bf16(oy, oz);
    f[15] = 0u;
}

__global__ void k_features(const float4* __restrict__ pos, const int* __restrict__ perm, int n,
                           const float* __restrict__ rho, int G, float inv_mean, __nv_bfloat16* __restrict__ out) {
    wait_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 p = pos[perm ? perm[i] : i];
    float f[32];
    if (p.x < 0.f) {
#pragma unroll
        for (int j = 0; j < 32; ++j) f[j] = 0.f;
    } else {
        particle_features(rho, G, inv_mean, p, f);
    }
    uint4* o = reinterpret_cast<uint4*>(out + (size_t)i * kIn);
#pragma unroll
    for (int q = 0; q < 4; ++q)
        o[q] = make_uint4(pack_bf16(f[8 * q], f[8 * q + 1]), pack_bf16(f[8 * q + 2], f[8 * q + 3]),
                          pack_bf16(f[8 * q + 4], f[8 * q + 5]), pack_bf16(f[8 * q + 6], f[8 * q + 7]));
}

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldm4(unsigned (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}
__device__ __forceinline__ void ldm4t(unsigned (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}

// ---- fused inference -----------------------------------------------------------------
// Each warp takes 32 particles, a lane each, through the network by itself: the lane
// forms its particle's features, the warp swaps them through a shared-memory row each
// into the A fragments of two m16n8k16 row tiles, and from there every layer stays in
// registers: the accumulators of 16 units, activated and packed to BF16, are one k-step
// of the next layer's A fragments. A step of layer 2 feeds layer 3 at once, so only
// layer 1's activations (32 registers) are held. The weights' B fragments come from
// shared memory by ldmatrix and serve both row tiles.
//
// No barrier follows the loading of the weights, and nothing waits but for operands: with
// tcgen05.mma, four CTAs of 128 rows an SM (their tensor memory) met at two barriers and a
// completion wait for each layer, and 2,097,152 particles on 128^3 took 172 us. Here 158
// with features from rho, 136 (and 2.7 for the table) with the cells' features made once
// and the biases as the products' first addend. What bounds it now are the products on
// this path (with 64 of a tile's 104 left out 86 us), then the 128 tanh a particle (58 us
// of the special-function unit); 4 to 6 CTAs an SM measure the same, and loading a tile's
// features beside the last one's layers gains nothing.
//
// The two hidden layers run on weights and biases scaled by 1/2 (exact in BF16 and
// FP32), so each accumulator holds u = z / 2 and SiLU(z) = z sigmoid(z) =
// u + u tanh(u): one tanh and one FMA per unit, rounded to BF16 once.
namespace inf {
constexpr int kThreads = 128, kWarps = kThreads / 32, kCtasPerSm = 5;
constexpr int kS = 72;   // BF16 elements of a 64-wide row: 8 rows of 16 bytes fall in 32 banks
constexpr int kSF = 40;  // of a row of features

struct Smem {
    __nv_bfloat16 w1[kIn][kS], w2[kH][kS], w3[kH][kOut];
    __nv_bfloat16 feat[kWarps][32][kSF];
    float4 b[2 * kH / 2];  // units 2 i, 2 i + 1 of the hidden layers, twice: an accumulator's first addend
    float b3[kOut];
};

// u + u tanh(u) of 16 units of the two row tiles -> one k-step of A fragments
__device__ __forceinline__ void activate(const float (&u)[2][2][4], unsigned (&h)[2][4]) {
#pragma unroll
    for (int q = 0; q < 2; ++q)
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            const float* v = u[mt][q];
            h[mt][2 * q] = pack_bf16(fmaf(v[0], tanh_approx(v[0]), v[0]), fmaf(v[1], tanh_approx(v[1]), v[1]));
            h[mt][2 * q + 1] = pack_bf16(fmaf(v[2], tanh_approx(v[2]), v[2]), fmaf(v[3], tanh_approx(v[3]), v[3]));
        }
}

// acc (two row tiles x 16 units) = bias + A * W[k][16 nc ..]
template <int KS>
__device__ __forceinline__ void layer16(float (&acc)[2][2][4], const unsigned (&a)[KS][2][4],
                                        const __nv_bfloat16* w, const float4* bias, int nc, int lane) {
    const float4 c0 = bias[8 * nc + (lane & 3)], c1 = bias[8 * nc + 4 + (lane & 3)];
#pragma unroll
    for (int s = 0; s < KS; ++s) {
        unsigned b[4];  // {k 0..7, k 8..15} of the two n-tiles
        ldm4t(b, smem_addr(w + (16 * s + (lane & 15)) * kS + 16 * nc + 8 * (lane >> 4)));
#pragma unroll
        for (int mt = 0; mt < 2; ++mt) {
            if (s == 0) {
                mma16816(acc[mt][0], a[s][mt], b[0], b[1], c0);
                mma16816(acc[mt][1], a[s][mt], b[2], b[3], c1);
            } else {
                mma16816(acc[mt][0], a[s][mt], b[0], b[1]);
                mma16816(acc[mt][1], a[s][mt], b[2], b[3]);
            }
        }
    }
}
}  // namespace inf

// TABLE: the density features come from `table` (k_feature_table); otherwise from rho.
template <bool TABLE>
__global__ void __launch_bounds__(inf::kThreads, inf::kCtasPerSm)
    k_mlp_infer(const float* __restrict__ params, const float4* __restrict__ pos, const int* __restrict__ perm, int n,
                const float* __restrict__ rho, const unsigned* __restrict__ table, int G, float inv_mean,
                float out_scale, float4* __restrict__ out) {
    wait_previous();
    __shared__ __align__(16) inf::Smem s;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    // the same BF16 rounding of the weights as the training's copies
    for (int e = tid; e < kIn * kH; e += inf::kThreads)
        s.w1[e / kH][e % kH] = __float2bfloat16_rn(0.5f * params[oW1 + e]);
    for (int e = tid; e < kH * kH; e += inf::kThreads)
        s.w2[e / kH][e % kH] = __float2bfloat16_rn(0.5f * params[oW2 + e]);
    for (int e = tid; e < kH * kOut; e += inf::kThreads) s.w3[e / kOut][e % kOut] = __float2bfloat16_rn(params[oW3 + e]);
    if (tid < kH) {
        const float* b = params + (tid < kH / 2 ? oB1 + 2 * tid : oB2 + 2 * tid - kH);
        s.b[tid] = make_float4(0.5f * b[0], 0.5f * b[1], 0.5f * b[0], 0.5f * b[1]);
    }
    if (tid < kOut) s.b3[tid] = params[oB3 + tid];
    __syncthreads();

    const int tiles = (n + 31) / 32, stride = gridDim.x * inf::kWarps;
    const float4 none = make_float4(-1.f, -1.f, -1.f, 0.f);
    // the next tile's particle and the index of the one after are on their way while a
    // tile runs
    auto index_at = [&](int tile) {
        const long long i = (long long)tile * 32 + lane;
        return i < n ? (perm ? perm[i] : (int)i) : -1;
    };
    int tile = blockIdx.x * inf::kWarps + w;
    int j = tile < tiles ? index_at(tile) : -1;
    float4 p = j >= 0 ? pos[j] : none;
    j = tile + stride < tiles ? index_at(tile + stride) : -1;
    float4 pn = j >= 0 ? pos[j] : none;
    for (; tile < tiles; tile += stride) {
        j = (long long)tile + 2ll * stride < tiles ? index_at(tile + 2 * stride) : -1;
        unsigned a[2][2][4];
        {
            uint4* row = reinterpret_cast<uint4*>(&s.feat[w][lane][0]);
            if (p.x < 0.f) {
#pragma unroll
                for (int q = 0; q < 4; ++q) row[q] = make_uint4(0u, 0u, 0u, 0u);
            } else if (TABLE) {
                unsigned f[16];
                table_features(table, G, p, f);
#pragma unroll
                for (int q = 0; q < 4; ++q) row[q] = make_uint4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3]);
            } else {
                float f[32];
                particle_features(rho, G, inv_mean, p, f);
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    row[q] = make_uint4(pack_bf16(f[8 * q], f[8 * q + 1]), pack_bf16(f[8 * q + 2], f[8 * q + 3]),
                                        pack_bf16(f[8 * q + 4], f[8 * q + 5]), pack_bf16(f[8 * q + 6], f[8 * q + 7]));
            }
            __syncwarp();
#pragma unroll
            for (int k = 0; k < 2; ++k)
#pragma unroll
                for (int mt = 0; mt < 2; ++mt)
                    ldm4(a[k][mt], smem_addr(&s.feat[w][16 * mt + (lane & 15)][16 * k + 8 * (lane >> 4)]));
            __syncwarp();
        }
        unsigned h1[4][2][4];
#pragma unroll
        for (int nc = 0; nc < 4; ++nc) {
            float acc[2][2][4];
            inf::layer16<2>(acc, a, &s.w1[0][0], s.b, nc, lane);
            inf::activate(acc, h1[nc]);
        }
        float y[2][4] = {};
#pragma unroll
        for (int nc = 0; nc < 4; ++nc) {
            float acc[2][2][4];
            unsigned h2[2][4];
            inf::layer16<4>(acc, h1, &s.w2[0][0], s.b + kH / 2, nc, lane);
            inf::activate(acc, h2);
            unsigned b0, b1;  // W3 rows 16 nc ..
            asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                         : "=r"(b0), "=r"(b1)
                         : "r"(smem_addr(&s.w3[16 * nc + (lane & 15)][0])));
            mma16816(y[0], h2[0], b0, b1);
            mma16816(y[1], h2[1], b0, b1);
        }
        // outputs 0 and 1 of a row sit in the first lane of its four, 2 in the second
        const unsigned live = __ballot_sync(0xffffffffu, p.x >= 0.f);
        const float b0 = s.b3[0], b1 = s.b3[1], b2 = s.b3[2];
#pragma unroll
        for (int mt = 0; mt < 2; ++mt)
#pragma unroll
            for (int hi = 0; hi < 2; ++hi) {
                const float y2 = __shfl_down_sync(0xffffffffu, y[mt][2 * hi], 1);
                const int r = 16 * mt + 8 * hi + g;
                const long long i = (long long)tile * 32 + r;
                if (t == 0 && i < n)
                    out[i] = ((live >> r) & 1u) ? make_float4((y[mt][2 * hi] + b0) * out_scale,
                                                              (y[mt][2 * hi + 1] + b1) * out_scale,
                                                              (y2 + b2) * out_scale, 0.f)
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        p = pn;
        pn = j >= 0 ? pos[j] : none;
    }
}

// ---- training: one batch's loss and gradients ----------------------------------------
// k_train_tile takes tiles of 128 rows, eight warps of 16 rows each. Forward, loss
// and backward of a warp's rows chain through registers: the accumulators of one
// m16n8k16 product, packed to BF16, are the A fragments of the next, so no
// activation passes through shared memory on the way. What the weight gradients
// contract over the rows (X, h1, h2, dz1, dz2, dy) is also left in shared memory as
// BF16 rows, and after one barrier the warps split the output tiles of
//   dW1 = X^T dz1 (32 x 64), dW2 = h1^T dz2 (64 x 64), dW3 = h2^T dy (64 x 8)
// over the tile's 128 rows, reading both operands with transposing ldmatrix.
// Accumulators live across the CTA's tiles; each CTA then writes one FP32 partial of
// the whole gradient and k_train_reduce adds the partials in CTA order, so the
// result does not depend on timing.
//
// A batch is a few megaflops: the time is the latency of one tile's chain plus the
// launches. One launch per matrix product, bias, activation and column sum (23 a
// batch, products reading 2-byte elements a whole row apart) took 289 us for a batch
// of 16,384 rows with its Adam step; these two kernels and the step take 26 us.
namespace tr {
constexpr int kThreads = 256, kWarps = 8, kRows = 128;
constexpr int kS = 72;   // BF16 elements of a 64-wide row: 144 bytes, so 8 rows of 16 bytes fall in 32 banks
constexpr int kSX = 40;  // of a 32-wide row
constexpr int kPart = kParams + 8;  // floats of one CTA's partial: the gradient and the squared error

struct Smem {
    __nv_bfloat16 w1[kIn][kS], w2[kH][kS], w3[kH][kOut];
    __nv_bfloat16 x[kRows][kSX], h1[kRows][kS], h2[kRows][kS], dz1[kRows][kS], dz2[kRows][kS], dy[kRows][kOut];
    float b[2 * kH + kOut];
    float colsum[kWarps][2 * kH + kOut + 1];
};

// acc (16 x 64) += A (16 x 16 KS, fragments) * W[k][n] (rows of kS elements)
template <int KS>
__device__ __forceinline__ void mul_w(float (&acc)[8][4], const unsigned (&a)[KS][4], const __nv_bfloat16* w,
                                      int lane) {
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            unsigned b[4];  // two n-tiles: {k 0..7, k 8..15} of each
            ldm4t(b, smem_addr(w + (16 * s + (lane & 15)) * kS + 16 * np + 8 * (lane >> 4)));
            mma16816(acc[2 * np], a[s], b[0], b[1]);
            mma16816(acc[2 * np + 1], a[s], b[2], b[3]);
        }
}

// z = acc + bias; h = bf16(SiLU(z)) as the next product's A fragments and as rows of `rows`
__device__ __forceinline__ void activate(float (&z)[8][4], const float* bias, unsigned (&h)[4][4],
                                         __nv_bfloat16 (*rows)[kS], int row, int t) {
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const float b0 = bias[8 * nt + 2 * t], b1 = bias[8 * nt + 2 * t + 1];
        z[nt][0] += b0;
        z[nt][1] += b1;
        z[nt][2] += b0;
        z[nt][3] += b1;
        const unsigned lo = pack_bf16(silu(z[nt][0]), silu(z[nt][1]));
        const unsigned hi = pack_bf16(silu(z[nt][2]), silu(z[nt][3]));
        h[nt >> 1][(nt & 1) * 2] = lo;
        h[nt >> 1][(nt & 1) * 2 + 1] = hi;
        *reinterpret_cast<unsigned*>(&rows[row][8 * nt + 2 * t]) = lo;
        *reinterpret_cast<unsigned*>(&rows[row + 8][8 * nt + 2 * t]) = hi;
    }
}

// dz = bf16(dh * SiLU'(z)): A fragments, rows, and this thread's share of the column sums
__device__ __forceinline__ void back_silu(const float (&dh)[8][4], const float (&z)[8][4], unsigned (&dz)[4][4],
                                          __nv_bfloat16 (*rows)[kS], int row, int t, float (&sum)[8][2]) {
#pragma unroll
    for (int nt = 0; nt < 8; ++nt) {
        const unsigned lo = pack_bf16(dh[nt][0] * silu_grad(z[nt][0]), dh[nt][1] * silu_grad(z[nt][1]));
        const unsigned hi = pack_bf16(dh[nt][2] * silu_grad(z[nt][2]), dh[nt][3] * silu_grad(z[nt][3]));
        dz[nt >> 1][(nt & 1) * 2] = lo;
        dz[nt >> 1][(nt & 1) * 2 + 1] = hi;
        *reinterpret_cast<unsigned*>(&rows[row][8 * nt + 2 * t]) = lo;
        *reinterpret_cast<unsigned*>(&rows[row + 8][8 * nt + 2 * t]) = hi;
        // a BF16 value is the high half of a float
        sum[nt][0] += __uint_as_float(lo << 16) + __uint_as_float(hi << 16);
        sum[nt][1] += __uint_as_float(lo & 0xffff0000u) + __uint_as_float(hi & 0xffff0000u);
    }
}

// A fragment of M^T for 16 rows: elements (m0.., r0..) of a row-major [row][m] matrix
__device__ __forceinline__ uint32_t at_a(const __nv_bfloat16* m, int stride, int r0, int m0, int lane) {
    return smem_addr(m + (r0 + (lane & 7) + 8 * (lane >> 4)) * stride + m0 + 8 * ((lane >> 3) & 1));
}
// B fragments of two n-tiles for 16 rows of a row-major [row][n] matrix
__device__ __forceinline__ uint32_t at_b(const __nv_bfloat16* m, int stride, int r0, int n0, int lane) {
    return smem_addr(m + (r0 + (lane & 15)) * stride + n0 + 8 * (lane >> 4));
}

// 16 x 8 accumulator tile to rows m0.. of a row-major float matrix
__device__ __forceinline__ void put(float* c, int ld, int m0, int n0, const float (&a)[4], int lane) {
    const int g = lane >> 2, t = lane & 3;
    float* q = c + (m0 + g) * ld + n0 + 2 * t;
    q[0] = a[0];
    q[1] = a[1];
    q[8 * ld] = a[2];
    q[8 * ld + 1] = a[3];
}
}  // namespace tr

__global__ void __launch_bounds__(tr::kThreads, 1) k_train_tile(const float* __restrict__ params,
                                                                const __nv_bfloat16* __restrict__ X,
                                                                const float* __restrict__ tgt, int rows,
                                                                float* __restrict__ part) {
    wait_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    tr::Smem& s = *reinterpret_cast<tr::Smem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, g = lane >> 2, t = lane & 3;
    for (int e = tid; e < kIn * kH; e += tr::kThreads) s.w1[e / kH][e % kH] = __float2bfloat16_rn(params[oW1 + e]);
    for (int e = tid; e < kH * kH; e += tr::kThreads) s.w2[e / kH][e % kH] = __float2bfloat16_rn(params[oW2 + e]);
    for (int e = tid; e < kH * kOut; e += tr::kThreads) s.w3[e / kOut][e % kOut] = __float2bfloat16_rn(params[oW3 + e]);
    if (tid < kH) {
        s.b[tid] = params[oB1 + tid];
        s.b[kH + tid] = params[oB2 + tid];
    }
    if (tid < kOut) s.b[2 * kH + tid] = params[oB3 + tid];

    const bool aligned = (reinterpret_cast<uintptr_t>(X) & 15u) == 0;
    float dw1[2][4] = {}, dw2[4][4] = {}, dw3[4] = {};  // this warp's tiles of the weight gradients
    float sum1[8][2] = {}, sum2[8][2] = {}, sum3[2] = {0.f, 0.f}, err = 0.f;
    const int tiles = (rows - 1) / tr::kRows + 1;
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const int r0 = tile * tr::kRows;
        __syncthreads();  // the last tile's rows are used up (first pass: orders the weights with the next barrier)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
            const int e = tid + q * tr::kThreads, r = e >> 2, c = e & 3;
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (r0 + r < rows) {
                const __nv_bfloat16* src = X + (size_t)(r0 + r) * kIn + 8 * c;
                if (aligned) {
                    v = *reinterpret_cast<const uint4*>(src);
                } else {  // features at any 2-byte address
                    const unsigned short* h = reinterpret_cast<const unsigned short*>(src);
                    v = make_uint4(h[0] | (unsigned)h[1] << 16, h[2] | (unsigned)h[3] << 16,
                                   h[4] | (unsigned)h[5] << 16, h[6] | (unsigned)h[7] << 16);
                }
            }
            *reinterpret_cast<uint4*>(&s.x[r][8 * c]) = v;
        }
        __syncthreads();
        const int row = 16 * w + g;  // this thread's rows of the tile: row, row + 8
        if (r0 + 16 * w < rows) {    // rows come in multiples of 16: a warp has all of its 16 or none
            float z1[8][4] = {}, z2[8][4] = {};
            unsigned h[4][4];
            {
                unsigned a[2][4];
                const uint32_t xa = smem_addr(&s.x[16 * w + (lane & 15)][8 * (lane >> 4)]);
                ldm4(a[0], xa);
                ldm4(a[1], xa + 32);
                tr::mul_w<2>(z1, a, &s.w1[0][0], lane);
            }
            tr::activate(z1, s.b, h, s.h1, row, t);
            tr::mul_w<4>(z2, h, &s.w2[0][0], lane);
            tr::activate(z2, s.b + kH, h, s.h2, row, t);
            float y[4] = {};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                unsigned b[4];  // k-steps 2q and 2q + 1
                ldm4t(b, smem_addr(&s.w3[32 * q + lane][0]));
                mma16816(y, h[2 * q], b[0], b[1]);
                mma16816(y, h[2 * q + 1], b[2], b[3]);
            }
            // dY = 2 (Y - T) / (3 rows) on the 3 real outputs
            float d[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int c = 2 * t + (q & 1), r = row + 8 * (q >> 1);
                d[q] = 0.f;
                if (c < 3) {
                    const float diff = y[q] + s.b[2 * kH + c] - tgt[(size_t)(r0 + r) * 3 + c];
                    err += diff * diff;
                    d[q] = 2.f * diff / (3.f * (float)rows);
                }
            }
            const unsigned lo = pack_bf16(d[0], d[1]), hi = pack_bf16(d[2], d[3]);
            *reinterpret_cast<unsigned*>(&s.dy[row][2 * t]) = lo;
            *reinterpret_cast<unsigned*>(&s.dy[row + 8][2 * t]) = hi;
            sum3[0] += __uint_as_float(lo << 16) + __uint_as_float(hi << 16);
            sum3[1] += __uint_as_float(lo & 0xffff0000u) + __uint_as_float(hi & 0xffff0000u);
            // dh2 = dY W3^T: k = the 8 outputs, the upper half of the k-step zero
            float dh[8][4] = {};
            const unsigned ay[4] = {lo, hi, 0u, 0u};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                unsigned b[4];  // units 32 q + 8 j: row n, 8 outputs along k
                ldm4(b, smem_addr(&s.w3[32 * q + lane][0]));
#pragma unroll
                for (int j = 0; j < 4; ++j) mma16816(dh[4 * q + j], ay, b[j], 0u);
            }
            unsigned dz[4][4];
            tr::back_silu(dh, z2, dz, s.dz2, row, t, sum2);
            // dh1 = dz2 W2^T: B[k = unit of layer 2][n = unit of layer 1] = W2[n][k]
            float dg[8][4] = {};
#pragma unroll
            for (int nt = 0; nt < 8; ++nt)
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    unsigned b[4];  // k-steps 2q, 2q + 1
                    ldm4(b, smem_addr(&s.w2[8 * nt + (lane & 7)][32 * q + 8 * (lane >> 3)]));
                    mma16816(dg[nt], dz[2 * q], b[0], b[1]);
                    mma16816(dg[nt], dz[2 * q + 1], b[2], b[3]);
                }
            tr::back_silu(dg, z1, dz, s.dz1, row, t, sum1);
        } else {  // rows past the batch add nothing: their gradients' factors are zero
            for (int e = lane; e < 16 * kH / 2; e += 32) {
                const int r = 16 * w + e / (kH / 2), c = 2 * (e % (kH / 2));
                *reinterpret_cast<unsigned*>(&s.h1[r][c]) = 0u;
                *reinterpret_cast<unsigned*>(&s.h2[r][c]) = 0u;
                *reinterpret_cast<unsigned*>(&s.dz1[r][c]) = 0u;
                *reinterpret_cast<unsigned*>(&s.dz2[r][c]) = 0u;
            }
            for (int e = lane; e < 16 * kOut / 2; e += 32)
                *reinterpret_cast<unsigned*>(&s.dy[16 * w + e / (kOut / 2)][2 * (e % (kOut / 2))]) = 0u;
        }
        __syncthreads();
        const int m2 = 16 * (w >> 1), n2 = 32 * (w & 1);  // dW2: 16 x 32 per warp
        const int m1 = 16 * (w >> 2), n1 = 16 * (w & 3);  // dW1: 16 x 16 per warp
        const int m3 = 16 * (w & 3);                      // dW3: 16 x 8 per warp, 64 rows each
#pragma unroll 2
        for (int k = 0; k < tr::kRows / 16; ++k) {
            unsigned a[4], b[4];
            ldm4t(a, tr::at_a(&s.h1[0][0], tr::kS, 16 * k, m2, lane));
            ldm4t(b, tr::at_b(&s.dz2[0][0], tr::kS, 16 * k, n2, lane));
            mma16816(dw2[0], a, b[0], b[1]);
            mma16816(dw2[1], a, b[2], b[3]);
            ldm4t(b, tr::at_b(&s.dz2[0][0], tr::kS, 16 * k, n2 + 16, lane));
            mma16816(dw2[2], a, b[0], b[1]);
            mma16816(dw2[3], a, b[2], b[3]);
            ldm4t(a, tr::at_a(&s.x[0][0], tr::kSX, 16 * k, m1, lane));
            ldm4t(b, tr::at_b(&s.dz1[0][0], tr::kS, 16 * k, n1, lane));
            mma16816(dw1[0], a, b[0], b[1]);
            mma16816(dw1[1], a, b[2], b[3]);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {  // warps 0..3: the tile's first 64 rows, 4..7: the rest
            const int k = 64 * (w >> 2) + 32 * q;
            unsigned a[4], b[4];
            ldm4t(b, smem_addr(&s.dy[k + lane][0]));
            ldm4t(a, tr::at_a(&s.h2[0][0], tr::kS, k, m3, lane));
            mma16816(dw3, a, b[0], b[1]);
            ldm4t(a, tr::at_a(&s.h2[0][0], tr::kS, k + 16, m3, lane));
            mma16816(dw3, a, b[2], b[3]);
        }
    }

    // the CTA's partial: weight tiles straight from the accumulators; column sums and the
    // squared error over the lanes of a warp, then over the warps
    float* p = part + (size_t)blockIdx.x * tr::kPart;
#pragma unroll
    for (int j = 0; j < 4; ++j) tr::put(p + oW2, kH, 16 * (w >> 1), 32 * (w & 1) + 8 * j, dw2[j], lane);
#pragma unroll
    for (int j = 0; j < 2; ++j) tr::put(p + oW1, kH, 16 * (w >> 2), 16 * (w & 3) + 8 * j, dw1[j], lane);
    auto over_rows = [](float v) {  // lanes that share t hold the same columns
        v += __shfl_xor_sync(0xffffffffu, v, 4);
        v += __shfl_xor_sync(0xffffffffu, v, 8);
        return v + __shfl_xor_sync(0xffffffffu, v, 16);
    };
#pragma unroll
    for (int nt = 0; nt < 8; ++nt)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float a = over_rows(sum1[nt][c]), b = over_rows(sum2[nt][c]);
            if (g == 0) {
                s.colsum[w][8 * nt + 2 * t + c] = a;
                s.colsum[w][kH + 8 * nt + 2 * t + c] = b;
            }
        }
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        const float a = over_rows(sum3[c]);
        if (g == 0) s.colsum[w][2 * kH + 2 * t + c] = a;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) err += __shfl_xor_sync(0xffffffffu, err, o);
    if (lane == 0) s.colsum[w][2 * kH + kOut] = err;
    __syncthreads();  // the last tile's rows are used up: h1's storage takes the upper half of dW3
    float* d3 = reinterpret_cast<float*>(&s.h1[0][0]);
    if (w >= 4) tr::put(d3, kOut, 16 * (w & 3), 0, dw3, lane);
    if (tid <= 2 * kH + kOut) {
        float v = 0.f;
#pragma unroll
        for (int q = 0; q < tr::kWarps; ++q) v += s.colsum[q][tid];
        const int o = tid < kH ? oB1 + tid : (tid < 2 * kH ? oB2 + tid - kH : oB3 + tid - 2 * kH);
        p[o] = v;  // the squared error lands after b3, at kParams
    }
    __syncthreads();
    if (w < 4) {
        float lo[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) lo[q] = dw3[q] + d3[(16 * w + g + 8 * (q >> 1)) * kOut + 2 * t + (q & 1)];
        tr::put(p + oW3, kOut, 16 * w, 0, lo, lane);
    }
}

// grad[i] = sum over the CTAs' partials, in a fixed order: 4 threads take a quarter of
// them each; *sse from the entry after the gradient.
__global__ void __launch_bounds__(256) k_train_reduce(const float* __restrict__ part, int parts,
                                                      float* __restrict__ grad, float* __restrict__ sse) {
    wait_previous();
    __shared__ float red[4][64];
    const int c = threadIdx.x & 63, q = threadIdx.x >> 6, i = blockIdx.x * 64 + c;
    const int per = (parts + 3) / 4, p0 = q * per, p1 = min(parts, p0 + per);
    float v = 0.f;
    if (i <= kParams) {
#pragma unroll 8
        for (int p = p0; p < p1; ++p) v += part[(size_t)p * tr::kPart + i];
    }
    red[q][c] = v;
    __syncthreads();
    if (q == 0 && i <= kParams) {
        v = (red[0][c] + red[1][c]) + (red[2][c] + red[3][c]);
        if (i < kParams) grad[i] = v;
        else *sse = v;
    }
}

__global__ void k_adam(float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ grad, int n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
    wait_previous();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float g = grad[i];
    const float mi = b1 * m[i] + (1.f - b1) * g;
    const float vi = b2 * v[i] + (1.f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
}

}  // namespace

size_t mlp_param_count() { return kParams; }

int launch_mlp_infer(const float* params, const float4* pos, const int* perm, int n, const float* rho, int G,
                     float inv_mean, float out_scale, float4* out, cudaStream_t s, unsigned* table) {
    if (n <= 0) return SD_OK;
    const int tiles = (n + 31) / 32, need = (tiles + inf::kWarps - 1) / inf::kWarps, wave = 148 * inf::kCtasPerSm;
    const int blocks = need < wave ? need : wave;
    if (table) {
        const size_t quads = (size_t)G * G * G / 4;
        launch(k_feature_table, (unsigned)((quads + 255) / 256), 256, 0, s, reinterpret_cast<const float4*>(rho), quads,
               inv_mean, reinterpret_cast<uint2*>(table));
        SD_LAUNCHED(s);
        launch(k_mlp_infer<true>, blocks, inf::kThreads, 0, s, params, pos, perm, n, rho, table, G, inv_mean, out_scale,
               out);
    } else {
        launch(k_mlp_infer<false>, blocks, inf::kThreads, 0, s, params, pos, perm, n, rho, nullptr, G, inv_mean, out_scale,
               out);
    }
    SD_LAUNCHED(s);
    return SD_OK;
}

// CTAs of a training batch: one per tile of 128 rows, at most one per SM (a CTA's
// partial gradient is 27 KB that the reduction reads again).
static int train_ctas(int rows) {
    const int tiles = rows > 0 ? (rows - 1) / tr::kRows + 1 : 1;
    return tiles < 148 ? tiles : 148;
}

}  // namespace sd

using namespace sd;

extern "C" {

int sd_mlp_param_count(void) { return kParams; }

// The inference has no wait that could give up.
int sd_mlp_wait_timeouts(void) { return SD_CUDA(cudaDeviceSynchronize()) ? SD_E_CUDA : 0; }

int sd_mlp_features(const float* pos, const int32_t* perm, int n, const float* rho, int G, float inv_mean,
                    void* features_bf16, void* stream) {
    if (!pos || !rho || !features_bf16 || n < 0 || G < 16 || (G & (G - 1)))
        return fail(SD_E_ARG, "mlp_features: bad arguments");
    if (n == 0) return SD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    launch(k_features, (n + 255) / 256, 256, 0, st, reinterpret_cast<const float4*>(pos), perm, n, rho, G, inv_mean,
           reinterpret_cast<__nv_bfloat16*>(features_bf16));
    SD_LAUNCHED(st);
    return SD_OK;
}

int sd_mlp_infer(const float* params, const float* pos, const int32_t* perm, int n, const float* rho, int G,
                 float inv_mean, float out_scale, float* out, void* stream) {
    if (!params || !pos || !rho || !out || n < 0 || G < 16 || (G & (G - 1)))
        return fail(SD_E_ARG, "mlp_infer: bad arguments");
    return launch_mlp_infer(params, reinterpret_cast<const float4*>(pos), perm, n, rho, G, inv_mean, out_scale,
                            reinterpret_cast<float4*>(out), (cudaStream_t)stream);
}

size_t sd_mlp_train_workspace_bytes(int rows) {
    return align_up(sizeof(float) * tr::kPart * (size_t)train_ctas(rows), 256);
}

// Loss and gradients of one batch: features X (bf16 [rows][32]), targets T
// (fp32 [rows][3]) -> grad (fp32 [kParams]) of the mean squared error over rows
// and the 3 components, and *sse = the sum of squared errors (device float).
// rows must be a multiple of 16.
int sd_mlp_loss_grad(const float* params, const void* features_bf16, const float* targets, int rows, float* grad,
                     float* sse, void* ws, size_t ws_bytes, void* stream) {
    if (!params || !features_bf16 || !targets || !grad || !sse || !ws || rows <= 0 || rows % 16)
        return fail(SD_E_ARG, "mlp_loss_grad: bad arguments (rows must be a positive multiple of 16)");
    if (ws_bytes < sd_mlp_train_workspace_bytes(rows)) return fail(SD_E_ARG, "mlp_loss_grad: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    const int ctas = train_ctas(rows);
    float* part = reinterpret_cast<float*>(ws);
    // the shared-memory limit is per device, so it is set on each call (a host-side look-up)
    if (SD_CUDA(cudaFuncSetAttribute(k_train_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(tr::Smem))))
        return SD_E_CUDA;
    launch(k_train_tile, ctas, tr::kThreads, sizeof(tr::Smem), st,
           params, reinterpret_cast<const __nv_bfloat16*>(features_bf16), targets, rows, part);
    SD_LAUNCHED(st);
    launch(k_train_reduce, (kParams + 1 + 63) / 64, 256, 0, st, part, ctas, grad, sse);
    SD_LAUNCHED(st);
    return SD_OK;
}

int sd_mlp_adam(float* params, float* m, float* v, const float* grad, int step, float lr, float beta1, float beta2,
                float eps, void* stream) {
    if (!params || !m || !v || !grad || step < 1) return fail(SD_E_ARG, "mlp_adam: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    const float c1 = 1.f / (1.f - powf(beta1, (float)step)), c2 = 1.f / (1.f - powf(beta2, (float)step));
    launch(k_adam, (kParams + 255) / 256, 256, 0, st, params, m, v, grad, kParams, lr, beta1, beta2, eps, c1, c2);
    SD_LAUNCHED(st);
    return SD_OK;
}

}  // extern "C"
