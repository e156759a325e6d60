// sd_mlp.cu -- learned sub-grid force correction: features, BF16 tensor-core
// MLP (30 -> 64 -> 64 -> 3, SiLU), its training kernels and the fused inference
// that feeds the kick. No counterpart in the reference; the correction is added
// on top of the plain PM acceleration (kIntegrate's accG sample, Sim.cu:822).
//
// Numerics: weights and activations are BF16, every matrix product accumulates
// in FP32 on the tensor cores (the inference with tcgen05.mma into tensor memory,
// the training's GEMMs with mma.sync m16n8k16), biases and the SiLU are FP32,
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
__device__ __forceinline__ float cell_feature(float r, float inv_mean) {
    return __logf(1.f + r * inv_mean) - 0.69314718055994531f;
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

__global__ void k_features(const float4* __restrict__ pos, const int* __restrict__ perm, int n,
                           const float* __restrict__ rho, int G, float inv_mean, __nv_bfloat16* __restrict__ out) {
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

// ---- fused inference on the 5th-generation tensor cores (tcgen05) -------------------
// One CTA of 128 threads takes tiles of 128 particles, thread r <-> row r of the
// tile <-> tensor-memory lane r. Each layer is one tcgen05.mma chain (M = 128,
// N = 64 or 16, K in steps of 16, BF16 x BF16 -> FP32) issued by thread 0: the
// activations (operand A) sit in tensor memory, the weights (operand B) in
// shared memory, the FP32 accumulator in 64 tensor-memory columns. Completion
// arrives on an mbarrier (tcgen05.commit); every thread reads its row back with
// tcgen05.ld, adds the bias, applies the SiLU and writes its row of the next
// layer's A with tcgen05.st -- no shared-memory round trip for the activations.
//
// A: row r in lane r, element k in column kAcol + k / 2 (two BF16 per 32-bit
// column, k even in the low half); k-step s reads columns kAcol + 8 s.
// B: the canonical K-major layout without swizzle, 8 x 16-byte core matrices
// (8 rows x 8 BF16): element (row n, k) of a matrix with K columns at byte
// (n / 8) * SBO + (k / 8) * 128 + (n % 8) * 16 + (k % 8) * 2, SBO = K * 16; the
// descriptor of k-step s starts 256 s bytes in (leading offset 128 bytes: the two
// 8-column halves of the step).
//
// Measured against the mma.sync kernel it replaced (2,097,152 particles on 128^3,
// identical outputs): 0.165 against 0.153 ms. The tensor pipe is 8 % busy; the
// kernel waits on the feature gathers from L2 and on the SiLU's dependent chains
// at four CTAs per SM (the tensor-memory columns), not on the products.
namespace tc {
constexpr int kThreads = 128;                  // one warpgroup: TMEM lanes 0..127
constexpr int kTmemCols = 128;                 // FP32 accumulator (columns 0..63) + BF16 operand A (64..95)
constexpr int kAcol = 64;                      // A: row r in lane r, BF16 pairs along K in consecutive columns
constexpr int kN3 = 16;                        // output layer N (3 outputs padded)
constexpr int kB1 = 0;                         // W1^T [64][32]
constexpr int kB2 = kB1 + kH * kIn * 2;        // W2^T [64][64]
constexpr int kB3 = kB2 + kH * kH * 2;         // W3^T [16][64] (rows 8..15 zero)
constexpr int kBias = kB3 + kN3 * kH * 2;      // b1[64], b2[64], b3[8] (float)
constexpr int kBar = kBias + (2 * kH + kOut) * 4 + 8;  // mbarrier (8-byte aligned)
constexpr int kTaddr = kBar + 8;
constexpr int kSmem = kTaddr + 8;
constexpr int kSmemLaunch = 46 * 1024;  // at most four CTAs per SM (see launch_mlp_infer)
static_assert(kBar % 8 == 0 && kB2 % 16 == 0 && kB3 % 16 == 0, "alignment");

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// byte offset of element (r, k) in a K-major shared-memory operand with K columns
__device__ __forceinline__ int op_off(int r, int k, int K) { return (r >> 3) * (K * 16) + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2; }

__device__ __forceinline__ uint64_t desc(uint32_t addr, int K) {
    const uint64_t lbo = 128 >> 4, sbo = (uint64_t)(K * 16) >> 4;
    return (uint64_t)((addr >> 4) & 0x3FFF) | (lbo << 16) | (sbo << 32) | (1ull << 46);  // version 1, no swizzle
}

// instruction descriptor: BF16 x BF16 -> FP32, both K-major, M = 128
__host__ __device__ constexpr uint32_t idesc(int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

// A from tensor memory (the activations), B from shared memory (the weights)
__device__ __forceinline__ void mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b, uint32_t id, uint32_t acc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}\n" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b), "r"(id), "r"(acc));
}

// 16 32-bit words into columns [col, col + 16) of this thread's TMEM lane
__device__ __forceinline__ void st16(uint32_t taddr, const unsigned (&w)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};\n" ::"r"(
            taddr),
        "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7]), "r"(w[8]), "r"(w[9]),
        "r"(w[10]), "r"(w[11]), "r"(w[12]), "r"(w[13]), "r"(w[14]), "r"(w[15])
        : "memory");
}
__device__ __forceinline__ void wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

__device__ __forceinline__ void commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
                 : "memory");
}

__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_proxy() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// Bounded wait for phase `parity` of the mbarrier; false if it gave up.
__device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity) {
    for (int it = 0; it < (1 << 22); ++it) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred q;\n\tmbarrier.try_wait.parity.shared::cta.b64 q, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    return false;
}

// FP32 columns [col, col + 16 X) of this thread's TMEM lane: X loads of 16 columns
// in flight together, one wait
__device__ __forceinline__ void ld16_issue(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
}
template <int X>
__device__ __forceinline__ void ld_cols(uint32_t taddr, float (&v)[16 * X]) {
    uint32_t r[X][16];
#pragma unroll
    for (int x = 0; x < X; ++x) ld16_issue(taddr + 16 * x, r[x]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int x = 0; x < X; ++x)
#pragma unroll
        for (int q = 0; q < 16; ++q) v[16 * x + q] = __uint_as_float(r[x][q]);
}
}  // namespace tc

// Waits that gave up (an mbarrier phase that never completed): the tile's outputs
// are NaN and the count is readable through sd_mlp_wait_timeouts.
__device__ unsigned g_mlp_wait_timeouts = 0;

// The two hidden layers run on weights and biases scaled by 1/2 (exact in BF16 and
// FP32), so each accumulator holds u = z / 2 and SiLU(z) = z sigmoid(z) =
// u + u tanh(u): one tanh and one FMA per unit, rounded to BF16 once.
__global__ void __launch_bounds__(tc::kThreads, 4) k_mlp_infer_tc(const float* __restrict__ params,
                                                              const float4* __restrict__ pos,
                                                              const int* __restrict__ perm, int n,
                                                              const float* __restrict__ rho, int G,
                                                              float inv_mean, float out_scale,
                                                              float4* __restrict__ out) {
    extern __shared__ __align__(1024) unsigned char sm[];
    const int r = threadIdx.x, warp = r >> 5;
    float* bias = reinterpret_cast<float*>(sm + tc::kBias);
    const uint32_t bar = tc::smem_u32(sm + tc::kBar);
    uint32_t* taddr_s = reinterpret_cast<uint32_t*>(sm + tc::kTaddr);
    // weights as K-major operands (W[k][n] -> row n, column k), the same BF16 rounding
    // as the training's copies
    for (int e = r; e < kH * kIn; e += tc::kThreads) {
        const int nn = e / kIn, k = e % kIn;
        *reinterpret_cast<__nv_bfloat16*>(sm + tc::kB1 + tc::op_off(nn, k, kIn)) =
            __float2bfloat16_rn(0.5f * params[oW1 + k * kH + nn]);
    }
    for (int e = r; e < kH * kH; e += tc::kThreads) {
        const int nn = e / kH, k = e % kH;
        *reinterpret_cast<__nv_bfloat16*>(sm + tc::kB2 + tc::op_off(nn, k, kH)) =
            __float2bfloat16_rn(0.5f * params[oW2 + k * kH + nn]);
    }
    for (int e = r; e < tc::kN3 * kH; e += tc::kThreads) {
        const int nn = e / kH, k = e % kH;
        *reinterpret_cast<__nv_bfloat16*>(sm + tc::kB3 + tc::op_off(nn, k, kH)) =
            __float2bfloat16_rn(nn < kOut ? params[oW3 + k * kOut + nn] : 0.f);
    }
    for (int e = r; e < kH; e += tc::kThreads) {
        bias[e] = 0.5f * params[oB1 + e];
        bias[kH + e] = 0.5f * params[oB2 + e];
    }
    if (r < kOut) bias[2 * kH + r] = params[oB3 + r];
    if (r == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(taddr_s)),
                     "r"(tc::kTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc::fence_proxy();  // the weights, written by the threads, are read by the tensor cores
    tc::fence_before();
    __syncthreads();
    tc::fence_after();
    const uint32_t tmem = *taddr_s;
    const uint32_t lane_addr = tmem + ((uint32_t)(warp * 32) << 16);  // this warp's 32 lanes
    const uint32_t a_lane = lane_addr + tc::kAcol;  // this thread's row of the operand A
    const uint32_t b1 = tc::smem_u32(sm + tc::kB1), b2 = tc::smem_u32(sm + tc::kB2),
                   b3 = tc::smem_u32(sm + tc::kB3);
    uint32_t phase = 0;
    bool ok = true;
    const int tiles = (n + tc::kThreads - 1) / tc::kThreads;
    // this thread's particle of the CTA's next tile, loaded while the current tile
    // runs through the network
    float4 pn = make_float4(-1.f, -1.f, -1.f, 0.f);
    if (blockIdx.x * tc::kThreads + r < n) {
        const int i0 = blockIdx.x * tc::kThreads + r;
        pn = pos[perm ? perm[i0] : i0];
    }
    for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x) {
        const int i = t * tc::kThreads + r;
        const float4 p = pn;
        {
            const int inx = i + gridDim.x * tc::kThreads;
            pn = make_float4(-1.f, -1.f, -1.f, 0.f);
            if (inx < n) pn = pos[perm ? perm[inx] : inx];
        }
        {
            unsigned w[16];
            if (p.x < 0.f) {
#pragma unroll
                for (int j = 0; j < 16; ++j) w[j] = 0u;
            } else {
                float f[32];
                particle_features(rho, G, inv_mean, p, f);
#pragma unroll
                for (int j = 0; j < 16; ++j) w[j] = pack_bf16(f[2 * j], f[2 * j + 1]);
            }
            tc::st16(a_lane, w);
            tc::wait_st();
        }
        // three layers; layer l reads A (K = 32 for the first, 64 after) and B_l
#pragma unroll 1
        for (int layer = 0; layer < 3; ++layer) {
            const int K = layer == 0 ? kIn : kH;
            tc::fence_before();  // this thread's operand row (tcgen05.st, waited) before the MMA
            __syncthreads();
            if (r == 0) {
                tc::fence_after();
                const uint32_t bb = layer == 0 ? b1 : (layer == 1 ? b2 : b3);
                const uint32_t id = tc::idesc(layer == 2 ? tc::kN3 : kH);
                // k-step s: A columns kAcol + 8 s (16 BF16 per row), B rows from byte 256 s
                for (int s = 0; s < K / 16; ++s)
                    tc::mma_ts(tmem, tmem + tc::kAcol + 8 * s, tc::desc(bb + 256 * s, K), id, s > 0);
                tc::commit(bar);
            }
            // every thread waits; the verdict is made uniform so the CTA's barriers stay matched
            if (!__syncthreads_and(tc::wait_bar(bar, phase))) {
                ok = false;
                if (r == 0) atomicAdd(&g_mlp_wait_timeouts, 1u);
                break;
            }
            phase ^= 1;
            tc::fence_after();
            if (layer < 2) {
                // this row's 64 pre-activations -> SiLU -> the next layer's operand row
                // (the MMA that read A has completed)
#pragma unroll
                for (int c2 = 0; c2 < kH / 32; ++c2) {
                    float v[32];
                    tc::ld_cols<2>(lane_addr + 32 * c2, v);
                    const float* b = bias + layer * kH + 32 * c2;
                    unsigned h[16];
#pragma unroll
                    for (int q = 0; q < 16; ++q) {
                        const float u0 = v[2 * q] + b[2 * q], u1 = v[2 * q + 1] + b[2 * q + 1];
                        h[q] = pack_bf16(fmaf(u0, tanh_approx(u0), u0), fmaf(u1, tanh_approx(u1), u1));
                    }
                    tc::st16(a_lane + 16 * c2, h);  // units 32 c2 .. 32 c2 + 31
                }
                tc::wait_st();
            } else {
                float v[16];
                tc::ld_cols<1>(lane_addr, v);
                const float* b = bias + 2 * kH;
                if (i < n)
                    out[i] = (p.x >= 0.f) ? make_float4((v[0] + b[0]) * out_scale, (v[1] + b[1]) * out_scale,
                                                        (v[2] + b[2]) * out_scale, 0.f)
                                          : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        if (!ok && i < n) out[i] = make_float4(__int_as_float(0x7fc00000), __int_as_float(0x7fc00000),
                                               __int_as_float(0x7fc00000), 0.f);
    }
    // every tcgen05.ld has completed (wait::ld) and no MMA is in flight once the
    // last wait returned; a CTA whose wait gave up drains with a second bounded wait
    if (!ok && r == 0) tc::wait_bar(bar, phase);
    tc::fence_before();
    __syncthreads();
    if (warp == 0) {
        tc::fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(tc::kTmemCols)
                     : "memory");
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

__device__ __forceinline__ uint32_t addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
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

// acc (16 x 64) += A (16 x 16 KS, fragments) * W[k][n] (rows of kS elements)
template <int KS>
__device__ __forceinline__ void mul_w(float (&acc)[8][4], const unsigned (&a)[KS][4], const __nv_bfloat16* w,
                                      int lane) {
#pragma unroll
    for (int s = 0; s < KS; ++s)
#pragma unroll
        for (int np = 0; np < 4; ++np) {
            unsigned b[4];  // two n-tiles: {k 0..7, k 8..15} of each
            ldm4t(b, addr(w + (16 * s + (lane & 15)) * kS + 16 * np + 8 * (lane >> 4)));
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
    return addr(m + (r0 + (lane & 7) + 8 * (lane >> 4)) * stride + m0 + 8 * ((lane >> 3) & 1));
}
// B fragments of two n-tiles for 16 rows of a row-major [row][n] matrix
__device__ __forceinline__ uint32_t at_b(const __nv_bfloat16* m, int stride, int r0, int n0, int lane) {
    return addr(m + (r0 + (lane & 15)) * stride + n0 + 8 * (lane >> 4));
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
                const uint32_t xa = tr::addr(&s.x[16 * w + (lane & 15)][8 * (lane >> 4)]);
                tr::ldm4(a[0], xa);
                tr::ldm4(a[1], xa + 32);
                tr::mul_w<2>(z1, a, &s.w1[0][0], lane);
            }
            tr::activate(z1, s.b, h, s.h1, row, t);
            tr::mul_w<4>(z2, h, &s.w2[0][0], lane);
            tr::activate(z2, s.b + kH, h, s.h2, row, t);
            float y[4] = {};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                unsigned b[4];  // k-steps 2q and 2q + 1
                tr::ldm4t(b, tr::addr(&s.w3[32 * q + lane][0]));
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
                tr::ldm4(b, tr::addr(&s.w3[32 * q + lane][0]));
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
                    tr::ldm4(b, tr::addr(&s.w2[8 * nt + (lane & 7)][32 * q + 8 * (lane >> 3)]));
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
            tr::ldm4t(a, tr::at_a(&s.h1[0][0], tr::kS, 16 * k, m2, lane));
            tr::ldm4t(b, tr::at_b(&s.dz2[0][0], tr::kS, 16 * k, n2, lane));
            mma16816(dw2[0], a, b[0], b[1]);
            mma16816(dw2[1], a, b[2], b[3]);
            tr::ldm4t(b, tr::at_b(&s.dz2[0][0], tr::kS, 16 * k, n2 + 16, lane));
            mma16816(dw2[2], a, b[0], b[1]);
            mma16816(dw2[3], a, b[2], b[3]);
            tr::ldm4t(a, tr::at_a(&s.x[0][0], tr::kSX, 16 * k, m1, lane));
            tr::ldm4t(b, tr::at_b(&s.dz1[0][0], tr::kS, 16 * k, n1, lane));
            mma16816(dw1[0], a, b[0], b[1]);
            mma16816(dw1[1], a, b[2], b[3]);
        }
#pragma unroll
        for (int q = 0; q < 2; ++q) {  // warps 0..3: the tile's first 64 rows, 4..7: the rest
            const int k = 64 * (w >> 2) + 32 * q;
            unsigned a[4], b[4];
            tr::ldm4t(b, tr::addr(&s.dy[k + lane][0]));
            tr::ldm4t(a, tr::at_a(&s.h2[0][0], tr::kS, k, m3, lane));
            mma16816(dw3, a, b[0], b[1]);
            tr::ldm4t(a, tr::at_a(&s.h2[0][0], tr::kS, k + 16, m3, lane));
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

__global__ void k_adam(
float* __restrict__ p, float* __restrict__ m, float* __restrict__ v,
                       const float* __restrict__ grad, int n, float lr, float b1, float b2, float eps, float c1,
                       float c2) {
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
                     float inv_mean, float out_scale, float4* out, cudaStream_t s) {
    if (n <= 0) return SD_OK;
    // tiles of 128 particles; four CTAs fill an SM's 512 tensor-memory columns (128 each).
    // The dynamic shared memory is padded so that no fifth CTA is placed on an SM, where
    // its tcgen05.alloc would wait for one of the four to finish.
    static_assert(tc::kSmemLaunch >= tc::kSmem && 5 * (tc::kSmemLaunch + 1024) > 228 * 1024, "four CTAs per SM");
    const int tiles = (n + tc::kThreads - 1) / tc::kThreads;
    const int blocks = tiles < 148 * 4 ? tiles : 148 * 4;
    k_mlp_infer_tc<<<blocks, tc::kThreads, tc::kSmemLaunch, s>>>(params, pos, perm, n, rho, G, inv_mean, out_scale,
                                                                 out);
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

int sd_mlp_wait_timeouts(void) {
    unsigned v = 0;
    if (SD_CUDA(cudaMemcpyFromSymbol(&v, g_mlp_wait_timeouts, sizeof(v)))) return SD_E_CUDA;
    return (int)v;
}

int sd_mlp_features(const float* pos, const int32_t* perm, int n, const float* rho, int G, float inv_mean,
                    void* features_bf16, void* stream) {
    if (!pos || !rho || !features_bf16 || n < 0 || G < 16 || (G & (G - 1)))
        return fail(SD_E_ARG, "mlp_features: bad arguments");
    if (n == 0) return SD_OK;
    cudaStream_t st = (cudaStream_t)stream;
    k_features<<<(n + 255) / 256, 256, 0, st>>>(reinterpret_cast<const float4*>(pos), perm, n, rho, G, inv_mean,
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
    k_train_tile<<<ctas, tr::kThreads, sizeof(tr::Smem), st>>>(
        params, reinterpret_cast<const __nv_bfloat16*>(features_bf16), targets, rows, part);
    SD_LAUNCHED(st);
    k_train_reduce<<<(kParams + 1 + 63) / 64, 256, 0, st>>>(part, ctas, grad, sse);
    SD_LAUNCHED(st);
    return SD_OK;
}

int sd_mlp_adam(float* params, float* m, float* v, const float* grad, int step, float lr, float beta1, float beta2,
                float eps, void* stream) {
    if (!params || !m || !v || !grad || step < 1) return fail(SD_E_ARG, "mlp_adam: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    const float c1 = 1.f / (1.f - powf(beta1, (float)step)), c2 = 1.f / (1.f - powf(beta2, (float)step));
    k_adam<<<(kParams + 255) / 256, 256, 0, st>>>(params, m, v, grad, kParams, lr, beta1, beta2, eps, c1, c2);
    SD_LAUNCHED(st);
    return SD_OK;
}

}  // extern "C"
