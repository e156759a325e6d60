// sd_common.cuh -- device helpers shared by the PM kernels (sm_100a).
//
// The CIC arithmetic below is written with explicit __fmaf_rn / __fmul_rn so the
// result of each expression is fixed by the source: the CPU oracle in oracle/
// uses the same forms with fmaf(), which is what makes keys, the fixed-point
// density and the kick bit-comparable between the two.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#define SD_FIXED_ONE 4294967296.0f           // 2^32: fixed-point scale of one deposit weight
#define SD_FIXED_INV 2.3283064365386963e-10f  // 2^-32

namespace sd {

// First statement of every kernel that launch() (sd_internal.h) starts: waits until the
// kernels before it in the stream are done and their writes can be seen. None of them
// lets the next one start early, so all of their blocks have left by then.
__device__ __forceinline__ void wait_previous() { cudaGridDependencySynchronize(); }

// CIC base cell and fraction along one axis: g = p*G - 1/2 (kScatter, Sim.cu:509-511).
__device__ __forceinline__ void cic_axis(float p, int G, int& i, float& f) {
    const float g = __fmaf_rn(p, (float)G, -0.5f);
    const float fl = floorf(g);
    i = __float2int_rz(fl);  // saturates
    f = __fsub_rn(g, fl);
}

// Containing cell along one axis, clamped (kCellKey, Sim.cu:2482-2485).
__device__ __forceinline__ int cell_axis(float p, int G) {
    return min(max(__float2int_rz(__fmul_rn(p, (float)G)), 0), G - 1);
}

// Cell index of a CIC corner: wrapped (periodic) or clamped to the edge cell
// (isolated; gidx3, Sim.cu:96-100 -- weights past the edge land on it).
__device__ __forceinline__ int cic_cell(int i, int G, bool periodic) {
    return periodic ? (i & (G - 1)) : min(max(i, 0), G - 1);
}

// Cell of corner o (0 or 1) of a stencil at base i. The sum is one of unsigned values: the
// base of a coordinate beyond 2^31 cells is 2^31 - 1, and where the compiler may take a sum
// not to overflow it clamps before it adds, and a corner of such a particle, or of one
// at infinity, lies outside the box's memory.
__device__ __forceinline__ int cic_corner(int i, int o, int G, bool periodic) {
    return cic_cell((int)((unsigned)i + (unsigned)o), G, periodic);
}

// Weight of corner k = ox | oy<<1 | oz<<2, as (wx*wy)*wz (Sim.cu:515).
__device__ __forceinline__ float cic_weight(int k, float fx, float fy, float fz) {
    const float wx = (k & 1) ? fx : __fsub_rn(1.f, fx);
    const float wy = (k & 2) ? fy : __fsub_rn(1.f, fy);
    const float wz = (k & 4) ? fz : __fsub_rn(1.f, fz);
    return __fmul_rn(__fmul_rn(wx, wy), wz);
}

__device__ __forceinline__ long long fixed_weight(float w) {
    return __float2ll_rn(__fmul_rn(w, SD_FIXED_ONE));
}

__device__ __forceinline__ float fixed_to_float(long long s) {
    return __fmul_rn(__ll2float_rn(s), SD_FIXED_INV);
}

// The 8 corners of one particle into an int64 fixed-point grid of side G.
__device__ __forceinline__ void deposit_particle(float4 p, int G, unsigned long long* __restrict__ acc, bool periodic) {
    if (p.x < 0.f) return;
    int ix, iy, iz;
    float fx, fy, fz;
    cic_axis(p.x, G, ix, fx);
    cic_axis(p.y, G, iy, fy);
    cic_axis(p.z, G, iz, fz);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int cx = cic_corner(ix, k & 1, G, periodic);
        const int cy = cic_corner(iy, (k >> 1) & 1, G, periodic);
        const int cz = cic_corner(iz, (k >> 2) & 1, G, periodic);
        const long long q = fixed_weight(cic_weight(k, fx, fy, fz));
        atomicAdd(acc + ((size_t)cz * G + cy) * G + cx, (unsigned long long)q);
    }
}

__device__ __forceinline__ uint32_t part1by2(uint32_t v) {
    v &= 0x3ffu;
    v = (v | (v << 16)) & 0x030000ffu;
    v = (v | (v << 8)) & 0x0300f00fu;
    v = (v | (v << 4)) & 0x030c30c3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// Order keys (see sd_cell_keys in stardust_pm.h). Row-major and Morton: key + 1,
// 0 = empty slot. Tiled: the row index itself (G^2 values, log2(G^2) bits), with
// empty slots sharing row 0 (the fused deposit skips them).
__device__ __forceinline__ uint32_t order_key(float4 p, int G, int order) {
    if (p.x < 0.f) return 0u;
    if (order == 2) {  // tile rows of the CIC base cell
        int iy, iz; float f;
        cic_axis(p.y, G, iy, f);
        cic_axis(p.z, G, iz, f);
        iy &= (G - 1); iz &= (G - 1);
        const int tiles = G >> 2;
        const int tile = (iz >> 2) * tiles + (iy >> 2);
        return (uint32_t)(tile * 16 + (iz & 3) * 4 + (iy & 3));
    }
    const int cx = cell_axis(p.x, G), cy = cell_axis(p.y, G), cz = cell_axis(p.z, G);
    if (order == 1)
        return (part1by2((uint32_t)cx) | (part1by2((uint32_t)cy) << 1) | (part1by2((uint32_t)cz) << 2)) + 1u;
    return (uint32_t)((cz * G + cy) * G + cx) + 1u;
}

// Row table of sorted keys: entry r is the first position whose key is at least
// row_low(r, shift). Tiled keys are rows themselves (shift < 0; entries 0..G^2).
// Row-major and Morton keys hold 2^shift = G cells of a row (or of a run of the
// Morton curve) next to each other: entry 0 is the empty slots (key 0), entry r + 1
// starts row r (entries 0..G^2 + 1). row_of is the last entry whose low key is not
// above a key.
__host__ __device__ __forceinline__ uint32_t row_low(int r, int shift) {
    return shift < 0 ? (uint32_t)r : (r ? ((uint32_t)(r - 1) << shift) + 1u : 0u);
}
__host__ __device__ __forceinline__ uint32_t row_of(uint32_t key, int shift) {
    return shift < 0 ? key : (key ? ((key - 1u) >> shift) + 1u : 0u);
}

// Whether the fused deposit would not add a live particle as k_deposit_fixed does (see
// k_deposit_plan): along y or z its stencil's base row is not where its key's row says
// (positions outside the box), or along any axis its weight is no number, which
// two 32-bit sums do not hold. The periodic tiled order leaves such weights out.
__device__ __forceinline__ bool stray_axis(float p, int G, int order, bool periodic, bool row) {
    int i;
    float f;
    cic_axis(p, G, i, f);
    if (order == 1 || (order == 2 && periodic)) return false;
    if (f != f) return true;
    if (!row || (order == 0 && !periodic)) return false;
    if (order == 2) return i < -1 || i >= G;
    const int c = cell_axis(p, G);
    return i != c && i != c - 1;
}
__device__ __forceinline__ bool stray_particle(float4 p, int G, int order, bool periodic) {
    return !(p.x < 0.f) && (stray_axis(p.x, G, order, periodic, false) || stray_axis(p.y, G, order, periodic, true) ||
                            stray_axis(p.z, G, order, periodic, true));
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

}  // namespace sd
