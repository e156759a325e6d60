// sd_fft.cuh -- shared-memory Stockham FFT over 16 interleaved lines (sm_100a).
//
// A CTA holds 16 lines of N complex values in shared memory, interleaved:
// element i of line l sits at s[at(i, l)], in row i, of 16 float2. All 16 lines are
// transformed at once. Threads are mapped line-fastest (item u -> line u & 15, butterfly
// u >> 4), so every load and store of every stage touches two rows of 16 consecutive
// float2 per warp: the two-wavefront minimum for 8-byte accesses, with no padding and no
// bank conflicts.
//
// Stages are mixed radix (32 or 16 where every thread still gets a butterfly,
// else 8, then 4 or 2 for the remainder) in the self-sorting
// Stockham form: the stage with radix R and sub-transform length Ns reads
// in[j + r*N/R], multiplies by W_{Ns*R}^{(j mod Ns)*r}, does an R-point DFT in
// registers and writes out[(j/Ns)*Ns*R + (j mod Ns) + r*Ns]. Output is in
// natural order. Each stage loads all its butterflies into registers,
// synchronises and stores back in place.
//
// Twiddles come from a table tw[m] = exp(-2 pi i m / M) of length M = N * TWS
// (TWS = table stride); the inverse uses conjugates. Transforms are unnormalised.
#pragma once

#include <cuda_runtime.h>

namespace sd {
namespace fft {

// Element `pos` of line l. TURN: the lines of a row are turned by 4 (pos mod 4). Passes B and
// D copy whole bricks in which 8 lanes take 16 bytes of four rows each: a 4-way bank
// conflict where rows are not turned (512^3 207 and 209 us, turned 201 and 207; 256^3
// 27.3 and 24.2). The others' copies have none (C) or small ones, and only pay for the turn
// (isolated C 25.9 -> 27.2, E at 256 33.2 -> 34.1).
template <bool TURN = false>
__device__ __forceinline__ int at(int pos, int l) {
    return pos * 16 + (TURN ? l ^ ((pos & 3) << 2) : l);
}

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 conjf2(float2 a) { return make_float2(a.x, -a.y); }
// a - i b (forward) or a + i b (inverse)
template <bool INV>
__device__ __forceinline__ float2 add_mi(float2 a, float2 b) {
    return INV ? make_float2(a.x - b.y, a.y + b.x) : make_float2(a.x + b.y, a.y - b.x);
}

// a + b, a - b and a + c b. PAIR: both halves in one instruction, each rounded as a
// scalar's.
template <bool PAIR>
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    if (!PAIR) return cadd(a, b);
    float2 r;
    asm("{ .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x; }"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
template <bool PAIR>
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
    if (!PAIR) return csub(a, b);
    float2 r;
    asm("{ .reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n sub.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x; }"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
template <bool PAIR>
__device__ __forceinline__ float2 fma2(float c, float2 b, float2 a) {
    if (!PAIR) return make_float2(fmaf(c, b.x, a.x), fmaf(c, b.y, a.y));
    float2 r;
    asm("{ .reg .b64 x, y, z;\n mov.b64 x, {%2, %2};\n mov.b64 y, {%3, %4};\n mov.b64 z, {%5, %6};\n"
        " fma.rn.f32x2 x, x, y, z;\n mov.b64 {%0, %1}, x; }"
        : "=f"(r.x), "=f"(r.y)
        : "f"(c), "f"(b.x), "f"(b.y), "f"(a.x), "f"(a.y));
    return r;
}

// exp(-2 pi i k / 32), 0 < k < 16, k != 8, as c (1 + i t) where the cosine is the larger
// part and as c (t + i) where the sine is (swap). Two fused operations then form
// u = b (1 + i t), and four more a + c u and a - c u, one rounding each: a butterfly is
// 6 instead of 8 instructions. (The inverse's: t changes sign, and c with swap.)
struct Turn {
    float t, c;
    bool swap;
};
namespace w32 {
constexpr double c1 = 0.98078528040323044913, s1 = 0.19509032201612826785;
constexpr double c2 = 0.92387953251128675613, s2 = 0.38268343236508977173;
constexpr double c3 = 0.83146961230254523708, s3 = 0.55557023301960222474;
constexpr double r = 0.70710678118654752440;
__device__ __forceinline__ Turn get(int k) {  // k is a compile-time constant after unrolling
    constexpr float t1 = (float)(s1 / c1), t2 = (float)(s2 / c2), t3 = (float)(s3 / c3);
    constexpr float f1 = (float)c1, f2 = (float)c2, f3 = (float)c3, fr = (float)r;
    switch (k) {
        case 1: return {-t1, f1, false};
        case 2: return {-t2, f2, false};
        case 3: return {-t3, f3, false};
        case 4: return {-1.f, fr, false};
        case 5: return {-t3, -f3, true};
        case 6: return {-t2, -f2, true};
        case 7: return {-t1, -f1, true};
        case 9: return {t1, -f1, true};
        case 10: return {t2, -f2, true};
        case 11: return {t3, -f3, true};
        case 12: return {1.f, -fr, false};
        case 13: return {t3, -f3, false};
        case 14: return {t2, -f2, false};
        default: return {t1, -f1, false};
    }
}
}  // namespace w32

template <int R, bool INV, bool PAIR = false>
__device__ __forceinline__ void dft(float2* v) {
    if constexpr (R == 16 || R == 32) {
        // radix-2 split: DFTs of the even and odd inputs, combined with W_R^k
        constexpr int H = R / 2;
        float2 e[H], o[H];
#pragma unroll
        for (int i = 0; i < H; ++i) {
            e[i] = v[2 * i];
            o[i] = v[2 * i + 1];
        }
        dft<H, INV, PAIR>(e);
        dft<H, INV, PAIR>(o);
        v[0] = add2<PAIR>(e[0], o[0]);
        v[H] = sub2<PAIR>(e[0], o[0]);
#pragma unroll
        for (int k = 1; k < H; ++k) {
            if (k == H / 2) {
                v[k] = add_mi<INV>(e[k], o[k]);
                v[k + H] = add_mi<!INV>(e[k], o[k]);
                continue;
            }
            const Turn w = w32::get(k * (32 / R));
            const float t = INV ? -w.t : w.t, c = INV && w.swap ? -w.c : w.c;
            const float2 u = w.swap ? make_float2(fmaf(t, o[k].x, -o[k].y), fmaf(t, o[k].y, o[k].x))
                                    : make_float2(fmaf(-t, o[k].y, o[k].x), fmaf(t, o[k].x, o[k].y));
            v[k] = fma2<PAIR>(c, u, e[k]);
            v[k + H] = fma2<PAIR>(-c, u, e[k]);
        }
    } else if constexpr (R == 2) {
        const float2 a = v[0], b = v[1];
        v[0] = add2<PAIR>(a, b);
        v[1] = sub2<PAIR>(a, b);
    } else if constexpr (R == 4) {
        const float2 t0 = add2<PAIR>(v[0], v[2]), t1 = sub2<PAIR>(v[0], v[2]);
        const float2 t2 = add2<PAIR>(v[1], v[3]), t3 = sub2<PAIR>(v[1], v[3]);
        v[0] = add2<PAIR>(t0, t2);
        v[2] = sub2<PAIR>(t0, t2);
        v[1] = add_mi<INV>(t1, t3);
        v[3] = add_mi<!INV>(t1, t3);
    } else {  // R == 8: two 4-point DFTs of the even and odd inputs
        float2 e[4] = {v[0], v[2], v[4], v[6]};
        float2 o[4] = {v[1], v[3], v[5], v[7]};
        dft<4, INV, PAIR>(e);
        dft<4, INV, PAIR>(o);
        constexpr float c = 0.70710678118654752440f;
        // W8^1 = c(1 -/+ i), W8^2 = -/+ i, W8^3 = -c(1 +/- i)
        const float2 o1 = add_mi<INV>(o[1], o[1]), o3 = add_mi<!INV>(o[3], o[3]);
        v[0] = add2<PAIR>(e[0], o[0]);
        v[4] = sub2<PAIR>(e[0], o[0]);
        v[1] = fma2<PAIR>(c, o1, e[1]);
        v[5] = fma2<PAIR>(-c, o1, e[1]);
        v[2] = add_mi<INV>(e[2], o[2]);
        v[6] = add_mi<!INV>(e[2], o[2]);
        v[3] = fma2<PAIR>(-c, o3, e[3]);
        v[7] = fma2<PAIR>(c, o3, e[3]);
    }
}

// Radix of the next stage for a remaining length REM of an N-point transform on
// NT threads: the largest of 32, 16 that divides REM and still gives every thread
// a butterfly (16 N / R >= NT), else 8, 4 or 2. Fewer, wider stages mean fewer
// shared-memory round trips.
template <int REM, int N, int NT>
struct radix_of {
    static constexpr int value = (REM % 32 == 0 && 16 * N / 32 >= NT)   ? 32
                                 : (REM % 16 == 0 && 16 * N / 16 >= NT) ? 16
                                 : (REM % 8 == 0)                       ? 8
                                 : (REM % 4 == 0)                       ? 4
                                                                        : 2;
};

// One Stockham stage on the 16 interleaved lines, then recurse.
// radix_of as a constexpr function, and the sub-transform length Ns of the last
// stage of an N-point transform on NT threads.
constexpr int radix_for(int rem, int N, int NT) {
    return (rem % 32 == 0 && 16 * N / 32 >= NT)   ? 32
           : (rem % 16 == 0 && 16 * N / 16 >= NT) ? 16
           : (rem % 8 == 0)                       ? 8
           : (rem % 4 == 0)                       ? 4
                                                  : 2;
}
constexpr int last_stage_ns(int N, int NT) {
    int ns = 1;
    while (ns * radix_for(N / ns, N, NT) < N) ns *= radix_for(N / ns, N, NT);
    return ns;
}

// Element `pos` of line l as the first stage reads it: plainly, or through a
// caller's functor that forms it from what s holds (a pre-processing step fused
// into the first stage's loads, saving a shared-memory round trip and a barrier).
struct PlainLoad {
    __device__ __forceinline__ float2 operator()(const float2* s, int l, int pos) const { return s[at(pos, l)]; }
};

// Stages from sub-transform length Ns on, stopping before the stage at STOP; the
// stage at Ns = 1 reads through `load`. HALF: positions N/2 and up of the input are
// zero and are not read (they are the upper half of the first stage's radix).
template <int N, int Ns, int NT, int TWS, bool INV, int STOP = N, class Load = PlainLoad, bool HALF = false,
          bool PAIR = false, bool TURN = false>
__device__ __forceinline__ void stages16(float2* s, const float2* tw, Load load = Load()) {
    if constexpr (Ns < N && Ns < STOP) {
        constexpr int R = radix_of<N / Ns, N, NT>::value;
        constexpr int NB = N / R;
        constexpr int TOT = 16 * NB;
        constexpr int PER = (TOT + NT - 1) / NT;
        float2 v[PER][R];
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const int u = threadIdx.x + p * NT;
            if (TOT % NT == 0 || u < TOT) {
                const int l = u & 15, j = u >> 4, k = j % Ns;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    if (HALF && Ns == 1 && r >= R / 2) {
                        v[p][r] = make_float2(0.f, 0.f);
                        continue;
                    }
                    float2 x = (Ns == 1 && !TURN) ? load(s, l, j + r * NB) : s[at<TURN>(j + r * NB, l)];
                    if (Ns > 1 && r > 0) {
                        float2 w = tw[(k * r * (N / (Ns * R))) * TWS];
                        if (INV) w.y = -w.y;
                        x = cmul(x, w);
                    }
                    v[p][r] = x;
                }
            }
        }
        __syncthreads();
#pragma unroll
        for (int p = 0; p < PER; ++p) {
            const int u = threadIdx.x + p * NT;
            if (TOT % NT == 0 || u < TOT) {
                const int l = u & 15, j = u >> 4, k = j % Ns;
                dft<R, INV, PAIR>(v[p]);
                const int base = (j / Ns) * Ns * R + k;
#pragma unroll
                for (int r = 0; r < R; ++r) s[at<TURN>(base + r * Ns, l)] = v[p][r];
            }
        }
        __syncthreads();
        stages16<N, Ns * R, NT, TWS, INV, STOP, PlainLoad, false, PAIR, TURN>(s, tw);
    }
}

// Transform the 16 interleaved lines of length N in s. The caller synchronises
// before the call; the routine ends with a barrier. HALF: the input's upper half is zero.
template <int N, int NT, int TWS, bool INV, bool HALF = false, bool TURN = false>
__device__ __forceinline__ void lines16(float2* s, const float2* tw) {
    stages16<N, 1, NT, TWS, INV, N, PlainLoad, HALF, false, TURN>(s, tw);
}

// Forward transform, a pointwise multiply, inverse transform of the 16 lines.
// The forward's last stage (radix R, sub-length Ns = N / R) leaves, in each
// thread's registers, the outputs at positions j + r Ns -- exactly the inputs of
// an inverse first stage of the same radix. So that stage, the multiply
// mul(line, position, position >= N / 2, value) and the inverse's first stage run in registers with
// no shared-memory round trip or barrier between them; the inverse then goes on
// from sub-length R. The caller synchronises before the call; it ends with a
// barrier. HALF: the input's upper half is zero (N takes at least two stages).
template <int N, int NT, int TWS, bool HALF = false, class Mul>
__device__ __forceinline__ void convolve16(float2* s, const float2* tw, Mul mul) {
    constexpr int NsL = last_stage_ns(N, NT);
    constexpr int R = N / NsL;
    constexpr int NB = N / R;  // == NsL
    constexpr int TOT = 16 * NB;
    constexpr int PER = (TOT + NT - 1) / NT;
    static_assert(!HALF || NsL > 1, "a half-zero input is pruned in a first stage of its own");
    stages16<N, 1, NT, TWS, false, NsL, PlainLoad, HALF, true>(s, tw);
    float2 v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * NT;
        if (TOT % NT == 0 || u < TOT) {
            const int l = u & 15, j = u >> 4;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 x = s[at(j + r * NB, l)];
                if (NsL > 1 && r > 0) x = cmul(x, tw[(j * r) * TWS]);
                v[p][r] = x;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * NT;
        if (TOT % NT == 0 || u < TOT) {
            const int l = u & 15, j = u >> 4;
            dft<R, false, true>(v[p]);
#pragma unroll
            for (int r = 0; r < R; ++r) v[p][r] = mul(l, j + r * NsL, r >= R / 2, v[p][r]);
            dft<R, true, true>(v[p]);
#pragma unroll
            for (int r = 0; r < R; ++r) s[at(j * R + r, l)] = v[p][r];
        }
    }
    __syncthreads();
    stages16<N, R, NT, TWS, true, N, PlainLoad, false, true>(s, tw);
}

// lines16, with the last stage writing its outputs row-major (line l at
// s[l * RS + position]) instead of interleaved, for callers that store rows; the
// first stage reads through `load`.
template <int N, int NT, int TWS, bool INV, int RS, class Load = PlainLoad>
__device__ __forceinline__ void lines16_rows(float2* s, const float2* tw, Load load = Load()) {
    constexpr int NsL = last_stage_ns(N, NT);
    constexpr int R = N / NsL;
    constexpr int NB = N / R;
    constexpr int TOT = 16 * NB;
    constexpr int PER = (TOT + NT - 1) / NT;
    stages16<N, 1, NT, TWS, INV, NsL>(s, tw, load);
    float2 v[PER][R];
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * NT;
        if (TOT % NT == 0 || u < TOT) {
            const int l = u & 15, j = u >> 4;
#pragma unroll
            for (int r = 0; r < R; ++r) {
                float2 x = (NsL == 1) ? load(s, l, j + r * NB) : s[at(j + r * NB, l)];
                if (NsL > 1 && r > 0) {
                    float2 w = tw[(j * r) * TWS];
                    if (INV) w.y = -w.y;
                    x = cmul(x, w);
                }
                v[p][r] = x;
            }
        }
    }
    __syncthreads();
#pragma unroll
    for (int p = 0; p < PER; ++p) {
        const int u = threadIdx.x + p * NT;
        if (TOT % NT == 0 || u < TOT) {
            const int l = u & 15, j = u >> 4;
            dft<R, INV>(v[p]);
#pragma unroll
            for (int r = 0; r < R; ++r) s[l * RS + j + r * NsL] = v[p][r];
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

}  // namespace fft
}  // namespace sd
