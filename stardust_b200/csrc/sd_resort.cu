// sd_resort.cu -- the step's sort as a merge.
//
// Between two steps a particle's key changes only when it crosses a row (tiled
// order) or a cell (row-major, Morton): a percent of the particles or less on the
// 16M/512^3 field. The previous step left the particles sorted by their old keys,
// its row table (row_start[r] = first position with old key >= row_low(r)) and,
// from its gather, the new key of every position plus a bit per position saying
// whether it changed.
// The stable sort of the new keys is then the merge of
//   U  the unchanged positions, already in (key, position) order, and
//   C  the changed ones, radix-sorted by key (stable, so in position order
//      within a key),
// ordered by (key, position) -- exactly the stable sort's order. Every output
// slot follows from counts, with no search over the whole array:
//   changed  (k, i) at rank r in C:  r + #U before it, where the unchanged
//            positions before it are those below row_start[k] plus those in
//            [row_start[k], row_start[k+1]) below i, less the changed ones
//            among them (prefix counts of the change bits); where a row holds many
//            keys (row-major, Morton), a binary search of the row's unchanged
//            positions, whose keys are still in order, takes the place of i;
//   unchanged (k, j):  j - #changed below j + #C with row below k's (a row table of
//            the sorted C) + #C of the same row and (key, position) below (k, j).
// The new row table needs no pass over the keys either: the positions below
// row r are the unchanged ones below the old row_start[r] plus the changed
// ones with key < r. The permutation is the one the radix sort gives; the
// sorted keys themselves are not written (the row table is all the step reads).
// Every formula holds for any set of marked positions that contains the changed
// ones: a marked position whose key did not change simply goes through C, so
// bits left over from a step whose merge never ran cost time, not correctness.
//
// Kernels, in order (the size of C stays on the device throughout):
//   k_chg_count      changed positions per chunk of 512 words
//   k_chg_compact    per word: changed positions before it; C in position order
//   (radix sort of C by key, on grids of about one wave looping over its tiles)
//   k_merge_changed  output slot of every C entry
//   k_rows           row table of C (a galloping search per row) and the new row table
//   k_merge_unchanged output slot of every unchanged position; clears the bits
#include <cuda_runtime.h>
#include <stdint.h>

#include "sd_common.cuh"
#include "sd_internal.h"

namespace sd {
namespace {

constexpr int kChgThreads = 64;
constexpr int kChgWordsPer = 8;                          // words per thread, two 16-byte loads
constexpr int kChunkWords = kChgThreads * kChgWordsPer;  // 512 words = 16,384 positions
constexpr int kCompactThreads = 256;                      // for the chunk's compaction
constexpr int kCompactWords = kChunkWords / (kCompactThreads / 32);  // words per warp
constexpr int kMergeThreads = 256;
constexpr int kMergeWordsPerWarp = 8;                            // 256 positions per warp
constexpr int kMergeWords = (kMergeThreads / 32) * kMergeWordsPerWarp;  // words per CTA

template <int NT>
__device__ __forceinline__ unsigned block_sum(unsigned v, unsigned* red) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[w] = v;
    __syncthreads();
    unsigned t = 0u;
#pragma unroll
    for (int k = 0; k < NT / 32; ++k) t += red[k];
    __syncthreads();
    return t;
}

// Exclusive scan across the block; *total receives the block sum.
template <int NT>
__device__ __forceinline__ unsigned block_exclusive(unsigned v, unsigned* red, unsigned* total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    unsigned inc = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned t = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= o) inc += t;
    }
    if (lane == 31) red[w] = inc;
    __syncthreads();
    unsigned before = 0u, tot = 0u;
#pragma unroll
    for (int k = 0; k < NT / 32; ++k) {
        const unsigned s = red[k];
        if (k < w) before += s;
        tot += s;
    }
    __syncthreads();
    *total = tot;
    return before + inc - v;
}

__device__ __forceinline__ void load_words8(const unsigned* __restrict__ p, unsigned (&w)[8]) {
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    const uint4 b = *reinterpret_cast<const uint4*>(p + 4);
    w[0] = a.x; w[1] = a.y; w[2] = a.z; w[3] = a.w;
    w[4] = b.x; w[5] = b.y; w[6] = b.z; w[7] = b.w;
}

// Changed positions in each chunk of kChunkWords words (the word buffers are
// padded to whole chunks, and the padding stays zero).
__global__ void __launch_bounds__(kChgThreads) k_chg_count(const unsigned* __restrict__ words,
                                                           unsigned* __restrict__ chunk_cnt) {
    wait_previous();
    __shared__ unsigned red[kChgThreads / 32];
    unsigned w[8];
    load_words8(words + (size_t)blockIdx.x * kChunkWords + threadIdx.x * kChgWordsPer, w);
    unsigned c = 0u;
#pragma unroll
    for (int q = 0; q < 8; ++q) c += __popc(w[q]);
    c = block_sum<kChgThreads>(c, red);
    if (threadIdx.x == 0) chunk_cnt[blockIdx.x] = c;
}

// CTA per chunk: the changed positions before each word (word_pre) and C =
// (new key, position) of the changed positions, in position order. The last
// CTA writes the size of C. A warp takes a word's 32 positions at once, sixteen words in
// flight, so keys are read and C is written in runs. (A thread that walked the bits of
// eight words alone read one key after another: the pair of galaxies, 4M particles on 256^3,
// 37.8 us, now 9.3; 8M row-major 9.1, now 6.7; 16M on 512^3, where few change, 10.0 and 11.)
__global__ void __launch_bounds__(kCompactThreads) k_chg_compact(const unsigned* __restrict__ words,
                                                                 const unsigned* __restrict__ chunk_cnt,
                                                                 const uint32_t* __restrict__ keys,
                                                                 unsigned* __restrict__ word_pre,
                                                                 uint32_t* __restrict__ ck, int32_t* __restrict__ ci,
                                                                 int* __restrict__ n_changed) {
    wait_previous();
    static_assert(kChunkWords == 2 * kCompactThreads, "two words per thread in the scan");
    __shared__ unsigned red[kCompactThreads / 32];
    __shared__ uint2 s_word[kChunkWords];  // (word, changed positions before it)
    const size_t chunk = (size_t)blockIdx.x * kChunkWords;
    const uint2 w = *reinterpret_cast<const uint2*>(words + chunk + 2 * threadIdx.x);
    unsigned before = 0u;  // changed positions in the chunks before this one
    for (int b = 0; b < (int)blockIdx.x; b += 8 * kCompactThreads) {  // eight loads in flight per thread
        unsigned v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = b + q * kCompactThreads + threadIdx.x;
            v[q] = c < (int)blockIdx.x ? chunk_cnt[c] : 0u;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) before += v[q];
    }
    before = block_sum<kCompactThreads>(before, red);
    const unsigned c0 = __popc(w.x), c1 = __popc(w.y);
    unsigned total;
    const unsigned base = before + block_exclusive<kCompactThreads>(c0 + c1, red, &total);
    *reinterpret_cast<uint2*>(word_pre + chunk + 2 * threadIdx.x) = make_uint2(base, base + c0);
    *reinterpret_cast<uint4*>(s_word + 2 * threadIdx.x) = make_uint4(w.x, base, w.y, base + c0);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) *n_changed = (int)(before + total);
    __syncwarp();  // a warp compacts the words that its own lanes put there
    const int lane = threadIdx.x & 31, first = (threadIdx.x >> 5) * kCompactWords;
    const unsigned below = (1u << lane) - 1u;
    constexpr int kBatch = 16;
#pragma unroll 1
    for (int i = first; i < first + kCompactWords; i += kBatch) {
        uint32_t key[kBatch];
#pragma unroll
        for (int q = 0; q < kBatch; ++q)
            if (s_word[i + q].x >> lane & 1u) key[q] = keys[(chunk + i + q) * 32 + lane];
#pragma unroll
        for (int q = 0; q < kBatch; ++q) {
            const uint2 v = s_word[i + q];
            if (v.x >> lane & 1u) {
                const unsigned at = v.y + __popc(v.x & below);
                ck[at] = key[q];
                ci[at] = (int)((chunk + i + q) * 32) + lane;
            }
        }
    }
}

// Changed positions below x (0 <= x <= n; the padding words are zero).
__device__ __forceinline__ unsigned changed_below(const unsigned* __restrict__ words,
                                                  const unsigned* __restrict__ word_pre, int x) {
    const unsigned m = (1u << (x & 31)) - 1u;
    return word_pre[x >> 5] + __popc(words[x >> 5] & m);
}

// First unchanged position at or after q (hi when there is none before hi).
__device__ __forceinline__ int next_unchanged(const unsigned* __restrict__ words, int q, int hi) {
    int w = q >> 5;
    unsigned u = ~words[w] & (0xffffffffu << (q & 31));
    while (u == 0u) {
        if ((++w << 5) >= hi) return hi;
        u = ~words[w];
    }
    return min(hi, (w << 5) + __ffs(u) - 1);
}

// WIDE: rows hold many keys (shift >= 0); otherwise the key is the row.
template <bool WIDE>
__global__ void k_merge_changed(const uint32_t* __restrict__ ck, const int32_t* __restrict__ ci,
                                const int* __restrict__ n_changed, const uint32_t* __restrict__ keys, int shift,
                                const int* __restrict__ row_start_old, const unsigned* __restrict__ words,
                                const unsigned* __restrict__ word_pre, int32_t* __restrict__ vals_out) {
    wait_previous();
    const int nc = *n_changed;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < nc; r += gridDim.x * blockDim.x) {
        const uint32_t k = ck[r];
        const int i = ci[r];
        const uint32_t row = WIDE ? row_of(k, shift) : k;
        const int lb = row_start_old[row], ub = row_start_old[row + 1];
        if (WIDE) {
            // the row's unchanged positions are in (key, position) order: find the first
            // that is not before (k, i), stepping over the changed ones
            int lo = lb, hi = ub;
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                const int q = next_unchanged(words, mid, hi);
                const uint32_t kq = q < hi ? keys[q] : 0xffffffffu;
                if (kq < k || (kq == k && q < i)) lo = q + 1;
                else hi = mid;
            }
            vals_out[r + lo - (int)changed_below(words, word_pre, lo)] = i;
        } else {
            const unsigned cl = changed_below(words, word_pre, lb);
            unsigned u = (unsigned)lb - cl;
            if (i > lb) {
                const int m = min(ub, i);
                u += (unsigned)(m - lb) - (changed_below(words, word_pre, m) - cl);
            }
            vals_out[r + u] = i;
        }
    }
}

// Thread per row r in [0, rows]: c_rows[r] = first rank of C with key >= row_low(r), and
// the new row start = unchanged positions below the old one + c_rows[r]. The
// search starts where r would fall if C were spread evenly over the rows and
// gallops outwards to a bracket, which a few steps find for an even spread.
__global__ void k_rows(const uint32_t* __restrict__ ck, const int* __restrict__ n_changed, int rows, int shift,
                       const unsigned* __restrict__ words, const unsigned* __restrict__ word_pre,
                       int* __restrict__ c_rows, int* __restrict__ row_start) {
    wait_previous();
    const int nc = *n_changed;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r <= rows; r += gridDim.x * blockDim.x) {
        const uint32_t low = row_low(r, shift);
        // bracket [lo, hi] with ck[lo - 1] < low <= ck[hi] (ck[-1] = -inf, ck[nc] = +inf)
        const int g = (int)(((long long)r * nc) / (rows > 0 ? rows : 1));
        int lo, hi;
        if (g < nc && ck[g] < low) {  // the answer lies above g
            int step = 1;
            lo = g + 1;
            hi = g + 1;
            while (hi < nc && ck[hi] < low) {
                lo = hi + 1;
                hi = min(nc, hi + step);
                step <<= 1;
            }
        } else {  // at or below g
            int step = 1;
            hi = g;
            lo = g;
            while (lo > 0 && ck[lo - 1] >= low) {
                hi = lo - 1;
                lo = max(0, lo - step);
                step <<= 1;
            }
        }
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (ck[mid] < low) lo = mid + 1;
            else hi = mid;
        }
        c_rows[r] = lo;
        const int rs = row_start[r];
        row_start[r] = rs - (int)changed_below(words, word_pre, rs) + lo;
    }
}

// Warp per 8 words (256 positions, lane-major: position = base + 32 q + lane), all
// loads issued before use. The changed positions were placed by k_merge_changed.
// Clears the change bits for the next gather.
template <bool WIDE>
__global__ void __launch_bounds__(kMergeThreads) k_merge_unchanged(const uint32_t* __restrict__ keys,
                                                                   unsigned* __restrict__ words,
                                                                   const unsigned* __restrict__ word_pre,
                                                                   const int* __restrict__ c_rows, int shift,
                                                                   const uint32_t* __restrict__ ck,
                                                                   const int32_t* __restrict__ ci, int n,
                                                                   int32_t* __restrict__ vals_out) {
    wait_previous();
    const int lane = threadIdx.x & 31;
    const size_t wb = (size_t)blockIdx.x * kMergeWords + (threadIdx.x >> 5) * kMergeWordsPerWarp;
    const int base = (int)(wb * 32);
    if (base >= n) return;
    unsigned bits[8], pre[8];
    load_words8(words + wb, bits);
    load_words8(word_pre + wb, pre);
    uint32_t k[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = base + q * 32 + lane;
        k[q] = (j < n) ? keys[j] : 0u;
    }
    int lo[8], hi[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const uint32_t row = WIDE ? row_of(k[q], shift) : k[q];
        lo[q] = c_rows[row];
        hi[q] = c_rows[row + 1];
    }
    const unsigned lt = lanemask_lt();
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int j = base + q * 32 + lane;
        if (j < n && !((bits[q] >> lane) & 1u)) {
            // C entries of k's row lie at ranks [c_rows[row], c_rows[row+1]) in (key, position) order
            int a = lo[q], b = hi[q];
            while (a < b) {  // first rank that is above (k, j)
                const int mid = (a + b) >> 1;
                bool before = ci[mid] < j;
                if (WIDE) {
                    const uint32_t kc = ck[mid];
                    before = kc < k[q] || (kc == k[q] && before);
                }
                if (before) a = mid + 1;
                else b = mid;
            }
            vals_out[j - (int)(pre[q] + __popc(bits[q] & lt)) + a] = j;
        }
    }
    __syncwarp();
    if (lane < kMergeWordsPerWarp) words[wb + lane] = 0u;  // every lane has used them
}

// Words for n positions plus one (changed_below(n) reads word n / 32), in whole chunks.
size_t padded_words(int n) {
    const size_t w = (size_t)n / 32 + 1;
    return (w + kChunkWords - 1) / kChunkWords * kChunkWords;
}

}  // namespace

size_t resort_words(int n) { return padded_words(n); }

size_t resort_bytes(int n, int G) {
    const size_t words = padded_words(n), chunks = words / kChunkWords;
    return align_up(sizeof(unsigned) * words, 256) * 2 + align_up(sizeof(unsigned) * chunks, 256) +
           align_up(sizeof(int32_t) * ((size_t)G * G + 2), 256) + align_up(sizeof(int), 256) +
           3 * align_up(sizeof(uint32_t) * (size_t)n, 256);
}

ResortBufs resort_layout(void* base, int n, int G, uint32_t* spare_k0, int32_t* spare_v0, uint32_t* spare_k1) {
    const size_t words = padded_words(n), chunks = words / kChunkWords;
    char* b = (char*)base;
    ResortBufs r;
    r.words = (unsigned*)b;
    b += align_up(sizeof(unsigned) * words, 256);
    r.word_pre = (unsigned*)b;
    b += align_up(sizeof(unsigned) * words, 256);
    r.chunk_cnt = (unsigned*)b;
    b += align_up(sizeof(unsigned) * chunks, 256);
    r.c_rows = (int*)b;
    b += align_up(sizeof(int32_t) * ((size_t)G * G + 2), 256);
    r.n_changed = (int*)b;
    b += align_up(sizeof(int), 256);
    r.ck_out = (uint32_t*)b;
    b += align_up(sizeof(uint32_t) * (size_t)n, 256);
    r.ci_out = (int32_t*)b;
    b += align_up(sizeof(int32_t) * (size_t)n, 256);
    r.ci_tmp = (int32_t*)b;
    r.ck_in = spare_k0;
    r.ci_in = spare_v0;
    r.ck_tmp = spare_k1;
    return r;
}

int launch_resort(const ResortBufs& r, const uint32_t* keys, int n, int G, int order, int key_bits, int* row_start,
                  int32_t* vals_out, void* sort_ws, size_t sort_ws_bytes, cudaStream_t s) {
    if (n <= 0) return SD_OK;
    const int chunks = (int)(padded_words(n) / kChunkWords);
    const int rows = row_last(G, order), shift = row_shift(G, order);
    launch(k_chg_count, chunks, kChgThreads, 0, s, r.words, r.chunk_cnt);
    SD_LAUNCHED(s);
    launch(k_chg_compact, chunks, kCompactThreads, 0, s, r.words, r.chunk_cnt, keys, r.word_pre, r.ck_in, r.ci_in,
           r.n_changed);
    SD_LAUNCHED(s);
    // C by key, stable: the radix sort with the count on the device
    int rc = launch_sort_pairs(r.ck_in, r.ci_in, r.ck_out, r.ci_out, r.ck_tmp, r.ci_tmp, n, key_bits, sort_ws,
                               sort_ws_bytes, s, true, false, r.n_changed);
    if (rc) return rc;
    auto changed = shift < 0 ? k_merge_changed<false> : k_merge_changed<true>;
    launch(changed, 148 * 4, 256, 0, s, r.ck_out, r.ci_out, r.n_changed, keys, shift, row_start, r.words, r.word_pre,
           vals_out);
    SD_LAUNCHED(s);
    launch(k_rows, (rows + 1 + 255) / 256, 256, 0, s, r.ck_out, r.n_changed, rows, shift, r.words, r.word_pre, r.c_rows,
           row_start);
    SD_LAUNCHED(s);
    const int warps = (n + 255) / 256;
    auto unchanged = shift < 0 ? k_merge_unchanged<false> : k_merge_unchanged<true>;
    launch(unchanged, (warps + kMergeThreads / 32 - 1) / (kMergeThreads / 32), kMergeThreads, 0, s,
           keys, r.words, r.word_pre, r.c_rows, shift, r.ck_out, r.ci_out, n, vals_out);
    SD_LAUNCHED(s);
    return SD_OK;
}

}  // namespace sd
