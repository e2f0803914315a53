// Bag relations on the device: canonical instance tuples, a stable LSD radix
// sort of uint32 tuples, and trie levels built from the sorted tuples.
//
// The reference materialises a bag as vector<vector<VertexID>> tuples
// (nodeJoin, matching/join.cpp:309-421), std::sorts them and groups them
// column by column into nested TrieLevel{values, children}
// (buildTrie, join.cpp:1713-1717; TrieLevel::buildTrieFromSortedMatchesBatch,
// relation/relation.cpp:340-379).  Here tuples are rows of a device array;
// the sort packs a tuple into a 64- or 128-bit key and runs an LSD radix sort
// over the bits in use (8-bit digits, stable scatter by warp match + per-warp
// digit counts), and each trie level is a flat array of values plus child
// offsets into the next level (CSR form of the same tree), all levels built
// in two passes over the rows.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "common.hpp"
#include "device_util.hpp"

using namespace sge;

namespace {

#define CUDA_TRY(expr)                                                                               \
    do {                                                                                             \
        cudaError_t _e = (expr);                                                                     \
        if (_e != cudaSuccess)                                                                       \
            return fail(_e == cudaErrorMemoryAllocation ? SGE_OOM : SGE_CUDA_ERROR, "%s: %s", #expr, \
                        cudaGetErrorString(_e));                                                     \
    } while (0)

constexpr int MAX_ARITY = 16;

// ---- canonical form: the lexicographically smallest image of a tuple under
// the pattern's automorphisms (one representative per automorphism class) ----
__global__ void canon_kernel(uint32_t *t, unsigned long long n, uint32_t k, const uint8_t *__restrict__ perms,
                             uint32_t naut) {
    unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint32_t *row = t + i * k;
    uint32_t best[MAX_ARITY], cur[MAX_ARITY];
    for (uint32_t j = 0; j < k; ++j) best[j] = row[j];
    for (uint32_t a = 0; a < naut; ++a) {
        const uint8_t *s = perms + (size_t)a * k;
        int cmp = 0;
        for (uint32_t j = 0; j < k; ++j) {
            cur[j] = row[s[j]];
            if (cmp == 0) cmp = cur[j] < best[j] ? -1 : (cur[j] > best[j] ? 1 : 0);
        }
        if (cmp < 0)
            for (uint32_t j = 0; j < k; ++j) best[j] = cur[j];
    }
    for (uint32_t j = 0; j < k; ++j) row[j] = best[j];
}

inline unsigned grid_for(unsigned long long n, unsigned b = 256) { return (unsigned)((n + b - 1) / b); }

constexpr int SORT_THREADS = 256, SORT_WARPS = SORT_THREADS / 32;
constexpr int SCAN_TILE = 4096;  // 256 threads x 16

// Exclusive prefix of one value per thread over a 256-thread block, and the total.
__device__ __forceinline__ uint32_t block_exclusive(uint32_t v, uint32_t *ws, uint32_t &total) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (uint32_t o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xFFFFFFFFu, incl, o);
        if (lane >= o) incl += t;
    }
    __syncthreads();  // (ws may still be read from the last call)
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
#pragma unroll
    for (uint32_t q = 0; q < SORT_WARPS; ++q) {
        if (q < w) before += ws[q];
        total += ws[q];
    }
    return before + incl - v;
}

// ---- keys: a tuple packed into 64 or 128 bits, first column highest ----
// The sort moves whole tuples as keys of exactly the bits their columns use
// (the OR of each column gives its width), so a pass reads and writes 8 or 16
// bytes a row in order.  Sorting a permutation instead gathers every digit
// from a random row: 8 passes over 32M (src, dst) rows took 8.4 ms, the keys
// 5 passes take 1.8 ms.
struct Key64 {
    unsigned long long lo;
    __device__ __forceinline__ uint32_t digit(uint32_t shift) const { return (uint32_t)(lo >> shift) & 0xFFu; }
    __device__ __forceinline__ void push(uint32_t v, uint32_t bits) { lo = (lo << bits) | v; }
    __device__ __forceinline__ uint32_t pop(uint32_t bits) {
        const uint32_t v = (uint32_t)(lo & ((1ull << bits) - 1ull));
        lo >>= bits;
        return v;
    }
};
struct alignas(16) Key128 {
    unsigned long long lo, hi;
    __device__ __forceinline__ uint32_t digit(uint32_t shift) const {
        if (shift >= 64) return (uint32_t)(hi >> (shift - 64)) & 0xFFu;
        uint32_t d = (uint32_t)(lo >> shift);
        if (shift > 56) d |= (uint32_t)(hi << (64 - shift));
        return d & 0xFFu;
    }
    __device__ __forceinline__ void push(uint32_t v, uint32_t bits) {
        if (!bits) return;
        hi = (hi << bits) | (lo >> (64 - bits));
        lo = (lo << bits) | v;
    }
    __device__ __forceinline__ uint32_t pop(uint32_t bits) {
        const uint32_t v = (uint32_t)(lo & ((1ull << bits) - 1ull));
        if (bits) {
            lo = (lo >> bits) | (hi << (64 - bits));
            hi >>= bits;
        }
        return v;
    }
};
struct Widths {
    uint8_t bits[MAX_ARITY];
};

// OR of every column (its width), 16 columns at most.
__global__ void column_or_kernel(const uint32_t *t, unsigned long long n, uint32_t arity, uint32_t *ors) {
    // a thread strides by a multiple of the arity, so it stays in one column
    const unsigned long long total = n * arity, step = (unsigned long long)gridDim.x * blockDim.x / arity * arity;
    const unsigned long long first = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x;
    __shared__ uint32_t s[MAX_ARITY];
    if (threadIdx.x < MAX_ARITY) s[threadIdx.x] = 0;
    __syncthreads();
    uint32_t v = 0;
    if (first < step)
        for (unsigned long long i = first; i < total; i += step) v |= t[i];
    if (v) atomicOr(&s[first % arity], v);
    __syncthreads();
    if (threadIdx.x < arity && s[threadIdx.x]) atomicOr(ors + threadIdx.x, s[threadIdx.x]);
}

template <class K>
__global__ void pack_kernel(const uint32_t *t, unsigned long long n, uint32_t arity, Widths w, K *keys) {
    const unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    K k{};
    for (uint32_t c = 0; c < arity; ++c) k.push(t[i * arity + c], w.bits[c]);
    keys[i] = k;
}
template <class K>
__global__ void unpack_kernel(const K *keys, unsigned long long n, uint32_t arity, Widths w, uint32_t *t) {
    const unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    K k = keys[i];
    for (uint32_t c = arity; c-- > 0;) t[i * arity + c] = k.pop(w.bits[c]);
}

// ---- one pass of the LSD radix sort over an 8-bit digit: tile histograms,
// one scan row per digit, stable scatter ----
template <class K>
constexpr int SORT_ITEMS = sizeof(K) == 8 ? 16 : 8;  // per thread: 32 KB of keys a tile
template <class K>
constexpr int SORT_TILE = SORT_THREADS *SORT_ITEMS<K>;

// digit counts of each tile, digit-major: hist[d * ntiles + tile]
template <class K>
__global__ void __launch_bounds__(SORT_THREADS) hist_kernel(const K *keys, unsigned long long n, uint32_t shift,
                                                            uint32_t *hist, uint32_t ntiles) {
    __shared__ uint32_t h[SORT_WARPS][256];   // a copy per warp: fewer conflicting atomics
    const uint32_t warp = threadIdx.x >> 5;
    for (uint32_t i = threadIdx.x; i < SORT_WARPS * 256; i += SORT_THREADS) (&h[0][0])[i] = 0;
    __syncthreads();
    const unsigned long long base = (unsigned long long)blockIdx.x * SORT_TILE<K>;
#pragma unroll 4
    for (int r = 0; r < SORT_ITEMS<K>; ++r) {
        const unsigned long long i = base + r * SORT_THREADS + threadIdx.x;
        if (i < n) atomicAdd(&h[warp][keys[i].digit(shift)], 1u);
    }
    __syncthreads();
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t w = 0; w < SORT_WARPS; ++w) sum += h[w][threadIdx.x];
    hist[(size_t)threadIdx.x * ntiles + blockIdx.x] = sum;
}

// Block d: exclusive prefix of row d in place; totals[d] = its sum.
__global__ void __launch_bounds__(SORT_THREADS) row_scan_kernel(uint32_t *hist, uint32_t ntiles, uint32_t *totals) {
    __shared__ uint32_t ws[SORT_WARPS];
    uint32_t *row = hist + (size_t)blockIdx.x * ntiles, run = 0;
    for (uint32_t b = 0; b < ntiles; b += SORT_THREADS) {
        const uint32_t i = b + threadIdx.x, v = i < ntiles ? row[i] : 0u;
        uint32_t total;
        const uint32_t at = block_exclusive(v, ws, total);
        if (i < ntiles) row[i] = run + at;
        run += total;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = run;
}

// Stable scatter.  A warp ranks its consecutive SORT_ITEMS x 32 keys by
// matching equal digits lane by lane; the tile is put in digit order in shared
// memory and written from there, so that a digit's keys leave as one run.
template <class K>
__global__ void __launch_bounds__(SORT_THREADS) scatter_kernel(const K *in, K *out, unsigned long long n,
                                                               uint32_t shift, const uint32_t *hist, uint32_t ntiles,
                                                               const uint32_t *totals) {
    constexpr int ITEMS = SORT_ITEMS<K>, TILE = SORT_TILE<K>;
    extern __shared__ __align__(16) unsigned char smem[];
    K *sorted = reinterpret_cast<K *>(smem);                                     // TILE keys
    uint32_t(*cnt)[256] = reinterpret_cast<uint32_t(*)[256]>(smem + TILE * sizeof(K));  // per warp and digit
    uint32_t *gbase = reinterpret_cast<uint32_t *>(cnt + SORT_WARPS);            // output index of a digit's run, less its start in the tile
    __shared__ uint32_t ws[SORT_WARPS];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    for (uint32_t i = threadIdx.x; i < SORT_WARPS * 256; i += SORT_THREADS) (&cnt[0][0])[i] = 0;
    __syncthreads();
    const unsigned long long tile = (unsigned long long)blockIdx.x * TILE;
    const uint32_t have = (uint32_t)min((unsigned long long)TILE, n - tile);
    K key[ITEMS];
    uint16_t rank[ITEMS];
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t i = warp * (ITEMS * 32) + r * 32 + lane;
        if (i < have) key[r] = in[tile + i];
    }
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t i = warp * (ITEMS * 32) + r * 32 + lane;
        const bool ok = i < have;
        const uint32_t d = ok ? key[r].digit(shift) : 256u + lane;  // (absent keys match nothing)
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, d);
        const uint32_t below = __popc(peers & ((1u << lane) - 1u));
        uint32_t before = 0;
        if (ok && below == 0) {
            before = cnt[warp][d];
            cnt[warp][d] = before + __popc(peers);
        }
        before = __shfl_sync(0xFFFFFFFFu, before, __ffs(peers) - 1);
        rank[r] = (uint16_t)(before + below);
        __syncwarp();
    }
    __syncthreads();
    // digit threadIdx.x: its warps' prefixes, its start in the tile and in the output
    {
        const uint32_t d = threadIdx.x;
        uint32_t sum = 0;
#pragma unroll
        for (uint32_t w = 0; w < SORT_WARPS; ++w) {
            const uint32_t c = cnt[w][d];
            cnt[w][d] = sum;
            sum += c;
        }
        uint32_t total;
        const uint32_t start = block_exclusive(sum, ws, total);
        const uint32_t digit_base = block_exclusive(totals[d], ws, total);
#pragma unroll
        for (uint32_t w = 0; w < SORT_WARPS; ++w) cnt[w][d] += start;
        gbase[d] = digit_base + hist[(size_t)d * ntiles + blockIdx.x] - start;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < ITEMS; ++r) {
        const uint32_t i = warp * (ITEMS * 32) + r * 32 + lane;
        if (i < have) sorted[cnt[warp][key[r].digit(shift)] + rank[r]] = key[r];
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < have; i += SORT_THREADS) {
        const K k = sorted[i];
        out[gbase[k.digit(shift)] + i] = k;
    }
}

// Sorts n keys by their bits [from, to); the result is in *a (a and b change
// places).  hist: 256 * ntiles + 256 words.
template <class K>
sge_status sort_keys(K *&a, K *&b, unsigned long long n, uint32_t from, uint32_t to, uint32_t *hist, cudaStream_t s) {
    const uint32_t ntiles = (uint32_t)((n + SORT_TILE<K> - 1) / SORT_TILE<K>);
    uint32_t *totals = hist + 256ull * ntiles;
    const size_t smem = SORT_TILE<K> * sizeof(K) + (SORT_WARPS + 1) * 256 * 4;
    CUDA_TRY(cudaFuncSetAttribute(scatter_kernel<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    for (uint32_t shift = from; shift < to; shift += 8) {
        hist_kernel<K><<<ntiles, SORT_THREADS, 0, s>>>(a, n, shift, hist, ntiles);
        row_scan_kernel<<<256, SORT_THREADS, 0, s>>>(hist, ntiles, totals);
        scatter_kernel<K><<<ntiles, SORT_THREADS, smem, s>>>(a, b, n, shift, hist, ntiles, totals);
        std::swap(a, b);
    }
    CUDA_TRY(cudaGetLastError());
    return SGE_OK;
}

// ---- rows wider than 128 bits: a permutation sorted by one 8-bit digit of
// one column at a time, each digit as a 64-bit (digit, index) key ----
__global__ void digit_keys_kernel(const uint32_t *t, const Key64 *perm, unsigned long long n, uint32_t arity,
                                  uint32_t col, Key64 *keys) {
    const unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t idx = perm ? (uint32_t)perm[i].lo : (uint32_t)i;
    keys[i].lo = (unsigned long long)t[(size_t)idx * arity + col] << 32 | idx;
}
__global__ void gather_rows(const uint32_t *in, const Key64 *perm, uint32_t *out, unsigned long long n,
                            uint32_t arity) {
    const unsigned long long i = blockIdx.x * (unsigned long long)blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t *src = in + (size_t)(uint32_t)perm[i].lo * arity;
    uint32_t *dst = out + i * arity;
    for (uint32_t j = 0; j < arity; ++j) dst[j] = src[j];
}

// ---- exclusive scan of n uint32: tile sums, one block over them, tile scans ----
__global__ void __launch_bounds__(256) tile_sums_kernel(const uint32_t *in, unsigned long long n, uint32_t *sums) {
    __shared__ uint32_t ws[SORT_WARPS];
    const unsigned long long base = blockIdx.x * (unsigned long long)SCAN_TILE;
    uint32_t v = 0, total;
#pragma unroll
    for (int r = 0; r < SCAN_TILE / 256; ++r) {
        const unsigned long long i = base + r * 256 + threadIdx.x;
        if (i < n) v += in[i];
    }
    block_exclusive(v, ws, total);
    if (threadIdx.x == 0) sums[blockIdx.x] = total;
}
// Exclusive prefix of m words in place, one block.
__global__ void __launch_bounds__(256) sums_scan_kernel(uint32_t *a, uint32_t m, uint32_t *grand) {
    __shared__ uint32_t ws[SORT_WARPS];
    uint32_t run = 0;
    for (uint32_t b = 0; b < m; b += 256 * 16) {
        uint32_t v[16], sum = 0, total;
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const uint32_t i = b + threadIdx.x * 16 + q;
            v[q] = i < m ? a[i] : 0u;
            sum += v[q];
        }
        uint32_t at = run + block_exclusive(sum, ws, total);
#pragma unroll
        for (int q = 0; q < 16; ++q) {
            const uint32_t i = b + threadIdx.x * 16 + q;
            if (i < m) a[i] = at;
            at += v[q];
        }
        run += total;
    }
    if (threadIdx.x == 0 && grand) *grand = run;
}
__global__ void __launch_bounds__(256) tile_scan_kernel(const uint32_t *in, uint32_t *out, unsigned long long n,
                                                        const uint32_t *sums) {
    __shared__ uint32_t ws[SORT_WARPS];
    __shared__ uint32_t buf[SCAN_TILE + SCAN_TILE / 16];   // (padded: a thread's 16 words are consecutive)
    const unsigned long long base = blockIdx.x * (unsigned long long)SCAN_TILE;
#pragma unroll
    for (int r = 0; r < SCAN_TILE / 256; ++r) {
        const uint32_t i = r * 256 + threadIdx.x;
        buf[i + i / 16] = base + i < n ? in[base + i] : 0u;
    }
    __syncthreads();
    uint32_t v[16], sum = 0, total;
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        v[q] = buf[threadIdx.x * 17 + q];
        sum += v[q];
    }
    uint32_t at = sums[blockIdx.x] + block_exclusive(sum, ws, total);
#pragma unroll
    for (int q = 0; q < 16; ++q) {
        buf[threadIdx.x * 17 + q] = at;
        at += v[q];
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < SCAN_TILE / 256; ++r) {
        const uint32_t i = r * 256 + threadIdx.x;
        if (base + i < n) out[base + i] = buf[i + i / 16];
    }
}

// ---- trie levels from sorted tuples ----
// Row i starts a node of every level from first_change(i) on (the first column
// that differs from row i - 1).  One pass counts the nodes of every level per
// tile, a scan numbers them, and a second pass writes all levels' values and
// child offsets: 2 reads of the rows where a flag, a scan and two gathers per
// level took 10 passes.
constexpr int TRIE_TILE = 1024;   // rows per block: 256 threads x 4
__device__ __forceinline__ uint32_t first_change(const uint32_t *t, unsigned long long i, uint32_t arity) {
    if (i == 0) return 0;
    const uint32_t *a = t + (i - 1) * arity, *b = a + arity;
    uint32_t c = 0;
    while (c < arity && a[c] == b[c]) ++c;
    return c;
}
// counts[l * ntiles + tile] = nodes of level l that start in the tile
__global__ void __launch_bounds__(256) trie_count_kernel(const uint32_t *t, unsigned long long n, uint32_t arity,
                                                         uint32_t ntiles, uint32_t *counts) {
    __shared__ uint32_t c[MAX_ARITY];
    if (threadIdx.x < MAX_ARITY) c[threadIdx.x] = 0;
    __syncthreads();
    const unsigned long long base = blockIdx.x * (unsigned long long)TRIE_TILE;
    for (int r = 0; r < TRIE_TILE / 256; ++r) {
        const unsigned long long i = base + r * 256 + threadIdx.x;
        const uint32_t f = i < n ? first_change(t, i, arity) : arity;
        for (uint32_t l = 0; l < arity; ++l) {
            const uint32_t b = __ballot_sync(0xFFFFFFFFu, f <= l);
            if ((threadIdx.x & 31u) == 0 && b) atomicAdd(&c[l], (uint32_t)__popc(b));
        }
    }
    __syncthreads();
    if (threadIdx.x < arity) counts[(size_t)threadIdx.x * ntiles + blockIdx.x] = c[threadIdx.x];
}
struct TriePtrs {
    uint32_t *values[MAX_ARITY];
    unsigned long long *child[MAX_ARITY];
};
__global__ void __launch_bounds__(256) trie_write_kernel(const uint32_t *t, unsigned long long n, uint32_t arity,
                                                         uint32_t ntiles, const uint32_t *counts, TriePtrs out) {
    __shared__ uint32_t ws[SORT_WARPS];
    const unsigned long long base = blockIdx.x * (unsigned long long)TRIE_TILE + threadIdx.x * (TRIE_TILE / 256);
    uint32_t f[TRIE_TILE / 256];
#pragma unroll
    for (int r = 0; r < TRIE_TILE / 256; ++r) f[r] = base + r < n ? first_change(t, base + r, arity) : arity;
    // from the deepest level up: a node's first child is the next level's node of the same row
    uint32_t below[TRIE_TILE / 256];
    for (uint32_t l = arity; l-- > 0;) {
        uint32_t mine = 0, total;
#pragma unroll
        for (int r = 0; r < TRIE_TILE / 256; ++r) mine += f[r] <= l;
        uint32_t at = counts[(size_t)l * ntiles + blockIdx.x] + block_exclusive(mine, ws, total);
#pragma unroll
        for (int r = 0; r < TRIE_TILE / 256; ++r)
            if (f[r] <= l) {
                out.values[l][at] = t[(base + r) * arity + l];
                if (l + 1 < arity) out.child[l][at] = below[r];
                below[r] = at++;
            }
    }
}
// End of each level's child array, and nothing else.
__global__ void trie_ends_kernel(uint32_t arity, const uint32_t *totals, TriePtrs out) {
    const uint32_t l = threadIdx.x;
    if (l + 1 < arity) out.child[l][totals[l]] = totals[l + 1];
}

}  // namespace

sge_status sge::device_exclusive_scan(const uint32_t *in, uint32_t *out, uint64_t n, cudaStream_t s) {
    if (n == 0) return SGE_OK;
    uint32_t *sums = nullptr;
    const uint32_t nb = (uint32_t)((n + SCAN_TILE - 1) / SCAN_TILE);
    CUDA_TRY(cudaMalloc(&sums, sizeof(uint32_t) * nb));
    tile_sums_kernel<<<nb, 256, 0, s>>>(in, n, sums);
    sums_scan_kernel<<<1, 256, 0, s>>>(sums, nb, nullptr);
    tile_scan_kernel<<<nb, 256, 0, s>>>(in, out, n, sums);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    cudaFree(sums);
    if (e != cudaSuccess) return fail(SGE_CUDA_ERROR, "device_exclusive_scan: %s", cudaGetErrorString(e));
    return SGE_OK;
}

sge_status sge::device_sort_keys(unsigned long long *&keys, unsigned long long *&tmp, uint64_t n, uint32_t bits,
                                 cudaStream_t s) {
    if (n <= 1) return SGE_OK;
    uint32_t *hist = nullptr;
    const uint64_t ntiles = (n + SORT_TILE<Key64> - 1) / SORT_TILE<Key64>;
    CUDA_TRY(cudaMalloc(&hist, (256 * ntiles + 256) * 4));
    Key64 *a = reinterpret_cast<Key64 *>(keys), *b = reinterpret_cast<Key64 *>(tmp);
    const sge_status st = sort_keys(a, b, n, 0u, bits, hist, s);
    keys = reinterpret_cast<unsigned long long *>(a);
    tmp = reinterpret_cast<unsigned long long *>(b);
    cudaError_t e = cudaStreamSynchronize(s);
    cudaFree(hist);
    if (st != SGE_OK) return st;
    if (e != cudaSuccess) return fail(SGE_CUDA_ERROR, "device_sort_keys: %s", cudaGetErrorString(e));
    return SGE_OK;
}

namespace {
// Wider rows: one stable sort of (column value, row) keys per column, last column first.
sge_status sort_wide(uint32_t *d_tuples, uint64_t n, uint32_t arity, const Widths &w) {
    Key64 *a = nullptr, *b = nullptr;
    uint32_t *hist = nullptr, *rows = nullptr;
    const uint64_t ntiles = (n + SORT_TILE<Key64> - 1) / SORT_TILE<Key64>;
    auto cleanup = [&]() { cudaFree(a); cudaFree(b); cudaFree(hist); cudaFree(rows); };
    cudaError_t e;
    if ((e = cudaMalloc(&a, n * 8)) != cudaSuccess || (e = cudaMalloc(&b, n * 8)) != cudaSuccess ||
        (e = cudaMalloc(&hist, (256 * ntiles + 256) * 4)) != cudaSuccess) {
        cleanup();
        return fail(SGE_OOM, "sge_sort_tuples: %s", cudaGetErrorString(e));
    }
    bool first = true;
    for (int col = (int)arity - 1; col >= 0; --col) {
        if (!w.bits[col] && !(first && col == 0)) continue;
        digit_keys_kernel<<<grid_for(n), 256>>>(d_tuples, first ? nullptr : a, n, arity, (uint32_t)col, first ? a : b);
        if (!first) std::swap(a, b);
        first = false;
        sge_status st = sort_keys(a, b, n, 32u, 32u + w.bits[col], hist, 0);
        if (st != SGE_OK) {
            cleanup();
            return st;
        }
    }
    cudaFree(b);   // (the rows' copy takes its place)
    b = nullptr;
    if ((e = cudaMalloc(&rows, n * arity * 4ull)) != cudaSuccess) {
        cleanup();
        return fail(SGE_OOM, "sge_sort_tuples: %s", cudaGetErrorString(e));
    }
    gather_rows<<<grid_for(n), 256>>>(d_tuples, a, rows, n, arity);
    e = cudaMemcpy(d_tuples, rows, n * arity * 4ull, cudaMemcpyDeviceToDevice);
    cudaError_t e2 = cudaDeviceSynchronize();
    cleanup();
    if (e != cudaSuccess || e2 != cudaSuccess)
        return fail(SGE_CUDA_ERROR, "sge_sort_tuples: %s", cudaGetErrorString(e != cudaSuccess ? e : e2));
    return SGE_OK;
}
// Packs, sorts and unpacks rows whose columns fit one key.
template <class K>
sge_status sort_packed(uint32_t *d_tuples, uint64_t n, uint32_t arity, const Widths &w, uint32_t bits) {
    K *a = nullptr, *b = nullptr;
    uint32_t *hist = nullptr;
    const uint64_t ntiles = (n + SORT_TILE<K> - 1) / SORT_TILE<K>;
    cudaError_t e;
    if ((e = cudaMalloc(&a, n * sizeof(K))) != cudaSuccess || (e = cudaMalloc(&b, n * sizeof(K))) != cudaSuccess ||
        (e = cudaMalloc(&hist, (256 * ntiles + 256) * 4)) != cudaSuccess) {
        cudaFree(a);
        cudaFree(b);
        cudaGetLastError();
        // (128-bit keys: the wide form's are half as large)
        if (sizeof(K) == 16 && arity > 1) return sort_wide(d_tuples, n, arity, w);
        return fail(SGE_OOM, "sge_sort_tuples: %s", cudaGetErrorString(e));
    }
    pack_kernel<K><<<grid_for(n), 256>>>(d_tuples, n, arity, w, a);
    const sge_status st = sort_keys(a, b, n, 0u, bits, hist, 0);
    if (st == SGE_OK) unpack_kernel<K><<<grid_for(n), 256>>>(a, n, arity, w, d_tuples);
    e = cudaDeviceSynchronize();
    cudaFree(a);
    cudaFree(b);
    cudaFree(hist);
    if (st != SGE_OK) return st;
    if (e != cudaSuccess) return fail(SGE_CUDA_ERROR, "sge_sort_tuples: %s", cudaGetErrorString(e));
    return SGE_OK;
}
}  // namespace

extern "C" {

sge_status sge_canonicalize(uint32_t *d_tuples, uint64_t n, uint32_t k, const uint8_t *perms, uint32_t naut) {
    if ((!d_tuples && n) || !perms || k == 0 || k > MAX_ARITY || naut == 0)
        return fail(SGE_BAD_INPUT, "sge_canonicalize: bad argument");
    if (n == 0) return SGE_OK;
    uint8_t *dp = nullptr;
    CUDA_TRY(cudaMalloc(&dp, (size_t)naut * k));
    CUDA_TRY(cudaMemcpy(dp, perms, (size_t)naut * k, cudaMemcpyHostToDevice));
    canon_kernel<<<grid_for(n), 256>>>(d_tuples, n, k, dp, naut);
    cudaError_t e = cudaDeviceSynchronize();
    cudaFree(dp);
    if (e != cudaSuccess) return fail(SGE_CUDA_ERROR, "canonicalize: %s", cudaGetErrorString(e));
    return SGE_OK;
}

// Lexicographic sort of n rows of `arity` uint32 (device, in place).
sge_status sge_sort_tuples(uint32_t *d_tuples, uint64_t n, uint32_t arity) {
    if ((!d_tuples && n) || arity == 0 || arity > MAX_ARITY) return fail(SGE_BAD_INPUT, "sge_sort_tuples: bad argument");
    if (n <= 1) return SGE_OK;
    if (n >= (1ull << 32)) return fail(SGE_UNSUPPORTED, "sge_sort_tuples: more than 2^32 rows");
    if (arity == 1 && n <= (1ull << 20)) {
        // a short column: its width saves less than finding it costs (100,000
        // values of 31 bits 0.38 ms with the look, 0.28 without)
        Widths w{};
        w.bits[0] = 32;
        return sort_packed<Key64>(d_tuples, n, arity, w, 32);
    }
    uint32_t *d_or = nullptr, h_or[MAX_ARITY] = {};
    CUDA_TRY(cudaMalloc(&d_or, sizeof h_or));
    cudaError_t e = cudaMemset(d_or, 0, sizeof h_or);
    if (e == cudaSuccess) {
        column_or_kernel<<<(unsigned)std::min<uint64_t>((n * arity + 255) / 256, 1216), 256>>>(d_tuples, n, arity, d_or);
        e = cudaMemcpy(h_or, d_or, sizeof h_or, cudaMemcpyDeviceToHost);
    }
    cudaFree(d_or);
    if (e != cudaSuccess) return fail(SGE_CUDA_ERROR, "sge_sort_tuples: %s", cudaGetErrorString(e));
    Widths w{};
    uint32_t bits = 0;
    for (uint32_t c = 0; c < arity; ++c) {
        w.bits[c] = h_or[c] ? (uint8_t)(32 - __builtin_clz(h_or[c])) : 0;
        bits += w.bits[c];
    }
    if (bits <= 64) return sort_packed<Key64>(d_tuples, n, arity, w, bits);
    if (bits <= 128) return sort_packed<Key128>(d_tuples, n, arity, w, bits);
    return sort_wide(d_tuples, n, arity, w);
}

// Trie levels of sorted tuples: level l has len[l] values (device array
// values[l]); node p of level l < arity-1 owns children
// [child[l][p], child[l][p+1]) of level l+1 (child[l] has len[l]+1 entries).
sge_status sge_trie_build(const uint32_t *d_sorted, uint64_t n, uint32_t arity, sge_trie *out) {
    if (!out || (!d_sorted && n) || arity == 0 || arity > SGE_TRIE_MAX_LEVELS)
        return fail(SGE_BAD_INPUT, "sge_trie_build: bad argument");
    memset(out, 0, sizeof *out);
    out->arity = arity;
    if (n == 0) return SGE_OK;
    if (n >= (1ull << 32)) return fail(SGE_UNSUPPORTED, "sge_trie_build: more than 2^32 rows");
    const uint32_t ntiles = (uint32_t)((n + TRIE_TILE - 1) / TRIE_TILE);
    uint32_t *counts = nullptr, totals[MAX_ARITY] = {};
    CUDA_TRY(cudaMalloc(&counts, ((size_t)arity * ntiles + MAX_ARITY) * 4));
    uint32_t *d_totals = counts + (size_t)arity * ntiles;
    trie_count_kernel<<<ntiles, 256>>>(d_sorted, n, arity, ntiles, counts);
    row_scan_kernel<<<arity, SORT_THREADS>>>(counts, ntiles, d_totals);
    cudaError_t e = cudaMemcpy(totals, d_totals, arity * 4, cudaMemcpyDeviceToHost);
    TriePtrs P{};
    for (uint32_t l = 0; l < arity && e == cudaSuccess; ++l) {
        out->level_len[l] = totals[l];
        e = cudaMalloc(&out->values[l], (size_t)totals[l] * 4);
        if (e == cudaSuccess && l + 1 < arity) e = cudaMalloc(&out->child[l], ((size_t)totals[l] + 1) * 8);
        P.values[l] = out->values[l];
        P.child[l] = out->child[l];
    }
    if (e == cudaSuccess) {
        trie_write_kernel<<<ntiles, 256>>>(d_sorted, n, arity, ntiles, counts, P);
        trie_ends_kernel<<<1, 32>>>(arity, d_totals, P);
        e = cudaGetLastError();
    }
    const cudaError_t e2 = cudaDeviceSynchronize();
    cudaFree(counts);
    if (e != cudaSuccess || e2 != cudaSuccess) {
        sge_trie_free(out);
        const cudaError_t err = e != cudaSuccess ? e : e2;
        return fail(err == cudaErrorMemoryAllocation ? SGE_OOM : SGE_CUDA_ERROR, "sge_trie_build: %s",
                    cudaGetErrorString(err));
    }
    return SGE_OK;
}

sge_status sge_trie_copy_level(const sge_trie *t, uint32_t level, uint32_t *values, unsigned long long *child) {
    if (!t || level >= t->arity || (!values && t->level_len[level])) return fail(SGE_BAD_INPUT, "sge_trie_copy_level: bad argument");
    const uint64_t n = t->level_len[level];
    if (n) CUDA_TRY(cudaMemcpy(values, t->values[level], n * 4, cudaMemcpyDeviceToHost));
    if (child && level + 1 < t->arity && t->child[level])
        CUDA_TRY(cudaMemcpy(child, t->child[level], (n + 1) * 8, cudaMemcpyDeviceToHost));
    return SGE_OK;
}

sge_status sge_trie_free(sge_trie *t) {
    if (!t) return SGE_OK;
    for (uint32_t l = 0; l < SGE_TRIE_MAX_LEVELS; ++l) {
        cudaFree(t->values[l]);
        cudaFree(t->child[l]);
        t->values[l] = nullptr;
        t->child[l] = nullptr;
    }
    return SGE_OK;
}

// The sorted instance set of a pattern (the embedding set -r writes; the
// reference never produces one): enumerate into a device buffer, canonicalise
// under the automorphisms, sort, copy to host.
sge_status sge_match_set(sge_graph *g, const sge_plan *p, uint32_t k, uint32_t m, const uint32_t *edges,
                         uint32_t *host_out, uint64_t cap_rows, uint64_t *n_rows) {
    if (!g || !p || !n_rows || (!host_out && cap_rows)) return fail(SGE_BAD_INPUT, "sge_match_set: null argument");
    // a buffer of the caller's own size is filled directly, unless it would
    // take much of the device: then the instances are counted first.  Without
    // room for a row the count alone answers (a random graph with 4M edges
    // and no gem: 4.2 ms, enumerated 8.7 ms)
    uint64_t inst = cap_rows, n2 = 0;
    auto count = [&]() {   // SGE_OK: the output has room for them
        uint64_t counts = 0;
        const sge_plan *pp = p;
        const sge_status st = sge_count(g, &pp, 1, nullptr, &counts, &inst, nullptr);
        if (st != SGE_OK) return st;
        *n_rows = inst;
        if (inst > cap_rows) return fail(SGE_OOM, "%llu instances exceed the %llu-row output", (unsigned long long)inst,
                                         (unsigned long long)cap_rows);
        return SGE_OK;
    };
    size_t free_b = 0, tot_b = 0;
    CUDA_TRY(cudaMemGetInfo(&free_b, &tot_b));
    const bool counted = cap_rows == 0 || cap_rows > std::min<uint64_t>(1ull << 30, free_b / 8) / (4ull * std::max<uint32_t>(k, 1));
    if (counted) {
        const sge_status cst = count();
        if (cst != SGE_OK || inst == 0) return cst;
    }
    uint32_t *d = nullptr;
    if (inst) CUDA_TRY(cudaMalloc(&d, inst * k * 4ull));
    sge_status st = enumerate_rows(g, p, d, inst, &n2, true);
    if (counted && st == SGE_OK && n2 != inst)
        st = fail(SGE_CUDA_ERROR, "enumeration produced %llu rows but the count is %llu", (unsigned long long)n2,
                  (unsigned long long)inst);
    if (!counted && st != SGE_OK && st != SGE_OOM) {
        // a plan that cannot be enumerated is an error where there are rows to write
        cudaFree(d);
        const sge_status cst = count();
        return cst == SGE_OK && inst ? st : cst;
    }
    if (!counted) {
        *n_rows = inst = n2;
        if (n2 > cap_rows) st = fail(SGE_OOM, "%llu instances exceed the %llu-row output", (unsigned long long)n2,
                                     (unsigned long long)cap_rows);
    }
    if (st != SGE_OK || inst == 0) {
        cudaFree(d);
        return st;
    }
    std::vector<uint8_t> perms((size_t)4096 * k);
    uint32_t naut = 0;
    if (st == SGE_OK) st = sge_pattern_automorphisms(k, m, edges, perms.data(), 4096, &naut);
    if (st == SGE_OK) st = sge_canonicalize(d, inst, k, perms.data(), naut);
    if (st == SGE_OK) st = sge_sort_tuples(d, inst, k);
    if (st == SGE_OK && cudaMemcpy(host_out, d, inst * k * 4ull, cudaMemcpyDeviceToHost) != cudaSuccess)
        st = fail(SGE_CUDA_ERROR, "sge_match_set: copy-out failed");
    cudaFree(d);
    return st;
}

}  // extern "C"
