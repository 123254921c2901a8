// CSR -> condensed row-window tiles on the GPU.  Same output, bit for bit, as the host converter
// (format.cpp) and therefore as the reference's CSR2BTCFNOBITMAP (src/utils/convert.h:146-225),
// for CSR whose rows hold ascending, distinct columns (what the reference's loader produces,
// src/utils/load.h:137-145,256).  The reference converts on one host thread; the largest
// benchmark matrix (5.2e8 entries) takes ten seconds on sixteen host cores and well under one on
// the device.
//
// A matrix of up to 744,000 columns is converted window by window: a warp sorts the entries of a window in registers, or, where
// they are more than kWarpEntries, a block marks their columns in a bit set in shared memory; either way an entry learns how many
// distinct columns lie below its own, which is its place in the window's tiles.  One scan over the windows says where those
// begin, and a pass over the entries writes column lists and values.
//
// Steps otherwise (all integer work, bound by HBM traffic):
//   1. one key (window, column) per entry, in as few bits as the matrix needs - 32-bit keys where they fit - since
//      every eight bits are a pass of the sort; the entry's row is found by binary search in row_ptr
//   2. radix sort of the keys, then unique -> the sorted distinct columns of every window
//      (CUB device primitives: sort, select-unique, scan)
//   3. every window finds its range of them by binary search; one scan of (holds entries, tiles) gives
//      rowOffset, rowIdx and all sizes.  The host waits for the device once on the way, for those sizes: a
//      wait in each step (entries, distinct columns, windows, tiles) left the device idle for 80 of 290 us on
//      a matrix of 700,000 entries.
//   4. column lists scattered into tcA2B (pre-filled with 0xFFFFFFFF padding); every entry finds its slot by binary search in its
//      window's column list and is written into the zero-filled tile array
#include <algorithm>
#include <cstdint>
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>
#include <new>

#include "../../include/b200_spmm.h"
#include "common.hpp"
#include "device_pool.hpp"
#include "format.hpp"

struct b200spmm_dbtcf {
    b200spmm_btcf_info_t info{};
    int device = 0;
    uint32_t *d_rowOffset = nullptr, *d_tcA2B = nullptr, *d_rowIdx = nullptr;
    void *d_data = nullptr;
};

namespace b200spmm {
namespace gpuconv {

constexpr int kBlock = 256;

constexpr uint32_t kKeyEntries = 4 * kBlock;  // entries a block takes at a time in make_keys_kernel

// last row r in [lo, hi) with row_ptr[r] <= p, or lo
__device__ __forceinline__ uint32_t row_of_entry(const uint32_t *__restrict__ row_ptr, uint32_t lo, uint32_t hi, uint32_t p) {
    while (hi - lo > 1) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (row_ptr[mid] <= p) lo = mid; else hi = mid;
    }
    return lo;
}

// The last window whose first entry is p or one before it, found by a whole warp: 32 windows at a time.
__device__ __forceinline__ uint32_t window_of_entry(const uint32_t *__restrict__ row_ptr, uint32_t n_windows, uint32_t row_window, uint32_t p) {
    uint32_t lo = 0, hi = n_windows;  // row_ptr[lo * row_window] <= p, and behind hi - 1 none
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32, w = lo + (threadIdx.x & 31u) * step;
        const uint32_t below = __ballot_sync(0xffffffffu, w < hi && (w == lo || row_ptr[w * row_window] <= p));
        lo += (31u - (uint32_t)__clz((int)below)) * step;  // (lane 0 is always there)
        hi = min(hi, lo + step);
    }
    return lo;
}

struct Totals {
    uint64_t n_unique;
    unsigned long long windows_tiles;  // windows that hold entries << 32 | their tiles
    uint32_t bad, hubs, long_windows;
};

// keys[p] = window(p) << col_bits | col[p]; flags row pointers that do not run from 0 to nnz, a column out
// of range or a row whose columns are not strictly ascending.  Neighbouring entries lie in few rows: a block searches
// the whole of row_ptr for its first and last entry only.
template <typename K>
__global__ void __launch_bounds__(kBlock)
make_keys_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ col_idx, uint32_t rows, uint32_t cols, uint64_t nnz,
                 uint32_t row_window, int col_bits, K *__restrict__ keys, Totals *__restrict__ totals) {
    __shared__ uint32_t range[2];
    if (blockIdx.x == 0 && threadIdx.x == 0 && (row_ptr[0] != 0 || row_ptr[rows] != nnz)) atomicOr(&totals->bad, 1u);
    for (uint64_t p0 = (uint64_t)blockIdx.x * kKeyEntries; p0 < nnz; p0 += (uint64_t)gridDim.x * kKeyEntries) {
        const uint64_t p1 = min(p0 + kKeyEntries, nnz);
        __syncthreads();
        if (threadIdx.x < 2) range[threadIdx.x] = row_of_entry(row_ptr, 0, rows, (uint32_t)(threadIdx.x ? p1 - 1 : p0));
        __syncthreads();
        const uint32_t first = range[0], end = max(range[1], first) + 1;
        for (uint64_t p = p0 + threadIdx.x; p < p1; p += kBlock) {
            const uint32_t r = row_of_entry(row_ptr, first, end, (uint32_t)p), c = col_idx[p], start = row_ptr[r];
            if (c >= cols || p < start || p >= row_ptr[r + 1] || (p > start && col_idx[p - 1] >= c)) atomicOr(&totals->bad, 1u);
            keys[p] = ((K)(r / row_window) << col_bits) | c;
        }
    }
}

// first[w] = distinct (window, column) pairs of the windows before w
template <typename K>
__global__ void window_bounds_kernel(const K *__restrict__ ukeys, const Totals *__restrict__ totals, uint32_t n_windows, int col_bits,
                                     uint32_t *__restrict__ first) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w > n_windows) return;
    uint32_t lo = 0, hi = totals->bad ? 0u : (uint32_t)totals->n_unique;  // (the keys of a bad matrix need not be sorted)
    if (w == n_windows) lo = hi;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (ukeys[mid] < (K)w << col_bits) lo = mid + 1; else hi = mid;
    }
    first[w] = lo;
}

constexpr int kBitsBlock = 1024;
constexpr size_t kBitsSmemMax = 125 * 1024, kSetsSmemMax = 220 * 1024;  // one set, the sets of a block
constexpr uint32_t kGroupWords = 8;  // words of the bit set that share a rank

inline uint32_t bit_words(uint64_t cols) { return (uint32_t)((cols + 32 * kGroupWords - 1) / (32 * kGroupWords)) * kGroupWords; }
// the set, how many columns lie below a word in its group (a byte), and below a group
inline size_t bits_smem(uint64_t cols) { return ((size_t)bit_words(cols) * 5 + (size_t)(bit_words(cols) / kGroupWords) * 4 + 15) / 16 * 16; }

// What a column needs of a key beside the row (4 bits) and the entry (8 bits), or the entry alone (9 bits), see sort_window.
constexpr uint32_t kKeyCols = (1u << 20) - 1u;
static_assert(kBitsSmemMax / 11 * 2 * 32 < kKeyCols, "a column of the largest set fits a key");

// The windows, where a block has room for a set.  Conversion of graphs in us, windows against the sort of all entries (four or
// more passes of ~20 bytes an entry): 157 / 276 for 1.8e6 in 262,144, 960 / 1,560 for 10.4e6 in 524,288.
inline bool by_windows_pays(uint64_t cols) { return bits_smem(cols) <= kBitsSmemMax; }

// What the kernels of the windows read and write.
struct WindowArgs {
    const uint32_t *row_ptr, *col_idx;
    uint32_t rows, cols, nnz, n_windows, row_window, log_cw, words;
    uint32_t *places, *count;  // an entry's place in its window's tiles (tile, row, column), a window's distinct columns
    uint32_t *listed;  // (the scan's output before it is written) windows for blocks: the longest from the front, others from the back
    Totals *totals;
    __device__ __forceinline__ uint32_t place(uint32_t column, uint32_t row) const {  // fewer than 2^24: 2^20 columns, 16 rows
        return (((column >> log_cw) * row_window + row) << log_cw) | (column & ((1u << log_cw) - 1u));
    }
    // Lane k: the first entry of row k of window w, from row_window on the end of the last one.  False for all lanes if they are none.
    __device__ __forceinline__ bool starts(uint32_t w, uint32_t lane, uint32_t *start) const {
        *start = row_ptr[min((uint64_t)w * row_window + min(lane, row_window), (uint64_t)rows)];
        const uint32_t prev = __shfl_up_sync(0xffffffffu, *start, 1);
        return __all_sync(0xffffffffu, *start <= nnz && (lane == 0 || prev <= *start));
    }
    // the last row that starts at entry p or before it (for a whole warp)
    __device__ __forceinline__ uint32_t row_of(uint64_t p, uint32_t start) const {
        uint32_t r = 0;
#pragma unroll
        for (uint32_t step = 8; step; step /= 2) {
            const uint32_t s = __shfl_sync(0xffffffffu, start, (int)(r + step));
            if (r + step < row_window && s <= p) r += step;
        }
        return r;
    }
};

constexpr uint32_t kHubEntries = 4096;
// Entries of a window that a warp sorts.
template <bool kWide>
constexpr uint32_t kWarpEntries = kWide ? 512 : 256;

// A warp's window of up to 32 * kN entries, one key of column, row and entry each: a bitonic sort over the places lane * kN + k,
// the strides below kN within a lane.  (A key has no room for the row of one of 512 entries, which is looked up again.)
template <int kN>
__device__ __forceinline__ void sort_window(const WindowArgs &a, uint32_t w, uint32_t lane, uint32_t start, uint32_t p0, uint32_t n) {
    constexpr bool kRowInKey = kN <= 8;
    constexpr int kEntryBits = kRowInKey ? 8 : 9, kColumnAt = kRowInKey ? 12 : 9;
    uint32_t key[kN], before = 0, row_before = 0xFFFFFFFFu;  // column and row of the entry before the first one of a step
    bool bad = false;
#pragma unroll
    for (int k = 0; k < kN; ++k) key[k] = k * 32 + lane < n ? a.col_idx[p0 + k * 32 + lane] : 0xFFFFFFFFu;
#pragma unroll
    for (int k = 0; k < kN; ++k) {
        const uint32_t i = k * 32 + lane, c = key[k], r = a.row_of((uint64_t)p0 + i, start);
        uint32_t left = __shfl_up_sync(0xffffffffu, c, 1), left_row = __shfl_up_sync(0xffffffffu, r, 1);
        if (lane == 0) left = before, left_row = row_before;
        before = __shfl_sync(0xffffffffu, c, 31);
        row_before = __shfl_sync(0xffffffffu, r, 31);
        const bool live = i < n, fits = c < a.cols;
        bad |= live && (!fits || (left_row == r && left >= c));
        key[k] = live && fits ? c << kColumnAt | (kRowInKey ? r << kEntryBits : 0u) | i : 0xFFFFFFFFu;
    }
    if (__any_sync(0xffffffffu, bad)) {
        if (lane == 0) {
            a.count[w] = 0;
            atomicOr(&a.totals->bad, 1u);
        }
        return;
    }
#pragma unroll
    for (int size = 2; size <= 32 * kN; size *= 2) {
#pragma unroll
        for (int stride = size / 2; stride; stride /= 2) {
            if (stride >= kN) {
                // of two lanes, the one with the lower place keeps the smaller key in a rising run
                const bool smaller = ((lane & (uint32_t)(stride / kN)) == 0) == ((lane & (uint32_t)(size / kN)) == 0);
#pragma unroll
                for (int k = 0; k < kN; ++k) {
                    const uint32_t other = __shfl_xor_sync(0xffffffffu, key[k], stride / kN);
                    key[k] = smaller ? min(key[k], other) : max(key[k], other);
                }
            } else {
#pragma unroll
                for (int k = 0; k < kN; ++k) {
                    if (k & stride) continue;
                    const bool rising = size < kN ? (k & size) == 0 : (lane & (uint32_t)(size / kN)) == 0;
                    const uint32_t lo = min(key[k], key[k + stride]), hi = max(key[k], key[k + stride]);
                    key[k] = rising ? lo : hi;
                    key[k + stride] = rising ? hi : lo;
                }
            }
        }
    }
    uint32_t prev = __shfl_up_sync(0xffffffffu, key[kN - 1], 1), mine = 0;
    if (lane == 0) prev = 0xFFFFFFFFu;  // (no entry's column)
    bool first[kN];
#pragma unroll
    for (int k = 0; k < kN; ++k) {
        first[k] = lane * kN + k < n && key[k] >> kColumnAt != prev >> kColumnAt;
        prev = key[k];
        mine += first[k];
    }
    uint32_t upto = mine;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= (uint32_t)d) upto += x;
    }
    if (lane == 31) a.count[w] = upto;
    uint32_t at = upto - mine - 1;  // (of the column before: a column's first entry steps on)
#pragma unroll
    for (int k = 0; k < kN; ++k) {
        at += first[k];
        const uint32_t entry = key[k] & ((1u << kEntryBits) - 1u);
        const uint32_t r = kRowInKey ? key[k] >> kEntryBits & 15u : a.row_of((uint64_t)p0 + entry, start);
        if (lane * kN + k < n) a.places[p0 + entry] = a.place(at, r);
    }
}

// A window a warp.  `clear`: the tile array, zeroed on the way where it is there already.  A median window of a graph has a few
// dozen entries: sorted by a warp that is some hundred instructions, marked in a set by a block of 256 threads it is 5,500,
// most of them to clear and to count an empty set (60,000 nodes, 720,000 entries: 40 us; this kernel takes 9 with the zeroing of
// 24 MB, the one for long windows 18 - 21).
//
// kWide: windows of up to 512 entries, for matrices of so many columns (655,361 and more) that a block has room for one set alone.
// There a window of just over 256 entries waits for a set of 110 KB to be cleared and counted, 5.6 us of an SM: 660,000 nodes, 17 /
// 20 / 30 entries a node 2,230 / 2,310 / 2,670 us, so 1,000 / 1,080 / 1,370 (through the sort of all entries 1,660 / 1,840 / 4,700).  Where
// two sets and more fit, the wide kernel's code costs a small matrix more than that: a graph of 2,000 nodes 70 -> 80, of 60,000 96 -> 104.
constexpr int kSortBlock = 256;
template <bool kWide>
__global__ void __launch_bounds__(kSortBlock, 4)
window_sort_kernel(const WindowArgs a, uint4 *__restrict__ clear, uint64_t n_clear) {
    const uint32_t lane = threadIdx.x & 31u;
    if (blockIdx.x == 0 && threadIdx.x == 0 && (a.row_ptr[0] != 0 || a.row_ptr[a.rows] != a.nnz)) atomicOr(&a.totals->bad, 1u);
    for (uint64_t w64 = (uint64_t)blockIdx.x * (kSortBlock / 32) + (threadIdx.x >> 5); w64 < a.n_windows; w64 += (uint64_t)gridDim.x * (kSortBlock / 32)) {
        const uint32_t w = (uint32_t)w64;
        uint32_t start;
        const bool ok = a.starts(w, lane, &start);
        const uint32_t p0 = __shfl_sync(0xffffffffu, start, 0), n = ok ? __shfl_sync(0xffffffffu, start, 31) - p0 : 0;
        if (n == 0) {
            if (lane == 0) {
                a.count[w] = 0;
                if (!ok) atomicOr(&a.totals->bad, 1u);
            }
        } else if (n <= 64) {
            sort_window<2>(a, w, lane, start, p0, n);
        } else if (n <= 128) {
            sort_window<4>(a, w, lane, start, p0, n);
        } else if (n <= 256) {
            sort_window<8>(a, w, lane, start, p0, n);
        } else if (n <= kWarpEntries<kWide>) {
            if constexpr (kWide) sort_window<16>(a, w, lane, start, p0, n);
        } else if (lane == 0) {
            const bool hub = n > kHubEntries;
            const uint32_t k = atomicAdd(hub ? &a.totals->hubs : &a.totals->long_windows, 1u);
            a.listed[hub ? k : a.n_windows - 1 - k] = w;
        }
    }
    for (uint64_t k = (uint64_t)blockIdx.x * kSortBlock + threadIdx.x; k < n_clear; k += (uint64_t)gridDim.x * kSortBlock)
        clear[k] = make_uint4(0, 0, 0, 0);
}

// A listed window by `threads` threads of the block (t of them this one), which have barrier `bar` and a set for themselves.
__device__ __forceinline__ void mark_window(const WindowArgs &a, uint32_t w, uint32_t t, uint32_t threads, uint32_t bar, uint32_t *bits, uint32_t *sums) {
    constexpr uint32_t kUnroll = 4;  // columns of a thread in flight
    auto sync = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(bar), "r"(threads) : "memory"); };
    const uint32_t lane = t & 31u, warp = t >> 5, groups = a.words / kGroupWords;
    uint32_t *rank = bits + a.words;  // columns in the groups before
    uint8_t *in_group = reinterpret_cast<uint8_t *>(rank + groups);
    uint32_t start;
    a.starts(w, lane, &start);  // (every warp for itself; a window is listed if they are in order)
    const uint32_t p0 = __shfl_sync(0xffffffffu, start, 0), n = __shfl_sync(0xffffffffu, start, 31) - p0;
    const uint32_t *col = a.col_idx + p0;
    start = lane < a.row_window ? start - p0 : 0xFFFFFFFFu;
    for (uint32_t i = t; i < a.words / 4; i += threads) reinterpret_cast<uint4 *>(bits)[i] = make_uint4(0, 0, 0, 0);
    sync();
    for (uint32_t i0 = t & ~31u; i0 < n; i0 += kUnroll * threads) {  // of the warp's first lane
        uint32_t c[kUnroll], left[kUnroll];
#pragma unroll
        for (uint32_t j = 0; j < kUnroll; ++j) {
            const uint32_t i = i0 + j * threads + lane;
            const bool live = j * threads < n - i0 && lane < n - i0 - j * threads;
            c[j] = live ? col[i] : 0xFFFFFFFFu;
            left[j] = live && lane == 0 && i ? col[i - 1] : 0u;
        }
#pragma unroll
        for (uint32_t j = 0; j < kUnroll; ++j) {
            if (j * threads >= n - i0) break;  // (the whole warp)
            const uint32_t i = i0 + j * threads + lane, of_left = __shfl_up_sync(0xffffffffu, c[j], 1);
            if (lane) left[j] = of_left;
            if (c[j] < a.cols) atomicOr(bits + (c[j] >> 5), 1u << (c[j] & 31u));
            if (i && left[j] >= c[j] && i < n) {  // only where a row starts
                bool row_start = false;
                for (uint32_t r = 1; r < a.row_window; ++r) row_start |= a.row_ptr[min((uint64_t)w * a.row_window + r, (uint64_t)a.rows)] == p0 + i;
                if (!row_start) atomicOr(&a.totals->bad, 1u);
            }
            if (c[j] >= a.cols && lane < n - i0 - j * threads) atomicOr(&a.totals->bad, 1u);
        }
        if (n - i0 <= kUnroll * threads) break;  // (the sum may not fit)
    }
    sync();
    uint32_t base = 0;
    for (uint32_t g0 = 0; g0 < groups; g0 += threads) {  // one group a thread
        const uint32_t g = g0 + t;
        uint32_t mine = 0;
        if (g < groups) {
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint4 b = reinterpret_cast<const uint4 *>(bits)[2 * g + h];
                const uint32_t word[4] = {b.x, b.y, b.z, b.w};
                uint32_t below = 0;
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    below |= mine << (8 * j);  // (224 at most)
                    mine += (uint32_t)__popc(word[j]);
                }
                reinterpret_cast<uint32_t *>(in_group)[2 * g + h] = below;
            }
        }
        uint32_t upto = mine;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= (uint32_t)d) upto += x;
        }
        if (g0) sync();  // `sums` of the round before has been read
        if (lane == 31) sums[warp] = upto;
        sync();
        const uint32_t of_lane = lane < threads / 32 ? sums[lane] : 0u;
        const uint32_t before = base + __reduce_add_sync(0xffffffffu, lane < warp ? of_lane : 0u);
        base += __reduce_add_sync(0xffffffffu, of_lane);
        if (g < groups) rank[g] = before + upto - mine;
    }
    sync();
    for (uint32_t i0 = t & ~31u; i0 < n; i0 += kUnroll * threads) {
        uint32_t c[kUnroll];
#pragma unroll
        for (uint32_t j = 0; j < kUnroll; ++j)
            c[j] = j * threads < n - i0 && lane < n - i0 - j * threads ? col[i0 + j * threads + lane] : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t j = 0; j < kUnroll; ++j) {
            if (j * threads >= n - i0) break;
            // the rows that start at the warp's first entry or before it; most often all of its entries are of the last one
            const uint32_t first = i0 + j * threads, rows = __ballot_sync(0xffffffffu, start <= first);
            uint32_t r = 31u - (uint32_t)__clz((int)rows);
            if (__any_sync(0xffffffffu, start > first && start - first < 32)) r = a.row_of(first + lane, start);
            const uint32_t word = c[j] >> 5;
            if (c[j] < a.cols)
                a.places[p0 + first + lane] = a.place(rank[word / kGroupWords] + in_group[word] + (uint32_t)__popc(bits[word] & ((1u << (c[j] & 31u)) - 1u)), r);
        }
        if (n - i0 <= kUnroll * threads) break;
    }
    if (t == 0) a.count[w] = base;
    sync();  // the next window clears the set
}

// The longest windows by a block each, of the others up to `most_parts` at a time.  Bound by the chain of a window - row
// pointers, columns, marks, ranks, columns, places, a barrier after each - and by the longest one: 20,000 entries of a graph's
// 720,000 take 20 us of one SM, where the others are done in 9.  Two blocks an SM, of 32 registers a thread, spill (23 us); lanes
// that put the bits of one word together before the atomics cost more than the conflicts (23).
__global__ void __launch_bounds__(kBitsBlock, 1)
window_marks_kernel(const WindowArgs a, uint32_t most_parts, uint32_t set_words) {
    extern __shared__ __align__(16) uint32_t sets[];
    __shared__ uint32_t sums[4][32];
    const uint32_t hubs = a.totals->hubs, n_long = a.totals->long_windows;
    for (uint32_t k = blockIdx.x; k < hubs; k += gridDim.x) mark_window(a, a.listed[k], threadIdx.x, kBitsBlock, 0, sets, sums[0]);
    uint32_t parts = most_parts;
    while (parts > 1 && n_long <= gridDim.x * (parts / 2)) parts /= 2;
    const uint32_t threads = kBitsBlock / parts, part = threadIdx.x / threads;
    // from the last block on: the first ones have the longest windows
    for (uint64_t k = (uint64_t)(gridDim.x - 1 - blockIdx.x) * parts + part; k < n_long; k += (uint64_t)gridDim.x * parts)
        mark_window(a, a.listed[a.n_windows - 1 - (uint32_t)k], threadIdx.x % threads, threads, 1 + part, sets + part * set_words, sums[part]);
}

// The window's terms of the scan.  Fewer than 2^32 entries make fewer than 2^30 full tiles, 2^29 windows as many more.
struct WindowTerms {
    const uint32_t *first, *count;  // one of the two
    uint32_t n_windows, col_window;
    __host__ __device__ uint32_t columns_of(uint32_t w) const { return count ? count[w] : first[w + 1] - first[w]; }
    __host__ __device__ unsigned long long operator()(uint32_t w) const {
        if (w >= n_windows) return 0;
        const uint32_t n = columns_of(w);
        return (unsigned long long)(n != 0) << 32 | ((unsigned long long)n + col_window - 1) / col_window;
    }
};

__global__ void window_tables_kernel(const unsigned long long *__restrict__ before, uint32_t n_windows,
                                     uint32_t row_window, uint32_t *__restrict__ rowOffset, uint32_t *__restrict__ rowIdx,
                                     uint32_t *__restrict__ tile_of, Totals *__restrict__ totals) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w > n_windows) return;
    const uint32_t e = (uint32_t)(before[w] >> 32), tile = (uint32_t)before[w];
    if (w == n_windows) {
        rowOffset[e] = tile;
        totals->windows_tiles = before[w];
        return;
    }
    tile_of[w] = tile;
    if ((uint32_t)(before[w + 1] >> 32) == e) return;
    rowOffset[e] = tile;
    rowIdx[e] = w * row_window;
}

// The same scan and tables by one block, a load, a sum and a store for each 4,096 windows: 6 us for 3,750 of them, where the two
// launches of the scan and the tables took 14.
constexpr int kScanBlock = 1024;
constexpr uint32_t kScanPer = 4, kOneBlockWindows = 16384;
__global__ void __launch_bounds__(kScanBlock)
scan_tables_kernel(const uint32_t *__restrict__ count, uint32_t n_windows, uint32_t row_window, uint32_t col_window,
                   uint32_t *__restrict__ rowOffset, uint32_t *__restrict__ rowIdx, uint32_t *__restrict__ tile_of, Totals *__restrict__ totals) {
    __shared__ unsigned long long warp_sums[kScanBlock / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    unsigned long long base = 0;
    const WindowTerms terms{nullptr, count, n_windows, col_window};
    for (uint32_t w0 = 0; w0 < n_windows; w0 += kScanBlock * kScanPer) {
        const uint32_t w = w0 + threadIdx.x * kScanPer;
        unsigned long long term[kScanPer], upto = 0;
#pragma unroll
        for (uint32_t k = 0; k < kScanPer; ++k) {
            term[k] = terms(w + k);
            upto += term[k];
        }
        const unsigned long long mine = upto;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const unsigned long long x = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= (uint32_t)d) upto += x;
        }
        if (w0) __syncthreads();  // the sums of the round before have been read
        if (lane == 31) warp_sums[warp] = upto;
        __syncthreads();
        const unsigned long long of_lane = warp_sums[lane];  // (as many warps as lanes)
        unsigned long long warps = of_lane;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const unsigned long long x = __shfl_up_sync(0xffffffffu, warps, d);
            if (lane >= (uint32_t)d) warps += x;
        }
        unsigned long long at = base + upto - mine + __shfl_sync(0xffffffffu, warps - of_lane, (int)warp);
        base += __shfl_sync(0xffffffffu, warps, 31);
#pragma unroll
        for (uint32_t k = 0; k < kScanPer; ++k) {
            if (w + k >= n_windows) break;
            tile_of[w + k] = (uint32_t)at;
            if (term[k]) {
                rowOffset[at >> 32] = (uint32_t)at;
                rowIdx[at >> 32] = (w + k) * row_window;
            }
            at += term[k];
        }
    }
    if (threadIdx.x == 0) {
        rowOffset[base >> 32] = (uint32_t)base;
        totals->windows_tiles = base;
    }
}
static_assert(kScanBlock / 32 == 32, "a lane for every warp's sum");

// Entry p's column and value at its place; the list's slots without a column.  10 us for 720,000 entries; the columns listed
// first, and every entry searching its column there, took 24.  A block takes kKeyEntries entries at a time
// and looks for the windows of the first and the last of them.
template <typename T>
__global__ void __launch_bounds__(kBlock)
place_entries_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ col_idx, const T *__restrict__ values,
                     const uint32_t *__restrict__ places, const uint32_t *__restrict__ count, const uint32_t *__restrict__ tile_of,
                     const Totals *__restrict__ totals, uint32_t nnz, uint32_t n_windows, uint32_t row_window, uint32_t log_cw,
                     uint32_t *__restrict__ tcA2B, T *__restrict__ data) {
    __shared__ uint32_t range[2];
    if (totals->bad) return;  // (places are missing, and the windows need not hold the entries)
    const uint32_t cw = 1u << log_cw, log_tile = log_cw + (row_window == 16 ? 4 : 3);
    for (uint64_t w = (uint64_t)blockIdx.x * kBlock + threadIdx.x; w < n_windows; w += (uint64_t)gridDim.x * kBlock) {
        const uint32_t n = count[w], padded = (n + cw - 1) & ~(cw - 1);
        for (uint32_t k = n; k < padded; ++k) tcA2B[((uint64_t)tile_of[w] << log_cw) + k] = 0xFFFFFFFFu;
    }
    for (uint64_t p0 = (uint64_t)blockIdx.x * kKeyEntries; p0 < nnz; p0 += (uint64_t)gridDim.x * kKeyEntries) {
        const uint32_t n = (uint32_t)min((uint64_t)kKeyEntries, nnz - p0);
        __syncthreads();
        if (threadIdx.x < 64) {
            const uint32_t w = window_of_entry(row_ptr, n_windows, row_window, (uint32_t)p0 + (threadIdx.x < 32 ? 0u : n - 1));
            if (threadIdx.x % 32 == 0) range[threadIdx.x / 32] = w;
        }
        __syncthreads();
        const uint32_t first = range[0], end = range[1] + 1;
#pragma unroll
        for (uint32_t k = 0; k < kKeyEntries / kBlock; ++k) {
            const uint32_t i = k * kBlock + threadIdx.x;
            if (i >= n) break;
            const uint32_t p = (uint32_t)p0 + i, place = places[p], c = col_idx[p];
            const T v = values[p];
            uint32_t lo = first, hi = end;
            while (hi - lo > 1) {
                const uint32_t mid = lo + (hi - lo) / 2;
                if (row_ptr[mid * row_window] <= p) lo = mid; else hi = mid;
            }
            const uint64_t tile0 = tile_of[lo];
            data[(tile0 << log_tile) + place] = v;
            tcA2B[((tile0 + (place >> log_tile)) << log_cw) + (place & (cw - 1))] = c;  // (as every other entry of the column)
        }
    }
}

// distinct column j (sorted by window, column) -> its place in the window's padded column list
template <typename K>
__global__ void scatter_columns_kernel(const K *__restrict__ ukeys, uint64_t n_unique, int col_bits, const uint32_t *__restrict__ first,
                                       const uint32_t *__restrict__ tile_of, uint32_t col_window, uint32_t *__restrict__ tcA2B) {
    for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n_unique; j += (uint64_t)gridDim.x * blockDim.x) {
        const K k = ukeys[j];
        const uint32_t w = (uint32_t)(k >> col_bits);
        tcA2B[(uint64_t)tile_of[w] * col_window + (j - first[w])] = (uint32_t)(k & (((K)1 << col_bits) - 1));
    }
}

// entry p -> its slot in the zero-filled tile array
template <typename T>
__global__ void __launch_bounds__(kBlock)
scatter_values_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ col_idx, const T *__restrict__ values, uint32_t rows,
                      uint64_t nnz, WindowTerms windows, const uint32_t *__restrict__ tile_of, const uint32_t *__restrict__ tcA2B,
                      uint32_t row_window, uint32_t col_window, T *__restrict__ data) {
    __shared__ uint32_t range[2];
    for (uint64_t p0 = (uint64_t)blockIdx.x * kKeyEntries; p0 < nnz; p0 += (uint64_t)gridDim.x * kKeyEntries) {
        const uint64_t p1 = min(p0 + kKeyEntries, nnz);
        __syncthreads();
        if (threadIdx.x < 2) range[threadIdx.x] = row_of_entry(row_ptr, 0, rows, (uint32_t)(threadIdx.x ? p1 - 1 : p0));
        __syncthreads();
        const uint32_t first = range[0], end = range[1] + 1;
        for (uint64_t p = p0 + threadIdx.x; p < p1; p += kBlock) {
            const uint32_t r = row_of_entry(row_ptr, first, end, (uint32_t)p), c = col_idx[p], w = r / row_window, tile0 = tile_of[w];
            const uint32_t *list = tcA2B + (uint64_t)tile0 * col_window;
            uint32_t lo = 0, hi = windows.columns_of(w);  // the window's real columns are ascending; padding follows them
            while (lo < hi) {
                const uint32_t mid = lo + (hi - lo) / 2;
                if (list[mid] < c) lo = mid + 1; else hi = mid;
            }
            const uint64_t tile = (uint64_t)tile0 + lo / col_window;
            data[tile * row_window * col_window + (uint64_t)(r % row_window) * col_window + lo % col_window] = values[p];
        }
    }
}

inline int grid_for(uint64_t n) { return (int)std::min<uint64_t>((n + kBlock - 1) / kBlock, 148 * 32); }

void scatter_values(const b200spmm_dbtcf *f, const uint32_t *d_row_ptr, const uint32_t *d_col_idx, const void *d_values,
                    const WindowTerms &windows, const uint32_t *tile_of, cudaStream_t stream) {
    const auto &i = f->info;
    const int grid = (int)std::min<uint64_t>((i.nnzs + kKeyEntries - 1) / kKeyEntries, 148 * 32);
    if (i.elt_size == 2)
        scatter_values_kernel<uint16_t><<<grid, kBlock, 0, stream>>>(d_row_ptr, d_col_idx, static_cast<const uint16_t *>(d_values),
                                                                     (uint32_t)i.rows, i.nnzs, windows, tile_of, f->d_tcA2B,
                                                                     (uint32_t)i.row_window, (uint32_t)i.col_window, static_cast<uint16_t *>(f->d_data));
    else
        scatter_values_kernel<uint32_t><<<grid, kBlock, 0, stream>>>(d_row_ptr, d_col_idx, static_cast<const uint32_t *>(d_values),
                                                                     (uint32_t)i.rows, i.nnzs, windows, tile_of, f->d_tcA2B,
                                                                     (uint32_t)i.row_window, (uint32_t)i.col_window, static_cast<uint32_t *>(f->d_data));
}

// Up to this size the tile array is made ahead, as large as it can become (no column shared by two entries, or every column in
// every window): it is cleared while the places are found, and the host waits once instead of twice (about 12 us of 80).  Without
// the second bound, and cleared by the blocks of the windows alone, dense matrices had several times their tiles cleared and held:
// pruned 1024 x 4096 / 2000 x 2000 at 30 % 166 / 118 us (113 / 105 with two waits), now 80 / 78.  Where windows share columns by
// blocks the array stays too large; moving what is used to one of its size took 20 to 30 of 110 us and gave the pool, which maps 64
// MB at a time, nothing to return.
constexpr uint64_t kAheadBytes = (uint64_t)64 << 20;

template <typename T>
void place_entries(const b200spmm_dbtcf *f, const uint32_t *d_row_ptr, const uint32_t *d_col_idx, const void *d_values, const uint32_t *places,
                   const uint32_t *count, const uint32_t *tile_of, const Totals *totals, uint32_t log_cw, cudaStream_t stream) {
    const auto &i = f->info;
    const int grid = (int)std::min<uint64_t>((i.nnzs + kKeyEntries - 1) / kKeyEntries, 148 * 32);
    place_entries_kernel<T><<<grid, kBlock, 0, stream>>>(d_row_ptr, d_col_idx, static_cast<const T *>(d_values), places, count, tile_of, totals,
                                                         (uint32_t)i.nnzs, (uint32_t)i.total_row_windows, (uint32_t)i.row_window, log_cw,
                                                         f->d_tcA2B, static_cast<T *>(f->d_data));
}

int convert_by_windows(b200spmm_dbtcf *f, const uint32_t *d_row_ptr, const uint32_t *d_col_idx, const void *d_values, cudaStream_t stream) {
    const uint32_t rows = (uint32_t)f->info.rows, cols = (uint32_t)f->info.cols, nnz = (uint32_t)f->info.nnzs;
    const uint32_t n_windows = (uint32_t)f->info.total_row_windows, RW = (uint32_t)f->info.row_window, CW = (uint32_t)f->info.col_window;
    const uint32_t log_cw = CW == 16 ? 4 : CW == 8 ? 3 : 2;
    const size_t smem = bits_smem(f->info.cols);
    const uint64_t tile_bytes = (uint64_t)RW * CW * f->info.elt_size;
    PoolScratch tmp(stream);
    Totals *totals = nullptr;
    uint32_t *places = nullptr, *count = nullptr, *tile_of = nullptr;
    B200_CUDA_TRY(tmp.alloc(&places, nnz));
    B200_CUDA_TRY(tmp.alloc(&totals, 1));
    B200_CUDA_TRY(tmp.alloc(&count, n_windows));
    B200_CUDA_TRY(tmp.alloc(&tile_of, n_windows));
    B200_CUDA_TRY(pool_alloc(&f->d_rowOffset, (size_t)n_windows + 1, stream));
    B200_CUDA_TRY(pool_alloc(&f->d_rowIdx, n_windows, stream));
    const uint64_t most_windows = std::min(n_windows, nnz);
    const uint64_t most_tiles = std::min((uint64_t)nnz / CW + most_windows, most_windows * (((uint64_t)cols + CW - 1) / CW));
    bool ahead = most_tiles * tile_bytes <= kAheadBytes;
    auto alloc_tiles = [&](uint64_t tiles) {
        const cudaError_t e = pool_alloc(&f->d_tcA2B, tiles * CW, stream);
        return e == cudaSuccess ? pool_alloc_bytes(&f->d_data, std::max<uint64_t>(tiles * tile_bytes, 16), stream) : e;
    };
    if (ahead) {
        const cudaError_t e = alloc_tiles(most_tiles);
        if (e == cudaErrorMemoryAllocation) {  // what is needed may still fit
            cudaGetLastError();
            pool_free(f->d_tcA2B, stream);
            f->d_tcA2B = nullptr;
            ahead = false;
        } else {
            B200_CUDA_TRY(e);
        }
    }
    const uint32_t parts = 4 * smem <= kSetsSmemMax ? 4 : 2 * smem <= kSetsSmemMax ? 2 : 1;
    if (parts * smem > 47 * 1024)  // (48 KB hold the kernel's own shared variables, too)
        B200_CUDA_TRY(cudaFuncSetAttribute(window_marks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSetsSmemMax));
    B200_CUDA_TRY(cudaMemsetAsync(totals, 0, sizeof(Totals), stream));
    const WindowArgs args{d_row_ptr, d_col_idx, rows, cols, nnz, n_windows, RW, log_cw, bit_words(f->info.cols), places, count, tile_of, totals};
    constexpr uint32_t kWarps = kSortBlock / 32;
    const bool wide = parts == 1;
    // as many blocks as there are windows, or as clear the tiles at the rate of the memory
    const uint64_t n_clear = ahead ? most_tiles * tile_bytes / 16 : 0;
    const uint32_t for_windows = std::min<uint32_t>((n_windows + kWarps - 1) / kWarps, 148 * 64);
    const uint32_t for_clearing = (uint32_t)std::min<uint64_t>((n_clear + 8 * kSortBlock - 1) / (8 * kSortBlock), 148 * 4);
    (wide ? window_sort_kernel<true> : window_sort_kernel<false>)<<<std::max(for_windows, for_clearing), kSortBlock, 0, stream>>>(
        args, static_cast<uint4 *>(f->d_data), n_clear);
    if (nnz > (wide ? kWarpEntries<true> : kWarpEntries<false>)) window_marks_kernel<<<std::min<uint32_t>(n_windows, 148), kBitsBlock, parts * smem, stream>>>(args, parts, (uint32_t)(smem / 4));
    B200_CUDA_TRY(cudaGetLastError());
    if (n_windows <= kOneBlockWindows) {
        scan_tables_kernel<<<1, kScanBlock, 0, stream>>>(count, n_windows, RW, CW, f->d_rowOffset, f->d_rowIdx, tile_of, totals);
    } else {
        unsigned long long *before = nullptr;
        uint8_t *scan_tmp = nullptr;
        size_t scan_bytes = 0;
        auto terms = thrust::make_transform_iterator(thrust::make_counting_iterator<uint32_t>(0), WindowTerms{nullptr, count, n_windows, CW});
        B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, terms, before, (int64_t)n_windows + 1, stream));
        B200_CUDA_TRY(tmp.alloc(&before, (size_t)n_windows + 1));
        B200_CUDA_TRY(tmp.alloc(&scan_tmp, scan_bytes));
        B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, terms, before, (int64_t)n_windows + 1, stream));
        window_tables_kernel<<<n_windows / kBlock + 1, kBlock, 0, stream>>>(before, n_windows, RW, f->d_rowOffset, f->d_rowIdx, tile_of, totals);
    }
    B200_CUDA_TRY(cudaGetLastError());
    auto place = [&]() {
        if (f->info.elt_size == 2) place_entries<uint16_t>(f, d_row_ptr, d_col_idx, d_values, places, count, tile_of, totals, log_cw, stream);
        else place_entries<uint32_t>(f, d_row_ptr, d_col_idx, d_values, places, count, tile_of, totals, log_cw, stream);
        return cudaGetLastError();
    };
    if (ahead) B200_CUDA_TRY(place());
    Totals h;
    B200_CUDA_TRY(cudaMemcpyAsync(&h, totals, sizeof(h), cudaMemcpyDeviceToHost, stream));
    B200_CUDA_TRY(cudaStreamSynchronize(stream));
    if (h.bad) return B200SPMM_ERR_BAD_CSR;
    f->info.eff_row_windows = h.windows_tiles >> 32;
    f->info.total_tiles = (uint32_t)h.windows_tiles;
    if (ahead) return B200SPMM_OK;
    B200_CUDA_TRY(alloc_tiles(f->info.total_tiles));
    B200_CUDA_TRY(cudaMemsetAsync(f->d_data, 0, f->info.total_tiles * tile_bytes, stream));
    B200_CUDA_TRY(place());
    B200_CUDA_TRY(cudaStreamSynchronize(stream));
    return B200SPMM_OK;
}

// Steps 1 - 4, with keys of key_bits bits (col_bits of them the column).
template <typename K>
int convert_on_device(b200spmm_dbtcf *f, const uint32_t *d_row_ptr, const uint32_t *d_col_idx, const void *d_values, int col_bits,
                      int key_bits, cudaStream_t stream) {
    const uint64_t rows = f->info.rows, cols = f->info.cols, nnz = f->info.nnzs, n_windows = f->info.total_row_windows;
    const uint32_t RW = (uint32_t)f->info.row_window, CW = (uint32_t)f->info.col_window;
    const int esz = f->info.elt_size;
    PoolScratch tmp(stream);
    K *keys = nullptr, *keys_sorted = nullptr, *ukeys = nullptr;
    Totals *totals = nullptr;
    uint32_t *first = nullptr, *tile_of = nullptr;
    unsigned long long *before = nullptr;
    B200_CUDA_TRY(tmp.alloc(&keys, nnz));
    B200_CUDA_TRY(tmp.alloc(&keys_sorted, nnz));
    B200_CUDA_TRY(tmp.alloc(&totals, 1));
    B200_CUDA_TRY(tmp.alloc(&first, n_windows + 1));
    B200_CUDA_TRY(tmp.alloc(&tile_of, n_windows));
    B200_CUDA_TRY(tmp.alloc(&before, n_windows + 1));
    ukeys = keys;  // the unsorted keys are dead once sorted: reuse their buffer for the distinct keys
    const WindowTerms windows{first, nullptr, (uint32_t)n_windows, CW};
    auto terms = thrust::make_transform_iterator(thrust::make_counting_iterator<uint32_t>(0), windows);
    size_t sort_bytes = 0, sel_bytes = 0, scan_bytes = 0;
    B200_CUDA_TRY(cub::DeviceRadixSort::SortKeys(nullptr, sort_bytes, keys, keys_sorted, (int64_t)nnz, 0, key_bits, stream));
    B200_CUDA_TRY(cub::DeviceSelect::Unique(nullptr, sel_bytes, keys_sorted, ukeys, &totals->n_unique, (int64_t)nnz, stream));
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, terms, before, (int64_t)n_windows + 1, stream));
    uint8_t *cub_tmp = nullptr;
    B200_CUDA_TRY(tmp.alloc(&cub_tmp, std::max({sort_bytes, sel_bytes, scan_bytes})));
    B200_CUDA_TRY(pool_alloc(&f->d_rowOffset, n_windows + 1, stream));
    B200_CUDA_TRY(pool_alloc(&f->d_rowIdx, n_windows, stream));

    // 1. keys
    B200_CUDA_TRY(cudaMemsetAsync(totals, 0, sizeof(Totals), stream));
    const int key_grid = (int)std::min<uint64_t>((nnz + kKeyEntries - 1) / kKeyEntries, 148 * 8);
    make_keys_kernel<<<key_grid, kBlock, 0, stream>>>(d_row_ptr, d_col_idx, (uint32_t)rows, (uint32_t)cols, nnz, RW, col_bits, keys,
                                                      totals);
    B200_CUDA_TRY(cudaGetLastError());

    // 2. sort, unique
    B200_CUDA_TRY(cub::DeviceRadixSort::SortKeys(cub_tmp, sort_bytes, keys, keys_sorted, (int64_t)nnz, 0, key_bits, stream));
    B200_CUDA_TRY(cub::DeviceSelect::Unique(cub_tmp, sel_bytes, keys_sorted, ukeys, &totals->n_unique, (int64_t)nnz, stream));

    // 3. windows
    const unsigned window_grid = (unsigned)(n_windows / kBlock + 1);
    window_bounds_kernel<<<window_grid, kBlock, 0, stream>>>(ukeys, totals, (uint32_t)n_windows, col_bits, first);
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(cub_tmp, scan_bytes, terms, before, (int64_t)n_windows + 1, stream));
    window_tables_kernel<<<window_grid, kBlock, 0, stream>>>(before, (uint32_t)n_windows, RW, f->d_rowOffset, f->d_rowIdx, tile_of,
                                                             totals);
    B200_CUDA_TRY(cudaGetLastError());
    Totals h;
    B200_CUDA_TRY(cudaMemcpyAsync(&h, totals, sizeof(h), cudaMemcpyDeviceToHost, stream));
    B200_CUDA_TRY(cudaStreamSynchronize(stream));
    if (h.bad) return B200SPMM_ERR_BAD_CSR;
    const uint64_t n_unique = h.n_unique;
    const uint32_t eff = (uint32_t)(h.windows_tiles >> 32), total_tiles = (uint32_t)h.windows_tiles;
    f->info.eff_row_windows = eff;
    f->info.total_tiles = total_tiles;

    // 4. column lists and values
    const uint64_t list_len = (uint64_t)total_tiles * CW, data_len = (uint64_t)total_tiles * RW * CW;
    B200_CUDA_TRY(pool_alloc(&f->d_tcA2B, list_len, stream));
    B200_CUDA_TRY(pool_alloc_bytes(&f->d_data, std::max<uint64_t>(data_len * esz, 16), stream));
    B200_CUDA_TRY(cudaMemsetAsync(f->d_tcA2B, 0xFF, list_len * 4, stream));  // kIdxMax padding
    B200_CUDA_TRY(cudaMemsetAsync(f->d_data, 0, data_len * esz, stream));
    scatter_columns_kernel<<<grid_for(n_unique), kBlock, 0, stream>>>(ukeys, n_unique, col_bits, first, tile_of, CW, f->d_tcA2B);
    B200_CUDA_TRY(cudaGetLastError());
    scatter_values(f, d_row_ptr, d_col_idx, d_values, windows, tile_of, stream);
    B200_CUDA_TRY(cudaGetLastError());
    B200_CUDA_TRY(cudaStreamSynchronize(stream));
    return B200SPMM_OK;
}

}  // namespace gpuconv
}  // namespace b200spmm

using namespace b200spmm;
using namespace b200spmm::gpuconv;

extern "C" {

void b200spmm_dbtcf_destroy(b200spmm_dbtcf_t *f) {
    if (!f) return;
    cudaSetDevice(f->device);
    cudaDeviceSynchronize();  // a product may still be reading the arrays
    pool_free(f->d_rowOffset);
    pool_free(f->d_tcA2B);
    pool_free(f->d_rowIdx);
    pool_free(f->d_data);
    delete f;
}

int b200spmm_dbtcf_info(const b200spmm_dbtcf_t *f, b200spmm_btcf_info_t *info) {
    if (!f || !info) return B200SPMM_ERR_INVALID_ARG;
    *info = f->info;
    return B200SPMM_OK;
}
const uint32_t *b200spmm_dbtcf_rowOffset(const b200spmm_dbtcf_t *f) { return f ? f->d_rowOffset : nullptr; }
const uint32_t *b200spmm_dbtcf_tcA2B(const b200spmm_dbtcf_t *f) { return f ? f->d_tcA2B : nullptr; }
const void *b200spmm_dbtcf_data(const b200spmm_dbtcf_t *f) { return f ? f->d_data : nullptr; }
const uint32_t *b200spmm_dbtcf_rowIdx(const b200spmm_dbtcf_t *f) { return f ? f->d_rowIdx : nullptr; }

int b200spmm_dbtcf_copy_to_host(const b200spmm_dbtcf_t *f, uint32_t *rowOffset, uint32_t *tcA2B, void *data,
                                uint32_t *rowIdx) {
    if (!f || !rowOffset || !tcA2B || !data || !rowIdx) return B200SPMM_ERR_INVALID_ARG;
    B200_CUDA_TRY(cudaSetDevice(f->device));
    const auto &i = f->info;
    const uint64_t tile_elems = (uint64_t)i.row_window * i.col_window;
    B200_CUDA_TRY(cudaMemcpy(rowOffset, f->d_rowOffset, (i.eff_row_windows + 1) * 4, cudaMemcpyDeviceToHost));
    if (i.total_tiles) {
        B200_CUDA_TRY(cudaMemcpy(tcA2B, f->d_tcA2B, i.total_tiles * i.col_window * 4, cudaMemcpyDeviceToHost));
        B200_CUDA_TRY(cudaMemcpy(data, f->d_data, i.total_tiles * tile_elems * i.elt_size, cudaMemcpyDeviceToHost));
        B200_CUDA_TRY(cudaMemcpy(rowIdx, f->d_rowIdx, i.eff_row_windows * 4, cudaMemcpyDeviceToHost));
    }
    return B200SPMM_OK;
}

int b200spmm_csr2btcf_nobitmap_device(uint64_t rows, uint64_t cols, uint64_t nnz, const uint32_t *d_row_ptr,
                                      const uint32_t *d_col_idx, const void *d_values, int dtype, int row_window,
                                      int col_window, int device, void *stream_v, b200spmm_dbtcf_t **out) {
    if (!out || !d_row_ptr || (nnz && (!d_col_idx || !d_values))) return B200SPMM_ERR_INVALID_ARG;
    *out = nullptr;
    if (dtype != B200SPMM_F16 && dtype != B200SPMM_TF32) return B200SPMM_ERR_INVALID_ARG;
    if (row_window != 8 && row_window != 16) return B200SPMM_ERR_INVALID_ARG;
    if (col_window == 0) col_window = dtype == B200SPMM_F16 ? 16 : 8;
    if (col_window != 4 && col_window != 8 && col_window != 16) return B200SPMM_ERR_INVALID_ARG;
    if (rows >= 0xFFFFFFFFull || cols > 0xFFFFFFFFull || nnz > 0xFFFFFFFFull) return B200SPMM_ERR_UNSUPPORTED;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    B200_CUDA_TRY(cudaSetDevice(device));
    const uint32_t RW = (uint32_t)row_window;
    const int esz = dtype == B200SPMM_F16 ? 2 : 4;
    const uint64_t n_windows = (rows + RW - 1) / RW;

    b200spmm_dbtcf *f = new (std::nothrow) b200spmm_dbtcf();
    if (!f) return B200SPMM_ERR_NO_MEMORY;
    f->device = device;
    f->info.rows = rows;
    f->info.cols = cols;
    f->info.nnzs = nnz;
    f->info.total_row_windows = n_windows;
    f->info.row_window = row_window;
    f->info.col_window = col_window;
    f->info.dtype = dtype;
    f->info.elt_size = esz;
    struct Guard {  // frees the half-built result unless released
        b200spmm_dbtcf *f;
        ~Guard() { if (f) b200spmm_dbtcf_destroy(f); }
    } guard{f};

    if (nnz == 0) {
        uint32_t head[2] = {0, 0};  // (with entries make_keys_kernel looks at them)
        B200_CUDA_TRY(cudaMemcpyAsync(&head[0], d_row_ptr, 4, cudaMemcpyDeviceToHost, stream));
        B200_CUDA_TRY(cudaMemcpyAsync(&head[1], d_row_ptr + rows, 4, cudaMemcpyDeviceToHost, stream));
        B200_CUDA_TRY(cudaStreamSynchronize(stream));
        if (head[0] != 0 || head[1] != 0) return B200SPMM_ERR_BAD_CSR;
        B200_CUDA_TRY(pool_alloc(&f->d_rowOffset, 4, stream));
        B200_CUDA_TRY(cudaMemsetAsync(f->d_rowOffset, 0, 16, stream));
        B200_CUDA_TRY(cudaStreamSynchronize(stream));
        guard.f = nullptr;
        *out = f;
        return B200SPMM_OK;
    }

    if (by_windows_pays(cols)) {
        const int st = convert_by_windows(f, d_row_ptr, d_col_idx, d_values, stream);
        if (st != B200SPMM_OK) return st;
        guard.f = nullptr;
        *out = f;
        return B200SPMM_OK;
    }
    int win_bits = 1, col_bits = 1;
    while ((1ull << win_bits) < n_windows) ++win_bits;
    while ((1ull << col_bits) < cols) ++col_bits;
    const int st = win_bits + col_bits <= 32
                       ? convert_on_device<uint32_t>(f, d_row_ptr, d_col_idx, d_values, col_bits, win_bits + col_bits, stream)
                       : convert_on_device<uint64_t>(f, d_row_ptr, d_col_idx, d_values, col_bits, win_bits + col_bits, stream);
    if (st != B200SPMM_OK) return st;
    guard.f = nullptr;
    *out = f;
    return B200SPMM_OK;
}

}  // extern "C"
