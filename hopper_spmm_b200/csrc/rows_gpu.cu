// Condensed tiles -> row units, on the device.
//
//   1. the tiles of every window in runs of at most kRunTiles; a warp counts the stored values of each of the
//      sixteen rows of its run (one 16-byte load per lane is half a tile row)
//   2. per (window, row): running sums over the window's runs -> row lengths; scans over the rows -> the units,
//      slots and bands
//   3. units sorted by length, longest first (CUB radix sort, a few key bits), their batches numbered in that order;
//      where there are bands, the list once more with the bands apart
//   4. the warps of step 1 write (column, value) to the place of their row's unit
// A stored value is one whose bits are not all zero (an explicit zero adds nothing to a product), in a row and a column
// of the matrix: the arrays may be a caller's, and what lies in a padded slot or below the last row multiplies nothing.
#include <algorithm>
#include <cub/cub.cuh>

#include "common.hpp"
#include "device_pool.hpp"
#include "rows_gpu.hpp"

namespace b200spmm {
namespace {

constexpr int kBlock = 256;
// A hub window has thousands of tiles: short runs, or its warps are what everybody waits for (60,000 nodes, hub
// row of 10,000 entries: 419 us for write_entries_kernel with runs of 256 tiles).
constexpr uint32_t kRunTiles = 16;
constexpr uint32_t kMaxBands = 8;
constexpr uint32_t kEmptyKey = 512;  // sort key of the units: longest first, rows without entries last
constexpr int kUnitKeyBits = 10;
constexpr uint32_t kEmptyBandKey = kMaxBands;  // sort key of the bands: their units, then their rows without entries
constexpr int kBandKeyBits = 4;
constexpr uint32_t kMaxLenAt = 4 + 2 * (kMaxBands + 1) + kLongUnits;  // in the table of totals: the longest row
constexpr uint64_t kMinBandedCost = 2000000;  // bands pay where one keeps the GPU busy for tens of microseconds
// For the bands a row counts as this many entries: its store is 4 bytes a feature where a gathered entry is 2.
constexpr uint64_t kRowCost = 2;
// Starting and reducing a row costs a warp of the narrow kernel about what 64 entries do.
constexpr uint64_t kNarrowRowCost = 64;

inline int grid_for(uint64_t n) { return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + kBlock - 1) / kBlock, 148 * 32)); }

__host__ __device__ __forceinline__ uint32_t pieces_of(uint32_t len, uint32_t cap) { return len <= cap ? 1u : (len + cap - 1) / cap; }

__global__ void run_counts_kernel(const uint32_t *__restrict__ rowOffset, uint32_t eff, uint32_t *__restrict__ n_runs) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w < eff) n_runs[w] = (rowOffset[w + 1] - rowOffset[w] + kRunTiles - 1) / kRunTiles;
    if (w == eff) n_runs[w] = 0;
}

__global__ void run_windows_kernel(const uint32_t *__restrict__ run_first, uint32_t eff, uint32_t *__restrict__ run_window) {
    const uint32_t w = blockIdx.x * blockDim.x + threadIdx.x;
    if (w >= eff) return;
    for (uint32_t r = run_first[w]; r < run_first[w + 1]; ++r) run_window[r] = w;
}

// a[k] of registers, by halves: two predicates less a register than comparing k with every index
template <int kN>
__device__ __forceinline__ uint32_t pick(const uint32_t (&a)[kN], int k) {
    const uint32_t lo = (k & 2) ? ((k & 1) ? a[3] : a[2]) : ((k & 1) ? a[1] : a[0]);
    if (kN == 4) return lo;
    const uint32_t hi = (k & 2) ? ((k & 1) ? a[kN - 1] : a[kN - 2]) : ((k & 1) ? a[kN - 3] : a[kN - 4]);
    return (k & 4) ? hi : lo;
}

// The lane's share of a tile: row lane / 2, its left or right half of the columns.
template <typename T>
struct Piece {
    static constexpr int kPer = 16 / (int)sizeof(T);
    alignas(16) T v[kPer];
    uint32_t mask;
    __device__ __forceinline__ T pick(int k) const {  // v[k]
        const uint32_t *w = reinterpret_cast<const uint32_t *>(v);
        const int i = sizeof(T) == 2 ? k >> 1 : k;
        const uint32_t word = (i & 2) ? ((i & 1) ? w[3] : w[2]) : ((i & 1) ? w[1] : w[0]);
        return sizeof(T) == 2 ? (T)(word >> ((k & 1) * 16)) : (T)word;
    }
    __device__ __forceinline__ void load(const T *__restrict__ data, uint64_t tile, uint32_t lane) {
        *reinterpret_cast<uint4 *>(v) = __ldcs(reinterpret_cast<const uint4 *>(data + tile * (32 * kPer) + lane * kPer));
        mask = 0;
#pragma unroll
        for (int k = 0; k < kPer; ++k) mask |= v[k] != 0 ? 1u << k : 0u;
    }
    // Leaves the values that count.  `cols`: of the lane's half, `n_cols`: 0 for a row below the last one.  Unless the lists
    // are loose, only the last tile of a window has slots without a column.
    __device__ __forceinline__ void keep(const uint32_t (&cols)[kPer], uint32_t n_cols) {
#pragma unroll
        for (int k = 0; k < kPer; ++k) mask &= cols[k] < n_cols ? 0xFFFFFFFFu : ~(1u << k);
    }
};

// The columns of the lane's half of a tile.
template <int kPer>
__device__ __forceinline__ void load_columns(uint32_t (&cols)[kPer], const uint32_t *__restrict__ tcA2B, uint64_t tile, uint32_t lane) {
#pragma unroll
    for (int k = 0; k < kPer / 4; ++k)
        reinterpret_cast<uint4 *>(cols)[k] = __ldg(reinterpret_cast<const uint4 *>(tcA2B + tile * (2 * kPer) + (lane & 1u) * kPer) + k);
}

// counts[run * 16 + row] = stored values of that row in the run's tiles
template <typename T>
__global__ void __launch_bounds__(kBlock)
run_rows_kernel(const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ tcA2B, const T *__restrict__ data,
                const uint32_t *__restrict__ rowIdx, const uint32_t *__restrict__ run_first, const uint32_t *__restrict__ run_window,
                uint32_t eff, uint32_t rows, uint32_t cols, bool loose, uint32_t *__restrict__ counts) {
    const uint32_t lane = threadIdx.x & 31u, n_runs = run_first[eff];
    for (uint32_t run = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); run < n_runs; run += gridDim.x * (kBlock / 32)) {
        const uint32_t w = run_window[run], t0 = rowOffset[w] + (run - run_first[w]) * kRunTiles;
        const uint32_t end = rowOffset[w + 1], t1 = min(t0 + kRunTiles, end);
        alignas(16) uint32_t of[Piece<T>::kPer];
        if (t1 == end) load_columns(of, tcA2B, end - 1, lane);
        uint32_t mine = 0;
        Piece<T> p;
        if (loose) {
            for (uint32_t t = t0; t < t1; ++t) {
                p.load(data, t, lane);
                load_columns(of, tcA2B, t, lane);
                p.keep(of, cols);
                mine += __popc(p.mask);
            }
        } else {
#pragma unroll 4
            for (uint32_t t = t0; t < t1; ++t) {
                p.load(data, t, lane);
                mine += __popc(p.mask);
            }
            if (t1 == end) {
                mine -= __popc(p.mask);
                p.keep(of, cols);
                mine += __popc(p.mask);
            }
        }
        if (rowIdx[w] + (lane >> 1) >= rows) mine = 0;
        mine += __shfl_xor_sync(0xffffffffu, mine, 1);
        if (!(lane & 1u)) counts[(uint64_t)run * 16 + (lane >> 1)] = mine;
    }
}

// thread (window, row of it): counts of its runs become what the earlier runs hold; the sum is the row's length
__global__ void row_lengths_kernel(const uint32_t *__restrict__ run_first, const uint32_t *__restrict__ rowIdx, uint32_t eff,
                                   uint32_t rows, uint32_t *__restrict__ counts, uint32_t *__restrict__ row_len,
                                   uint32_t *__restrict__ max_len) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t w = (uint32_t)(i >> 4), r = (uint32_t)i & 15u;
    if (w >= eff) return;
    uint32_t sum = 0;
    const uint32_t end = run_first[w + 1];
    for (uint32_t run = run_first[w]; run < end; run += 8) {
        uint32_t c[8];
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) c[k] = run + k < end ? counts[(uint64_t)(run + k) * 16 + r] : 0u;
#pragma unroll
        for (uint32_t k = 0; k < 8; ++k) {
            if (run + k < end) counts[(uint64_t)(run + k) * 16 + r] = sum;
            sum += c[k];
        }
    }
    if (rowIdx[w] + r < rows) row_len[rowIdx[w] + r] = sum;
    if (sum > *max_len) atomicMax(max_len, sum);
}

// Inclusive scans follow over both: (entries << 32 | units) and (cut rows << 32 | slots).
__global__ void row_terms_kernel(const uint32_t *__restrict__ row_len, uint32_t rows, uint32_t cap, unsigned long long *__restrict__ a,
                                 unsigned long long *__restrict__ b) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const uint32_t len = row_len[r], n = pieces_of(len, cap);
    a[r] = ((unsigned long long)len << 32) | n;
    b[r] = n > 1 ? (1ull << 32) | n : 0ull;
}

// totals[0..3]: entries, units, cut rows, slots; then per band its first row and cut row
__global__ void row_bands_kernel(uint32_t rows, const unsigned long long *__restrict__ a, const unsigned long long *__restrict__ b,
                                 uint32_t *__restrict__ totals) {
    const uint32_t k = threadIdx.x;
    if (k == 0) {
        totals[0] = (uint32_t)(a[rows - 1] >> 32);
        totals[1] = (uint32_t)a[rows - 1];
        totals[2] = (uint32_t)(b[rows - 1] >> 32);
        totals[3] = (uint32_t)b[rows - 1];
    }
    if (k > kMaxBands) return;
    const uint64_t cost = (a[rows - 1] >> 32) + kRowCost * rows;
    const uint32_t bands = cost >= kMinBandedCost ? kMaxBands : 1u;
    uint32_t lo = 0, hi = rows;  // rows before which k / bands of the cost lie
    const uint64_t want = cost * k / bands;
    while (k < bands && lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if ((a[mid] >> 32) + kRowCost * (mid + 1) <= want) lo = mid + 1; else hi = mid;
    }
    if (k >= bands) lo = rows;
    totals[4 + k * 2] = lo;
    totals[5 + k * 2] = lo ? (uint32_t)(b[lo - 1] >> 32) : 0u;
}

// one thread per row: sort keys of its units, and its line of the split table
__global__ void unit_keys_kernel(const uint32_t *__restrict__ row_len, uint32_t rows, uint32_t cap,
                                 const unsigned long long *__restrict__ a, const unsigned long long *__restrict__ b,
                                 uint32_t *__restrict__ keys, uint32_t *__restrict__ ids,
                                 uint32_t *__restrict__ unit_row, RowSplit *__restrict__ splits) {
    const uint32_t r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= rows) return;
    const uint32_t len = row_len[r], n = pieces_of(len, cap), first = (uint32_t)a[r] - n;
    for (uint32_t q = 0; q < n; ++q) {
        const uint32_t part = min(len - q * cap, cap);
        keys[first + q] = part ? kMaxUnitEntries - part : kEmptyKey;
        ids[first + q] = first + q;
        unit_row[first + q] = r;
    }
    if (n > 1) splits[(uint32_t)(b[r] >> 32) - 1] = RowSplit{r, (uint32_t)b[r] - n, (uint32_t)b[r]};
}

__device__ __forceinline__ uint32_t batches_of_key(uint32_t key) {
    return key == kEmptyKey ? 0u : (kMaxUnitEntries - key + kUnitBatch - 1) / kUnitBatch;
}

// Four neighbours of the sorted list form a quad and are stored batch by batch side by side (batch k of all four,
// then batch k + 1): the groups of a warp, which walk neighbours, read their entries from the same lines.
__global__ void quad_lengths_kernel(const uint32_t *__restrict__ keys, uint32_t n_units, uint32_t n_quads, uint32_t *__restrict__ quads) {
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q > n_quads) return;
    uint32_t most = 0;
    for (uint32_t i = 4 * q; i < min(4 * q + 4, n_units); ++i) most = max(most, batches_of_key(keys[i]));
    quads[q] = most;  // (0 for q == n_quads: its place in the running sum is the total)
}

// place i of the sorted list: where the unit's batches lie, the targets in them, and the key of its band
template <bool kTf32>
__global__ void place_units_kernel(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ ids, const uint32_t *__restrict__ quads,
                                   uint32_t n_units, uint32_t cap, const uint32_t *__restrict__ unit_row, const uint32_t *__restrict__ row_len,
                                   const unsigned long long *__restrict__ a, const unsigned long long *__restrict__ b,
                                   uint2 *__restrict__ units, uint32_t *__restrict__ unit_batch, uint32_t *__restrict__ batches,
                                   uint32_t bands, const uint32_t *__restrict__ totals, uint32_t *__restrict__ band_keys) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n_units) return;
    const uint32_t u = ids[i], r = unit_row[u], n = pieces_of(row_len[r], cap), first = quads[i >> 2] * 4 + (i & 3u);
    const uint32_t q = u - ((uint32_t)a[r] - n);  // which piece of its row
    const uint32_t n_batches = batches_of_key(keys[i]);
    units[i] = make_uint2(n_batches ? first : r, n_batches);
    unit_batch[u] = first;
    if (bands > 1) {
        uint32_t band = 0;
        for (uint32_t k = 1; k < bands; ++k) band += r >= totals[4 + k * 2] ? 1u : 0u;
        band_keys[i] = (n_batches ? 0u : kEmptyBandKey) | band;
    }
    for (uint32_t k = 0; k < n_batches; ++k)
        batches[(uint64_t)(first + 4 * k) * kBatchWords<kTf32> + kTargetWord<kTf32>] =
            k + 1 < n_batches ? kNoTarget : n > 1 ? kSlotTarget | ((uint32_t)b[r] - n + q) : r;
    if (i == n_units - 1) {  // the batch that belongs to nobody
        uint32_t *w = batches + (uint64_t)quads[(n_units + 3) / 4] * 4 * kBatchWords<kTf32>;
        for (uint32_t k = 0; k < kBatchWords<kTf32>; ++k) w[k] = k == kTargetWord<kTf32> ? kNoTarget : 0u;
    }
}

// band k <= bands: the places of its first unit and of its first row without entries (keys: of the bands, or of the units
// where there is one band); the number of batches; and how many units have at least 2 << j batches (unit_keys)
__global__ void band_units_kernel(const uint32_t *__restrict__ keys, const uint32_t *__restrict__ unit_keys, const uint32_t *__restrict__ quads,
                                  uint32_t n_units, uint32_t bands, uint32_t *__restrict__ out) {
    const uint32_t i = threadIdx.x, k = i >> 1, n_bounds = 2 * bands + 2;
    if (i > n_bounds + kLongUnits) return;
    if (i == n_bounds) {
        out[i] = 4 * quads[(n_units + 3) / 4];
        return;
    }
    uint32_t want = ((i & 1u) ? (bands > 1 ? kEmptyBandKey : kEmptyKey) : 0u) + k;
    if (i > n_bounds) {  // the first key that stands for fewer batches
        keys = unit_keys;
        want = kMaxUnitEntries - kUnitBatch * ((2u << (i - n_bounds - 1)) - 1u);
    }
    uint32_t lo = 0, hi = n_units;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if (keys[mid] < want) lo = mid + 1; else hi = mid;
    }
    out[i] = lo;
}

// v as first + n * unit, all three of v's sign, for the slots that fill a batch up: v's significand less n, and ones of its
// last place (tf32 has the same ten bits of it as fp16, thirteen places further up).  Times a value of B and added one after
// the other, first to nothing, every partial sum has the 22 bits of a product at most: the sum of the parts is the product,
// bit for bit, and infinite where it is.  (Zeros as fillers would make zero times infinity of it.)  A subnormal of n units
// and less has no such parts: it is followed by zeros.
template <typename T>
__device__ __forceinline__ void split_value(T v, uint32_t n, T *first, T *unit) {
    constexpr uint32_t kLow = sizeof(T) == 2 ? 0 : 13, kExp = sizeof(T) == 2 ? 31u : 255u;
    const uint32_t exp = ((uint32_t)v >> (10 + kLow)) & kExp, sign = (uint32_t)v & ((kExp + 1) << (10 + kLow));
    const uint32_t below = ((uint32_t)v >> kLow) & 1023u, m = below | (exp ? 1024u : 0u);
    *first = *unit = v;
    if (exp == kExp || m == 0) return;
    if (m <= n) {
        *unit = 0;
        return;
    }
    // under a power of two the places are half as wide
    *first = (T)((uint32_t)v - ((below >= n || exp <= 1 ? n : 2 * n - below) << kLow));
    *unit = (T)(sign | (exp > 10 ? (exp - 10) << (10 + kLow) : 1u << (max(exp, 1u) - 1 + kLow)));
}

template <typename T>
__global__ void __launch_bounds__(kBlock)
write_entries_kernel(const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ tcA2B, const T *__restrict__ data,
                     const uint32_t *__restrict__ rowIdx, const uint32_t *__restrict__ run_first,
                     const uint32_t *__restrict__ run_window, uint32_t eff, uint32_t rows, uint32_t n_cols, bool loose, uint32_t cap,
                     const uint32_t *__restrict__ counts,
                     const uint32_t *__restrict__ row_len, const unsigned long long *__restrict__ a,
                     const uint32_t *__restrict__ unit_batch, uint32_t *__restrict__ batches) {
    constexpr int kPer = Piece<T>::kPer;
    constexpr uint32_t kWords = kBatchWords<sizeof(T) == 4>;
    const uint32_t lane = threadIdx.x & 31u, n_runs = run_first[eff];
    for (uint32_t run = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); run < n_runs; run += gridDim.x * (kBlock / 32)) {
        const uint32_t w = run_window[run], t0 = rowOffset[w] + (run - run_first[w]) * kRunTiles;
        const uint32_t w_end = rowOffset[w + 1], t1 = min(t0 + kRunTiles, w_end), row = min(rowIdx[w] + (lane >> 1), rows - 1);
        const uint32_t len = row_len[row], limit = rowIdx[w] + (lane >> 1) < rows ? n_cols : 0u;
        const uint32_t *unit = unit_batch + ((uint32_t)a[row] - pieces_of(len, cap));  // first batches of the row's units
        uint32_t at = counts[(uint64_t)run * 16 + (lane >> 1)];  // entries of the row so far
        // Everything a lane reads comes ahead of its stores and for all lanes at once - the unit it starts in, a tile's
        // columns and values while the tile before is written: fetched at its first entry, one by one, they cost the warp
        // a round trip to L2 per entry (43 us of a matrix of 700,000 entries, 60,000 rows; now 32).
        uint32_t piece = min(at / cap, pieces_of(len, cap) - 1u), piece_end = (piece + 1) * cap;
        uint32_t fill = (0u - min(len - piece * cap, cap)) % kUnitBatch;  // slots before the second entry of the unit
        uint32_t *out = batches + (uint64_t)unit[piece] * kWords;
        auto put = [&](uint32_t e, uint32_t col, T v) {
            uint32_t *words = out + (e / kUnitBatch) * (4 * kWords);
            words[e % kUnitBatch] = col;
            reinterpret_cast<T *>(words + kUnitBatch)[e % kUnitBatch] = v;
        };
        Piece<T> next;
        alignas(16) uint32_t next_cols[kPer];
        auto fetch = [&](uint32_t t) {
            next.load(data, t, lane);
            load_columns(next_cols, tcA2B, t, lane);
        };
        fetch(t0);
        for (uint32_t t = t0; t < t1; ++t) {
            Piece<T> p = next;
            uint32_t cols[kPer];
#pragma unroll
            for (int k = 0; k < kPer; ++k) cols[k] = next_cols[k];
            if (loose || t + 1 == w_end || limit == 0) p.keep(cols, limit);
            if (t + 1 < t1) fetch(t + 1);
            const uint32_t mine = (uint32_t)__popc(p.mask), other = __shfl_xor_sync(0xffffffffu, mine, 1);
            uint32_t k_out = at + ((lane & 1u) ? other : 0u);
            at += mine + other;
            for (uint32_t m = p.mask; m; m &= m - 1u) {  // (two or three steps a warp; one per column would be eight)
                const int k = __ffs((int)m) - 1;
                const uint32_t col = pick(cols, k);
                const T v = sizeof(T) == 2 ? p.pick(k) : (T)((uint32_t)p.pick(k) & 0xFFFFE000u);  // as the tensor core reads it
                if (k_out >= piece_end) {
                    piece = k_out / cap;
                    piece_end = (piece + 1) * cap;
                    out = batches + (uint64_t)unit[piece] * kWords;
                    fill = (0u - min(len - piece * cap, cap)) % kUnitBatch;
                }
                const uint32_t e = k_out - piece * cap;
                ++k_out;
                T value = v, one;
                if (!e && fill) {
                    split_value(v, fill, &value, &one);
                    for (uint32_t f = 1; f <= fill; ++f) put(f, col, one);
                }
                put(e ? e + fill : 0u, col, value);
            }
        }
    }
}

// Entries of one row that are summed in one go; a longer row is cut.  A piece costs its slot, written and read
// once - 3 % of the rows of B that 256 entries gather - so large matrices keep to the maximum.  On small ones a
// warp's whole share is a few hundred entries and a unit of 256 would be the longest thing in the launch; but
// ordinary rows stay whole (up to twice the mean), because cut rows cost a second launch.
uint32_t unit_entries_for(uint64_t nnz, uint64_t rows, int n_sms) {
    const uint64_t share = nnz / ((uint64_t)n_sms * 128), mean = rows ? nnz / rows : 0;
    uint32_t cap = 64;
    while (cap < kMaxUnitEntries && (cap < share || cap < 2 * mean)) cap *= 2;
    return cap;
}

// ---- entries for narrow B

// columns and values of the rows one after the other, in column order
template <typename T>
__global__ void __launch_bounds__(kBlock)
write_csr_kernel(const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ tcA2B, const T *__restrict__ data,
                 const uint32_t *__restrict__ rowIdx, const uint32_t *__restrict__ run_first, const uint32_t *__restrict__ run_window,
                 uint32_t eff, uint32_t rows, uint32_t n_cols, const uint32_t *__restrict__ counts,
                 const unsigned long long *__restrict__ a, uint32_t *__restrict__ cols_out, T *__restrict__ vals_out) {
    constexpr int kPer = Piece<T>::kPer;
    const uint32_t lane = threadIdx.x & 31u, n_runs = run_first[eff];
    for (uint32_t run = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); run < n_runs; run += gridDim.x * (kBlock / 32)) {
        const uint32_t w = run_window[run], t0 = rowOffset[w] + (run - run_first[w]) * kRunTiles;
        const uint32_t t1 = min(t0 + kRunTiles, rowOffset[w + 1]), row = min(rowIdx[w] + (lane >> 1), rows - 1);
        const uint32_t limit = rowIdx[w] + (lane >> 1) < rows ? n_cols : 0u;
        uint32_t at = (row ? (uint32_t)(a[row - 1] >> 32) : 0u) + counts[(uint64_t)run * 16 + (lane >> 1)];
#pragma unroll 2
        for (uint32_t t = t0; t < t1; ++t) {
            Piece<T> p;
            alignas(16) uint32_t cols[kPer];
            p.load(data, t, lane);
            load_columns(cols, tcA2B, t, lane);
            p.keep(cols, limit);
            const uint32_t mine = (uint32_t)__popc(p.mask), other = __shfl_xor_sync(0xffffffffu, mine, 1);
            uint32_t k_out = at + ((lane & 1u) ? other : 0u);
            at += mine + other;
#pragma unroll
            for (int k = 0; k < kPer; ++k)
                if (p.mask & (1u << k)) {
                    cols_out[k_out] = cols[k];
                    vals_out[k_out++] = p.v[k];
                }
        }
    }
}

// One warp per row.  The kernel reads shared memory at 16 bytes x (column mod 8) for eight neighbouring entries at a
// time, so inside a block the entries are dealt out by column mod 8: first the first column of every class, then the
// second of every class, and so on.  Entry of rank r in class c comes behind min(count, r) entries of every class
// and one more of the classes below c that have it.
template <typename T>
__global__ void __launch_bounds__(kBlock)
narrow_entries_kernel(const uint32_t *__restrict__ cols, const T *__restrict__ vals, const unsigned long long *__restrict__ a, uint32_t rows,
                      uint32_t n_blocks, uint32_t *__restrict__ seg, uint32_t *__restrict__ entries) {
    extern __shared__ uint32_t narrow_smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, row = blockIdx.x * (kBlock / 32) + warp;
    uint32_t *count = narrow_smem + warp * (2 * n_blocks * 8), *run = count + n_blocks * 8;
    if (row >= rows) return;
    for (uint32_t k = lane; k < 2 * n_blocks * 8; k += 32) count[k] = 0;
    __syncwarp();
    const uint32_t begin = row ? (uint32_t)(a[row - 1] >> 32) : 0u, end = (uint32_t)(a[row] >> 32);
    for (uint32_t e = begin + lane; e < end; e += 32) atomicAdd(&count[(cols[e] / kNarrowCols) * 8 + (cols[e] & 7u)], 1u);
    __syncwarp();
    uint32_t *my_seg = seg + (uint64_t)row * (n_blocks + 1);
    if (lane == 0) {
        uint32_t at = begin;
        for (uint32_t b = 0; b < n_blocks; ++b) {
            my_seg[b] = at;
            for (uint32_t c = 0; c < 8; ++c) at += count[b * 8 + c];
        }
        my_seg[n_blocks] = at;
    }
    __syncwarp();
    for (uint32_t e0 = begin; e0 < end; e0 += 32) {
        const bool live = e0 + lane < end;
        const uint32_t col = live ? cols[e0 + lane] : 0xFFFFFFFFu, c = col & 7u, b = col / kNarrowCols;
        const uint32_t same = __match_any_sync(0xffffffffu, live ? b * 8 + c : 0xFFFFFFFFu);
        if (live) {
            const uint32_t rank = run[b * 8 + c] + (uint32_t)__popc(same & ((1u << lane) - 1u));
            uint32_t at = my_seg[b];
#pragma unroll
            for (uint32_t k = 0; k < 8; ++k) {
                const uint32_t n = count[b * 8 + k];
                at += min(n, rank) + (k < c && n > rank ? 1u : 0u);
            }
            if constexpr (sizeof(T) == 2) entries[at] = ((uint32_t)vals[e0 + lane] << 16) | (col & 0xFFFFu);
            else reinterpret_cast<uint2 *>(entries)[at] = make_uint2(col, (uint32_t)vals[e0 + lane] & 0xFFFFE000u);
        }
        __syncwarp();
        if (live && (same >> lane) == 1u) run[b * 8 + c] += (uint32_t)__popc(same);  // the last lane of the class
        __syncwarp();
    }
}

// CTA k: rows from the first one whose cost reaches k / n_ctas of the total on
__global__ void narrow_cuts_kernel(const unsigned long long *__restrict__ a, uint32_t rows, uint32_t n_ctas, uint32_t *__restrict__ cut) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > n_ctas) return;
    const uint64_t total = (a[rows - 1] >> 32) + kNarrowRowCost * rows, want = total * k / n_ctas;
    uint32_t lo = 0, hi = rows;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if ((a[mid] >> 32) + kNarrowRowCost * (mid + 1ull) <= want) lo = mid + 1; else hi = mid;
    }
    cut[k] = k == n_ctas ? rows : lo;
}

}  // namespace

void free_narrow(NarrowFormat *f) {
    pool_free(f->d_entries);
    pool_free(f->d_seg);
    pool_free(f->d_cut);
    *f = NarrowFormat();
}

void free_rows(RowsFormat *r) {
    pool_free(r->d_batches);
    pool_free(r->d_units);
    pool_free(r->d_band_units);
    pool_free(r->d_splits);
    *r = RowsFormat();
}

namespace {

// CTAs hold whole rows and a row is a warp's work: rows of a few steps of 32 lanes at least on average, and none
// longer than a quarter of a CTA's share.
bool narrow_pays(uint64_t nnz, uint64_t rows, uint64_t cols, uint64_t max_len, int n_sms) {
    return cols <= 65536 && nnz >= 48 * rows && max_len * (uint64_t)n_sms <= 4 * nnz + 32 * (uint64_t)n_sms * 32;
}

int build_narrow(const b200spmm_btcf_info_t &info, uint64_t nnz, const uint32_t *d_rowOffset, const uint32_t *d_tcA2B, const void *d_data,
                 const uint32_t *d_rowIdx, int n_sms, const uint32_t *run_first, const uint32_t *run_window, int run_grid,
                 const uint32_t *counts, const unsigned long long *a, NarrowFormat *out) {
    const uint32_t rows = (uint32_t)info.rows, eff = (uint32_t)info.eff_row_windows, words = (uint32_t)info.elt_size / 2;
    const uint32_t n_cols = (uint32_t)info.cols;
    NarrowFormat f;
    struct Guard {
        NarrowFormat *f;
        ~Guard() { if (f) free_narrow(f); }
    } guard{&f};
    PoolScratch tmp;
    f.n_blocks = (uint32_t)((info.cols + kNarrowCols - 1) / kNarrowCols);
    f.n_ctas = (uint32_t)std::min<uint64_t>((uint64_t)n_sms, rows);
    uint32_t *cols = nullptr;
    void *vals = nullptr;
    cudaError_t e = pool_alloc(&f.d_entries, nnz * words);
    if (e == cudaSuccess) e = pool_alloc(&f.d_seg, (uint64_t)rows * (f.n_blocks + 1));
    if (e == cudaSuccess) e = pool_alloc(&f.d_cut, f.n_ctas + 1);
    if (e == cudaSuccess) e = tmp.alloc(&cols, nnz);
    if (e == cudaSuccess) e = tmp.alloc(reinterpret_cast<uint16_t **>(&vals), nnz * words);
    if (e == cudaErrorMemoryAllocation) {  // no room: the tile kernels still work
        cudaGetLastError();
        return B200SPMM_OK;
    }
    B200_CUDA_TRY(e);
    const int grid = (int)((rows + kBlock / 32 - 1) / (kBlock / 32));
    const size_t smem = (size_t)(kBlock / 32) * 2 * f.n_blocks * 8 * 4;
    if (info.elt_size == 2) {
        write_csr_kernel<uint16_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, static_cast<const uint16_t *>(d_data), d_rowIdx, run_first,
                                                         run_window, eff, rows, n_cols, counts, a, cols, static_cast<uint16_t *>(vals));
        narrow_entries_kernel<uint16_t><<<grid, kBlock, smem>>>(cols, static_cast<const uint16_t *>(vals), a, rows, f.n_blocks, f.d_seg, f.d_entries);
    } else {
        write_csr_kernel<uint32_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, static_cast<const uint32_t *>(d_data), d_rowIdx, run_first,
                                                         run_window, eff, rows, n_cols, counts, a, cols, static_cast<uint32_t *>(vals));
        narrow_entries_kernel<uint32_t><<<grid, kBlock, smem>>>(cols, static_cast<const uint32_t *>(vals), a, rows, f.n_blocks, f.d_seg, f.d_entries);
    }
    narrow_cuts_kernel<<<(int)(f.n_ctas / kBlock + 1), kBlock>>>(a, rows, f.n_ctas, f.d_cut);
    B200_CUDA_TRY(cudaGetLastError());
    std::vector<uint32_t> cut(f.n_ctas + 1);
    B200_CUDA_TRY(cudaMemcpy(cut.data(), f.d_cut, cut.size() * 4, cudaMemcpyDeviceToHost));
    for (uint32_t k = 0; k < f.n_ctas; ++k) f.max_rows = std::max(f.max_rows, cut[k + 1] - cut[k]);
    B200_CUDA_TRY(cudaDeviceSynchronize());
    *out = f;
    guard.f = nullptr;
    return B200SPMM_OK;
}

}  // namespace

int build_row_formats(const b200spmm_btcf_info_t &info, const uint32_t *d_rowOffset, const uint32_t *d_tcA2B,
                      const void *d_data, const uint32_t *d_rowIdx, bool loose, int n_sms, double max_fill, bool force_rows,
                      RowsFormat *out, NarrowFormat *narrow) {
    *out = RowsFormat();
    *narrow = NarrowFormat();
    const uint64_t tiles = info.total_tiles;
    // (the product is refused for more columns, and the running sums of entries are 32-bit)
    if (!info.eff_row_windows || !tiles || info.rows >= kSlotTarget || info.cols > 0x7FFFFFFFull || info.nnzs > 0xFFFFFFFFull) return B200SPMM_OK;
    const uint32_t rows = (uint32_t)info.rows, cols = (uint32_t)info.cols, eff = (uint32_t)info.eff_row_windows;
    const uint32_t cap = unit_entries_for(info.nnzs, info.rows, n_sms);
    RowsFormat f;
    struct Guard {
        RowsFormat *f;
        ~Guard() { if (f) free_rows(f); }
    } guard{&f};
    PoolScratch tmp;
    const uint64_t max_runs = eff + tiles / kRunTiles;
    uint32_t *n_runs = nullptr, *run_first = nullptr, *run_window = nullptr, *counts = nullptr, *row_len = nullptr, *totals = nullptr;
    unsigned long long *a = nullptr, *b = nullptr;
    B200_CUDA_TRY(tmp.alloc(&n_runs, eff + 1));
    B200_CUDA_TRY(tmp.alloc(&run_first, eff + 1));
    B200_CUDA_TRY(tmp.alloc(&run_window, max_runs));
    B200_CUDA_TRY(tmp.alloc(&counts, max_runs * 16));
    B200_CUDA_TRY(tmp.alloc(&row_len, rows));
    B200_CUDA_TRY(tmp.alloc(&a, rows));
    B200_CUDA_TRY(tmp.alloc(&b, rows));
    B200_CUDA_TRY(tmp.alloc(&totals, kMaxLenAt + 1));
    size_t run_bytes = 0, row_bytes = 0;
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, run_bytes, n_runs, run_first, (int64_t)eff + 1));
    B200_CUDA_TRY(cub::DeviceScan::InclusiveSum(nullptr, row_bytes, a, a, (int64_t)rows));
    uint8_t *scan_tmp = nullptr;
    B200_CUDA_TRY(tmp.alloc(&scan_tmp, std::max(run_bytes, row_bytes)));

    run_counts_kernel<<<eff / kBlock + 1, kBlock>>>(d_rowOffset, eff, n_runs);
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(scan_tmp, run_bytes, n_runs, run_first, (int64_t)eff + 1));
    run_windows_kernel<<<(eff + kBlock - 1) / kBlock, kBlock>>>(run_first, eff, run_window);
    const bool f16 = info.elt_size == 2;
    const uint16_t *data16 = static_cast<const uint16_t *>(d_data);
    const uint32_t *data32 = static_cast<const uint32_t *>(d_data);
    const int run_grid = grid_for(max_runs * 32), row_grid = (int)((rows + kBlock - 1) / kBlock);
    if (f16) run_rows_kernel<uint16_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data16, d_rowIdx, run_first, run_window, eff, rows, cols, loose, counts);
    else run_rows_kernel<uint32_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data32, d_rowIdx, run_first, run_window, eff, rows, cols, loose, counts);
    uint32_t *max_len = totals + kMaxLenAt;
    B200_CUDA_TRY(cudaMemsetAsync(row_len, 0, (size_t)rows * 4));
    B200_CUDA_TRY(cudaMemsetAsync(max_len, 0, 4));
    row_lengths_kernel<<<(unsigned)(((uint64_t)eff * 16 + kBlock - 1) / kBlock), kBlock>>>(run_first, d_rowIdx, eff, rows, counts, row_len, max_len);
    row_terms_kernel<<<row_grid, kBlock>>>(row_len, rows, cap, a, b);
    B200_CUDA_TRY(cub::DeviceScan::InclusiveSum(scan_tmp, row_bytes, a, a, (int64_t)rows));
    B200_CUDA_TRY(cub::DeviceScan::InclusiveSum(scan_tmp, row_bytes, b, b, (int64_t)rows));
    row_bands_kernel<<<1, 32>>>(rows, a, b, totals);
    B200_CUDA_TRY(cudaGetLastError());
    uint32_t h[kMaxLenAt + 1];
    B200_CUDA_TRY(cudaMemcpy(h, totals, sizeof(h), cudaMemcpyDeviceToHost));
    if (!force_rows && (double)h[0] > max_fill * (double)tiles * 16.0 * info.col_window) {
        if (narrow_pays(h[0], rows, info.cols, h[kMaxLenAt], n_sms))
            return build_narrow(info, h[0], d_rowOffset, d_tcA2B, d_data, d_rowIdx, n_sms, run_first, run_window, run_grid, counts, a, narrow);
        return B200SPMM_OK;
    }
    const uint32_t h_max_len = h[kMaxLenAt];
    f.nnz = h[0];
    f.n_units = h[1];
    f.n_splits = h[2];
    f.n_slots = h[3];
    uint32_t bands = 0;
    while (h[4 + 2 * bands] != rows) ++bands;
    for (uint32_t k = 0; k <= bands; ++k) f.bands.push_back(RowBand{0, 0, h[5 + 2 * k], h[4 + 2 * k]});

    // Every unit rounds up to a batch, every quad to its longest unit: up to three longest units in all, as the lengths
    // fall from first to last, and three more where a quad holds the last units.
    const uint64_t max_batches = f.nnz / kUnitBatch + f.n_units + 6 * (kMaxUnitEntries / kUnitBatch) + 8;
    if (max_batches > 0xFFFFFFFFull || f.n_slots >= kSlotTarget - 1) return B200SPMM_OK;
    const uint32_t words = info.elt_size == 2 ? kBatchWords<false> : kBatchWords<true>;
    uint32_t *keys[2] = {}, *ids[2] = {}, *unit_row = nullptr;
    cudaError_t e = pool_alloc(&f.d_batches, max_batches * words);
    if (e == cudaSuccess) e = pool_alloc(&f.d_units, f.n_units);
    if (e == cudaSuccess && bands > 1) e = pool_alloc(&f.d_band_units, f.n_units);
    if (e == cudaSuccess) e = pool_alloc(&f.d_splits, f.n_splits);
    for (int k = 0; k < 2 && e == cudaSuccess; ++k) {
        e = tmp.alloc(&keys[k], f.n_units);
        if (e == cudaSuccess) e = tmp.alloc(&ids[k], f.n_units);
    }
    if (e == cudaSuccess) e = tmp.alloc(&unit_row, f.n_units);
    if (e == cudaErrorMemoryAllocation) {  // no room: the tile kernels still work
        cudaGetLastError();
        return B200SPMM_OK;
    }
    B200_CUDA_TRY(e);
    const uint32_t n_quads = (f.n_units + 3) / 4;
    uint32_t *quads = nullptr, *unit_batch = keys[0], *band_keys = ids[0];  // (free again once the pairs are sorted)
    B200_CUDA_TRY(tmp.alloc(&quads, n_quads + 1));
    unit_keys_kernel<<<row_grid, kBlock>>>(row_len, rows, cap, a, b, keys[0], ids[0], unit_row, f.d_splits);
    size_t sort_bytes = 0, batch_bytes = 0, band_bytes = 0;
    B200_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, keys[0], keys[1], ids[0], ids[1], (int64_t)f.n_units, 0, kUnitKeyBits));
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, batch_bytes, quads, quads, (int64_t)n_quads + 1));
    if (bands > 1)
        B200_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, band_bytes, band_keys, unit_row, f.d_units, f.d_band_units, (int64_t)f.n_units, 0, kBandKeyBits));
    uint8_t *sort_tmp = nullptr;
    B200_CUDA_TRY(tmp.alloc(&sort_tmp, std::max({sort_bytes, batch_bytes, band_bytes})));
    B200_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, keys[0], keys[1], ids[0], ids[1], (int64_t)f.n_units, 0, kUnitKeyBits));
    quad_lengths_kernel<<<(int)(n_quads / kBlock + 1), kBlock>>>(keys[1], f.n_units, n_quads, quads);
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(sort_tmp, batch_bytes, quads, quads, (int64_t)n_quads + 1));
    const int unit_grid = (int)((f.n_units + kBlock - 1) / kBlock);
    if (f16) {
        place_units_kernel<false><<<unit_grid, kBlock>>>(keys[1], ids[1], quads, f.n_units, cap, unit_row, row_len, a, b, f.d_units,
                                                         unit_batch, f.d_batches, bands, totals, band_keys);
        write_entries_kernel<uint16_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data16, d_rowIdx, run_first, run_window, eff, rows, cols, loose, cap,
                                                             counts, row_len, a, unit_batch, f.d_batches);
    } else {
        place_units_kernel<true><<<unit_grid, kBlock>>>(keys[1], ids[1], quads, f.n_units, cap, unit_row, row_len, a, b, f.d_units,
                                                        unit_batch, f.d_batches, bands, totals, band_keys);
        write_entries_kernel<uint32_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data32, d_rowIdx, run_first, run_window, eff, rows, cols, loose, cap,
                                                             counts, row_len, a, unit_batch, f.d_batches);
    }
    const uint32_t *sorted_bands = keys[1];
    if (bands > 1) {  // (the units of a band keep their order)
        B200_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sort_tmp, band_bytes, band_keys, unit_row, f.d_units, f.d_band_units, (int64_t)f.n_units, 0, kBandKeyBits));
        sorted_bands = unit_row;
    }
    band_units_kernel<<<1, 32>>>(sorted_bands, keys[1], quads, f.n_units, bands, totals);
    B200_CUDA_TRY(cudaGetLastError());
    B200_CUDA_TRY(cudaMemcpy(h, totals, (2 * bands + 3 + kLongUnits) * 4, cudaMemcpyDeviceToHost));
    for (uint32_t k = 0; k <= bands; ++k) {
        f.bands[k].unit = h[2 * k];
        f.bands[k].empty = h[2 * k + 1];
    }
    f.bands[bands].unit = f.bands[0].empty;  // (all units, then all rows without entries)
    f.bands[bands].empty = f.n_units;
    f.n_batches = h[2 * bands + 2];
    f.most_batches = (std::min(h_max_len, cap) + kUnitBatch - 1) / kUnitBatch;
    for (uint32_t k = 0; k < kLongUnits; ++k) f.long_units[k] = h[2 * bands + 3 + k];
    if (!force_rows && narrow_pays(f.nnz, rows, info.cols, h_max_len, n_sms)) {
        const int st = build_narrow(info, f.nnz, d_rowOffset, d_tcA2B, d_data, d_rowIdx, n_sms, run_first, run_window, run_grid, counts, a, narrow);
        if (st != B200SPMM_OK) return st;
    }
    *out = f;
    guard.f = nullptr;
    return B200SPMM_OK;
}

}  // namespace b200spmm
