// Condensed tiles -> row units, on the device.
//
//   1. the tile stream in runs of kRunTiles, and a run cut where a window ends; a warp counts the stored values of each of
//      the sixteen rows of its run (one 16-byte load per lane is half a tile row)
//   2. per (window, row): running sums over the window's runs -> row lengths, and how many units there are of every length;
//      running sums over the rows -> the units, slots and bands.  The longest come first, so the lengths alone say where every
//      unit of a length lies and where its batches do: the host's one wait, which brings what the look over a caller's tables
//      has found as well
//   3. every row puts its units into the list (build_band_units makes the one with the bands apart, CUB radix sort, four key bits)
//   4. the warps of step 1 write (column, value) to the place of their row's unit
// Seven launches and one wait before the last.  The plan of a graph of 60,000 nodes and 720,000 entries takes 95 us, of 10,000
// nodes 80; with a wait for the tables, a scan in two launches, a hub row's pieces placed by one thread and values written as they
// are found it was 138 and 99, with the units sorted, three scans and a launch for each small step (26 of them) 232 and 200.
// A stored value is one whose bits are not all zero (an explicit zero adds nothing to a product), in a row and a column
// of the matrix: the arrays may be a caller's, and what lies in a padded slot or below the last row multiplies nothing.
#include <algorithm>
#include <cub/cub.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include "common.hpp"
#include "device_pool.hpp"
#include "rows_gpu.hpp"

namespace b200spmm {
namespace {

constexpr int kBlock = 256;
// A hub window has thousands of tiles: short runs, or its warps are what everybody waits for (60,000 nodes, hub
// row of 10,000 entries: 419 us for write_entries_kernel with runs of 256 tiles).  A plan, in us, with runs of 16 / 8 / 4:
// 60,000 nodes 147 / 138 / 136, 10,000 nodes 122 / 99 / 91, 150,001 nodes, tf32 276 / 280 / 300.
constexpr uint32_t kRunTiles = 8;
constexpr uint32_t kMaxBands = 8;
// The lengths of the units: kMaxUnitEntries - entries, so the longest come first; rows without entries are behind all of them.
constexpr uint32_t kLengths = kMaxUnitEntries, kEmpty = kLengths;
constexpr uint32_t kEmptyBandKey = kMaxBands;  // sort key of the bands: their units, then their rows without entries
constexpr int kBandKeyBits = 4;
constexpr uint64_t kMinBandedCost = 2000000;  // bands pay where one keeps the GPU busy for tens of microseconds
// For the bands a row counts as this many entries: its store is 4 bytes a feature where a gathered entry is 2.
constexpr uint64_t kRowCost = 2;
// Starting and reducing a row costs a warp of the narrow kernel about what 64 entries do.
constexpr uint64_t kNarrowRowCost = 64;

inline int grid_for(uint64_t n) { return (int)std::max<uint64_t>(1, std::min<uint64_t>((n + kBlock - 1) / kBlock, 148 * 32)); }

__host__ __device__ __forceinline__ uint32_t pieces_of(uint32_t len, uint32_t cap) { return len <= cap ? 1u : (len + cap - 1) / cap; }

// Running sums over the rows, this one included: (entries << 32 | units) and (cut rows << 32 | slots).
struct RowSums {
    unsigned long long a, b;
};
struct AddSums {
    __host__ __device__ RowSums operator()(const RowSums &x, const RowSums &y) const { return {x.a + y.a, x.b + y.b}; }
};
// Rows a block of row_sums_kernel sums up, and how many such chunks one can have before it.
constexpr uint32_t kChunkRows = 4 * kBlock, kMaxChunks = kBlock;

struct RowTerms {
    const uint32_t *row_len;
    uint32_t cap;
    __host__ __device__ RowSums operator()(uint32_t r) const {
        const uint32_t len = row_len[r], n = pieces_of(len, cap);
        return {((unsigned long long)len << 32) | n, n > 1 ? (1ull << 32) | n : 0ull};
    }
};

// What the host waits for.
struct RowTotals {
    uint32_t entries, units, cut_rows, slots;
    uint32_t with_entries, n_batches, long_units[kLongUnits];  // units that have entries; and see RowsFormat
    uint32_t max_len;
    uint32_t band_row[kMaxBands + 1], band_cut[kMaxBands + 1];  // the bands' first rows and cut rows
    formatcheck::Found found;
    uint32_t blocks_done;  // of row_sums_kernel
};

// The look over the tables that runs ahead of the kernels here, if there is one, or what is known of them.
struct Tables {
    const formatcheck::Found *check;
    bool known_loose;
    __device__ __forceinline__ bool bad() const { return check && check->bad(); }
    __device__ __forceinline__ bool loose() const { return check ? check->loose() : known_loose; }
};

// Where the units of a length lie in the list, and the four neighbours' batches (quads) in front of theirs.
struct LengthTables {
    uint32_t count[kLengths];         // units of every length
    uint32_t start[kLengths + 1];     // place of the first one; of the first row without entries
    uint32_t quad_steps[kLengths];    // steps of the quads that begin before it
    uint32_t cursor[kLengths + 1];    // places taken so far
};

// Run `id` of window w (tiles chunk * kRunTiles .. of the stream, as far as they are the window's; none where a window ends
// with a chunk) has the number chunk + w.
__host__ __device__ __forceinline__ uint32_t first_run(uint32_t tile, uint32_t w) { return tile / kRunTiles + w; }

// run -> window; clears what the kernels behind it count in
__global__ void run_windows_kernel(const uint32_t *__restrict__ rowOffset, uint32_t eff, uint32_t rows, Tables found, uint32_t *__restrict__ run_window,
                                   uint32_t *__restrict__ row_len, LengthTables *__restrict__ tables, RowTotals *__restrict__ totals,
                                   RowSums *__restrict__ chunks) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < kMaxChunks) chunks[i] = {0, 0};
    if (i < eff && !found.bad())
        for (uint32_t r = first_run(rowOffset[i], i), end = first_run(rowOffset[i + 1], i + 1); r < end; ++r) run_window[r] = i;
    if (i < rows) row_len[i] = 0;
    if (blockIdx.x == 0) {
        for (uint32_t k = threadIdx.x; k < kLengths; k += blockDim.x) tables->count[k] = 0;
        if (threadIdx.x == 0) totals->max_len = totals->blocks_done = 0;
    }
}

// The tiles of a run.
struct RunTiles {
    uint32_t w, t0, t1, end;  // window, tiles [t0, t1), end of the window
    __device__ __forceinline__ RunTiles(uint32_t run, const uint32_t *__restrict__ run_window, const uint32_t *__restrict__ rowOffset) {
        w = run_window[run];
        const uint32_t chunk = (run - w) * kRunTiles;
        end = rowOffset[w + 1];
        t0 = max(chunk, rowOffset[w]);
        t1 = min(chunk + kRunTiles, end);
    }
};

// The lane's share of a tile: row lane / 2, its left or right half of the columns.
template <typename T>
struct Piece {
    static constexpr int kPer = 16 / (int)sizeof(T);
    alignas(16) T v[kPer];
    uint32_t mask;
    __device__ __forceinline__ void load(const T *__restrict__ data, uint64_t tile, uint32_t lane) {
        *reinterpret_cast<uint4 *>(v) = __ldcs(reinterpret_cast<const uint4 *>(data + tile * (32 * kPer) + lane * kPer));
        mask = 0;
        if (sizeof(T) == 2) {  // two values a word: a carry into the top bit of each half that is not zero
            const uint32_t *w = reinterpret_cast<const uint32_t *>(v);
            uint32_t m = 0;
#pragma unroll
            for (int k = 0; k < 4; ++k) m |= ((w[k] | ((w[k] & 0x7FFF7FFFu) + 0x7FFF7FFFu)) & 0x80008000u) >> (15 - 2 * k);
            mask = (m | m >> 15) & 0xFFu;
        } else {
#pragma unroll
            for (int k = 0; k < kPer; ++k) mask |= v[k] != 0 ? 1u << k : 0u;
        }
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
                const uint32_t *__restrict__ rowIdx, const uint32_t *__restrict__ run_window,
                uint32_t n_runs, uint32_t rows, uint32_t cols, Tables found, uint32_t *__restrict__ counts) {
    const uint32_t lane = threadIdx.x & 31u;
    if (found.bad()) return;
    const bool loose = found.loose();
    for (uint32_t run = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); run < n_runs; run += gridDim.x * (kBlock / 32)) {
        const RunTiles tiles(run, run_window, rowOffset);
        const uint32_t w = tiles.w, t0 = tiles.t0, t1 = tiles.t1, end = tiles.end;
        if (t0 >= t1) {
            if (lane < 16) counts[(uint64_t)run * 16 + lane] = 0;
            continue;
        }
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
__global__ void __launch_bounds__(kBlock)
row_lengths_kernel(const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ rowIdx, uint32_t eff, uint32_t rows, uint32_t cap, Tables found,
                   uint32_t *__restrict__ counts, uint32_t *__restrict__ row_len, LengthTables *__restrict__ tables,
                   RowTotals *__restrict__ totals, RowSums *__restrict__ chunks, uint32_t n_chunks) {
    __shared__ uint32_t here[kLengths];
    if (found.bad()) return;
    for (uint32_t k = threadIdx.x; k < kLengths; k += kBlock) here[k] = 0;
    __syncthreads();
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t w = (uint32_t)(i >> 4), r = (uint32_t)i & 15u;
    uint32_t sum = 0, chunk = 0;
    if (w < eff) {
        const uint32_t end = first_run(rowOffset[w + 1], w + 1);
        for (uint32_t run = first_run(rowOffset[w], w); run < end; run += 8) {
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
        chunk = (rowIdx[w] + r) / kChunkRows;
    }
    const uint32_t n = pieces_of(sum, cap);
    if (n_chunks) {
        // what the rows of a chunk add to the running sums, without the unit that every row has: a lane for each chunk of the warp
        // (one or two, or a lane each where a caller's windows lie far apart)
        const uint32_t same = __match_any_sync(0xffffffffu, chunk), lane = threadIdx.x & 31u;
        const uint32_t len = __reduce_add_sync(same, sum), more = __reduce_add_sync(same, n - 1), slots = __reduce_add_sync(same, n > 1 ? n : 0u);
        const uint32_t cut = __popc(__ballot_sync(0xffffffffu, n > 1) & same);
        if (len && (uint32_t)__ffs((int)same) - 1u == lane) {
            atomicAdd(&chunks[chunk].a, (unsigned long long)len << 32 | more);
            if (cut) atomicAdd(&chunks[chunk].b, (unsigned long long)cut << 32 | slots);
        }
    }
    if (sum) {  // (none below the last row)
        if (n > 1) atomicAdd(&here[kMaxUnitEntries - cap], n - 1);
        atomicAdd(&here[kMaxUnitEntries - (sum - (n - 1) * cap)], 1u);
    }
    const uint32_t most = __reduce_max_sync(0xffffffffu, sum);
    if ((threadIdx.x & 31u) == 0 && most > totals->max_len) atomicMax(&totals->max_len, most);
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < kLengths; k += kBlock)
        if (here[k]) atomicAdd(&tables->count[k], here[k]);
}

__device__ __forceinline__ uint32_t batches_of_length(uint32_t key) { return (kMaxUnitEntries - key + kUnitBatch - 1) / kUnitBatch; }
__device__ __forceinline__ uint32_t quads_before(uint32_t place) { return (place + 3) / 4; }

// Sum over the threads before this one.
__device__ __forceinline__ uint32_t block_exclusive_sum(uint32_t mine, uint32_t *warp_sums) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t upto = mine;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
        if (lane >= (uint32_t)d) upto += x;
    }
    __syncthreads();
    if (lane == 31) warp_sums[warp] = upto;
    __syncthreads();
    uint32_t before = upto - mine;
    for (uint32_t k = 0; k < warp; ++k) before += warp_sums[k];
    return before;
}

// One block of a thread per length.  Four neighbours of the list form a quad and are stored batch by batch side by side (batch
// k of all four, then batch k + 1): the groups of a warp, which walk neighbours, read their entries from the same lines.  A
// quad takes the steps of its first unit, which is its longest.
static_assert(kLengths == kBlock, "a thread for every length");
__device__ __forceinline__ void row_totals(uint32_t rows, Tables found, const RowSums *sums, LengthTables *tables, RowTotals *totals, uint32_t *warp_sums) {
    const uint32_t k = threadIdx.x, count = tables->count[k], start = block_exclusive_sum(count, warp_sums);
    const uint32_t steps = (quads_before(start + count) - quads_before(start)) * batches_of_length(k);  // of the quads that begin here
    const uint32_t steps_before = block_exclusive_sum(steps, warp_sums);
    tables->start[k] = tables->cursor[k] = start;
    tables->quad_steps[k] = steps_before;
    // units of at least 2 << j batches: those of at most this key
    for (uint32_t j = 0; j < kLongUnits; ++j)
        if (k == kMaxUnitEntries - kUnitBatch * ((2u << j) - 1u) - 1u) totals->long_units[j] = start + count;
    if (k == kLengths - 1) {
        tables->start[kEmpty] = tables->cursor[kEmpty] = totals->with_entries = start + count;
        totals->n_batches = 4 * (steps_before + steps);
    }
    const RowSums all = {__ldcg(&sums[rows - 1].a), __ldcg(&sums[rows - 1].b)};  // (other blocks may have written them just now)
    if (k == 0) {
        totals->entries = (uint32_t)(all.a >> 32);
        totals->units = (uint32_t)all.a;
        totals->cut_rows = (uint32_t)(all.b >> 32);
        totals->slots = (uint32_t)all.b;
        totals->found = found.check ? *found.check : formatcheck::Found{};
    }
    if (k > kMaxBands) return;
    const uint64_t cost = (all.a >> 32) + kRowCost * rows;
    const uint32_t bands = cost >= kMinBandedCost ? kMaxBands : 1u;
    uint32_t lo = 0, hi = rows;  // rows before which k / bands of the cost lie
    const uint64_t want = cost * k / bands;
    while (k && k < bands && lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if ((__ldcg(&sums[mid].a) >> 32) + kRowCost * (mid + 1) <= want) lo = mid + 1; else hi = mid;
    }
    if (!k || k >= bands) lo = k ? rows : 0u;
    totals->band_row[k] = lo;
    totals->band_cut[k] = lo ? (uint32_t)(__ldcg(&sums[lo - 1].b) >> 32) : 0u;
}

__global__ void __launch_bounds__(kBlock)
row_totals_kernel(uint32_t rows, Tables found, const RowSums *sums, LengthTables *tables, RowTotals *totals) {
    __shared__ uint32_t warp_sums[kBlock / 32];
    row_totals(rows, found, sums, tables, totals, warp_sums);
}

__device__ __forceinline__ unsigned long long shfl_up(unsigned long long x, int d) { return __shfl_up_sync(0xffffffffu, x, d); }

// The running sums of up to kMaxChunks chunks of rows: a block adds up what row_lengths_kernel has summed of the chunks before its
// own, and the last block to finish makes the totals.  60,000 rows: 8 us, where a scan in two launches and the totals took 15.
__global__ void __launch_bounds__(kBlock)
row_sums_kernel(const uint32_t *__restrict__ row_len, uint32_t rows, uint32_t cap, Tables found, const RowSums *__restrict__ chunks, RowSums *sums,
                LengthTables *tables, RowTotals *totals) {
    __shared__ RowSums warp_sums[kBlock / 32], warp_chunks[kBlock / 32];
    __shared__ uint32_t totals_sums[kBlock / 32], last;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, r0 = blockIdx.x * kChunkRows + threadIdx.x * 4;
    RowSums before = threadIdx.x < blockIdx.x ? chunks[threadIdx.x] : RowSums{0, 0};
    uint32_t len[4];
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) len[k] = r0 + k < rows ? row_len[r0 + k] : 0u;
    RowSums of[4], upto{0, 0};
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        const uint32_t n = pieces_of(len[k], cap);
        upto.a += (unsigned long long)len[k] << 32 | n;
        if (n > 1) upto.b += 1ull << 32 | n;
        of[k] = upto;
    }
    const RowSums mine = upto;
#pragma unroll
    for (int d = 1; d < 32; d *= 2) {
        const RowSums x{shfl_up(upto.a, d), shfl_up(upto.b, d)};
        if (lane >= (uint32_t)d) upto = AddSums{}(upto, x);
    }
#pragma unroll
    for (int d = 16; d; d /= 2) {
        before.a += __shfl_xor_sync(0xffffffffu, before.a, d);
        before.b += __shfl_xor_sync(0xffffffffu, before.b, d);
    }
    if (lane == 31) {
        warp_sums[warp] = upto;
        warp_chunks[warp] = before;
    }
    __syncthreads();
    RowSums base{(unsigned long long)blockIdx.x * kChunkRows + upto.a - mine.a, upto.b - mine.b};  // every row before has a unit
#pragma unroll
    for (uint32_t k = 0; k < kBlock / 32; ++k) {
        base = AddSums{}(base, warp_chunks[k]);
        if (k < warp) base = AddSums{}(base, warp_sums[k]);
    }
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)
        if (r0 + k < rows) sums[r0 + k] = AddSums{}(base, of[k]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(&totals->blocks_done, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!last) return;
    __threadfence();
    row_totals(rows, found, sums, tables, totals, totals_sums);
}

// Thread r: the units of row r take places among those of their length (in the order in which blocks of rows ask), and its
// line of the split table.
__global__ void __launch_bounds__(kBlock)
place_units_kernel(const uint32_t *__restrict__ row_len, uint32_t rows, uint32_t cap, const RowSums *__restrict__ sums, LengthTables *__restrict__ tables,
                   const RowTotals *__restrict__ totals, uint2 *__restrict__ units, uint32_t *__restrict__ unit_batch,
                   RowSplit *__restrict__ splits, uint32_t *__restrict__ batches, uint32_t batch_words) {
    __shared__ uint32_t base[kLengths + 1], start[kLengths + 1], quad_steps[kLengths];
    for (uint32_t k = threadIdx.x; k <= kLengths; k += kBlock) {
        base[k] = 0;
        start[k] = tables->start[k];
        if (k < kLengths) quad_steps[k] = tables->quad_steps[k];
    }
    __syncthreads();
    const uint32_t r = blockIdx.x * kBlock + threadIdx.x;
    uint32_t n = 0, full = 0, last_key = 0, rank_full = 0, rank_last = 0;
    const uint32_t full_key = kMaxUnitEntries - cap;
    if (r < rows) {
        const uint32_t len = row_len[r];
        n = pieces_of(len, cap);
        full = n - 1;
        last_key = len ? kMaxUnitEntries - (len - full * cap) : kEmpty;
        if (full) rank_full = atomicAdd(&base[full_key], full);
        rank_last = atomicAdd(&base[last_key], 1u);
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k <= kLengths; k += kBlock)
        if (base[k]) base[k] = atomicAdd(&tables->cursor[k], base[k]);
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x < batch_words)  // the batch that belongs to nobody
        batches[(uint64_t)totals->n_batches * batch_words + threadIdx.x] = batch_words == kBatchWords<true> ? (threadIdx.x == kTargetWord<true> ? kNoTarget : 0u)
                                                                                                 : (threadIdx.x == kTargetWord<false> ? kNoTarget : 0u);
    const uint32_t lane = threadIdx.x & 31u;
    const RowSums sum = r < rows ? sums[r] : RowSums{0, 0};
    // a piece of `key` at `place` of the list, the unit_at-th unit of the rows' order
    auto put = [&](uint32_t place, uint32_t key, uint32_t unit_at) {
        uint32_t of = key;  // the length of the quad's first unit
        while (start[of] > (place & ~3u)) --of;
        const uint32_t first = 4 * (quad_steps[of] + (place / 4 - quads_before(start[of])) * batches_of_length(of)) + (place & 3u);
        unit_batch[unit_at] = first;
        units[place] = make_uint2(first, batches_of_length(key));
    };
    // the full pieces of a long row by the whole warp: a hub row has hundreds (60,000 nodes: by its own thread 16 us, now 9)
    for (uint32_t cut = __ballot_sync(0xffffffffu, full != 0); cut; cut &= cut - 1u) {
        const int from = __ffs((int)cut) - 1;
        const uint32_t pieces = __shfl_sync(0xffffffffu, full, from), place = base[full_key] + __shfl_sync(0xffffffffu, rank_full, from);
        const uint32_t unit_at = __shfl_sync(0xffffffffu, (uint32_t)sum.a - n, from);
        for (uint32_t q = lane; q < pieces; q += 32) put(place + q, full_key, unit_at + q);
    }
    if (r >= rows) return;
    const uint32_t place = base[last_key] + rank_last;
    if (last_key != kEmpty) put(place, last_key, (uint32_t)sum.a - 1);
    else units[place] = make_uint2(r, 0u);
    if (n > 1) splits[(uint32_t)(sum.b >> 32) - 1] = RowSplit{r, (uint32_t)sum.b - n, (uint32_t)sum.b};
}

// The first rows of the bands.
struct BandRows {
    uint32_t row[kMaxBands];
};

// The band of every unit in the list, from the row that it adds to: its last batch names the row, or the slot of a cut one.
__global__ void __launch_bounds__(kBlock)
band_keys_kernel(const uint2 *__restrict__ units, uint32_t n_units, const uint32_t *__restrict__ batches, uint32_t batch_words, uint32_t target_word,
                 const RowSplit *__restrict__ splits, uint32_t n_splits, BandRows first, uint32_t bands, uint32_t *__restrict__ keys) {
    const uint32_t i = blockIdx.x * kBlock + threadIdx.x;
    if (i >= n_units) return;
    const uint2 unit = units[i];
    uint32_t row = unit.x;
    if (unit.y) {
        row = batches[(uint64_t)(unit.x + 4u * (unit.y - 1u)) * batch_words + target_word];
        if (row & kSlotTarget) {
            const uint32_t slot = row & ~kSlotTarget;
            uint32_t lo = 0, hi = n_splits - 1;  // the last cut row that starts at or before the slot
            while (lo < hi) {
                const uint32_t mid = hi - (hi - lo) / 2;
                if (splits[mid].slot_begin <= slot) lo = mid; else hi = mid - 1;
            }
            row = splits[lo].row;
        }
    }
    uint32_t band = 0;
    for (uint32_t k = 1; k < bands; ++k) band += row >= first.row[k] ? 1u : 0u;
    keys[i] = (unit.y ? 0u : kEmptyBandKey) | band;
}

// band k <= bands: the places of its first unit and of its first row without entries in the list of the bands
__global__ void band_units_kernel(const uint32_t *__restrict__ keys, uint32_t n_units, uint32_t bands, uint32_t *__restrict__ out) {
    const uint32_t i = threadIdx.x, k = i >> 1;
    if (k > bands) return;
    const uint32_t want = ((i & 1u) ? kEmptyBandKey : 0u) + k;
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

// A warp lists the stored values of its run - tile, lane and place in the lane's half row - and then takes 32 of the list at a
// time: written as they are found, lane by lane, a tile of a graph with 16 values kept 13 lanes of 32 busy in three rounds
// (720,000 entries, 60,000 rows: 30 us, 330 instructions a tile; now 21, 210).  Bound by instructions: neither more of the list in
// flight nor the list in the order of the rows' entries, which makes fewer and wider stores, is faster.
template <typename T>
__global__ void __launch_bounds__(kBlock)
write_entries_kernel(const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ tcA2B, const T *__restrict__ data,
                     const uint32_t *__restrict__ rowIdx, const uint32_t *__restrict__ run_window, uint32_t n_runs, uint32_t rows, uint32_t n_cols,
                     bool loose, uint32_t cap_bits, const uint32_t *__restrict__ counts, const uint32_t *__restrict__ row_len,
                     const RowSums *__restrict__ sums, const uint32_t *__restrict__ unit_batch, uint32_t *__restrict__ batches) {
    constexpr uint32_t kPer = Piece<T>::kPer, kWords = kBatchWords<sizeof(T) == 4>, kTo = kTargetWord<sizeof(T) == 4>;
    __shared__ uint16_t lists[kBlock / 32][kRunTiles * 32 * kPer];
    static_assert(kRunTiles * kPer <= 64, "a bit for each of a lane's values");
    const uint32_t lane = threadIdx.x & 31u, cap = 1u << cap_bits;
    uint16_t *list = lists[threadIdx.x >> 5];
    for (uint32_t run = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); run < n_runs; run += gridDim.x * (kBlock / 32)) {
        const RunTiles tiles(run, run_window, rowOffset);
        const uint32_t w = tiles.w, t0 = tiles.t0, n_tiles = tiles.t1 - t0, first_row = rowIdx[w], row = min(first_row + (lane >> 1), rows - 1);
        if (t0 >= tiles.t1) continue;
        const uint32_t limit = first_row + (lane >> 1) < rows ? n_cols : 0u;
        // of the lane's row
        const uint32_t len = row_len[row], at = counts[(uint64_t)run * 16 + (lane >> 1)];  // its entries, those in front of the run
        const RowSums sum = sums[row];
        const uint32_t pieces = pieces_of(len, cap), unit = (uint32_t)sum.a - pieces, slot = (uint32_t)sum.b - pieces;
        uint64_t found = 0;  // the lane's values, kPer bits a tile
#pragma unroll
        for (uint32_t t = 0; t < kRunTiles; ++t) {
            if (t >= n_tiles) break;
            Piece<T> p;
            p.load(data, t0 + t, lane);
            if (loose || t0 + t + 1 == tiles.end || limit == 0) {
                alignas(16) uint32_t cols[kPer];
                load_columns(cols, tcA2B, t0 + t, lane);
                p.keep(cols, limit);
            }
            found |= (uint64_t)p.mask << (t * kPer);
        }
        const uint32_t mine = (uint32_t)__popcll(found);
        uint32_t upto = mine;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
            if (lane >= (uint32_t)d) upto += x;
        }
        const uint32_t n = __shfl_sync(0xffffffffu, upto, 31);
        uint32_t to = upto - mine;
        const uint32_t first_entry = at - to;  // of the lane's values, were there none in the other half
        for (uint64_t m = found; m; m &= m - 1) list[to++] = (uint16_t)((uint32_t)(__ffsll((long long)m) - 1) << 5 | lane);
        __syncwarp();
        for (uint32_t i0 = 0; i0 < n; i0 += 32) {
            const uint32_t i = i0 + lane;
            const uint32_t which = i < n ? list[i] : 0u, from = which & 31u, bit = which >> 5, tile = bit / kPer, k = bit % kPer;
            uint32_t col = 0;
            T v = 0;
            if (i < n) {
                col = tcA2B[(uint64_t)(t0 + tile) * (2 * kPer) + (from & 1u) * kPer + k];
                v = data[(uint64_t)(t0 + tile) * (32 * kPer) + from * kPer + k];
            }
            // in front of it in the row, too: the other half's values up to this tile, or with it if that is the left one
            const uint32_t other_bits = (tile + (from & 1u)) * kPer;
            const uint64_t other = __shfl_sync(0xffffffffu, found, (int)(from ^ 1u)) & (other_bits == 64 ? ~0ull : (1ull << other_bits) - 1);
            const uint32_t entry = i + __shfl_sync(0xffffffffu, first_entry, (int)from) + (uint32_t)__popcll(other);
            const uint32_t row_entries = __shfl_sync(0xffffffffu, len, (int)from);
            const uint32_t first_unit = __shfl_sync(0xffffffffu, unit, (int)from), first_slot = __shfl_sync(0xffffffffu, slot, (int)from);
            if (i >= n) continue;
            if (sizeof(T) == 4) v = (T)((uint32_t)v & 0xFFFFE000u);  // as the tensor core reads it
            const uint32_t n_pieces = pieces_of(row_entries, cap), piece = min(entry >> cap_bits, n_pieces - 1), e = entry - (piece << cap_bits);
            const uint32_t entries = min(row_entries - (piece << cap_bits), cap), fill = (0u - entries) % kUnitBatch;  // slots before the second entry
            uint32_t *out = batches + (uint64_t)unit_batch[first_unit + piece] * kWords;
            // the unit's last batch holds its target, the others none; a batch's first entry writes it
            auto put = [&](uint32_t e, T value) {
                uint32_t *words = out + (e / kUnitBatch) * (4 * kWords);
                words[e % kUnitBatch] = col;
                if (e % kUnitBatch == 0)
                    words[kTo] = e / kUnitBatch + 1 < (entries + kUnitBatch - 1) / kUnitBatch ? kNoTarget
                                 : n_pieces > 1                                              ? kSlotTarget | (first_slot + piece)
                                                                                             : first_row + (from >> 1);
                reinterpret_cast<T *>(words + kUnitBatch)[e % kUnitBatch] = value;
            };
            T value = v, one;
            if (!e && fill) {
                split_value(v, fill, &value, &one);
                for (uint32_t f = 1; f <= fill; ++f) put(f, one);
            }
            put(e ? e + fill : 0u, value);
        }
        __syncwarp();
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
                 const uint32_t *__restrict__ rowIdx, const uint32_t *__restrict__ run_window,
                 uint32_t n_runs, uint32_t rows, uint32_t n_cols, const uint32_t *__restrict__ counts,
                 const RowSums *__restrict__ sums, uint32_t *__restrict__ cols_out, T *__restrict__ vals_out) {
    constexpr int kPer = Piece<T>::kPer;
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t run = blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5); run < n_runs; run += gridDim.x * (kBlock / 32)) {
        const RunTiles tiles(run, run_window, rowOffset);
        const uint32_t w = tiles.w, t0 = tiles.t0, t1 = tiles.t1, row = min(rowIdx[w] + (lane >> 1), rows - 1);
        const uint32_t limit = rowIdx[w] + (lane >> 1) < rows ? n_cols : 0u;
        uint32_t at = (row ? (uint32_t)(sums[row - 1].a >> 32) : 0u) + counts[(uint64_t)run * 16 + (lane >> 1)];
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
narrow_entries_kernel(const uint32_t *__restrict__ cols, const T *__restrict__ vals, const RowSums *__restrict__ sums, uint32_t rows,
                      uint32_t n_blocks, uint32_t *__restrict__ seg, uint32_t *__restrict__ entries) {
    extern __shared__ uint32_t narrow_smem[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, row = blockIdx.x * (kBlock / 32) + warp;
    uint32_t *count = narrow_smem + warp * (2 * n_blocks * 8), *run = count + n_blocks * 8;
    if (row >= rows) return;
    for (uint32_t k = lane; k < 2 * n_blocks * 8; k += 32) count[k] = 0;
    __syncwarp();
    const uint32_t begin = row ? (uint32_t)(sums[row - 1].a >> 32) : 0u, end = (uint32_t)(sums[row].a >> 32);
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
__global__ void narrow_cuts_kernel(const RowSums *__restrict__ sums, uint32_t rows, uint32_t n_ctas, uint32_t *__restrict__ cut) {
    const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k > n_ctas) return;
    const uint64_t total = (sums[rows - 1].a >> 32) + kNarrowRowCost * rows, want = total * k / n_ctas;
    uint32_t lo = 0, hi = rows;
    while (lo < hi) {
        const uint32_t mid = lo + (hi - lo) / 2;
        if ((sums[mid].a >> 32) + kNarrowRowCost * (mid + 1ull) <= want) lo = mid + 1; else hi = mid;
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
                 const uint32_t *d_rowIdx, int n_sms, const uint32_t *run_window, uint32_t n_runs, int run_grid,
                 const uint32_t *counts, const RowSums *sums, NarrowFormat *out) {
    const uint32_t rows = (uint32_t)info.rows, words = (uint32_t)info.elt_size / 2;
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
        write_csr_kernel<uint16_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, static_cast<const uint16_t *>(d_data), d_rowIdx,
                                                         run_window, n_runs, rows, n_cols, counts, sums, cols, static_cast<uint16_t *>(vals));
        narrow_entries_kernel<uint16_t><<<grid, kBlock, smem>>>(cols, static_cast<const uint16_t *>(vals), sums, rows, f.n_blocks, f.d_seg, f.d_entries);
    } else {
        write_csr_kernel<uint32_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, static_cast<const uint32_t *>(d_data), d_rowIdx,
                                                         run_window, n_runs, rows, n_cols, counts, sums, cols, static_cast<uint32_t *>(vals));
        narrow_entries_kernel<uint32_t><<<grid, kBlock, smem>>>(cols, static_cast<const uint32_t *>(vals), sums, rows, f.n_blocks, f.d_seg, f.d_entries);
    }
    narrow_cuts_kernel<<<(int)(f.n_ctas / kBlock + 1), kBlock>>>(sums, rows, f.n_ctas, f.d_cut);
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

int build_band_units(RowsFormat *f, bool tf32) {
    if (f->d_band_units || f->bands.size() <= 2) return B200SPMM_OK;
    const uint32_t bands = (uint32_t)f->bands.size() - 1, n = f->n_units;
    struct Units {
        uint2 *ptr = nullptr;
        ~Units() { pool_free(ptr); }
    } units;
    PoolScratch tmp;
    uint32_t *keys[2] = {}, *band_places = nullptr;
    uint8_t *sort_tmp = nullptr;
    size_t sort_bytes = 0;
    B200_CUDA_TRY(cub::DeviceRadixSort::SortPairs(nullptr, sort_bytes, keys[0], keys[1], f->d_units, units.ptr, (int64_t)n, 0, kBandKeyBits));
    cudaError_t e = pool_alloc(&units.ptr, n);
    for (int k = 0; k < 2 && e == cudaSuccess; ++k) e = tmp.alloc(&keys[k], n);
    if (e == cudaSuccess) e = tmp.alloc(&band_places, 2 * bands + 2);
    if (e == cudaSuccess) e = tmp.alloc(&sort_tmp, sort_bytes);
    if (e == cudaErrorMemoryAllocation) {  // no room: one band
        cudaGetLastError();
        return B200SPMM_OK;
    }
    B200_CUDA_TRY(e);
    BandRows first{};
    for (uint32_t k = 0; k < bands; ++k) first.row[k] = (uint32_t)f->bands[k].row;
    band_keys_kernel<<<(unsigned)((n + kBlock - 1) / kBlock), kBlock>>>(f->d_units, n, f->d_batches, tf32 ? kBatchWords<true> : kBatchWords<false>,
                                                                      tf32 ? kTargetWord<true> : kTargetWord<false>, f->d_splits, f->n_splits, first, bands, keys[0]);
    B200_CUDA_TRY(cudaGetLastError());
    // (the units of a band keep their order)
    B200_CUDA_TRY(cub::DeviceRadixSort::SortPairs(sort_tmp, sort_bytes, keys[0], keys[1], f->d_units, units.ptr, (int64_t)n, 0, kBandKeyBits));
    band_units_kernel<<<1, 32>>>(keys[1], n, bands, band_places);
    B200_CUDA_TRY(cudaGetLastError());
    uint32_t places[2 * kMaxBands + 2];
    B200_CUDA_TRY(cudaMemcpy(places, band_places, (2 * bands + 2) * 4, cudaMemcpyDeviceToHost));
    for (uint32_t k = 0; k < bands; ++k) {
        f->bands[k].unit = places[2 * k];
        f->bands[k].empty = places[2 * k + 1];
    }
    f->d_band_units = units.ptr;
    units.ptr = nullptr;
    return B200SPMM_OK;
}

int build_row_formats(const b200spmm_btcf_info_t &info, const uint32_t *d_rowOffset, const uint32_t *d_tcA2B,
                      const void *d_data, const uint32_t *d_rowIdx, const formatcheck::Found *d_found, formatcheck::Found *found, bool *found_known,
                      int n_sms, double max_fill, bool force_rows, RowsFormat *out, NarrowFormat *narrow) {
    *out = RowsFormat();
    *narrow = NarrowFormat();
    const uint64_t tiles = info.total_tiles;
    // (the product is refused for more columns, and the running sums of entries are 32-bit; a caller's tables may name windows of a
    // matrix without rows, which the look over them refuses)
    if (!info.rows || !info.eff_row_windows || !tiles || info.rows >= kSlotTarget || info.cols > 0x7FFFFFFFull || info.nnzs > 0xFFFFFFFFull) return B200SPMM_OK;
    const uint32_t rows = (uint32_t)info.rows, cols = (uint32_t)info.cols, eff = (uint32_t)info.eff_row_windows;
    const uint32_t cap = unit_entries_for(info.nnzs, info.rows, n_sms);
    RowsFormat f;
    struct Guard {
        RowsFormat *f;
        ~Guard() { if (f) free_rows(f); }
    } guard{&f};
    PoolScratch tmp;
    const uint64_t n_runs64 = tiles / kRunTiles + eff;  // first_run behind the last window
    if (n_runs64 > 0xFFFFFFFFull) return B200SPMM_OK;
    const uint32_t n_runs = (uint32_t)n_runs64;
    uint32_t *run_window = nullptr, *counts = nullptr, *row_len = nullptr;
    RowSums *sums = nullptr;
    LengthTables *tables = nullptr;
    RowTotals *totals = nullptr;
    B200_CUDA_TRY(tmp.alloc(&run_window, n_runs));
    B200_CUDA_TRY(tmp.alloc(&counts, n_runs64 * 16));
    B200_CUDA_TRY(tmp.alloc(&row_len, rows));
    B200_CUDA_TRY(tmp.alloc(&sums, rows));
    B200_CUDA_TRY(tmp.alloc(&tables, 1));
    B200_CUDA_TRY(tmp.alloc(&totals, 1));
    RowSums *chunks = nullptr;
    B200_CUDA_TRY(tmp.alloc(&chunks, kMaxChunks));
    const uint32_t n_chunks = rows <= kMaxChunks * kChunkRows ? (rows + kChunkRows - 1) / kChunkRows : 0;
    const Tables look{*found_known ? nullptr : d_found, found->loose()};

    const bool f16 = info.elt_size == 2;
    const uint16_t *data16 = static_cast<const uint16_t *>(d_data);
    const uint32_t *data32 = static_cast<const uint32_t *>(d_data);
    const int run_grid = grid_for(n_runs64 * 32), row_grid = (int)(((uint64_t)rows + kBlock - 1) / kBlock);
    run_windows_kernel<<<(unsigned)((std::max<uint64_t>(eff, rows) + kBlock - 1) / kBlock), kBlock>>>(d_rowOffset, eff, rows, look, run_window, row_len, tables, totals, chunks);
    if (f16) run_rows_kernel<uint16_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data16, d_rowIdx, run_window, n_runs, rows, cols, look, counts);
    else run_rows_kernel<uint32_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data32, d_rowIdx, run_window, n_runs, rows, cols, look, counts);
    row_lengths_kernel<<<(unsigned)(((uint64_t)eff * 16 + kBlock - 1) / kBlock), kBlock>>>(d_rowOffset, d_rowIdx, eff, rows, cap, look, counts, row_len, tables, totals,
                                                                                         chunks, n_chunks);
    if (n_chunks) {
        row_sums_kernel<<<n_chunks, kBlock>>>(row_len, rows, cap, look, chunks, sums, tables, totals);
    } else {
        auto terms = thrust::make_transform_iterator(thrust::make_counting_iterator<uint32_t>(0), RowTerms{row_len, cap});
        size_t scan_bytes = 0;
        B200_CUDA_TRY(cub::DeviceScan::InclusiveScan(nullptr, scan_bytes, terms, sums, AddSums{}, (int64_t)rows));
        uint8_t *scan_tmp = nullptr;
        B200_CUDA_TRY(tmp.alloc(&scan_tmp, scan_bytes));
        B200_CUDA_TRY(cub::DeviceScan::InclusiveScan(scan_tmp, scan_bytes, terms, sums, AddSums{}, (int64_t)rows));
        row_totals_kernel<<<1, kBlock>>>(rows, look, sums, tables, totals);
    }
    B200_CUDA_TRY(cudaGetLastError());
    RowTotals h;
    B200_CUDA_TRY(cudaMemcpy(&h, totals, sizeof(h), cudaMemcpyDeviceToHost));
    if (!*found_known) {
        *found = h.found;
        *found_known = true;
        if (found->bad()) return B200SPMM_OK;  // (the caller refuses them)
    }
    const bool loose = found->loose();
    if (!force_rows && (double)h.entries > max_fill * (double)tiles * 16.0 * info.col_window) {
        if (narrow_pays(h.entries, rows, info.cols, h.max_len, n_sms))
            return build_narrow(info, h.entries, d_rowOffset, d_tcA2B, d_data, d_rowIdx, n_sms, run_window, n_runs, run_grid, counts, sums, narrow);
        return B200SPMM_OK;
    }
    f.nnz = h.entries;
    f.n_units = h.units;
    f.n_splits = h.cut_rows;
    f.n_slots = h.slots;
    f.n_batches = h.n_batches;
    f.most_batches = (std::min(h.max_len, cap) + kUnitBatch - 1) / kUnitBatch;
    std::copy(h.long_units, h.long_units + kLongUnits, f.long_units);
    uint32_t bands = 0;
    while (h.band_row[bands] != rows) ++bands;
    for (uint32_t k = 0; k <= bands; ++k) f.bands.push_back(RowBand{0, h.with_entries, h.band_cut[k], h.band_row[k]});
    f.bands[bands].unit = h.with_entries;  // (all units, then all rows without entries)
    f.bands[bands].empty = f.n_units;

    // (the last batch belongs to nobody)
    const uint64_t n_batches = (uint64_t)f.nnz / kUnitBatch + f.n_units + 6 * (kMaxUnitEntries / kUnitBatch) + 8;
    if (n_batches > 0xFFFFFFFFull || f.n_slots >= kSlotTarget - 1) return B200SPMM_OK;
    const uint32_t words = info.elt_size == 2 ? kBatchWords<false> : kBatchWords<true>;
    uint32_t *unit_batch = nullptr;
    cudaError_t e = pool_alloc(&f.d_batches, ((uint64_t)f.n_batches + 1) * words);
    if (e == cudaSuccess) e = pool_alloc(&f.d_units, f.n_units);
    if (e == cudaSuccess) e = pool_alloc(&f.d_splits, f.n_splits);
    if (e == cudaSuccess) e = tmp.alloc(&unit_batch, f.n_units);
    if (e == cudaErrorMemoryAllocation) {  // no room: the tile kernels still work
        cudaGetLastError();
        return B200SPMM_OK;
    }
    B200_CUDA_TRY(e);
    uint32_t cap_bits = 0;  // (a power of two)
    while ((1u << cap_bits) < cap) ++cap_bits;
    place_units_kernel<<<row_grid, kBlock>>>(row_len, rows, cap, sums, tables, totals, f.d_units, unit_batch, f.d_splits, f.d_batches, words);
    if (f16)
        write_entries_kernel<uint16_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data16, d_rowIdx, run_window, n_runs, rows, cols, loose, cap_bits, counts,
                                                             row_len, sums, unit_batch, f.d_batches);
    else
        write_entries_kernel<uint32_t><<<run_grid, kBlock>>>(d_rowOffset, d_tcA2B, data32, d_rowIdx, run_window, n_runs, rows, cols, loose, cap_bits, counts,
                                                             row_len, sums, unit_batch, f.d_batches);
    B200_CUDA_TRY(cudaGetLastError());
    B200_CUDA_TRY(cudaDeviceSynchronize());
    if (!force_rows && narrow_pays(f.nnz, rows, info.cols, h.max_len, n_sms)) {
        const int st = build_narrow(info, f.nnz, d_rowOffset, d_tcA2B, d_data, d_rowIdx, n_sms, run_window, n_runs, run_grid, counts, sums, narrow);
        if (st != B200SPMM_OK) return st;
    }
    *out = f;
    guard.f = nullptr;
    return B200SPMM_OK;
}

}  // namespace b200spmm
