// 16-row condensed format -> super-windows of 128 or 256 rows, on the device.  Same result as converting the
// matrix at that window height with the reference's algorithm (src/utils/convert.h:146-225):
// sorted distinct columns per window, padded to whole tiles; entries at (row % 128, column slot).
//
//   1. count_kernel: a block marks the columns of a 256-row window and of its two halves in bit sets in shared memory and
//      counts them.  The host makes the tile offsets of both heights from that, its one wait.
//   2. lists_kernel: the same bit set once more per window; the rank of a word gives its columns their places
//   3. tiles_kernel: a block makes kRunTiles neighbouring tiles of 128 rows in shared memory - each warp takes a
//      16-row tile that has columns there, eight values a lane, and looks their slots up in the run's list - and writes them
//      in one piece, as the product kernel's shared-memory image (the two 16-byte halves of a tile row swapped when
//      row / 4 is odd: the 32-byte swizzle)
// Large matrices are bound by the bytes of both formats and the driver's memory, small ones by the copies and waits around
// three launches.  A whole plan, in us, with a sort of all columns and a scatter of single values into cleared tiles, and so:
// pruned 28672 x 8192 at 10 % 5,270 and 3,190, 14336 x 4096 2,300 and 730, 1777 x 7404 at 15 % 870 and 445.
#include <algorithm>
#include <cstring>
#include <vector>

#include "common.hpp"
#include "device_pool.hpp"
#include "format.hpp"
#include "tall_gpu.hpp"

namespace b200spmm {
namespace {

constexpr uint32_t kShort = 16;
constexpr int kMergeBlock = 512;
constexpr uint32_t kChunkWords = 12288;  // words of a bit set: wider matrices go through chunks of columns
constexpr uint32_t kRunTiles = 8;        // 32 KB of tiles a block: six of them an SM
constexpr int kTilesBlock = 256;

inline uint32_t chunk_words(uint64_t cols) { return (uint32_t)std::min<uint64_t>((cols + 127) / 128 * 4, kChunkWords); }

// Marks the columns [col0, col0 + 32 * words) of the lists in tiles [t0, t1).
__device__ __forceinline__ void mark_columns(uint32_t *bits, uint32_t words, const uint32_t *__restrict__ tcA2B, uint32_t t0, uint32_t t1, uint32_t cw,
                                             uint32_t col0) {
    const uint4 *lists = reinterpret_cast<const uint4 *>(tcA2B + (uint64_t)t0 * cw);
    const uint32_t n = (t1 - t0) * (cw / 4);
#pragma unroll 4
    for (uint32_t q = threadIdx.x; q < n; q += kMergeBlock) {
        const uint4 v = __ldg(lists + q);
        const uint32_t c[4] = {v.x - col0, v.y - col0, v.z - col0, v.w - col0};
#pragma unroll
        for (int k = 0; k < 4; ++k)  // (no column: past every word)
            if ((c[k] >> 5) < words) atomicOr(bits + (c[k] >> 5), 1u << (c[k] & 31u));
    }
}

// One block per 256-row window: distinct columns of its upper half, its lower half, and both.
struct WindowPair {
    uint32_t t0, t_mid, t1;  // 16-row tiles of the two halves
};
__global__ void __launch_bounds__(kMergeBlock)
count_kernel(const WindowPair *__restrict__ pairs, const uint32_t *__restrict__ tcA2B, uint32_t cw, uint64_t cols, uint32_t words,
             uint32_t *__restrict__ counts) {
    extern __shared__ __align__(16) uint32_t merge_smem[];
    __shared__ uint32_t total[3];
    uint32_t *upper = merge_smem, *lower = merge_smem + words;
    const WindowPair p = pairs[blockIdx.x];
    if (threadIdx.x < 3) total[threadIdx.x] = 0;
    for (uint64_t col0 = 0; col0 < cols; col0 += 32ull * words) {
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < 2 * words; k += kMergeBlock) merge_smem[k] = 0;
        __syncthreads();
        mark_columns(upper, words, tcA2B, p.t0, p.t_mid, cw, (uint32_t)col0);
        mark_columns(lower, words, tcA2B, p.t_mid, p.t1, cw, (uint32_t)col0);
        __syncthreads();
        uint32_t n[3] = {};
        for (uint32_t k = threadIdx.x; k < words; k += kMergeBlock) {
            const uint32_t a = upper[k], b = lower[k];
            n[0] += __popc(a);
            n[1] += __popc(b);
            n[2] += __popc(a | b);
        }
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            n[k] = __reduce_add_sync(0xffffffffu, n[k]);
            if ((threadIdx.x & 31u) == 0 && n[k]) atomicAdd(&total[k], n[k]);
        }
    }
    __syncthreads();
    if (threadIdx.x < 3) counts[blockIdx.x * 3 + threadIdx.x] = total[threadIdx.x];
}

// One block per super-window: its sorted distinct columns, padded to whole tiles; and how many of the tiles name one aligned
// group of rows of B (added to *aligned).
struct WindowLists {
    uint32_t t0, t1, out, n_tiles;  // 16-row tiles, first tile of the list, tiles
};
__global__ void __launch_bounds__(kMergeBlock)
lists_kernel(const WindowLists *__restrict__ windows, const uint32_t *__restrict__ tcA2B, uint32_t cw, uint64_t cols, uint32_t words,
             uint32_t *__restrict__ lists, uint32_t *__restrict__ aligned) {
    extern __shared__ __align__(16) uint32_t merge_smem[];
    __shared__ uint32_t sums[kMergeBlock / 32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const WindowLists w = windows[blockIdx.x];
    uint32_t *out = lists + (uint64_t)w.out * cw, base = 0;
    for (uint64_t col0 = 0; col0 < cols; col0 += 32ull * words) {
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < words; k += kMergeBlock) merge_smem[k] = 0;
        __syncthreads();
        mark_columns(merge_smem, words, tcA2B, w.t0, w.t1, cw, (uint32_t)col0);
        __syncthreads();
        for (uint32_t k0 = 0; k0 < words; k0 += kMergeBlock) {  // one word a thread
            const uint32_t k = k0 + threadIdx.x;
            uint32_t b = k < words ? merge_smem[k] : 0u;
            const uint32_t mine = __popc(b);
            uint32_t upto = mine;
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= (uint32_t)d) upto += x;
            }
            __syncthreads();  // `sums` of the round before has been read
            if (lane == 31) sums[warp] = upto;
            __syncthreads();
            uint32_t at = base + upto - mine;
            for (uint32_t i = 0; i < kMergeBlock / 32; ++i) {
                if (i < warp) at += sums[i];
                base += sums[i];
            }
            for (; b; b &= b - 1u) out[at++] = (uint32_t)col0 + k * 32u + (uint32_t)__ffs((int)b) - 1u;
        }
    }
    for (uint32_t k = base + threadIdx.x; k < w.n_tiles * cw; k += kMergeBlock) out[k] = kIdxMax;
    __syncthreads();
    uint32_t n = 0;
    for (uint32_t t = threadIdx.x; t < w.n_tiles; t += kMergeBlock) {
        const uint32_t from = out[t * cw];
        n += from % cw == 0 && out[t * cw + cw - 1] - from == cw - 1;
    }
    n = __reduce_add_sync(0xffffffffu, n);
    if (lane == 0 && n) atomicAdd(aligned, n);
}

// One block per run of tiles of 128 rows.
struct TileRun {
    uint32_t w0, w1, row0;          // 16-row windows of the 128 rows, and the first of these
    uint32_t list, n_tiles, image;  // first tile of the run in the lists, its tiles, and its first image
};
template <typename T>
__global__ void __launch_bounds__(kTilesBlock)
tiles_kernel(const TileRun *__restrict__ runs, const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ tcA2B,
             const T *__restrict__ data, const uint32_t *__restrict__ rowIdx, const uint32_t *__restrict__ lists, uint8_t *__restrict__ images) {
    constexpr uint32_t kPer = 16 / sizeof(T), kCW = 2 * kPer, kWindows = 128 / kShort;  // kPer: values of a lane, half a tile row
    __shared__ __align__(16) uint8_t image[kRunTiles * 4096];
    __shared__ uint32_t list[kRunTiles * kCW], first[kWindows], tiles_before[kWindows + 1], bound[2 * kWindows];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const TileRun r = runs[blockIdx.x];
    const uint32_t n_windows = r.w1 - r.w0, n_list = r.n_tiles * kCW;
    for (uint32_t k = threadIdx.x; k < n_list; k += kTilesBlock) list[k] = __ldg(lists + (uint64_t)r.list * kCW + k);
    for (uint32_t k = threadIdx.x; k < r.n_tiles * 256; k += kTilesBlock) reinterpret_cast<uint4 *>(image)[k] = make_uint4(0, 0, 0, 0);
    __syncthreads();
    const uint32_t lowest = list[0];
    uint32_t n_real = n_list;  // the padding is at the end
    while (list[n_real - 1] == kIdxMax) --n_real;
    const uint32_t highest = list[n_real - 1];
    if (threadIdx.x < 2 * n_windows) {  // where the run's columns begin and end in the windows' lists
        const uint32_t w = r.w0 + threadIdx.x / 2, t0 = rowOffset[w];
        const uint32_t *own = tcA2B + (uint64_t)t0 * kCW;
        uint32_t lo = 0, hi = (rowOffset[w + 1] - t0) * kCW;
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2, c = own[mid];
            if ((threadIdx.x & 1u) ? c <= highest : c < lowest) lo = mid + 1; else hi = mid;
        }
        bound[threadIdx.x] = lo;
        if (!(threadIdx.x & 1u)) first[threadIdx.x / 2] = t0;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t sum = 0;
        for (uint32_t k = 0; k < n_windows; ++k) {
            const uint32_t begin = bound[2 * k], end = bound[2 * k + 1];
            tiles_before[k] = sum;
            first[k] += begin / kCW;
            if (end > begin) sum += (end - 1) / kCW + 1 - begin / kCW;
        }
        tiles_before[n_windows] = sum;
    }
    __syncthreads();
    const uint32_t n_tiles = tiles_before[n_windows];
    struct Source {
        uint32_t column, row;
        alignas(16) T v[kPer];
    };
    auto load = [&](uint32_t i, Source &s) {
        uint32_t k = 0;
        while (i >= tiles_before[k + 1]) ++k;
        const uint64_t t = first[k] + (i - tiles_before[k]);
        s.column = __ldg(tcA2B + t * kCW + lane % kCW);
        *reinterpret_cast<uint4 *>(s.v) = __ldcs(reinterpret_cast<const uint4 *>(data + (t * 32 + lane) * kPer));
        s.row = __ldg(rowIdx + r.w0 + k) - r.row0 + (lane >> 1);
    };
    Source now, next;
    if (warp < n_tiles) load(warp, next);
    for (uint32_t i = warp; i < n_tiles; i += kTilesBlock / 32) {
        now = next;
        if (i + kTilesBlock / 32 < n_tiles) load(i + kTilesBlock / 32, next);
        uint32_t lo = 0, hi = n_real;  // the slot of the lane's column
        while (lo < hi) {
            const uint32_t mid = lo + (hi - lo) / 2;
            if (list[mid] < now.column) lo = mid + 1; else hi = mid;
        }
        const uint32_t slot = lo < n_real && list[lo] == now.column ? lo : kIdxMax;
        uint8_t *row = image + now.row * 32u;
        const uint32_t flip = (now.row >> 2) & 1u;
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t at = __shfl_sync(0xffffffffu, slot, (lane & 1u) * kPer + k);
            if (at == kIdxMax) continue;
            const uint32_t in_tile = at % kCW;
            *reinterpret_cast<T *>(row + at / kCW * 4096u + ((in_tile / kPer) ^ flip) * 16u + in_tile % kPer * sizeof(T)) = now.v[k];
        }
    }
    __syncthreads();
    uint4 *out = reinterpret_cast<uint4 *>(images + (uint64_t)r.image * 4096u);
    for (uint32_t k = threadIdx.x; k < r.n_tiles * 256; k += kTilesBlock) __stcs(out + k, reinterpret_cast<const uint4 *>(image)[k]);
}

// Distinct columns in the lists of a run of 16-row tiles, one block per run.
__global__ void __launch_bounds__(1024)
distinct_columns_kernel(const uint32_t *__restrict__ tcA2B, const uint2 *__restrict__ ranges, uint32_t cw, uint64_t cols, uint64_t words,
                        uint32_t *__restrict__ bits, uint32_t *__restrict__ distinct) {
    __shared__ uint32_t total;
    if (threadIdx.x == 0) total = 0;
    __syncthreads();
    const uint64_t end = (uint64_t)ranges[blockIdx.x].y * cw;
    uint32_t *mine = bits + blockIdx.x * words, n = 0;
    for (uint64_t e = (uint64_t)ranges[blockIdx.x].x * cw + threadIdx.x; e < end; e += 1024) {
        const uint32_t c = tcA2B[e];
        if (c < cols && c != kIdxMax && !(atomicOr(mine + (c >> 5), 1u << (c & 31u)) & (1u << (c & 31u)))) ++n;
    }
    atomicAdd(&total, n);
    __syncthreads();
    if (threadIdx.x == 0) distinct[blockIdx.x] = total;
}

// Runs of 16-row windows that fall into the same 128-row window.
void group_windows(const uint32_t *h_rowIdx, uint64_t eff, uint32_t kTall, std::vector<uint32_t> *win_group,
                   std::vector<uint64_t> *group_first) {
    win_group->resize(eff);
    group_first->clear();
    for (uint64_t i = 0; i < eff; ++i) {
        if (i == 0 || h_rowIdx[i] / kTall != h_rowIdx[i - 1] / kTall) group_first->push_back(i);
        (*win_group)[i] = (uint32_t)(group_first->size() - 1);
    }
    group_first->push_back(eff);
}

// (always the same limit, whoever else is about to launch)
template <typename K>
int allow_bit_sets(K kernel, int sets) {
    B200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sets * (int)kChunkWords * 4));
    return B200SPMM_OK;
}

}  // namespace

int estimate_tall_tile_ratio(const b200spmm_btcf_info_t &info, const uint32_t *h_rowOffset, const uint32_t *h_rowIdx,
                             const uint32_t *d_tcA2B, uint32_t tall_rows, int max_samples, double *ratio,
                             uint64_t *n_super_windows) {
    const uint64_t eff = info.eff_row_windows, cw = (uint64_t)info.col_window;
    std::vector<uint32_t> win_group;
    std::vector<uint64_t> group_first;
    group_windows(h_rowIdx, eff, tall_rows, &win_group, &group_first);
    const uint64_t n_groups = group_first.size() - 1;
    *n_super_windows = n_groups;
    *ratio = 1.0;
    if (!n_groups || max_samples < 1) return B200SPMM_OK;
    // one bit per column and sampled super-window, at most 64 MB of them
    const uint64_t words = info.cols / 32 + 1;
    const uint64_t n_samples = std::max<uint64_t>(1, std::min({(uint64_t)max_samples, n_groups, ((uint64_t)16 << 20) / words}));
    std::vector<uint2> ranges;
    uint64_t short_tiles = 0, tall_tiles = 0;
    for (uint64_t k = 0; k < n_samples; ++k) {
        const uint64_t g = (2 * k + 1) * n_groups / (2 * n_samples);
        ranges.push_back(make_uint2(h_rowOffset[group_first[g]], h_rowOffset[group_first[g + 1]]));
        short_tiles += ranges.back().y - ranges.back().x;
    }
    PoolScratch tmp;
    uint2 *d_ranges = nullptr;
    uint32_t *bits = nullptr, *d_distinct = nullptr;
    B200_CUDA_TRY(tmp.alloc(&d_ranges, n_samples));
    B200_CUDA_TRY(tmp.alloc(&d_distinct, n_samples));
    B200_CUDA_TRY(tmp.alloc(&bits, n_samples * words));
    B200_CUDA_TRY(cudaMemsetAsync(bits, 0, n_samples * words * 4));
    B200_CUDA_TRY(cudaMemcpy(d_ranges, ranges.data(), n_samples * sizeof(uint2), cudaMemcpyHostToDevice));
    distinct_columns_kernel<<<(unsigned)n_samples, 1024>>>(d_tcA2B, d_ranges, (uint32_t)cw, info.cols, words, bits, d_distinct);
    B200_CUDA_TRY(cudaGetLastError());
    std::vector<uint32_t> distinct(n_samples);
    B200_CUDA_TRY(cudaMemcpy(distinct.data(), d_distinct, n_samples * 4, cudaMemcpyDeviceToHost));
    for (uint32_t d : distinct) tall_tiles += (d + cw - 1) / cw;
    if (short_tiles) *ratio = (double)tall_tiles / (double)short_tiles;
    return B200SPMM_OK;
}

int count_super_windows(const b200spmm_btcf_info_t &info, const uint32_t *h_rowOffset, const uint32_t *h_rowIdx, const uint32_t *d_tcA2B,
                        SuperCounts *out) {
    *out = SuperCounts();
    const uint64_t eff = info.eff_row_windows;
    std::vector<WindowPair> pairs;
    for (uint64_t i = 0; i < eff;) {
        SuperCounts::Pair w{(uint32_t)(h_rowIdx[i] / 256u * 256u), (uint32_t)i, (uint32_t)i, (uint32_t)i, {}};
        while (w.mid < eff && h_rowIdx[w.mid] - w.row0 < 128u) ++w.mid;
        w.end = w.mid;
        while (w.end < eff && h_rowIdx[w.end] - w.row0 < 256u) ++w.end;
        pairs.push_back(WindowPair{h_rowOffset[w.begin], h_rowOffset[w.mid], h_rowOffset[w.end]});
        out->pairs.push_back(w);
        i = w.end;
    }
    if (pairs.empty()) return B200SPMM_OK;
    PoolScratch tmp;
    WindowPair *d_pairs = nullptr;
    uint32_t *d_counts = nullptr;
    B200_CUDA_TRY(tmp.alloc(&d_pairs, pairs.size()));
    B200_CUDA_TRY(tmp.alloc(&d_counts, 3 * pairs.size()));
    B200_CUDA_TRY(cudaMemcpy(d_pairs, pairs.data(), pairs.size() * sizeof(WindowPair), cudaMemcpyHostToDevice));
    const uint32_t words = chunk_words(info.cols);
    const int st = allow_bit_sets(count_kernel, 2);
    if (st != B200SPMM_OK) return st;
    count_kernel<<<(unsigned)pairs.size(), kMergeBlock, 2 * words * 4>>>(d_pairs, d_tcA2B, (uint32_t)info.col_window, info.cols, words, d_counts);
    B200_CUDA_TRY(cudaGetLastError());
    std::vector<uint32_t> counts(3 * pairs.size());
    B200_CUDA_TRY(cudaMemcpy(counts.data(), d_counts, counts.size() * 4, cudaMemcpyDeviceToHost));
    const uint32_t cw = (uint32_t)info.col_window;
    for (size_t k = 0; k < pairs.size(); ++k) {
        for (int j = 0; j < 3; ++j) out->pairs[k].tiles[j] = (counts[3 * k + j] + cw - 1) / cw;
        out->tall_tiles += (uint64_t)out->pairs[k].tiles[0] + out->pairs[k].tiles[1];
        out->pair_tiles += out->pairs[k].tiles[2];
        out->tall_windows += (out->pairs[k].tiles[0] != 0) + (out->pairs[k].tiles[1] != 0);
    }
    return B200SPMM_OK;
}

void free_tall(TallFormat *t) {
    pool_free(t->d_rowOffset);  // (d_rowIdx is behind it)
    pool_free(t->d_tcA2B);
    pool_free(t->d_data);
    *t = TallFormat();
}

int build_tall_device(const b200spmm_btcf_info_t &info, const SuperCounts &counts, const uint32_t *h_rowOffset, const uint32_t *d_rowOffset,
                      const uint32_t *d_tcA2B, const void *d_data, const uint32_t *d_rowIdx, uint32_t tall_rows, TallFormat *out) {
    *out = TallFormat();
    if (info.row_window != (int)kShort || (tall_rows != 128 && tall_rows != 256)) return B200SPMM_ERR_UNSUPPORTED;
    const uint32_t cw = (uint32_t)info.col_window, parts = tall_rows / 128;
    // (images are numbered in 32 bits here, and rowOffset is 32-bit)
    if ((tall_rows == 256 ? 2 * counts.pair_tiles : counts.tall_tiles) > 0xFFFFFFFFull) return B200SPMM_ERR_UNSUPPORTED;
    std::vector<uint32_t> rowOffset{0}, rowIdx;
    std::vector<WindowLists> windows;
    std::vector<TileRun> runs;
    TallFormat t;
    t.rows = tall_rows;
    // windows [begin, end) of 16 rows with `n` tiles when merged; half j of a 256-row window has images [j n, j n + n)
    auto add = [&](const SuperCounts::Pair &w, uint32_t begin, uint32_t end, uint32_t row0, uint32_t n) {
        if (!n) return;
        const uint32_t list = rowOffset.back();
        windows.push_back(WindowLists{h_rowOffset[begin], h_rowOffset[end], list, n});
        rowIdx.push_back(row0);
        rowOffset.push_back(list + n);
        t.max_window_tiles = std::max<uint64_t>(t.max_window_tiles, n);
        t.min_window_tiles = windows.size() == 1 ? n : std::min<uint64_t>(t.min_window_tiles, n);
        for (uint32_t j = 0; j < parts; ++j) {
            const uint32_t b = parts == 1 ? begin : j ? w.mid : w.begin, e = parts == 1 ? end : j ? w.end : w.mid;
            for (uint32_t k = 0; k < n; k += kRunTiles)
                runs.push_back(TileRun{b, e, row0 + j * 128u, list + k, std::min(kRunTiles, n - k), list * parts + j * n + k});
        }
    };
    for (const SuperCounts::Pair &w : counts.pairs) {
        if (parts == 2) {
            add(w, w.begin, w.end, w.row0, w.tiles[2]);
        } else {
            add(w, w.begin, w.mid, w.row0, w.tiles[0]);
            add(w, w.mid, w.end, w.row0 + 128u, w.tiles[1]);
        }
    }
    t.eff = windows.size();
    t.tiles = rowOffset.back();
    if (!t.tiles) return B200SPMM_OK;
    struct Guard {
        TallFormat *t;
        ~Guard() { if (t) free_tall(t); }
    } guard{&t};
    // one copy brings all tables (a copy is 8 us, whatever it holds): rowOffset, the aligned tiles, rowIdx, windows, runs
    std::vector<uint32_t> tables(rowOffset);
    auto append = [&](const void *from, size_t bytes) {
        const size_t at = tables.size();
        tables.resize(at + bytes / 4);
        std::memcpy(tables.data() + at, from, bytes);
        return at;
    };
    const uint32_t none = 0;
    const size_t aligned_at = append(&none, 4), rowIdx_at = append(rowIdx.data(), rowIdx.size() * 4),
                 windows_at = append(windows.data(), windows.size() * sizeof(WindowLists)), runs_at = append(runs.data(), runs.size() * sizeof(TileRun));
    B200_CUDA_TRY(pool_alloc(&t.d_rowOffset, tables.size()));
    B200_CUDA_TRY(cudaMemcpy(t.d_rowOffset, tables.data(), tables.size() * 4, cudaMemcpyHostToDevice));
    t.d_rowIdx = t.d_rowOffset + rowIdx_at;
    t.d_aligned = t.d_rowOffset + aligned_at;
    const auto *d_windows = reinterpret_cast<const WindowLists *>(t.d_rowOffset + windows_at);
    const auto *d_runs = reinterpret_cast<const TileRun *>(t.d_rowOffset + runs_at);
    B200_CUDA_TRY(pool_alloc(&t.d_tcA2B, t.tiles * cw));
    B200_CUDA_TRY(pool_alloc_bytes(&t.d_data, t.tiles * parts * 4096, nullptr));
    const uint32_t words = chunk_words(info.cols);
    const int st = allow_bit_sets(lists_kernel, 1);
    if (st != B200SPMM_OK) return st;
    lists_kernel<<<(unsigned)windows.size(), kMergeBlock, words * 4>>>(d_windows, d_tcA2B, cw, info.cols, words, t.d_tcA2B, t.d_aligned);
    B200_CUDA_TRY(cudaGetLastError());
    if (info.elt_size == 2)
        tiles_kernel<uint16_t><<<(unsigned)runs.size(), kTilesBlock>>>(d_runs, d_rowOffset, d_tcA2B, static_cast<const uint16_t *>(d_data), d_rowIdx,
                                                                       t.d_tcA2B, static_cast<uint8_t *>(t.d_data));
    else
        tiles_kernel<uint32_t><<<(unsigned)runs.size(), kTilesBlock>>>(d_runs, d_rowOffset, d_tcA2B, static_cast<const uint32_t *>(d_data), d_rowIdx,
                                                                       t.d_tcA2B, static_cast<uint8_t *>(t.d_data));
    B200_CUDA_TRY(cudaGetLastError());
    t.h_rowOffset = std::move(rowOffset);
    *out = t;
    guard.t = nullptr;
    return B200SPMM_OK;
}

}  // namespace b200spmm
