// CSR -> condensed row-window tiles on the GPU.  Same output, bit for bit, as the host converter
// (format.cpp) and therefore as the reference's CSR2BTCFNOBITMAP (src/utils/convert.h:146-225),
// for CSR whose rows hold ascending, distinct columns (what the reference's loader produces,
// src/utils/load.h:137-145,256).  The reference converts on one host thread; the largest
// benchmark matrix (5.2e8 entries) takes ten seconds on sixteen host cores and well under one on
// the device.
//
// A matrix whose windows are not too empty for it (see window_bits_pay) is converted window by window: a block marks
// the window's columns in a bit set in shared memory and lists them in order; after one scan over the windows the lists
// move to their places.  60,000 nodes, 700,000 entries: 67 us with the values, where the sort took 101.  A block of 512 or 1024
// threads is slower (conversion 140 us a call with 256, 164 with 512): most windows have a few hundred entries.
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
//   4. column lists scattered into tcA2B (pre-filled with 0xFFFFFFFF padding); every entry finds its slot by binary search in its window's column list and is written into
//      the zero-filled tile array
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

struct Totals {
    uint64_t n_unique;
    unsigned long long windows_tiles;  // windows that hold entries << 32 | their tiles
    uint32_t bad;
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

constexpr int kBitsBlock = 256;
constexpr size_t kBitsSmemMax = 100 * 1024;
constexpr uint32_t kGroupWords = 8;  // words of the bit set that share a rank

inline uint32_t bit_words(uint64_t cols) { return (uint32_t)((cols + 32 * kGroupWords - 1) / (32 * kGroupWords)) * kGroupWords; }
inline size_t bits_smem(uint64_t cols) { return (size_t)bit_words(cols) * 4 + (size_t)(bit_words(cols) / kGroupWords) * 4; }

// A pass over the bit set costs a window its words, four at a time, where the sort costs an entry four or more passes
// of ~20 bytes each.  Conversion of graphs in us, sets against sort, at words of the sets per entry: 133 / 212 at 10,
// 151 / 218 at 23, 3,930 / 5,208 at 36, 272 / 268 at 58, 705 / 490 at 90.  The set has to leave room for two blocks an SM.
inline bool window_bits_pay(uint64_t n_windows, uint64_t cols, uint64_t nnz) {
    return bits_smem(cols) <= kBitsSmemMax && n_windows * bit_words(cols) <= 40 * nnz;
}

// The distinct columns of every window in order, at columns[first entry of the window ..], and how many they are.
__global__ void __launch_bounds__(kBitsBlock)
window_columns_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ col_idx, uint32_t rows, uint32_t cols, uint32_t nnz,
                      uint32_t row_window, uint32_t n_windows, uint32_t words, uint32_t *__restrict__ columns, uint32_t *__restrict__ count,
                      Totals *__restrict__ totals) {
    constexpr int kUnroll = 8;  // columns of a thread in flight
    extern __shared__ __align__(16) uint32_t bits[];
    __shared__ uint32_t start[32], sums[kBitsBlock / 32];
    const uint32_t groups = words / kGroupWords, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t *rank = bits + words;  // columns in the groups before
    if (blockIdx.x == 0 && threadIdx.x == 0 && (row_ptr[0] != 0 || row_ptr[rows] != nnz)) atomicOr(&totals->bad, 1u);
    for (uint32_t w = blockIdx.x; w < n_windows; w += gridDim.x) {
        bool ok = true;
        if (threadIdx.x <= row_window) {
            const uint64_t r = (uint64_t)w * row_window + threadIdx.x;
            const uint32_t s = row_ptr[min(r, (uint64_t)rows)], prev = threadIdx.x ? row_ptr[min(r - 1, (uint64_t)rows)] : 0u;
            start[threadIdx.x] = s;
            ok = s <= nnz && prev <= s;
        }
        for (uint32_t k = threadIdx.x; k < words / 4; k += kBitsBlock) reinterpret_cast<uint4 *>(bits)[k] = make_uint4(0, 0, 0, 0);
        ok = __syncthreads_and(ok);
        const uint32_t p0 = start[0], p1 = start[row_window];
        if (!ok || p0 == p1) {
            if (threadIdx.x == 0) {
                count[w] = 0;
                if (!ok) atomicOr(&totals->bad, 1u);
            }
            __syncthreads();
            continue;
        }
        for (uint32_t q = p0 + threadIdx.x; q < p1; q += kUnroll * kBitsBlock) {  // (no overflow: p1 <= 2^32 - 1 is checked by the host)
            uint32_t c[kUnroll], left[kUnroll];
#pragma unroll
            for (int k = 0; k < kUnroll; ++k) {
                const uint64_t p = (uint64_t)q + (uint32_t)k * kBitsBlock;
                c[k] = p < p1 ? col_idx[p] : 0u;
                left[k] = p < p1 && p > p0 ? col_idx[p - 1] : 0u;
            }
#pragma unroll
            for (int k = 0; k < kUnroll; ++k) {
                const uint64_t p = (uint64_t)q + (uint32_t)k * kBitsBlock;
                if (p >= p1) break;
                if (p > p0 && left[k] >= c[k]) {  // only where a row starts
                    bool row_start = false;
                    for (uint32_t r = 1; r < row_window; ++r) row_start |= start[r] == p;
                    if (!row_start) atomicOr(&totals->bad, 1u);
                }
                if (c[k] < cols) atomicOr(bits + (c[k] >> 5), 1u << (c[k] & 31u));
                else atomicOr(&totals->bad, 1u);
            }
            if (p1 - q <= kUnroll * kBitsBlock) break;
        }
        __syncthreads();
        uint32_t base = 0;
        for (uint32_t g0 = 0; g0 < groups; g0 += kBitsBlock) {  // one group a thread
            const uint32_t g = g0 + threadIdx.x;
            uint32_t mine = 0;
            if (g < groups)
#pragma unroll
                for (uint32_t k = 0; k < kGroupWords; ++k) mine += __popc(bits[g * kGroupWords + k]);
            uint32_t upto = mine;
#pragma unroll
            for (int d = 1; d < 32; d *= 2) {
                const uint32_t x = __shfl_up_sync(0xffffffffu, upto, d);
                if (lane >= (uint32_t)d) upto += x;
            }
            __syncthreads();  // `sums` of the round before has been read
            if (lane == 31) sums[warp] = upto;
            __syncthreads();
            uint32_t before = base;
            for (uint32_t k = 0; k < kBitsBlock / 32; ++k) {
                if (k < warp) before += sums[k];
                base += sums[k];
            }
            if (g < groups) rank[g] = before + upto - mine;
        }
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < words; k += kBitsBlock) {
            uint32_t b = bits[k];
            if (!b) continue;
            uint32_t at = p0 + rank[k / kGroupWords];
            for (uint32_t j = k / kGroupWords * kGroupWords; j < k; ++j) at += __popc(bits[j]);
            for (; b; b &= b - 1u) columns[at++] = k * 32u + (uint32_t)__ffs((int)b) - 1u;
        }
        if (threadIdx.x == 0) count[w] = base;
        __syncthreads();  // the next window clears the set
    }
}

// The lists at their places, padded to whole tiles.
__global__ void __launch_bounds__(kBitsBlock)
place_columns_kernel(const uint32_t *__restrict__ row_ptr, const uint32_t *__restrict__ columns, const uint32_t *__restrict__ count,
                     const uint32_t *__restrict__ tile_of, uint32_t n_windows, uint32_t row_window, uint32_t col_window,
                     uint32_t *__restrict__ tcA2B) {
    for (uint32_t w = blockIdx.x; w < n_windows; w += gridDim.x) {
        const uint32_t n = count[w], padded = (n + col_window - 1) / col_window * col_window;
        if (!n) continue;
        const uint32_t *from = columns + row_ptr[w * row_window];
        uint32_t *list = tcA2B + (uint64_t)tile_of[w] * col_window;
#pragma unroll 4
        for (uint32_t k = threadIdx.x; k < padded; k += kBitsBlock) list[k] = k < n ? from[k] : 0xFFFFFFFFu;
    }
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

int convert_by_windows(b200spmm_dbtcf *f, const uint32_t *d_row_ptr, const uint32_t *d_col_idx, const void *d_values, cudaStream_t stream) {
    const uint32_t rows = (uint32_t)f->info.rows, cols = (uint32_t)f->info.cols, nnz = (uint32_t)f->info.nnzs;
    const uint32_t n_windows = (uint32_t)f->info.total_row_windows, RW = (uint32_t)f->info.row_window, CW = (uint32_t)f->info.col_window;
    const uint32_t words = bit_words(f->info.cols);
    const size_t smem = bits_smem(f->info.cols);
    const int esz = f->info.elt_size;
    PoolScratch tmp(stream);
    Totals *totals = nullptr;
    uint32_t *columns = nullptr, *count = nullptr, *tile_of = nullptr;
    B200_CUDA_TRY(tmp.alloc(&columns, nnz));
    unsigned long long *before = nullptr;
    B200_CUDA_TRY(tmp.alloc(&totals, 1));
    B200_CUDA_TRY(tmp.alloc(&count, n_windows));
    B200_CUDA_TRY(tmp.alloc(&tile_of, n_windows));
    B200_CUDA_TRY(tmp.alloc(&before, (size_t)n_windows + 1));
    const WindowTerms windows{nullptr, count, n_windows, CW};
    auto terms = thrust::make_transform_iterator(thrust::make_counting_iterator<uint32_t>(0), windows);
    size_t scan_bytes = 0;
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(nullptr, scan_bytes, terms, before, (int64_t)n_windows + 1, stream));
    uint8_t *scan_tmp = nullptr;
    B200_CUDA_TRY(tmp.alloc(&scan_tmp, scan_bytes));
    B200_CUDA_TRY(pool_alloc(&f->d_rowOffset, (size_t)n_windows + 1, stream));
    B200_CUDA_TRY(pool_alloc(&f->d_rowIdx, n_windows, stream));
    if (smem > 47 * 1024)  // (48 KB hold the kernel's own shared variables, too)
        B200_CUDA_TRY(cudaFuncSetAttribute(window_columns_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBitsSmemMax));
    const unsigned grid = std::min<uint32_t>(n_windows, 148 * 64), table_grid = n_windows / kBlock + 1;
    B200_CUDA_TRY(cudaMemsetAsync(totals, 0, sizeof(Totals), stream));
    window_columns_kernel<<<grid, kBitsBlock, smem, stream>>>(d_row_ptr, d_col_idx, rows, cols, nnz, RW, n_windows, words, columns, count,
                                                                 totals);
    B200_CUDA_TRY(cudaGetLastError());
    B200_CUDA_TRY(cub::DeviceScan::ExclusiveSum(scan_tmp, scan_bytes, terms, before, (int64_t)n_windows + 1, stream));
    window_tables_kernel<<<table_grid, kBlock, 0, stream>>>(before, n_windows, RW, f->d_rowOffset, f->d_rowIdx, tile_of, totals);
    B200_CUDA_TRY(cudaGetLastError());
    Totals h;
    B200_CUDA_TRY(cudaMemcpyAsync(&h, totals, sizeof(h), cudaMemcpyDeviceToHost, stream));
    B200_CUDA_TRY(cudaStreamSynchronize(stream));
    if (h.bad) return B200SPMM_ERR_BAD_CSR;
    f->info.eff_row_windows = h.windows_tiles >> 32;
    f->info.total_tiles = (uint32_t)h.windows_tiles;
    const uint64_t data_bytes = f->info.total_tiles * RW * CW * esz;
    B200_CUDA_TRY(pool_alloc(&f->d_tcA2B, f->info.total_tiles * CW, stream));
    B200_CUDA_TRY(pool_alloc_bytes(&f->d_data, std::max<uint64_t>(data_bytes, 16), stream));
    B200_CUDA_TRY(cudaMemsetAsync(f->d_data, 0, data_bytes, stream));
    place_columns_kernel<<<grid, kBitsBlock, 0, stream>>>(d_row_ptr, columns, count, tile_of, n_windows, RW, CW, f->d_tcA2B);
    scatter_values(f, d_row_ptr, d_col_idx, d_values, windows, tile_of, stream);
    B200_CUDA_TRY(cudaGetLastError());
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

    if (window_bits_pay(n_windows, cols, nnz)) {
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
