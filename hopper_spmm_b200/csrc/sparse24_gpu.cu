// Dense tiles of 256-row super-windows -> the 2:4 form, on the device.
//
// tcgen05.mma.sp multiplies 32 columns where tcgen05.mma multiplies 16, in the same time and with the same sixteen values a
// row, if a row has at most two entries in every four neighbouring columns of the list.  At 10 % unstructured density one
// group in 270 has more; its first entries beyond two, 0.9 % of all, become the row's rest, which the kernel's epilogue warps
// multiply while the tensor core works.
//
// The instruction multiplies two columns of a group whatever the row has there.  A zero times an infinity in B is NaN, and a
// row that meets the infinity must keep it: idle places name columns that the row has no entry in, which the dense tile
// multiplies by zero, too.  There are always enough of them.
//
//   1. tiles_kernel: a block takes kBlockTiles tiles of a window and a thread a row.  It marks the entries that go to the rest in
//      shared memory and, when it knows how many they are, asks for places in the row's list
//   2. rest_kernel: blocks have asked in any order; every row's list is sorted by column
// Only the length of a row's list is limited (kSparse24MaxRest).  With a limit of seven for every 16 tiles of a row as well,
// one row-block of 2.5e-7 decided for the whole matrix: one 28672 x 8192 weight of ten at 10 %, 45 of a hundred at 10.9 %.
// Bound by reading the dense tiles.
#include <algorithm>
#include <vector>

#include "common.hpp"
#include "device_pool.hpp"
#include "format.hpp"
#include "sparse24_gpu.hpp"

namespace b200spmm {
namespace {

constexpr int kRows = 256;            // of a window, and threads of a block
constexpr uint32_t kBlockTiles = 16;  // of 32 columns
// Entries of the rest a row and dense tile, up to which the form pays: the epilogue warps get through 0.02 while the tensor core
// does a tile.  28672 x 8192, dense and so in turn, us of a loop of calls (and of single ones after 3 ms of rest): 192 columns, half
// results, 10 % (0.015) 109 and 98 (117 and 102), 11 % (0.020) 107 and 104 (117 and 106), 12 % (0.026) 108 and 115 (118 and 117), 14 %
// (0.040) 107 and 139; 2,048 columns, 10 % 738 and 688 at 1,635 MHz under the power cap (692 and 608), 11 % 735 and 731 (691 and 637),
// 12 % 735 and 802 (695 and 703), 14 % 733 and 990.
constexpr double kMostRest = 0.02;

constexpr unsigned long long kUnfit = 1ull << 63;  // in the number of all entries of the rest: some row has too many

struct Row {
    uint32_t w[8];  // sixteen fp16
    __device__ __forceinline__ void load(const uint4 *__restrict__ image, uint32_t r) {  // r: row of 128
        const uint32_t flip = (r >> 2) & 1u;
        reinterpret_cast<uint4 *>(w)[0] = __ldcs(image + 2 * r + flip);
        reinterpret_cast<uint4 *>(w)[1] = __ldcs(image + 2 * r + (flip ^ 1u));
    }
    // value of column idx (0..3) of group g, and which of the four have bits
    __device__ __forceinline__ uint32_t value(int g, uint32_t idx) const { return ((idx & 2u) ? w[2 * g + 1] : w[2 * g]) >> ((idx & 1u) * 16u) & 0xFFFFu; }
    __device__ __forceinline__ uint32_t mask(int g) const {
        return ((w[2 * g] & 0xFFFFu) ? 1u : 0u) | ((w[2 * g] >> 16) ? 2u : 0u) | ((w[2 * g + 1] & 0xFFFFu) ? 4u : 0u) | ((w[2 * g + 1] >> 16) ? 8u : 0u);
    }
};

// What a sample of the matrix has beyond two in a group of four: totals[0] entries in totals[1] dense tiles.  A block takes as
// many tiles as in tiles_kernel.
constexpr uint32_t kSampleBlocks = 296;
__global__ void __launch_bounds__(kRows)
sample_kernel(const uint32_t *__restrict__ denseOffset, const uint4 *__restrict__ dense, uint32_t n_windows, unsigned long long *__restrict__ totals) {
    const uint32_t w = (uint32_t)((2ull * blockIdx.x + 1) * n_windows / (2 * kSampleBlocks)), first = denseOffset[w], n = denseOffset[w + 1] - first;
    const uint32_t runs = (n + kBlockTiles - 1) / kBlockTiles, t0 = blockIdx.x * 5u % runs * kBlockTiles, t1 = min(t0 + kBlockTiles, n);
    const uint32_t half = threadIdx.x >> 7, r = threadIdx.x & 127u;
    const uint4 *from = dense + ((uint64_t)first * 2 + half * n) * 256;
    uint32_t beyond = 0;
#pragma unroll 4
    for (uint32_t t = t0; t < t1; ++t) {
        Row row;
        row.load(from + (uint64_t)t * 256, r);
#pragma unroll
        for (int g = 0; g < 4; ++g) beyond += (uint32_t)max(__popc(row.mask(g)) - 2, 0);
    }
    beyond = __reduce_add_sync(0xffffffffu, beyond);
    if ((threadIdx.x & 31u) == 0 && beyond) atomicAdd(totals, (unsigned long long)beyond);
    if (threadIdx.x == 0) atomicAdd(totals + 1, (unsigned long long)(t1 - t0));
}

__global__ void __launch_bounds__(kRows)
tiles_kernel(const uint32_t *__restrict__ denseOffset, const uint32_t *__restrict__ dense_lists, const uint4 *__restrict__ dense,
             const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ quads, uint32_t *__restrict__ lists, uint4 *__restrict__ data,
             uint16_t *__restrict__ meta, uint32_t *__restrict__ n_rest, uint32_t *__restrict__ rest, unsigned long long *__restrict__ total) {
    __shared__ uint32_t beyond[kBlockTiles][kRows];  // columns of a row and tile that go to the rest
    const uint32_t w = blockIdx.x, first = denseOffset[w], n = denseOffset[w + 1] - first, out = rowOffset[w], n_out = rowOffset[w + 1] - out;
    const uint32_t k0 = blockIdx.y * kBlockTiles, k1 = min(k0 + kBlockTiles, n_out), half = threadIdx.x >> 7, r = threadIdx.x & 127u, flip = (r >> 2) & 1u;
    uint32_t n_mine = 0;
    const uint32_t *list = dense_lists + (uint64_t)first * 16u;
    if (k0 < k1) {
        for (uint32_t k = k0 * 32u + threadIdx.x; k < k1 * 32u; k += kRows) lists[(uint64_t)out * 32u + k] = k < n * 16u ? list[k] : kIdxMax;
        const uint4 *from = dense + ((uint64_t)first * 2 + half * n) * 256;
        uint4 *to = data + ((uint64_t)out * 2 + half * n_out) * 256 + 2 * r;
        // Tensor memory wants the rows 16 m2 + 8 m1 + m0 in lanes 16 m2 + m0 (columns 0-15) and 16 m2 + 8 + m0 (16-31), m1 in a half word.
        uint16_t *m_to = meta + ((uint64_t)quads[w] * 2 + half * (quads[w + 1] - quads[w])) * 1024u + ((r >> 4) * 16u + (r & 7u)) * 8u + (r >> 3 & 1u);
#pragma unroll 2
        for (uint32_t k = k0; k < k1; ++k) {
            uint32_t v[8] = {}, m[2] = {0x4444u, 0x4444u}, over = 0;
#pragma unroll
            for (uint32_t h = 0; h < 2; ++h) {
                const uint32_t t = 2 * k + h;
                if (t >= n) break;
                Row row;
                row.load(from + (uint64_t)t * 256, r);
                m[h] = 0;
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const uint32_t met = row.mask(g);
                    uint32_t have = met;
                    while (__popc(have) > 2) have &= have - 1u;
                    over |= (met ^ have) << (16 * h + 4 * g);
                    uint32_t two = have, idle = ~met & 15u;
                    while (__popc(two) < 2) {
                        two |= idle & (0u - idle);
                        idle &= idle - 1u;
                    }
                    const uint32_t lo = (uint32_t)__ffs((int)two) - 1u, hi = 31u - (uint32_t)__clz((int)two);
                    m[h] |= (lo | hi << 2) << (4 * g);
                    v[4 * h + g] = (have >> lo & 1u ? row.value(g, lo) : 0u) | (have >> hi & 1u ? row.value(g, hi) : 0u) << 16;
                }
            }
            __stcs(to + (uint64_t)k * 256 + flip, make_uint4(v[0], v[1], v[2], v[3]));
            __stcs(to + (uint64_t)k * 256 + (flip ^ 1u), make_uint4(v[4], v[5], v[6], v[7]));
            uint16_t *mk = m_to + (uint64_t)(k / 4) * 1024u + (k & 3u) * 2u;
            mk[0] = (uint16_t)m[0];
            mk[64] = (uint16_t)m[1];
            beyond[k - k0][threadIdx.x] = over;
            n_mine += (uint32_t)__popc(over);
        }
        if (n_mine) {
            uint32_t at = atomicAdd(n_rest + (uint64_t)w * kRows + threadIdx.x, n_mine);
            const uint16_t *values = reinterpret_cast<const uint16_t *>(from + 2 * r);
            for (uint32_t k = k0; k < k1; ++k)
                for (uint32_t over = beyond[k - k0][threadIdx.x]; over; over &= over - 1u, ++at) {
                    const uint32_t in_tile = (uint32_t)__ffs((int)over) - 1u, c = in_tile & 15u;
                    const uint64_t t = 2 * k + (in_tile >> 4);
                    if (at < kSparse24MaxRest)
                        rest[((uint64_t)w * kSparse24MaxRest + at) * kRows + threadIdx.x] =
                            list[t * 16u + c] << 16 | values[t * 2048 + ((c >> 3) ^ flip) * 8u + (c & 7u)];
                }
        }
    }
    const uint32_t sum = __reduce_add_sync(0xffffffffu, n_mine);
    if ((threadIdx.x & 31u) == 0 && sum) atomicAdd(total, (unsigned long long)sum);
}

__global__ void __launch_bounds__(kRows)
rest_kernel(const uint32_t *__restrict__ n_rest, uint32_t *__restrict__ rest, unsigned long long *__restrict__ total) {
    __shared__ uint32_t sorted[kSparse24MaxRest][kRows];
    const uint32_t r = threadIdx.x, n = n_rest[(uint64_t)blockIdx.x * kRows + r];
    uint32_t *list = rest + (uint64_t)blockIdx.x * (kSparse24MaxRest * kRows) + r;
    if (n > kSparse24MaxRest) {
        atomicOr(total, kUnfit);
        return;
    }
    for (uint32_t i = 0; i < n; ++i) {
        const uint32_t entry = list[i * kRows];
        uint32_t at = i;
        for (; at && sorted[at - 1][r] > entry; --at) sorted[at][r] = sorted[at - 1][r];
        sorted[at][r] = entry;
    }
    for (uint32_t i = 0; i < n; ++i) list[i * kRows] = sorted[i][r];
}

}  // namespace

void free_sparse24(Sparse24Format *f) {
    pool_free(f->d_data);  // (all lie there)
    *f = Sparse24Format();
}

int build_sparse24(const TallFormat &pair, uint64_t cols, bool always, Sparse24Format *out) {
    *out = Sparse24Format();
    if (pair.rows != (uint32_t)kRows || !pair.tiles || cols > 65536) return B200SPMM_OK;
    Sparse24Format f;
    struct Guard {
        Sparse24Format *f;
        ~Guard() { if (f) free_sparse24(f); }
    } guard{&f};
    const uint64_t n_windows = pair.eff;
    if (!always) {
        // A look at 38 MB of the tiles first, since the form is made before its rest is known: a plan of 28449 x 8119 at 26 % took
        // 6.5 ms with the form made and thrown away, 5.3 without it, now 5.4.  Up to a tenth beyond the limit all tiles decide.
        PoolScratch tmp;
        unsigned long long *d_totals = nullptr, totals[2] = {};
        cudaError_t e = tmp.alloc(&d_totals, 2);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            return B200SPMM_OK;
        }
        B200_CUDA_TRY(e);
        B200_CUDA_TRY(cudaMemsetAsync(d_totals, 0, sizeof(totals)));
        sample_kernel<<<kSampleBlocks, kRows>>>(pair.d_rowOffset, static_cast<const uint4 *>(pair.d_data), (uint32_t)n_windows, d_totals);
        B200_CUDA_TRY(cudaGetLastError());
        B200_CUDA_TRY(cudaMemcpy(totals, d_totals, sizeof(totals), cudaMemcpyDeviceToHost));
        if ((double)totals[0] > 1.1 * kMostRest * (double)kRows * (double)totals[1]) return B200SPMM_OK;
    }
    const std::vector<uint32_t> &dense = pair.h_rowOffset;
    std::vector<uint32_t> tables(2 * (n_windows + 1));
    uint32_t *rowOffset = tables.data(), *quads = rowOffset + n_windows + 1, longest = 0;
    for (uint64_t w = 0; w < n_windows; ++w) {
        const uint32_t n = (dense[w + 1] - dense[w] + 1) / 2;
        rowOffset[w + 1] = rowOffset[w] + n;
        quads[w + 1] = quads[w] + (n + 3) / 4;
        longest = std::max(longest, n);
    }
    f.tiles = rowOffset[n_windows];
    const uint32_t blocks = (longest + kBlockTiles - 1) / kBlockTiles;
    // all in one buffer, which is the driver's own where it is large (new memory costs the pool more)
    size_t bytes = 0;
    auto place = [&](size_t n) {
        const size_t at = bytes;
        bytes += (n + 255) / 256 * 256;
        return at;
    };
    const size_t data_at = place(f.tiles * 8192), meta_at = place((size_t)quads[n_windows] * 4096), lists_at = place(f.tiles * 128),
                 n_rest_at = place(n_windows * kRows * 4), total_at = place(8), rest_at = place(n_windows * kRows * kSparse24MaxRest * 4), tables_at = place(tables.size() * 4);
    const cudaError_t e = pool_alloc_bytes(&f.d_data, bytes, nullptr);
    if (e == cudaErrorMemoryAllocation) {  // no room: the dense tiles still work
        cudaGetLastError();
        return B200SPMM_OK;
    }
    B200_CUDA_TRY(e);
    auto *base = static_cast<uint8_t *>(f.d_data) + data_at;
    f.d_meta = base + meta_at;
    f.d_tcA2B = reinterpret_cast<uint32_t *>(base + lists_at);
    f.d_n_rest = reinterpret_cast<uint32_t *>(base + n_rest_at);
    f.d_rest = reinterpret_cast<uint32_t *>(base + rest_at);
    f.d_rowOffset = reinterpret_cast<uint32_t *>(base + tables_at);
    f.d_quads = f.d_rowOffset + n_windows + 1;
    B200_CUDA_TRY(cudaMemcpy(f.d_rowOffset, tables.data(), tables.size() * 4, cudaMemcpyHostToDevice));
    auto *d_total = reinterpret_cast<unsigned long long *>(base + total_at);
    B200_CUDA_TRY(cudaMemsetAsync(base + n_rest_at, 0, total_at + 8 - n_rest_at));
    tiles_kernel<<<dim3((unsigned)n_windows, blocks), kRows>>>(pair.d_rowOffset, pair.d_tcA2B, static_cast<const uint4 *>(pair.d_data), f.d_rowOffset,
                                                               f.d_quads, f.d_tcA2B, static_cast<uint4 *>(f.d_data), static_cast<uint16_t *>(f.d_meta),
                                                               f.d_n_rest, f.d_rest, d_total);
    rest_kernel<<<(unsigned)n_windows, kRows>>>(f.d_n_rest, f.d_rest, d_total);
    B200_CUDA_TRY(cudaGetLastError());
    unsigned long long total = 0;
    B200_CUDA_TRY(cudaMemcpy(&total, d_total, 8, cudaMemcpyDeviceToHost));
    if ((total & kUnfit) || (!always && (double)total > kMostRest * (double)kRows * (double)pair.tiles)) return B200SPMM_OK;
    *out = f;
    guard.f = nullptr;
    return B200SPMM_OK;
}

}  // namespace b200spmm
