// SpMM over 16-row windows by single warps: the kernel for matrices of short windows.
//
// The pipelined kernel (spmm_kernel.cuh) hands every window from its producers to the thread that issues the matrix
// instructions and on to the epilogue: a chain that costs a window what twelve tiles cost, in each pass over the
// features.  A window of ten tiles (16,384^2 of 16 x 8 blocks at 0.5 %) has nothing to hide that behind.  Here a
// warp owns a window and the features of one 128-byte line of B's rows, and nothing is handed on: D[16 rows x
// features] += Atile[16 x CW] * Bgather[CW x features] by mma.sync, whose operands lie in the warp's registers and whose
// sums stay there; there is no tensor memory to hand over and no barrier.
//
//   A  lane (g, t) = (lane / 4, lane % 4) holds 8 bytes of row g and 8 of row g + 8, four fp16 or two tf32 columns: the
//      instruction's k index is any numbering of the tile's columns as long as A and B agree on it
//   B  lane (g, t) has 16 bytes of the row of B that each of those columns names: eight lanes cover 128 bytes of a
//      row.  Element j of the 16 bytes belongs to instruction j, so that lane group g's n index stands for features
//      vec * block(g) + j; block(g) is chosen so that neighbouring t store neighbouring pieces of C
//   C  the sixteen rows leave the registers as 16-byte pieces of whole sectors
//
// Copies run two stages ahead of the products in a ring of shared memory that the warp has to itself: it waits for its
// own copies and for nobody else.  Lanes read the rows as 16 bytes of four rows at a time, whose places are exclusive-ored
// with the row so that eight lanes read different banks.  Loading them straight into registers touches four lines with
// every eight lanes and is bound by the load unit's wavefronts, 40 a kilobyte of gathered rows where a copy and its reads
// take 24 (16,384^2 of blocks at 3 %, tf32, 512 columns 165 us; 116 through the ring of one line, 103 of two).  A warp that
// multiplies two lines reads tile, columns and addresses once for both: 99 instructions a kilobyte fell to about 50.  Three
// stages of 4 KB give 16 warps an SM; two or three of 8 KB and four of 4 KB are 8 to 30 % slower.
// Where tiles and lists are not in L2 their prefetch at the start gives 12 % (16,384^2 at 0.5 %, 256 columns, matrices in turn 17.8 -> 15.6).
//
// A window's products are added in the order, and cut as, in the pipelined kernel: C has the same bits.
#pragma once

#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "common.hpp"
#include "ptx_sm100.cuh"

namespace b200spmm {

struct WindowParams {
    const uint32_t *rowOffset;  // [eff + 1] tiles
    const uint32_t *tcA2B;      // [tiles * CW]
    const uint32_t *rowIdx;     // [eff]
    const uint8_t *tiles;       // [tiles][512 bytes], row-major, or as the shared-memory image (`swizzled`)
    const void *B;              // [cols, n] row-major
    void *C;                    // [rows, n] row-major
    int64_t ldc;                // elements
    uint32_t pitch;             // bytes of a row of B
    uint32_t rows, cols, n, eff;
    uint32_t lines;             // 128-byte lines of a row of B
    uint32_t swizzled, c_is_half;
};

constexpr int kWindowWarps = 4;  // of a block
constexpr uint32_t kWindowStages = 3, kWindowStageBytes = 4096;  // of every warp
constexpr uint32_t kWindowMaxLines = 2;

namespace windowdev {

template <bool kTf32>
__device__ __forceinline__ void mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    if constexpr (kTf32)
        asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
    else
        asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
            : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
            : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// 16 bytes to shared memory, or zeros.
__device__ __forceinline__ void copy_if(uint32_t dst, const void *src, bool want) {
    ptx::cp_async_16(dst, src, want ? 16u : 0u);
}
// Brings a piece of memory into L2: whole 16-byte words.
__device__ __forceinline__ void prefetch(const void *p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// One line of a window: acc[j][0..1] / [2..3] are row g / g + 8, feature j of the blocks t and t + 4 of the line.
template <bool kTf32>
__device__ __forceinline__ void store_line(const WindowParams &p, const float (&acc)[kTf32 ? 4 : 8][4], uint32_t line, uint32_t w, uint32_t row0, uint32_t g, uint32_t t) {
    constexpr uint32_t kVec = kTf32 ? 4 : 8;
    const uint32_t f0 = line * 8u * kVec + t * kVec;
#pragma unroll
    for (uint32_t half = 0; half < 2; ++half) {
        const uint32_t row = row0 + g + 8u * half;
#pragma unroll
        for (uint32_t blk = 0; blk < 2; ++blk) {
            const uint32_t f = f0 + blk * 4u * kVec, i = 2u * half + blk;
            if constexpr (kTf32) {
                if (row >= p.rows || f >= p.n) continue;
                if (p.c_is_half) {
                    const __half2 lo = __floats2half2_rn(acc[0][i], acc[1][i]), hi = __floats2half2_rn(acc[2][i], acc[3][i]);
                    __stcs(reinterpret_cast<uint2 *>(static_cast<__half *>(p.C) + (int64_t)row * p.ldc + f),
                           make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi)));
                } else {
                    __stcs(reinterpret_cast<float4 *>(static_cast<float *>(p.C) + (int64_t)row * p.ldc + f),
                           make_float4(acc[0][i], acc[1][i], acc[2][i], acc[3][i]));
                }
            } else if (p.c_is_half) {
                uint32_t h[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const __half2 v = __floats2half2_rn(acc[2 * j][i], acc[2 * j + 1][i]);
                    h[j] = *reinterpret_cast<const uint32_t *>(&v);
                }
                if (row < p.rows && f < p.n)
                    __stcs(reinterpret_cast<uint4 *>(static_cast<__half *>(p.C) + (int64_t)row * p.ldc + f), make_uint4(h[0], h[1], h[2], h[3]));
            } else {
                // eight floats a lane: lanes t and t ^ 1 swap halves, so that a store covers whole sectors
                float mine[4], other[4];
#pragma unroll
                for (uint32_t j = 0; j < 4; ++j) {
                    const float send = (t & 1u) ? acc[j][i] : acc[4 + j][i];
                    other[j] = __shfl_xor_sync(0xffffffffu, send, 1);
                    mine[j] = (t & 1u) ? acc[4 + j][i] : acc[j][i];
                }
                const float4 m = make_float4(mine[0], mine[1], mine[2], mine[3]), o = make_float4(other[0], other[1], other[2], other[3]);
                // even t: first half of its own block and of t + 1's; odd t: second half of t - 1's and of its own
                const uint32_t fe = f - (t & 1u) * kVec + (t & 1u) * 4u;  // in the even lane's block
                float *c = static_cast<float *>(p.C) + (int64_t)row * p.ldc;
                if (row < p.rows) {
                    if (fe < p.n) __stcs(reinterpret_cast<float4 *>(c + fe), (t & 1u) ? o : m);
                    if (fe + kVec < p.n) __stcs(reinterpret_cast<float4 *>(c + fe + kVec), (t & 1u) ? m : o);
                }
            }
        }
    }
    // rows of windows without entries: those behind this window, and those ahead of the first one
    const uint32_t gap_end = w + 1 < p.eff ? __ldg(p.rowIdx + w + 1) : p.rows;
    const uint32_t csz = p.c_is_half ? 2u : 4u, line_bytes = min(8u * kVec, p.n - line * 8u * kVec) * csz;
    auto clear = [&](uint32_t from, uint32_t to) {
        for (uint32_t r = from + g; r < to; r += 8u) {
            uint8_t *c = static_cast<uint8_t *>(p.C) + ((int64_t)r * p.ldc + line * 8u * kVec) * csz;
            for (uint32_t k = t * 16u; k < line_bytes; k += 64u) *reinterpret_cast<uint4 *>(c + k) = make_uint4(0, 0, 0, 0);
        }
    };
    if (w == 0) clear(0, row0);
    if (row0 + 16u < gap_end) clear(row0 + 16u, gap_end);
}

}  // namespace windowdev

template <bool kTf32, uint32_t kLines>
__global__ void __launch_bounds__(kWindowWarps * 32, 4) spmm_window_kernel(const WindowParams p) {
    constexpr uint32_t kCW = kTf32 ? 8 : 16;
    constexpr uint32_t kVec = kTf32 ? 4 : 8;        // features of 16 bytes, and instructions a tile and line
    constexpr uint32_t kOwn = kCW / 4;              // columns of a tile that a lane has
    constexpr uint32_t kTileBytes = kCW * 128 * kLines, kTiles = kWindowStageBytes / kTileBytes;  // of a stage
    static_assert(kTiles * kTileBytes == kWindowStageBytes, "whole tiles");
    extern __shared__ __align__(128) uint8_t ring[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, g = lane >> 2, t = lane & 3u;
    const uint32_t item = blockIdx.x * kWindowWarps + warp, groups = (p.lines + kLines - 1) / kLines;  // windows x groups of lines
    const uint32_t w = item / groups, line0 = (item - w * groups) * kLines, lines = min(kLines, p.lines - line0);
    if (w >= p.eff) {
        ptx::wait_for_grids_before();
        return;
    }
    uint32_t tile = __ldg(p.rowOffset + w);
    const uint32_t end = __ldg(p.rowOffset + w + 1), row0 = __ldg(p.rowIdx + w);
    if (line0 == 0 && lane == 0) {  // all of the window's list and tiles at once; fetched stage by stage, each stage waits for DRAM
        const uint32_t n_tiles = min(end - tile, 1024u);
        windowdev::prefetch(p.tcA2B + (uint64_t)tile * kCW, n_tiles * kCW * 4u);
        windowdev::prefetch(p.tiles + (uint64_t)tile * 512u, n_tiles * 512u);
    }
    // copies: eight lanes bring 128 bytes of a row, lane quad q those of the columns q * kOwn + j of a tile, to row 4 j + q
    const uint32_t q = lane >> 3, chunk = lane & 7u;
    const uint8_t *b_base = static_cast<const uint8_t *>(p.B) + line0 * 128u + chunk * 16u;
    uint32_t limit[kLines];  // columns of B that the lane has something of
#pragma unroll
    for (uint32_t l = 0; l < kLines; ++l) limit[l] = (line0 + l) * 128u + chunk * 16u < p.n * (kTf32 ? 4u : 2u) ? p.cols : 0u;
    const uint32_t my_ring = ptx::smem_u32(ring) + warp * (kWindowStages * kWindowStageBytes);
    const uint32_t put = my_ring + q * 128u + ((chunk ^ q) << 4);
    const uint32_t get = my_ring + t * 128u + ((((g >> 1) + (g & 1u) * 4u) ^ t) << 4);
    uint32_t col[kTiles][kOwn];
    auto fetch_columns = [&](uint32_t at) {
        const uint32_t *list = p.tcA2B + (uint64_t)at * kCW + q * kOwn;
#pragma unroll
        for (uint32_t k = 0; k < kTiles; ++k) {
            if (at + k >= end) break;
            if constexpr (kTf32) {
                const uint2 c = __ldg(reinterpret_cast<const uint2 *>(list + k * kCW));
                col[k][0] = c.x; col[k][1] = c.y;
            } else {
                const uint4 c = __ldg(reinterpret_cast<const uint4 *>(list + k * kCW));
                col[k][0] = c.x; col[k][1] = c.y; col[k][2] = c.z; col[k][3] = c.w;
            }
        }
    };
    uint32_t put_slot = 0, get_slot = 0;
    auto copy_stage = [&](uint32_t at) {
#pragma unroll
        for (uint32_t k = 0; k < kTiles; ++k) {
            if (at + k >= end) break;
#pragma unroll
            for (uint32_t j = 0; j < kOwn; ++j) {
                const uint8_t *row = b_base + (uint64_t)col[k][j] * p.pitch;
#pragma unroll
                for (uint32_t l = 0; l < kLines; ++l)
                    windowdev::copy_if(put + put_slot + ((k * kLines + l) * kOwn + j) * 512u, row + l * 128u, col[k][j] < limit[l]);
            }
        }
        ptx::cp_async_commit();
        put_slot = put_slot == (kWindowStages - 1) * kWindowStageBytes ? 0u : put_slot + kWindowStageBytes;
    };
    const uint8_t *a_base = p.tiles + g * 32u + ((t * 8u) ^ (p.swizzled ? (g & 4u) << 2 : 0u));
    uint2 a[2][kTiles][2];  // of this stage and of the next one
    auto fetch_tiles = [&](uint32_t at) {
        const uint8_t *from = a_base + (uint64_t)at * 512u;
#pragma unroll
        for (uint32_t k = 0; k < kTiles; ++k) {
            if (at + k >= end) break;
            a[1][k][0] = __ldg(reinterpret_cast<const uint2 *>(from + k * 512u));
            a[1][k][1] = __ldg(reinterpret_cast<const uint2 *>(from + k * 512u + 256u));
        }
    };
    float acc[kLines][kVec][4] = {};
    fetch_columns(tile);
    fetch_tiles(tile);
    ptx::wait_for_grids_before();
#pragma unroll
    for (uint32_t s = 0; s + 1 < kWindowStages; ++s) {
        copy_stage(tile + s * kTiles);
        fetch_columns(tile + (s + 1) * kTiles);
    }
    for (; tile < end; tile += kTiles) {
#pragma unroll
        for (uint32_t k = 0; k < kTiles; ++k)
#pragma unroll
            for (uint32_t i = 0; i < 2; ++i) a[0][k][i] = a[1][k][i];
        copy_stage(tile + (kWindowStages - 1) * kTiles);
        fetch_columns(tile + kWindowStages * kTiles);
        fetch_tiles(tile + kTiles);
        asm volatile("cp.async.wait_group %0;" ::"n"(kWindowStages - 1) : "memory");
        __syncwarp();
#pragma unroll
        for (uint32_t k = 0; k < kTiles; ++k) {
            if (tile + k >= end) break;
            const uint32_t av[4] = {a[0][k][0].x, a[0][k][1].x, a[0][k][0].y, a[0][k][1].y};
#pragma unroll
            for (uint32_t l = 0; l < kLines; ++l) {
                uint32_t b[kOwn][4];
#pragma unroll
                for (uint32_t j = 0; j < kOwn; ++j)
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];"
                                 : "=r"(b[j][0]), "=r"(b[j][1]), "=r"(b[j][2]), "=r"(b[j][3])
                                 : "r"(get + get_slot + ((k * kLines + l) * kOwn + j) * 512u)
                                 : "memory");
                if constexpr (kTf32) {
#pragma unroll
                    for (uint32_t j = 0; j < kVec; ++j) windowdev::mma<true>(acc[l][j], av, b[0][j], b[1][j]);
                } else {
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j) {
                        windowdev::mma<false>(acc[l][2 * j], av, __byte_perm(b[0][j], b[1][j], 0x5410), __byte_perm(b[2][j], b[3][j], 0x5410));
                        windowdev::mma<false>(acc[l][2 * j + 1], av, __byte_perm(b[0][j], b[1][j], 0x7632), __byte_perm(b[2][j], b[3][j], 0x7632));
                    }
                }
            }
        }
        get_slot = get_slot == (kWindowStages - 1) * kWindowStageBytes ? 0u : get_slot + kWindowStageBytes;
        __syncwarp();  // the slot is free for the next copies
    }
#pragma unroll
    for (uint32_t l = 0; l < kLines; ++l) {
        if (l >= lines) break;
        windowdev::store_line<kTf32>(p, acc[l], line0 + l, w, row0, g, t);
    }
}

}  // namespace b200spmm
