// SpMM row by row: the kernel for matrices whose condensed tiles are nearly empty.
//
// A tile of the condensed format costs the tile kernels its CW gathered rows of B whatever it holds.  On a
// power-law graph (17 entries per 256-slot tile: about one per gathered row) the matrix instruction has
// nothing to share, and what remains is the traffic of the gathered rows, which TMA's gather4 delivers at ~39
// bytes per clock and SM (11 TB/s).  16-byte loads by the lanes of a warp reach 17 TB/s as long as B lies in
// L2 (10 on a graph of 2^20 nodes, where it does not), and they need no tiles (512 bytes for 17 entries), so here every entry is one coalesced row load and one
// FMA per feature.
//
// A unit (a row, or a piece of a long one, see rows_gpu.hpp) is walked by the group of lanes that covers the
// features of a pass at 16 bytes per lane - 8 lanes for 64 fp16 features, 10 for 40 tf32 ones - so a warp walks
// 32 / lanes units side by side.  A group that is through with a unit goes on with the next of its share, every
// n-th unit of a list in order of length, longest first: the last blocks have the shortest units.
//
// A long row leaves pieces in fp32 slots that rows_fixup_kernel adds in order: C does not depend on timing,
// bands or feature halves.
#pragma once

#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "ptx_sm100.cuh"
#include "rows_gpu.hpp"

namespace b200spmm {

struct RowsParams {
    const uint32_t *batches;    // [n_batches + 1][kBatchWords]
    const uint2 *units;               // first batch and number of batches, or a row without entries
    uint32_t unit_begin, unit_end;    // units with entries: their first batches
    uint32_t empty_begin, empty_end;  // rows without entries
    uint32_t team_end, team_blocks;   // kTeams: units before team_end are walked by whole warps, of the first team_blocks blocks
    uint32_t n_batches;
    const void *B;              // [cols, n] row-major
    void *C;                    // [rows, n] row-major
    float *partial;             // [n_slots][n] pieces of cut rows
    int64_t ldb, ldc;           // elements
    uint32_t n, slab;           // features, features per pass (blockIdx.y)
    uint32_t c_is_half;
};

// Two warps a block and 16 blocks an SM: the SM favours its older warps, so equal shares end at very different
// times, and the shares are handed out by the hardware as small blocks instead, the longest units first (2^20-node R-MAT
// graph, 64 fp16 features, 220 us now: 15 to 35 % faster than one resident wave with fixed shares).  A share of 16
// batches still hides its start, three dependent loads; with 8 the start shows (7 %), with 32 nothing changes.
// The bound of 64 registers lets the compiler keep all four rows of a batch in flight; at 48 it does not (30 % slower).
constexpr int kRowsThreads = 64;
constexpr int kRowsBlocksPerSm = 16;
constexpr uint64_t kRowsGroupBatches = 16;
constexpr uint32_t kRowsWarpsPerSm = kRowsBlocksPerSm * kRowsThreads / 32;

namespace rowsdev {

// 16 bytes of a row of B times one value, added to the lane's fp32 accumulators.
template <bool kTf32>
__device__ __forceinline__ void accumulate(float (&acc)[kTf32 ? 4 : 8], const uint4 &b, uint32_t a) {
    const uint32_t w[4] = {b.x, b.y, b.z, b.w};
    if constexpr (kTf32) {  // the tensor core reads fp32 as tf32: low 13 mantissa bits dropped
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[k] = fmaf(__uint_as_float(a), __uint_as_float(w[k] & 0xFFFFE000u), acc[k]);
    } else {
        const uint16_t ah = (uint16_t)a;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            asm("fma.rn.f32.f16 %0, %1, %2, %0;" : "+f"(acc[2 * k]) : "h"(ah), "h"((uint16_t)w[k]));
            asm("fma.rn.f32.f16 %0, %1, %2, %0;" : "+f"(acc[2 * k + 1]) : "h"(ah), "h"((uint16_t)(w[k] >> 16)));
        }
    }
}

template <int kN>
__device__ __forceinline__ void store_f32(float *dst, const float (&acc)[kN]) {
#pragma unroll
    for (int k = 0; k < kN / 4; ++k)
        __stcs(reinterpret_cast<float4 *>(dst) + k, make_float4(acc[4 * k], acc[4 * k + 1], acc[4 * k + 2], acc[4 * k + 3]));
}

template <int kN>
__device__ __forceinline__ void store_f16(__half *dst, const float (&acc)[kN]) {
    uint32_t w[4] = {};
#pragma unroll
    for (int k = 0; k < kN / 2; ++k) {
        const __half2 h = __floats2half2_rn(acc[2 * k], acc[2 * k + 1]);
        w[k] = *reinterpret_cast<const uint32_t *>(&h);
    }
    if constexpr (kN == 4) __stcs(reinterpret_cast<uint2 *>(dst), make_uint2(w[0], w[1]));
    else __stcs(reinterpret_cast<uint4 *>(dst), make_uint4(w[0], w[1], w[2], w[3]));
}

}  // namespace rowsdev

// kTeams: in launches that leave the GPU half empty a unit is a chain of batches, each a round trip to L2, that too few
// others hide.  There all groups of a warp share a unit - group t takes every groups-th batch from t on - and are summed
// by shuffles (always in the same order).  It costs the loop registers and instructions, 8 % of a large launch, so it is a
// kernel of its own; launch_rows has the rule and what it gives.
template <bool kTf32, bool kTeams>
__global__ void __launch_bounds__(kRowsThreads, kRowsBlocksPerSm) spmm_rows_kernel(const RowsParams p) {
    constexpr uint32_t kVec = kTf32 ? 4 : 8;  // features per lane: 16 bytes
    constexpr uint32_t kEsz = kTf32 ? 4 : 2;
    constexpr uint32_t kQ = kBatchWords<kTf32> / 4;  // 16-byte words of a batch
    const uint32_t f0 = blockIdx.y * p.slab, width = min(p.slab, p.n - f0);
    const uint32_t lanes = width / kVec, groups = 32u / lanes;  // lanes per unit, units per warp
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t g = min(lane / lanes, groups - 1), pos = lane - g * lanes;
    const bool live = pos < lanes;  // (lanes left over when 32 is no multiple follow the last group and store nothing)
    const uint32_t feat = f0 + (live ? pos : 0u) * kVec;
    const uint8_t *Bf = static_cast<const uint8_t *>(p.B) + (size_t)feat * kEsz;
    const uint32_t pitch = (uint32_t)p.ldb * kEsz;
    const uint32_t everyone = gridDim.x * (kRowsThreads / 32) * groups;
    const uint32_t me = (blockIdx.x * (kRowsThreads / 32) + warp) * groups + g;
    const bool team = kTeams && blockIdx.x < p.team_blocks;
    const uint32_t step = team ? groups : 1u, t = team ? g : 0u;  // groups that share a unit, and which of them this one is
    uint32_t stride = everyone, first = p.unit_begin + me, end = p.unit_end;
    if (kTeams) {
        const uint32_t warps = kRowsThreads / 32, block = team ? blockIdx.x : blockIdx.x - p.team_blocks;
        stride = (team ? p.team_blocks : (gridDim.x - p.team_blocks) * groups) * warps;
        first = team ? p.unit_begin + block * warps + warp : p.team_end + (block * warps + warp) * groups + g;
        if (team) end = p.team_end;
    }

    float acc[kVec] = {};
    auto store_row = [&](uint32_t to) {
        if (!live || (kTeams && to == kNoTarget)) return;
        if (to & kSlotTarget) rowsdev::store_f32(p.partial + (size_t)(to & ~kSlotTarget) * p.n + feat, acc);
        else if (p.c_is_half) rowsdev::store_f16(static_cast<__half *>(p.C) + (int64_t)to * p.ldc + feat, acc);
        else rowsdev::store_f32(static_cast<float *>(p.C) + (int64_t)to * p.ldc + feat, acc);
    };
    uint32_t u = first;
    auto load_unit = [&](uint32_t k) { return k < end ? __ldg(p.units + k) : make_uint2(p.n_batches, kTeams ? 0u : 0xFFFFFFFFu); };
    const uint4 *batches = reinterpret_cast<const uint4 *>(p.batches);
    uint2 unit = load_unit(u), next = load_unit(u + stride);
    uint4 e[kQ];  // entries of the next batch
    auto fetch = [&]() {
        // (a group of a team has nothing to fetch where fewer batches than groups are left)
        const uint32_t at = !kTeams ? unit.x : t < unit.y ? unit.x + 4u * t : p.n_batches;
#pragma unroll
        for (uint32_t k = 0; k < kQ; ++k) e[k] = ptx::ld_global_nc_v4_ahead(batches + (uint64_t)at * kQ + k);
    };
    u += stride;
    fetch();
    ptx::wait_for_grids_before();
    for (uint32_t k = p.empty_begin + me; k < p.empty_end; k += everyone) store_row(__ldg(p.units + k).x);
    while (!__all_sync(0xffffffffu, kTeams ? unit.y == 0 : unit.x == p.n_batches)) {  // a group that is through stays at the spare batch
        uint4 b[kUnitBatch];
        const uint32_t col[4] = {e[0].x, e[0].y, e[0].z, e[0].w};
#pragma unroll
        for (uint32_t k = 0; k < kUnitBatch; ++k) b[k] = ptx::ld_global_v4(Bf + (uint64_t)col[k] * pitch);
        uint32_t val[4], to;
        if constexpr (kTf32) {
            val[0] = e[1].x; val[1] = e[1].y; val[2] = e[1].z; val[3] = e[1].w;
            to = e[2].x;
        } else {
            val[0] = e[1].x; val[1] = e[1].x >> 16; val[2] = e[1].y; val[3] = e[1].y >> 16;
            to = e[1].z;
        }
        // the batch behind this one, or the first one of the next unit
        const uint32_t left = unit.y;  // batches of the unit, this one and those of the other groups of a team among them
        bool last;
        if (kTeams) {
            last = left <= step;
            unit.x += 4u * step;
            unit.y -= step;
        } else {
            last = --unit.y == 0;
        }
        if (last) {
            unit = next;
            u += stride;
            next = load_unit(u);
        } else if (!kTeams && unit.x != p.n_batches) {
            unit.x += 4;
        }
        fetch();
        if (!kTeams || t < left) {
#pragma unroll
            for (uint32_t k = 0; k < kUnitBatch; ++k) rowsdev::accumulate<kTf32>(acc, b[k], val[k]);
        }
        if (last) {
            if (kTeams && left == 0) to = kNoTarget;  // (through)
            if (team) {
                to = __shfl_sync(0xffffffffu, to, (left - 1) * lanes);  // the group of the last batch knows the target
                if ((lanes & (lanes - 1)) == 0) {
                    for (uint32_t o = lanes; o < 32; o *= 2) {
#pragma unroll
                        for (uint32_t k = 0; k < kVec; ++k) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
                    }
                } else {
                    float sum[kVec] = {};
                    for (uint32_t j = 0; j < groups; ++j) {
#pragma unroll
                        for (uint32_t k = 0; k < kVec; ++k) sum[k] += __shfl_sync(0xffffffffu, acc[k], j * lanes + pos);
                    }
#pragma unroll
                    for (uint32_t k = 0; k < kVec; ++k) acc[k] = sum[k];
                }
                if (g != 0) to = kNoTarget;
            }
            store_row(to);
#pragma unroll
            for (uint32_t k = 0; k < kVec; ++k) acc[k] = 0.f;
        }
    }
}

// Adds the pieces of every cut row and writes the row of C.  One block per row: 8 runs of pieces (piece k
// belongs to run k mod 8, whatever the width) times 32 lanes of four features.
__global__ void __launch_bounds__(256)
rows_fixup_kernel(const RowSplit *__restrict__ splits, const float *partial, void *C, int64_t ldc,
                  uint32_t n, uint32_t c_is_half) {
    __shared__ float4 part[8][32];
    const RowSplit sp = splits[blockIdx.x];
    const uint32_t lane = threadIdx.x & 31u, run = threadIdx.x >> 5;
    ptx::wait_for_grids_before();
    for (uint32_t f0 = 0; f0 < n; f0 += 128) {
        const uint32_t feat = f0 + lane * 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (feat < n) {
#pragma unroll 4
            for (uint32_t s = sp.slot_begin + run; s < sp.slot_end; s += 8) {
                const float4 v = __ldcs(reinterpret_cast<const float4 *>(partial + (size_t)s * n + feat));
                acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
            }
        }
        __syncthreads();
        part[run][lane] = acc;
        __syncthreads();
        if (run == 0 && feat < n) {
#pragma unroll
            for (int k = 1; k < 8; ++k) {
                const float4 v = part[k][lane];
                acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
            }
            if (c_is_half) {
                const __half2 lo = __floats2half2_rn(acc.x, acc.y), hi = __floats2half2_rn(acc.z, acc.w);
                uint2 packed;
                packed.x = *reinterpret_cast<const uint32_t *>(&lo);
                packed.y = *reinterpret_cast<const uint32_t *>(&hi);
                *reinterpret_cast<uint2 *>(static_cast<__half *>(C) + (int64_t)sp.row * ldc + feat) = packed;
            } else {
                *reinterpret_cast<float4 *>(static_cast<float *>(C) + (int64_t)sp.row * ldc + feat) = acc;
            }
        }
    }
}

}  // namespace b200spmm
