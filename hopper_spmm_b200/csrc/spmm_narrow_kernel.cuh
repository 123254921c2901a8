// SpMM for narrow B (token-by-token decoding through a pruned weight): A is read once, B comes from shared memory.
//
// With eight columns of B the product is a stream over A - 94 MB of 4-byte entries for 23.5 M stored values, 14 us
// of HBM time - as long as the gathers from B cost less.  From L1 they do not: 32 lanes hit 32 different lines, one
// per clock (83 us).  Shared memory serves eight 16-byte reads a clock when they fall into different bank groups,
// so the entries of a row are stored in an order in which neighbours do (narrow_entries_kernel), and B is laid out
// in planes of 16 bytes per column.  Every CTA (one per SM, 32 warps) owns a run of rows, balanced by entries, and
// goes over the columns of B in groups that fit its shared memory, all rows for each group; sums of several groups
// wait in shared memory.  A warp takes a row: 32 entries a step, one per lane, and a butterfly at the row's end.
#pragma once

#include <cstdint>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include "ptx_sm100.cuh"
#include "rows_gpu.hpp"
#include "spmm_rows_kernel.cuh"

namespace b200spmm {

struct NarrowParams {
    const uint32_t *entries, *seg, *cut;  // NarrowFormat
    uint32_t n_blocks, group_blocks;      // column blocks in all, and in shared memory at one time
    const void *B;
    void *C;
    int64_t ldb, ldc;
    uint32_t cols, n;
    uint32_t c_is_half;
};

constexpr int kNarrowThreads = 1024;
// Steps whose entries are loaded at one time, and again one ahead.  With one word of B a step is short and eight of them hide
// the stream's latency (28672 x 8192 at 10 %, 8 columns 33.1 us, with four 35.2); with more, the idle steps at the end of a
// row cost more than that (16 columns 68.9 with eight, 63.5 with four; tf32 14000 x 8192, 8 columns 49.2 and 39.2).
template <int kVecs>
constexpr int kNarrowSteps = kVecs == 1 ? 8 : 4;
constexpr int kNarrowMaxVecs = 4;      // 16-byte words of a row of B
constexpr size_t kNarrowSmemMax = 232448;

// Columns of B and (with several groups) fp32 sums in shared memory.
inline size_t narrow_smem_bytes(uint32_t vecs, uint32_t cols, uint32_t group_blocks, uint32_t n_blocks, uint32_t max_rows, uint32_t n) {
    const size_t group_cols = group_blocks < n_blocks ? (size_t)group_blocks * kNarrowCols : (size_t)cols;
    return group_cols * vecs * 16 + (group_blocks < n_blocks ? (size_t)max_rows * n * 4 : 0);
}

template <bool kTf32, int kVecs>
__global__ void __launch_bounds__(kNarrowThreads, 1) spmm_narrow_kernel(const NarrowParams p) {
    constexpr int kPer = kTf32 ? 4 : 8;  // features of a 16-byte word
    constexpr int kW = kVecs * kPer <= 8 ? 8 : kVecs * kPer <= 16 ? 16 : kVecs * kPer <= 32 ? 32 : 64;
    constexpr uint32_t kEsz = kTf32 ? 4 : 2;
    constexpr int kSteps = kNarrowSteps<kVecs>;
    extern __shared__ __align__(16) uint8_t narrow_b[];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t row0 = p.cut[blockIdx.x], row1 = p.cut[blockIdx.x + 1], stride = p.n_blocks + 1;
    const uint32_t max_cols = p.group_blocks < p.n_blocks ? p.group_blocks * kNarrowCols : p.cols;
    const uint32_t b_addr = ptx::smem_u32(narrow_b), plane = max_cols * 16u;
    float *sums = reinterpret_cast<float *>(narrow_b + (size_t)plane * kVecs);
    const bool several = p.group_blocks < p.n_blocks;
    // feature that ends up in this lane, and its register, see the reduction
    const uint32_t feat = ((lane & 16u) ? kW / 2 : 0u) + ((lane & 8u) ? kW / 4 : 0u) + ((lane & 4u) ? kW / 8 : 0u) +
                          ((lane & 2u) && kW >= 16 ? kW / 16 : 0u) + ((lane & 1u) && kW >= 32 ? kW / 32 : 0u);
    const bool owner = kW >= 32 || (kW == 16 ? (lane & 1u) == 0 : (lane & 3u) == 0);

    for (uint32_t g0 = 0; g0 < p.n_blocks; g0 += p.group_blocks) {
        const uint32_t g1 = min(g0 + p.group_blocks, p.n_blocks), col0 = g0 * kNarrowCols, n_cols = min(p.cols - col0, max_cols);
        uint32_t row = row0 + warp;
        uint32_t e = 0, end = 0, next_e = 0, next_end = 0;
        auto segment = [&](uint32_t r, uint32_t &lo, uint32_t &hi) {
            if (r < row1) {
                lo = __ldg(p.seg + (uint64_t)r * stride + g0);
                hi = __ldg(p.seg + (uint64_t)r * stride + g1);
            }
        };
        uint2 w[kSteps];
        auto load = [&](uint2 (&to)[kSteps], uint32_t from, uint32_t limit) {
#pragma unroll
            for (int k = 0; k < kSteps; ++k) {
                const uint32_t i = from + k * 32 + lane;
                if (i < limit) {
                    if (kTf32) to[k] = __ldcs(reinterpret_cast<const uint2 *>(p.entries) + i);
                    else to[k].x = __ldcs(p.entries + i);
                }
            }
        };
        segment(row, e, end);
        segment(row + kNarrowThreads / 32, next_e, next_end);
        if (g0) __syncthreads();  // everybody is through with the group before
        else ptx::wait_for_grids_before();
        for (uint32_t i = threadIdx.x; i < n_cols * kVecs; i += kNarrowThreads) {
            const uint32_t c = i / kVecs, v = i % kVecs;
            ptx::cp_async_16(b_addr + v * plane + c * 16u,
                             static_cast<const uint8_t *>(p.B) + (uint64_t)(col0 + c) * ((uint64_t)p.ldb * kEsz) + v * 16u, 16u);
        }
        ptx::cp_async_commit();
        load(w, e, end);
        ptx::cp_async_wait_group<0>();
        __syncthreads();
        for (; row < row1; row += kNarrowThreads / 32) {
            float acc[kW] = {};
            uint32_t after_e = 0, after_end = 0;
            segment(row + 2 * (kNarrowThreads / 32), after_e, after_end);
            for (bool last = false; !last;) {
                last = e + kSteps * 32 >= end;
                uint2 ahead[kSteps];
                if (last) load(ahead, next_e, next_end);
                else load(ahead, e + kSteps * 32, end);
#pragma unroll
                for (int k = 0; k < kSteps; ++k) {
                    if (e + k * 32 + lane < end) {
                        const uint32_t c = kTf32 ? w[k].x - col0 : (w[k].x - col0) & 0xFFFFu, a = kTf32 ? w[k].y : w[k].x >> 16;
#pragma unroll
                        for (int v = 0; v < kVecs; ++v)
                            rowsdev::accumulate<kTf32>(*reinterpret_cast<float(*)[kPer]>(acc + v * kPer),
                                                       ptx::ld_shared_v4(b_addr + v * plane + c * 16u), a);
                    }
                }
                e += kSteps * 32;
#pragma unroll
                for (int k = 0; k < kSteps; ++k) w[k] = ahead[k];
            }
            // Sum over the lanes: every step halves the features a lane holds while there are several.
#pragma unroll
            for (int s = 0; s < 5; ++s) {
                const int off = 16 >> s, half = (kW >> s) / 2;
                if (half >= 1) {
                    const bool up = lane & off;
#pragma unroll
                    for (int i = 0; i < (half ? half : 1); ++i) {
                        const float give = up ? acc[i] : acc[i + half], keep = up ? acc[i + half] : acc[i];
                        acc[i] = keep + __shfl_xor_sync(0xffffffffu, give, off);
                    }
                } else {
                    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], off);
                }
            }
#pragma unroll
            for (int i = 0; i < (kW > 32 ? kW / 32 : 1); ++i) {
                const uint32_t f = feat + i;
                if (owner && f < p.n) {
                    if (several) {
                        float *s = sums + (size_t)(row - row0) * p.n + f;
                        *s = g0 ? *s + acc[i] : acc[i];
                        if (g1 == p.n_blocks) acc[i] = *s;
                    }
                    if (g1 == p.n_blocks) {
                        if (p.c_is_half) static_cast<__half *>(p.C)[(int64_t)row * p.ldc + f] = __float2half_rn(acc[i]);
                        else static_cast<float *>(p.C)[(int64_t)row * p.ldc + f] = acc[i];
                    }
                }
            }
            e = next_e;
            end = next_end;
            next_e = after_e;
            next_end = after_end;
        }
    }
}

}  // namespace b200spmm
