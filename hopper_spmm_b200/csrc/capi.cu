// C ABI of the library (include/b200_spmm.h): format handles, device plans, launches.
// Replaces the host side of the reference's operator, fp16_spmm (src/fp16.cu:221-281).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <new>
#include <string>
#include <vector>

#include "../../include/b200_spmm.h"
#include "common.hpp"
#include "compress_gpu.hpp"
#include "device_pool.hpp"
#include "format.hpp"
#include "handles.hpp"
#include "sparse24_gpu.hpp"
#include "spmm_kernel.cuh"
#include "spmm_narrow_kernel.cuh"
#include "spmm_pair_kernel.cuh"
#include "spmm_rows_kernel.cuh"
#include "spmm_tall_kernel.cuh"
#include "spmm_window_kernel.cuh"
#include "tall_gpu.hpp"
#include "tensormap.hpp"

namespace b200spmm {

namespace {
// The last error of the calling thread: either a composed text (CUDA failures: the failing call
// and the runtime's message) or a pointer to a fixed message, which needs no allocation.
thread_local std::string g_last_cuda_error;
thread_local const char *g_last_static_error = nullptr;
}

void record_cuda_error(cudaError_t e, const char *what) {
    try {
        g_last_cuda_error = std::string(what) + ": " + cudaGetErrorString(e);
        g_last_static_error = nullptr;
    } catch (const std::exception &) {  // no room for the text
        g_last_static_error = cudaGetErrorString(e);
    }
    cudaGetLastError();  // clear the sticky-free error so later calls start clean
}

void set_last_error_static(const char *message) { g_last_static_error = message; }

}  // namespace b200spmm

using namespace b200spmm;


struct b200spmm_plan {
    b200spmm_btcf_info_t info{};
    int device = 0;
    bool owns_format = false;
    uint32_t *d_rowOffset = nullptr, *d_tcA2B = nullptr, *d_rowIdx = nullptr;
    void *d_data = nullptr;
    // The schedule: the tile stream cut into chunks (tile cuts, first / last window and the
    // partial-result slots of each chunk), which the CTAs claim at run time, plus the split
    // windows and their slots for the fix-up kernel.
    struct Sched {
        int n_ctas = 0;
        uint32_t n_chunks = 0;
        uint32_t *d_tables = nullptr;  // holds all that follow
        uint32_t *d_tile = nullptr, *d_wfirst = nullptr, *d_wlast = nullptr, *d_head_slot = nullptr, *d_tail_slot = nullptr;
        SplitWindow *d_splits = nullptr;
        uint32_t *d_piece_slots = nullptr;
        uint32_t n_splits = 0, n_slots = 0;
        // Bands: the chunk table cut into a few runs of whole windows, so that a caller can launch
        // band after band and start copying a band's rows of C out while the next one is computed.
        // Band k covers chunks [band_chunk[k], band_chunk[k+1]), rows [band_row[k], band_row[k+1])
        // and the split windows [band_split[k], band_split[k+1]).
        std::vector<uint32_t> band_chunk, band_split;
        std::vector<uint64_t> band_row;
    } sched;
    cudaStream_t copy_stream = nullptr;       // host-buffer call: C goes out on this one
    cudaStream_t upload_stream = nullptr;     // ... and the second half of B's features comes in on this one
    cudaEvent_t half_up[2] = {nullptr, nullptr};
    bool host_split = true;                   // B200SPMM_HOST_SPLIT=0 (read when the plan is made) turns the halves off
    std::vector<cudaEvent_t> band_done;
    const Sched *launch_sched = nullptr;  // the one the next launch uses
    CompressedTiles comp;                 // the tiles as bitmap + stored values (empty: dense tiles only)
    // fp16 tiles as records of 32 (position, value) words (SpmmParams::tile_entries), or null: B200SPMM_TILES=entries
    uint32_t *d_tile_entries = nullptr;
    uint64_t entry_dense_tiles = 0;       // tiles with more than 32 entries, which stay dense
    // The same matrix in 128-row super-windows, built when merging eight windows shortens the tile
    // stream enough for the wide-MMA kernel (spmm_tall_kernel.cuh) to win; empty otherwise.
    TallFormat tall;
    bool tall_forced = false;  // B200SPMM_WINDOW=128 or 256: use it whatever the launch's size
    // ... and in 256-row super-windows for the CTA-pair kernel (spmm_pair_kernel.cuh), which takes the
    // launches wider than 128 features when doubling the window height again halves the tile count.
    TallFormat pair;
    Sparse24Format sparse;     // the same windows in the tensor core's 2:4 form (fp16), or empty
    int pair_clusters = 0;     // two-CTA clusters of that kernel the GPU runs at the same time
    // ... and as row units for the kernel that loads rows of B entry by entry (spmm_rows_kernel.cuh).  A matrix
    // whose tiles are nearly empty keeps nothing else (rows_only).
    RowsFormat rows_fmt;
    bool rows_only = false;
    NarrowFormat narrow;       // the entries once more for narrow B (spmm_narrow_kernel.cuh), or empty
    // A caller's column lists that are not as the converter makes them: only what takes any list may run, the 16-row
    // kernel without row boxes and the kernels that go by entries.
    bool loose_lists = false;
    bool has_tile_path = false;  // schedule and tile image of the 16-row kernel are there
    // Launches of kernels with bounded waits whose status word no sync has read yet: of one stream, or more than that can
    // be said about (a captured launch runs again without passing through the host).
    enum class Unread { none, one_stream, any } unread = Unread::none;
    unsigned long long unread_stream = 0;  // its id (a handle may come back as another stream)
    // Most tiles of the super-window format name one aligned group of CW consecutive rows of B: then B
    // is re-laid as shared-memory images at every launch (scratch of the plan, as large as B) and such a
    // tile's operand arrives by one bulk copy.
    bool tall_pack_b = false;
    // Scratch of launches, grown to the largest need seen (take_scratch).  A graph runs at the addresses its launches were
    // captured with: memory that one of them was given is not freed when it is outgrown, but with the plan.
    struct Scratch {
        void *ptr = nullptr;
        size_t bytes = 0;
        bool in_graph = false;
    };
    Scratch b_packed;
    Scratch partial;  // fp32: pieces of windows or rows that are computed in parts, parts of super-windows
    std::vector<void *> outgrown;
    // The kernel of single warps may take launches (windows_fit), or has to (windows_forced: B200SPMM_WINDOW=warps).
    uint32_t max_short_tiles = 0;  // of a 16-row window
    uint32_t max_gap = 0;          // windows without entries one after the other, the ends of the matrix among them
    bool windows_fit = false, windows_forced = false;
    int n_sms = 0;
    // The tiles as the kernel's shared-memory image (spmm_kernel.cuh, SpmmParams::tiles_image): the plan's own
    // array swizzled in place when it owns the format, a swizzled copy when the arrays are the caller's.
    void *d_tiles_image = nullptr;
    bool image_is_copy = false;
    uint32_t *d_status = nullptr;
    CUtensorMap tmap_a{};
    // Tensor map over B, kept between launches: B's address, pitch and width rarely change from call
    // to call, and encoding a map costs the host several microseconds of a 10-microsecond launch.
    CUtensorMap tmap_b{};   // box: 128 bytes of one row (the unit of tile::gather4)
    CUtensorMap tmap_bt{};  // box: 128 bytes of CW consecutive rows (tiles whose columns are neighbours)
    const void *tmap_b_ptr = nullptr;
    int64_t tmap_b_ldb = 0;
    uint32_t tmap_b_n = 0;
    bool row_boxes = false;       // keep tmap_bt (the allocation-free call encodes one map only)
    bool gather_cpasync = false;  // B200SPMM_GATHER=cpasync, read when the plan is made
    size_t scratch_limit = ~(size_t)0;  // b200spmm_kat_scratch_limit only: who needs more asks for more than there is
    unsigned long long wait_limit_ns = kDeviceWaitLimitNs;  // how long a wait inside the kernel may last
    bool starve_gathers = false;  // b200spmm_kat_spmm_starved only: B's tensor map delivers half the bytes
    // buffers of the host-pointer entry point, grown on demand
    void *d_B = nullptr, *d_C = nullptr;
    size_t d_B_bytes = 0, d_C_bytes = 0;
    b200spmm_launch_info_t last{};
};

namespace tileimage {
// dst row r (32 bytes) = src row r with its 16-byte halves swapped when (r / 4) is odd; dst may be src.
__global__ void swizzle_tiles_kernel(const uint4 *__restrict__ src, uint4 *__restrict__ dst, uint64_t n_rows) {
    for (uint64_t r = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n_rows; r += (uint64_t)gridDim.x * blockDim.x) {
        const uint4 lo = src[2 * r], hi = src[2 * r + 1];
        const bool flip = (r >> 2) & 1u;
        dst[2 * r] = flip ? hi : lo;
        dst[2 * r + 1] = flip ? lo : hi;
    }
}

// One warp per fp16 tile of the reference's layout (16 rows x 16 columns, row-major): the tile's record of 32
// words.  Lane l looks at row l / 2, columns 8 (l % 2) .. +7; a stored entry is any value whose bits are not
// zero; its word is (byte offset in the tile's shared-memory image << 16) | bits, where the image swaps the
// two 16-byte halves of a row when row / 4 is odd (the 32-byte swizzle).
__global__ void __launch_bounds__(256)
tile_entries_kernel(const uint16_t *__restrict__ data, uint64_t tiles, uint32_t *__restrict__ records,
                    unsigned long long *__restrict__ n_dense) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint64_t t = (uint64_t)blockIdx.x * 8u + (threadIdx.x >> 5); t < tiles; t += (uint64_t)gridDim.x * 8u) {
        const uint4 v = *reinterpret_cast<const uint4 *>(data + t * 256u + lane * 8u);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        uint32_t mask = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) mask |= (((w[k >> 1] >> ((k & 1) * 16)) & 0xFFFFu) != 0u) ? (1u << k) : 0u;
        const uint32_t mine = (uint32_t)__popc(mask);
        uint32_t before = mine;  // inclusive warp scan
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t up = __shfl_up_sync(0xffffffffu, before, d);
            if ((int)lane >= d) before += up;
        }
        const uint32_t total = __shfl_sync(0xffffffffu, before, 31);
        before -= mine;
        uint32_t *rec = records + (t << 5);
        if (total > 32u) {
            rec[lane] = b200spmm::kDenseTile;
            if (lane == 0) atomicAdd(n_dense, 1ull);
            continue;
        }
        rec[lane] = b200spmm::kNoEntry;
        __syncwarp();
        const uint32_t row = lane >> 1, half = lane & 1u;
        const uint32_t base = row * 32u + ((half ^ ((row >> 2) & 1u)) << 4);
        uint32_t k_out = before;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            if (mask & (1u << k)) {
                const uint32_t bits = (w[k >> 1] >> ((k & 1) * 16)) & 0xFFFFu;
                rec[k_out++] = ((base + (uint32_t)k * 2u) << 16) | bits;
            }
        }
    }
}

}  // namespace tileimage

// Looks over the tables of a caller's format.  Bad tables: window offsets that do not rise from 0 to the number of tiles,
// window rows that are past the end or closer than a window; nothing can run on them.  Loose lists: a window's columns are
// not ascending and distinct with less than a tile of padding behind them, one is past the end, or a window starts off the
// 16-row grid.  A column that does not rise is right where a window starts and nowhere else, so the lists are read once, four
// entries a thread, and the windows take their own falls off the count (searching the window of every fall: 8 us for
// 60,000 nodes and 700,000 entries, now 5).  Reads inside [eff + 1], [eff] and [tiles * cw] whatever the tables hold.
__global__ void __launch_bounds__(256)
tables_kernel(const uint32_t *__restrict__ rowOffset, const uint32_t *__restrict__ tcA2B, const uint32_t *__restrict__ rowIdx, uint32_t eff,
              uint32_t tiles, uint64_t rows, uint64_t cols, uint32_t cw, formatcheck::Found *__restrict__ found) {
    uint32_t flags = 0;
    int32_t falls = 0;
    const uint64_t first = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, step = (uint64_t)gridDim.x * blockDim.x;
    if (first == 0 && (rowOffset[0] != 0 || rowOffset[eff] != tiles)) flags |= formatcheck::kBadTables;
    auto fall = [](uint32_t before, uint32_t c) { return c != kIdxMax && before >= c; };
    for (uint64_t w = first; w < eff; w += step) {
        const uint32_t t = rowOffset[w], row = rowIdx[w];
        if (rowOffset[w + 1] <= t || row >= rows) flags |= formatcheck::kBadTables;
        if (row % kRowWindow) flags |= formatcheck::kLooseLists;
        if (!w) continue;
        const uint32_t row_before = rowIdx[w - 1];
        if (row < row_before || row - row_before < (uint32_t)kRowWindow) flags |= formatcheck::kBadTables;
        if (t && t < tiles && fall(tcA2B[(uint64_t)t * cw - 1], tcA2B[(uint64_t)t * cw])) --falls;
    }
    for (uint64_t q = first; q < (uint64_t)tiles * cw / 4; q += step) {
        const uint4 v = __ldg(reinterpret_cast<const uint4 *>(tcA2B) + q);
        const uint32_t c[4] = {v.x, v.y, v.z, v.w};
        uint32_t before = q ? __ldg(tcA2B + q * 4 - 1) : 0u;
        if (q * 4 % cw == 0 && c[0] == kIdxMax) flags |= formatcheck::kLooseLists;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (c[k] != kIdxMax && c[k] >= cols) flags |= formatcheck::kLooseLists;
            if ((q || k) && fall(before, c[k])) ++falls;
            before = c[k];
        }
    }
    falls = __reduce_add_sync(0xffffffffu, falls);
    flags = __reduce_or_sync(0xffffffffu, flags);
    if ((threadIdx.x & 31u) == 0) {
        if (falls) atomicAdd(&found->falls, falls);
        if (flags) atomicOr(&found->flags, flags);
    }
}

namespace {

// Launches a kernel of a product: it may start when the last block of the kernel before it in the stream has ended, and
// waits itself for that one's results (ptx::wait_for_grids_before).  What a launch costs on the GPU between two others - the
// results' way, the blocks' start, what they set up - overlaps: 4.1 -> 2.8 us a call for 1003 x 997 at 2 %, 32 columns,
// 8.2 -> 6.2 for 4096 x 4096 at 1 %, 128 columns.  The kernels do not let the next one in any earlier: its blocks would take
// the places that become free, unevenly (the same 4096 x 4096: 8.8 us).
template <typename... P, typename... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem, unsigned cluster, cudaStream_t stream, A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = cluster;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

template <bool kTf32, int kNs, bool kTma, int kTiles>
int launch_one(b200spmm_plan *p, const SpmmParams &prm, const CUtensorMap &tmap_b, cudaStream_t stream) {
    using Cfg = SpmmCfg<kTf32, kNs, kTma, kTiles>;
    auto kernel = spmm_sm100_kernel<kTf32, kNs, kTma, kTiles>;
    static thread_local int configured_device = -1;
    if (configured_device != p->device) {
        B200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmemBytes));
        // all of the SM's shared-memory/L1 array as shared memory: two CTAs of the narrow slabs fit only then
        B200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        configured_device = p->device;
    }
    B200_CUDA_TRY(launch_after(kernel, dim3(p->launch_sched->n_ctas), Cfg::kThreads, Cfg::kSmemBytes, 1, stream, p->tmap_a, tmap_b, p->tmap_bt, prm));
    p->last.n_ctas = p->launch_sched->n_ctas;
    p->last.threads = Cfg::kThreads;
    p->last.stages = Cfg::kStages;
    p->last.feature_slab = kNs;
    p->last.n_slabs = (int)prm.n_slabs;
    p->last.smem_bytes = (int64_t)Cfg::kSmemBytes;
    p->last.kernel_launches = 1;
    p->last.tma_gather = kTma ? 1 : 0;
    p->last.bitmap_tiles = kTiles;
    p->last.row_window = kRowWindow;
    return B200SPMM_OK;
}

// Feature slab a launch uses for B of width n, and how many CTAs of that kernel share an SM.
constexpr uint64_t kMaxChunksPerCta = 16;
constexpr uint32_t kRowBands = 8;  // bands of the host-buffer call (large matrices only)
// Up to 128 features per pass: a CTA of that width leaves room for a second one on the SM, and two
// MMA-issuing threads per SM outweigh streaming the tiles once more per extra pass (n = 2048:
// 4.27 ms in sixteen passes of 128 against 4.65 ms in eight of 256).
inline uint32_t slab_for(uint32_t n) { return std::min(128u, (n + 63u) / 64u * 64u); }
constexpr int kCtasPerSm = 2;  // every kernel variant in use is sized for two resident CTAs per SM

template <bool kTf32, bool kTma, int kTiles>
int launch_slab(b200spmm_plan *p, SpmmParams &prm, const CUtensorMap &tmap_b, cudaStream_t stream) {
    const uint32_t ns = slab_for(prm.n);
    prm.n_slabs = (prm.n + ns - 1) / ns;
    switch (ns) {
        case 64: return launch_one<kTf32, 64, kTma, kTiles>(p, prm, tmap_b, stream);
        default: return launch_one<kTf32, 128, kTma, kTiles>(p, prm, tmap_b, stream);
    }
}

// A buffer of the plan that launches on any stream may use: what is there is given back once nothing uses it.
template <typename T>
int grow_buffer(T **buf, size_t bytes) {
    if (*buf) B200_CUDA_TRY(cudaDeviceSynchronize());
    pool_free(*buf);
    *buf = nullptr;
    void *ptr = nullptr;
    B200_CUDA_TRY(pool_alloc_bytes(&ptr, bytes, nullptr));
    B200_CUDA_TRY(cudaStreamSynchronize(nullptr));  // from here on the memory is there for every stream
    *buf = static_cast<T *>(ptr);
    return B200SPMM_OK;
}

// (The default stream does not answer while another one is being captured; a launch there will say so.)
bool is_captured(cudaStream_t stream) {
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) == cudaSuccess) return capture != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    return true;
}

// Scratch for a launch on `stream`.  A captured launch has it like any other, so that a graph holds the kernels that the call
// would run; but a capture allows no wait for the device, and what is outgrown then may be in use.
int take_scratch(b200spmm_plan *p, b200spmm_plan::Scratch *s, size_t bytes, cudaStream_t stream) {
    if (bytes > s->bytes) {
        const bool captured = is_captured(stream);
        if (s->ptr && (captured || s->in_graph)) {
            p->outgrown.push_back(s->ptr);
            s->ptr = nullptr;
        }
        s->in_graph = false;
        s->bytes = 0;
        const size_t ask = bytes <= p->scratch_limit ? bytes : (size_t)1 << 60;
        if (captured) {
            B200_CUDA_TRY(pool_alloc_under_capture(&s->ptr, ask));
        } else {
            const int st = grow_buffer(&s->ptr, ask);
            if (st != B200SPMM_OK) return st;
        }
        s->bytes = bytes;
    }
    if (bytes && !s->in_graph) s->in_graph = is_captured(stream);
    return B200SPMM_OK;
}

// The environment is consulted when a plan is made (and once per process for the plan-less
// allocation-free call), never on a launch.
bool env_is(const char *name, const char *value) {
    const char *v = std::getenv(name);
    return v && std::strcmp(v, value) == 0;
}

// Tensor map over B seen as [cols][n] with its real row pitch; a box is 128 bytes of one row.
// Rows or features past the end read as zeros.  Re-encoded only when B's address, pitch or width
// differ from the previous launch of this plan.
int b_tensor_map(b200spmm_plan *p, const void *B, int64_t ldb, uint32_t n, uint32_t cols, bool tf32) {
    if (p->tmap_b_ptr == B && p->tmap_b_ldb == ldb && p->tmap_b_n == n) return B200SPMM_OK;
    const uint32_t esz = tf32 ? 4 : 2, box = (p->starve_gathers ? 64 : 128) / esz;
    p->tmap_b_ptr = nullptr;
    if (!encode_2d(&p->tmap_b, tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, B, n,
                   cols, (uint64_t)ldb * esz, box, 1,
                   tf32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B,
                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) {
        set_last_error_static("cuTensorMapEncodeTiled failed for B");
        return B200SPMM_ERR_CUDA;
    }
    if (p->row_boxes &&
        !encode_2d(&p->tmap_bt, tf32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16, B, n, cols,
                   (uint64_t)ldb * esz, box, std::min<uint32_t>((uint32_t)p->info.col_window, cols),
                   tf32 ? CU_TENSOR_MAP_SWIZZLE_128B_ATOM_32B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B)) {
        set_last_error_static("cuTensorMapEncodeTiled failed for B (row boxes)");
        return B200SPMM_ERR_CUDA;
    }
    p->tmap_b_ptr = B;
    p->tmap_b_ldb = ldb;
    p->tmap_b_n = n;
    return B200SPMM_OK;
}

// How the rows of B are gathered: TMA tile::gather4 unless the plan was made with B200SPMM_GATHER=cpasync.  The
// features a 128-byte box has beyond n arrive as zeros; a narrow row costs a whole box of shared memory, but the
// cp.async copies cost the producer warps far more (pruned 28672 x 8192 weight, 8 columns: 306 us).
template <bool kTf32>
int launch_dtype(b200spmm_plan *p, SpmmParams &prm, cudaStream_t stream) {
    if (p->gather_cpasync) return launch_slab<kTf32, false, 0>(p, prm, p->tmap_b, stream);
    {
        int st = b_tensor_map(p, prm.B, prm.ldb, prm.n, prm.cols, kTf32);
        if (st != B200SPMM_OK) return st;
    }
    const CUtensorMap &tmap_b = p->tmap_b;
    prm.row_boxes = p->row_boxes ? 1u : 0u;
    if (p->comp.tcBit) {  // stream the compressed tiles
        prm.tcBit = p->comp.tcBit;
        prm.nnzOffset = p->comp.nnzOffset;
        prm.values = p->comp.values;
        return launch_slab<kTf32, true, 1>(p, prm, tmap_b, stream);
    }
    if constexpr (!kTf32) {
        if (p->d_tile_entries && prm.tiles_image) {  // stream the entry lists; tiles with many entries come from the image
            prm.tile_entries = p->d_tile_entries;
            return launch_slab<false, true, 2>(p, prm, tmap_b, stream);
        }
    }
    return launch_slab<kTf32, true, 0>(p, prm, tmap_b, stream);
}

// Tensor map over `data` seen as rows of 32 bytes: one tile is 16 consecutive rows, one box is
// the eight consecutive tiles of a ring stage.
int encode_tile_map(b200spmm_plan *p) {
    const auto &info = p->info;
    if (!info.total_tiles) return B200SPMM_OK;
    const bool f16 = info.dtype == B200SPMM_F16;
    if (!encode_2d(&p->tmap_a, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, p->d_data,
                   f16 ? 16 : 8, info.total_tiles * kRowWindow, 32, f16 ? 16 : 8, kRowWindow * kTilesPerStage,
                   CU_TENSOR_MAP_SWIZZLE_32B)) {
        set_last_error_static("cuTensorMapEncodeTiled failed for the tile array");
        return B200SPMM_ERR_CUDA;
    }
    return B200SPMM_OK;
}

#ifdef B200SPMM_PROFILE
unsigned long long *g_prof = nullptr;
#endif

// ---- 128-row super-windows
template <bool kTf32, int kNs>
int launch_tall_one(b200spmm_plan *p, TallParams &prm, cudaStream_t stream) {
    using Cfg = TallCfg<kTf32, kNs>;
    auto kernel = spmm_tall_kernel<kTf32, kNs>;
    static thread_local int configured_device = -1;
    if (configured_device != p->device) {
        B200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmemBytes));
        configured_device = p->device;
    }
    prm.n_slabs = (prm.n + kNs - 1) / kNs;
    prm.n_items = prm.eff_row_windows * prm.n_slabs * prm.parts;
    const int n_ctas = (int)std::min<uint32_t>(prm.n_items, (uint32_t)p->n_sms);
    B200_CUDA_TRY(launch_after(kernel, dim3(n_ctas), Cfg::kThreads, Cfg::kSmemBytes, 1, stream, p->tmap_b, p->tmap_bt, prm));
    p->last.n_ctas = n_ctas;
    p->last.threads = Cfg::kThreads;
    p->last.stages = Cfg::kStages;
    p->last.feature_slab = kNs;
    p->last.n_slabs = (int)prm.n_slabs;
    p->last.smem_bytes = (int64_t)Cfg::kSmemBytes;
    p->last.kernel_launches = prm.b_packed ? 2 : 1;
    p->last.tma_gather = 1;
    p->last.bitmap_tiles = 0;
    p->last.row_window = kTallRows;
    return B200SPMM_OK;
}

template <bool kTf32, bool kSparse>
int launch_pair_one(b200spmm_plan *p, TallParams &prm, cudaStream_t stream) {
    using Cfg = PairCfg<kTf32, kSparse>;
    auto kernel = spmm_pair_kernel<kTf32, kSparse>;
    prm.n_slabs = (prm.n + Cfg::kNs - 1) / Cfg::kNs;
    prm.n_items = prm.eff_row_windows * prm.n_slabs * prm.parts;
    const int n_pairs = (int)std::min<uint32_t>(prm.n_items, (uint32_t)p->pair_clusters);
    B200_CUDA_TRY(launch_after(kernel, dim3(2 * n_pairs), Cfg::kThreads, Cfg::kSmemBytes, 2, stream, p->tmap_b, p->tmap_bt, prm));
    p->last.n_ctas = 2 * n_pairs;
    p->last.threads = Cfg::kThreads;
    p->last.stages = Cfg::kStages;
    p->last.feature_slab = Cfg::kNs;
    p->last.n_slabs = (int)prm.n_slabs;
    p->last.smem_bytes = (int64_t)Cfg::kSmemBytes;
    p->last.kernel_launches = prm.b_packed ? 2 : 1;
    p->last.tma_gather = 1;
    p->last.bitmap_tiles = 0;
    p->last.row_window = kPairRows;
    return B200SPMM_OK;
}

// How many two-CTA clusters of the pair kernel the device runs at once (0: it cannot run it).
template <bool kTf32, bool kSparse = false>
int pair_max_clusters(int *out) {
    using Cfg = PairCfg<kTf32, kSparse>;
    auto kernel = spmm_pair_kernel<kTf32, kSparse>;
    B200_CUDA_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Cfg::kSmemBytes));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(2 * 148);
    cfg.blockDim = dim3(Cfg::kThreads);
    cfg.dynamicSmemBytes = Cfg::kSmemBytes;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = 2;
    attr.val.clusterDim.y = 1;
    attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    int n = 0;
    B200_CUDA_TRY(cudaOccupancyMaxActiveClusters(&n, kernel, &cfg));
    *out = n;
    return B200SPMM_OK;
}

// ---- row units
// A tile costs the 16-row kernel its gathered rows and one matrix instruction per 128 features whatever it
// holds; a row unit costs a row load per entry.
constexpr double kRowsMaxFill = 0.08;  // share of a tile's slots in use
// Up to this fill the row units still win over 16-row tiles (128 fp16 features: graph of 10,000 nodes, degree 40, 15.0
// against 21.7 us; 3000 x 3000 at 7 %, 10 % fill, 25.2 against 25.1 us), but not where super-windows do: those take a
// matrix whose merged tiles are at least kTallMinFill full (pruned at 5 %) and that has enough of them for the SMs.  A
// graph of 20,000 nodes merges well too, and waits for its hub window: 148 us against 35.  Matrices of fewer tiles
// than two a CTA take the same few microseconds either way and stay with their tiles.
constexpr double kRowsMaxFillWide = 0.11, kTallMinFill = 0.03;
constexpr uint64_t kRowsWideMinTiles = 592, kRowsWideAnyTiles = 16384;  // (below the second, whatever super-windows would do)
// Super-windows are made from this many short tiles on: 1100 x 1100 at 20 % (4,638), fp16, 72 / 256 / 512 / 2,048 columns 16.4
// / 22.5 / 38.5 / 135 us with 16 rows, 10.9 / 15.7 / 16.7 / 35.7 with them; the plan takes 285 us instead of 276.  Those of
// 256 rows from the second number on: in parts the two heights take the same (1682 x 1536 at 11 %, 8,614 tiles, 816 columns
// 21.5 and 22.5 us), and the plan takes 50 us less with one of them.
constexpr uint64_t kTallMinShortTiles = 2048, kPairMinShortTiles = 16384;
constexpr uint64_t kSparse24MinTiles = 20000;  // of 256 rows
constexpr uint64_t kTallMaxCounted = 1 << 25, kTallMaxCountedCols = 393216;  // entries of lists; columns of one bit set

bool use_rows(const b200spmm_plan *p, int64_t ldb) {
    return p->rows_only && ldb * p->info.elt_size <= 0xFFFFFFFFll;  // (the kernel's row pitch is 32-bit)
}

// How many of the longest units of a launch are walked by whole warps (spmm_rows_kernel<., true>).  They pay where the
// longest unit would take longer than all the work does: a batch is a round trip to L2 of about 0.35 us, and an SM gets through
// a warp's four entries a group in 0.025, so where the longest unit has a sixteenth of an SM's steps.  Then the units of
// at least 2, 4, 8 ... batches, as many as are resident at one time and leave the launch with at most half as many warps
// again: where all are teams and start in two waves, the starts cost more than the chains (6578 x 2298 at 2.5 %, 80 columns
// 8.5 -> 9.4).  4096 x 4096 at 1 %, 32 / 128 columns 4.9 -> 4.0 / 6.0 -> 5.2 us; 600 x 8000 at 2 %,
// 128 columns (passes of 32) 12.8 -> 4.4; graphs of 2,000 nodes, 64 columns 7.3 -> 4.4 and of 10,000, 128 columns 9.5 -> 7.9;
// but 8000 x 3000 at 1 %, 128 columns 6.5 -> 8.0 and 6000 x 6000 at 1 %, tf32, 64 columns 8.9 -> 10.2.
// (Rows without entries are only stored, but by all warps; where they alone would fill the GPU, the launch has to.)
uint32_t team_units(const b200spmm_plan *p, uint32_t n_units, uint32_t n_empty, uint32_t groups, uint32_t n_slabs) {
    const RowsFormat &f = p->rows_fmt;
    const uint64_t resident = (uint64_t)p->n_sms * kRowsWarpsPerSm, steps = (uint64_t)f.n_batches * n_slabs / groups / p->n_sms;
    if (groups < 2 || 16ull * f.most_batches < steps || (uint64_t)n_empty / groups * n_slabs > resident) return 0;
    for (uint32_t longest : f.long_units)
        if (longest && (uint64_t)longest * n_slabs <= resident && 2 * ((uint64_t)longest + (n_units - longest) / groups) * n_slabs <= 3 * resident)
            return longest;
    return 0;
}

int launch_rows_grid(b200spmm_plan *p, const RowsParams &prm, dim3 grid, void (*kernel)(const RowsParams), uint32_t s0, uint32_t s1,
                     cudaStream_t stream) {
    B200_CUDA_TRY(launch_after(kernel, grid, kRowsThreads, 0, 1, stream, prm));
    p->last.n_ctas = (int)(grid.x * grid.y);
    p->last.threads = kRowsThreads;
    p->last.feature_slab = (int)slab_for(prm.n);  // (what a pass covers; teams share a pass out by features, too)
    p->last.n_slabs = (int)((prm.n + slab_for(prm.n) - 1) / slab_for(prm.n));
    p->last.row_window = kRowWindow;
    p->last.kernel_launches = 1;
    if (s1 == s0) return B200SPMM_OK;
    B200_CUDA_TRY(launch_after(rows_fixup_kernel, dim3(s1 - s0), 256, 0, 1, stream, p->rows_fmt.d_splits + s0, (const float *)prm.partial, prm.C,
                               prm.ldc, prm.n, prm.c_is_half));
    p->last.kernel_launches = 2;
    return B200SPMM_OK;
}

int launch_rows(b200spmm_plan *p, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                cudaStream_t stream, int band) {
    const RowsFormat &f = p->rows_fmt;
    if (band >= 0 && ((size_t)band + 1 >= f.bands.size() || (f.bands.size() > 2 && !f.d_band_units))) return B200SPMM_ERR_INVALID_ARG;
    const RowBand &from = f.bands[band < 0 ? 0 : band], &to = band < 0 ? f.bands.back() : f.bands[band + 1];
    RowsParams prm{};
    prm.batches = f.d_batches;
    prm.units = band >= 0 && f.bands.size() > 2 ? f.d_band_units : f.d_units;
    prm.unit_begin = from.unit;
    prm.unit_end = to.unit;
    prm.empty_begin = from.empty;
    prm.empty_end = to.empty;
    prm.n_batches = f.n_batches;
    prm.B = d_B;
    prm.C = d_C;
    prm.ldb = ldb;
    prm.ldc = ldc;
    prm.n = (uint32_t)n;
    prm.c_is_half = c_dtype == B200SPMM_C_F16;
    if (f.n_slots) {
        int st = take_scratch(p, &p->partial, (size_t)f.n_slots * (size_t)n * 4, stream);
        if (st != B200SPMM_OK) return st;
    }
    prm.partial = static_cast<float *>(p->partial.ptr);
    const uint32_t vec = 16u / (uint32_t)p->info.elt_size;
    uint32_t n_slabs = 0, groups = 0;
    auto set_slab = [&](uint32_t slab) {
        prm.slab = slab;
        n_slabs = (prm.n + slab - 1) / slab;
        groups = 32u / (std::min(slab, prm.n) / vec);
    };
    const uint32_t whole = slab_for(prm.n), all_units = to.unit - from.unit, n_empty = prm.empty_end - prm.empty_begin;
    uint32_t n_team = 0;
    if (band < 0 && f.bands.size() == 2) {
        set_slab(whole);
        if (groups < 2) set_slab(whole / 2);  // (128 tf32 features take all lanes)
        n_team = team_units(p, all_units, n_empty, groups, n_slabs);
    }
    if (n_team) {
        // a pass shared out by features gives more groups a warp, down to 64 bytes of a row, while all warps are resident
        while (n_team == all_units && prm.slab > 4 * vec && (uint64_t)all_units * n_slabs * 2 <= (uint64_t)p->n_sms * kRowsWarpsPerSm)
            set_slab(prm.slab / 2);
        const uint32_t warps = kRowsThreads / 32, rest = all_units - n_team;
        prm.team_end = prm.unit_begin + n_team;
        prm.team_blocks = (n_team + warps - 1) / warps;
        const dim3 grid(prm.team_blocks + (rest + groups * warps - 1) / (groups * warps), n_slabs);
        return launch_rows_grid(p, prm, grid, p->info.dtype == B200SPMM_TF32 ? spmm_rows_kernel<true, true> : spmm_rows_kernel<false, true>,
                                from.split, to.split, stream);
    }
    set_slab(whole);
    // a group of lanes for every kRowsGroupBatches batches, but enough of them for one wave where there are units for it
    const uint32_t n_units = std::max(all_units, n_empty), per_block = groups * (kRowsThreads / 32);
    const uint64_t share = (uint64_t)f.n_batches * n_units / f.n_units / kRowsGroupBatches / per_block;
    const dim3 grid(std::min((n_units + per_block - 1) / per_block, std::max((uint32_t)share, (uint32_t)(p->n_sms * kRowsBlocksPerSm))), n_slabs);
    if (!n_units) return B200SPMM_OK;
    return launch_rows_grid(p, prm, grid, p->info.dtype == B200SPMM_TF32 ? spmm_rows_kernel<true, false> : spmm_rows_kernel<false, false>,
                            from.split, to.split, stream);
}

// ---- windows of single warps
int launch_windows(b200spmm_plan *p, uint32_t lines, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                   cudaStream_t stream) {
    const bool tf32 = p->info.dtype == B200SPMM_TF32;
    WindowParams prm{};
    prm.rowOffset = p->d_rowOffset;
    prm.tcA2B = p->d_tcA2B;
    prm.rowIdx = p->d_rowIdx;
    prm.swizzled = p->d_tiles_image != nullptr;
    prm.tiles = static_cast<const uint8_t *>(p->d_tiles_image ? p->d_tiles_image : p->d_data);
    prm.B = d_B;
    prm.C = d_C;
    prm.ldc = ldc;
    prm.pitch = (uint32_t)(ldb * p->info.elt_size);
    prm.rows = (uint32_t)p->info.rows;
    prm.cols = (uint32_t)p->info.cols;
    prm.n = (uint32_t)n;
    prm.eff = (uint32_t)p->info.eff_row_windows;
    const uint32_t line = 128u / (uint32_t)p->info.elt_size;
    prm.lines = (prm.n + line - 1) / line;
    prm.c_is_half = c_dtype == B200SPMM_C_F16;
    using Kernel = void (*)(const WindowParams);
    static constexpr Kernel kernels[2][kWindowMaxLines] = {{spmm_window_kernel<false, 1>, spmm_window_kernel<false, 2>},
                                                           {spmm_window_kernel<true, 1>, spmm_window_kernel<true, 2>}};
    constexpr uint32_t threads = kWindowWarps * 32, smem = kWindowWarps * kWindowStages * kWindowStageBytes;
    static_assert(smem <= 48 * 1024, "needs no attribute");
    const uint32_t groups = (prm.lines + lines - 1) / lines;
    const uint64_t blocks = ((uint64_t)prm.eff * groups + kWindowWarps - 1) / kWindowWarps;
    B200_CUDA_TRY(launch_after(kernels[tf32][lines - 1], dim3((unsigned)blocks), threads, smem, 1, stream, prm));
    p->last.n_ctas = (int)blocks;
    p->last.threads = (int)threads;
    p->last.stages = (int)kWindowStages;
    p->last.feature_slab = (int)(line * lines);
    p->last.n_slabs = (int)groups;
    p->last.smem_bytes = (int64_t)smem;
    p->last.kernel_launches = 1;
    p->last.row_window = kRowWindow;
    return B200SPMM_OK;
}

// ---- narrow B
template <bool kTf32>
int launch_narrow_vecs(const NarrowParams &prm, int vecs, unsigned n_ctas, size_t smem, cudaStream_t stream) {
    using Kernel = void (*)(const NarrowParams);
    constexpr Kernel kernels[kNarrowMaxVecs] = {spmm_narrow_kernel<kTf32, 1>, spmm_narrow_kernel<kTf32, 2>, spmm_narrow_kernel<kTf32, 3>,
                                                spmm_narrow_kernel<kTf32, 4>};
    static thread_local int configured_device = -1;
    int device = 0;
    B200_CUDA_TRY(cudaGetDevice(&device));
    if (configured_device != device) {
        for (Kernel k : kernels) B200_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNarrowSmemMax));
        configured_device = device;
    }
    B200_CUDA_TRY(launch_after(kernels[vecs - 1], dim3(n_ctas), kNarrowThreads, smem, 1, stream, prm));
    return B200SPMM_OK;
}

// How long a launch takes, in microseconds, to choose between the tile kernels.  A super-window launch lasts as many
// rounds of its CTAs or pairs as its items need, each as long as the longest window, so a matrix with one heavy window
// stays with 16 rows; the 16-row kernel spreads its tiles evenly over all CTAs.  It pays long before every SM has an
// item: pruned 14336 x 4096, 10 %, fp16, 64 / 128 / 192 columns 33 / 36 / 43 us (56 windows of 256 rows for 74 pairs)
// against 62 / 79 / 146 with 16 rows; 3000 x 3000, 12 %, 192 columns 33 against 45, but at 64 columns 25 against 23.
// A tf32 tile takes what an fp16 one does, eight rows of B of twice the bytes.  Pruned, uniform and block matrices and
// graphs of at least 16,384 tiles, 32 to 1,024 columns, against the best of the three kernels when forced: the
// choice is 0.3 % slower on average in tf32 (84 products, at most 7 %), and in fp16 as fast on average (77 products, at
// most 15 % slower: 3000 x 3000 with 128 columns, 29 us against 25).
//
// With fewer items than CTAs or pairs the windows are cut into parts, as many as fit in one round: a tile takes the time it
// takes a CTA by itself then, and the sums go through L2 twice, where a launch of their own adds them up.  Parts in us,
// whole / 2 / 4 / 8 (16-row kernel): 1777 x 7404 at 15 %, fp16, 104 columns 38.6 / 26.2 / 19.1 / 15.9 (43); 1668 x 5737 at
// 28 %, tf32, 392 columns 67 / 46 / 35 / - (114); 1682 x 1536 at 11 %, fp16, 816 columns 28 / 21.5 / - / - (78); more than one
// round of parts is slower again (2000 x 8000 at 10 %, 1,024 columns 56 / 45 / 55 / 81).
// Up to 64 columns a matrix of fewer than kOneLaunchTiles tiles whose 16-row schedule cuts no window keeps to whole windows or to
// that kernel, which then is one launch and not two: 1024 x 1024 / 2048 x 1024 / 4096 x 1024 at 25 %, fp16, 64 columns 8.9 / 9.2 /
// 9.3 us, in parts 11.0 / 10.7 / 11.7.  Parts are as fast above (4736 x 1090, 20,424 tiles, 12.1 both, and 4736 x 1500 13.4 -> 12.1),
// and where windows are cut from the smallest matrices on (1040 x 1040 at 30 %, tf32, 40 columns 11.3 and 11.5; 1024 x 1700, 64
// columns 12.4 and 12.4; 3000 x 3000 at 12 %, fp16 19.1 -> 13.2, tf32 24.7 -> 16.3; 2001 x 6167 at 28 %, 40 columns 33.2 -> 13.6).
//
// The tensor core cuts what it adds, so the error of a sum grows with the tiles it runs through: 1.4e-8 a tile here, and with 16
// rows 1.6e-8 and more in fp16, 1.1e-8 in tf32, over the tiles of a piece of a window.  Where whole super-windows are not
// expected to be faster than 16 rows, or the matrix is small, the windows are cut so far that the sums are no less exact than
// those of the 16-row kernel's pieces (tall_least_parts), in more than one round if it takes that; or that kernel stays.
struct TallLaunch {
    double micros;
    uint32_t parts;
};
constexpr uint64_t kOneLaunchTiles = 20000;
constexpr double kTallMaxSums = 128e6;  // bytes of scratch that a plan may keep for them
double short_micros(const b200spmm_plan *p, int64_t n) {  // (tiles over 148 SMs)
    return 14.0 + (double)p->info.total_tiles * (148.0 / p->n_sms) * (n <= 64 ? 0.28e-3 : 0.4e-3 * (double)((n + 127) / 128));
}


bool tall_is_pair(const TallFormat &f) { return f.rows == (uint32_t)kPairRows; }
int64_t tall_items(const TallFormat &f, int64_t n) {
    const int64_t slab = tall_is_pair(f) || n > 128 ? 256 : 128;
    return (int64_t)f.eff * ((n + slab - 1) / slab);
}
double tall_whole_micros(const b200spmm_plan *p, const TallFormat &f, int64_t n) {
    const int64_t units = tall_is_pair(f) ? p->pair_clusters : p->n_sms;
    return 12.0 + (double)((tall_items(f, n) + units - 1) / units) * (double)f.max_window_tiles * (n > 128 ? 0.11 : 0.085);
}

uint32_t tall_least_parts(const b200spmm_plan *p, int64_t n) {
    const bool pair = p->pair.tiles && p->pair_clusters > 0 && n > 128;
    if (p->info.total_tiles >= kPairMinShortTiles && p->tall.eff * 16 >= (uint64_t)p->n_sms &&
        ((pair && tall_whole_micros(p, p->pair, n) < short_micros(p, n)) || tall_whole_micros(p, p->tall, n) < short_micros(p, n)))
        return 1;
    const double pieces = (double)std::max<uint64_t>(p->info.eff_row_windows, (uint64_t)p->n_sms * kCtasPerSm);
    const double tiles = (double)p->info.total_tiles / pieces * (p->info.dtype == B200SPMM_TF32 ? 0.65 : 1.0);
    return (uint32_t)std::ceil((double)p->tall.max_window_tiles / std::max(tiles, 1.0));
}

TallLaunch tall_launch(const b200spmm_plan *p, const TallFormat &f, int64_t n, uint32_t least) {
    const double whole = tall_whole_micros(p, f, n);
    if (p->tall_forced) return {whole, 1};
    TallLaunch best{least > 1 ? 1e30 : whole, 1};
    if (n <= 64 && p->sched.n_splits == 0 && p->info.total_tiles < kOneLaunchTiles) return best;
    const bool pair = tall_is_pair(f);
    const int64_t units = pair ? p->pair_clusters : p->n_sms, items = tall_items(f, n);
    const double longest = (double)f.max_window_tiles, alone = pair ? 0.088 : n > 128 ? 0.105 : 0.068;
    double lowest = least > 1 ? 1e30 : 12.0 + longest * alone;
    const uint64_t stages = (f.min_window_tiles + kTallStageTiles - 1) / kTallStageTiles;
    for (uint32_t parts = std::max(2u, least); parts <= 16 && parts <= stages; ++parts) {
        const int64_t rounds = (items * parts + units - 1) / units;
        const double sums = (double)parts * (double)f.eff * f.rows * (double)n * 4.0;
        if ((rounds > 1 && parts > least) || sums > kTallMaxSums) break;
        const double micros = 12.0 + (double)rounds * longest / parts * (rounds > 1 ? (n > 128 ? 0.11 : 0.085) : alone) + 1.5 + 2.0 * sums * 0.22e-6;
        if (micros < lowest) {
            lowest = micros;
            best = {micros, parts};
        }
    }
    return best;
}

// Whether a launch goes to the super-window kernels, how, and what it needs of the plan's scratch.  Worked out once a launch.
// Only with the TMA gathers, and - unless forced, for B at least one 128-byte box wide - only when it is expected to be faster.
struct TallChoice {
    bool use, pair, sparse;  // sparse: the pair kernel on 2:4 tiles
    uint32_t parts, least_parts;  // with fewer than the second the sums would be less exact than those of 16 rows
    size_t partial_bytes, packed_bytes;
};
TallChoice choose_tall(const b200spmm_plan *p, int64_t n) {
    TallChoice c{};
    if (!p->tall.tiles || p->gather_cpasync) return c;
    const bool can_pair = p->pair.tiles && p->pair_clusters > 0 && n > 128;
    if (p->tall_forced) {
        c.use = n * p->info.elt_size >= 128;
        c.pair = can_pair;
        c.parts = c.least_parts = 1;
    } else {
        const uint32_t least = c.least_parts = tall_least_parts(p, n);
        const double short_time = short_micros(p, n);
        TallLaunch l{};
        if (can_pair) l = tall_launch(p, p->pair, n, least);
        c.use = c.pair = can_pair && l.micros < short_time;
        if (!c.pair) {
            // (the 16-row kernel is better than its estimate where every SM has a window: 3000 x 1100 at 10 %, 128 columns 12.4 us against 13.3)
            const double margin = p->info.total_tiles < kPairMinShortTiles && p->info.eff_row_windows >= (uint64_t)p->n_sms ? 1.1 : 1.0;
            l = tall_launch(p, p->tall, n, least);
            c.use = l.micros * margin < short_time;
        }
        c.parts = l.parts;
    }
    const TallFormat &f = c.pair ? p->pair : p->tall;
    // (2:4 windows in parts: 4096^2 at 10 %, 256 columns 24.8 us with dense tiles, 30.4 so)
    c.sparse = c.pair && p->sparse.tiles && c.parts == 1;
    if (c.parts > 1) c.partial_bytes = (size_t)c.parts * (size_t)f.eff * f.rows * (size_t)n * 4;  // kTallMaxSums
    if (p->tall_pack_b) {
        // the pair kernel's CTAs fetch 128-feature halves of a 256-feature slab: both halves of the last slab must
        // exist in the packed copy (as zeros past n), so an even number of 128-feature blocks
        const size_t features = c.pair || n > 128 ? (size_t)(n + 255) / 256 * 256 : 128;
        const size_t group = c.sparse ? 32 : (size_t)p->info.col_window;  // rows of B
        c.packed_bytes = features * (size_t)p->info.elt_size * group * (((size_t)p->info.cols + group - 1) / group);
    }
    return c;
}

// Lines of 128 bytes that a warp of the kernel of single warps (spmm_window_kernel.cuh) multiplies, or 0 where the pipelined
// 16-row kernel is expected to be faster, or would cut windows into pieces: here they are whole, and their sums have its bits.
//
// The estimates are least-squares fits to forced launches of block, uniform and pruned matrices of the ranges that the
// benchmark draws, 8 to 2,000 columns (1,143 here, 15 % rms; 62 of the pipelined kernel on blocks, 7 %).  Here: a start, a step
// for every stage of a long window, the copies of all tiles, and the warps to start.  There: a start, and per pass of 128
// features a start of its own, the tiles and what it costs to hand a window over.  Us, pipelined / here, operands in L2:
// blocks, tf32, 16384^2 at 0.5 %, 256 columns 16.2 / 13.0 (matrices in turn, from DRAM: 16.8 / 15.7); 13040 x 2960 at 0.9 %, 504
// columns 15.5 / 11.2, 128 columns 7.3 / 4.9; 1648 x 5712 at 0.8 %, 512 columns 10.2 / 4.7; 1088 x 14304 at 0.3 %, 96 columns
// 6.3 / 3.7; fp16, 16384^2 at 0.5 %, 64 columns 8.4 / 5.0, 256 columns 13.3 / 8.2.  Long windows stay: 1024^2 pruned to 10 %,
// fp16, 64 columns 9.4 / 24.
//
// Rows of missing windows are cleared by whoever has the window in front of them, and from five windows on the longest gap ends
// last: 0.17 us a window and line of a warp (0.15 where a line of B is 256 bytes of C), 0.145 a window and pass of the pipelined
// kernel's CTA (0.18 up to 96 columns, where half its lanes store).  16384 x 8192 of blocks at 0.5 %, 32 / 256 / 1,024 empty windows
// behind: tf32, 128 columns, two lines 15 / 91 / 352, pipelined 12 / 45 / 156; 256 columns, two lines 18 / 95 / 356, one line 16 / 54
// / 185, pipelined 20 / 86 / 311; fp16, 128 columns, one line 8.7 / 42 / 158, pipelined 12 / 44 / 156.
struct WindowCost {
    double start, step, tile, warp;  // us; of a stage, of 1,000 tiles x groups of lines, of 1,000 warps
};
struct PipelinedCost {
    double start, pass, tile, window;  // us; of 1,000 tiles and of 1,000 windows in a pass
};
constexpr WindowCost kWindowCost[2][kWindowMaxLines] = {{{2.4, 0.34, 0.174, 1.08}, {2.7, 0.33, 0.258, 1.61}}, {{1.8, 0.49, 0.085, 0.83}, {2.2, 0.345, 0.137, 1.02}}};
constexpr PipelinedCost kPipelinedCost[2] = {{4.3, 1.71, 0.40, 0.17}, {4.9, 1.08, 0.36, 0.62}};
constexpr double kWindowGap[2] = {0.15, 0.17}, kPipelinedGap = 0.145, kPipelinedGapNarrow = 0.18;  // us
constexpr uint32_t kHiddenGap = 5;
uint32_t choose_window_lines(const b200spmm_plan *p, int64_t ldb, int64_t n) {
    const bool tf32 = p->info.dtype == B200SPMM_TF32;
    const uint64_t eff = p->info.eff_row_windows;
    const uint32_t line = 128u / (uint32_t)p->info.elt_size, n_lines = (uint32_t)((n + line - 1) / line);
    if (!p->windows_fit || (uint64_t)ldb * p->info.elt_size > 0xFFFFFFFFull || eff * n_lines > 0x7FFFFFFFull) return 0;  // 32-bit row pitch, grid
    const double tiles = (double)p->info.total_tiles, scale = 1e-3 * (148.0 / p->n_sms);
    const double gap = p->max_gap > kHiddenGap ? (double)(p->max_gap - kHiddenGap) : 0.0;
    double least = 1e30;
    if (!p->windows_forced) {
        const PipelinedCost &c = kPipelinedCost[tf32];
        const double passes = (double)((n + 127) / 128);
        least = c.start + passes * (c.pass + (c.tile * tiles + c.window * (double)eff) * scale) +
                gap * (n <= 96 ? kPipelinedGapNarrow : passes * kPipelinedGap);
    }
    const uint32_t longest = (uint32_t)((tiles / (double)eff + p->max_short_tiles) / 2);  // (of ten tiles on average: two standard deviations above)
    uint32_t best = 0;
    for (uint32_t lines = 1; lines <= kWindowMaxLines && lines <= n_lines; ++lines) {
        const WindowCost &c = kWindowCost[tf32][lines - 1];
        const uint32_t stage = kWindowStageBytes / (128u * (uint32_t)p->info.col_window * lines), steps = (longest + stage - 1) / stage;
        const double micros = c.start + c.step * steps + (c.tile * tiles + c.warp * (double)eff) * scale * (double)((n_lines + lines - 1) / lines) +
                              kWindowGap[tf32] * lines * gap;
        if (micros < least) {
            least = micros;
            best = lines;
        }
    }
    return best;
}

// Column blocks per group for B of width n: as many as fit shared memory, 0 if the kernel does not take it.  Every
// 16-byte word of a row of B adds to its time - pruned 28672 x 8192 weight, fp16: 33, 64, 84, 123 us for 8, 16, 24, 32
// columns; a warp has a row, so 33 rows a CTA take as long as 64 - while the tile kernels take the same up to 64 features (89
// us; tf32: 98 us for 8 and 16 columns).  Up to 24 fp16 and 16 tf32 columns it is taken all the same, also where super-windows
// would be faster (6000 x 8192 at 20 %, 24 columns 49.6 us against 23.4): its fp32 sums are thirty times as exact as the
// tensor core's.  32 fp16 columns go to it where all of B fits shared memory and it is expected to be faster than the tiles (1100 x
// 1100 at 20 % 11.6 -> 7.5 us, 1682 x 1536 at 11 % 13.5 -> 10.0, 3000 x 3000 at 12 % 19.2 -> 17.0; 2000 x 8000 at 6 %, in two
// halves, 36 against 20).  Below kNarrowPartsTiles tiles than 16 rows or whole windows: windows in parts would be faster (4885 x
// 1335 at 25 % 15.4 and 12.4 us, 3513 x 3235 at 26 % 23.4 and 12.6), and here too its sums are what it is kept for; above, it
// would take twice the time of the parts (8221 x 3229 at 25 % 33.4 and 17.0; 16972 x 2328 at 28 % 43.1 and 18.2).
constexpr uint64_t kNarrowPartsTiles = 80000;
uint32_t narrow_group_blocks(const b200spmm_plan *p, int64_t n) {
    const NarrowFormat &f = p->narrow;
    const int64_t vecs = n * p->info.elt_size / 16;
    const bool tf32 = p->info.dtype == B200SPMM_TF32;
    if (!f.n_ctas || vecs > kNarrowMaxVecs) return 0;
    uint32_t g = f.n_blocks;
    while (g && narrow_smem_bytes((uint32_t)vecs, (uint32_t)p->info.cols, g, f.n_blocks, f.max_rows, (uint32_t)n) > kNarrowSmemMax) --g;
    if (!g || vecs < kNarrowMaxVecs || tf32) return g;
    if (p->rows_only || g < f.n_blocks) return 0;
    const double rows = (double)p->info.rows / f.n_ctas, rounds = std::ceil(rows / 32.0) * 32.0 / rows;
    const double micros = 4.0 + (double)p->info.nnzs * (double)vecs * 1.05e-6 * (148.0 / p->n_sms) * rounds;
    double tall = 1e30;
    if (p->tall.tiles && !p->gather_cpasync) {
        const uint32_t least = p->tall_forced ? 1 : tall_least_parts(p, n);
        if (p->info.total_tiles >= kNarrowPartsTiles) tall = tall_launch(p, p->tall, n, least).micros;
        else if (least <= 1) tall = tall_whole_micros(p, p->tall, n);
    }
    return micros < tall && micros < short_micros(p, n) ? g : 0;
}

int launch_narrow(b200spmm_plan *p, uint32_t group_blocks, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                  cudaStream_t stream) {
    const NarrowFormat &f = p->narrow;
    NarrowParams prm{};
    prm.entries = f.d_entries;
    prm.seg = f.d_seg;
    prm.cut = f.d_cut;
    prm.n_blocks = f.n_blocks;
    prm.group_blocks = group_blocks;
    prm.B = d_B;
    prm.C = d_C;
    prm.ldb = ldb;
    prm.ldc = ldc;
    prm.cols = (uint32_t)p->info.cols;
    prm.n = (uint32_t)n;
    prm.c_is_half = c_dtype == B200SPMM_C_F16;
    const int vecs = (int)(n * p->info.elt_size / 16);
    const size_t smem = narrow_smem_bytes((uint32_t)vecs, prm.cols, group_blocks, f.n_blocks, f.max_rows, prm.n);
    const int st = p->info.dtype == B200SPMM_TF32 ? launch_narrow_vecs<true>(prm, vecs, f.n_ctas, smem, stream)
                                                  : launch_narrow_vecs<false>(prm, vecs, f.n_ctas, smem, stream);
    if (st != B200SPMM_OK) return st;
    p->last.n_ctas = (int)f.n_ctas;
    p->last.threads = kNarrowThreads;
    p->last.feature_slab = 64;
    p->last.n_slabs = 1;
    p->last.smem_bytes = (int64_t)smem;
    p->last.kernel_launches = 1;
    p->last.row_window = kRowWindow;
    return B200SPMM_OK;
}

int launch_tall(b200spmm_plan *p, const TallChoice &choice, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                cudaStream_t stream) {
    const bool tf32 = p->info.dtype == B200SPMM_TF32;
    int st = b_tensor_map(p, d_B, ldb, (uint32_t)n, (uint32_t)p->info.cols, tf32);
    if (st != B200SPMM_OK) return st;
    const bool pair = choice.pair;
    const TallFormat &fmt = pair ? p->pair : p->tall;
    TallParams prm{};
    prm.rowOffset = fmt.d_rowOffset;
    prm.tcA2B = fmt.d_tcA2B;
    prm.rowIdx = fmt.d_rowIdx;
    prm.data = static_cast<const uint8_t *>(fmt.d_data);
    if (choice.sparse) {
        prm.rowOffset = p->sparse.d_rowOffset;
        prm.tcA2B = p->sparse.d_tcA2B;
        prm.data = static_cast<const uint8_t *>(p->sparse.d_data);
        prm.meta = static_cast<const uint8_t *>(p->sparse.d_meta);
        prm.quads = p->sparse.d_quads;
        prm.n_rest = p->sparse.d_n_rest;
        prm.rest = p->sparse.d_rest;
        prm.B = static_cast<const uint8_t *>(d_B);
        prm.ldb_bytes = (uint64_t)ldb * 2u;
    }
    if (p->tall_pack_b) {
        const uint32_t cw = choice.sparse ? 32u : (uint32_t)p->info.col_window, esz = (uint32_t)p->info.elt_size;
        const uint32_t slab = (n <= 128 || pair) ? 128u : 256u;
        const uint32_t n_slabs = pair ? 2u * (uint32_t)((n + 255) / 256) : (uint32_t)((n + slab - 1) / slab);
        const uint32_t groups = (uint32_t)((p->info.cols + cw - 1) / cw);
        const size_t need = choice.packed_bytes;  // n_slabs * groups * cw * esz * slab
        st = take_scratch(p, &p->b_packed, need, stream);
        if (st != B200SPMM_OK) return st;
        const int grid = (int)std::min<size_t>((need / 16 + 255) / 256, (size_t)p->n_sms * 16);
        B200_CUDA_TRY(launch_after(tf32 ? pack_b_kernel<true> : choice.sparse ? pack_b_kernel<false, 32> : pack_b_kernel<false>, dim3(grid), 256, 0, 1, stream, static_cast<const uint8_t *>(d_B),
                                   ldb * esz, (uint32_t)p->info.cols, (uint32_t)n, slab, n_slabs, groups, static_cast<uint8_t *>(p->b_packed.ptr)));
        prm.b_packed = static_cast<const uint8_t *>(p->b_packed.ptr);
        prm.b_groups = groups;
    }
    prm.parts = choice.parts;
    prm.partial = static_cast<float *>(p->partial.ptr);
    prm.partial_rows = (uint32_t)(fmt.eff * fmt.rows);
    prm.sched_counter = p->d_status + 1;
    prm.C = d_C;
    prm.ldc = ldc;
    prm.rows = (uint32_t)p->info.rows;
    prm.cols = (uint32_t)p->info.cols;
    prm.n = (uint32_t)n;
    prm.eff_row_windows = (uint32_t)fmt.eff;
    prm.c_is_half = c_dtype == B200SPMM_C_F16;
    prm.status = p->d_status;
    prm.wait_limit_ns = p->wait_limit_ns;
    prm.starve_bytes = p->starve_gathers ? 16u : 0u;
#ifdef B200SPMM_PROFILE
    if (const char *dbg = std::getenv("B200SPMM_DEBUG")) prm.debug = (uint32_t)std::atoi(dbg);  // results invalid
    if (!g_prof) cudaMalloc(&g_prof, 1024 * 32 * 8);
    cudaMemsetAsync(g_prof, 0, 1024 * 32 * 8, stream);
    prm.prof = g_prof;
#endif
    if (pair) st = tf32 ? launch_pair_one<true, false>(p, prm, stream) : choice.sparse ? launch_pair_one<false, true>(p, prm, stream) : launch_pair_one<false, false>(p, prm, stream);
    else if (n <= 128) st = tf32 ? launch_tall_one<true, 128>(p, prm, stream) : launch_tall_one<false, 128>(p, prm, stream);
    else st = tf32 ? launch_tall_one<true, 256>(p, prm, stream) : launch_tall_one<false, 256>(p, prm, stream);
    if (st != B200SPMM_OK || prm.parts == 1) return st;
    const uint64_t sums = (uint64_t)fmt.eff * fmt.rows * (prm.n / 4);
    B200_CUDA_TRY(launch_after(tall_sum_parts_kernel, dim3((unsigned)((sums + 255) / 256)), 256, 0, 1, stream, (const float *)prm.partial, prm.parts,
                               fmt.d_rowIdx, prm.eff_row_windows, fmt.rows, d_C, ldc, prm.rows, prm.n, prm.c_is_half));
    ++p->last.kernel_launches;
    return B200SPMM_OK;
}

// Builds the super-window copy of the matrix when it pays.  The 16-row kernel spends about 100 SM
// clocks per tile and 128 features whatever the tile holds; the super-window kernel about 70 per
// 128-row tile and 128 features.  So the merge pays when it leaves fewer than ~0.7 of the tiles -
// i.e. when the parts of a super-window share most of their columns (a pruned weight matrix: 0.15;
// a power-law graph: ~0.9, stays with 16 rows).  B200SPMM_WINDOW=16 / 128 overrides the choice.
int plan_build_tall(b200spmm_plan *p, const uint32_t *h_rowOffset, const uint32_t *h_rowIdx) {
    const auto &info = p->info;
    if (!info.total_tiles || env_is("B200SPMM_WINDOW", "16")) return B200SPMM_OK;
    const bool want_pair = env_is("B200SPMM_WINDOW", "256");
    p->tall_forced = env_is("B200SPMM_WINDOW", "128") || want_pair;
    SuperCounts counts;
    bool counted = false;
    if (!p->tall_forced) {
        if (info.total_tiles < kTallMinShortTiles) return B200SPMM_OK;
        double ratio = 1.0;
        uint64_t n_super = 0;
        // counting all windows takes a look at every list, several where the columns are many: large graphs are sampled first
        counted = info.total_tiles * (uint64_t)info.col_window <= kTallMaxCounted && info.cols <= kTallMaxCountedCols;
        int st;
        if (counted) {
            st = count_super_windows(info, h_rowOffset, h_rowIdx, p->d_tcA2B, &counts);
            ratio = (double)counts.tall_tiles / (double)info.total_tiles;
            n_super = counts.tall_windows;
        } else {
            st = estimate_tall_tile_ratio(info, h_rowOffset, h_rowIdx, p->d_tcA2B, kTallRows, 48, &ratio, &n_super);
        }
        if (st != B200SPMM_OK) return st;
        // fewer super-windows than SMs / 32 leave the GPU half empty even in sixteen parts each
        if (ratio > 0.7 || n_super * 32 < (uint64_t)p->n_sms) return B200SPMM_OK;
    }
    int st = counted ? B200SPMM_OK : count_super_windows(info, h_rowOffset, h_rowIdx, p->d_tcA2B, &counts);
    if (st != B200SPMM_OK) return st;
    st = build_tall_device(info, counts, h_rowOffset, p->d_rowOffset, p->d_tcA2B, p->d_data, p->d_rowIdx, kTallRows, &p->tall);
    if (st == B200SPMM_ERR_UNSUPPORTED) return B200SPMM_OK;  // too many tiles for 32-bit offsets: 16-row kernel
    if (st != B200SPMM_OK || !p->tall.tiles) return st;
    // The pair kernel does twice the work per tile: it pays when a 256-row window has (about) the column
    // list of its halves, i.e. half the tiles.  B200SPMM_WINDOW=256 forces it, =128 keeps it out.
    if (!env_is("B200SPMM_WINDOW", "128")) {
        st = info.dtype == B200SPMM_TF32 ? pair_max_clusters<true>(&p->pair_clusters) : pair_max_clusters<false>(&p->pair_clusters);
        if (st != B200SPMM_OK) return st;
        if (p->pair_clusters > 0 && (want_pair || ((double)counts.pair_tiles <= 0.55 * (double)counts.tall_tiles && info.total_tiles >= kPairMinShortTiles))) {
            st = build_tall_device(info, counts, h_rowOffset, p->d_rowOffset, p->d_tcA2B, p->d_data, p->d_rowIdx, kPairRows, &p->pair);
            if (st != B200SPMM_OK && st != B200SPMM_ERR_UNSUPPORTED) return st;
        }
    }
    uint32_t aligned = 0;
    B200_CUDA_TRY(cudaMemcpy(&aligned, p->tall.d_aligned, 4, cudaMemcpyDeviceToHost));
    const bool most_aligned = (uint64_t)aligned * 2 >= p->tall.tiles;
    p->tall_pack_b = most_aligned && !env_is("B200SPMM_PACK_B", "0");
    // The windows once more in 2:4 form, where most of their lists name neighbouring rows of B (the kernel has no room for gathers
    // in every stage): 0.6 of their memory again, for launches of more than 128 columns in whole windows.  28672 x 8192 at 10 %
    // (57,344 tiles): plan 3.3 -> 3.9 ms, 1,323 -> 1,598 MB, 738 -> 688 us a product of 2,048 columns.  14336 x 4096 at 8 % (14,336): plan 0.8
    // -> 0.9 ms where the pool has room for its buffers, 1.1 -> 1.5 to 2.0 where it has not, 39 -> 31 us a product of 256 columns: up
    // to a hundred products, more than a plan that is made anew has before it.  Sizes between were not measured.
    // B200SPMM_SPARSE24=0 keeps it out, =1 asks for it wherever it fits.
    const bool always = env_is("B200SPMM_SPARSE24", "1");
    if (p->pair.tiles && most_aligned && info.dtype == B200SPMM_F16 && (always || p->pair.tiles >= kSparse24MinTiles) && !env_is("B200SPMM_SPARSE24", "0")) {
        int clusters = 0;
        st = pair_max_clusters<false, true>(&clusters);
        if (st == B200SPMM_OK && clusters >= p->pair_clusters) st = build_sparse24(p->pair, info.cols, always, &p->sparse);
        if (st != B200SPMM_OK) return st;
    }
    B200_CUDA_TRY(cudaDeviceSynchronize());
    return B200SPMM_OK;
}

// Gives the plan its tile image.  Called last in plan_finish: everything that reads the tiles in the
// reference's layout (compression, the super-window merge) has run by then.
int plan_build_tile_image(b200spmm_plan *p) {
    const uint64_t n_rows = p->info.total_tiles * (uint64_t)kRowWindow;
    if (!n_rows || p->comp.tcBit) return B200SPMM_OK;  // compressed tiles are expanded in the kernel
    void *dst = p->d_data;
    if (!p->owns_format) {
        if (pool_alloc_bytes(&dst, n_rows * 32, nullptr) != cudaSuccess) {  // no room for a copy: the tiled loads still work
            cudaGetLastError();
            return B200SPMM_OK;
        }
        p->image_is_copy = true;
    }
    const int grid = (int)std::min<uint64_t>((n_rows + 255) / 256, 148 * 16);
    tileimage::swizzle_tiles_kernel<<<grid, 256>>>(static_cast<const uint4 *>(p->d_data), static_cast<uint4 *>(dst), n_rows);
    B200_CUDA_TRY(cudaGetLastError());
    B200_CUDA_TRY(cudaDeviceSynchronize());
    p->d_tiles_image = dst;
    return B200SPMM_OK;
}

// The schedule of the 16-row kernel, on the device.
int plan_build_schedule(b200spmm_plan *p, const uint32_t *h_rowOffset, const uint32_t *h_rowIdx, int n_ctas) {
    const auto &info = p->info;
    {
        b200spmm_plan::Sched &ps = p->sched;
        ps.n_ctas = n_ctas > 0 ? n_ctas : p->n_sms * kCtasPerSm;
        // Several chunks per CTA, taken from all over the matrix, even out regions whose tiles
        // cost more than the schedule's model says; a chunk stays long enough (512 tiles or
        // more) for the hand-over at its start not to matter.
        const uint64_t per_cta = info.total_tiles / (uint64_t)ps.n_ctas;
        const int chunks_per_cta = (int)std::min<uint64_t>(kMaxChunksPerCta, std::max<uint64_t>(1, per_cta / 512));
        ps.n_chunks = (uint32_t)(ps.n_ctas * chunks_per_cta);
        TileSchedule sc;
        build_tile_schedule(h_rowOffset, info.eff_row_windows, (int)ps.n_chunks, /*allow_split=*/true, &sc);
        std::vector<SplitWindow> splits;
        for (const auto &sp : sc.splits) splits.push_back(SplitWindow{sp.window, sp.piece_begin, sp.piece_end});
        // one copy brings all tables
        std::vector<uint32_t> tables;
        auto append = [&](const auto &v) {
            const size_t at = tables.size();
            tables.resize(at + v.size() * sizeof(v[0]) / 4);
            std::memcpy(tables.data() + at, v.data(), v.size() * sizeof(v[0]));
            return at;
        };
        const size_t tile = append(sc.tile), wfirst = append(sc.wfirst), wlast = append(sc.wlast), head = append(sc.head_slot),
                     tail = append(sc.tail_slot), split = append(splits), pieces = append(sc.piece_slots);
        B200_CUDA_TRY(pool_alloc(&ps.d_tables, tables.size()));
        B200_CUDA_TRY(cudaMemcpy(ps.d_tables, tables.data(), tables.size() * 4, cudaMemcpyHostToDevice));
        ps.d_tile = ps.d_tables + tile;
        ps.d_wfirst = ps.d_tables + wfirst;
        ps.d_wlast = ps.d_tables + wlast;
        ps.d_head_slot = ps.d_tables + head;
        ps.d_tail_slot = ps.d_tables + tail;
        ps.d_splits = reinterpret_cast<SplitWindow *>(ps.d_tables + split);
        ps.d_piece_slots = ps.d_tables + pieces;
        ps.n_splits = (uint32_t)splits.size();
        ps.n_slots = sc.n_slots;
        RowBands bands;  // only schedules with many chunks are worth launching in bands
        build_row_bands(sc, h_rowIdx, info.rows, ps.n_chunks >= (uint32_t)ps.n_ctas * 8u ? kRowBands : 1u, &bands);
        ps.band_chunk = bands.chunk;
        ps.band_row = bands.row;
        ps.band_split = bands.split;
    }
    return B200SPMM_OK;
}

// What the tile kernels need beside the format: schedule, compressed tiles or super-windows, tile image.
int plan_build_tile_path(b200spmm_plan *p, const uint32_t *h_rowOffset, const uint32_t *h_rowIdx, int n_ctas) {
    const auto &info = p->info;
    {
        int st = plan_build_schedule(p, h_rowOffset, h_rowIdx, n_ctas);
        if (st == B200SPMM_OK) st = encode_tile_map(p);
        if (st != B200SPMM_OK) return st;
    }
    // On request (B200SPMM_TILES=bitmap) the kernels stream the tiles in compressed form - bitmap +
    // stored values, expanded by the producer warps - instead of the dense 512-byte tiles; both
    // give the same C bit for bit.  The compressed form moves an eighth of the tile bytes at a
    // few per cent fill but costs the producer warps more instructions per tile than they can
    // spare today, so dense tiles are the default.
    if (info.total_tiles && env_is("B200SPMM_TILES", "bitmap")) {
        int st = compress_tiles_device(p->d_data, info.total_tiles, info.dtype, &p->comp);
        if (st != B200SPMM_OK) return st;
    }
    // B200SPMM_TILES=entries (fp16): the kernels stream the tiles as records of 32 (position, value) words - a
    // quarter of the dense bytes - which a producer warp expands with two stores per lane; tiles with more than
    // 32 entries still come from the dense image.  Same C bit for bit.
    if (info.total_tiles && info.dtype == B200SPMM_F16 && env_is("B200SPMM_TILES", "entries")) {
        B200_CUDA_TRY(pool_alloc(&p->d_tile_entries, info.total_tiles * 32));
        unsigned long long *d_count = nullptr;
        B200_CUDA_TRY(cudaMalloc(&d_count, 8));
        B200_CUDA_TRY(cudaMemset(d_count, 0, 8));
        const int grid = (int)std::min<uint64_t>((info.total_tiles + 7) / 8, (uint64_t)p->n_sms * 32);
        tileimage::tile_entries_kernel<<<grid, 256>>>(static_cast<const uint16_t *>(p->d_data), info.total_tiles, p->d_tile_entries, d_count);
        cudaError_t e = cudaGetLastError();
        unsigned long long n_dense = 0;
        if (e == cudaSuccess) e = cudaMemcpy(&n_dense, d_count, 8, cudaMemcpyDeviceToHost);
        cudaFree(d_count);
        B200_CUDA_TRY(e);
        p->entry_dense_tiles = n_dense;
    }
    // an explicit CTA count or compressed tiles ask for the 16-row kernel, and loose lists cannot be merged
    if (n_ctas <= 0 && !p->comp.tcBit && !p->loose_lists) {
        int st = plan_build_tall(p, h_rowOffset, h_rowIdx);
        if (st != B200SPMM_OK) return st;
    }
    p->has_tile_path = true;
    // An explicit CTA count, window height, form of the tiles or way to fetch rows asks for the pipelined kernels, and so does a
    // matrix of which less than one window in sixteen holds entries.  (How long its gaps may be: choose_window_lines.)
    p->windows_forced = env_is("B200SPMM_WINDOW", "warps");
    p->windows_fit = n_ctas <= 0 && !p->loose_lists && !p->gather_cpasync && !std::getenv("B200SPMM_TILES") &&
                     (p->windows_forced || (!std::getenv("B200SPMM_WINDOW") && !p->sched.n_splits && info.total_row_windows <= 16 * info.eff_row_windows));
    uint64_t row = 0;  // behind the last window so far
    for (uint64_t w = 0; w < info.eff_row_windows; ++w) {
        p->max_short_tiles = std::max(p->max_short_tiles, h_rowOffset[w + 1] - h_rowOffset[w]);
        p->max_gap = std::max(p->max_gap, (uint32_t)((h_rowIdx[w] - row) / kRowWindow));
        row = (uint64_t)h_rowIdx[w] + kRowWindow;
    }
    if (info.rows > row) p->max_gap = std::max(p->max_gap, (uint32_t)((info.rows - row + kRowWindow - 1) / kRowWindow));
    return plan_build_tile_image(p);
}

// The window tables on the host, where the caller has them on the device only.
int read_window_tables(b200spmm_plan *p, std::vector<uint32_t> *rowOffset, std::vector<uint32_t> *rowIdx) {
    rowOffset->resize(p->info.eff_row_windows + 1);
    rowIdx->resize(p->info.eff_row_windows);
    B200_CUDA_TRY(cudaMemcpy(rowOffset->data(), p->d_rowOffset, rowOffset->size() * 4, cudaMemcpyDeviceToHost));
    if (!rowIdx->empty()) B200_CUDA_TRY(cudaMemcpy(rowIdx->data(), p->d_rowIdx, rowIdx->size() * 4, cudaMemcpyDeviceToHost));
    return B200SPMM_OK;
}

int plan_add_tile_path(b200spmm_plan *p, int n_ctas) {
    std::vector<uint32_t> h_rowOffset, h_rowIdx;
    const int st = read_window_tables(p, &h_rowOffset, &h_rowIdx);
    if (st != B200SPMM_OK) return st;
    return plan_build_tile_path(p, h_rowOffset.data(), h_rowIdx.data(), n_ctas);
}

// What every plan starts with: a format and a device the kernels take, and the status word.
int plan_start(b200spmm_plan *p) {
    const auto &info = p->info;
    if (info.row_window != kRowWindow) return B200SPMM_ERR_UNSUPPORTED;
    const int cw = info.dtype == B200SPMM_F16 ? 16 : 8;
    if (info.col_window != cw) return B200SPMM_ERR_UNSUPPORTED;
    if (info.total_tiles * (uint64_t)kRowWindow >= 0x7FFFFFFFull) return B200SPMM_ERR_UNSUPPORTED;  // TMA row coordinate
    int major = 0;
    B200_CUDA_TRY(cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, p->device));
    if (major != 10) return B200SPMM_ERR_NO_DEVICE;
    B200_CUDA_TRY(cudaDeviceGetAttribute(&p->n_sms, cudaDevAttrMultiProcessorCount, p->device));
    // status word, then the two counters of the chunk hand-out (the kernel leaves them at zero), then what tables_kernel finds
    B200_CUDA_TRY(pool_alloc(&p->d_status, 6));
    B200_CUDA_TRY(cudaMemset(p->d_status, 0, 6 * sizeof(uint32_t)));
    return B200SPMM_OK;
}

formatcheck::Found *tables_found(const b200spmm_plan *p) { return reinterpret_cast<formatcheck::Found *>(p->d_status + 4); }

// A caller's device arrays: looked over while the plan is made.
int plan_start_table_check(b200spmm_plan *p) {
    const auto &info = p->info;
    if (info.eff_row_windows > info.total_tiles) return B200SPMM_ERR_INVALID_ARG;  // every window holds a tile
    const uint64_t n = std::max<uint64_t>(info.eff_row_windows, info.total_tiles * (uint64_t)info.col_window / 4);
    const int grid = (int)std::max<uint64_t>(1, std::min<uint64_t>((n + 255) / 256, (uint64_t)p->n_sms * 8));
    tables_kernel<<<grid, 256>>>(p->d_rowOffset, p->d_tcA2B, p->d_rowIdx, (uint32_t)info.eff_row_windows, (uint32_t)info.total_tiles,
                                              info.rows, info.cols, (uint32_t)info.col_window, tables_found(p));
    B200_CUDA_TRY(cudaGetLastError());
    return B200SPMM_OK;
}

// Refused, or marked as loose (see tables_kernel).
int plan_take_found(b200spmm_plan *p, const formatcheck::Found &found) {
    if (found.bad()) {
        set_last_error_static("rowOffset or rowIdx does not describe windows of the matrix");
        return B200SPMM_ERR_INVALID_ARG;
    }
    p->loose_lists = found.loose();
    p->row_boxes = !p->loose_lists;
    return B200SPMM_OK;
}

// h_rowOffset and h_rowIdx may be null: they are read back if the plan needs them.  A caller's device arrays (checked) are being
// looked over: what that finds comes with the sizes of the row units where those are asked for, or is waited for.
int plan_finish(b200spmm_plan *p, const uint32_t *h_rowOffset, const uint32_t *h_rowIdx, int n_ctas, bool checked) {
    const auto &info = p->info;
    formatcheck::Found found{};
    bool found_known = !checked;
    auto wait_for_check = [&]() -> int {
        if (!found_known) B200_CUDA_TRY(cudaMemcpy(&found, tables_found(p), sizeof(found), cudaMemcpyDeviceToHost));
        found_known = true;
        return plan_take_found(p, found);
    };
    const int cw = info.col_window;
    p->gather_cpasync = env_is("B200SPMM_GATHER", "cpasync");
    p->host_split = !env_is("B200SPMM_HOST_SPLIT", "0");
    // An explicit CTA count, a way to fetch tiles or rows, or a window height asks for a tile kernel.
    // B200SPMM_WINDOW=rows asks for the row units whatever the matrix.
    const bool force_rows = env_is("B200SPMM_WINDOW", "rows");
    if (n_ctas <= 0 && (force_rows || (!std::getenv("B200SPMM_WINDOW") && !std::getenv("B200SPMM_TILES") && !p->gather_cpasync))) {
        const double fill = info.total_tiles ? (double)info.nnzs / ((double)info.total_tiles * kRowWindow * cw) : 0.0;
        double max_fill = kRowsMaxFill;
        if (fill > kRowsMaxFill && fill <= kRowsMaxFillWide && info.total_tiles >= kRowsWideMinTiles && !force_rows) {
            int st = wait_for_check();
            if (st != B200SPMM_OK) return st;
            std::vector<uint32_t> tables[2];
            if (!h_rowOffset) {
                st = read_window_tables(p, &tables[0], &tables[1]);
                if (st != B200SPMM_OK) return st;
            }
            double ratio = 1.0;
            uint64_t n_super = 0;
            st = estimate_tall_tile_ratio(info, h_rowOffset ? h_rowOffset : tables[0].data(), h_rowOffset ? h_rowIdx : tables[1].data(),
                                              p->d_tcA2B, kTallRows, 48, &ratio, &n_super);
            if (st != B200SPMM_OK) return st;
            // (an eighth of the short tiles is the least that merging eight windows can leave)
            if (fill / (8.0 * ratio) < kTallMinFill || info.total_tiles < kRowsWideAnyTiles) max_fill = kRowsMaxFillWide;
        }
        const int built = build_row_formats(info, p->d_rowOffset, p->d_tcA2B, p->d_data, p->d_rowIdx, checked ? tables_found(p) : nullptr, &found, &found_known,
                                            p->n_sms, max_fill, force_rows, &p->rows_fmt, &p->narrow);
        const int st = wait_for_check();  // (bad tables are refused as such, whatever became of the row units)
        if (st != B200SPMM_OK) return st;
        if (built != B200SPMM_OK) return built;
        p->rows_only = p->rows_fmt.n_units > 0;
        if (p->rows_only) return B200SPMM_OK;
    }
    const int st = wait_for_check();
    if (st != B200SPMM_OK) return st;
    return h_rowOffset ? plan_build_tile_path(p, h_rowOffset, h_rowIdx, n_ctas) : plan_add_tile_path(p, n_ctas);
}

}  // namespace

// ------------------------------------------------------------------ allocation-free launch path
namespace noalloc {
//
// Working memory of b200spmm_spmm_noalloc: the schedule tables (tile cuts, first and last window
// per CTA) and the kernel status word.  It is part of the library image, so every GPU that loads
// the library holds these 16 KiB until the process exits and no call ever has to allocate them.
constexpr int kNoAllocMaxCtas = 1024;
constexpr int kNoAllocTile = 0;                                  // [kNoAllocMaxCtas + 1]
constexpr int kNoAllocWfirst = kNoAllocTile + kNoAllocMaxCtas + 1;  // [kNoAllocMaxCtas]
constexpr int kNoAllocWlast = kNoAllocWfirst + kNoAllocMaxCtas;     // [kNoAllocMaxCtas]
constexpr int kNoAllocStatusWord = kNoAllocWlast + kNoAllocMaxCtas;
static __device__ __align__(256) uint32_t g_noalloc_scratch[4096];

// Cuts of the effective row windows over n_ctas CTAs by the same cost model as the host
// scheduler, always on window boundaries (no window is shared between CTAs, so no partial-result
// slots are needed).  One block; also clears the status word.
__global__ void noalloc_schedule_kernel(const uint32_t *__restrict__ rowOffset, uint32_t eff, int n_ctas,
                                        uint32_t *__restrict__ scratch) {
    __shared__ uint32_t cut[kNoAllocMaxCtas + 1];
    if (threadIdx.x == 0) scratch[kNoAllocStatusWord] = 0;
    auto cost = [&](uint64_t w) { return (uint64_t)rowOffset[w] + kWindowCharge * w; };
    const uint64_t total = eff ? cost(eff) : 0;
    for (int c = (int)threadIdx.x; c <= n_ctas; c += (int)blockDim.x) {
        uint64_t lo = 0, hi = eff;
        if (c == n_ctas) {
            lo = eff;
        } else if (c > 0) {
            const uint64_t target = total * (uint64_t)c / (uint64_t)n_ctas;
            while (lo < hi) {
                const uint64_t mid = (lo + hi) / 2;
                if (cost(mid) < target) lo = mid + 1; else hi = mid;
            }
        }
        cut[c] = (uint32_t)lo;
        scratch[kNoAllocTile + c] = rowOffset[lo];
    }
    __syncthreads();
    for (int c = (int)threadIdx.x; c < n_ctas; c += (int)blockDim.x) {
        scratch[kNoAllocWfirst + c] = cut[c];
        scratch[kNoAllocWlast + c] = cut[c + 1] > cut[c] ? cut[c + 1] - 1 : cut[c];
    }
}

// Device address of g_noalloc_scratch on `device`, looked up on first use.  The name of a
// __device__ array is only a host-side handle; kernels must be given this address.
int noalloc_scratch_address(int device, uint32_t **out) {
    constexpr int kMaxDevices = 64;
    static uint32_t *cache[kMaxDevices] = {};
    static std::mutex lock;
    if (device < 0 || device >= kMaxDevices) return B200SPMM_ERR_INVALID_ARG;
    std::lock_guard<std::mutex> guard(lock);
    if (!cache[device]) {
        void *ptr = nullptr;
        B200_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_noalloc_scratch));  // `device` is current (set by the caller)
        cache[device] = static_cast<uint32_t *>(ptr);
    }
    *out = cache[device];
    return B200SPMM_OK;
}

}  // namespace noalloc
using namespace noalloc;

#ifdef B200SPMM_PROFILE
extern "C" int b200spmm_debug_read_profile(unsigned long long *out, int n_ctas) {
    return cudaMemcpy(out, g_prof, (size_t)n_ctas * 32 * 8, cudaMemcpyDeviceToHost) == cudaSuccess ? 0 : -5;
}
#endif

extern "C" {

const char *b200spmm_status_string(int status) {
    switch (status) {
        case B200SPMM_OK: return "ok";
        case B200SPMM_ERR_INVALID_ARG: return "invalid argument";
        case B200SPMM_ERR_BAD_CSR: return "malformed CSR (row_ptr not monotone, wrong nnz, or column out of range)";
        case B200SPMM_ERR_UNSUPPORTED: return "shape, size or alignment not supported";
        case B200SPMM_ERR_NO_MEMORY: return "host allocation failed";
        case B200SPMM_ERR_CUDA: return "CUDA call failed (see b200spmm_last_cuda_error)";
        case B200SPMM_ERR_NO_DEVICE: return "no sm_100 device available";
        case B200SPMM_ERR_DEVICE_TIMEOUT: return "a bounded wait inside the kernel ran out";
        default: return "unknown status";
    }
}

const char *b200spmm_last_cuda_error(void) { return g_last_static_error ? g_last_static_error : g_last_cuda_error.c_str(); }

int b200spmm_version(void) { return 100; }

int b200spmm_csr2btcf_nobitmap(uint64_t rows, uint64_t cols, uint64_t nnz, const uint32_t *row_ptr,
                               const uint32_t *col_idx, const void *values, int dtype, int row_window,
                               int col_window, int n_threads, b200spmm_btcf_t **out) {
    if (!out) return B200SPMM_ERR_INVALID_ARG;
    *out = nullptr;
    b200spmm_btcf *h = new (std::nothrow) b200spmm_btcf();
    if (!h) return B200SPMM_ERR_NO_MEMORY;
    int st = guarded([&]() { return convert_csr_to_btcf(rows, cols, nnz, row_ptr, col_idx, values, dtype, row_window, col_window, n_threads, &h->f); });
    if (st != B200SPMM_OK) {
        delete h;
        return st;
    }
    *out = h;
    return B200SPMM_OK;
}

int b200spmm_btcf_transpose_tiles(b200spmm_btcf_t *f) {
    if (!f) return B200SPMM_ERR_INVALID_ARG;
    return guarded([&]() -> int {
        transpose_tiles(&f->f);
        return B200SPMM_OK;
    });
}

int b200spmm_btcf_tiles_col_major(const b200spmm_btcf_t *f) { return f && f->f.col_major_tiles ? 1 : 0; }

int b200spmm_btcf_rewindow(const b200spmm_btcf_info_t *info, const uint32_t *rowOffset, const uint32_t *tcA2B,
                           const void *data, const uint32_t *rowIdx, int row_window, int n_threads,
                           b200spmm_btcf_t **out) {
    if (!out) return B200SPMM_ERR_INVALID_ARG;
    *out = nullptr;
    if (!info || !rowOffset) return B200SPMM_ERR_INVALID_ARG;
    if (rowOffset[info->eff_row_windows] != info->total_tiles) return B200SPMM_ERR_INVALID_ARG;
    b200spmm_btcf *h = new (std::nothrow) b200spmm_btcf();
    if (!h) return B200SPMM_ERR_NO_MEMORY;
    int st = guarded([&]() {
        return rewindow_btcf(info->rows, info->cols, info->nnzs, info->dtype, info->row_window, info->col_window,
                             info->eff_row_windows, rowOffset, tcA2B, data, rowIdx, row_window, n_threads, &h->f);
    });
    if (st != B200SPMM_OK) {
        delete h;
        return st;
    }
    *out = h;
    return B200SPMM_OK;
}

int b200spmm_btcf_info(const b200spmm_btcf_t *h, b200spmm_btcf_info_t *info) {
    if (!h || !info) return B200SPMM_ERR_INVALID_ARG;
    const Btcf &f = h->f;
    info->rows = f.rows;
    info->cols = f.cols;
    info->nnzs = f.nnzs;
    info->total_row_windows = f.total_row_windows;
    info->eff_row_windows = f.eff_row_windows;
    info->total_tiles = f.total_tiles;
    info->row_window = f.row_window;
    info->col_window = f.col_window;
    info->dtype = f.dtype;
    info->elt_size = f.elt_size;
    return B200SPMM_OK;
}

const uint32_t *b200spmm_btcf_rowOffset(const b200spmm_btcf_t *h) { return h ? h->f.rowOffset.data() : nullptr; }
const uint32_t *b200spmm_btcf_tcA2B(const b200spmm_btcf_t *h) { return h ? h->f.tcA2B.data() : nullptr; }
const void *b200spmm_btcf_data(const b200spmm_btcf_t *h) { return h ? h->f.data.data() : nullptr; }
const uint32_t *b200spmm_btcf_rowIdx(const b200spmm_btcf_t *h) { return h ? h->f.rowIdx.data() : nullptr; }
void b200spmm_btcf_destroy(b200spmm_btcf_t *h) { delete h; }

int b200spmm_shard_rows(uint64_t rows, const uint32_t *row_ptr, int row_window, int parts, uint64_t *row_begin) {
    return shard_rows(rows, row_ptr, row_window, parts, 0, row_begin);
}

int b200spmm_shard_rows_weighted(uint64_t rows, const uint32_t *row_ptr, int row_window, int parts,
                                 uint64_t row_charge, uint64_t *row_begin) {
    return shard_rows(rows, row_ptr, row_window, parts, row_charge, row_begin);
}

int b200spmm_allgather_plan(const uint64_t *cut, int n_parts, uint64_t *even_part, uint64_t *pieces) {
    if (!cut || !even_part || n_parts < 1 || (n_parts > 1 && !pieces)) return B200SPMM_ERR_INVALID_ARG;
    for (int d = 0; d < n_parts; ++d)
        if (cut[d + 1] < cut[d]) return B200SPMM_ERR_INVALID_ARG;
    *even_part = exchange_even_part(cut, n_parts);
    for (int d = 0; d < n_parts; ++d)
        for (int step = 1; step < n_parts; ++step) {
            uint64_t *out = pieces + ((size_t)d * (size_t)(n_parts - 1) + (size_t)(step - 1)) * 10;
            int to = 0, from = 0;
            exchange_pieces(cut, n_parts, *even_part, d, step, &to, &from, out + 2);
            out[0] = (uint64_t)to;
            out[1] = (uint64_t)from;
        }
    return B200SPMM_OK;
}

int b200spmm_build_schedule(const uint32_t *rowOffset, uint64_t eff_row_windows, int n_ctas, uint32_t *cta_window) {
    return guarded([&]() -> int {
        if (!rowOffset || !cta_window || n_ctas < 1) return B200SPMM_ERR_INVALID_ARG;
        std::vector<uint32_t> cuts;
        build_cta_schedule(rowOffset, eff_row_windows, n_ctas, &cuts);
        std::memcpy(cta_window, cuts.data(), cuts.size() * sizeof(uint32_t));
        return B200SPMM_OK;
    });
}

int b200spmm_build_tile_schedule(const uint32_t *rowOffset, uint64_t eff_row_windows, int n_ctas, uint32_t *cta_tile,
                                 uint32_t *cta_wfirst, uint32_t *cta_wlast, uint32_t *slot_window) {
    return guarded([&]() -> int {
        if (!rowOffset || !cta_tile || !cta_wfirst || !cta_wlast || !slot_window || n_ctas < 1) return B200SPMM_ERR_INVALID_ARG;
        TileSchedule sc;
        build_tile_schedule(rowOffset, eff_row_windows, n_ctas, /*allow_split=*/true, &sc);
        std::memcpy(cta_tile, sc.tile.data(), sc.tile.size() * sizeof(uint32_t));
        std::memcpy(cta_wfirst, sc.wfirst.data(), sc.wfirst.size() * sizeof(uint32_t));
        std::memcpy(cta_wlast, sc.wlast.data(), sc.wlast.size() * sizeof(uint32_t));
        for (int c = 0; c < n_ctas; ++c) {
            slot_window[2 * c] = sc.head_slot[c] != kNoSlot ? sc.wfirst[c] : 0xFFFFFFFFu;
            slot_window[2 * c + 1] = sc.tail_slot[c] != kNoSlot ? sc.wlast[c] : 0xFFFFFFFFu;
        }
        return B200SPMM_OK;
    });
}

int b200spmm_build_row_bands(const uint32_t *rowOffset, const uint32_t *rowIdx, uint64_t eff_row_windows, uint64_t rows,
                             int n_parts, int max_bands, uint32_t *band_chunk, uint64_t *band_row, int *n_bands) {
    return guarded([&]() -> int {
        if (!rowOffset || !band_chunk || !band_row || !n_bands || n_parts < 1 || max_bands < 1 || (eff_row_windows && !rowIdx))
            return B200SPMM_ERR_INVALID_ARG;
        TileSchedule sc;
        build_tile_schedule(rowOffset, eff_row_windows, n_parts, /*allow_split=*/true, &sc);
        RowBands bands;
        build_row_bands(sc, rowIdx, rows, (uint32_t)max_bands, &bands);
        *n_bands = (int)bands.chunk.size() - 1;
        std::memcpy(band_chunk, bands.chunk.data(), bands.chunk.size() * sizeof(uint32_t));
        std::memcpy(band_row, bands.row.data(), bands.row.size() * sizeof(uint64_t));
        return B200SPMM_OK;
    });
}

void b200spmm_plan_destroy(b200spmm_plan_t *p) {
    if (!p) return;
    cudaSetDevice(p->device);
    cudaDeviceSynchronize();  // a launch may still be using the plan
    if (p->owns_format) {
        pool_free(p->d_rowOffset);
        pool_free(p->d_tcA2B);
        pool_free(p->d_rowIdx);
        pool_free(p->d_data);
    }
    {
        auto &ps = p->sched;
        pool_free(ps.d_tables);
    }
    free_compressed_tiles(&p->comp);
    free_rows(&p->rows_fmt);
    free_narrow(&p->narrow);
    pool_free(p->d_tile_entries);
    free_tall(&p->tall);
    free_tall(&p->pair);
    free_sparse24(&p->sparse);
    pool_free(p->b_packed.ptr);
    pool_free(p->partial.ptr);
    for (void *old : p->outgrown) pool_free(old);
    if (p->image_is_copy) pool_free(p->d_tiles_image);
    for (cudaEvent_t e : p->band_done) cudaEventDestroy(e);
    if (p->copy_stream) cudaStreamDestroy(p->copy_stream);
    if (p->upload_stream) cudaStreamDestroy(p->upload_stream);
    for (cudaEvent_t e : p->half_up)
        if (e) cudaEventDestroy(e);
    pool_free(p->d_status);
    pool_free(p->d_B);
    pool_free(p->d_C);
    delete p;
}

int b200spmm_plan_create(const b200spmm_btcf_t *h, int device, int n_ctas, b200spmm_plan_t **out) {
    if (!h || !out) return B200SPMM_ERR_INVALID_ARG;
    *out = nullptr;
    if (h->f.col_major_tiles) {  // the kernels read row-major tiles (the reference's default build)
        set_last_error_static("tiles are stored column-major: b200spmm_btcf_transpose_tiles brings them back");
        return B200SPMM_ERR_UNSUPPORTED;
    }
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || device < 0 || device >= n_dev) {
        cudaGetLastError();
        return B200SPMM_ERR_NO_DEVICE;
    }
    B200_CUDA_TRY(cudaSetDevice(device));
    b200spmm_plan *p = new (std::nothrow) b200spmm_plan();
    if (!p) return B200SPMM_ERR_NO_MEMORY;
    p->device = device;
    p->owns_format = true;
    b200spmm_btcf_info(h, &p->info);
    const Btcf &f = h->f;
    auto upload = [&](void **dst, const void *src, size_t bytes) -> int {
        B200_CUDA_TRY(pool_alloc_bytes(dst, std::max<size_t>(bytes, 16), nullptr));
        if (bytes)
            return guarded([&]() -> int {
                B200_CUDA_TRY(upload_pageable(*dst, src, bytes));
                return B200SPMM_OK;
            });
        return B200SPMM_OK;
    };
    int st = upload((void **)&p->d_rowOffset, f.rowOffset.data(), f.rowOffset.size() * 4);
    if (st == B200SPMM_OK) st = upload((void **)&p->d_tcA2B, f.tcA2B.data(), f.tcA2B.size() * 4);
    if (st == B200SPMM_OK) st = upload((void **)&p->d_rowIdx, f.rowIdx.data(), f.rowIdx.size() * 4);
    if (st == B200SPMM_OK) st = upload(&p->d_data, f.data.data(), f.data.size());
    if (st == B200SPMM_OK) st = plan_start(p);
    if (st == B200SPMM_OK) st = guarded([&]() { return plan_finish(p, f.rowOffset.data(), f.rowIdx.data(), n_ctas, false); });
    if (st != B200SPMM_OK) {
        b200spmm_plan_destroy(p);
        return st;
    }
    *out = p;
    return B200SPMM_OK;
}

int b200spmm_plan_create_device(const b200spmm_btcf_info_t *info, const uint32_t *d_rowOffset, const uint32_t *d_tcA2B,
                                const void *d_data, const uint32_t *d_rowIdx, int device, int n_ctas,
                                b200spmm_plan_t **out) {
    if (!info || !out || !d_rowOffset) return B200SPMM_ERR_INVALID_ARG;
    if (info->total_tiles && (!d_tcA2B || !d_data || !d_rowIdx)) return B200SPMM_ERR_INVALID_ARG;
    if (((reinterpret_cast<uintptr_t>(d_data) | reinterpret_cast<uintptr_t>(d_tcA2B)) & 15u) != 0) return B200SPMM_ERR_UNSUPPORTED;
    *out = nullptr;
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || device < 0 || device >= n_dev) {
        cudaGetLastError();
        return B200SPMM_ERR_NO_DEVICE;
    }
    B200_CUDA_TRY(cudaSetDevice(device));
    b200spmm_plan *p = new (std::nothrow) b200spmm_plan();
    if (!p) return B200SPMM_ERR_NO_MEMORY;
    p->device = device;
    p->owns_format = false;
    p->info = *info;
    p->d_rowOffset = const_cast<uint32_t *>(d_rowOffset);
    p->d_tcA2B = const_cast<uint32_t *>(d_tcA2B);
    p->d_rowIdx = const_cast<uint32_t *>(d_rowIdx);
    p->d_data = const_cast<void *>(d_data);
    p->info.elt_size = info->dtype == B200SPMM_F16 ? 2 : 4;
    int st = plan_start(p);
    if (st == B200SPMM_OK) st = plan_start_table_check(p);
    if (st == B200SPMM_OK) st = guarded([&]() { return plan_finish(p, nullptr, nullptr, n_ctas, true); });
    if (st != B200SPMM_OK) {
        b200spmm_plan_destroy(p);
        return st;
    }
    *out = p;
    return B200SPMM_OK;
}

int b200spmm_plan_info(const b200spmm_plan_t *p, b200spmm_btcf_info_t *info) {
    if (!p || !info) return B200SPMM_ERR_INVALID_ARG;
    *info = p->info;
    return B200SPMM_OK;
}

static int super_window_info(const b200spmm_plan_t *p, const TallFormat &f, int rows, b200spmm_btcf_info_t *info) {
    if (!p || !info) return B200SPMM_ERR_INVALID_ARG;
    *info = p->info;
    info->row_window = f.tiles ? rows : 0;
    info->total_row_windows = (p->info.rows + rows - 1) / rows;
    info->eff_row_windows = f.eff;
    info->total_tiles = f.tiles;
    return B200SPMM_OK;
}

static int super_window_copy_to_host(const b200spmm_plan_t *p, const TallFormat &f, uint32_t *rowOffset, uint32_t *tcA2B,
                                     void *data, uint32_t *rowIdx) {
    return guarded([&]() -> int {
        if (!p || !rowOffset || !tcA2B || !data || !rowIdx) return B200SPMM_ERR_INVALID_ARG;
        if (!f.tiles) return B200SPMM_ERR_UNSUPPORTED;
        B200_CUDA_TRY(cudaSetDevice(p->device));
        const uint64_t cw = (uint64_t)p->info.col_window, parts = f.rows / 128u;
        B200_CUDA_TRY(cudaMemcpy(rowOffset, f.d_rowOffset, (f.eff + 1) * 4, cudaMemcpyDeviceToHost));
        B200_CUDA_TRY(cudaMemcpy(rowIdx, f.d_rowIdx, f.eff * 4, cudaMemcpyDeviceToHost));
        B200_CUDA_TRY(cudaMemcpy(tcA2B, f.d_tcA2B, f.tiles * cw * 4, cudaMemcpyDeviceToHost));
        // The device copy holds 128-row images as they lie in shared memory (the halves of a row swapped when
        // row / 4 is odd), for 256-row windows per window first rows 0-127 of all its tiles, then rows 128-255:
        // put the halves back and the images where the converter would have them.
        std::vector<uint8_t> img(f.tiles * parts * 4096);
        B200_CUDA_TRY(cudaMemcpy(img.data(), f.d_data, img.size(), cudaMemcpyDeviceToHost));
        uint8_t *bytes = static_cast<uint8_t *>(data);
        for (uint64_t g = 0; g < f.eff; ++g) {
            const uint64_t first = rowOffset[g], n_tiles = rowOffset[g + 1] - first;
            for (uint64_t part = 0; part < parts; ++part)
                for (uint64_t t = 0; t < n_tiles; ++t) {
                    const uint8_t *src = img.data() + (first * parts + part * n_tiles + t) * 4096;
                    uint8_t *dst = bytes + ((first + t) * parts + part) * 4096;
                    for (uint32_t r = 0; r < 128; ++r) {
                        const uint32_t flip = (r >> 2) & 1u;
                        std::memcpy(dst + r * 32, src + r * 32 + (flip ? 16 : 0), 16);
                        std::memcpy(dst + r * 32 + 16, src + r * 32 + (flip ? 0 : 16), 16);
                    }
                }
        }
        return B200SPMM_OK;
    });
}

int b200spmm_plan_tall_info(const b200spmm_plan_t *p, b200spmm_btcf_info_t *info) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    return super_window_info(p, p->tall, kTallRows, info);
}
int b200spmm_plan_tall_copy_to_host(const b200spmm_plan_t *p, uint32_t *rowOffset, uint32_t *tcA2B, void *data,
                                    uint32_t *rowIdx) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    return super_window_copy_to_host(p, p->tall, rowOffset, tcA2B, data, rowIdx);
}
int b200spmm_plan_pair_info(const b200spmm_plan_t *p, b200spmm_btcf_info_t *info) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    return super_window_info(p, p->pair, kPairRows, info);
}
int b200spmm_plan_pair_copy_to_host(const b200spmm_plan_t *p, uint32_t *rowOffset, uint32_t *tcA2B, void *data,
                                    uint32_t *rowIdx) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    return super_window_copy_to_host(p, p->pair, rowOffset, tcA2B, data, rowIdx);
}

int b200spmm_plan_launch_info(const b200spmm_plan_t *p, b200spmm_launch_info_t *info) {
    if (!p || !info) return B200SPMM_ERR_INVALID_ARG;
    *info = p->last;
    return B200SPMM_OK;
}

}  // extern "C"

namespace {

// cudaSetDevice costs a launch-bound call more than asking.
cudaError_t make_current(int device) {
    int now = -1;
    const cudaError_t e = cudaGetDevice(&now);
    return e == cudaSuccess && now != device ? cudaSetDevice(device) : e;
}

// A kernel that may raise the status word goes to `stream`.
void note_bounded_waits(b200spmm_plan_t *p, cudaStream_t stream) {
    using Unread = b200spmm_plan::Unread;
    if (p->unread == Unread::any) return;
    unsigned long long id = 0;
    const bool known = !is_captured(stream) && cudaStreamGetId(stream, &id) == cudaSuccess;  // (asking a stream for its id ends its capture)
    if (!known) cudaGetLastError();
    if (!known || (p->unread == Unread::one_stream && p->unread_stream != id)) {
        p->unread = Unread::any;
        return;
    }
    p->unread = Unread::one_stream;
    p->unread_stream = id;
}

// The product, or one band of it (band < 0: every chunk; otherwise the chunks, rows and split
// windows of that band of the schedule the launch selects - see b200spmm_plan::Sched).
int spmm_launch(b200spmm_plan_t *p, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                void *stream_v, int band) {
    if (!p || !d_B || !d_C || n <= 0 || ldb < n || ldc < n) return B200SPMM_ERR_INVALID_ARG;
    if (c_dtype != B200SPMM_C_F32 && c_dtype != B200SPMM_C_F16) return B200SPMM_ERR_INVALID_ARG;
    const int esz = p->info.elt_size, csz = c_dtype == B200SPMM_C_F32 ? 4 : 2;
    if (n % 8 || n > 0x7FFFFFFF || p->info.cols > 0x7FFFFFFFull) return B200SPMM_ERR_UNSUPPORTED;
    if ((reinterpret_cast<uintptr_t>(d_B) & 15u) || (reinterpret_cast<uintptr_t>(d_C) & 15u)) return B200SPMM_ERR_UNSUPPORTED;
    if ((ldb * esz) % 16 || (ldc * csz) % 16) return B200SPMM_ERR_UNSUPPORTED;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    B200_CUDA_TRY(make_current(p->device));
    p->last = b200spmm_launch_info_t{};
    if (p->info.eff_row_windows == 0) {  // nothing stored: C is all zeros
        B200_CUDA_TRY(cudaMemset2DAsync(d_C, (size_t)ldc * csz, 0, (size_t)n * csz, p->info.rows, stream));
        return B200SPMM_OK;
    }
    if (const uint32_t g = p->starve_gathers || band >= 0 ? 0u : narrow_group_blocks(p, n))
        return launch_narrow(p, g, d_B, ldb, n, d_C, ldc, c_dtype, stream);
    if (!p->starve_gathers && use_rows(p, ldb)) return launch_rows(p, d_B, ldb, n, d_C, ldc, c_dtype, stream, band);
    if (!p->has_tile_path) {  // only row units were kept; the starved test launch and a huge ldb ask for more
        int st = plan_add_tile_path(p, 0);
        if (st != B200SPMM_OK) return st;
    }
    TallChoice tall = band < 0 ? choose_tall(p, n) : TallChoice{};
    if (const uint32_t lines = tall.use || band >= 0 || p->starve_gathers ? 0u : choose_window_lines(p, ldb, n))
        return launch_windows(p, lines, d_B, ldb, n, d_C, ldc, c_dtype, stream);
    note_bounded_waits(p, stream);
    if (tall.parts > 1 && tall.use && take_scratch(p, &p->partial, tall.partial_bytes, stream) != B200SPMM_OK) {
        // no room for the parts' sums: whole windows where they are as exact, else the 16-row kernel
        tall.use = tall.least_parts <= 1;
        tall.parts = 1;
    }
    if (tall.use) return launch_tall(p, tall, d_B, ldb, n, d_C, ldc, c_dtype, stream);
    SpmmParams prm{};
    prm.rowOffset = p->d_rowOffset;
    prm.tcA2B = p->d_tcA2B;
    prm.rowIdx = p->d_rowIdx;
    const b200spmm_plan::Sched &sc = p->sched;
    p->launch_sched = &sc;
    prm.chunk_tile = sc.d_tile;
    prm.chunk_wfirst = sc.d_wfirst;
    prm.chunk_wlast = sc.d_wlast;
    prm.chunk_head_slot = sc.d_head_slot;
    prm.chunk_tail_slot = sc.d_tail_slot;
    if (band >= 0 && (size_t)band + 1 >= sc.band_chunk.size()) return B200SPMM_ERR_INVALID_ARG;
    prm.chunk_begin = band < 0 ? 0u : sc.band_chunk[band];
    prm.chunk_end = band < 0 ? sc.n_chunks : sc.band_chunk[band + 1];
    const uint32_t split_begin = band < 0 ? 0u : sc.band_split[band];
    const uint32_t split_end = band < 0 ? sc.n_splits : sc.band_split[band + 1];
    prm.sched_counter = sc.n_chunks > (uint32_t)sc.n_ctas ? p->d_status + 1 : nullptr;
    if (sc.n_slots) {  // slots for the pieces of windows that span chunks
        int st = take_scratch(p, &p->partial, (size_t)sc.n_slots * kRowWindow * (size_t)n * 4, stream);
        if (st != B200SPMM_OK) return st;
    }
    prm.partial = static_cast<float *>(p->partial.ptr);
    prm.tiles_image = static_cast<const uint8_t *>(p->d_tiles_image);
    prm.total_tiles = (uint32_t)p->info.total_tiles;
    prm.B = d_B;
    prm.C = d_C;
    prm.ldb = ldb;
    prm.ldc = ldc;
    prm.rows = (uint32_t)p->info.rows;
    prm.cols = (uint32_t)p->info.cols;
    prm.n = (uint32_t)n;
    prm.eff_row_windows = (uint32_t)p->info.eff_row_windows;
    prm.c_is_half = c_dtype == B200SPMM_C_F16;
    prm.status = p->d_status;
    prm.wait_limit_ns = p->wait_limit_ns;
#ifdef B200SPMM_PROFILE
    if (!g_prof) cudaMalloc(&g_prof, 1024 * 32 * 8);
    cudaMemsetAsync(g_prof, 0, 1024 * 32 * 8, stream);
    prm.prof = g_prof;
    if (const char *dbg = std::getenv("B200SPMM_DEBUG")) prm.debug = (uint32_t)std::atoi(dbg);  // results invalid
#endif
    int st = p->info.dtype == B200SPMM_F16 ? launch_dtype<false>(p, prm, stream) : launch_dtype<true>(p, prm, stream);
    if (st != B200SPMM_OK || split_end == split_begin) return st;
    // windows shared out over several CTAs: sum their pieces
    B200_CUDA_TRY(launch_after(spmm_fixup_kernel, dim3(split_end - split_begin), 256, 0, 1, stream, sc.d_splits + split_begin, sc.d_piece_slots,
                               (const float *)prm.partial, p->d_rowIdx, d_C, ldc, prm.rows, prm.n, prm.c_is_half));
    p->last.kernel_launches = 2;
    return B200SPMM_OK;
}

}  // namespace

extern "C" {

int b200spmm_spmm(b200spmm_plan_t *p, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                  void *stream_v) {
    return guarded([&]() { return spmm_launch(p, d_B, ldb, n, d_C, ldc, c_dtype, stream_v, -1); });
}

int b200spmm_fp16_spmm(b200spmm_plan_t *p, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                       void *stream) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    if (p->info.dtype != B200SPMM_F16) return B200SPMM_ERR_INVALID_ARG;
    return b200spmm_spmm(p, d_B, ldb, n, d_C, ldc, c_dtype, stream);
}

int b200spmm_tf32_spmm(b200spmm_plan_t *p, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                       void *stream) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    if (p->info.dtype != B200SPMM_TF32) return B200SPMM_ERR_INVALID_ARG;
    return b200spmm_spmm(p, d_B, ldb, n, d_C, ldc, c_dtype, stream);
}

int b200spmm_plan_sync(b200spmm_plan_t *p, void *stream_v) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    B200_CUDA_TRY(cudaSetDevice(p->device));
    B200_CUDA_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream_v)));
    using Unread = b200spmm_plan::Unread;
    if (p->unread == Unread::none) return B200SPMM_OK;  // (row units and the narrow kernel wait for nothing)
    uint32_t status = 0;
    B200_CUDA_TRY(cudaMemcpy(&status, p->d_status, sizeof(status), cudaMemcpyDeviceToHost));
    unsigned long long id = 0;
    if (p->unread == Unread::one_stream && cudaStreamGetId(static_cast<cudaStream_t>(stream_v), &id) == cudaSuccess && id == p->unread_stream)
        p->unread = Unread::none;  // what was launched there is done, and read
    if (status) {
        // status and the hand-out counters, cleared before the caller can launch again (on any stream)
        B200_CUDA_TRY(cudaMemset(p->d_status, 0, 4 * sizeof(uint32_t)));
        B200_CUDA_TRY(cudaStreamSynchronize(nullptr));
        return B200SPMM_ERR_DEVICE_TIMEOUT;
    }
    return B200SPMM_OK;
}

static int run_host(b200spmm_plan_t *p, const void *h_B, int64_t n, void *h_C, int c_dtype) {
    if (!p || !h_B || !h_C || n <= 0) return B200SPMM_ERR_INVALID_ARG;
    if (c_dtype != B200SPMM_C_F32 && c_dtype != B200SPMM_C_F16) return B200SPMM_ERR_INVALID_ARG;
    B200_CUDA_TRY(cudaSetDevice(p->device));
    const size_t b_bytes = (size_t)p->info.cols * n * p->info.elt_size;
    const size_t c_bytes = (size_t)p->info.rows * n * (c_dtype == B200SPMM_C_F32 ? 4 : 2);
    if (b_bytes > p->d_B_bytes) {
        p->d_B_bytes = 0;
        int st = grow_buffer(&p->d_B, b_bytes);
        if (st != B200SPMM_OK) return st;
        p->d_B_bytes = b_bytes;
    }
    if (c_bytes > p->d_C_bytes) {
        p->d_C_bytes = 0;
        int st = grow_buffer(&p->d_C, c_bytes);
        if (st != B200SPMM_OK) return st;
        p->d_C_bytes = c_bytes;
    }
    const bool rows = use_rows(p, n);
    std::vector<uint64_t> band_row;
    if (!narrow_group_blocks(p, n)) {
        if (rows) {
            const int st = build_band_units(&p->rows_fmt, p->info.dtype == B200SPMM_TF32);
            if (st != B200SPMM_OK) return st;
            if (p->rows_fmt.d_band_units)
                for (const RowBand &b : p->rows_fmt.bands) band_row.push_back(b.row);
        } else if (!choose_tall(p, n).use) {
            band_row = p->sched.band_row;
        }
    }
    const size_t bands = band_row.size() > 1 ? band_row.size() - 1 : 1;
    if (bands == 1 || p->info.eff_row_windows == 0) {
        B200_CUDA_TRY(cudaMemcpyAsync(p->d_B, h_B, b_bytes, cudaMemcpyHostToDevice, nullptr));
        int st = b200spmm_spmm(p, p->d_B, n, n, p->d_C, n, c_dtype, nullptr);
        if (st != B200SPMM_OK) return st;
        B200_CUDA_TRY(cudaMemcpyAsync(h_C, p->d_C, c_bytes, cudaMemcpyDeviceToHost, nullptr));
        return b200spmm_plan_sync(p, nullptr);
    }
    // Large matrix: band after band on the compute stream; as soon as a band is done its rows of C
    // leave on a second stream while the next band is computed.
    //
    // Every row of C needs all rows of B, so the two copies of a step cannot overlap - except by
    // features: with the features cut in two halves, the first half of C goes out while the second
    // half of B comes in, and the host link carries both directions at once for the middle third of
    // the step.  Each half is a product of its own (B and C as views with the full leading dimension).
    // The copy engines move a piece of a row at a time: 55 + 57 GB/s (in, out; 50 each way at once) for 256 bytes and whole
    // rows, 51 + 53 (36) for 128 and 40 + 43 (20) for 64.  Halves of H bytes take H / in + H / both + H / out against 2 H / in +
    // 2 H / out in one piece: 0.066 against 0.072 ns a byte for pieces of 128 bytes, 0.099 for 64.  So the line is at 128.
    const size_t esz = (size_t)p->info.elt_size, csz = c_dtype == B200SPMM_C_F32 ? 4 : 2;
    const int64_t n_first = n / 2;
    const bool halves = p->host_split && n % 16 == 0 && (size_t)n_first * esz >= 128;
    const int n_parts = halves ? 2 : 1;
    if (!p->copy_stream) B200_CUDA_TRY(cudaStreamCreateWithFlags(&p->copy_stream, cudaStreamNonBlocking));
    if (halves && !p->upload_stream) {
        B200_CUDA_TRY(cudaStreamCreateWithFlags(&p->upload_stream, cudaStreamNonBlocking));
        for (cudaEvent_t &e : p->half_up) B200_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    while (p->band_done.size() < bands * (size_t)n_parts) {
        cudaEvent_t e;
        B200_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        p->band_done.push_back(e);
    }
    const size_t b_pitch = (size_t)n * esz, c_pitch = (size_t)n * csz;
    if (!halves) {
        B200_CUDA_TRY(cudaMemcpyAsync(p->d_B, h_B, b_bytes, cudaMemcpyHostToDevice, nullptr));
    } else {  // first half on the compute stream, the second one behind it on a stream of its own
        B200_CUDA_TRY(cudaMemcpy2DAsync(p->d_B, b_pitch, h_B, b_pitch, (size_t)n_first * esz, (size_t)p->info.cols,
                                        cudaMemcpyHostToDevice, nullptr));
        B200_CUDA_TRY(cudaEventRecord(p->half_up[0], nullptr));
        B200_CUDA_TRY(cudaStreamWaitEvent(p->upload_stream, p->half_up[0], 0));
        B200_CUDA_TRY(cudaMemcpy2DAsync(static_cast<char *>(p->d_B) + (size_t)n_first * esz, b_pitch,
                                        static_cast<const char *>(h_B) + (size_t)n_first * esz, b_pitch,
                                        (size_t)(n - n_first) * esz, (size_t)p->info.cols, cudaMemcpyHostToDevice, p->upload_stream));
        B200_CUDA_TRY(cudaEventRecord(p->half_up[1], p->upload_stream));
    }
    int64_t launches = 0;
    for (int part = 0; part < n_parts; ++part) {
        const int64_t f0 = part == 0 ? 0 : n_first, nf = halves ? (part == 0 ? n_first : n - n_first) : n;
        if (part == 1) B200_CUDA_TRY(cudaStreamWaitEvent(nullptr, p->half_up[1], 0));
        const char *b_part = static_cast<const char *>(p->d_B) + (size_t)f0 * esz;
        char *c_part = static_cast<char *>(p->d_C) + (size_t)f0 * csz;
        for (size_t k = 0; k < bands; ++k) {
            int st = spmm_launch(p, b_part, n, nf, c_part, n, c_dtype, nullptr, (int)k);
            if (st != B200SPMM_OK) return st;
            launches += p->last.kernel_launches;
            cudaEvent_t done = p->band_done[(size_t)part * bands + k];
            B200_CUDA_TRY(cudaEventRecord(done, nullptr));
            B200_CUDA_TRY(cudaStreamWaitEvent(p->copy_stream, done, 0));
            const uint64_t r0 = band_row[k], r1 = band_row[k + 1];
            if (r1 == r0) continue;
            B200_CUDA_TRY(cudaMemcpy2DAsync(static_cast<char *>(h_C) + r0 * c_pitch + (size_t)f0 * csz, c_pitch, c_part + r0 * c_pitch,
                                            c_pitch, (size_t)nf * csz, r1 - r0, cudaMemcpyDeviceToHost, p->copy_stream));
        }
    }
    p->last.kernel_launches = launches;
    B200_CUDA_TRY(cudaStreamSynchronize(p->copy_stream));
    return b200spmm_plan_sync(p, nullptr);
}

int b200spmm_spmm_host(b200spmm_plan_t *p, const void *h_B, int64_t n, void *h_C, int c_dtype) {
    const int st = guarded([&]() { return run_host(p, h_B, n, h_C, c_dtype); });
    if (st != B200SPMM_OK && p) {  // copies may have been started: they must not outlive the call, nor the caller's buffers
        cudaStreamSynchronize(nullptr);
        if (p->upload_stream) cudaStreamSynchronize(p->upload_stream);
        if (p->copy_stream) cudaStreamSynchronize(p->copy_stream);
    }
    return st;
}

int b200spmm_bench(b200spmm_plan_t *p, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc, int c_dtype,
                   int warmup, int runs, void *stream_v, float *total_ms) {
    if (!p || !total_ms || warmup < 0 || runs < 1) return B200SPMM_ERR_INVALID_ARG;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    B200_CUDA_TRY(cudaSetDevice(p->device));
    for (int i = 0; i < warmup; ++i) {
        int st = b200spmm_spmm(p, d_B, ldb, n, d_C, ldc, c_dtype, stream_v);
        if (st != B200SPMM_OK) return st;
    }
    cudaEvent_t e0, e1;
    B200_CUDA_TRY(cudaEventCreate(&e0));
    B200_CUDA_TRY(cudaEventCreate(&e1));
    int st = B200SPMM_OK;
    cudaEventRecord(e0, stream);
    for (int i = 0; i < runs && st == B200SPMM_OK; ++i) st = b200spmm_spmm(p, d_B, ldb, n, d_C, ldc, c_dtype, stream_v);
    cudaEventRecord(e1, stream);
    if (st == B200SPMM_OK) st = b200spmm_plan_sync(p, stream_v);
    if (st == B200SPMM_OK && cudaEventElapsedTime(total_ms, e0, e1) != cudaSuccess) {
        record_cuda_error(cudaGetLastError(), "cudaEventElapsedTime");
        st = B200SPMM_ERR_CUDA;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return st;
}

/* Declared in b200_spmm_kat.h: the product launched so that its stage barriers can never complete. */
int b200spmm_kat_spmm_starved(b200spmm_plan_t *p, const void *d_B, int64_t ldb, int64_t n, void *d_C, int64_t ldc,
                              unsigned long long limit_ns, void *stream) {
    if (!p || limit_ns == 0 || limit_ns > kDeviceWaitLimitNs) return B200SPMM_ERR_INVALID_ARG;
    if (p->gather_cpasync || n * p->info.elt_size < 128) return B200SPMM_ERR_UNSUPPORTED;  // needs whole TMA boxes
    p->starve_gathers = true;
    p->wait_limit_ns = limit_ns;
    p->tmap_b_ptr = nullptr;  // a map encoded for a normal launch must not be reused, nor this one later
    const int st = guarded([&]() { return spmm_launch(p, d_B, ldb, n, d_C, ldc, B200SPMM_C_F32, stream, -1); });
    p->starve_gathers = false;
    p->wait_limit_ns = kDeviceWaitLimitNs;
    p->tmap_b_ptr = nullptr;
    return st;
}

/* Declared in b200_spmm_kat.h: a device without room for more scratch. */
int b200spmm_kat_scratch_limit(b200spmm_plan_t *p, uint64_t bytes) {
    if (!p) return B200SPMM_ERR_INVALID_ARG;
    p->scratch_limit = (size_t)bytes;
    return B200SPMM_OK;
}

int b200spmm_spmm_noalloc_status(int device, void *stream_v) {
    B200_CUDA_TRY(cudaSetDevice(device));
    uint32_t *scratch = nullptr;
    int st = noalloc_scratch_address(device, &scratch);
    if (st != B200SPMM_OK) return st;
    B200_CUDA_TRY(cudaStreamSynchronize(static_cast<cudaStream_t>(stream_v)));
    uint32_t status = 0;  // a copy into a stack word: nothing is allocated
    B200_CUDA_TRY(cudaMemcpy(&status, scratch + kNoAllocStatusWord, sizeof(status), cudaMemcpyDeviceToHost));
    return (status & kDevStatusTimeout) ? B200SPMM_ERR_DEVICE_TIMEOUT : B200SPMM_OK;
}

int b200spmm_spmm_noalloc(const b200spmm_btcf_info_t *info, const uint32_t *d_rowOffset, const uint32_t *d_tcA2B,
                          const void *d_data, const uint32_t *d_rowIdx, const void *d_B, int64_t ldb, int64_t n,
                          void *d_C, int64_t ldc, int c_dtype, int device, int n_ctas, void *stream_v) {
    if (!info || !d_rowOffset || !d_B || !d_C || n <= 0 || ldb < n || ldc < n) return B200SPMM_ERR_INVALID_ARG;
    if (info->total_tiles && (!d_tcA2B || !d_data || !d_rowIdx)) return B200SPMM_ERR_INVALID_ARG;
    if (c_dtype != B200SPMM_C_F32 && c_dtype != B200SPMM_C_F16) return B200SPMM_ERR_INVALID_ARG;
    if (info->dtype != B200SPMM_F16 && info->dtype != B200SPMM_TF32) return B200SPMM_ERR_INVALID_ARG;
    if (info->row_window != kRowWindow || info->col_window != (info->dtype == B200SPMM_F16 ? 16 : 8))
        return B200SPMM_ERR_UNSUPPORTED;
    if (n_ctas > kNoAllocMaxCtas) {
        set_last_error_static("b200spmm_spmm_noalloc: n_ctas exceeds the 1024 CTAs the built-in schedule table holds");
        return B200SPMM_ERR_UNSUPPORTED;
    }
    if (info->total_tiles * (uint64_t)kRowWindow >= 0x7FFFFFFFull || info->cols > 0x7FFFFFFFull || n > 0x7FFFFFFF || n % 8)
        return B200SPMM_ERR_UNSUPPORTED;
    const int esz = info->dtype == B200SPMM_F16 ? 2 : 4, csz = c_dtype == B200SPMM_C_F32 ? 4 : 2;
    if ((reinterpret_cast<uintptr_t>(d_B) & 15u) || (reinterpret_cast<uintptr_t>(d_C) & 15u) ||
        (reinterpret_cast<uintptr_t>(d_data) & 15u) || (reinterpret_cast<uintptr_t>(d_tcA2B) & 15u) ||
        (ldb * esz) % 16 || (ldc * csz) % 16)
        return B200SPMM_ERR_UNSUPPORTED;
    cudaStream_t stream = static_cast<cudaStream_t>(stream_v);
    B200_CUDA_TRY(cudaSetDevice(device));
    if (n_ctas <= 0) {
        B200_CUDA_TRY(cudaDeviceGetAttribute(&n_ctas, cudaDevAttrMultiProcessorCount, device));
        n_ctas *= kCtasPerSm;
        if (n_ctas > kNoAllocMaxCtas) n_ctas = kNoAllocMaxCtas;
    }
    if (info->eff_row_windows == 0) {  // nothing stored: C is all zeros
        B200_CUDA_TRY(cudaMemset2DAsync(d_C, (size_t)ldc * csz, 0, (size_t)n * csz, info->rows, stream));
        return B200SPMM_OK;
    }
    uint32_t *scratch = nullptr;
    int st = noalloc_scratch_address(device, &scratch);
    if (st != B200SPMM_OK) return st;

    b200spmm_plan tmp;  // lives on the stack; owns nothing
    static const bool cpasync = env_is("B200SPMM_GATHER", "cpasync");  // read once per process
    tmp.gather_cpasync = cpasync;
    tmp.info = *info;
    tmp.device = device;
    tmp.sched.n_ctas = n_ctas;  // the tables themselves are in the built-in array
    tmp.launch_sched = &tmp.sched;
    tmp.d_rowOffset = const_cast<uint32_t *>(d_rowOffset);
    tmp.d_tcA2B = const_cast<uint32_t *>(d_tcA2B);
    tmp.d_rowIdx = const_cast<uint32_t *>(d_rowIdx);
    tmp.d_data = const_cast<void *>(d_data);
    st = encode_tile_map(&tmp);
    if (st != B200SPMM_OK) return st;

    // The table and the status word keep the previous call's contents: both are rewritten here,
    // on the same stream, before the SpMM kernel reads them.
    noalloc_schedule_kernel<<<1, 256, 0, stream>>>(
        d_rowOffset, (uint32_t)info->eff_row_windows, n_ctas, scratch);
    B200_CUDA_TRY(cudaGetLastError());

    SpmmParams prm{};
    prm.rowOffset = d_rowOffset;
    prm.tcA2B = d_tcA2B;
    prm.rowIdx = d_rowIdx;
    prm.chunk_tile = scratch + kNoAllocTile;  // one chunk per CTA
    prm.chunk_wfirst = scratch + kNoAllocWfirst;
    prm.chunk_wlast = scratch + kNoAllocWlast;
    prm.chunk_head_slot = prm.chunk_tail_slot = nullptr;  // cuts lie on window boundaries: no shared windows
    prm.chunk_begin = 0;
    prm.chunk_end = (uint32_t)n_ctas;
    prm.sched_counter = nullptr;
    prm.partial = nullptr;
    prm.tiles_image = nullptr;  // the caller's tiles, as they are, through the tensor map
    prm.total_tiles = (uint32_t)info->total_tiles;
    prm.B = d_B;
    prm.C = d_C;
    prm.ldb = ldb;
    prm.ldc = ldc;
    prm.rows = (uint32_t)info->rows;
    prm.cols = (uint32_t)info->cols;
    prm.n = (uint32_t)n;
    prm.eff_row_windows = (uint32_t)info->eff_row_windows;
    prm.c_is_half = c_dtype == B200SPMM_C_F16;
    prm.status = scratch + kNoAllocStatusWord;
    prm.wait_limit_ns = kDeviceWaitLimitNs;
    return info->dtype == B200SPMM_F16 ? launch_dtype<false>(&tmp, prm, stream) : launch_dtype<true>(&tmp, prm, stream);
}

}  // extern "C"
