// 256-row super-windows in the 2:4 form of the tensor core, built on the device from the dense ones (sparse24_gpu.cu).
#pragma once

#include <cstdint>

#include "tall_gpu.hpp"

namespace b200spmm {

// Tiles of 256 rows x 32 columns of which every row keeps two in each group of four: sixteen fp16 values a row, and four bits
// a group that say which two.  What a row has beyond that is its rest: (column << 16) | value bits, in order of columns.
// The windows are those of the dense format, whose d_rowIdx goes with these arrays.
struct Sparse24Format {
    uint64_t tiles = 0;               // 0: there is none
    uint32_t *d_rowOffset = nullptr;  // [eff + 1] tiles
    uint32_t *d_quads = nullptr;      // [eff + 1] quads of tiles (a window's last one may be short)
    uint32_t *d_tcA2B = nullptr;      // [tiles * 32] columns, as the dense list has them; kIdxMax past its end
    void *d_data = nullptr;           // (owns all) per window the images of rows 0-127 of all its tiles (4 KB each: TallFormat::d_data), then of rows 128-255
    void *d_meta = nullptr;           // per window 2 KB for every quad and half, as tcgen05.cp takes them to tensor memory: 128 lanes x 4 words
    uint32_t *d_n_rest = nullptr;     // [eff * 256]
    uint32_t *d_rest = nullptr;       // [eff][kSparse24MaxRest][256]
};
constexpr uint32_t kSparse24MaxRest = 48;  // of a row

// Leaves *out empty where the form does not fit, rows have more in their rest than pays (unless `always`), or device memory is
// short.  fp16, at most 65,536 columns.
int build_sparse24(const TallFormat &pair, uint64_t cols, bool always, Sparse24Format *out);
void free_sparse24(Sparse24Format *f);

}  // namespace b200spmm
