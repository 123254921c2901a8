// The matrix of a plan as row units (see spmm_rows_kernel.cuh), built on the device from the condensed tiles.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>
#include <vector>

#include "../../include/b200_spmm.h"
#include "format.hpp"

namespace b200spmm {

// A unit is a row, or a piece of a long one.  Its entries lie in consecutive batches of four; the first batch is
// filled up with parts of the unit's first value (split_value in rows_gpu.cu).  A batch is kBatchWords 32-bit words: four columns, four
// values (fp16: two words, tf32: four, low 13 bits dropped), the target of the unit's sum in the unit's last
// batch and kNoTarget in the others, padding to 16 bytes.
constexpr uint32_t kMaxUnitEntries = 256;  // no unit is longer, see unit_entries_for
constexpr uint32_t kUnitBatch = 4;
template <bool kTf32>
constexpr uint32_t kBatchWords = kTf32 ? 12 : 8;
template <bool kTf32>
constexpr uint32_t kTargetWord = kTf32 ? 8 : 6;
constexpr uint32_t kLongUnits = 5;
constexpr uint32_t kSlotTarget = 0x80000000u, kNoTarget = 0xFFFFFFFFu;  // a row, or kSlotTarget | slot of a piece

// A row that was cut: its pieces lie in slots [slot_begin, slot_end), in entry order.
struct RowSplit {
    uint32_t row, slot_begin, slot_end;
};

// A band of whole rows: where in the list of the bands its units (longest first) and its rows without entries (behind
// the units of all bands) begin, its cut rows and its rows.
struct RowBand {
    uint32_t unit, empty, split;
    uint64_t row;
};

struct RowsFormat {
    uint32_t *d_batches = nullptr;    // [n_batches + 1][kBatchWords], the last one belongs to nobody
    uint2 *d_units = nullptr;         // [n_units] first batch and number of batches, longest first, then (row, 0) for rows without entries
    uint2 *d_band_units = nullptr;    // the same band by band, once build_band_units has run
    RowSplit *d_splits = nullptr;     // [n_splits] by row
    uint64_t nnz = 0;
    uint32_t n_batches = 0, n_units = 0, n_splits = 0, n_slots = 0;
    uint32_t most_batches = 0;             // of a unit
    uint32_t long_units[kLongUnits] = {};  // units of at least 2 << i batches
    std::vector<RowBand> bands;       // one more than there are bands: the last one holds the totals
};

// The same entries for narrow B (see spmm_narrow_kernel.cuh): row after row, and inside a row column block after
// column block of kNarrowCols columns.  fp16: (value << 16) | low half of the column; tf32: (column, value bits).
constexpr uint32_t kNarrowCols = 2048;
struct NarrowFormat {
    uint32_t *d_entries = nullptr;    // [nnz] words (fp16) or pairs of words (tf32)
    uint32_t *d_seg = nullptr;        // [rows][n_blocks + 1] first entry of every (row, block), and the row's end
    uint32_t *d_cut = nullptr;        // [n_ctas + 1] rows of every CTA
    uint32_t n_blocks = 0, n_ctas = 0, max_rows = 0;  // max_rows: of one CTA
};

// What a look over the tables of a caller's format finds (tables_kernel in capi.cu).
namespace formatcheck {

enum : uint32_t { kBadTables = 1u, kLooseLists = 2u };

struct Found {
    uint32_t flags;
    int32_t falls;  // places where a column is not above the one before it, less those where a window starts
    __host__ __device__ bool bad() const { return (flags & kBadTables) != 0; }
    __host__ __device__ bool loose() const { return flags || falls; }
};

}  // namespace formatcheck

// Builds what the kernels outside the tile path want from a matrix: row units when `force_rows` or when at most
// max_fill of the tiles' slots are in use, and the format for narrow B where it fits (at most 65,536 columns, rows
// of some length, none so long that CTAs of whole rows could not be balanced).  The tiles must be in the reference's layout
// (row-major 16 x CW).  `found`: of the tables; loose: slots without a column may lie anywhere in a window, and not only in its last
// tile.  While a look over them is still under way it writes d_found, and *found is set from that unless *found_known says that it
// already is: on return it does, if the host had to wait for the device.  Nothing is built from bad tables.  A format stays empty
// when device memory is short.
int build_row_formats(const b200spmm_btcf_info_t &info, const uint32_t *d_rowOffset, const uint32_t *d_tcA2B,
                      const void *d_data, const uint32_t *d_rowIdx, const formatcheck::Found *d_found, formatcheck::Found *found, bool *found_known,
                      int n_sms, double max_fill, bool force_rows, RowsFormat *rows, NarrowFormat *narrow);
// The list of the bands, where there are several and no list yet: only calls that copy C out band by band need it, and it is 8
// bytes a row.  Waits for the device.  Stays empty when device memory is short; then everything is one band.
int build_band_units(RowsFormat *f, bool tf32);
void free_rows(RowsFormat *r);
void free_narrow(NarrowFormat *f);

}  // namespace b200spmm
