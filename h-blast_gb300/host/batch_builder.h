// batch_builder.h -- host-side construction of a query batch: query packing
// into groups, six-frame translation for BLASTX, and the neighbourhood-word
// lookup tables.  Pure C++ (no CUDA); the runtime uploads the result.
#ifndef HBG_BATCH_BUILDER_H
#define HBG_BATCH_BUILDER_H

#include <stdint.h>

#include <string>
#include <vector>

#include "../csrc/hbg_internal.h"

namespace hbg {

// Shared-memory diagonal tables (16-bit cells) hold at most this many
// entries per warp; groups whose table is longer use 32-bit tables in the
// global scratch.  Measured on GB300: 2048-entry tables are faster in shared
// memory (four 8-warp CTAs per SM fit); longer shared tables cut resident
// warps to 8-20 per SM, and L2-resident global tables with 32 warps per SM
// beat them by 13-23 % (4096 to 32768 entries, BLASTP and six-frame BLASTX).
constexpr int32_t kSmemDiagMax = 2048;
// Default group length (letters, gaps included): 4056, the longest whose
// table has 4096 entries, which byte_kernel keeps in 16-bit cells with 22 warps
// per SM.  64 queries of 50..1500 letters against 500,000 subjects, word-finder
// ms by group length (and scans of the database): 1000 187 (52), 2008 167 (37),
// 4056 143 (16), 6000 146 (10), 8152 144 (7), 16,000 189 (4).  wordfinder_kernel
// has the same best range: 2,000,000 subjects, tables in global memory, 4056
// 862, 6000 858, with 15 times the DRAM writes above 4096 entries.
constexpr int32_t kDefaultGroupLen = 4056;
// Groups whose expected hits per subject offset reach this use offset mode
// (off by default: chunk mode at high occupancy measured faster; the autotuner
// and hbg_batch_set_mode choose offset mode explicitly).
constexpr double kOffsetModeHits = 1e30;
// Queries per group are bounded so per-query counters fit in shared memory.
constexpr int32_t kMaxQueriesPerGroup = 64;

struct HostBatch {
    int32_t threshold = 11;
    int32_t window = 40;
    std::vector<HbgGroup> groups;
    std::vector<HbgContext> contexts;
    std::vector<HbgQueryDesc> queries;
    struct Run {                         // letters of one context
        int32_t group, at, len;          // offset in the group
    };
    std::vector<Run> runs;               // by group, contexts that hold a word
    std::vector<uint8_t> letters;        // all groups, gaps included
    std::vector<int32_t> ctx_of;         // per letter, -1 outside contexts
    // lookup tables: empty until build_tables
    std::vector<uint32_t> cells;         // groups x HBG_CELL_STRIDE
    std::vector<uint16_t> entries;       // group-local query offsets
    std::vector<uint32_t> pv;            // groups x HBG_PV_WORDS
    std::vector<uint16_t> query_cells;   // queries x HBG_NUM_CELLS cell sizes
    int32_t max_query_len = 0;
    int32_t max_diag_len = 0;            // over groups with global placement
    int32_t smem_diag_len = 64;          // per-warp shared table: max over shared-placed groups
    double mode_hits = 0;                // offset-mode threshold
    bool counted = false;                // the groups' n_entries and max_cell are known
};

// One query already in NCBI concatenated form.
struct QueryIn {
    const uint8_t *seq;
    int32_t len;
    std::vector<int32_t> ctx_off, ctx_len, xdrop, cutoff;
};

// Packs the queries into groups; the lookup tables come later (build_tables).
// Returns an empty string on success, else the reason.
// max_group_len 0 = default; mode_hits < 0 = default offset-mode threshold,
// 0 = offset mode for every group, a huge value = chunk mode for every group.
std::string build_batch(const std::vector<QueryIn> &queries, int32_t threshold,
                        int32_t window, int32_t max_group_len, HostBatch *out,
                        double mode_hits = -1.0);

// The lookup tables of a batch on the host; searches build theirs on the device.
void build_tables(HostBatch *b);
// Lookup entries the tables hold, without building them; per group in n_entries,
// with a bound for its fullest cell in max_cell.
int64_t count_entries(HostBatch *b);

// Standard-code six-frame translation (frames +1,+2,+3,-1,-2,-3, one sentinel
// between frames).  Returns the concatenated letters; fills offsets/lengths.
std::vector<uint8_t> translate_six_frames(const uint8_t *nt, int32_t nt_len,
                                          std::vector<int32_t> *ctx_off,
                                          std::vector<int32_t> *ctx_len);

// SEG low-complexity masking of one protein sequence in place (masked
// letters become X); returns the number of letters masked.  seg.cpp.
int64_t seg_mask(uint8_t *seq, int32_t len, int32_t window, double locut, double hicut);

// Substitution score of NCBIstdaa letters (BLOSUM62).
int32_t blosum62(int32_t a, int32_t b);
const int8_t *blosum62_table();   // 28 rows x 32 columns, row = query letter

}  // namespace hbg

#endif
