// kernels.h -- launch wrappers of the device code (host-callable).
#ifndef HBG_KERNELS_H
#define HBG_KERNELS_H

#include <cuda_runtime.h>
#include <stdint.h>

#include "hbg_internal.h"

namespace hbg {

struct WordFinderArgs {
    // resident database
    const uint8_t *db;            // letters, one sentinel between subjects
    const int64_t *db_off;        // start of subject i
    const int32_t *db_len;        // length of subject i
    const int32_t *order;         // scheduling order of subjects (longest first)
    int32_t n_subj;
    // batch
    const HbgGroup *groups;
    int32_t n_groups;
    const int32_t *group_list;    // groups this launch processes (one hit mode per launch)
    const uint32_t *cells;        // n_groups x HBG_CELL_STRIDE
    const uint16_t *entries;
    const uint32_t *pv;           // n_groups x HBG_PV_WORDS
    const uint8_t *letters;
    const int32_t *ctx_of;
    const HbgContext *contexts;
    const HbgQueryDesc *queries;
    int32_t window;
    // scheduling: tile t covers groups group_list[(t / tiles_per_group) * team
    // .. + team) (those below n_list) and scheduled subjects
    // [(t % tiles_per_group) * tile_subjects, + tile_subjects); warp w of a
    // CTA works on the tile's group w % team
    int32_t tile_subjects;
    int32_t tiles_per_group;
    int64_t n_tiles;
    int32_t team;                 // groups per tile: warps that share each subject, 1..warps per CTA
    int32_t n_list;               // groups in group_list
    unsigned int *tile_counter;   // zeroed before launch
    // outputs
    hbg_hsp *hsps;
    unsigned long long *hsp_count;  // zeroed before launch
    int64_t hsp_cap;
    unsigned long long *q_extended; // per batch query, zeroed
    unsigned long long *q_kept;     // per batch query, zeroed
    unsigned long long *g_hits;     // per group lookup hits, zeroed
    // global-memory diagonal tables (groups with placement 1): one slice of
    // gdiag_len entries per (block, warp); warps clear theirs
    uint32_t *gdiag;
    int32_t gdiag_len;
    // entries per warp of the 16-bit shared-memory tables (a multiple of 8)
    int32_t smem_diag;
};

// Shared memory the word-finder kernel needs for a CTA of `threads` threads.
size_t wordfinder_smem_bytes(int threads, int smem_diag, int team);
cudaError_t wordfinder_configure();
// mode: bit 0 = offset mode (else chunk mode); bit 1 = the groups keep
// their diagonal tables in global memory (kernel built to favour L1); the
// instantiation for tiles of several groups (team > 1) is chosen from
// WordFinderArgs::team / the team argument
cudaError_t wordfinder_occupancy(int mode, int threads, int smem_diag, int team, int *blocks_per_sm);
cudaError_t launch_wordfinder(const WordFinderArgs &a, int mode, int blocks, int threads,
                              cudaStream_t stream);

// The word finder with small diagonal cells in shared memory (bytefinder.cu):
// the scheduled subjects [sub_lo, sub_lo + n_subj), for the groups of
// group_list.
constexpr int kByteThreads = 768;     // largest CTA
constexpr int kByteMinWindow = 5;     // smallest and largest two-hit window
constexpr int kByteMaxWindow = 64;
constexpr int kByteWide = 1023;       // packed cells say no higher count: see the cells
constexpr int kByteMaxEntries = 1 << 22;   // entries of a group are fewer
struct ByteArgs {
    const uint8_t *db;
    const int64_t *db_off;
    const int32_t *db_len;
    const int32_t *order;
    int32_t sub_lo, n_subj;
    const HbgGroup *groups;
    const int32_t *group_list;
    const uint32_t *packed;       // n_groups x HBG_NUM_CELLS: first entry | min(count, kByteWide) << 22
    const uint32_t *cells;        // n_groups x HBG_CELL_STRIDE
    const uint16_t *entries;
    const uint32_t *pv;
    const uint8_t *letters;
    const int32_t *ctx_of;
    const HbgContext *contexts;
    const HbgQueryDesc *queries;
    int32_t window;
    int32_t table_len;            // cells per warp: diag_len, for 8-bit cells the longest group's byte_table_len
    int32_t n_list;
    int32_t chunk;                // subjects a warp takes at a time, 1..32
    unsigned long long *next;     // per group: subjects taken, zeroed before launch
    uint16_t *side;               // 8-bit cells: blocks x warps x table_len flag ends (need no clearing)
    hbg_hsp *hsps;
    unsigned long long *hsp_count;
    int64_t hsp_cap;
    unsigned long long *q_extended;
    unsigned long long *q_kept;
};
// length of an 8-bit table for a group of `letters` letters and gap
__host__ __device__ constexpr int byte_table_len(int letters) { return (letters + 127) / 128 * 128; }
size_t byte_smem_bytes(int cell_bytes, int threads, int table_len);
cudaError_t byte_configure();
// wide: the groups may have cells of kByteWide entries or more (8-bit cells: always allowed)
cudaError_t launch_byte(const ByteArgs &a, int cell_bytes, bool wide, int blocks, int threads, cudaStream_t stream);

// The lookup tables of a batch (tables.cu): from letters, contexts and queries
// to cells, presence vectors, packed cells, entries and per-query cell counts.
struct TableSegment {             // letters of one query, up to kTableSegment words
    int32_t group, query;         // of the batch
    int32_t begin, end;           // group-local offsets of its words
};
constexpr int kTableSegment = 512;
struct TableArgs {
    const HbgGroup *groups;
    const TableSegment *segs;     // in query order; a group's are seg_base ..
    int32_t first_group, first_seg;   // of the groups and segments built by this launch
    const uint8_t *letters;
    const int32_t *ctx_of;
    int32_t threshold;
    uint32_t *cells;
    uint32_t *packed;
    uint32_t *pv;
    uint16_t *entries;            // a group's start at its entry_base
    uint16_t *query_cells;
    uint32_t *counts;             // scratch: HBG_NUM_CELLS per segment of the launch
};
cudaError_t launch_tables(const TableArgs &a, int32_t n_groups, int32_t n_segs, cudaStream_t stream);
cudaError_t launch_pack_cells(const uint32_t *cells, int32_t n_groups, uint32_t *packed, cudaStream_t stream);

// Ordering pass: sort HSPs by (query, subject, subject offset, query offset),
// and count the lookup hits of every query.
constexpr int kOrderMaxGrid = 512;    // most CTAs of the pass
struct OrderArgs {
    const hbg_hsp *in;
    hbg_hsp *out;
    const unsigned long long *count;  // device count of HSPs (clamped to cap)
    int64_t cap;
    uint64_t *keys[2];
    uint32_t *vals[2];
    uint32_t *hist;                   // 256 x kOrderMaxGrid
    int bits_q, bits_s, bits_so, bits_qo;
    // optional (null = skip): per-query first / end index in `out` and the
    // number of subjects with HSPs, each n_queries entries, zeroed beforehand
    unsigned long long *q_first, *q_end, *q_passed;
    unsigned long long *barrier, *error;   // zeroed beforehand; *error: the grid barrier gave up
    // lookup_hits[q] = sum_w db_hist[w] * query_cells[q][w]
    const unsigned long long *db_hist;
    const uint16_t *query_cells;
    int32_t n_queries;
    unsigned long long *lookup_hits;
};
int order_grid(int device);
cudaError_t launch_order(const OrderArgs &a, int grid, cudaStream_t stream);

// Letters of subjects that lie back to back (subject i at [first[i],
// first[i + 1]) of the caller's numbering), `count` of them from letter `from`
// on, into the resident layout: one zero before every subject and after the
// last.  *bad = min(*bad, subject with a letter outside 1..27).
cudaError_t launch_spread_letters(const uint8_t *raw, int64_t from, int64_t count, const int64_t *first, int32_t n,
                                  uint8_t *out, int32_t *bad, cudaStream_t stream);

// Database word histogram: hist[w] += positions whose three letters are
// non-sentinel and form word w.
cudaError_t launch_db_histogram(const uint8_t *db, int64_t n, unsigned long long *hist,
                                cudaStream_t stream);

// Device bytes that one search of the batch with these options takes besides the
// database (cap 0: default capacity).  In api.cu; for the server.
int search_bytes(const hbg_db *db, const hbg_batch *b, const hbg_gpu_options *opt, int64_t cap, int64_t *bytes);

}  // namespace hbg

#endif
