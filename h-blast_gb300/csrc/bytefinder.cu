// bytefinder.cu -- the word finder with its diagonal tables in shared memory:
// one warp per (query group, subject), hits applied 32 at a time.
//
// Subject letters are staged by cp.async and words filtered by a presence
// vector in shared memory as in wordfinder.cu; the cells are smaller and the
// per-hit rule is cut to what the common cases need:
//
//   A cell holds the position of its diagonal's last hit, position = subject
//   offset + rel, where rel moves up by subject length + window from subject
//   to subject (NCBI's diagonal offset), or a special value above every
//   position.  One subtraction diff = position - cell sorts a hit: diff >=
//   window: no recent hit, the cell takes the position; 0..2: overlaps the
//   last hit, passed; 3..window-1: second hit, an extension is queued and the
//   cell marked pending; negative: the cell is special.
//
//   16-bit cells: positions to 0x7ffe, 0x8000 | end for a diagonal flagged up
//   to position `end` (NCBI's DiagStruct flag), 0xffff pending.  The table is
//   cleared when a subject's positions would not fit.
//
//   8-bit cells (for longer tables, whose length is then exact instead of a
//   power of two): positions to 247; 248..254 a flag of the subject with that
//   number modulo 7, its end in a side table in global memory; 255 pending.
//   Every ~200 letters `sweep` moves the base up.
//
// The rules are NCBI aa_ungapped.c's two-hit state machine (H-BLAST
// h_blast_kernel.cu:672-871); the extension is in extend.h.
//
// What bounds it: issued instructions (3.0 of 4 per cycle); 24 warps of 80
// registers (32 of 64 spill: 2 % faster for one 350-letter query against 400,000
// subjects, 20 % slower against 20,000, where a warp's latency counts).  One 4056-letter
// query against 400,000 subjects (1.22e9 hits): 8.9 ms, 1.37e11 hits/s, 13.9 ms
// with wordfinder_kernel; of 223 warp instructions per batch of 32 hits the
// extensions take 93 (75 of them the walks), shared diagonals 22, scanning,
// locating and the common case 107.  DRAM traffic is the subject letters once per group.
#include <cuda_runtime.h>
#include <stddef.h>

#include "extend.h"
#include "kernels.h"

namespace hbg {

namespace {

constexpr int kMaxQ = 64;             // kMaxQueriesPerGroup
constexpr unsigned kAll = 0xffffffffu;

__constant__ int8_t c_blosum[28 * 32] = {
#include "blosum62.inc"
};

template <typename Cell>
struct Cells;
template <>
struct Cells<uint16_t> {
    static constexpr int kPending = 0xffff, kFlag = 0x8000, kMaxPos = 0x7ffe;
};
template <>
struct Cells<uint8_t> {
    static constexpr int kPending = 255, kFlag = 248, kMaxPos = 247;
};

constexpr int kFlushAt = 32;       // queued extensions that start a round
constexpr int kQueue = 64;
constexpr int kStageBlock = 64;    // staged letters per block: 16 bytes for each of lanes 0..3
constexpr int kStageRing = 4;      // blocks held: the scan's two, and two in flight
constexpr int kStageLanes = kStageBlock / 16;

struct WarpMem {
    uint4 stage[kStageRing * kStageBlock / 16];   // ring of subject letters
    uint2 list[32];          // the chunk's non-empty offsets: offset, entry index minus stream position
    uint2 task[kQueue];      // queued extensions: subject offset | query offset << 16, distance to the first hit
    uint32_t chain[32];      // lanes that share lane k's diagonal; zero between batches
    uint32_t blk[2 * kQueue]; // two lists of hits behind a queued extension: subject offset | query offset << 16
};

struct __align__(16) Head {
    Score matrix[28 * 32];   // scaled BLOSUM62, query letter x 32 + subject letter
    uint32_t pv[HBG_PV_WORDS];
    unsigned int q_ext[kMaxQ];
    unsigned int q_kept[kMaxQ];
    int go;                  // place in turn of the next group to search
    int pad[3];
};
static_assert(sizeof(Head) % 16 == 0 && sizeof(WarpMem) % 16 == 0, "16-byte shared-memory regions");

extern __shared__ __align__(16) unsigned char g_byte_smem[];

template <typename Cell>
struct Item {
    const uint8_t *s;        // subject letters
    int S, j;                // its length and ordinal id
    unsigned tab, mem;       // shared-memory offsets of the warp's cells and WarpMem
    unsigned len;            // table length: a power of two for 16-bit cells, exact for 8-bit ones
    unsigned span;           // window - 3
    int rel;                 // position of subject offset 0
    int code;                // 8-bit cells: flag code of this subject
    uint16_t *side;          // 8-bit cells: flag ends (subject offsets)
    const uint8_t *gseq;
    const int32_t *gctx;
    int first_query;
};

struct Queues {
    int n_tasks, n_blk, blk_cur;   // blk_cur: 0 or kQueue, the first entry of the list in use
};

// Shared memory by its byte offset from g_byte_smem: the compiler then forms
// 32-bit addresses.
template <typename T>
__device__ __forceinline__ T &smem_at(unsigned off) {
    return *reinterpret_cast<T *>(g_byte_smem + off);
}
__device__ __forceinline__ unsigned smem_address(unsigned off) {
    return (unsigned)__cvta_generic_to_shared(g_byte_smem) + off;
}

template <typename Cell>
__device__ __forceinline__ bool is_flag(int v) {
    return (unsigned)(v - Cells<Cell>::kFlag) < (unsigned)(Cells<Cell>::kPending - Cells<Cell>::kFlag);
}

// A hit's place in the subject as the batches carry it: the offset, for 8-bit
// cells with the offset modulo the table length in the upper half.  The cell of
// query offset q is (q - offset) modulo the table length.
template <typename Cell>
__device__ __forceinline__ int offset_of(unsigned place) {
    return (int)(sizeof(Cell) == 1 ? place & 0xffffu : place);
}
template <typename Cell>
__device__ __forceinline__ unsigned place_of(const Item<Cell> &it, int s_h) {
    return sizeof(Cell) == 1 ? (unsigned)s_h | (((unsigned)s_h % it.len) << 16) : (unsigned)s_h;
}
template <typename Cell>
__device__ __forceinline__ unsigned cell_of(const Item<Cell> &it, unsigned place, int q) {
    if (sizeof(Cell) == 2)
        return ((unsigned)q - place) & (it.len - 1u);
    const unsigned d = (unsigned)q - (place >> 16);
    return min(d, d + it.len);
}

// The general case of apply_hits: chains of lanes that share a diagonal, and
// special states.  A chain's state goes from lane to lane, in order, by
// shuffles, and its last lane writes the cell.  Chains are found through the
// cells: every lane writes its number and reads back whose number stayed; who
// reads another's says so in that lane's word of `chain`.  Warp-collective.
template <typename Cell>
__device__ __forceinline__ void apply_chains(const Item<Cell> &it, Queues &W, bool act, unsigned d, int s_h, int q, int v, int &nv,
                                             int &diff, bool &trig) {
    using K = Cells<Cell>;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int pos = s_h + it.rel;
    Cell &cell = smem_at<Cell>(it.tab + d * (unsigned)sizeof(Cell));
    if (act)
        cell = (Cell)lane;
    __syncwarp();
    const int t = act ? (int)cell : lane;
    bool over = false, blk = v == K::kPending;
    if (__any_sync(kAll, is_flag<Cell>(v))) {
        // a flagged diagonal: a hit before the flag's end changes nothing, one
        // at or beyond it finds no recent hit (state 0)
        if (is_flag<Cell>(v)) {
            if (sizeof(Cell) == 2)
                over = pos >= (v & (K::kFlag - 1));
            else
                over = v != it.code || s_h >= (int)it.side[d];
            nv = over ? pos : nv;
        }
    }
    const unsigned mine = smem_address(it.mem + (unsigned)offsetof(WarpMem, chain)) + 4u * (unsigned)t;
    unsigned m;
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %1, %2; @p red.shared.or.b32 [%0], %3; }" ::"r"(mine), "r"(t), "r"(lane),
                 "r"(lt + 1u)
                 : "memory");
    __syncwarp();
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(m) : "r"(mine) : "memory");
    __syncwarp();
    asm volatile("{ .reg .pred p; setp.ne.s32 p, %1, %2; @p st.shared.u32 [%0], %3; }" ::"r"(mine), "r"(t), "r"(lane), "r"(0)
                 : "memory");
    m |= 1u << t;                            // lanes of this diagonal
    const unsigned below = m & lt;
    const int rank = __popc(below), prev = 31 - __clz(below);
    for (int r = 1; __any_sync(kAll, rank >= r); ++r) {
        const int x = __shfl_sync(kAll, nv, prev);
        if (rank == r) {
            const int ps = over && is_flag<Cell>(x) ? 0 : x;
            diff = pos - ps;
            trig = (unsigned)(diff - 3) < it.span;
            nv = diff >= (int)it.span + 3 ? pos : ps;
            nv = trig ? K::kPending : nv;
            blk = x == K::kPending;
        }
    }
    if (act && (m & ~(2u * lt + 1u)) == 0)   // none above
        cell = (Cell)nv;
    blk = blk && act;
    const unsigned bm = __ballot_sync(kAll, blk);
    if (blk)
        smem_at<uint32_t>(it.mem + (unsigned)offsetof(WarpMem, blk) + 4u * (unsigned)(W.blk_cur + W.n_blk + __popc(bm & lt))) =
            (unsigned)s_h | ((unsigned)q << 16);
    W.n_blk += __popc(bm);
}

// Apply one batch of hits, one per active lane, in CPU order by lane.
//
// Every lane reads its cell, writes its position and reads the cell again: who
// then finds another position shares its diagonal with that lane.  (match.any
// finds this in one instruction, but took 30 cycles of the SM per batch, 30 %
// of the kernel on a 4056-letter group.)  95 % of the batches have lanes that
// share one, nearly always hits of consecutive offsets, and then each lane's
// outcome from the old state alone is right:
//   both less than 3 after the last hit: the cell stays;
//   both without a recent hit: the earlier one's position is the new state
// (the later one overlaps it).  Other batches -- a lane that shares its
// diagonal triggers an extension or is further off, or a cell holds a special
// state -- go through apply_chains.  Full: every lane is active.
// Warp-collective.
template <bool Full, typename Cell>
__device__ __forceinline__ void apply_hits(const Item<Cell> &it, Queues &W, bool act, unsigned place, int q) {
    using K = Cells<Cell>;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const int s_h = offset_of<Cell>(place);
    const unsigned d = cell_of(it, place, q);
    const int pos = s_h + it.rel;
    Cell &cell = smem_at<Cell>(it.tab + d * (unsigned)sizeof(Cell));
    int v = 0, t = pos;
    if (Full || act)
        v = cell;
    __syncwarp();
    if (Full || act)
        cell = (Cell)pos;
    __syncwarp();
    if (Full || act)
        t = cell;
    // diff >= window: no recent hit; 3..window-1: second hit; 0..2: overlap;
    // negative: a special state, which stays
    int diff = pos - v;
    bool trig = (unsigned)(diff - 3) < it.span;
    const bool reset = diff >= (int)it.span + 3;
    int nv = reset ? pos : v;
    nv = trig ? K::kPending : nv;
    const bool shared = t != pos;
    const bool hard = v >= K::kFlag ||
                      (shared && ((unsigned)(t - pos + 1) > 2u || trig || (unsigned)(t - v - 3) < it.span));
    bool store = (Full || act) && (shared ? reset && pos < t : nv != pos);
    if (__any_sync(kAll, hard)) {
        apply_chains(it, W, Full || act, d, s_h, q, v, nv, diff, trig);
        store = false;
    }
    if (store)
        cell = (Cell)nv;
    trig = (Full || act) && trig;
    const unsigned tm = __ballot_sync(kAll, trig);
    if (trig)
        smem_at<uint2>(it.mem + (unsigned)offsetof(WarpMem, task) + 8u * (unsigned)(W.n_tasks + __popc(tm & lt))) =
            make_uint2((unsigned)s_h | ((unsigned)q << 16), (unsigned)diff);
    W.n_tasks += __popc(tm);
    __syncwarp();
}

// One round: run queued extensions, a lane each (the newest 32 when more
// wait), then replay the blocked hits in order; with drain, until
// none is left.  A diagonal has at most one queued extension and extensions of
// different diagonals are independent, so any subset may run first; a replay
// batch starts only while at most 32 extensions wait, so the queue's 64 places
// suffice.  Warp-collective.
template <typename Cell>
__device__ __noinline__ Queues flush(const Item<Cell> it, const ByteArgs &a, Queues W, bool drain) {
    WarpMem &wm = smem_at<WarpMem>(it.mem);
    using K = Cells<Cell>;
    Head &hd = *reinterpret_cast<Head *>(g_byte_smem);
    const int lane = threadIdx.x & 31;
    const Letters subject = letters_of(it.s), group = letters_of(it.gseq);
    do {
        const int first = (!drain && W.n_tasks > 32) ? W.n_tasks - 32 : 0;
        for (int t0 = first; t0 < W.n_tasks; t0 += 32) {
            const int i = t0 + lane;
            if (i < W.n_tasks) {
                const uint2 task = wm.task[i];
                const int s_h = (int)(task.x & 0xffffu), q = (int)(task.x >> 16);
                const int ci = __ldg(it.gctx + q);
                const HbgContext C = a.contexts[ci];
                const HbgQueryDesc Q = a.queries[C.query];
                const int ql = q - Q.start;
                const Ext e = extend_two_hit(hd.matrix, subject, it.S, group, Q.start, Q.len, s_h - (int)task.y + 3, s_h, ql,
                                             C.x_dropoff);
                atomicAdd(&hd.q_ext[C.query - it.first_query], 1u);
                if (e.score >= C.cutoff) {
                    atomicAdd(&hd.q_kept[C.query - it.first_query], 1u);
                    const unsigned long long o = atomicAdd(a.hsp_count, 1ull);
                    if ((long long)o < a.hsp_cap) {
                        hbg_hsp out;
                        out.query = C.query;
                        out.subject = it.j;
                        out.q_start = e.q_start;
                        out.s_start = e.s_start;
                        out.q_off = ql;
                        out.s_off = s_h;
                        out.len = e.len;
                        out.score = e.score;
                        out.context = C.local;
                        a.hsps[o] = out;
                    }
                }
                const unsigned d = cell_of(it, place_of(it, s_h), q);
                int v = s_h + it.rel;
                if (e.right) {
                    const int end = e.s_last_off - 2;      // hits before it are passed
                    if (end <= s_h + 1) {
                        v = 0;                             // none is: later hits are at s_h + 1 or beyond
                    } else if (sizeof(Cell) == 2) {
                        v = K::kFlag | (end + it.rel);
                    } else {
                        v = it.code;
                        it.side[d] = (uint16_t)end;
                    }
                }
                smem_at<Cell>(it.tab + d * (unsigned)sizeof(Cell)) = (Cell)v;
            }
        }
        __syncwarp();
        W.n_tasks = first;
        const int nb = W.n_blk, src = W.blk_cur;
        W.n_blk = 0;
        W.blk_cur ^= kQueue;
        for (int b0 = 0; b0 < nb; b0 += 32) {
            if (W.n_tasks > 32) {
                // the rest of the list follows the re-blocked hits, in order
                for (int i = b0 + lane; i < nb; i += 32)
                    wm.blk[W.blk_cur + W.n_blk + i - b0] = wm.blk[src + i];
                W.n_blk += nb - b0;
                __syncwarp();
                break;
            }
            const bool act = b0 + lane < nb;
            const uint32_t rec = act ? wm.blk[src + b0 + lane] : 0u;
            apply_hits<false>(it, W, act, place_of(it, (int)(rec & 0xffffu)), (int)(rec >> 16));
        }
    } while (drain && (W.n_tasks > 0 || W.n_blk > 0));
    return W;
}

// 8-bit cells: move the base up by r, so that positions stay below the special
// values; cells that are `window` or more behind the scan become 0, which
// still reads as "no recent hit".  Flags of earlier subjects go, flags of the
// current one stay.  Nothing is pending.
__device__ __forceinline__ void sweep(unsigned tab, int len, int r, int code) {
    using K = Cells<uint8_t>;
    const int lane = threadIdx.x & 31;
    __syncwarp();
    const unsigned mr = ((unsigned)(-r) & 0xffffu) * 0x10001u;
#pragma unroll 4
    for (unsigned p = tab + 4u * lane; p < tab + (unsigned)len; p += 128) {
        const uint32_t v = smem_at<uint32_t>(p);
        const uint32_t lo = v & 0x00ff00ffu, hi = (v >> 8) & 0x00ff00ffu;
        uint32_t n = __viaddmax_s16x2(lo, mr, 0u) | (__viaddmax_s16x2(hi, mr, 0u) << 8);
        if ((((lo + 0x00080008u) | (hi + 0x00080008u)) & 0x01000100u) != 0u) {
            n = 0;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int c = (int)((v >> (8 * b)) & 255u);
                const int x = c >= K::kFlag ? (c == code ? c : 0) : max(c - r, 0);
                n |= (uint32_t)x << (8 * b);
            }
        }
        smem_at<uint32_t>(p) = n;
    }
    __syncwarp();
}

// Subject letters staged for the scan: blocks of kStageBlock letters counted
// from the 16-byte aligned address at or before the subject's first letter,
// block k in ring slot k % kStageRing; blocks next and next + 1 are issued.
// Issue block k: lanes 0..kStageLanes-1 copy 16 bytes each when they hold a
// letter of the subject (the copy then ends at most 15 bytes past it, inside
// the database buffer), else zero-fill.  Every lane commits one copy group.
__device__ __forceinline__ void stage_issue(WarpMem &wm, const uint8_t *s, int S, int k, int lane) {
    const uintptr_t sa = reinterpret_cast<uintptr_t>(s);
    const int delta = (int)(sa & 15);
    const int r = k * kStageBlock + lane * 16;
    if (lane < kStageLanes) {
        const bool in = r < delta + S;
        const uint8_t *src = reinterpret_cast<const uint8_t *>(sa & ~(uintptr_t)15) + (in ? r : 0);
        const unsigned dst = (unsigned)__cvta_generic_to_shared(&wm.stage[(k & (kStageRing - 1)) * kStageLanes + lane]);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(in ? 16 : 0)
                     : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Cell of the word at offset s0 + lane, 0 when it is empty: first entry |
// count << 22, counts of kByteWide and more as that.  Blocks up to the chunk's last letter are made resident first:
// for each newly needed block b, wait for its copy (all but the newest group)
// and issue b + 2 into the slot of b - 2, which no chunk needs any more.
// Warp-collective.
__device__ __forceinline__ uint32_t scan_words(const uint8_t *s, int S, int &next, WarpMem &wm, const uint32_t *pv,
                                               const uint32_t *packed, int s0) {
    const int lane = threadIdx.x & 31;
    const int delta = (int)(reinterpret_cast<uintptr_t>(s) & 15);
    const int blk = (delta + s0 + 33) / kStageBlock;
    while (next <= blk) {
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncwarp();
        stage_issue(wm, s, S, next + 2, lane);
        next++;
    }
    const uint8_t *ring = reinterpret_cast<const uint8_t *>(wm.stage);
    constexpr int kMask = kStageRing * kStageBlock - 1;
    const int sp = s0 + lane;
    const int r = delta + sp;
    if (sp > S - 3)
        return 0u;
    const uint32_t w = ((uint32_t)ring[r & kMask] << 10) | ((uint32_t)ring[(r + 1) & kMask] << 5) |
                       (uint32_t)ring[(r + 2) & kMask];
    return ((pv[w >> 5] >> (w & 31)) & 1u) ? __ldg(packed + w) : 0u;
}

// Entries of the word at s when its packed cell says kByteWide or more.
__device__ __noinline__ uint32_t wide_count(const uint8_t *s, const uint32_t *packed, const ByteArgs &a) {
    const unsigned w = ((unsigned)s[0] << 10) | ((unsigned)s[1] << 5) | s[2];
    const uint32_t *cs = a.cells + (size_t)((packed - a.packed) / HBG_NUM_CELLS) * HBG_CELL_STRIDE + w;
    return __ldg(cs + 1) - __ldg(cs);
}

// One (group, subject) item: scanned 32 offsets at a time; the subject's hit
// stream (CPU order) is applied 32 hits at a time across chunk boundaries.  A
// chunk's last, partial batch waits in lanes 0..carry-1 for the next chunk's
// first hits.  Warp-collective.
template <typename Cell, bool Wide>
__device__ __forceinline__ void process_item(Item<Cell> &it, const ByteArgs &a, const uint32_t *pv, const uint32_t *packed,
                                             const uint16_t *ents) {
    using K = Cells<Cell>;
    const int lane = threadIdx.x & 31;
    const unsigned le = 0xffffffffu >> (31 - lane);
    WarpMem &wm = smem_at<WarpMem>(it.mem);
    const unsigned list = it.mem + (unsigned)offsetof(WarpMem, list);
    Queues W{0, 0, 0};
    stage_issue(wm, it.s, it.S, 0, lane);
    stage_issue(wm, it.s, it.S, 1, lane);
    int next = 0;
    uint32_t carry = 0;        // hits of earlier chunks not applied yet, in lanes 0..carry-1
    unsigned s_n = 0;          // this lane's next hit
    int q_n = 0;
    unsigned s_mod = 0;        // 8-bit cells: s0 modulo the table length
    // the next chunk's cells are loaded while this chunk's hits are applied,
    // and each batch's query offsets while the previous batch is applied
    uint32_t cell_next = it.S >= 3 ? scan_words(it.s, it.S, next, wm, pv, packed, 0) : 0u;
    for (int s0 = 0; s0 <= it.S - 3; s0 += 32) {
        if (sizeof(Cell) == 1 && s0 + 31 + it.rel > K::kMaxPos) {
            // positions run out: apply what waits, then move the base
            if (carry > 0) {
                apply_hits<false>(it, W, (uint32_t)lane < carry, s_n, q_n);
                carry = 0;
            }
            if (W.n_tasks > 0 || W.n_blk > 0)
                W = flush(it, a, W, true);
            const int r = s0 + it.rel - (int)it.span - 3;
            sweep(it.tab, it.len, r, it.code);
            it.rel -= r;
        }
        unsigned place = (unsigned)(s0 + lane);
        if (sizeof(Cell) == 1) {
            const unsigned m = s_mod + lane;
            place |= (m >= it.len ? m - it.len : m) << 16;
            s_mod = s_mod + 32 >= it.len ? s_mod + 32 - it.len : s_mod + 32;
        }
        const uint32_t cell = cell_next;
        if (s0 + 32 <= it.S - 3)
            cell_next = scan_words(it.s, it.S, next, wm, pv, packed, s0 + 32);
        uint32_t c = cell >> 22;
        if (Wide && c == (uint32_t)kByteWide)
            c = wide_count(it.s + s0 + lane, packed, a);
        const unsigned nz = __ballot_sync(kAll, c != 0);
        if (nz == 0)
            continue;
        uint32_t incl = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t t = __shfl_up_sync(kAll, incl, o);
            if (lane >= o)
                incl += t;
        }
        // hit stream: position p of this chunk's hits starts at carry
        const uint32_t total = carry + __shfl_sync(kAll, incl, 31);
        uint32_t start = carry + incl - c;
        __syncwarp();              // the previous chunk's list has been read
        if (c != 0)
            smem_at<uint2>(list + 8u * (unsigned)__popc(nz & (le >> 1))) =
                make_uint2(place, (cell & 0x3fffffu) - start);
        else
            start = 0x80000000u;   // starts nothing
        __syncwarp();
        // the hits of stream positions cb + lane: the list entry is the last
        // that starts at or before the position
        unsigned before = list - 8u;   // entry that starts last before the batch
        auto starts = [&](uint32_t cb) {
            uint32_t bit;              // 0 for shifts of 32 or more
            asm("shl.b32 %0, 1, %1;" : "=r"(bit) : "r"(start - cb));
            return __reduce_or_sync(kAll, bit);
        };
        {
            const unsigned m = starts(0);
            if ((uint32_t)lane >= carry && (uint32_t)lane < total) {
                const uint2 e = smem_at<uint2>(before + 8u * (unsigned)__popc(m & le));
                s_n = e.x;
                q_n = (int)__ldg(ents + (e.y + lane));
            }
            before += 8u * (unsigned)__popc(m);
        }
        uint32_t cb = 0;
        for (; cb + 32 <= total; cb += 32) {       // full batches
            const unsigned at = s_n;
            const int q = q_n;
            {
                // lanes past the last hit read entries past its cell (the
                // entries end with padding); they are not applied
                const unsigned m = starts(cb + 32);
                const uint2 e = smem_at<uint2>(before + 8u * (unsigned)__popc(m & le));
                s_n = e.x;
                q_n = (int)__ldg(ents + (e.y + cb + 32 + lane));
                before += 8u * (unsigned)__popc(m);
            }
            apply_hits<true>(it, W, true, at, q);
            if (W.n_tasks >= kFlushAt || W.n_blk >= 32) {
                do                                 // keep room for one more batch
                    W = flush(it, a, W, false);
                while (W.n_tasks >= kFlushAt || W.n_blk >= 32);
            }
        }
        carry = total - cb;
    }
    if (carry > 0)                                 // the subject's last batch
        apply_hits<false>(it, W, (uint32_t)lane < carry, s_n, q_n);
    if (W.n_tasks > 0 || W.n_blk > 0)
        W = flush(it, a, W, true);
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");   // no copy may still write the ring
    __syncwarp();
}

__device__ __forceinline__ int turn(int i, int n) { return i < n ? i : i - n; }

}  // namespace

// The warps of a CTA take subjects of one group from the group's counter, a
// few at a time, longest first; a CTA moves to the next group (CTAs start at
// different ones) when the counter has run out.  Only then do its warps wait
// for one another.  Groups that are done are passed a CTA's width at a time:
// 5000 groups of 60 letters against 50 subjects 0.85 ms, one by one 2.6.
//
// Wide: packed cells may say kByteWide.  The check costs the 16-bit instantiation
// 3 to 6 % (350 letters against 300,000 subjects 1.30 -> 1.38 ms), the 8-bit one
// nothing.
template <typename Cell, bool Wide>
__global__ void __launch_bounds__(kByteThreads, 1) byte_kernel(ByteArgs a) {
    using K = Cells<Cell>;
    Head &hd = *reinterpret_cast<Head *>(g_byte_smem);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int window = a.window;
    const unsigned mem = (unsigned)sizeof(Head) + (unsigned)warp * (unsigned)(sizeof(WarpMem) + a.table_len * sizeof(Cell));
    const unsigned tab = mem + (unsigned)sizeof(WarpMem);
    uint16_t *side = sizeof(Cell) == 1 ? a.side + ((size_t)blockIdx.x * nwarps + warp) * a.table_len : nullptr;
    for (int i = threadIdx.x; i < 28 * 32; i += blockDim.x)
        load_scores(hd.matrix, c_blosum, i);
    for (unsigned i = lane; i < a.table_len * (unsigned)sizeof(Cell) / 4; i += 32)
        smem_at<uint32_t>(tab + 4 * i) = 0;
    smem_at<WarpMem>(mem).chain[lane] = 0;
    int top = 0;             // positions used so far
    int since = 0;           // 8-bit cells: subjects since the last sweep
    int code = K::kFlag;
    const int first = (int)((long long)blockIdx.x * a.n_list / gridDim.x);
    for (int step = 0; step < a.n_list;) {
        // the next group with subjects left: every thread looks at one
        __syncthreads();
        if (threadIdx.x == 0)
            hd.go = a.n_list;
        for (int i = threadIdx.x; i < kMaxQ; i += blockDim.x)
            hd.q_ext[i] = hd.q_kept[i] = 0;
        __syncthreads();
        const int look = step + (int)threadIdx.x;
        const bool left = look < a.n_list && *(volatile unsigned long long *)(a.next + a.group_list[turn(first + look, a.n_list)]) <
                                                 (unsigned long long)a.n_subj;
        const unsigned any = __ballot_sync(kAll, left);
        if (any != 0 && lane == 0)
            atomicMin(&hd.go, look + __ffs(any) - 1);
        __syncthreads();
        const int at = hd.go;
        step = at < a.n_list ? at + 1 : step + (int)blockDim.x;
        if (at >= a.n_list)
            continue;
        const int g = a.group_list[turn(first + at, a.n_list)];
        unsigned long long *const counter = a.next + g;
        for (int i = threadIdx.x; i < HBG_PV_WORDS; i += blockDim.x)
            hd.pv[i] = a.pv[(size_t)g * HBG_PV_WORDS + i];
        __syncthreads();
        const HbgGroup G = a.groups[g];
        const uint32_t *packed = a.packed + (size_t)g * HBG_NUM_CELLS;
        const uint16_t *ents = a.entries + G.entry_base;
        const unsigned len = sizeof(Cell) == 2 ? (unsigned)G.diag_len : (unsigned)byte_table_len(G.glen + window);
        if (sizeof(Cell) == 1) {
            // sweeps move the base of this group's cells alone: start it clean
            for (unsigned i = lane; i < len / 4; i += 32)
                smem_at<uint32_t>(tab + 4 * i) = 0;
            __syncwarp();
            top = since = 0;
        }
        // lane k holds the k-th subject of the warp's chunk
        const uint8_t *ds = nullptr;
        int dS = 0, dj = 0, ck = 0, cc = 0;
        for (;; ++ck) {
            if (ck >= cc) {
                unsigned long long base = 0;
                if (lane == 0)
                    base = atomicAdd(counter, (unsigned long long)a.chunk);
                base = __shfl_sync(kAll, base, 0);
                if (base >= (unsigned long long)a.n_subj)
                    break;
                const unsigned long long left = (unsigned long long)a.n_subj - base;
                cc = left < (unsigned long long)a.chunk ? (int)left : a.chunk;
                ck = 0;
                if (lane < cc) {
                    dj = a.order[a.sub_lo + (int)base + lane];
                    dS = a.db_len[dj];
                    ds = a.db + a.db_off[dj];
                }
            }
            const int S = __shfl_sync(kAll, dS, ck);
            int rel = top + window;
            if (sizeof(Cell) == 2) {
                if (rel + S > K::kMaxPos) {
                    __syncwarp();
                    for (unsigned i = lane; i < a.table_len / 2u; i += 32)
                        smem_at<uint32_t>(tab + 4 * i) = 0;
                    __syncwarp();
                    rel = window;
                }
            } else {
                code = code == K::kPending - 1 ? K::kFlag : code + 1;
                if (++since >= K::kPending - K::kFlag - 1 || rel > K::kMaxPos) {
                    // the flag codes run out (subjects of a few letters), or the positions
                    sweep(tab, (int)len, rel - window, code);
                    rel = window;
                    since = 0;
                }
            }
            Item<Cell> it{(const uint8_t *)(uintptr_t)__shfl_sync(kAll, (unsigned long long)(uintptr_t)ds, ck), S,
                          __shfl_sync(kAll, dj, ck), tab, mem, len, (unsigned)window - 3u, rel, code, side,
                          a.letters + G.seq_base, a.ctx_of + G.seq_base, G.first_query};
            process_item<Cell, Wide>(it, a, hd.pv, packed, ents);
            top = S + it.rel;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < G.n_queries && i < kMaxQ; i += blockDim.x) {
            if (hd.q_ext[i])
                atomicAdd(a.q_extended + G.first_query + i, (unsigned long long)hd.q_ext[i]);
            if (hd.q_kept[i])
                atomicAdd(a.q_kept + G.first_query + i, (unsigned long long)hd.q_kept[i]);
        }
    }
}

namespace {

const void *byte_kernel_of(int cell_bytes, bool wide) {
    return cell_bytes == 1 ? (const void *)byte_kernel<uint8_t, true>
                           : wide ? (const void *)byte_kernel<uint16_t, true> : (const void *)byte_kernel<uint16_t, false>;
}

}  // namespace

size_t byte_smem_bytes(int cell_bytes, int threads, int table_len) {
    return sizeof(Head) + (size_t)(threads / 32) * (sizeof(WarpMem) + (size_t)table_len * cell_bytes);
}

cudaError_t byte_configure() {
    int dev = 0, optin = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    for (const void *k : {byte_kernel_of(1, true), byte_kernel_of(2, false), byte_kernel_of(2, true)}) {
        cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, optin);
        if (e != cudaSuccess)
            return e;
    }
    return cudaSuccess;
}

cudaError_t launch_byte(const ByteArgs &a, int cell_bytes, bool wide, int blocks, int threads, cudaStream_t stream) {
    ByteArgs args = a;
    void *params[] = {&args};
    return cudaLaunchKernel(byte_kernel_of(cell_bytes, wide), dim3((unsigned)blocks), dim3((unsigned)threads), params,
                            byte_smem_bytes(cell_bytes, threads, a.table_len), stream);
}

}  // namespace hbg
