// tables.cu -- the neighbourhood-word lookup tables of a batch, built on the
// device from its letters (batch_builder.cpp builds the same tables on the host
// when a caller asks to see them; the rule is there).
//
// A warp owns one row of 32 words (x, y, *) and walks the letters of one segment
// (up to kTableSegment letters of one query) 32 at a time: lane i tests whether the word at its place can reach
// the threshold with x, y and the best third letter, and the warp then scores
// the few places that can against all 32 third letters, lane z word (x, y, z).
// Places are visited in ascending order, so every cell's entries come out
// ascending.  Two such walks (count, fill) with prefix sums between.  Bound by
// the walks' chains of shuffles and look-ups, so long queries are cut into
// segments walked side by side (20,000 letters in one: 300 us a walk).
// From the call to the end of a search of one subject, upload and build
// included: 300 letters 0.16 ms, 20,000 letters 0.39, 64 queries of 50,000 letters
// 0.60, of which the caller waits 0.05, 0.07 and 0.14; the host build alone took
// 0.13, 3.4 and 2.2 ms.
#include <cuda_runtime.h>

#include "kernels.h"

namespace hbg {

namespace {

constexpr unsigned kAll = 0xffffffffu;
constexpr int kLetters = HBG_ALPHABET;            // rows (x, y) with x, y < 28 have words
constexpr int kRowsPerCta = 8;
constexpr int kCtas = (kLetters * kLetters + kRowsPerCta - 1) / kRowsPerCta;

__constant__ int8_t c_blosum[28 * 32] = {
#include "blosum62.inc"
};

// Fill false: the counts of a segment's words; true: its entries.
template <bool Fill>
__global__ void __launch_bounds__(kRowsPerCta * 32)
walk_rows(TableArgs a) {
    __shared__ int8_t m[28 * 32];
    __shared__ int8_t most[32];                   // best score of each letter against any
    const int lane = threadIdx.x & 31;
    const TableSegment S = a.segs[a.first_seg + blockIdx.y];
    const int g = S.group;
    for (int i = threadIdx.x; i < 28 * 32; i += blockDim.x)
        m[i] = c_blosum[i];
    __syncthreads();
    if (threadIdx.x < kLetters) {
        int best = -128;
        for (int z = 0; z < kLetters; ++z)
            best = max(best, (int)m[threadIdx.x * 32 + z]);
        most[threadIdx.x] = (int8_t)best;
    }
    __syncthreads();
    const HbgGroup &G = a.groups[g];
    const uint8_t *gs = a.letters + G.seq_base;
    const int32_t *gc = a.ctx_of + G.seq_base;
    const int r = blockIdx.x * kRowsPerCta + (threadIdx.x >> 5);
    if (r >= kLetters * kLetters)
        return;
    const int x = r / kLetters, y = r % kLetters;
    const int row = x * 32 + y;
    uint32_t *const counts = a.counts + (size_t)blockIdx.y * HBG_NUM_CELLS + row * 32 + lane;
    uint32_t n = Fill ? a.cells[(size_t)g * HBG_CELL_STRIDE + row * 32 + lane] + *counts : 0u;
    uint16_t *const ents = a.entries + G.entry_base;
    for (int p0 = S.begin; p0 < S.end; p0 += 32) {
        const int p = p0 + lane;
        int t = 0, c = 0;
        bool on = false;
        if (p < S.end) {
            const int ctx = gc[p];
            c = gs[p + 2];
            t = m[gs[p] * 32 + x] + m[gs[p + 1] * 32 + y];
            on = ctx >= 0 && gc[p + 1] == ctx && gc[p + 2] == ctx && t + most[c] >= a.threshold;
        }
        for (unsigned mask = __ballot_sync(kAll, on); mask; mask &= mask - 1) {
            const int i = __ffs(mask) - 1;
            const int ti = __shfl_sync(kAll, t, i), ci = __shfl_sync(kAll, c, i);
            if (lane < kLetters && ti + m[ci * 32 + lane] >= a.threshold) {
                if (Fill)
                    ents[n] = (uint16_t)(p0 + i);
                ++n;
            }
        }
    }
    if (!Fill)
        *counts = n;
}

// Per word of a group: a segment's count becomes the count of those before it,
// and the sums are the word's count per query and (in packed) in the group.
__global__ void __launch_bounds__(256) sum_segments(TableArgs a) {
    const int g = a.first_group + blockIdx.y;
    const HbgGroup &G = a.groups[g];
    const int w = blockIdx.x * 256 + threadIdx.x;
    uint32_t n = 0;
    const bool used = (w >> 10) < kLetters && ((w >> 5) & 31) < kLetters;
    for (int k = 0; k < G.n_segs; ++k) {
        const int q = a.segs[G.seg_base + k].query;
        uint32_t first = n;
        for (;; ++k) {
            uint32_t *const c = a.counts + (size_t)(G.seg_base - a.first_seg + k) * HBG_NUM_CELLS + w;
            const uint32_t here = used ? *c : 0u;
            *c = n;
            n += here;
            if (k + 1 >= G.n_segs || a.segs[G.seg_base + k + 1].query != q)
                break;
        }
        a.query_cells[(size_t)q * HBG_NUM_CELLS + w] = (uint16_t)(n - first);
    }
    a.packed[(size_t)g * HBG_NUM_CELLS + w] = n;
}

// First entry and count of a cell in one word; where the count does not fit,
// byte_kernel reads the cells.
__device__ __forceinline__ uint32_t pack(uint32_t first, uint32_t count) {
    return first | (min(count, (uint32_t)kByteWide) << 22);
}

// One CTA per group: cells, presence vector, packed cells (from the words'
// counts in packed).  Thread t has row t.
__global__ void __launch_bounds__(1024) scan_rows(TableArgs a) {
    __shared__ uint32_t sums[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = a.first_group + blockIdx.x;
    uint32_t *const pk = a.packed + (size_t)g * HBG_NUM_CELLS + t * 32;
    uint32_t total = 0, bits = 0;
#pragma unroll 8
    for (int z = 0; z < 32; ++z) {
        const uint32_t c = pk[z];
        total += c;
        bits |= c ? 1u << z : 0u;
    }
    uint32_t incl = total;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kAll, incl, o);
        if (lane >= o)
            incl += v;
    }
    if (lane == 31)
        sums[warp] = incl;
    __syncthreads();
    const uint32_t before = __reduce_add_sync(kAll, lane < warp ? sums[lane] : 0u);
    uint32_t at = before + incl - total;
    uint32_t *const cs = a.cells + (size_t)g * HBG_CELL_STRIDE + t * 32;
#pragma unroll 8
    for (int z = 0; z < 32; ++z) {
        const uint32_t c = pk[z];
        cs[z] = at;
        pk[z] = pack(at, c);
        at += c;
    }
    a.pv[(size_t)g * HBG_PV_WORDS + t] = bits;
    if (t == 1023)
        cs[32] = at;
}

// The cells of every group in one word each.
__global__ void __launch_bounds__(256)
pack_cells(const uint32_t *cells, uint32_t *packed) {
    const uint32_t *cs = cells + (size_t)blockIdx.y * HBG_CELL_STRIDE;
    const int w = blockIdx.x * 256 + threadIdx.x;
    packed[(size_t)blockIdx.y * HBG_NUM_CELLS + w] = pack(cs[w], cs[w + 1] - cs[w]);
}

}  // namespace

cudaError_t launch_tables(const TableArgs &a, int32_t n_groups, int32_t n_segs, cudaStream_t stream) {
    const dim3 grid(kCtas, (unsigned)n_segs);
    walk_rows<false><<<grid, kRowsPerCta * 32, 0, stream>>>(a);
    sum_segments<<<dim3(HBG_NUM_CELLS / 256, n_groups), 256, 0, stream>>>(a);
    scan_rows<<<n_groups, 1024, 0, stream>>>(a);
    walk_rows<true><<<grid, kRowsPerCta * 32, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_pack_cells(const uint32_t *cells, int32_t n_groups, uint32_t *packed, cudaStream_t stream) {
    constexpr int kMost = 32768;                  // the grid's second dimension is limited
    for (int32_t g0 = 0; g0 < n_groups; g0 += kMost) {
        const int32_t n = n_groups - g0 < kMost ? n_groups - g0 : kMost;
        pack_cells<<<dim3(HBG_NUM_CELLS / 256, n), 256, 0, stream>>>(cells + (size_t)g0 * HBG_CELL_STRIDE,
                                                                     packed + (size_t)g0 * HBG_NUM_CELLS);
    }
    return cudaGetLastError();
}

}  // namespace hbg
