// extend.h -- the ungapped X-drop extension of byte_kernel (bytefinder.cu)
// (s_BlastAaExtendTwoHit/Left/Right; H-BLAST h_blast_kernel.cu:1069-1540, with
// the left walk also taken when min(s, q) == 0 as NCBI does).
#ifndef HBG_EXTEND_H
#define HBG_EXTEND_H

#include <cuda_runtime.h>
#include <stdint.h>

namespace hbg {
namespace {

// Scores are kept scaled: the table in shared memory holds 16 * score - 1 for
// (query letter x 32 + subject letter).  A running sum over the letters of one
// block of eight is then 16 * (prefix score) - (letters taken), so that the
// largest sum is the largest prefix and, among equal ones, the first: the
// block's best place comes out of a plain maximum.  The letters taken are added
// back between blocks.
constexpr int kScoreScale = 16;
typedef int16_t Score;

// X-drops are taken up to this.  No walk falls further: it has at most 65,000
// letter pairs of -128 (a sentinel) to 11, so at most 9.1 million lie between its
// best score and any other.  The scaled value and sums with it fit 32 bits.
constexpr int kMaxDrop = 1 << 24;

__device__ __forceinline__ void load_scores(Score *m, const int8_t *blosum, int i) {
    m[i] = (Score)(kScoreScale * blosum[i] - 1);
}

// A sequence by an aligned base (the same in all lanes of a warp) and 32-bit
// offsets from it; the base lies 64 letters before the first one, so that the
// blocks that reach past the start have offsets too.
struct Letters {
    const uint32_t *base;
    unsigned first;                          // offset of letter 0
};
__device__ __forceinline__ Letters letters_of(const uint8_t *p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p) - 64;
    return Letters{reinterpret_cast<const uint32_t *>(a & ~(uintptr_t)3), 64u + (unsigned)(a & 3)};
}

// Eight letters from offset `at` (any alignment), as two words: three aligned
// 32-bit loads and two funnel shifts.  Reads the aligned words that hold them.
__device__ __forceinline__ uint2 load8(const uint32_t *base, unsigned at) {
    const uint32_t *w = base + (at >> 2);
    const uint32_t sh = at * 8;              // funnel shifts take it modulo 32
    const uint32_t w0 = __ldg(w), w1 = __ldg(w + 1), w2 = __ldg(w + 2);
    return make_uint2(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh));
}

// Scaled scores of four letter pairs, in byte order.  The table indices of two
// pairs are formed in one word.
__device__ __forceinline__ void score4(const Score *m, uint32_t qw, uint32_t sw, int *x) {
    const uint32_t s2 = sw * 2u;             // letters are below 32: byte offsets into the table
    const uint32_t e = (qw & 0x00ff00ffu) * 64u + (s2 & 0x00ff00ffu);
    const uint32_t o = ((qw >> 8) & 0x00ff00ffu) * 64u + ((s2 >> 8) & 0x00ff00ffu);
    const char *b = reinterpret_cast<const char *>(m);
    x[0] = *reinterpret_cast<const Score *>(b + (e & 0xffffu));
    x[1] = *reinterpret_cast<const Score *>(b + (o & 0xffffu));
    x[2] = *reinterpret_cast<const Score *>(b + (e >> 16));
    x[3] = *reinterpret_cast<const Score *>(b + (o >> 16));
}

__device__ __forceinline__ int max8(const int *p) {
    return max(__vimax3_s32(p[0], p[1], p[2]), __vimax3_s32(p[3], p[4], __vimax3_s32(p[5], p[6], p[7])));
}
__device__ __forceinline__ int min8(const int *p) {
    return min(__vimin3_s32(p[0], p[1], p[2]), __vimin3_s32(p[3], p[4], __vimin3_s32(p[5], p[6], p[7])));
}

// An X-drop walk, eight letters at a time.  Letters past the end of a sequence
// count as zero, which neither raises the best score nor ends the walk.
struct Walk {
    int score, best;         // scaled, without the letters taken; a multiple of kScoreScale
    int best_len;            // letters in the best walk
    bool stop;
};

// x[0..7]: the scaled scores of the next letters in walking order, `taken`
// letters before them.  Right: the walk also ends where the score is <= 0, and
// *adv is the number of letters before the one that ends it (8: none).  The
// first `skip` letters do not belong to the walk (zeros).
template <bool Right>
__device__ __forceinline__ void walk8(Walk &w, const int *x, int taken, int drop, int skip, int *adv) {
    int p[8];
    p[0] = w.score + x[0];
#pragma unroll
    for (int i = 1; i < 8; ++i)
        p[i] = p[i - 1] + x[i];
    const int top = max8(p), low = min8(p);
    w.score = p[7] + 8;
    *adv = 8;
    // 16 (largest prefix) is in top + 1 .. top + 8, so it beats the best if top
    // + 8 reaches the next score; 16 (a prefix) <= limit if and only if its sum
    // is below limit, for any limit that is a multiple of 16
    const bool up = top >= w.best + (kScoreScale - 8);
    if (up && (top - low >= drop - 8 || (Right && low <= 0))) {
        // better, and perhaps the end: letter by letter
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int c = p[i] + i + 1;
            const bool better = !w.stop && c > w.best;
            w.best_len = better ? taken + i + 1 : w.best_len;
            w.best = better ? c : w.best;
            const bool end = !w.stop && i >= skip && ((Right && c <= 0) || w.best - c >= drop);
            *adv = end ? i : *adv;
            w.stop = w.stop || end;
        }
    } else {
        // nothing better: the best so far decides about the end; better: no end
        const int limit = Right ? max(w.best - drop, 0) : w.best - drop;
        const int b = (top + kScoreScale - 1) & -kScoreScale;
        w.stop = !up && low < limit;
        w.best_len = up ? taken + (b - top) : w.best_len;
        w.best = up ? b : w.best;
        if (Right && w.stop) {
#pragma unroll
            for (int i = 7; i >= 0; --i)
                *adv = p[i] < limit ? i : *adv;
        }
    }
}

// Letters from the n-th on are past the end of a sequence.
__device__ __forceinline__ void cut8(int *x, int n) {
    if (n < 8) {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            x[i] = i < n ? x[i] : -1;
    }
}

struct Ext {
    int q_start, s_start, len, score, s_last_off;
    bool right;
};

// The extension of a second hit (word at s_h, q_h; the query's letters start at
// q_start of G) whose first hit's word ends before s_left: the best prefix of the word, the walk to the left from its
// end, and the walk to the right if the left one reached the first hit.  The
// first block of the left walk holds the word.  Reads up to 8 letters before
// and 11 after the sequences' ends (the letter buffers are padded).
__device__ __forceinline__ Ext extend_two_hit(const Score *m, const Letters &S, int s_len, const Letters &G, int q_start,
                                              int q_len, int s_left, int s_h, int q_h, int dropoff) {
    const unsigned s0 = S.first + (unsigned)s_h - 5u, q0 = G.first + (unsigned)(q_start + q_h) - 5u;
    const int drop = kScoreScale * min(dropoff, kMaxDrop);
    Walk w{0, 0, 0, false};
    int x[8], y[8], adv;
    const int n_left = min(s_h, q_h) + 3;    // letters up to the end of the word
    int skip, k = 0;
    {
        const uint2 sw = load8(S.base, s0), qw = load8(G.base, q0);
        score4(m, qw.x, sw.x, y);
        score4(m, qw.y, sw.y, y + 4);
        // prefixes of the word, as 16 (score) - (letters): the largest, first one wins
        const int a1 = y[5], a2 = a1 + y[6], a3 = a2 + y[7];
        const int a = __vimax3_s32(a1, a2, a3);
        const int right_d = a < 0 ? 0 : (a == a1 ? 1 : (a == a2 ? 2 : 3));
        skip = 3 - right_d;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            x[i] = y[7 - i];
        x[0] = skip > 0 ? -1 : x[0];
        x[1] = skip > 1 ? -1 : x[1];
        x[2] = skip > 2 ? -1 : x[2];
        cut8(x, n_left);
        walk8<false>(w, x, 0, drop, skip, &adv);
    }
    for (k = 8; !w.stop && k < n_left; k += 8) {
        const uint2 sw = load8(S.base, s0 - (unsigned)k), qw = load8(G.base, q0 - (unsigned)k);
        score4(m, qw.x, sw.x, y);
        score4(m, qw.y, sw.y, y + 4);
#pragma unroll
        for (int i = 0; i < 8; ++i)
            x[i] = y[7 - i];
        cut8(x, n_left - k);
        walk8<false>(w, x, k, drop, 0, &adv);
    }
    const int left_d = w.best > 0 ? w.best_len - skip : 0;
    const int left_score = w.best;
    const int s_r = s_h + 3 - skip, q_r = q_h + 3 - skip;    // where the right walk starts
    Ext e;
    e.right = left_d >= s_r - s_left;
    e.s_last_off = s_r;
    int rlen = 0;
    if (e.right) {
        const int n = min(s_len - s_r, q_len - q_r);
        w.score = w.best;
        w.best_len = 0;
        w.stop = false;
        int i = 0;
        while (!w.stop && i < n) {
            const uint2 sw = load8(S.base, s0 + 8u - (unsigned)skip + (unsigned)i),
                        qw = load8(G.base, q0 + 8u - (unsigned)skip + (unsigned)i);
            score4(m, qw.x, sw.x, x);
            score4(m, qw.y, sw.y, x + 4);
            cut8(x, n - i);
            walk8<true>(w, x, i, drop, 0, &adv);
            i += min(adv, n - i);
        }
        rlen = w.best_len;
        e.s_last_off = s_r + i;
    }
    e.q_start = q_r - left_d;
    e.s_start = s_r - left_d;
    e.len = left_d + rlen;
    e.score = (e.right ? w.best : left_score) / kScoreScale;
    return e;
}

}  // namespace
}  // namespace hbg

#endif
