// batch_builder.cpp -- query packing, six-frame translation and the
// neighbourhood-word lookup tables of a batch (host side).
//
// Lookup-table rule (NCBI BLAST+ 2.2.28 blast_aalookup.c, the table H-BLAST
// consumes at h_blast_v1.1/H-BLAST/h_blast.cu:940-958): word size 3 over the
// 28-letter NCBIstdaa alphabet, 5 bits per letter (index (a<<10)|(b<<5)|c,
// as the kernel builds it at h_blast_kernel.cu:610-614); query offset p is
// stored in cell w when the three letters at p lie inside one context and
// score(query[p..p+2], w) >= threshold.  Cells hold offsets in ascending
// order, the order lut_sorting enforces (h_blast.cu:165-194).
#include "batch_builder.h"

#include <string.h>

#include <algorithm>
#include <array>
#include <atomic>
#include <exception>
#include <functional>
#include <map>
#include <memory>
#include <mutex>
#include <thread>

namespace hbg {

namespace {

const int8_t kBlosum62[28 * 32] = {
#include "../csrc/blosum62.inc"
};

// Neighbour words of every query word, computed once per distinct word and
// kept for the life of the process (one cache per threshold), so batches
// built one after another -- a serving loop -- reuse the enumerations.
class NeighbourCache {
  public:
    explicit NeighbourCache(int32_t threshold) : threshold_(threshold) {
        for (int x = 0; x < HBG_ALPHABET; ++x) {
            int m = -1000;
            for (int y = 0; y < HBG_ALPHABET; ++y)
                m = std::max<int>(m, kBlosum62[x * 32 + y]);
            row_max_[x] = m;
        }
        done_.assign(HBG_NUM_CELLS, 0);
        lists_.resize(HBG_NUM_CELLS);
    }

    // The neighbours of a word that prepare() has enumerated; read-only, so
    // any number of threads may call it.
    const std::vector<uint16_t> &get(uint8_t a, uint8_t b, uint8_t c) const {
        return lists_[(a << 10) | (b << 5) | c];
    }

    // Enumerate the neighbourhoods of those words not seen before, in
    // parallel.  Builds running at the same time take turns here; a list,
    // once written, never changes.
    template <typename ParallelFor>
    void prepare(const std::vector<int32_t> &words, ParallelFor &&pfor) {
        std::lock_guard<std::mutex> lock(mu_);
        std::vector<int32_t> keys;
        for (int32_t k : words)
            if (!done_[k])
                keys.push_back(k);
        std::sort(keys.begin(), keys.end());  // each listed once
        keys.erase(std::unique(keys.begin(), keys.end()), keys.end());
        pfor((int64_t)keys.size(), [&](int64_t i) {
            const int32_t k = keys[i];
            lists_[k].clear();                // of a build that ran out of memory
            enumerate((uint8_t)(k >> 10), (uint8_t)((k >> 5) & 31), (uint8_t)(k & 31), &lists_[k]);
        });
        for (int32_t k : keys)
            done_[k] = 1;
    }

  private:
    void enumerate(uint8_t a, uint8_t b, uint8_t c, std::vector<uint16_t> *out) {
        const int8_t *ra = kBlosum62 + a * 32;
        const int8_t *rb = kBlosum62 + b * 32;
        const int8_t *rc = kBlosum62 + c * 32;
        for (int x = 0; x < HBG_ALPHABET; ++x) {
            int s1 = ra[x];
            if (s1 + row_max_[b] + row_max_[c] < threshold_)
                continue;
            for (int y = 0; y < HBG_ALPHABET; ++y) {
                int s2 = s1 + rb[y];
                if (s2 + row_max_[c] < threshold_)
                    continue;
                for (int z = 0; z < HBG_ALPHABET; ++z)
                    if (s2 + rc[z] >= threshold_)
                        out->push_back((uint16_t)((x << 10) | (y << 5) | z));
            }
        }
    }

    int32_t threshold_;
    std::array<int, HBG_ALPHABET> row_max_;
    std::vector<uint8_t> done_;
    std::vector<std::vector<uint16_t>> lists_;
    std::mutex mu_;
};

NeighbourCache &neighbour_cache(int32_t threshold) {
    static std::mutex mu;
    static std::map<int32_t, std::unique_ptr<NeighbourCache>> caches;
    std::lock_guard<std::mutex> lock(mu);
    std::unique_ptr<NeighbourCache> &c = caches[threshold];
    if (!c)
        c.reset(new NeighbourCache(threshold));
    return *c;
}

// Run body(i) for i in [0, n) on up to 16 host threads (items taken from a
// shared counter), on fewer when no more can be started.  The first exception
// of a body ends the run and comes out of the call.
void parallel_for(int64_t n, const std::function<void(int64_t)> &body) {
    const int64_t nt = std::min<int64_t>({n, 16, (int64_t)std::max(1u, std::thread::hardware_concurrency())});
    if (nt <= 1) {
        for (int64_t i = 0; i < n; ++i)
            body(i);
        return;
    }
    std::atomic<int64_t> next{0};
    std::mutex mu;
    std::exception_ptr first;
    auto run = [&] {
        try {
            for (int64_t i = next++; i < n; i = next++)
                body(i);
        } catch (...) {
            std::lock_guard<std::mutex> lock(mu);
            if (!first)
                first = std::current_exception();
            next = n;
        }
    };
    std::vector<std::thread> th;
    try {
        for (int64_t t = 1; t < nt; ++t)
            th.emplace_back(run);
    } catch (const std::exception &) {
    }
    run();
    for (std::thread &x : th)
        x.join();
    if (first)
        std::rethrow_exception(first);
}

// Every letter is in 1..27, eight at a time.
bool letters_valid(const uint8_t *s, int32_t n) {
    constexpr uint64_t kOnes = 0x0101010101010101ull, kTop = 0x80 * kOnes;
    uint64_t bad = 0;
    int32_t i = 0;
    for (; i + 8 <= n; i += 8) {
        uint64_t w;
        memcpy(&w, s + i, 8);
        // the top bit of a byte: set if it is zero (or follows one that is), 28..127, 128..255
        bad |= ((w - kOnes) & ~w) | (w + (0x80 - HBG_ALPHABET) * kOnes) | w;
    }
    bad &= kTop;
    for (; i < n; ++i)
        bad |= s[i] == 0 || s[i] >= HBG_ALPHABET;
    return bad == 0;
}

int32_t next_pow2(int32_t v) {
    int32_t n = 1;
    while (n < v)
        n <<= 1;
    return n;
}

}  // namespace

int32_t blosum62(int32_t a, int32_t b) {
    if (a < 0 || a >= HBG_ALPHABET || b < 0 || b >= HBG_ALPHABET)
        return -128;
    return kBlosum62[a * 32 + b];
}

const int8_t *blosum62_table() { return kBlosum62; }

std::string build_batch(const std::vector<QueryIn> &qs, int32_t threshold,
                        int32_t window, int32_t max_group_len, HostBatch *out, double mode_hits) {
    if (window < 1 || window > 100000)
        return "window must be in 1..100000";
    if (qs.empty())
        return "empty batch";
    if (max_group_len <= 0)
        max_group_len = kDefaultGroupLen;
    // offsets in a group are kept in 16 bits: lookup entries, queued extensions
    max_group_len = std::min<int32_t>(max_group_len, HBG_MAX_QUERY_LEN);
    if (mode_hits < 0)
        mode_hits = kOffsetModeHits;
    HostBatch &b = *out;
    b = HostBatch();
    b.threshold = threshold;
    b.window = window;

    // --- validate and pack queries into groups (in order) ---
    std::vector<int32_t> group_of(qs.size());
    int32_t cur_len = 0, cur_n = 0;
    int32_t n_groups = 0;
    int64_t total = 0;                           // letters of the groups before this one
    for (size_t k = 0; k < qs.size(); ++k) {
        const QueryIn &q = qs[k];
        if (q.len <= 0 || q.len > HBG_MAX_QUERY_LEN)
            return "query " + std::to_string(k) + ": length must be in 1.." +
                   std::to_string(HBG_MAX_QUERY_LEN);
        size_t nc = q.ctx_off.size();
        if (nc == 0 || q.ctx_len.size() != nc || q.xdrop.size() != nc || q.cutoff.size() != nc)
            return "query " + std::to_string(k) + ": bad context arrays";
        for (size_t c = 0; c < nc; ++c) {
            if (q.ctx_off[c] < 0 || q.ctx_len[c] < 0 ||
                q.ctx_off[c] + q.ctx_len[c] > q.len)
                return "query " + std::to_string(k) + ": context outside the query";
            if (c > 0 && q.ctx_off[c] < q.ctx_off[c - 1] + q.ctx_len[c - 1])
                return "query " + std::to_string(k) + ": contexts overlap or are unordered";
            if (q.xdrop[c] < 0)
                return "query " + std::to_string(k) + ": negative x_dropoff";
            if (!letters_valid(q.seq + q.ctx_off[c], q.ctx_len[c]))
                return "query " + std::to_string(k) + ": letter outside NCBIstdaa 1..27";
        }
        int32_t need = (cur_n > 0 ? window : 0) + q.len;
        if (cur_n == 0 || cur_len + need > max_group_len || cur_n >= kMaxQueriesPerGroup) {
            if (cur_n > 0)
                ++n_groups;
            total += cur_len;
            cur_len = q.len;
            cur_n = 1;
        } else {
            cur_len += need;
            ++cur_n;
        }
        group_of[k] = n_groups;
        b.max_query_len = std::max(b.max_query_len, q.len);
    }
    ++n_groups;

    // --- lay out letters, queries, contexts ---
    b.groups.resize(n_groups);
    b.queries.resize(qs.size());
    b.letters.reserve((size_t)(total + cur_len));
    b.ctx_of.reserve((size_t)(total + cur_len));
    int64_t seq_pos = 0;
    for (int32_t g = 0, k = 0; g < n_groups; ++g) {
        HbgGroup &G = b.groups[g];
        memset(&G, 0, sizeof(G));
        G.seq_base = seq_pos;
        G.first_query = k;
        int32_t glen = 0;
        while (k < (int32_t)qs.size() && group_of[k] == g) {
            const QueryIn &q = qs[k];
            if (glen > 0) {
                b.letters.insert(b.letters.end(), window, 0);
                b.ctx_of.insert(b.ctx_of.end(), window, -1);
                glen += window;
            }
            HbgQueryDesc &Q = b.queries[k];
            memset(&Q, 0, sizeof(Q));
            Q.group = g;
            Q.start = glen;
            Q.len = q.len;
            Q.first_ctx = (int32_t)b.contexts.size();
            Q.n_ctx = (int32_t)q.ctx_off.size();
            // contexts in order; letters between them are sentinels whatever the
            // caller put there
            int32_t put = 0;
            auto gap = [&](int32_t end) {
                b.letters.insert(b.letters.end(), end - put, 0);
                b.ctx_of.insert(b.ctx_of.end(), end - put, -1);
                put = end;
            };
            for (int32_t c = 0; c < Q.n_ctx; ++c) {
                HbgContext C;
                C.query = k;
                C.local = c;
                C.x_dropoff = q.xdrop[c];
                C.cutoff = q.cutoff[c];
                int32_t ci = (int32_t)b.contexts.size();
                b.contexts.push_back(C);
                gap(q.ctx_off[c]);
                b.letters.insert(b.letters.end(), q.seq + put, q.seq + put + q.ctx_len[c]);
                b.ctx_of.insert(b.ctx_of.end(), q.ctx_len[c], ci);
                put += q.ctx_len[c];
                if (q.ctx_len[c] >= HBG_WORD_SIZE)
                    b.runs.push_back({g, glen + q.ctx_off[c], q.ctx_len[c]});
            }
            gap(q.len);
            glen += q.len;
            ++k;
        }
        G.n_queries = k - G.first_query;
        G.glen = glen;
        G.diag_len = next_pow2(glen + window);
        G.placement = G.diag_len <= kSmemDiagMax ? 0 : 1;
        if (G.placement)
            b.max_diag_len = std::max(b.max_diag_len, G.diag_len);
        else
            b.smem_diag_len = std::max(b.smem_diag_len, G.diag_len);
        seq_pos += glen;
    }

    b.mode_hits = mode_hits;
    if (mode_hits < kOffsetModeHits)             // the hit mode depends on the tables
        build_tables(out);
    return std::string();
}

namespace {

// A word is stored when its three letters lie inside one context.
bool valid(const int32_t *gc, int32_t p) {
    const int32_t c0 = gc[p];
    return c0 >= 0 && gc[p + 1] == c0 && gc[p + 2] == c0;
}

// The neighbourhoods of every word in the batch, enumerated in parallel.
NeighbourCache &prepared_cache(const HostBatch &b) {
    NeighbourCache &nb = neighbour_cache(b.threshold);
    std::vector<int32_t> words;
    words.reserve(b.letters.size());
    for (const HbgGroup &G : b.groups) {
        const uint8_t *gs = b.letters.data() + G.seq_base;
        const int32_t *gc = b.ctx_of.data() + G.seq_base;
        for (int32_t p = 0; p + HBG_WORD_SIZE <= G.glen; ++p)
            if (valid(gc, p))
                words.push_back((gs[p] << 10) | (gs[p + 1] << 5) | gs[p + 2]);
    }
    nb.prepare(words, parallel_for);
    return nb;
}

}  // namespace

// Neighbours of every word at a threshold, without listing them: sums of two
// letters' scores are counted once (at[a][b][v]: pairs (x, y) with score(a, x) +
// score(b, y) >= v), and a word's neighbours are the pairs that each third
// letter's score leaves room for.  One table per threshold, kept: 64 KiB, at most
// 418 of them (lower and higher thresholds count as the ends of the range).
constexpr int kScoreMin = -128, kScoreMax = 11;

const uint16_t *neighbour_counts(int32_t threshold) {
    constexpr int kPairMin = 2 * kScoreMin, kPairs = 2 * (kScoreMax - kScoreMin) + 1;
    typedef std::array<uint16_t, kPairs + 1> Sums;
    struct Row {
        std::vector<std::pair<int, int>> values;   // score, letters with it
    };
    static std::mutex mu;
    static std::vector<Row> rows;
    static std::vector<Sums> at;
    static std::map<int32_t, std::vector<uint16_t>> tables;
    threshold = std::min(std::max(threshold, 3 * kScoreMin), 3 * kScoreMax + 1);
    std::lock_guard<std::mutex> lock(mu);
    if (at.empty()) {
        std::vector<Row> r(HBG_ALPHABET);
        for (int x = 0; x < HBG_ALPHABET; ++x) {
            std::map<int, int> n;
            for (int y = 0; y < HBG_ALPHABET; ++y)
                ++n[kBlosum62[x * 32 + y]];
            r[x].values.assign(n.begin(), n.end());
        }
        std::vector<Sums> sums(HBG_ALPHABET * HBG_ALPHABET, Sums{});
        for (int x = 0; x < HBG_ALPHABET; ++x)
            for (int y = 0; y < HBG_ALPHABET; ++y) {
                Sums &c = sums[x * HBG_ALPHABET + y];
                for (const auto &u : r[x].values)
                    for (const auto &v : r[y].values)
                        c[u.first + v.first - kPairMin] += (uint16_t)(u.second * v.second);
                for (int k = kPairs - 1; k >= 0; --k)
                    c[k] = (uint16_t)(c[k] + c[k + 1]);
            }
        rows.swap(r);
        at.swap(sums);
    }
    std::vector<uint16_t> &t = tables[threshold];
    if (t.empty()) {
        std::vector<uint16_t> n(HBG_NUM_CELLS, 0);
        for (int x = 0; x < HBG_ALPHABET; ++x)
            for (int y = 0; y < HBG_ALPHABET; ++y)
                for (int z = 0; z < HBG_ALPHABET; ++z) {
                    int sum = 0;
                    for (const auto &v : rows[z].values) {
                        const int k = threshold - v.first - kPairMin;
                        if (k < kPairs)
                            sum += v.second * at[x * HBG_ALPHABET + y][std::max(k, 0)];
                    }
                    n[(x << 10) | (y << 5) | z] = (uint16_t)sum;
                }
        t.swap(n);
    }
    return t.data();
}

// Groups of so few words need no bound for their fullest cell, any count fits a
// packed cell; nor do those of so many letters: byte_kernel's 8-bit tables, which
// they have, take any count.
constexpr int64_t kMaxCellAlways = 1022, kMaxCellNever = 4096;

int64_t count_entries(HostBatch *out) {
    HostBatch &b = *out;
    if (!b.cells.empty())
        return (int64_t)b.entries.size();
    if (!b.counted) {
        const uint16_t *count = neighbour_counts(b.threshold);
        for (HbgGroup &G : b.groups)
            G.n_entries = 0;
        for (const HostBatch::Run &r : b.runs) {
            const uint8_t *s = b.letters.data() + b.groups[r.group].seq_base + r.at;
            auto of = [&](uint32_t x, uint32_t y, uint32_t z) { return (uint32_t)count[(x << 10) | (y << 5) | z]; };
            uint32_t n[4] = {0, 0, 0, 0};          // a run has less than 2^32 entries
            int32_t p = 0;
            for (; p + 6 <= r.len; p += 4) {
                n[0] += of(s[p], s[p + 1], s[p + 2]);
                n[1] += of(s[p + 1], s[p + 2], s[p + 3]);
                n[2] += of(s[p + 2], s[p + 3], s[p + 4]);
                n[3] += of(s[p + 3], s[p + 4], s[p + 5]);
            }
            for (; p + HBG_WORD_SIZE <= r.len; ++p)
                n[0] += of(s[p], s[p + 1], s[p + 2]);
            b.groups[r.group].n_entries += (int32_t)(n[0] + n[1] + n[2] + n[3]);
        }
        for (HbgGroup &G : b.groups) {
            const int64_t words = std::max(0, G.glen - HBG_WORD_SIZE + 1);
            G.max_cell = (int32_t)words;
            if (b.threshold <= 0 || words <= kMaxCellAlways || G.glen > kMaxCellNever)
                continue;
            const uint8_t *gs = b.letters.data() + G.seq_base;
            int32_t letters[4][32] = {{0}};            // by place: equal letters in a row would wait for one another
            for (int32_t p = 0; p < G.glen; ++p)
                ++letters[p & 3][gs[p] & 31];
            // The scores of a cell's words against it sum to at least threshold
            // each, and to no more than three times what all letters of the
            // group score against the best letter, negative scores left out.
            // (Random proteins: 0.17 entries a letter at threshold 11.)
            int64_t most = 0;
            for (int x = 0; x < HBG_ALPHABET; ++x) {
                int64_t sum = 0;
                for (int y = 1; y < HBG_ALPHABET; ++y)
                    sum += (int64_t)(letters[0][y] + letters[1][y] + letters[2][y] + letters[3][y]) *
                           std::max<int>(kBlosum62[y * 32 + x], 0);
                most = std::max(most, sum);
            }
            G.max_cell = (int32_t)std::min(words, 3 * most / b.threshold);
        }
        b.counted = true;
    }
    int64_t n = 0;
    for (const HbgGroup &G : b.groups)
        n += G.n_entries;
    return n;
}

// Count, then fill, per group (in parallel: groups own disjoint cells, queries
// and entries).
void build_tables(HostBatch *out) {
    HostBatch &b = *out;
    struct Undo {                      // an exception leaves no half-built tables
        HostBatch *b;
        ~Undo() {
            if (b) {
                b->cells = std::vector<uint32_t>();
                b->pv = std::vector<uint32_t>();
                b->query_cells = std::vector<uint16_t>();
                b->entries = std::vector<uint16_t>();
            }
        }
    } undo{out};
    const int32_t n_groups = (int32_t)b.groups.size();
    const double mode_hits = b.mode_hits;
    const NeighbourCache &nb = prepared_cache(b);
    b.cells.assign((size_t)n_groups * HBG_CELL_STRIDE, 0);
    b.pv.assign((size_t)n_groups * HBG_PV_WORDS, 0);
    b.query_cells.assign(b.queries.size() * (size_t)HBG_NUM_CELLS, 0);
    std::vector<uint32_t> group_entries(n_groups, 0);
    parallel_for(n_groups, [&](int64_t gi) {
        const int32_t g = (int32_t)gi;
        HbgGroup &G = b.groups[g];
        const uint8_t *gs = b.letters.data() + G.seq_base;
        const int32_t *gc = b.ctx_of.data() + G.seq_base;
        std::vector<uint32_t> count(HBG_NUM_CELLS, 0);
        for (int32_t p = 0; p + HBG_WORD_SIZE <= G.glen; ++p) {
            if (!valid(gc, p))
                continue;
            const std::vector<uint16_t> &ws = nb.get(gs[p], gs[p + 1], gs[p + 2]);
            uint16_t *qc = b.query_cells.data() + (size_t)b.contexts[gc[p]].query * HBG_NUM_CELLS;
            for (uint16_t w : ws) {
                ++count[w];
                ++qc[w];
            }
        }
        uint32_t *cs = b.cells.data() + (size_t)g * HBG_CELL_STRIDE;
        uint32_t *pv = b.pv.data() + (size_t)g * HBG_PV_WORDS;
        uint32_t acc = 0, most = 0;
        for (int32_t w = 0; w < HBG_NUM_CELLS; ++w) {
            cs[w] = acc;
            acc += count[w];
            most = std::max(most, count[w]);
            if (count[w])
                pv[w >> 5] |= 1u << (w & 31);
        }
        cs[HBG_NUM_CELLS] = acc;
        group_entries[g] = acc;
        G.n_entries = (int32_t)acc;
        G.max_cell = (int32_t)most;
        // expected hits per subject offset on typical proteins: entries of
        // words over the 20 standard letters, each such word taken as
        // equally likely (1 / 8000)
        static const uint8_t kStd[20] = {1, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15, 16, 17, 18, 19, 20, 22};
        uint64_t std_entries = acc;            // an upper bound, enough for most groups
        if ((double)std_entries / 8000.0 >= mode_hits) {
            std_entries = 0;
            for (int x = 0; x < 20; ++x)
                for (int y = 0; y < 20; ++y)
                    for (int z = 0; z < 20; ++z)
                        std_entries += count[(kStd[x] << 10) | (kStd[y] << 5) | kStd[z]];
        }
        if (mode_hits < kOffsetModeHits)
            G.mode = (double)std_entries / 8000.0 >= mode_hits ? 1 : 0;
    });
    int64_t entry_pos = 0;
    for (int32_t g = 0; g < n_groups; ++g) {
        b.groups[g].entry_base = entry_pos;
        entry_pos += group_entries[g];
    }
    b.entries.resize((size_t)entry_pos);
    parallel_for(n_groups, [&](int64_t gi) {
        const int32_t g = (int32_t)gi;
        const HbgGroup &G = b.groups[g];
        const uint8_t *gs = b.letters.data() + G.seq_base;
        const int32_t *gc = b.ctx_of.data() + G.seq_base;
        const uint32_t *cs = b.cells.data() + (size_t)g * HBG_CELL_STRIDE;
        // fill, ascending p inside each cell
        std::vector<uint32_t> cursor(cs, cs + HBG_NUM_CELLS);
        uint16_t *ge = b.entries.data() + G.entry_base;
        for (int32_t p = 0; p + HBG_WORD_SIZE <= G.glen; ++p) {
            if (!valid(gc, p))
                continue;
            const std::vector<uint16_t> &ws = nb.get(gs[p], gs[p + 1], gs[p + 2]);
            for (uint16_t w : ws)
                ge[cursor[w]++] = (uint16_t)p;
        }
    });
    undo.b = nullptr;
}

// --- six-frame translation ------------------------------------------------

namespace {
// Standard genetic code (NCBI transl_table 1), codons in TCAG order.
const char kStdCode[] = "FFLLSSSSYY**CC*WLLLLPPPPHHQQRRRRIIIMTTTTNNKKSSRRVVVVAAAADDEEGGGG";
const char kStdaa[] = "-ABCDEFGHIKLMNPQRSTVWXYZU*OJ";

struct CodonTable {
    uint8_t aa[64];
    CodonTable() {
        for (int i = 0; i < 64; ++i) {
            const char *p = strchr(kStdaa, kStdCode[i]);
            aa[i] = (uint8_t)(p - kStdaa);
        }
    }
};
const CodonTable kCodons;

// A=0 C=1 G=2 T=3 -> position in TCAG order; -1 for anything else
inline int tcag(uint8_t nt) {
    static const int8_t m[4] = {2, 1, 3, 0};
    return nt < 4 ? m[nt] : -1;
}
inline uint8_t codon(uint8_t a, uint8_t b, uint8_t c) {
    int x = tcag(a), y = tcag(b), z = tcag(c);
    if (x < 0 || y < 0 || z < 0)
        return 21;  // X
    return kCodons.aa[x * 16 + y * 4 + z];
}
inline uint8_t comp(uint8_t nt) { return nt < 4 ? (uint8_t)(3 - nt) : (uint8_t)4; }
}  // namespace

std::vector<uint8_t> translate_six_frames(const uint8_t *nt, int32_t n,
                                          std::vector<int32_t> *ctx_off,
                                          std::vector<int32_t> *ctx_len) {
    std::vector<uint8_t> out;
    out.reserve((size_t)(2 * n + 6));
    ctx_off->assign(6, 0);
    ctx_len->assign(6, 0);
    for (int f = 0; f < 6; ++f) {
        int32_t start = f % 3;
        int32_t len = n > start ? (n - start) / 3 : 0;
        if (f > 0)
            out.push_back(0);
        (*ctx_off)[f] = (int32_t)out.size();
        (*ctx_len)[f] = len;
        for (int32_t i = 0; i < len; ++i) {
            int32_t p = start + 3 * i;
            if (f < 3)
                out.push_back(codon(nt[p], nt[p + 1], nt[p + 2]));
            else
                out.push_back(codon(comp(nt[n - 1 - p]), comp(nt[n - 2 - p]),
                                    comp(nt[n - 3 - p])));
        }
    }
    return out;
}

}  // namespace hbg
