"""The shared-memory word finder at the edges of its ranges: table sizes (16- and
8-bit cells, up to the longest query), two-hit windows, subject lengths
around its chunks, sweeps and position limits, X-drop extremes, and the batches
it leaves to the general kernel.  Bit-exact against the CPU oracle (integer
work, tolerance 0)."""
import numpy as np
import pytest

import hblast
from hblast import synth
from oracle import oracle
from test_gpu_parity import check, contexts_query
from test_host import smallbone_from_csr

pytestmark = pytest.mark.gpu


def database(rng, q, extra=()):
    """Subjects of every length 1..70 and some around a sweep, cut from mutated
    copies of q, so that they hold hits, and a few of the given lengths."""
    lens = list(range(1, 71)) + [150, 191, 192, 193, 206, 207, 208, 248, 249, 300, 1000, 3000] + list(extra)
    subs = []
    for n in lens:
        s = synth.random_letters(rng, n)
        for at in range(0, n, 160):
            m = min(n - at, 90, len(q))
            a = int(rng.integers(0, len(q) - m + 1))
            s[at:at + m] = synth.mutate(rng, q[a:a + m], rng.uniform(0.4, 1.0))
        subs.append(s)
    off = np.zeros(len(subs) + 1, np.int64)
    off[1:] = np.cumsum([len(s) for s in subs])
    return np.concatenate(subs), off


@pytest.mark.parametrize("qlen,window", [(3, 40), (24, 40), (25, 40), (700, 5), (700, 4), (700, 64), (700, 65), (2008, 40),
                                         (2009, 40), (4056, 40), (4057, 40), (8152, 40), (8152, 7), (8153, 40), (16341, 40),
                                         (16345, 64), (33000, 40), (65000, 64)])
def test_table_edges(built, qlen, window):
    rng = np.random.default_rng(qlen + window)
    q = synth.random_letters(rng, qlen)
    res, off = database(rng, q)
    pqs = [hblast.ProteinQuery.blastp(q, 16, 20)]
    gdb = hblast.Database(res, off)
    got = hblast.search(gdb, hblast.Batch.proteins(pqs, window=window))
    # check() compares with the default window
    ref, subj, cnt = oracle.search(oracle.Query.blastp(q, 16, 20), res, off, window=window)
    h = got.hsps
    assert len(h) == len(ref) and np.array_equal(h["subject"], subj)
    for f, g in (("q_start", "q_start"), ("s_start", "s_start"), ("q_off", "q_off"), ("s_off", "s_off"),
                 ("len", "len"), ("score", "score")):
        assert np.array_equal(h[g], ref[f]), f
    st = got.stats[0]
    assert (st["lookup_hits"], st["init_extends"], st["good_init_extends"]) == tuple(int(c) for c in cnt)


@pytest.mark.parametrize("qlen,lens", [(300, (32725, 32726, 32727, 32766, 40000)), (5000, (32726, 65534, 65535, 65536, 70000))])
def test_long_subjects(built, qlen, lens):
    """Subjects at and past the largest position a cell holds: the longer ones
    go to the general kernel, all in one result."""
    rng = np.random.default_rng(qlen)
    q = synth.random_letters(rng, qlen)
    res, off = database(rng, q, lens)
    pqs = [hblast.ProteinQuery.blastp(q, 16, 30)]
    check(hblast.search(hblast.Database(res, off), hblast.Batch.proteins(pqs)), pqs, res, off)


def test_many_tiny_subjects_and_repeats(built):
    """Hundreds of subjects of a few letters in a row (flag codes of the 8-bit
    cells go round), low-complexity subjects and queries: long chains on one
    diagonal, blocked hits, cells of about a thousand entries and more."""
    rng = np.random.default_rng(5)
    unit = synth.random_letters(rng, 11)
    q8 = np.concatenate([np.tile(unit, 40), synth.random_letters(rng, 5000)])
    subs = [q8[a:a + int(rng.integers(3, 9))] for a in rng.integers(0, 5000, 900)]
    subs += [np.tile(unit, int(rng.integers(2, 30))) for _ in range(60)]
    subs += [np.full(n, 11, np.uint8) for n in (3, 40, 500)]
    off = np.zeros(len(subs) + 1, np.int64)
    off[1:] = np.cumsum([len(s) for s in subs])
    res = np.concatenate(subs)
    pqs = [hblast.ProteinQuery.blastp(x, 16, 20) for x in
           (q8, np.tile(unit, 60), np.full(1000, 11, np.uint8), np.full(1030, 11, np.uint8))]
    gdb = hblast.Database(res, off)
    for k, pq in enumerate(pqs):
        check(hblast.search(gdb, hblast.Batch.proteins([pq])), [pq], res, off)


@pytest.mark.parametrize("xdrop", [0, 1, 7, 200])
def test_xdrop_extremes(built, xdrop):
    rng = np.random.default_rng(xdrop)
    parts = [synth.random_letters(rng, n) for n in (40, 300, 5)]
    pq = contexts_query(parts, [xdrop] * 3, [11, 25, 11])
    res, off = database(rng, parts[1])
    check(hblast.search(hblast.Database(res, off), hblast.Batch.proteins([pq])), [pq], res, off)


def test_table_with_repeated_offsets(built):
    """A caller's own table that lists offsets twice: the second hit in one
    place changes nothing."""
    rng = np.random.default_rng(9)
    q = synth.random_letters(rng, 200)
    res, off = database(rng, q)
    pq = hblast.ProteinQuery.blastp(q, 16, 20)
    cs, ents = oracle.lookup_table(oracle.Query.blastp(q, 16, 20), 11)

    def table(rep):
        return hblast.Batch.from_smallbone(pq, *smallbone_from_csr(cs * rep, np.repeat(ents, rep)))

    gdb = hblast.Database(res, off)
    one, two = hblast.search(gdb, table(1)), hblast.search(gdb, table(2))
    assert len(one.hsps) > 0
    assert np.array_equal(one.hsps, two.hsps)
    check(one, [pq], res, off)


def test_groups_of_different_lengths(built):
    """8-bit tables of one launch have their groups' lengths, and a warp goes
    from group to group with what the last one left in its table: here from a
    long masked group, soon done, to a shorter one and on to a long one."""
    rng = np.random.default_rng(21)
    qs = [np.concatenate([np.full(5500, 21, np.uint8), synth.random_letters(rng, 2500)])]
    qs += [synth.random_letters(rng, n) for n in (4100, 8100)]
    db = synth.make_db(rng, 15000, 300, 0.6, 30, 3000, 0.01, qs[1:], 100, 0.5)
    pqs = [hblast.ProteinQuery.blastp(q) for q in qs]
    check(hblast.search(hblast.Database(db.residues, db.offsets), hblast.Batch.proteins(pqs)), pqs, db.residues,
          db.offsets, threads=16)


@pytest.mark.parametrize("threshold,qlens", [(8, (300,)), (9, (700, 40, 3, 2)), (11, (33, 34, 35, 1500)), (14, (64, 65)),
                                             (30, (50,)), (-400, (3, 5))])
def test_device_built_tables(built, threshold, qlens):
    """Lookup tables built on the device, from thresholds whose entries outgrow
    the block they are given (-400: every word of 28 letters is a neighbour) to
    none at all: hits, extensions and HSPs as the oracle finds them."""
    rng = np.random.default_rng(threshold + 1000)
    qs = [synth.random_letters(rng, n) for n in qlens]
    res, off = database(rng, qs[0] if len(qs[0]) > 10 else synth.random_letters(rng, 90))
    pqs = [hblast.ProteinQuery.blastp(q, 16, 20) for q in qs]
    got = hblast.search(hblast.Database(res, off), hblast.Batch.proteins(pqs, threshold=threshold))
    for k, q in enumerate(qs):
        ref, subj, cnt = oracle.search(oracle.Query.blastp(q, 16, 20), res, off, threshold=threshold)
        h = got.hsps[got.hsps["query"] == k]
        assert len(h) == len(ref) and np.array_equal(h["subject"], subj)
        for f in ("q_start", "s_start", "q_off", "s_off", "len", "score"):
            assert np.array_equal(h[f], ref[f]), f
        st = got.stats[k]
        assert (st["lookup_hits"], st["init_extends"], st["good_init_extends"]) == tuple(int(c) for c in cnt)


@pytest.mark.parametrize("xdrop", [1 << 24, (1 << 24) + 1, (1 << 27) - 1, 1 << 27, 1 << 28, (1 << 28) + 1, 2**31 - 1])
@pytest.mark.parametrize("qlen", [300, 5000])
def test_xdrop_without_limit(built, xdrop, qlen):
    """X-drops so large that no walk ends by them, the plain way to ask for
    none, with either size of cells."""
    rng = np.random.default_rng(qlen)
    parts = [synth.random_letters(rng, n) for n in (40, qlen, 5)]
    pq = contexts_query(parts, [xdrop, 16, xdrop], [11, 25, 11])
    res, off = database(rng, parts[0])
    check(hblast.search(hblast.Database(res, off), hblast.Batch.proteins([pq])), [pq], res, off)
    pq = contexts_query(parts, [xdrop] * 3, [30] * 3)
    res, off = database(rng, parts[1])
    check(hblast.search(hblast.Database(res, off), hblast.Batch.proteins([pq])), [pq], res, off)


@pytest.mark.parametrize("form", ["tiles", "tile bytes", "threads", "offset", "team", "window"])
def test_general_kernel_takes_long_groups_together(built, form):
    """Groups of every table length, left to the general kernel by the caller's
    choice or by the window: those with global tables share one launch against
    a small database."""
    rng = np.random.default_rng(31)
    qs = [synth.random_letters(rng, n) for n in (2500, 5000, 9000, 17000)]
    res, off = database(rng, qs[0])
    pqs = [hblast.ProteinQuery.blastp(q, 16, 20) for q in qs]
    gdb = hblast.Database(res, off)
    window = 70 if form == "window" else 40
    b = hblast.Batch.proteins(pqs, window=window, max_group_len=1)
    if form == "tiles":
        b.tune(64)
    if form == "tile bytes":
        b.schedule(1, 65536)
    if form == "team":
        b.schedule(3)
    if form == "offset":
        b.set_mode(1)
    s = hblast.Searcher(gdb, b, hblast.default_options(num_threadsx=128) if form == "threads" else None)
    s.launch()
    s.wait()
    assert s.timing()[2] == 2                    # the word finder and the ordering
    got = s.result()
    if window == 40:
        check(got, pqs, res, off)
    else:
        other = hblast.search(gdb, hblast.Batch.proteins(pqs, window=window, max_group_len=1).tune(64))
        assert len(got.hsps) > 0 and np.array_equal(got.hsps, other.hsps) and got.stats == other.stats


@pytest.mark.parametrize("n_groups,n_subjects", [(151, 30), (153, 30), (770, 30), (1700, 30), (608, 20), (609, 20), (1700, 2)])
def test_many_groups_few_subjects(built, n_groups, n_subjects):
    """More groups than CTAs and than a CTA has threads, against databases of
    about as many subjects as a CTA has warps: every query as the general kernel
    has it, and a few as the oracle."""
    rng = np.random.default_rng(n_groups)
    qs = [synth.random_letters(rng, int(n)) for n in rng.integers(20, 70, n_groups)]
    subs = [np.concatenate([synth.mutate(rng, qs[int(i)], 0.8) for i in rng.integers(0, n_groups, 12)]) for _ in range(n_subjects)]
    off = np.zeros(n_subjects + 1, np.int64)
    off[1:] = np.cumsum([len(s) for s in subs])
    res = np.concatenate(subs)
    gdb = hblast.Database(res, off)
    pqs = [hblast.ProteinQuery.blastp(q, 16, 25) for q in qs]
    got = hblast.search(gdb, hblast.Batch.proteins(pqs, max_group_len=1))
    ref = hblast.search(gdb, hblast.Batch.proteins(pqs, max_group_len=1).tune(8))
    assert len(got.hsps) > n_subjects and np.array_equal(got.hsps, ref.hsps) and got.stats == ref.stats
    for k in (0, 1, n_groups // 2, n_groups - 1):
        hsps, subj, cnt = oracle.search(oracle.Query.blastp(qs[k], 16, 25), res, off)
        mine = got.for_query(k)
        assert len(mine) == len(hsps) and np.array_equal(mine["subject"], subj)
        assert np.array_equal(mine["score"], hsps["score"]) and np.array_equal(mine["s_start"], hsps["s_start"])
        st = got.stats[k]
        assert (st["lookup_hits"], st["init_extends"], st["good_init_extends"]) == tuple(int(c) for c in cnt)


@pytest.mark.parametrize("qlens,lens", [((300,), (32727,)), ((300, 2000, 4000, 5000), (32726, 32727, 40000, 65535, 65536, 70000)),
                                        ((5000, 20), (65536,) * 20)])
@pytest.mark.parametrize("own_stream", [False, True])
def test_long_subjects_beside_the_others(built, qlens, lens, own_stream):
    """Subjects too long for the cells are searched on a stream of their own beside
    the others: the same result from the first launch, a captured one and its replays."""
    import torch
    rng = np.random.default_rng(len(qlens))
    qs = [synth.random_letters(rng, n) for n in qlens]
    res, off = database(rng, qs[0], lens)
    pqs = [hblast.ProteinQuery.blastp(q, 16, 30) for q in qs]
    gdb = hblast.Database(res, off)
    s = hblast.Searcher(gdb, hblast.Batch.proteins(pqs))
    stream = torch.cuda.Stream() if own_stream else None
    first = None
    for _ in range(4):
        s.launch(stream.cuda_stream if stream else None)
        s.wait()
        got = s.result()
        if first is None:
            first = got
            check(got, pqs, res, off, threads=16)
        assert np.array_equal(got.hsps, first.hsps) and got.stats == first.stats


@pytest.mark.parametrize("own_table", [False, True])
@pytest.mark.parametrize("qlen", [1024, 1025, 1026, 1800, 4000, 9000])
def test_cells_of_a_thousand_entries_and_more(built, qlen, own_table):
    """A packed cell counts to 1022; here 1022, 1023, 1024 and more query offsets
    share a word, in tables built on the device and in a caller's own."""
    rng = np.random.default_rng(qlen)
    q = np.concatenate([np.full(qlen, 11, np.uint8), synth.random_letters(rng, 60)])
    subs = [np.full(n, 11, np.uint8) for n in (3, 4, 35, 70)]
    subs += [np.concatenate([synth.random_letters(rng, 50), np.full(n, 11, np.uint8), q[-55:]]) for n in (0, 3, 10, 40)]
    subs += [synth.random_letters(rng, 300)]
    off = np.zeros(len(subs) + 1, np.int64)
    off[1:] = np.cumsum([len(s) for s in subs])
    res = np.concatenate(subs)
    pq = hblast.ProteinQuery.blastp(q, 16, 30)
    gdb = hblast.Database(res, off)
    if own_table:
        cs, ents = oracle.lookup_table(oracle.Query.blastp(q, 16, 30), 11)
        batch = hblast.Batch.from_smallbone(pq, *smallbone_from_csr(cs, ents))
    else:
        batch = hblast.Batch.proteins([pq])
    check(hblast.search(gdb, batch), [pq], res, off)


@pytest.mark.parametrize("lens", [(5000, 9000), (20, 100, 300, 900, 2000, 4000, 5000, 9000, 17000), (4000, 17000, 33000)])
@pytest.mark.parametrize("own_stream", [False, True])
def test_launches_side_by_side(built, lens, own_stream):
    """One launch per table length, side by side on up to four streams, 8-bit ones
    with flag ends of their own: as the oracle, and the same in every repetition."""
    import torch
    rng = np.random.default_rng(len(lens))
    qs = [synth.random_letters(rng, n) for n in lens]
    res, off = database(rng, np.concatenate(qs), (5000, 20000))
    pqs = [hblast.ProteinQuery.blastp(q, 16, 25) for q in qs]
    s = hblast.Searcher(hblast.Database(res, off), hblast.Batch.proteins(pqs, threshold=10, max_group_len=1))
    stream = torch.cuda.Stream() if own_stream else None
    first = None
    for _ in range(6):
        s.launch(stream.cuda_stream if stream else None)
        s.wait()
        got = s.result()
        if first is None:
            assert s.timing()[2] == len(lens) + 1
            first = got
            for k, q in enumerate(qs):
                ref, subj, cnt = oracle.search(oracle.Query.blastp(q, 16, 25), res, off, threshold=10, nthreads=8)
                mine = got.for_query(k)
                assert len(mine) == len(ref) and np.array_equal(mine["subject"], subj)
                for f in ("q_start", "s_start", "q_off", "s_off", "len", "score"):
                    assert np.array_equal(mine[f], ref[f]), (k, f)
                st = got.stats[k]
                assert (st["lookup_hits"], st["init_extends"], st["good_init_extends"]) == tuple(int(c) for c in cnt)
        assert np.array_equal(got.hsps, first.hsps) and got.stats == first.stats
