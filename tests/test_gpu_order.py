"""The ordering pass around the number of HSPs where it changes from ranking
every one against all others to the radix sort, and at the remainders of the
sort's rounds.  The database holds k copies of a query, so the HSPs are known:
one per query and subject, the whole query."""
import numpy as np
import pytest

import hblast
from hblast import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k,nq", [(1, 1), (31, 1), (1024, 1), (1025, 1), (341, 3), (342, 3), (4863, 1), (4865, 2), (16383, 1),
                                  (16384, 1), (16385, 1), (8192, 2), (3001, 7),
                                  (70001, 2), (1300003, 1)])
def test_order_of_known_hsps(built, k, nq):
    q = synth.random_letters(np.random.default_rng(3), 60)
    m = synth.blosum62()
    score = int(sum(m[a, a] for a in q))
    gdb = hblast.Database(np.tile(q, k), np.arange(k + 1, dtype=np.int64) * 60)
    # the cutoff leaves only the query's own diagonal
    pqs = [hblast.ProteinQuery.blastp(q, 16, score) for _ in range(nq)]
    res = hblast.search(gdb, hblast.Batch.proteins(pqs))
    h = res.hsps
    assert len(h) == k * nq
    assert np.array_equal(h["query"], np.repeat(np.arange(nq), k))
    assert np.array_equal(h["subject"], np.tile(np.arange(k), nq))
    for f, v in (("q_start", 0), ("s_start", 0), ("len", 60), ("score", score), ("context", 0)):
        assert (h[f] == v).all(), f
    for f in ("q_off", "s_off"):
        assert (h[f] == h[f][0]).all() and np.array_equal(h["q_off"], h["s_off"])
    for st in res.stats:
        assert st["subjects_passed"] == k and st["good_init_extends"] == k
