"""What a search asks of the device and the host beside its result: its memory,
hbg_mem_required against what the device hands out (in a process of its own so that
no buffer of an earlier search is used again), and no waiting for other searches."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import hblast
from hblast import synth
from test_gpu_parity import check

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parent.parent

_SEARCH = """
import sys
sys.path[:0] = {paths!r}
import ctypes as C
import numpy as np, torch, hblast
from hblast import synth
n, qlen, extra = {args!r}
rng = np.random.default_rng(n)
db = synth.make_db(rng, 1000, 300, 0.6, 30, 5000, 0, [synth.random_letters(rng, 300)], 100, 0.5)
res, off = db.residues, db.offsets
if extra:
    res, off = np.concatenate([res, synth.random_letters(rng, extra)]), np.append(off, off[-1] + extra)
gdb = hblast.Database(res, off)
batch = hblast.Batch.proteins([hblast.ProteinQuery.blastp(synth.random_letters(rng, qlen)) for _ in range(n)])
need = C.c_int64()
assert hblast.lib().hbg_mem_required(gdb.handle, batch.handle, 1 << 20, C.byref(need)) == 0
torch.cuda.synchronize()
before = torch.cuda.mem_get_info()[0]
s = hblast.Searcher(gdb, batch, hsp_capacity=1 << 20)
s.launch()
s.sync()
print(need.value, before - torch.cuda.mem_get_info()[0], batch.info()["device_bytes"])
"""


@pytest.mark.parametrize("n,qlen,extra", [(1, 300, 0), (4000, 60, 0), (64, 1500, 0), (1, 20000, 0), (1, 65000, 0),
                                          (1, 300, 40000), (1, 20000, 70000)])
def test_memory_required_is_what_a_search_takes(built, n, qlen, extra):
    """The device gives memory in blocks of 2 MiB, a dozen of them here, and the
    kernels' code may be loaded at their first launch: 64 MiB of room either way."""
    code = _SEARCH.format(paths=[str(ROOT / "h-blast_gb300"), str(ROOT)], args=(n, qlen, extra))
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr
    need, taken, batch = map(int, r.stdout.split())
    room = 64 << 20
    assert batch <= need
    assert taken <= need + room, (need, taken)
    assert need <= taken + room, (need, taken)


def test_first_search_of_a_batch_does_not_wait_for_another(built):
    """While a search of 50 ms and more runs on one stream, a new batch is searched
    on two others: the launches return while the first search still runs, and the
    results are right although the batch's tables are built behind it."""
    import torch
    qs, db = synth.batched_blastp(seed=7, n_queries=64, n_subjects=200_000)
    gdb = hblast.Database(db.residues, db.offsets)
    long = hblast.Searcher(gdb, hblast.Batch.proteins([hblast.ProteinQuery.blastp(q) for q in qs]))
    first, second, third = (torch.cuda.Stream() for _ in range(3))
    pqs = [hblast.ProteinQuery.blastp(q[:200]) for q in qs[:2]]
    want = hblast.search(gdb, hblast.Batch.proteins(pqs), hsp_capacity=1 << 20)      # (and buffers for the next ones)
    check(want, pqs, db.residues, db.offsets, threads=16)
    long.launch(first.cuda_stream)
    long.sync()
    for _ in range(3):
        batch = hblast.Batch.proteins(pqs)
        a, b = (hblast.Searcher(gdb, batch, hsp_capacity=1 << 20) for _ in range(2))
        long.launch(first.cuda_stream)
        a.launch(second.cuda_stream)
        b.launch(third.cuda_stream)
        assert not first.query()
        for s in (b, a):
            s.wait()
            got = s.result()
            assert np.array_equal(got.hsps, want.hsps) and got.stats == want.stats
            s.close()
        batch.close()
        long.sync()


def test_batch_may_go_before_its_result(built):
    """hbg_batch_destroy waits for the device: a search that it ends is then read
    without the batch."""
    rng = np.random.default_rng(3)
    q = synth.random_letters(rng, 400)
    db = synth.make_db(rng, 2000, 300, 0.6, 30, 3000, 0.05, [q], 100, 0.6)
    gdb = hblast.Database(db.residues, db.offsets)
    pqs = [hblast.ProteinQuery.blastp(q)]
    s = hblast.Searcher(gdb, hblast.Batch.proteins(pqs))
    s.launch()
    s.batch.close()
    more = [hblast.Batch.proteins(pqs * 50) for _ in range(20)]      # over the freed batch
    s.sync()
    assert s.n_hsps() > 0
    s.wait()
    check(s.result(), pqs, db.residues, db.offsets)
    s.close()
    del more


def test_threads_capture_and_destroy(built):
    """Four threads that launch kept results again, which captures a graph, and
    destroy batches, which waits for the device: neither disturbs the other."""
    import threading

    import torch
    rng = np.random.default_rng(8)
    qs = [synth.random_letters(rng, n) for n in (60, 300, 900, 2500, 6000)]
    db = synth.make_db(rng, 2000, 300, 0.6, 30, 3000, 0.05, qs, 50, 0.6)
    gdb = hblast.Database(db.residues, db.offsets)
    pqs = [hblast.ProteinQuery.blastp(q, 16, 30) for q in qs]
    want = {n: hblast.search(gdb, hblast.Batch.proteins(pqs[:n], max_group_len=1)) for n in range(1, 6)}
    check(want[5], pqs, db.residues, db.offsets, threads=16)
    faults = []

    def work(k):
        stream = torch.cuda.Stream()
        try:
            for i in range(40):
                n = 1 + (i + k) % 5
                batch = hblast.Batch.proteins(pqs[:n], max_group_len=1)
                s = hblast.Searcher(gdb, batch)
                for _ in range(3):
                    s.launch(stream.cuda_stream)
                    s.wait()
                    got = s.result()
                    if not np.array_equal(got.hsps, want[n].hsps) or got.stats != want[n].stats:
                        faults.append((k, i))
                s.close()
                batch.close()
        except Exception as e:
            faults.append((k, repr(e)))

    threads = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not faults
