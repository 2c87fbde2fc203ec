"""Opening a database from host arrays: the letters are spread out and checked
on the device, a warp taking 1024 letters and a piece 64 MiB."""
import numpy as np
import pytest

import hblast
from hblast import synth
from test_gpu_parity import check

pytestmark = pytest.mark.gpu


def test_layout_with_empty_subjects_and_offset_start(built):
    rng = np.random.default_rng(1)
    q = synth.random_letters(rng, 200)
    lens = np.array([0, 0, 1, 1023, 1, 0, 1024, 1025, 0, 0, 3, 31, 32, 33, 0] + [int(x) for x in rng.integers(0, 700, 300)] + [0])
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    res = synth.random_letters(rng, int(off[-1]))
    for at in range(40, len(res) - 100, 400):
        res[at:at + 80] = synth.mutate(rng, q[60:140], 0.6)
    pqs = [hblast.ProteinQuery.blastp(q, 16, 30)]
    gdb = hblast.Database(res, off)
    assert gdb.info()[:2] == (len(lens), int(off[-1]))
    r = hblast.search(gdb, hblast.Batch.proteins(pqs))
    assert len(r.hsps) > 50
    check(r, pqs, res, off)
    # the same subjects, starting inside a larger array
    shifted = hblast.Database(np.concatenate([np.zeros(777, np.uint8), res]), off + 777)
    assert np.array_equal(hblast.search(shifted, hblast.Batch.proteins(pqs)).hsps, r.hsps)


def test_several_pieces(built):
    """More than one piece of letters: copies of one subject across the seam."""
    rng = np.random.default_rng(2)
    q = synth.random_letters(rng, 111)
    k = (64 << 20) // 111 + 2000
    score = int(sum(synth.blosum62()[a, a] for a in q))
    gdb = hblast.Database(np.tile(q, k), np.arange(k + 1, dtype=np.int64) * 111)
    h = hblast.search(gdb, hblast.Batch.proteins([hblast.ProteinQuery.blastp(q, 16, score)])).hsps
    assert np.array_equal(h["subject"], np.arange(k)) and (h["len"] == 111).all() and (h["s_start"] == 0).all()


@pytest.mark.parametrize("where", [0, 1, 499, 1023, 1024, 1025, 49_999])
@pytest.mark.parametrize("letter", [0, 28, 255])
def test_bad_letter_names_the_first_subject(built, where, letter):
    off = np.arange(0, 50_001, 50, dtype=np.int64)
    res = np.full(50_000, 1, np.uint8)
    res[where] = letter
    res[49_999] = 99
    with pytest.raises(hblast.HblastError, match=rf"subject {where // 50}: letter") as e:
        hblast.Database(res, off)
    assert e.value.code == -1


def test_bad_length_after_bad_letter(built):
    off = np.array([0, 10, 20, 15, 30], np.int64)
    res = np.full(30, 3, np.uint8)
    with pytest.raises(hblast.HblastError, match="subject 2: bad length"):
        hblast.Database(res, off)
    res[12] = 0
    with pytest.raises(hblast.HblastError, match="subject 1: letter"):
        hblast.Database(res, off)
