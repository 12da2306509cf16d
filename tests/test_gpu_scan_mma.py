"""The scan whose comparison runs on the tensor cores (csrc/scan_mma.cuh)
against the POPC scan and the oracle, at the sizes where it can go wrong: one
pattern, the edges of 16 pattern rows and of 64 accumulator columns, sets too
large for shared memory, 20 and 31 compared cells, batches, slices, and an
overflowing hit list.  Rows are text, so every comparison is exact."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu
MMA = "13"
SHAPES = {f: (f, mk, mm) for f, mk, mm in randgen.REQUEST_SHAPES}


def _rows(text):
    return sorted(text.splitlines())


def _genome(cof_mod, records, seed=2, max_chunk=5000):
    g = cof_mod.Genome()
    for name, data, _nibs, s, e in randgen.chunk_records(random.Random(seed), records, max_chunk):
        g.add_chunk(name, data, s, e)
    return g


def _guides(rng, n, mk, length=25):
    return [mk("".join(rng.choice("ACGT") for _ in range(length))) for _ in range(n)]


def _same(monkeypatch, g, *args, **kw):
    monkeypatch.setenv("COF_SCAN_VARIANT", "0")
    ref = g.search(*args, **kw)
    monkeypatch.setenv("COF_SCAN_VARIANT", MMA)
    got = g.search(*args, **kw)
    assert g.tuning()["last"].startswith("mma-f8")
    assert got == ref
    return got


@pytest.mark.parametrize("n_pat", [1, 15, 16, 17, 48, 63, 64, 65, 81, 128, 129])
@pytest.mark.parametrize("shape", sorted(SHAPES))
def test_pattern_counts_and_shapes(cof_mod, monkeypatch, n_pat, shape):
    filt, mk, mm = SHAPES[shape]
    rng = random.Random(10 * n_pat + len(filt))
    _, records = randgen.random_genome(rng, 3, 20000, 40000)
    pats = _guides(rng, n_pat, mk)
    for p in pats[:8]:
        randgen.plant_sites(rng, records, p.upper(), filt, 6, mm)
    _same(monkeypatch, _genome(cof_mod, records), filt, pats, mm + 3)


@pytest.mark.parametrize("guide_len", [17, 20, 21, 25, 28, 29, 31, 40])
def test_compared_cells(cof_mod, oracle_mod, monkeypatch, guide_len):
    # up to 20 compared cells take two K steps, up to 31 three; of 32 (a
    # window-filling pattern) one is left to the exact decision
    rng = random.Random(guide_len)
    _, records = randgen.random_genome(rng, 2, 30000, 40000)
    for filt, pre, post in (("N" * (guide_len + 1) + "RG", "", "NNN"),
                            ("TTTN" + "N" * guide_len, "NNNN", ""), ("N" * guide_len, "", "")):
        pats = [pre + p + post for p in _guides(rng, 20, lambda x: x, guide_len)]
        for p in pats:
            randgen.plant_sites(rng, records, p, filt, 3, 4)
        g = _genome(cof_mod, records)
        text, n = _same(monkeypatch, g, filt, pats, 5)
        o = oracle_mod.OracleGenome()
        for name, data, _nibs, s, e in randgen.chunk_records(random.Random(2), records, 5000):
            o.add_chunk(name, data, s, e)
        ref, nref = o.search(filt, pats, 5)
        assert n == nref > 0 and _rows(text) == _rows(ref)


@pytest.mark.parametrize("n_pat,guide_len", [(1300, 20), (700, 25)])
def test_sets_beyond_shared_memory(cof_mod, monkeypatch, n_pat, guide_len):
    rng = random.Random(n_pat)
    _, records = randgen.random_genome(rng, 2, 20000, 30000)
    filt = "N" * (guide_len + 1) + "RG"
    pats = _guides(rng, n_pat, lambda x: x + "NNN", guide_len)
    for p in pats[::50] + pats[-2:]:
        randgen.plant_sites(rng, records, p, filt, 2, 3)
    assert _same(monkeypatch, _genome(cof_mod, records), filt, pats, 5)[1] > 0


@pytest.mark.parametrize("cps", [0, 2, 3])
def test_batch_of_mixed_requests(cof_mod, monkeypatch, cps):
    # sets of different PAMs, lengths and limits in one pass, and many batch
    # segments (small chunks_per_search), with a row block per batch
    rng = random.Random(90 + cps)
    _, records = randgen.random_genome(rng, 3, 20000, 40000)
    reqs = []
    for filt, mk, mm in randgen.REQUEST_SHAPES:
        pats = _guides(rng, rng.randint(1, 40), mk)
        for p in pats:
            randgen.plant_sites(rng, records, p.upper(), filt, 2, 2)
        reqs.append(dict(search_filter=filt, patterns=pats, max_mismatches=mm, chunks_per_search=cps))
    for n in (17, 22, 25):
        reqs.append(dict(search_filter="N" * (n + 1) + "RG",
                         patterns=_guides(rng, 9, lambda x: x[:n] + "NNN"), max_mismatches=n % 5,
                         chunks_per_search=cps))
    g = _genome(cof_mod, records, max_chunk=400)
    monkeypatch.setenv("COF_SCAN_VARIANT", "0")
    ref = g.search_batch(reqs)
    monkeypatch.setenv("COF_SCAN_VARIANT", MMA)
    assert g.search_batch(reqs) == ref and sum(n for _, n in ref) > 0
    assert g.tuning()["last"].startswith("mma-f8")


def test_hit_list_overflow_and_slices(cof_mod, monkeypatch):
    rng = random.Random(4)
    _, records = randgen.random_genome(rng, 3, 30000, 50000)
    pats = _guides(rng, 70, lambda x: x[:20] + "NNN")
    monkeypatch.setenv("COF_CAND_CAP", "64")
    g = _genome(cof_mod, records)
    monkeypatch.setenv("COF_SCAN_VARIANT", MMA)
    text, n = g.search("N" * 21 + "RG", pats, 9)
    assert g.last_stats()["raw_hits"] > 64
    monkeypatch.setenv("COF_SLICE_NT", "7000")
    assert g.search("N" * 21 + "RG", pats, 9) == (text, n)
    assert g.tuning()["slices"] > 5 and g.tuning()["last"].startswith("mma-f8")
    monkeypatch.delenv("COF_SLICE_NT")
    monkeypatch.setenv("COF_SCAN_VARIANT", "0")
    assert g.search("N" * 21 + "RG", pats, 9) == (text, n)


@pytest.mark.parametrize("guides,mm,mma", [(63, 4, False), (64, 4, True), (64, 12, False)])
def test_rule(cof_mod, monkeypatch, guides, mm, mma):
    # from 64 patterns per set on, unless hits are common
    monkeypatch.delenv("COF_SCAN_VARIANT", raising=False)
    rng = random.Random(guides + mm)
    _, records = randgen.random_genome(rng, 2, 20000, 30000)
    g = _genome(cof_mod, records)
    g.search("N" * 21 + "RG", _guides(rng, guides, lambda x: x[:20] + "NNN"), mm)
    assert g.tuning()["last"].startswith("mma-f8") == mma


@pytest.mark.parametrize("size", [1000, 1025, 4095, 4097, 5119, 8193, 12289])
def test_steps_of_four_tiles(cof_mod, monkeypatch, size):
    # segments that end inside, at and just after a step's four tiles, with more
    # than a row block of passing starts in a step and fewer than one
    rng = random.Random(size)
    records = [randgen.random_seq(rng, size - 1 + i) for i in range(3)]
    for filt, mk in (("N" * 21 + "RG", lambda x: x + "NNN"), ("TTTN" + "N" * 20, lambda x: "NNNN" + x)):
        pats = _guides(rng, 70, mk, 20)
        for p in pats[:8]:
            randgen.plant_sites(rng, records, p.upper(), filt, 2, 3)
        _same(monkeypatch, _genome(cof_mod, records, max_chunk=2 * size), filt, pats, 6)
