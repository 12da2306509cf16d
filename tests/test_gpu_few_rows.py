"""Passes of few hits, whose rows one block takes from the scan's hit list to
text in host memory (few_rows_kernel): the edges of its hit list, of its text
stage and of its requests, against the general path and the oracle.  Rows are
text: comparisons are exact."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu
FILT = "N" * 21 + "RG"


def _genome(cls, chunks):
    g = cls()
    for name, data, _nibs, s, e in chunks:
        g.add_chunk(name, data, s, e)
    return g


def _site_genome(rng, site, n, name="chr"):
    """n copies of `site`, 7 to 40 cells apart, in one record of even chunks."""
    seq = "".join(site + "".join(rng.choice("CT") for _ in range(rng.randint(7, 40))) for _ in range(n))
    return [(name, *randgen.pack(seq[s:s + 3000]), s, min(s + 3000, len(seq)))
            for s in range(0, len(seq), 3000)]


@pytest.mark.parametrize("n", [1, 31, 32, 33, 511, 512, 513, 1023, 1024, 1025, 3000])
def test_hit_list_edges(cof_mod, oracle_mod, n):
    rng = random.Random(n)
    guide = "".join(rng.choice("AG") for _ in range(20))
    chunks = _site_genome(rng, guide + "TGG", n)
    g, o = _genome(cof_mod.Genome, chunks), _genome(oracle_mod.OracleGenome, chunks)
    text, rows = g.search(FILT, [guide + "NNN"], 1)
    ref, nref = o.search(FILT, [guide + "NNN"], 1)
    assert rows == nref >= n and sorted(text.splitlines()) == sorted(ref.splitlines())
    # a pass with another, matchless request gives the same text
    other = dict(search_filter=FILT, patterns=["C" * 20 + "NNN"], max_mismatches=0)
    both = g.search_batch([other, dict(search_filter=FILT, patterns=[guide + "NNN"], max_mismatches=1)])
    assert both == [("", 0), (text, rows)]


@pytest.mark.parametrize("name_len", [0, 1, 400])
def test_long_record_names_and_text_stage(cof_mod, oracle_mod, name_len):
    # 300 rows of about 470 bytes pass the 96 KB stage: the general path
    rng = random.Random(name_len)
    guide = "".join(rng.choice("AG") for _ in range(20))
    chunks = _site_genome(rng, guide + "TGG", 300, "n" * name_len)
    g, o = _genome(cof_mod.Genome, chunks), _genome(oracle_mod.OracleGenome, chunks)
    text, rows = g.search(FILT, [guide + "NNN"], 1)
    ref, nref = o.search(FILT, [guide + "NNN"], 1)
    assert rows == nref >= 300 and sorted(text.splitlines()) == sorted(ref.splitlines())


@pytest.mark.parametrize("n_reqs", [1, 2, 255, 256, 257])
def test_requests_of_a_pass(cof_mod, n_reqs):
    rng = random.Random(n_reqs)
    _, records = randgen.random_genome(rng, 3, 20000, 40000)
    reqs = []
    for i in range(n_reqs):
        p = "".join(rng.choice("ACGT") for _ in range(20)) + "NNN"
        if i % 3 == 0:
            randgen.plant_sites(rng, records, p, FILT, 2, 2)
        reqs.append(dict(search_filter=FILT, patterns=[p], max_mismatches=2))
    g = _genome(cof_mod.Genome, randgen.chunk_records(rng, records, 2500))
    batch = g.search_batch(reqs)
    assert sum(n for _, n in batch) > 0
    for r, got in list(zip(reqs, batch))[:: max(1, n_reqs // 40)]:
        assert g.search_batch([r])[0] == got
    pieces = {}
    counts = g.search_stream(reqs, lambda req, text, n, _m: pieces.setdefault(req, []).append((text, n)))
    assert counts == [n for _, n in batch]
    for i, (text, n) in enumerate(batch):
        assert b"".join(t for t, _ in pieces.get(i, [])).decode() == text
        assert sum(k for _, k in pieces.get(i, [])) == n


def test_cancel_and_overflow(cof_mod, monkeypatch):
    rng = random.Random(3)
    guide = "".join(rng.choice("AG") for _ in range(20))
    chunks = _site_genome(rng, guide + "TGG", 400)
    g = _genome(cof_mod.Genome, chunks)
    req = dict(search_filter=FILT, patterns=[guide + "NNN"], max_mismatches=1)
    with pytest.raises(cof_mod.CofError) as e:
        g.search_stream([req], lambda *a: True)
    assert e.value.code == cof_mod.COF_E_CANCELLED
    want = g.search_batch([req])
    monkeypatch.setenv("COF_CAND_CAP", "64")  # the hit list overflows and grows
    assert _genome(cof_mod.Genome, chunks).search_batch([req]) == want
