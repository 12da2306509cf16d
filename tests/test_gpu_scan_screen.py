"""The screened scan of one or two guides and few mismatches
(scan_screen_kernel) against scan_direct_kernel and the oracle: PAMs, lengths,
every limit it takes and the first it does not, IUPAC guides, batches, slices
and an overflowing hit list.  Rows are text: comparisons are exact."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu
PAMS = [("", "NRG"), ("", "NNGRRT"), ("TTTN", ""), ("", "NGG"), ("", "NNAGAAW")]


def _chunks(records, seed=2, max_chunk=5000):
    return randgen.chunk_records(random.Random(seed), records, max_chunk)


def _genome(cls, chunks):
    g = cls()
    for name, data, _nibs, s, e in chunks:
        g.add_chunk(name, data, s, e)
    return g


def _request(rng, pre, post, n_guides, length):
    guides = ["".join(rng.choice("ACGT") for _ in range(length)) for _ in range(n_guides)]
    return (pre + "N" * length + post,
            ["N" * len(pre) + g + "N" * len(post) for g in guides])


@pytest.mark.parametrize("n_guides", [1, 2])
@pytest.mark.parametrize("pre,post", PAMS)
@pytest.mark.parametrize("length,mm", [(20, 0), (20, 3), (20, 4), (18, 2), (25, 4), (16, 3), (20, 5)])
def test_rows(cof_mod, oracle_mod, monkeypatch, n_guides, pre, post, length, mm):
    rng = random.Random(length * 10 + mm + n_guides)
    _, records = randgen.random_genome(rng, 3, 20000, 60000)
    filt, pats = _request(rng, pre, post, n_guides, length)
    for p in pats:
        randgen.plant_sites(rng, records, p, filt, 30, mm + 1)
    chunks = _chunks(records)
    g, o = _genome(cof_mod.Genome, chunks), _genome(oracle_mod.OracleGenome, chunks)
    monkeypatch.delenv("COF_SCAN_VARIANT", raising=False)
    got = g.search(filt, pats, mm)
    # (a rare PAM leaves few starts to screen; short guides share too few cells
    # between the strands)
    screened = mm <= 4 and post in ("NRG", "NGG") and length >= 20
    assert ("screen" in g.tuning()["last"]) == screened
    seen = g.last_stats()
    monkeypatch.setenv("COF_SCAN_VARIANT", str(8 + n_guides))
    assert g.search(filt, pats, mm) == got and "screen" not in g.tuning()["last"]
    assert [g.last_stats()[k] for k in ("candidates", "pairs")] == [seen[k] for k in ("candidates", "pairs")]
    ref, n = o.search(filt, pats, mm)
    assert got[1] == n > 0 and sorted(got[0].splitlines()) == sorted(ref.splitlines())


def test_iupac_guide_batch_slices_overflow(cof_mod, monkeypatch):
    rng = random.Random(8)
    _, records = randgen.random_genome(rng, 3, 30000, 60000)
    filt, (p,) = _request(rng, "", "NRG", 1, 25)
    p = p[:4] + "R" + p[5:11] + "N" + p[12:]
    randgen.plant_sites(rng, records, p, filt, 200, 3)
    chunks = _chunks(records, max_chunk=700)
    g = _genome(cof_mod.Genome, chunks)
    for cps in (0, 3):
        monkeypatch.setenv("COF_SCAN_VARIANT", "9")
        want = g.search(filt, [p], 3, chunks_per_search=cps)
        monkeypatch.delenv("COF_SCAN_VARIANT")
        assert want[1] > 100 and g.search(filt, [p], 3, chunks_per_search=cps) == want
        assert cps or "screen" in g.tuning()["last"]
        monkeypatch.setenv("COF_SLICE_NT", "5000")
        assert g.search(filt, [p], 3, chunks_per_search=cps) == want and g.tuning()["slices"] > 5
        monkeypatch.delenv("COF_SLICE_NT")
        # two requests of one filter are one pair of two patterns
        req = dict(search_filter=filt, patterns=[p], max_mismatches=3, chunks_per_search=cps)
        assert g.search_batch([req, req]) == [want, want]
    monkeypatch.setenv("COF_CAND_CAP", "64")
    assert _genome(cof_mod.Genome, chunks).search(filt, [p], 3) == g.search(filt, [p], 3)
