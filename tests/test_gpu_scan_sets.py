"""Scan kernel by set: of a pass, each set of patterns (one strand of the requests
with one PAM) goes to the tensor cores or to the POPC scan by its own patterns and
limits, whatever the others are, and a set's batches are one group.  Rows are
text: exact."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu
NRG = "N" * 21 + "RG"


def _genome(cof_mod, records, max_chunk=5000):
    g = cof_mod.Genome()
    for name, data, _nibs, s, e in randgen.chunk_records(random.Random(2), records, max_chunk):
        g.add_chunk(name, data, s, e)
    return g


def _req(rng, pam, n, mm, length=20, **kw):
    if pam == "TTTN":
        pats = ["NNNN" + "".join(rng.choice("ACGT") for _ in range(length)) for _ in range(n)]
        return dict(search_filter="TTTN" + "N" * length, patterns=pats, max_mismatches=mm, **kw)
    pats = ["".join(rng.choice("ACGT") for _ in range(length)) + "N" * len(pam) for _ in range(n)]
    return dict(search_filter="N" * length + pam, patterns=pats, max_mismatches=mm, **kw)


def _plant(rng, records, reqs):
    for r in reqs:
        for p in r["patterns"][:6]:
            randgen.plant_sites(rng, records, p, r["search_filter"], 3, min(r["max_mismatches"], 4))


# (sets, what the scan is reported as)
MIXES = {
    "one large, three small": ([("NRG", 200, 4), ("NNGRRT", 1, 4), ("TTTN", 1, 3), ("NGCG", 1, 2)], "mma+popc"),
    "just enough beside one guide": ([("NRG", 64, 4), ("TTTN", 1, 4)], "mma+popc"),
    "two large": ([("NRG", 64, 4), ("TTTN", 64, 4)], "mma"),
    "large in sum only": ([("NRG", 63, 4), ("TTTN", 63, 4), ("NGCG", 63, 4)], "popc"),
    "large and loose beside large": ([("NRG", 70, 4), ("TTTN", 70, 12)], "mma+popc"),
    "several requests of one set": ([("NRG", 30, 4), ("NRG", 34, 2), ("TTTN", 2, 3)], "mma+popc"),
    "one loose guide beside a library": ([("NRG", 1200, 4), ("TTTN", 1, 12)], "mma+popc"),
}


@pytest.mark.parametrize("mix", sorted(MIXES))
@pytest.mark.parametrize("cps", [0, 2])
def test_each_set_by_its_own_patterns(cof_mod, monkeypatch, mix, cps):
    monkeypatch.delenv("COF_SCAN_VARIANT", raising=False)
    sets, kernels = MIXES[mix]
    rng = random.Random(len(mix) + cps)
    _, records = randgen.random_genome(rng, 3, 30000, 60000)
    reqs = [_req(rng, pam, n, mm, chunks_per_search=cps) for pam, n, mm in sets]
    _plant(rng, records, reqs)
    # with cps 2 more batches than one scan group holds
    g = _genome(cof_mod, records, 5000 if cps == 0 else 500)
    got = g.search_batch(reqs)
    shape = g.tuning()["last"]
    assert shape.startswith("mma-f8") == kernels.startswith("mma")
    assert ("+" in shape) == (kernels == "mma+popc")
    monkeypatch.setenv("COF_SCAN_VARIANT", "0")
    assert g.search_batch(reqs) == got and all(n for _, n in got)
    assert not g.tuning()["last"].startswith("mma")


@pytest.mark.parametrize("n", [127, 128, 129])
def test_strands_apart_in_slices(cof_mod, monkeypatch, n):
    # an odd list without reverse complements: 63 forward patterns by POPC, 64
    # reverse ones on the tensor cores, in one pass and in slices
    monkeypatch.delenv("COF_SCAN_VARIANT", raising=False)
    rng = random.Random(n)
    _, records = randgen.random_genome(rng, 3, 30000, 50000)
    fwd = ["".join(rng.choice("ACGT") for _ in range(20)) + "NNN" for _ in range(n // 2)]
    comp = str.maketrans("ACGTN", "TGCAN")
    pats = fwd + [("".join(rng.choice("ACGT") for _ in range(20)) + "NNN").translate(comp)[::-1]
                  for _ in range(n - n // 2)]
    for p in fwd[:8]:
        randgen.plant_sites(rng, records, p, NRG, 6, 4)
    g = _genome(cof_mod, records)
    one = g.search(NRG, pats, 6, add_revcomp=False)
    shape = g.tuning()["last"]
    assert one[1] > 0 and shape.startswith("mma-f8") and ("+" in shape) == (n == 127)
    monkeypatch.setenv("COF_SLICE_NT", "7000")
    assert g.search(NRG, pats, 6, add_revcomp=False) == one
    assert g.tuning()["slices"] > 5 and g.tuning()["last"] == shape
    monkeypatch.setenv("COF_SCAN_VARIANT", "0")
    assert g.search(NRG, pats, 6, add_revcomp=False) == one
