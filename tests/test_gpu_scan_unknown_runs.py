"""Runs of N under a filter without PAM cells: the tensor-core scan reports no hits
inside them (the code of N is that of a base, so a guide of one base repeated
would meet every window there), at their edges the rows are those of the POPC scan,
and patterns that any window meets keep theirs.  Rows are text: exact."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu


def _genome(cof_mod, seqs):
    g = cof_mod.Genome()
    for i, seq in enumerate(seqs):
        for s in range(0, len(seq), 30000):
            e = min(len(seq), s + 30000)
            g.add_chunk("rec%d" % i, randgen.pack(seq[s:e])[0], s, e)
    return g


def _guides(rng, n, length):
    return ["".join(rng.choice("ACGT") for _ in range(length)) for _ in range(n)]


@pytest.mark.parametrize("length", [14, 20, 28, 31, 32, 36])
def test_no_hits_inside_runs(cof_mod, monkeypatch, length):
    rng = random.Random(length)

    def bases(n):
        return "".join(rng.choice("ACGT") for _ in range(n))
    # runs around the 32 cells of a window and a long one; bases between them
    seqs = ["".join(bases(rng.randint(40, 300)) + "N" * n
                    for n in (1, 19, 20, 30, 31, 32, 33, 34, 63, 64, 65, 96, 200_000)) + bases(500),
            "N" * 5000 + bases(3000) + "N" * 5000]
    pats = ["T" * length, "T" * (length - 3) + "ACG", "A" * length, "G" * length] + _guides(rng, 70, length)
    g = _genome(cof_mod, seqs)
    monkeypatch.setenv("COF_SCAN_VARIANT", "0")
    want = g.search("N" * length, pats, 5)
    popc_hits = g.last_stats()["raw_hits"]
    monkeypatch.setenv("COF_SCAN_VARIANT", "13")
    got = g.search("N" * length, pats, 5)
    assert g.tuning()["last"].startswith("mma-f8") and got == want
    # at most the windows over an edge of a run, for every pattern of one base
    assert g.last_stats()["raw_hits"] <= popc_hits + 16 * 2 * 32 * 4


@pytest.mark.parametrize("mm", [4, 6, 7])
def test_patterns_that_any_window_meets(cof_mod, monkeypatch, mm):
    # IUPAC cells are not compared by the scan: six compared cells with as many
    # mismatches allowed, among 70 guides that are all compared
    rng = random.Random(mm)
    seqs = [randgen.random_seq(rng, 3000) + "N" * 3000 + randgen.random_seq(rng, 3000)]
    pats = _guides(rng, 70, 20) + ["ACGTAC" + "R" * 14, "ACGTAC" + "RYKMBDHVSWRYKM"]
    g = _genome(cof_mod, seqs)
    monkeypatch.setenv("COF_SCAN_VARIANT", "0")
    want = g.search("N" * 20, pats, mm)
    for variant in ("13", ""):
        monkeypatch.setenv("COF_SCAN_VARIANT", variant)
        assert g.search("N" * 20, pats, mm) == want
