"""How the bulge path divides its work: end positions per Myers tile, and
candidate chunks planned from a probe.  Rows are text: comparisons are exact."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nt,guides", [(700, 1), (40_000, 1), (60_000, 12), (120_000, 40),
                                       (200_000, 150)])
def test_myers_tile_lengths(cof_mod, oracle_mod, nt, guides):
    # the end positions per Myers tile follow from genome and pattern count
    # (64 for the smallest, 1024 for the largest): rows equal the oracle's
    import synth
    rng = np.random.default_rng(nt + guides)
    sg = synth.make_genome(rng, [nt // 3, nt - nt // 3], [(0, nt // 20)])
    pats = [synth.random_guide(rng, 20) + "NNN" for _ in range(guides)]
    for i, p in enumerate(pats[:6]):
        synth.plant(rng, sg, p, "N" * 20 + "NRG", 2, 2, [], i, bulge=(1, 0))
    g, o = cof_mod.Genome(), oracle_mod.OracleGenome()
    sg.load_into(g)
    for name, data, s, e in sg.chunks():
        o.add_chunk(name, data, s, e)
    for filt, ps in (("N" * 21 + "RG", pats), ("TTTN" + "N" * 20, ["NNNN" + p[:20] for p in pats])):
        text, n = g.search(filt, ps, 2, 1, 1)
        ref, nref = o.search(filt, ps, 2, 1, 1)
        assert n == nref and sorted(text.splitlines()) == sorted(ref.splitlines())


def test_planned_chunks_equal_one_chunk(cof_mod, monkeypatch):
    # more than two probe chunks of surviving candidates: a probe, then chunks
    # sized from its rows per candidate; the rows are those of one chunk
    import synth
    cfg = synth.config_bulge(seed=9, scale=0.007, n_guides=20, planted=4)
    g = cof_mod.Genome()
    cfg["genome"].load_into(g)
    prepared = g.prepare([dict(search_filter=cfg["filter"], patterns=cfg["patterns"],
                               max_mismatches=4, max_dna_bulges=2, max_rna_bulges=2)])
    monkeypatch.setenv("COF_BULGE_CHUNK", str(1 << 21))
    (one, n1), = g.run_prepared(prepared, as_text=False)
    launches = g.last_stats()["kernel_launches"]
    monkeypatch.delenv("COF_BULGE_CHUNK")
    (text, n), = g.run_prepared(prepared, as_text=False)
    assert g.last_stats()["kernel_launches"] > launches
    assert n == n1 > 1_000_000 and len(text) == len(one)
    assert sorted(text.splitlines()) == sorted(one.splitlines())


@pytest.mark.parametrize("filt,pam_lead,pam_tail,core", [
    ("N" * 12 + "G", "", "N", 12),                       # one cell
    ("N" * 10 + "RSWNYKMBDHVNNRSWG", "", "N" * 17, 10),  # longer than a 16-cell word
    ("TTTV" + "N" * 14, "NNNN", "", 14),                 # leads the pattern: several spans
    ("N" * 16, "", "", 16),                              # none
])
@pytest.mark.parametrize("size", [15, 33, 63, 64, 65, 1023, 1057])
def test_pam_of_every_start(cof_mod, oracle_mod, size, filt, pam_lead, pam_tail, core):
    # batches that begin and end inside a word of 32 starts and of 16 cells,
    # unknown bases and codes of several bases among the cells
    import random

    import randgen
    rng = random.Random(size * 100 + len(filt))
    records = [randgen.random_seq(rng, size + i) for i in range(4)]
    pats = [pam_lead + "".join(rng.choice("ACGT") for _ in range(core)) + pam_tail
            for _ in range(3)]
    for p in pats:
        randgen.plant_sites(rng, records, p, filt, 4, 2)
    g, o = cof_mod.Genome(), oracle_mod.OracleGenome()
    for name, data, _nibs, s, e in randgen.chunk_records(rng, records, max(20, size // 2)):
        g.add_chunk(name, data, s, e)
        o.add_chunk(name, data, s, e)
    text, n = g.search(filt, pats, 3, 1, 1)
    ref, nref = o.search(filt, pats, 3, 1, 1)
    assert n == nref and sorted(text.splitlines()) == sorted(ref.splitlines())
