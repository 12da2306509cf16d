"""A product of the tensor-core scan that is not seen within its wait's limit
(COF_MMA_WAIT lowers it; 0: no wait sees its product) ends the search with
COF_E_TIMEOUT instead of wrong rows: the team leaves before its next product, also
in the middle of a set of several column blocks, and the genome answers the next
search as before."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("guides", [5, 64, 200, 700])
@pytest.mark.parametrize("slices", [False, True])
def test_a_wait_that_runs_out(cof_mod, monkeypatch, guides, slices):
    rng = random.Random(guides)
    _, records = randgen.random_genome(rng, 2, 20000, 30000)
    pats = ["".join(rng.choice("ACGT") for _ in range(20)) + "NNN" for _ in range(guides)]
    filt = "N" * 21 + "RG"
    for p in pats[:8]:
        randgen.plant_sites(rng, records, p, filt, 4, 3)
    g = cof_mod.Genome()
    for name, data, _nibs, s, e in randgen.chunk_records(random.Random(2), records, 5000):
        g.add_chunk(name, data, s, e)
    monkeypatch.setenv("COF_SCAN_VARIANT", "13")
    if slices:
        monkeypatch.setenv("COF_SLICE_NT", "7000")
    want = g.search(filt, pats, 5)
    assert want[1] > 0 and g.tuning()["last"].startswith("mma-f8")
    for _ in range(2):
        monkeypatch.setenv("COF_MMA_WAIT", "0")
        with pytest.raises(cof_mod.CofError) as e:
            g.search(filt, pats, 5)
        assert "-7" in str(e.value) or "gave up" in str(e.value)
        monkeypatch.delenv("COF_MMA_WAIT")
        assert g.search(filt, pats, 5) == want
