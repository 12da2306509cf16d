"""A COF_TUNE_CACHE file is read as it comes, from this version of the library or
another: a choice that names no scan shape is passed over, one that does is taken."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu
KEY = "pat4-grp2-pam2-L23-mm5"  # 3 guides at NRG, both strands


@pytest.mark.parametrize("cached,taken", [(4, 4), (12, None), (13, None), (14, None), (99, None),
                                          (2**31 - 1, None), (-1, None), (-2**31, None)])
def test_choices_of_a_file(cof_mod, monkeypatch, tmp_path, cached, taken):
    monkeypatch.delenv("COF_SCAN_VARIANT", raising=False)
    rng = random.Random(1)
    _, records = randgen.random_genome(rng, 2, 20000, 30000)
    pats = ["".join(rng.choice("ACGT") for _ in range(20)) + "NNN" for _ in range(3)]
    for p in pats:
        randgen.plant_sites(rng, records, p, "N" * 21 + "RG", 5, 4)

    def search():
        g = cof_mod.Genome()
        for name, data, _nibs, s, e in randgen.chunk_records(random.Random(2), records, 5000):
            g.add_chunk(name, data, s, e)
        return g.search("N" * 21 + "RG", pats, 5), g.tuning()
    want, tuning = search()
    default = tuning["variant"]
    path = tmp_path / "tune.txt"
    path.write_text("%s %d\n" % (KEY, cached))
    monkeypatch.setenv("COF_TUNE_CACHE", str(path))
    got, tuning = search()
    assert tuning["cache"].get(KEY) == cached  # the file was read, the key is this search's
    assert got == want and tuning["variant"] == (default if taken is None else taken)
