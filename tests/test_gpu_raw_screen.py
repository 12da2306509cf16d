"""The raw Match stream's bit-parallel screen (raw_screen_kernel) against the
oracle: pattern lengths to the 32 cells of a plane window, every limit it
takes and the first it does not, genomes with runs of N and IUPAC letters, batch
ends inside a window, and guides with IUPAC cells.  Lines are text: exact."""
import random

import pytest

import randgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length,mm", [(14, 0), (15, 4), (20, 2), (23, 4), (23, 5), (28, 3), (31, 4), (32, 4),
                                       (33, 4)])
@pytest.mark.parametrize("cps", [0, 3])
def test_raw_lines(cof_mod, oracle_mod, length, mm, cps):
    rng = random.Random(100 * length + mm + cps)
    _, records = randgen.random_genome(rng, 3, 8000, 20000)
    filt = "N" * (length - 3) + "NRG"
    pats = ["".join(rng.choice("ACGT") for _ in range(length - 3)) + "NNN" for _ in range(5)]
    for p in pats:
        randgen.plant_sites(rng, records, p, filt, 20, mm + 1)
    # guides with IUPAC cells, which count by the letters they hold
    extra = [pats[0][:2] + "RYN" + pats[0][5:], "N" * 3 + pats[1][3:]]
    g, o = cof_mod.Genome(), oracle_mod.OracleGenome()
    for name, data, _nibs, s, e in randgen.chunk_records(rng, records, 900):
        g.add_chunk(name, data, s, e)
        o.add_chunk(name, data, s, e)
    found = 0
    for ps in (pats, pats + extra):
        text, n = g.search(filt, ps, mm, raw=True, chunks_per_search=cps)
        ref, nref = o.search(filt, ps, mm, raw=True, chunks_per_search=cps)
        assert n == nref and sorted(text.split("\n")) == sorted(ref.split("\n"))
        found += n
    assert found > 0


def test_more_rows_than_the_first_room(cof_mod, oracle_mod):
    # over 4,096 raw matches: the rows' buffers grow and the hits are verified
    # again
    rng = random.Random(6)
    seq = "".join(rng.choice("ACGT") for _ in range(6000))
    chunks = [("rec", *randgen.pack(seq), 0, len(seq))]
    g, o = cof_mod.Genome(), oracle_mod.OracleGenome()
    for name, data, _nibs, s, e in chunks:
        g.add_chunk(name, data, s, e)
        o.add_chunk(name, data, s, e)
    pats = ["".join(rng.choice("ACGT") for _ in range(14)) for _ in range(10)]
    text, n = g.search("N" * 14, pats, 12, raw=True)
    ref, nref = o.search("N" * 14, pats, 12, raw=True)
    assert n == nref > 65536 and sorted(text.split("\n")) == sorted(ref.split("\n"))
