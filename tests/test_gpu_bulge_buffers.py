"""Page-locked memory of bulge searches that are walked in several chunks: the
pieces and results of equal calls differ by a few per cent, and use one buffer, not
a new one whenever one is a little larger than all before it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def searched(cof_mod):
    import synth
    cfg = synth.config_bulge(seed=9, scale=0.02, n_guides=20, planted=20)
    g = cof_mod.Genome()
    cfg["genome"].load_into(g)
    p = g.prepare([dict(search_filter=cfg["filter"], patterns=cfg["patterns"],
                        max_mismatches=4, max_dna_bulges=2, max_rna_bulges=2)])
    g.search(cfg["filter"], cfg["patterns"][:1], 2)  # upload, and buffers of every search
    return g, p


def test_equal_searches_pin_once(searched):
    g, p = searched
    before = g.tuning()["pinned"]
    rows = {g.run_prepared(p, as_text=None)[0] for _ in range(8)}
    assert len(rows) == 1 and rows.pop()[1] > 2_000_000
    assert g.tuning()["pinned"] - before <= 2


@pytest.mark.parametrize("matches", [False, True])
def test_equal_streams_pin_once(searched, matches):
    g, p = searched
    before = g.tuning()["pinned"]
    res = [g.stream_count(p, matches=matches) for _ in range(8)]
    assert len({r[:2] for r in res}) == 1 and res[0][2] > 2  # several pieces
    # the probe's piece and a planned one, with records two of each, and one that
    # passed its size class
    assert g.tuning()["pinned"] - before <= (3 if not matches else 5)
