"""Hand-on passes of the bulge path's slot traceback: dense sites, whose trees go
on over more passes than are launched before the host looks, with many subtrees per
warp in some passes and few in others.  Rows are text: exact."""
import pytest

pytestmark = pytest.mark.gpu


def _config(nt, guides, planted):
    import synth
    return synth.config_bulge(seed=9, scale=nt / 500e6, n_guides=guides, planted=planted)


def _prepare(g, cfg, guides=None):
    return g.prepare([dict(search_filter=cfg["filter"], patterns=cfg["patterns"][:guides],
                           max_mismatches=4, max_dna_bulges=2, max_rna_bulges=2)])


@pytest.mark.parametrize("nt,guides,planted", [(20_000, 1, 20), (60_000, 4, 50), (150_000, 20, 50),
                                               (1_000_000, 20, 12)])
def test_passes_at_the_default_budgets(cof_mod, monkeypatch, nt, guides, planted):
    cfg = _config(nt, guides, planted)
    g = cof_mod.Genome()
    cfg["genome"].load_into(g)
    p = _prepare(g, cfg)
    (text, n), = g.run_prepared(p)
    launches = g.last_stats()["kernel_launches"]
    # one budget in every pass: trees that stay where they are (one group of
    # passes), and trees handed on at once
    monkeypatch.setenv("COF_TB_BUDGET", "30000")
    (one, n_one), = g.run_prepared(p)
    # more than one group of passes
    assert launches >= g.last_stats()["kernel_launches"] + 4
    monkeypatch.setenv("COF_TB_BUDGET", "3")
    (soon, n_soon), = g.run_prepared(p)
    assert n == n_one == n_soon > 5000
    assert sorted(text.splitlines()) == sorted(one.splitlines()) == sorted(soon.splitlines())


def test_passes_against_the_oracle(cof_mod, oracle_mod):
    cfg = _config(30_000, 2, 40)
    g, o = cof_mod.Genome(), oracle_mod.OracleGenome()
    cfg["genome"].load_into(g)
    for name, data, s, e in cfg["genome"].chunks():
        o.add_chunk(name, data, s, e)
    (text, n), = g.run_prepared(_prepare(g, cfg))
    ref, nref = o.search(cfg["filter"], cfg["patterns"], 4, 2, 2)
    assert n == nref > 50_000 and sorted(text.splitlines()) == sorted(ref.splitlines())
