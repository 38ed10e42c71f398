"""The genealogy update from generators whose word count is past the state's
end: MT19937 makes the next state at 624 words drawn and at any number above
(625 is what a generator that was never seeded holds), and so does the update."""
import numpy as np
import pytest

from ima2p_gb300 import api, popmodel, workloads

pytestmark = pytest.mark.gpu


def run(w, mti, nsweeps=2):
    nl, nch = len(w.base), w.nch
    ctx = api.Context(0)
    for L in w.loci:
        ctx.add_locus_hky(L.seq, L.mult, L.totsites)
    ctx.set_chains(1, nch)
    pm = popmodel.build(w.tree, w.npops, nomig=True)
    th_max, th_min, _, _, _ = popmodel.priors(pm, 30.0, 0.0)
    ctx.set_popmodel(pm, th_max, th_min)
    ci, li = np.repeat(np.arange(nch), nl), np.tile(np.arange(nl), nch)
    flat = w.base * nch
    cat = lambda f: np.concatenate([getattr(g.g, f) for g in flat])  # noqa: E731
    ctx.set_genealogies(ci, li, cat("up0"), cat("up1"), cat("down"), cat("time"))
    ctx.set_labels(ci, li, flat)
    ctx.set_locus_pops(np.ones(nl), w.samppop)
    for c in range(nch):
        for l in range(nl):
            ctx.set_pi(c, l, w.loci[l].pi)
    rngs = [api.UgRng(40 + c) for c in range(nch)]
    for g in rngs:
        assert g.mt.mti == 624
        g.mt.mti = mti
    acc, top, probg = ctx.updategenealogy_sweep(np.arange(nch), np.tile(w.tvals, (nch, 1)), nsweeps, rngs, np.tile(w.u, nch),
                                                np.tile(w.kappa, nch))
    trees = [ctx.get_genealogy(c, l, len(w.base[l].pop)) for c in range(nch) for l in range(nl)]
    words = [(g.mt.mti, list(g.mt.mt), g.iset, g.gset, g.iseed) for g in rngs]
    return [acc, top, probg] + [a for t in trees for a in t], words


@pytest.mark.parametrize("nloci", [1, 9])  # a launch per locus, several loci a launch
@pytest.mark.parametrize("mti", [625, 700, 2 ** 31 - 1])
def test_word_count_past_the_end(nloci, mti):
    w = workloads.make_updgen(nloci=nloci, nch=3, ncopies=5, nbases=200)
    want, words = run(w, 624)
    got, gwords = run(w, mti)
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
    assert gwords == words
