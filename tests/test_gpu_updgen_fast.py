"""The genealogy update in the float-float form over launches of several loci:
the runs of test_gpu_updgen_runs, decision for decision against the oracle
(the likelihood ratios differ from FP64's by 1e-9 at most, so a decision only
where its deviate lies that near), and the partials that the sweeps leave --
roots, which hold every pattern, have moved -- through an evaluation from
edited edges, which reads them, against the FP64 form (1e-6 per locus)."""
import numpy as np
import pytest

from ima2p_gb300 import api, popmodel, workloads
from tests import test_gpu_updgen_runs as runs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,nsweeps", [
    ([runs.HKY] * 8, 3), ([runs.SW, runs.HKY, runs.HKY, runs.IS, runs.HKY, runs.HKY, runs.HKY, runs.SW, 2, 4, runs.IS], 5),
    ([runs.HKY] * 20 + [runs.SW] * 13 + [runs.IS] + [2] * 9 + [runs.HKY] * 5, 4)])
def test_runs_in_float_float(order, nsweeps, monkeypatch):
    monkeypatch.setattr(api, "PREC_FP64", api.PREC_FAST)  # the precision that the runs ask for
    runs.test_runs_of_loci_against_the_oracle(order, nsweeps)


@pytest.mark.parametrize("nloci,ncopies,nbases", [(8, 3, 100), (30, 10, 400), (50, 20, 1000)])
def test_partials_after_sweeps(nloci, ncopies, nbases):
    w = workloads.make_updgen(nloci=nloci, nch=4, ncopies=ncopies, nbases=nbases)
    nl, nch = nloci, w.nch
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
    u, kap = np.tile(w.u, nch), np.tile(w.kappa, nch)
    rngs = [api.UgRng(5 + c) for c in range(nch)]
    for _ in range(3):
        acc, _, _ = ctx.updategenealogy_sweep(np.arange(nch), np.tile(w.tvals, (nch, 1)), 4, rngs, u, kap,
                                              precision=api.PREC_FAST)
        assert acc.sum() > 0
        pdg = ctx.get_pdg().reshape(-1)
        # from the edge of tip 0: its ancestors anew, the rest from the sweeps
        edited, _ = ctx.eval(ci, li, u, kap, edits=np.tile([0, -1, -1, -1], (len(ci), 1)), precision=api.PREC_FAST)
        full, _ = ctx.eval(ci, li, u, kap, precision=api.PREC_FAST)
        want, _ = ctx.eval(ci, li, u, kap, precision=api.PREC_FP64)
        np.testing.assert_array_equal(edited, full)
        np.testing.assert_array_equal(pdg, full)
        np.testing.assert_allclose(full, want, rtol=1e-11, atol=1e-6)
