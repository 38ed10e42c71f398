"""The genealogy update over runs of loci of one model, which go through one
launch of each kernel: runs shorter than, as long as and longer than a launch
takes (a quarter of the loci, at most 12), runs broken by infinite-sites loci,
whose decisions draw from the generator, one locus, and more draws than one
state of the generator holds (624) -- against the oracle's restatement.
Accepted proposals, topologies, labels and alleles exact, node times 1e-12
(the device's log and sqrt in the slide's normal deviate), p(G) 1e-9 (its
terms' logarithms)."""
import numpy as np
import pytest

from ima2p_gb300 import api
from oracle import pyoracle as O
from tests.test_updgen_oracle import _case

pytestmark = pytest.mark.gpu

SW, IS, HKY = 0, 1, 3  # loci of the fixture (three stepwise ones: 0, 2, 4)


@pytest.mark.parametrize("order,nsweeps", [
    ([HKY], 3), ([SW] * 7, 3), ([HKY] * 8, 3), ([SW, HKY, HKY, IS, HKY, HKY, HKY, SW, 2, 4, IS, IS], 5),
    ([HKY] * 20 + [SW] * 13 + [IS] + [2] * 9 + [HKY] * 5, 4), ([4] * 50, 4)])
def test_runs_of_loci_against_the_oracle(order, nsweeps):
    d, pm, _, u, kap, pi, th_max, th_min, gens, alleles = _case("golden_ug_sw.npz")
    nch, nl0, nl = 2, len(d["kinds"]), len(order)
    kinds = [str(d["kinds"][k]) for k in order]
    base = [gens[0][k] for k in order]
    tv, betas, samps = np.tile(d["tv0"], (nch, 1)), d["betas"][:nch], d["samps"].astype(np.int32)[order]
    pick = lambda a: np.tile(a[:nl0][order], (nch,) + (1,) * (a.ndim - 1))  # noqa: E731
    u, kap, pi = pick(u), pick(kap), pick(pi)
    loci, arange = [], np.zeros((nl, 2), np.int32)
    ctx = api.Context(0)
    for j, k in enumerate(order):
        if kinds[j] == "is":
            ctx.add_locus_is(d["seq_%d" % k])
            loci.append(("is", d["seq_%d" % k], O.is_sumlogk(d["seq_%d" % k], base[j].g)[1]))
        elif kinds[j] == "hky":
            ctx.add_locus_hky(d["seq_%d" % k], d["mult_%d" % k], int(d["totsites_%d" % k]))
            loci.append(("hky", type("L", (), {"seq": d["seq_%d" % k], "mult": d["mult_%d" % k],
                                               "totsites": int(d["totsites_%d" % k])})))
        else:
            arange[j] = d["arange_%d" % k]
            ctx.add_locus_sw(len(base[j].pop) // 2 + 1, 1)
            loci.append(("sw", len(base[j].pop) // 2 + 1, int(arange[j, 0]), int(arange[j, 1])))
    ctx.set_chains(1, nch)
    ctx.set_popmodel(pm, th_max, th_min)
    ci, li = np.repeat(np.arange(nch, dtype=np.int32), nl), np.tile(np.arange(nl, dtype=np.int32), nch)
    flat = base * nch
    cat = lambda f: np.concatenate([getattr(g.g, f) for g in flat])  # noqa: E731
    ctx.set_genealogies(ci, li, cat("up0"), cat("up1"), cat("down"), cat("time"), length=np.full(len(flat), -1.0))
    ctx.set_labels(ci, li, flat)
    ctx.set_locus_pops(np.ones(nl), samps)
    al = {}
    for c in range(nch):
        for j, k in enumerate(order):
            if kinds[j] == "hky":
                ctx.set_pi(c, j, d["pi_%d" % k])
            elif kinds[j] == "sw":
                ctx.set_alleles(c, j, d["alleles_%d" % k])
                al[(c, j)] = d["alleles_%d" % k]
    ctx.set_betas(betas)
    acc, top, probg = ctx.updategenealogy_sweep(np.arange(nch), tv, nsweeps, [api.UgRng(70 + c) for c in range(nch)], u,
                                                kap, precision=api.PREC_FP64, allele_range=arange)
    st, res, _, _, pg, fin = O.ug_run(pm, th_max, th_min, O.UgLoci(loci, np.ones(nl), samps), [base] * nch, tv, betas,
                                      u, kap, pi, nsweeps, [O.UgRng(70 + c) for c in range(nch)], alleles=al)
    assert st == 0
    np.testing.assert_array_equal(acc, res[..., 0].sum(axis=1))
    np.testing.assert_allclose(probg, pg, rtol=0, atol=1e-9)
    o = 0
    for k in range(nch * nl):
        nlines = len(flat[k].pop)
        got = ctx.get_genealogy(int(ci[k]), int(li[k]), nlines)
        sl = slice(o, o + nlines)
        for j in (0, 1, 2, 4):
            np.testing.assert_array_equal(got[j], fin[j][sl])
        nonroot = fin[2][sl] != -1
        np.testing.assert_allclose(got[3][nonroot], fin[3][sl][nonroot], rtol=1e-12)
        if kinds[li[k]] == "sw":
            np.testing.assert_array_equal(ctx.get_alleles(int(ci[k]), int(li[k]), nlines), fin[5][sl])
        o += nlines
    ctx.close()
