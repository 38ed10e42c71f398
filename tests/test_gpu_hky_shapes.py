"""HKY loci that keep one partial per state and loci that keep every pattern
(unrelated sequences, or too many patterns for the masks), by themselves and
in one batch, in every launch shape, against the FP64 form: full evaluations
and evaluations from edited edges, sizes around a warp's 32 patterns.

Tolerance: the float-float form's documented 1e-6 per locus, FP32's 2e-6
relative."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth

pytestmark = pytest.mark.gpu

# genes, patterns, share of states drawn without regard to the others: 1 and
# 0.9 keep every pattern, 0.5 and less one partial per state
KINDS = {
    "alike": [(5, 31, 0.1), (40, 64, 0.05), (12, 33, 0.3)],
    "unrelated": [(2, 1, 1.0), (3, 32, 1.0), (40, 65, 1.0), (24, 200, 0.9)],
    "both": [(5, 31, 0.1), (40, 65, 1.0), (33, 96, 0.5), (2, 7, 1.0), (90, 40, 0.9), (12, 33, 0.3)],
    "masks": [(90, 3000, 0.05), (20, 64, 0.1)],
}


@pytest.mark.parametrize("prec", [api.PREC_FAST, api.PREC_FP32])
@pytest.mark.parametrize("kind", KINDS)
def test_shapes(kind, prec):
    rng = np.random.default_rng(len(kind))
    nch = 3
    ctx = api.Context(0)
    trees = []
    for n, S, p in KINDS[kind]:
        seq = np.repeat(rng.integers(0, 4, (1, S)), n, axis=0)
        seq = np.where(rng.random((n, S)) < p, rng.integers(0, 4, (n, S)), seq).astype(np.int8)
        mult = rng.integers(1, 5, S).astype(np.int32)
        ctx.add_locus_hky(seq, mult, int(mult.sum()))
        trees.append([synth.two_pop_tree(rng, n - n // 2, n // 2, 10.0, 0.2, 1.5) for _ in range(nch)])
    nl = len(trees)
    ctx.set_chains(1, nch)
    ci, li = np.repeat(np.arange(nch), nl), np.tile(np.arange(nl), nch)
    for c, l in zip(ci, li):
        ctx.set_pi(c, l, rng.dirichlet([5.0] * 4))
        ctx.set_genealogy(c, l, trees[l][c])
    u, kap = rng.uniform(0.3, 2.0, len(ci)), rng.uniform(1.5, 9.0, len(ci))
    one = np.ones(len(ci), np.uint8)

    def check(got):
        want, _ = ctx.eval(ci, li, u, kap, precision=api.PREC_FP64)
        if prec == api.PREC_FAST:
            np.testing.assert_allclose(got, want, rtol=1e-11, atol=1e-6)
        else:
            np.testing.assert_allclose(got, want, rtol=2e-6)

    first, st = ctx.eval(ci, li, u, kap, precision=prec)
    assert np.all(st == 0)
    check(first)
    b = ctx.batch_create(ci, li, u, kap, precision=prec)
    for v in range(6):
        b.set_variants(v, 0)
        b.run(use_graph=False)
        check(b.results()[0])
    ctx.eval(ci, li, u, kap, precision=prec)
    ctx.commit(ci, li, one)
    # one tip's edge shortened or lengthened with its sister's: their node moved
    edits = np.full((len(ci), 4), -1, np.int32)
    for k, (c, l) in enumerate(zip(ci, li)):
        g = trees[l][c].copy()
        v = int(g.down[0])
        a, o = int(g.up0[v]), int(g.up1[v])
        low = max(g.time[g.up0[x]] if g.up0[x] >= 0 else 0.0 for x in (a, o))
        top = float(g.time[v]) if g.down[v] >= 0 else g.time[a] * 1.5
        g.time[a] = g.time[o] = low + (top - low) * 0.37
        edits[k, :3] = a, o, v
        ctx.set_genealogy(c, l, g)
    edited, _ = ctx.eval(ci, li, u, kap, edits=edits, precision=prec)
    check(edited)
    e = ctx.batch_create(ci, li, u, kap, edits=edits, precision=prec)
    for v in range(6):
        e.set_variants(v, 0)
        e.run(use_graph=False)
        check(e.results()[0])
    full, _ = ctx.eval(ci, li, u, kap, precision=prec)
    np.testing.assert_array_equal(full, edited)
