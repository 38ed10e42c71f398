"""The task list that a full HKY evaluation keeps per chain-locus, through
evaluations from edited edges of the same topology (a slide that lands on its
own branch, then a split-time update): the edited evaluation's own list is
longer than shared memory holds (640 tasks; the root alone has one per
pattern) or shorter, and the full evaluations after it must not read from it.

An evaluation from edited edges combines the same values in the same order as
a full one, so both give the same bits.  Against the FP64 form: the
float-float form's documented 1e-6 per locus, FP32's 2e-6 relative."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth

pytestmark = pytest.mark.gpu

SIZES = [(2, 1), (3, 700), (5, 33), (12, 700), (40, 60), (40, 800), (90, 160), (90, 1200)]


def make(n, S, sparse, nch=2):
    rng = np.random.default_rng(n * 7919 + S * 2 + sparse)
    seq = rng.integers(0, 4, (1 if sparse else n, S))
    if sparse:  # a common state per pattern, few tips off it
        seq = np.where(rng.random((n, S)) < 1.5 / n, rng.integers(0, 4, (n, S)), np.repeat(seq, n, axis=0))
    mult = rng.integers(1, 5, S).astype(np.int32)
    ctx = api.Context(0)
    ctx.add_locus_hky(seq.astype(np.int8), mult, int(mult.sum()))
    ctx.set_chains(1, nch)
    trees = [synth.two_pop_tree(rng, n - n // 2, n // 2, 10.0, 0.2, 1.5) for _ in range(nch)]
    pi = rng.dirichlet([5.0] * 4)
    for c in range(nch):
        ctx.set_pi(c, 0, pi)
        ctx.set_genealogy(c, 0, trees[c])
    ci, li = np.arange(nch), np.zeros(nch, np.int64)
    return rng, ctx, trees, ci, li, rng.uniform(0.5, 1.5, nch), rng.uniform(2.0, 8.0, nch)


def retimed(rng, g):
    """One internal node moved between its daughters and its parent: the
    genealogy (its topology kept) and the edges whose length changed."""
    h = g.copy()
    n = h.n
    v = int(rng.integers(n, 2 * n - 1))
    a, b = int(h.up0[v]), int(h.up1[v])
    node = lambda k: h.time[h.up0[k]] if h.up0[k] >= 0 else 0.0  # noqa: E731
    lo = max(node(a), node(b))
    hi = float(h.time[v]) if h.down[v] >= 0 else node(v) * 1.5
    t = lo + (hi - lo) * float(rng.uniform(0.2, 0.8))
    h.time[a] = h.time[b] = t
    return h, [a, b, v if h.down[v] >= 0 else -1, -1]


def cat(trees):
    return np.concatenate([g.time for g in trees])


def check64(ctx, ci, li, u, kap, got, prec):
    want, _ = ctx.eval(ci, li, u, kap, precision=api.PREC_FP64)
    if prec == api.PREC_FAST:
        np.testing.assert_allclose(got, want, rtol=1e-11, atol=1e-6)
    else:
        np.testing.assert_allclose(got, want, rtol=2e-6)


@pytest.mark.parametrize("prec", [api.PREC_FAST, api.PREC_FP32])
@pytest.mark.parametrize("sparse", [True, False])
@pytest.mark.parametrize("n,S", SIZES)
def test_eval(n, S, sparse, prec):
    rng, ctx, trees, ci, li, u, kap = make(n, S, sparse)
    one = np.ones(len(ci), np.uint8)
    ctx.eval(ci, li, u, kap, precision=prec)
    ctx.commit(ci, li, one)
    for step in range(6):
        moved = [retimed(rng, g) for g in trees]
        if step % 2:  # as an upload of the whole genealogy, or of its times
            for c in ci:
                ctx.set_genealogy(c, 0, moved[c][0])
        else:
            ctx.set_times(ci, li, cat([m[0] for m in moved]))
        edited, st = ctx.eval(ci, li, u, kap, edits=np.array([m[1] for m in moved]), precision=prec)
        assert np.all(st == 0)
        full, _ = ctx.eval(ci, li, u, kap, precision=prec)
        np.testing.assert_array_equal(edited, full)
        check64(ctx, ci, li, u, kap, full, prec)
        ctx.eval(ci, li, u, kap, edits=np.array([m[1] for m in moved]), precision=prec)
        keep = np.array([step % 3 != 0, step % 3 != 1], np.uint8)
        ctx.commit(ci, li, keep)
        trees = [m[0] if k else g for m, g, k in zip(moved, trees, keep)]
        back, _ = ctx.eval_times(ci, li, cat(trees), u, kap, precision=prec)
        check64(ctx, ci, li, u, kap, back, prec)
        ctx.eval(ci, li, u, kap, precision=prec)
        ctx.commit(ci, li, one)


@pytest.mark.parametrize("graph", [False, True])
@pytest.mark.parametrize("n,S", [(12, 700), (40, 60), (90, 1200)])
def test_batches(n, S, graph):
    rng, ctx, trees, ci, li, u, kap = make(n, S, True)
    one = np.ones(len(ci), np.uint8)
    whole = ctx.batch_create(ci, li, u, kap)
    whole.run(use_graph=graph)
    ctx.commit(ci, li, one)
    moved = [retimed(rng, g) for g in trees]
    part = ctx.batch_create(ci, li, u, kap, edits=np.array([m[1] for m in moved]))
    ctx.set_times(ci, li, cat([m[0] for m in moved]))
    got = []
    for b in (part, whole, part, part, whole, whole):
        b.run(use_graph=graph)
        got.append(b.results()[0])
    for g in got[1:]:
        np.testing.assert_array_equal(g, got[0])
    check64(ctx, ci, li, u, kap, got[-1], api.PREC_FAST)


def test_likelihoodHKY():
    rng, ctx, trees, ci, li, u, kap = make(40, 900, True, nch=1)
    g = trees[0]
    ctx.likelihoodHKY(0, 0, u[0], kap[0])
    ctx.copyfraclike(0, 0)
    for _ in range(4):
        h, e = retimed(rng, g)
        ctx.set_genealogy(0, 0, h)
        edited = ctx.likelihoodHKY(0, 0, u[0], kap[0], *e)
        ctx.restorescalefactors(0, 0)
        full = ctx.likelihoodHKY(0, 0, u[0], kap[0])
        assert edited == full
        check64(ctx, ci, li, u, kap, np.array([full]), api.PREC_FAST)
        ctx.likelihoodHKY(0, 0, u[0], kap[0])
        ctx.copyfraclike(0, 0)
        g = h
