"""HKY partials kept once per state where the tips below a node agree: the
float-float and FP32 forms against the FP64 form (which keeps every pattern)
at the sizes where the entries' masks and task lists can go wrong -- one word
of patterns less and more, one pattern, two genes, lists longer than shared
memory holds, masks past their limit (every pattern kept) -- for patterns
that are nearly uniform and for random ones, through full evaluations,
repeated ones (the list read back), new topologies evaluated from their edited
edges, accepted and rejected.

Tolerance: the float-float form's documented 1e-6 per locus (its pairs carry
46 bits: below 1e-12 of the sum), FP32's 2e-6 relative."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth

pytestmark = pytest.mark.gpu


def regraft(rng, g):
    """A tip moved to another branch below the root: (genealogy, edited edges)."""
    h = g.copy()
    n = h.n
    for _ in range(50):
        e = int(rng.integers(n))
        p = int(h.down[e])
        if p == h.root:
            continue
        s = int(h.up1[p] if h.up0[p] == e else h.up0[p])
        gp = int(h.down[p])
        f = int(rng.integers(2 * n - 1))
        if f in (e, p, s, h.root):
            continue
        lo = h.time[h.up0[f]] if h.up0[f] >= 0 else 0.0
        hi = h.time[f]
        if not hi > lo + 1e-9:
            continue
        t = float(rng.uniform(lo + 0.1 * (hi - lo), hi - 0.1 * (hi - lo)))
        if h.up0[gp] == p:
            h.up0[gp] = s
        else:
            h.up1[gp] = s
        h.down[s], h.time[s] = gp, h.time[p]
        fp, top = int(h.down[f]), float(h.time[f])
        if h.up0[fp] == f:
            h.up0[fp] = p
        else:
            h.up1[fp] = p
        h.up0[p], h.up1[p] = f, e
        h.down[e] = h.down[f] = p
        h.down[p] = fp
        h.time[e] = h.time[f] = t
        h.time[p] = top
        return h, [e, s, f, p]
    return None, None


def data(rng, n, S, sparse):
    if sparse:  # a common state per pattern, few tips off it
        seq = np.repeat(rng.integers(0, 4, (1, S)), n, axis=0)
        off = rng.random((n, S)) < 1.5 / n
        seq = np.where(off, rng.integers(0, 4, (n, S)), seq)
    else:
        seq = rng.integers(0, 4, (n, S))
    return seq.astype(np.int8), rng.integers(1, 5, S).astype(np.int32)


@pytest.mark.parametrize("n,S", [(2, 1), (3, 4), (5, 31), (5, 32), (6, 33), (40, 64), (24, 130), (90, 160), (12, 700),
                                 (60, 4500)])
@pytest.mark.parametrize("sparse", [True, False])
def test_uniform_entries(n, S, sparse):
    rng = np.random.default_rng(n * 1000 + S + sparse)
    seq, mult = data(rng, n, S, sparse)
    ctx = api.Context(0)
    ctx.add_locus_hky(seq, mult, int(mult.sum()))
    ctx.set_chains(1, 2)
    trees = [synth.two_pop_tree(rng, n - n // 2, n // 2, 10.0, 0.2, 1.5) for _ in range(2)]
    ci, li = np.array([0, 1]), np.array([0, 0])
    u, kap = np.array([1.3, 0.7]), np.array([3.0, 5.0])
    pi = rng.dirichlet([5.0] * 4)
    for c in range(2):
        ctx.set_pi(c, 0, pi)
        ctx.set_genealogy(c, 0, trees[c])

    def check(edits=None):
        want, _ = ctx.eval(ci, li, u, kap, precision=api.PREC_FP64)  # in full
        got, st = ctx.eval(ci, li, u, kap, edits=edits, precision=api.PREC_FAST)
        assert np.all(st == 0)
        np.testing.assert_allclose(got, want, rtol=1e-11, atol=1e-6)
        return got

    check()
    first = check()  # the list read back
    ctx.commit(ci, li, np.ones(2, np.uint8))
    got32, _ = ctx.eval(ci, li, u, kap, precision=api.PREC_FP32)
    np.testing.assert_allclose(got32, first, rtol=2e-6)
    ctx.eval(ci, li, u, kap, precision=api.PREC_FAST)
    ctx.commit(ci, li, np.ones(2, np.uint8))
    for step in range(6):
        moved = [regraft(rng, t) for t in trees]
        if any(m[0] is None for m in moved):
            return  # too few genes to move one
        for c in range(2):
            ctx.set_genealogy(c, 0, moved[c][0])
        check(np.array([m[1] for m in moved]))
        keep = np.array([step % 2, 1 - step % 2], np.uint8)
        ctx.commit(ci, li, keep)
        for c in range(2):
            if keep[c]:
                trees[c] = moved[c][0]
            else:
                ctx.set_genealogy(c, 0, trees[c])
    check()
