"""The most genes an HKY locus may have: what a CTA's shared memory holds (227
KB) of a branch's 141 bytes in the FP64 and float-float forms, of 77 in FP32
-- 824 and 1,509 genes.

Against pruning in numpy, whose 1 - e^-b of the shortest branches (b down to
1e-10) keeps 6 digits, as the FP64 form's does; a site's likelihood has a few
such factors among some hundred, so 1e-7 of the sum is far above that.  FP32:
2e-6."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth

pytestmark = pytest.mark.gpu


def pruned(seq, mult, totsites, g, pi, u, kappa):
    mu = u / (totsites * synth.hky_standfactor(pi, kappa))
    b = g.branch() * mu
    part, scale = {}, np.zeros(seq.shape[1])
    for c in synth.postorder(g):
        L = np.eye(4)[seq[c]] if g.up0[c] < 0 else part.pop(int(g.up0[c])) * part.pop(int(g.up1[c]))
        m = L.max(axis=1)
        L, scale = L / m[:, None], scale + np.log(m)
        part[c] = L @ pi if c == g.root else L @ synth.hky_pmatrix(pi, kappa, b[c]).T
    return float(np.dot(mult, np.log(part[g.root]) + scale))


@pytest.mark.parametrize("n,prec,rtol", [(802, api.PREC_FP64, 1e-7), (824, api.PREC_FP64, 1e-7),
                                         (824, api.PREC_FAST, 1e-7), (1509, api.PREC_FP32, 2e-6)])
@pytest.mark.parametrize("share", [0.01, 1.0])
def test_most_genes(n, prec, rtol, share):
    rng = np.random.default_rng(n)
    S = 40
    g = synth.two_pop_tree(rng, n - n // 2, n // 2, 10.0, 0.2, 1.5)
    seq = np.repeat(rng.integers(0, 4, (1, S)), n, axis=0)
    seq = np.where(rng.random((n, S)) < share, rng.integers(0, 4, (n, S)), seq).astype(np.int8)
    mult = rng.integers(1, 5, S).astype(np.int32)
    pi = rng.dirichlet([5.0] * 4)
    ctx = api.Context(0)
    ctx.add_locus_hky(seq, mult, int(mult.sum()))
    ctx.set_chains(1, 2)
    for c in range(2):
        ctx.set_pi(c, 0, pi)
        ctx.set_genealogy(c, 0, g)
    got, st = ctx.eval([0, 1], [0, 0], [1.3, 0.4], [3.0, 6.0], precision=prec)
    assert np.all(st == 0)
    want = [pruned(seq, mult, int(mult.sum()), g, pi, u, k) for u, k in ((1.3, 3.0), (0.4, 6.0))]
    np.testing.assert_allclose(got, want, rtol=rtol)
