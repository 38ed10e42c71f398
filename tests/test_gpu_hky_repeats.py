"""HKY chain-loci listed several times in one call, with other parameters: the
entries share the chain-locus's partials, so each has to give the bits of a
call of its own, and the last one's partials are the ones committed.  Sizes
whose partials fit in shared memory and sizes far past it."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [api.PREC_FAST, api.PREC_FP32, api.PREC_FP64])
@pytest.mark.parametrize("n,S", [(2, 3), (10, 40), (40, 300), (90, 900)])
def test_repeats(n, S, prec):
    rng = np.random.default_rng(n + S)
    ctx = api.Context(0)
    trees = []
    for l in range(3):
        seq = np.repeat(rng.integers(0, 4, (1, S)), n, axis=0)
        seq = np.where(rng.random((n, S)) < 1.5 / n, rng.integers(0, 4, (n, S)), seq)
        ctx.add_locus_hky(seq.astype(np.int8), rng.integers(1, 5, S).astype(np.int32), 5 * S)
        trees.append(synth.two_pop_tree(rng, n - n // 2, n // 2, 10.0, 0.2, 1.5))
    ctx.set_chains(1, 2)
    for c in range(2):
        for l in range(3):
            ctx.set_pi(c, l, rng.dirichlet([5.0] * 4))
            ctx.set_genealogy(c, l, trees[l])
    # chain-locus (0, 1) eight times, (1, 2) three times, the others once
    pairs = [(0, 0), (0, 1), (1, 2), (0, 1), (0, 1), (1, 0), (0, 1), (1, 2), (0, 2), (0, 1), (0, 1), (1, 1), (0, 1),
             (1, 2), (0, 1)]
    ci, li = np.array(pairs).T
    u, kap = rng.uniform(0.3, 3.0, len(ci)), rng.uniform(1.5, 9.0, len(ci))
    want = np.array([ctx.eval(ci[k:k + 1], li[k:k + 1], u[k:k + 1], kap[k:k + 1], precision=prec)[0][0]
                     for k in range(len(ci))])
    for _ in range(3):
        got, st = ctx.eval(ci, li, u, kap, precision=prec)
        assert np.all(st == 0)
        np.testing.assert_array_equal(got, want)
    b = ctx.batch_create(ci, li, u, kap, precision=prec)
    for _ in range(3):
        b.run(use_graph=True)
        np.testing.assert_array_equal(b.results()[0], want)
    # the last entry's partials: an evaluation from one tip's edge (the same
    # genealogy, that entry's parameters) reads them for the clean nodes
    ctx.commit([0], [1], np.ones(1, np.uint8))
    last = len(pairs) - 1
    got, _ = ctx.eval([0], [1], u[last:], kap[last:], edits=np.array([[0, -1, -1, -1]]), precision=prec)
    np.testing.assert_array_equal(got, want[last:])
