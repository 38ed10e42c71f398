"""The HKY fast forms' inputs are rounded to nearest: on branches of no length
a pattern's likelihood is the frequency of its state, here between two floats
in [0.5, 1), whose logarithm is taken of a mantissa near 1 (so that FP32's own
logarithm adds below 1e-11).

Tolerance: half a unit in the last place of a float at 0.5, 3e-8 / 0.5, for
the nearest float; cut off, the value would be 1.2e-7 away.  Float-float: a
pair holds 2^-49 of it, its logarithm 1e-13."""
import math

import numpy as np
import pytest

from ima2p_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("share", [0.02, 0.3, 0.49, 0.51, 0.75, 0.98])
@pytest.mark.parametrize("state", range(4))
@pytest.mark.parametrize("n", [2, 5])
def test_frequencies(n, state, share):
    p = 0.5 + (1000 + share) * 2.0 ** -24
    pi = np.full(4, (1.0 - p) / 3)
    pi[state] = p
    g = synth.two_pop_tree(np.random.default_rng(n), n - n // 2, n // 2, 10.0, 0.2, 1.5)
    ctx = api.Context(0)
    ctx.add_locus_hky(np.full((n, 1), state, np.int8), np.ones(1, np.int32), 1)
    ctx.set_chains(1, 1)
    g.time = np.where(g.time > 0, g.time * 1e-30, g.time)
    ctx.set_pi(0, 0, pi)
    ctx.set_genealogy(0, 0, g)
    for prec, tol in ((api.PREC_FP32, 6.1e-8), (api.PREC_FAST, 2e-13)):
        got, st = ctx.eval([0], [0], [1.0], [4.0], precision=prec)
        assert st[0] == 0 and abs(got[0] - math.log(p)) <= tol, (prec, got[0] - math.log(p))
