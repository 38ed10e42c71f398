"""The tensor-core surface over genealogies some of which have no weight: a log
normaliser of -inf, or an infinite rate.  The others count as if those were
absent (but for log G), in calls taken by the direct form, by the screen with
and without its pre-pass, and by both.

Tolerance: that of test_gpu_screen (a compensated dot product within K 2^-46
of its terms, and the terms left out); both calls have it, hence twice."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth
from tests._gpu import ctx_with

pytestmark = pytest.mark.gpu


def surface(rows, norm, np_, nm, x):
    ctx = ctx_with([("sw", 2, 1)])
    ctx.surface_load(rows, np_, nm, 3, lognorm=norm)
    first = ctx.surface_eval(x, modeltype=0, method=api.SURF_TC)
    again = ctx.surface_eval(x, modeltype=0, method=api.SURF_TC)
    for a, b in zip(first, again):
        np.testing.assert_array_equal(a, b)
    return first


@pytest.mark.parametrize("what", ["norm", "fc", "fm"])
@pytest.mark.parametrize("G,P,spread", [(300, 20, 3.0), (900, 130, 60.0), (5000, 40, 3.0), (5000, 200, 100.0),
                                        (20000, 150, 25.0)])
def test_genealogies_without_weight(G, P, spread, what):
    rng = np.random.default_rng(G + P)
    np_, nm = 5, 8
    rows = synth.peaked_stats(rng, G, np_, nm, 2)
    off = synth.gsamp_layout(np_, nm, 2)
    cc, fc = rows[:, off["cc"]:off["cc"] + np_], rows[:, off["fc"]:off["fc"] + np_]
    mc, fm = rows[:, off["mc"]:off["mc"] + nm], rows[:, off["fm"]:off["fm"] + nm]
    p = (cc * np.log(2 / 6.0) - 2 * fc / 6.0).sum(1) - fm.sum(1)
    norm = -p + rng.normal(0.0, spread, G)
    x = synth.surface_points(rng, P, np_, nm)
    gone = np.zeros(G, bool)
    gone[rng.choice(G, 7, replace=False)] = True
    want, wess = surface(rows[~gone], norm[~gone], np_, nm, x)
    r, v = rows.copy(), norm.copy()
    if what == "norm":
        v[gone] = -np.inf
    else:
        r[gone, off[what]] = np.inf
    q, ess = surface(r, v, np_, nm, x)
    mag = np.abs(norm).max() + 100 * np.abs(p).max()
    np.testing.assert_allclose(q, want + np.log(G / (G - 7)), rtol=0, atol=2e-9 + 8.6e-13 * mag)
    np.testing.assert_allclose(ess, wess, rtol=1e-8 + 4e-12 * mag)
