"""The direct form of the split-precision surface (points where most terms
count) against the FP64 form, at the edges of its tiles and groups: one
genealogy, tile remainders (64 genealogies), sizes with and without the
max-only pre-pass, point counts around a warp, every column count of the
model types, and calls whose points are taken both ways.

Tolerance: a term's compensated dot product is within K 2^-46 sum |s phi|
(26 columns, sums below 1,000: 4e-10 in the worst case, far less on average)
and its weight within 3e-14, so the log of the sum agrees within 1e-9; the
effective sample size has twice the weights' relative error."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth
from tests._gpu import ctx_with

pytestmark = pytest.mark.gpu


def rows_of(rng, G, pops, spread):
    """Rows whose terms lie within `spread` nats or so of one another: the
    normaliser is the log density at a central point, plus noise."""
    np_, nm = (3, 2) if pops == 2 else (5, 8)
    rows = synth.peaked_stats(rng, G, np_, nm, pops - 1)
    off = synth.gsamp_layout(np_, nm, pops - 1)
    th, m = 6.0, 1.0
    cc, fc = rows[:, off["cc"]:off["cc"] + np_], rows[:, off["fc"]:off["fc"] + np_]
    mc, fm = rows[:, off["mc"]:off["mc"] + nm], rows[:, off["fm"]:off["fm"] + nm]
    p = (cc * np.log(2 / th) - 2 * fc / th).sum(1) + (mc * np.log(m) - fm * m).sum(1)
    return rows, -p + rng.normal(0.0, spread, G), np_, nm


@pytest.mark.parametrize("G,P,pops,mt,spread", [
    (1, 1, 2, 0, 1.0), (63, 33, 2, 0, 3.0), (64, 32, 3, 1, 3.0), (65, 31, 3, 2, 3.0), (129, 200, 3, 0, 2.0),
    (1023, 1, 3, 0, 2.0), (1024, 5, 2, 1, 3.0), (4097, 130, 2, 2, 5.0), (5000, 300, 3, 0, 4.0),
    (20000, 150, 3, 0, 25.0), (20000, 150, 2, 0, 60.0)])
def test_surface_direct_form(G, P, pops, mt, spread):
    rng = np.random.default_rng(G * 7 + P)
    rows, norm, np_, nm = rows_of(rng, G, pops, spread)
    x = synth.surface_points(rng, P, np_, nm)
    ctx = ctx_with([("sw", 2, 1)])
    ctx.surface_load(rows, np_, nm, pops, lognorm=norm)
    q, ess = ctx.surface_eval(x, modeltype=mt, method=api.SURF_TC)
    q64, ess64 = ctx.surface_eval(x, modeltype=mt, method=api.SURF_FP64)
    assert np.max(np.abs(q - q64)) <= 1e-9
    np.testing.assert_allclose(ess, ess64, rtol=4e-9)
    q2, ess2 = ctx.surface_eval(x, modeltype=mt, method=api.SURF_TC)
    np.testing.assert_array_equal(q2, q)
    np.testing.assert_array_equal(ess2, ess)
