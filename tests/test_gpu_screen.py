"""The tensor-core screen with FP16 operands against the FP64 form, where its
operands are hardest: statistics far from 1 and not whole numbers, a column
that is zero throughout, coefficients large enough to be clamped, a bias that
dwarfs the statistics, the most columns it takes, and the edges of its tiles
(128 points, 256 genealogies, the pre-pass from 769 genealogies on).

Tolerance: the screen only selects terms; those left out are 32 nats below
the maximum, under G e^-32 < 1e-9 of the sum.  A term's compensated dot
product is within K 2^-46 < 4.3e-13 of sum |s phi| + |bias|, and so is the
log of the sum."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth
from tests._gpu import ctx_with

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("G,P,np_,nm,scale,xlo", [
    (1, 1, 3, 2, 1.0, 0.5), (255, 127, 5, 8, 1.0, 0.5), (256, 128, 5, 8, 300.0, 0.5), (769, 129, 5, 8, 1e-3, 0.5),
    (3000, 40, 5, 8, 1e5, 0.5), (3000, 140, 7, 8, 7.3, 0.1), (20001, 257, 5, 8, 1.7, 1e-6), (20001, 33, 3, 2, 1e-2, 1e-3)])
def test_screen_keeps_every_term_that_counts(G, P, np_, nm, scale, xlo):
    pops = {5: 2, 13: 3, 15: 4}[np_ + nm]
    rng = np.random.default_rng(G + P + np_)
    rows = synth.peaked_stats(rng, G, np_, nm, pops - 1)
    off = synth.gsamp_layout(np_, nm, pops - 1)
    rows[:, off["fc"]:off["fc"] + np_] *= np.float32(scale * 1.2345)
    rows[:, off["fm"]:off["fm"] + nm] *= np.float32(scale / 3.0)
    rows[:, off["cc"]:off["cc"] + np_] *= max(1, round(scale))
    rows[:, off["mc"] + nm - 1] = 0.0
    norm = rng.normal(0.0, 40.0 * max(scale, 1.0), G)
    x = synth.surface_points(rng, P, np_, nm) * rng.uniform(xlo, 1.0, (P, 1))
    ctx = ctx_with([("sw", 2, 1)])
    ctx.surface_load(rows, np_, nm, pops, lognorm=norm)
    q, ess = ctx.surface_eval(x, modeltype=0, method=api.SURF_TC)
    q64, ess64 = ctx.surface_eval(x, modeltype=0, method=api.SURF_FP64)
    r = np.abs(rows.astype(np.float64))
    cc, fc = r[:, off["cc"]:off["cc"] + np_], r[:, off["fc"]:off["fc"] + np_]
    mc, fm = r[:, off["mc"]:off["mc"] + nm], r[:, off["fm"]:off["fm"] + nm]
    hcc = r[:, off["hcc"]:off["hcc"] + np_].sum(1)
    th, m = x[:, :np_], x[:, np_:]
    mag = (cc.max(0) * np.abs(np.log(2 / th)) + 2 * fc.max(0) / th).sum(1) + \
        (mc.max(0) * np.abs(np.log(m)) + fm.max(0) * m).sum(1) + np.abs(norm).max() + hcc.max()
    assert np.all(np.abs(q - q64) <= 1e-9 + 4.3e-13 * mag), np.max(np.abs(q - q64) / mag)
    np.testing.assert_allclose(ess, ess64, rtol=4e-9 + 2e-12 * mag.max())
