"""2NM densities under the uniform prior by the size of a call: points of one
term around the 32 that share a warp's genealogies, several terms in one call
(padded blocks), genealogy counts around a warp's 32 and a chunk's 128, rows
without events of the term's population or migration (left to the FP64 form),
and points beyond the term's range -- against the oracle, at the 1e-9 that an
ulp of the reference's logarithms makes of single genealogies (see
test_gpu_popmig.py)."""
import os

import numpy as np
import pytest

from ima2p_gb300 import api, synth
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu

GOLD = np.load(os.path.join(os.path.dirname(__file__), "golden", "golden_popmig.npz"))


@pytest.mark.parametrize("G", [1, 31, 32, 33, 129, 400])
@pytest.mark.parametrize("counts", [(1,), (33,), (2, 5, 32), (31, 1, 17, 40)])
def test_blocks_of_points(G, counts):
    rng = np.random.default_rng(G + sum(counts))
    rows = GOLD["rows"][rng.integers(0, len(GOLD["rows"]), G)].copy()
    off = synth.gsamp_layout(3, 2, 1)
    if G > 1:
        none = rng.random(G) < 0.125
        rows[none, off["cc"]:off["cc"] + 3] = 0.0
        rows[none, off["mc"]:off["mc"] + 2] = 0.0
    q, m = GOLD["qmax"], GOLD["mmax"]
    terms = [(0, 0), (1, 1), (0, 1), (1, 0)][:len(counts)]
    th = np.repeat([t for t, _ in terms], counts)
    mi = np.repeat([j for _, j in terms], counts)
    x = q[th] * m[mi] / 2.0 * rng.uniform(0.01, 1.1, len(th))
    order = rng.permutation(len(th))
    th, mi, x = th[order], mi[order], x[order]
    ctx = api.Context(0)
    ctx.surface_load(rows, 3, 2, 2)
    y = ctx.popmig(th, mi, x, q, m)
    want = np.array([O.popmig(rows, 3, 2, int(t), int(j), float(v), q[t], m[j]) for t, j, v in zip(th, mi, x)])
    np.testing.assert_allclose(y, want, rtol=1e-9, atol=1e-300)
    ctx.close()
