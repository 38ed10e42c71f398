"""The marginal densities' common factors: x (or 1/x) times log2 e is the same
for every genealogy, and a genealogy's base times log2 e for every x, so their
roundings would stay in the sum.

Rates alone (no counts, 4,000 rates near 20, so that the terms' own roundings,
at most 1.8e-15 each and independent, average to below 1e-16) and bases alone
(every genealogy the same), against extended precision.  Tolerance: 4e-16, the
sum's and the result's roundings (1.1e-16 each) and that average; the factor's
own rounding is up to 20 x 1.1e-16 = 2.2e-15."""
import numpy as np
import pytest

from ima2p_gb300 import synth
from tests._gpu import ctx_with

pytestmark = pytest.mark.gpu

L = np.longdouble
NP, NM = 3, 2
OFF = synth.gsamp_layout(NP, NM, 1)


def loaded(rows):
    ctx = ctx_with([("sw", 2, 1)])
    ctx.surface_load(rows.astype(np.float32), NP, NM, 2)
    return ctx


@pytest.mark.parametrize("param", [0, NP])
@pytest.mark.parametrize("each", [1, 300])  # a point a call, and all in one
def test_rates(param, each):
    rng = np.random.default_rng(param + each)
    G, P = 4000, 300 if each > 1 else 40
    r = np.zeros((G, OFF["rowlen"]), np.float32)
    f = rng.uniform(19.5, 20.5, G).astype(np.float32)
    r[:, OFF["fc" if param == 0 else "fm"]] = f / 2 if param == 0 else f
    ctx = loaded(r)
    x = rng.uniform(0.9, 1.1, P)
    got = np.concatenate([ctx.margincalc(np.full(len(c), param), c) for c in np.split(x, range(each, P, each))])
    b = 1.0 / x if param == 0 else x
    want = np.array([np.exp(-f.astype(L) * L(v)).sum() / L(G) for v in b])
    err = np.abs((got.astype(L) - want) / want).astype(float)
    assert err.max() <= 4e-16, err.max()


def test_bases():
    rng = np.random.default_rng(5)
    for q in rng.uniform(-21.0, 21.0, 60).astype(np.float32):
        r = np.zeros((300, OFF["rowlen"]), np.float32)
        r[:, OFF["qi"]] = r[:, OFF["mi"] + 1] = q
        ctx = loaded(r)
        want = np.exp(-L(q))
        for param in (0, NP + 1):
            got = ctx.margincalc([param], [1.0])
            assert abs((L(got[0]) - want) / want) <= 4e-16, (q, got)
