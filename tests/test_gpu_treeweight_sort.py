"""The weights' event sort: genealogies of 2 events, around a lane's and a
warp's worth, the 128 that are ranked and the first sizes beyond, with times
all different and with times rounded so that many events tie (ties keep the
list's order), one genealogy and batches of several to a warp -- the oracle's
weights bit for bit (the sums' order follows the sort)."""
import numpy as np
import pytest

from ima2p_gb300 import api, popmodel, synth
from oracle import pyoracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("copies", [1, 8, 15, 16, 17, 31, 32, 33, 63, 64, 65, 130])
@pytest.mark.parametrize("grid", [0.0, 0.25])
@pytest.mark.parametrize("ngen", [1, 700])
def test_event_order(copies, grid, ngen):
    pm = popmodel.build("(0,1):2", 2, nomig=True)
    rng = np.random.default_rng(copies + ngen)
    kinds = []
    for _ in range(min(ngen, 5)):
        lg = synth.sim_im_labeled(rng, [copies] * 2, [4.0] * 3, 0.0, [(1.5, 0, 1, 2)])
        if grid:
            lg.g.time = np.where(lg.g.down < 0, lg.g.time, np.ceil(lg.g.time / grid) * grid)
        kinds.append(lg)
    gens = [kinds[k % len(kinds)] for k in range(ngen)]
    packed = api.pack_labelled(gens)
    zero, hval, samp, tv = np.zeros(ngen, np.int32), np.ones(1), np.array([[copies] * 2], np.int32), np.array([[1.5]])
    bad, want = O.treeweight_batch(pm, packed, zero, zero, hval, samp, tv)
    ctx = api.Context(0)
    ctx.set_popmodel(pm, *popmodel.priors(pm, 30.0, 0.0)[:2])
    if bad:
        with pytest.raises(api.ImaError):
            ctx.treeweight(packed, zero, zero, hval, samp, tv)
    else:
        w = ctx.treeweight(packed, zero, zero, hval, samp, tv)
        for f in ("cc", "hcc", "fc", "lens"):
            np.testing.assert_array_equal(w[f], want[f], err_msg=f)
    ctx.close()
