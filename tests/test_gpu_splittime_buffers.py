"""Split-time updates of many chains in one call (parameter blocks of more
than 64 KB, which a copy from pageable memory need not have read when it
returns) against the same moves made one synchronised call at a time:
the times bit for bit, through accepted and rejected moves, with the host's
memory put to other use between the calls."""
import numpy as np
import pytest

from ima2p_gb300 import api, popmodel, splittime, synth

pytestmark = pytest.mark.gpu


def chain_set(nch, nl):
    rng = np.random.default_rng(nch)
    pm = popmodel.build("((0,1):3,2):4", 3)
    gens = [synth.sim_im_labeled(rng, [2, 3, 2], [4.0] * 5, 0.2, [(0.6, 0, 1, 3), (1.4, 3, 2, 4)]) for _ in range(nl)]
    ctx = api.Context(0)
    for g in gens:
        ctx.add_locus_is(synth.is_data(rng, g.g, 1.0, min_sites=1))
    ctx.set_chains(1, nch)
    nth, nmg = len(pm.th_cells), len(pm.mg_cells)
    ctx.set_popmodel(pm, [15.0] * nth, [0.0] * nth, [2.0] * nmg, [0.0] * nmg, [1.0] * nmg)
    cs = splittime.ResidentChainSet(ctx, [gens] * nch, np.tile([0.6, 1.4], (nch, 1)), np.linspace(1.0, 0.5, nch),
                                    np.ones(nl), [[2, 3, 2]] * nl, np.ones(nl))
    return ctx, cs, [len(g.pop) for g in gens]


@pytest.mark.parametrize("nch,nl", [(5, 1), (3000, 1), (2000, 3)])
def test_many_chains(nch, nl):
    a, cs, lines = chain_set(nch, nl)
    b, _, _ = chain_set(nch, nl)
    rng = np.random.default_rng(3)
    chains, rows = np.arange(nch), np.arange(nch)
    tv = np.tile([0.6, 1.4], (nch, 1))
    u = np.ones(nch * nl)
    for step in range(6):
        period = rng.integers(0, 2, nch)
        old = tv[rows, period]
        t_u = np.where(period == 0, 0.0, tv[:, 0])
        t_d = np.where(period == 1, 1000000.0, tv[:, 1])
        new = np.where(period == 0, rng.uniform(0.1, 0.9, nch) * tv[:, 1], tv[:, 0] + rng.uniform(0.1, 1.5, nch))
        lhu = np.log((new - t_u) / (old - t_u))
        lhd = np.log(np.where(period == 1, 1.0, (t_d - new) / (t_d - old)))
        want = rng.random(nch) < [0.5, 0.0, 1.0, 0.1, 0.9, 0.5][step]
        tnew = tv.copy()
        tnew[rows, period] = new
        acc, _, _ = a.changet_ry1_sweep(chains, period, old, new, t_u, t_d, lhu, lhd, np.where(want, -1e300, 1e300), tnew, u)
        np.testing.assert_array_equal(acc, want)
        np.random.default_rng(step).random(200000).sort()  # the host's freed memory written over
        b.rubber_band(chains, period, old, new, t_u, t_d)
        rej = np.flatnonzero(~want)
        if len(rej):
            b.rubber_band(chains[rej], period[rej], old[rej], new[rej], t_u[rej], t_d[rej], inverse=True)
        tv[rows[want], period[want]] = new[want]
        np.testing.assert_array_equal(a.get_split_times(), tv)
        for c in rng.permutation(nch)[:400]:
            for l in range(nl):
                x, y = a.get_times(c, l, lines[l]), b.get_times(c, l, lines[l])
                np.testing.assert_array_equal(x[0], y[0])
                np.testing.assert_array_equal(x[1], y[1])
