"""The launch counter of HKY batches that take several launches: one per size
class where the classes fill the device, one more per repeated entry."""
import numpy as np
import pytest

from ima2p_gb300 import api, synth

pytestmark = pytest.mark.gpu


def context(ns, nch):
    rng = np.random.default_rng(len(ns))
    ctx = api.Context(0)
    g = []
    for n in ns:
        ctx.add_locus_hky(rng.integers(0, 4, (n, 3)).astype(np.int8), np.ones(3, np.int32), 3)
        g.append(synth.two_pop_tree(rng, n - n // 2, n // 2, 10.0, 0.2, 1.5))
    ctx.set_chains(1, nch)
    ci = np.repeat(np.arange(nch, dtype=np.int32), len(ns))
    li = np.tile(np.arange(len(ns), dtype=np.int32), nch)
    ctx.set_genealogies(ci, li, *[np.concatenate([getattr(t, f) for t in g] * nch) for f in ("up0", "up1", "down", "time")])
    for c in range(nch):
        for l in range(len(ns)):
            ctx.set_pi(c, l, [0.3, 0.2, 0.2, 0.3])
    return ctx, ci, li


def counted(ctx, f):
    before = ctx.launch_count()
    f()
    return ctx.launch_count() - before


@pytest.mark.parametrize("ns,nch,pairs,kernels", [
    ([4], 8, None, 1),
    ([40, 4], 8, None, 1),           # two classes, too few of each
    ([40, 4], 1500, None, 2),        # two classes that fill the device
    ([4, 6], 1, [(0, 0), (0, 1), (0, 0), (0, 0)], 3),
])
def test_hky_launches(ns, nch, pairs, kernels):
    ctx, ci, li = context(ns, nch)
    if pairs:
        ci, li = np.array(pairs, np.int32).T
    one = np.ones(len(ci))
    ctx.eval(ci, li, one, 2 * one)  # uploads and first allocations
    assert counted(ctx, lambda: ctx.eval(ci, li, one, 2 * one)) == kernels
    b = ctx.batch_create(ci, li, one, 2 * one)
    for graph in (False, True, True):
        assert counted(ctx, lambda: b.run(use_graph=graph)) == kernels
    b64 = ctx.batch_create(ci, li, one, 2 * one, precision=api.PREC_FP64)
    b64.run(use_graph=True)
    assert counted(ctx, lambda: b64.run(use_graph=True)) == (kernels if pairs else 1)
    if not pairs:
        for graph in (False, True):
            b.sweep(1, use_graph=graph)
            assert counted(ctx, lambda: b.sweep(1, use_graph=graph)) == kernels + 2 + (nch >= 2)
