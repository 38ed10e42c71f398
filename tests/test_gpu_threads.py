"""Contexts of several threads whose kernels need different amounts of shared
memory: genealogy updates with 12 loci a launch beside some with 5 and with
genealogies of 400 genes, HKY loci of 20 and of 800 genes.  The limit is set
per kernel, so one thread's must hold for the others' launches too.  Results
are those of each context by itself."""
import threading

import numpy as np
import pytest

from ima2p_gb300 import api, popmodel, synth, workloads

pytestmark = pytest.mark.gpu


def updater(nloci, ncopies, nch, seed):
    w = workloads.make_updgen(seed=seed, nloci=nloci, nch=nch, ncopies=ncopies, nbases=100)
    ctx = api.Context(0)
    for L in w.loci:
        ctx.add_locus_hky(L.seq, L.mult, L.totsites)
    ctx.set_chains(1, nch)
    pm = popmodel.build(w.tree, w.npops, nomig=True)
    th_max, th_min, _, _, _ = popmodel.priors(pm, 30.0, 0.0)
    ctx.set_popmodel(pm, th_max, th_min)
    ci, li = np.repeat(np.arange(nch), nloci), np.tile(np.arange(nloci), nch)
    flat = w.base * nch
    cat = lambda f: np.concatenate([getattr(g.g, f) for g in flat])  # noqa: E731
    ctx.set_genealogies(ci, li, cat("up0"), cat("up1"), cat("down"), cat("time"))
    ctx.set_labels(ci, li, flat)
    ctx.set_locus_pops(np.ones(nloci), w.samppop)
    for c in range(nch):
        for l in range(nloci):
            ctx.set_pi(c, l, w.loci[l].pi)
    rngs = [api.UgRng(seed + c) for c in range(nch)]

    def step():
        acc, top, pg = ctx.updategenealogy_sweep(np.arange(nch), np.tile(w.tvals, (nch, 1)), 1, rngs, np.tile(w.u, nch),
                                                 np.tile(w.kappa, nch), precision=api.PREC_FAST)
        return acc, top, pg
    return step


def evaluator(n, S):
    rng = np.random.default_rng(n)
    ctx = api.Context(0)
    ctx.add_locus_hky(rng.integers(0, 4, (n, S)).astype(np.int8), np.ones(S, np.int32), S)
    ctx.set_chains(1, 2)
    g = synth.two_pop_tree(rng, n - n // 2, n // 2, 10.0, 0.2, 1.5)
    for c in range(2):
        ctx.set_pi(c, 0, [0.3, 0.2, 0.2, 0.3])
        ctx.set_genealogy(c, 0, g)
    return lambda: (ctx.eval([0, 1], [0, 0], [1.0, 2.0], [3.0, 4.0])[0],)


def test_threads():
    makers = [lambda: updater(48, 20, 2, 5), lambda: updater(20, 20, 2, 6), lambda: updater(4, 200, 2, 7),
              lambda: evaluator(20, 60), lambda: evaluator(800, 40)]
    steps = 30
    want = []
    for m in makers:
        f = m()
        want.append([f() for _ in range(steps)])
    fs = [m() for m in makers]
    got, errors = [[] for _ in fs], []
    start = threading.Barrier(len(fs))

    def work(k):
        try:
            start.wait()
            for _ in range(steps):
                got[k].append(fs[k]())
        except Exception as e:  # noqa: BLE001
            errors.append((k, e))
    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(fs))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors
    for g, w in zip(got, want):
        for a, b in zip(g, w):
            for x, y in zip(a, b):
                np.testing.assert_array_equal(x, y)
