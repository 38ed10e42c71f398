"""Performance cases of the library: what an IMa2p-style host program has it do.

Every case goes through the public Python view of the C ABI
(ima2p_gb300.api), with host arrays in and host arrays out, as such a program
calls it; the resident state (loci, genealogies, partial likelihoods,
population labels, saved-genealogy rows) is what the program keeps between
calls.  prepare() makes that state from a seed, run() is one pass, exact()
gives the same outputs from plain FP64 numpy / torch, and work() the bytes
and operations a pass cannot do without.

The kinds of case, with the sizes of the repository's own workloads:

  mc3_is     one MC3 step of the small infinite-sites model: new node times
             and likelihoods of every chain-locus, commit, temperature swaps
  hky        likelihoods of every HKY chain-locus after a re-timing move
  hky_edit   one locus's genealogy proposals on every chain: new topologies,
             pruning from the edited edges, commit
  sw         likelihoods of every stepwise chain-locus after a re-timing move
  mixed      the same for HKY and stepwise loci of uneven size together
  surface    jointp at many points: a differential-evolution generation over
             a two-population run's saved genealogies (prior integrals in the
             rows), or a parameter grid with a log normaliser per genealogy
  curves     the 1-D marginal curves of every parameter
  popmig     the 2NM curves
  splittime  one split-time update of every resident chain
  genealogy  genealogy updates of resident chains, HKY or stepwise loci
"""
import math

import numpy as np
import torch

from ima2p_gb300 import api, popmodel, splittime, synth

THETA_MAX, MIG_MAX = 20.0, 2.0


# ------------------------------------------------------------------- cases
def listed():
    return [
        # the smallest call: twenty chain-loci of twenty genes, where launches
        # and copies are all there is (the infinite-sites configuration)
        {"name": "mc3_is_small", "kind": "mc3_is", "loci": 5, "copies": 10, "chains": 4},
        # a host-side proposal loop: one locus of 32 chains at a time
        {"name": "hky_edits", "kind": "hky_edit", "copies": 20, "bases": 1000, "chains": 32},
        # the HKY configuration: 50 loci x (20+20) x 1000 bp, 32 chains
        {"name": "hky_full", "kind": "hky", "loci": 50, "copies": 20, "bases": 1000, "chains": 32},
        # the stepwise configuration: 100 loci x 90 copies, 64 chains
        {"name": "sw_full", "kind": "sw", "loci": 100, "copies": 30, "chains": 64},
        # the mixed configuration's loci (U(4,60) copies per population,
        # U(200,3000) bp) in one run of 128 chains
        {"name": "mixed_300", "kind": "mixed", "hky": 200, "sw": 100, "chains": 128},
        # one generation of the peak search: 100 trial vectors per parameter
        {"name": "surface_search", "kind": "surface", "pops": 2, "G": 100000, "P": 500, "grid": False},
        # the surface configuration's genealogies, half its grid
        {"name": "surface_grid", "kind": "surface", "pops": 3, "G": 2097152, "P": 32768, "grid": True},
        # every marginal curve of a three-population model
        {"name": "curves", "kind": "curves", "pops": 3, "G": 100000, "points": 1000},
        # its eight 2NM curves
        {"name": "popmig", "kind": "popmig", "terms": 8, "G": 10000, "points": 1000},
        # one split-time update of each of 128 chains
        {"name": "splittime", "kind": "splittime", "loci": 100, "chains": 128},
        # genealogy updates between two swap steps, few chains and many
        {"name": "genealogy_hky", "kind": "genealogy", "model": "hky", "loci": 50, "copies": 20, "chains": 32,
         "sweeps": 2},
        {"name": "genealogy_sw", "kind": "genealogy", "model": "sw", "loci": 100, "copies": 30, "chains": 64,
         "sweeps": 2},
    ]


def _between(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.49)))))))


def draw(rng):
    kind = rng.choice(["mc3_is", "hky_edit", "hky", "sw", "mixed", "surface", "surface", "curves", "popmig",
                       "splittime", "genealogy"])
    if kind == "mc3_is":
        return {"kind": kind, "loci": _between(rng, 2, 60), "copies": _between(rng, 4, 50),
                "chains": _between(rng, 2, 64)}
    if kind == "hky_edit":
        return {"kind": kind, "copies": _between(rng, 4, 60), "bases": _between(rng, 200, 3000),
                "chains": _between(rng, 1, 128)}
    if kind == "hky":
        return {"kind": kind, "loci": _between(rng, 1, 50), "copies": _between(rng, 3, 40),
                "bases": _between(rng, 200, 3000), "chains": _between(rng, 1, 64)}
    if kind == "sw":
        return {"kind": kind, "loci": _between(rng, 1, 100), "copies": _between(rng, 3, 60),
                "chains": _between(rng, 1, 128)}
    if kind == "mixed":
        return {"kind": kind, "hky": _between(rng, 10, 200), "sw": _between(rng, 5, 100),
                "chains": _between(rng, 4, 128)}
    if kind == "surface":
        return {"kind": kind, "pops": rng.choice([2, 3]), "G": _between(rng, 1000, 2000000),
                "P": _between(rng, 1, 16384), "grid": rng.random() < 0.5}
    if kind == "curves":
        return {"kind": kind, "pops": rng.choice([2, 3]), "G": _between(rng, 1000, 100000),
                "points": _between(rng, 100, 1000)}
    if kind == "popmig":
        return {"kind": kind, "terms": rng.randint(1, 8), "G": _between(rng, 500, 10000),
                "points": _between(rng, 100, 1000)}
    if kind == "splittime":
        return {"kind": kind, "loci": _between(rng, 4, 100), "chains": _between(rng, 4, 128)}
    if rng.random() < 0.5:
        return {"kind": kind, "model": "hky", "loci": _between(rng, 4, 50), "copies": _between(rng, 4, 30),
                "chains": _between(rng, 2, 128), "sweeps": rng.randint(1, 2)}
    return {"kind": kind, "model": "sw", "loci": _between(rng, 4, 100), "copies": _between(rng, 4, 30),
            "chains": _between(rng, 2, 128), "sweeps": rng.randint(1, 2)}


# ------------------------------------------------------------- genealogies
def _rescaled(g, f):
    """Node times of a genealogy with every time scaled by f (root: -1)."""
    return np.where(g.time >= 0, g.time * f, g.time)


def _moved(rng, g, tries=20):
    """g after one prune-and-regraft below the root: (genealogy, the four
    edges whose length or attachment changed), or (copy, None)."""
    h = g.copy()
    n = h.n
    low = np.where(h.up0 >= 0, h.time[np.maximum(h.up0, 0)], 0.0)  # time of node c itself
    for _ in range(tries):
        e = int(rng.integers(2 * n - 1))
        p = int(h.down[e])
        if e == h.root or p < 0 or p == h.root:
            continue
        s = int(h.up1[p] if h.up0[p] == e else h.up0[p])
        gp = int(h.down[p])
        f = int(rng.integers(2 * n - 1))
        if f in (e, p, s, h.root):
            continue
        c, inside = f, False
        while c >= 0:  # not below the pruned edge
            if c == e:
                inside = True
                break
            c = int(h.down[c])
        fp = int(h.down[f])
        if inside or fp < 0:
            continue
        lo, hi = max(low[e], low[f]), h.time[f]
        if not hi > lo * 1.0001 + 1e-9:
            continue
        t = float(rng.uniform(lo + 0.05 * (hi - lo), hi - 0.05 * (hi - lo)))
        for q, old, new in ((gp, p, s),):  # the sister takes the freed node's place
            if h.up0[q] == old:
                h.up0[q] = new
            else:
                h.up1[q] = new
        h.down[s] = gp
        h.time[s] = h.time[p]
        fp = int(h.down[f])
        top = float(h.time[f])
        if h.up0[fp] == f:
            h.up0[fp] = p
        else:
            h.up1[fp] = p
        h.up0[p], h.up1[p] = e, f
        h.down[e] = h.down[f] = p
        h.down[p] = fp
        h.time[e] = h.time[f] = t
        h.time[p] = top
        return h, [e, s, f, p]
    return g.copy(), None


def _variants(rng, g, count, moves):
    """count genealogies around g: g after `moves` random regrafts each."""
    out = []
    for _ in range(count):
        h = g
        for _ in range(moves):
            h, _ = _moved(rng, h)
        out.append(h)
    return out


def _rates(rng, n):
    u = rng.lognormal(0.0, 0.5, n)
    return u / np.exp(np.mean(np.log(u)))


class _Chains:
    """Genealogies of every chain-locus: per locus a few topologies, per
    chain-locus one of them with its times rescaled."""

    def __init__(self, rng, variants, nch, scale=0.15):
        nl = len(variants)
        self.variants, self.nch, self.nl = variants, nch, nl
        self.which = np.stack([(np.arange(nch) + rng.integers(1 << 20)) % len(v) for v in variants], axis=1)
        self.fac = np.exp(rng.normal(0.0, scale, (nch, nl)))
        self.ci = np.repeat(np.arange(nch, dtype=np.int32), nl)
        self.li = np.tile(np.arange(nl, dtype=np.int32), nch)
        self.scale = scale

    def tree(self, c, l):
        return self.variants[l][self.which[c, l]]

    def nodes(self):
        gs = [self.tree(c, l) for c in range(self.nch) for l in range(self.nl)]
        cat = lambda f: np.concatenate([getattr(g, f) for g in gs])  # noqa: E731
        return cat("up0"), cat("up1"), cat("down")

    def times(self, fac):
        return np.concatenate([_rescaled(self.tree(c, l), fac[c, l])
                               for c in range(self.nch) for l in range(self.nl)])


def _alleles(rng, g, A, n, steps=0.2):
    """Allele states of another chain: some internal states a step away."""
    B = A.copy()
    inner = np.arange(n, 2 * n - 1)
    flip = rng.uniform(size=len(inner)) < steps
    B[inner[flip]] += rng.choice([-1, 1], size=int(flip.sum()))
    return np.maximum(B, 4).astype(np.int32)


# -------------------------------------------- likelihoods: mc3_is, hky, sw, mixed
def _loci(case, seed):
    """The loci, chain genealogies and parameters of a likelihood case."""
    rng = np.random.default_rng([seed, 17])
    kind, nch = case["kind"], case["chains"]
    loci, variants = [], []
    if kind == "mc3_is":
        u = _rates(rng, case["loci"])
        for l in range(case["loci"]):
            g = synth.two_pop_tree(rng, case["copies"], case["copies"], 5.0, 0.1, 1.0)
            loci.append(("is", synth.is_data(rng, g, float(u[l]), min_sites=3)))
            variants.append([g])
    elif kind == "hky":
        u = _rates(rng, case["loci"])
        for l in range(case["loci"]):
            g = synth.two_pop_tree(rng, case["copies"], case["copies"], 10.0, 0.2, 1.5)
            kap = float(rng.uniform(2.0, 8.0))
            loci.append(("hky", synth.hky_data(rng, g, case["bases"], float(u[l]), kap, rng.dirichlet([5] * 4)), kap))
            variants.append(_variants(rng, g, min(8, nch), max(2, g.n // 4)))
    elif kind == "sw":
        u = _rates(rng, case["loci"])
        for l in range(case["loci"]):
            g = synth.three_pop_tree(rng, [case["copies"]] * 3, 4.0, 0.05)
            loci.append(("sw", g.n, synth.sw_alleles(rng, g, float(u[l]))))
            variants.append([g])
    else:  # mixed: sixty distinct loci, repeated with other rates
        nb = case["hky"] + case["sw"]
        u = _rates(rng, nb)
        base = []
        for k in range(min(40, case["hky"])):
            g = synth.three_pop_tree(rng, [int(v) for v in rng.integers(4, 61, 3)], 10.0, 0.05)
            kap = float(rng.uniform(2.0, 8.0))
            d = synth.hky_data(rng, g, int(rng.integers(200, 3001)), float(rng.lognormal(0.0, 0.5)), kap,
                               rng.dirichlet([5] * 4))
            base.append((("hky", d, kap), _variants(rng, g, 2, max(2, g.n // 4))))
        sbase = []
        for k in range(min(20, case["sw"])):
            g = synth.three_pop_tree(rng, [int(v) for v in rng.integers(4, 61, 3)], 4.0, 0.05)
            sbase.append((("sw", g.n, synth.sw_alleles(rng, g, float(rng.lognormal(0.0, 0.5)))), [g]))
        for l in range(nb):
            spec, v = base[l % len(base)] if l < case["hky"] else sbase[(l - case["hky"]) % len(sbase)]
            loci.append(spec)
            variants.append(v)
    ch = _Chains(rng, variants, nch)
    par = np.tile(np.array([x[2] if x[0] == "hky" else 1.0 for x in loci]), nch)
    al = {}
    for l, x in enumerate(loci):
        if x[0] == "sw":
            g = variants[l][0]
            for c in range(nch):
                al[(c, l)] = x[2] if c == 0 else _alleles(rng, g, x[2], x[1])
    fac2 = np.exp(rng.normal(0.0, ch.scale, (nch, ch.nl)))  # the re-timing move
    return loci, ch, np.tile(u, nch), par, al, ch.fac * fac2, rng


def _context(loci, nch):
    ctx = api.Context(0)
    for x in loci:
        if x[0] == "is":
            ctx.add_locus_is(x[1])
        elif x[0] == "hky":
            ctx.add_locus_hky(x[1].seq, x[1].mult, x[1].totsites)
        else:
            ctx.add_locus_sw(x[1], 1)
    ctx.set_chains(1, nch)
    return ctx


def _prepare_likelihood(case, seed):
    loci, ch, u, par, al, fac, rng = _loci(case, seed)
    nch = case["chains"]
    ctx = _context(loci, nch)
    up0, up1, down = ch.nodes()
    ctx.set_genealogies(ch.ci, ch.li, up0, up1, down, ch.times(ch.fac))
    for l, x in enumerate(loci):
        for c in range(nch):
            if x[0] == "hky":
                ctx.set_pi(c, l, x[1].pi)
            elif x[0] == "sw":
                ctx.set_alleles(c, l, al[(c, l)])
    ctx.eval(ch.ci, ch.li, u, par)
    ctx.commit(ch.ci, ch.li, np.ones(len(ch.ci), np.uint8))
    s = {"kind": case["kind"], "ctx": ctx, "ci": ch.ci, "li": ch.li, "time": ch.times(fac), "u": u, "par": par,
         "all": np.ones(len(ch.ci), np.uint8)}
    if case["kind"] == "mc3_is":
        ctx.setheat(0.9, 0.8, 1)
        ctx.set_probg(rng.normal(-50.0, 2.0, nch))
        s["uniform"] = np.random.default_rng([seed, 18])
    return s


def _run_likelihood(s):
    ctx = s["ctx"]
    res, st = ctx.eval_times(s["ci"], s["li"], s["time"], s["u"], s["par"])
    if s["kind"] != "mc3_is":
        return {"loglik": res, "status": st}
    ctx.commit(s["ci"], s["li"], s["all"])
    tries = max(1, ctx.nchains - 1)
    ok, used = ctx.swapchains(tries, True, uniforms=s["uniform"].random((1, 64 + 64 * tries)))
    return {"loglik": res, "status": st, "swaps": ok, "used": used, "betas": ctx.get_betas()}


def _exact_likelihood(case, seed):
    loci, ch, u, par, al, fac, _ = _loci(case, seed)
    nch, nl = case["chains"], len(loci)
    u, par = u.reshape(nch, nl), par.reshape(nch, nl)
    res = np.zeros((nch, nl))
    for l, x in enumerate(loci):
        for v, g in enumerate(ch.variants[l]):
            cs = np.flatnonzero(ch.which[:, l] == v)
            if not len(cs):
                continue
            t = np.stack([_rescaled(g, fac[c, l]) for c in cs])
            if x[0] == "is":
                res[cs, l] = _is64(x[1], g, t, u[cs, l])
            elif x[0] == "hky":
                res[cs, l] = _hky64(x[1], g, t, u[cs, l], par[cs, l])
            else:
                res[cs, l] = _sw64(np.stack([al[(c, l)] for c in cs]), g, t, u[cs, l])
    out = {"loglik": res.reshape(-1), "status": None}
    if case["kind"] == "mc3_is":
        out |= {"swaps": None, "used": None, "betas": None}
    return out


def _lengths(g, t):
    """Branch lengths [B, nodes] of node times t (0 at the root)."""
    low = np.where(g.up0 >= 0, t[:, np.maximum(g.up0, 0)], 0.0)
    b = t - low
    b[:, g.root] = 0.0
    return b


def _is64(seq, g, t, u):
    """sum over sites of log(branch u), less length u and sum log k!."""
    b = _lengths(g, t)
    n = g.n
    below = {}
    for c in synth.postorder(g):
        below[c] = frozenset([c]) if g.up0[c] < 0 else below[g.up0[c]] | below[g.up1[c]]
    every = frozenset(range(n))
    edge = {}
    for c in range(2 * n - 1):
        if c != g.root:
            edge.setdefault(below[c], []).append(c)
            edge.setdefault(every - below[c], []).append(c)
    total = -b.sum(axis=1) * u
    count = {}
    for k in range(seq.shape[1]):
        on = sorted(set(edge[frozenset(np.flatnonzero(seq[:, k]).tolist())]))
        total = total + np.log(b[:, on].sum(axis=1) * u)
        node = int(g.down[on[0]])
        count[node] = count.get(node, 0) + 1
    return total - sum(math.lgamma(k + 1) for k in count.values())


def _hky64(loc, g, t, u, kappa):
    """HKY85 pruning of one topology for B sets of node times."""
    pi = np.asarray(loc.pi, np.float64)
    sf = np.array([synth.hky_standfactor(pi, k) for k in kappa])
    b = _lengths(g, t) * (u / (loc.totsites * sf))[:, None]
    P2 = np.array([pi[0] + pi[2], pi[1] + pi[3]] * 2)
    A = 1.0 + P2[None, :] * (kappa[:, None] - 1.0)
    part = {}
    for c in synth.postorder(g):
        if c == g.root:
            continue
        # P(b) with 1 - exp taken from expm1: short branches do not cancel
        e1 = -np.expm1(-b[:, c])[:, None]
        e2 = -np.expm1(-b[:, c][:, None] * A)
        own = pi / P2 * (e2 - e1 * (1.0 - P2))          # [B, k], within the class of k
        M = np.repeat((pi * e1)[:, None, :], 4, axis=1)  # [B, j, k]
        for k in range(4):
            M[:, k ^ 2, k] = own[:, k]
            M[:, k, k] = own[:, k] + 1.0 - e2[:, k]
        if g.up0[c] < 0:
            v = np.transpose(M[:, :, loc.seq[c]], (0, 2, 1))
        else:
            v = (part.pop(g.up0[c]) * part.pop(g.up1[c])) @ np.transpose(M, (0, 2, 1))
        part[c] = v
    L = (part[g.up0[g.root]] * part[g.up1[g.root]]) @ pi
    return np.log(L) @ loc.mult.astype(np.float64)


_I0S = [1.0, 3.5156229, 3.0899424, 1.2067492, 0.2659732, 0.360768e-1, 0.45813e-2]
_I0L = [0.39894228, 0.1328592e-1, 0.225319e-2, -0.157565e-2, 0.916281e-2, -0.2057706e-1, 0.2635537e-1, -0.1647633e-1,
        0.392377e-2]
_I1S = [0.5, 0.87890594, 0.51498869, 0.15084934, 0.2658733e-1, 0.301532e-2, 0.32411e-3]
_I1L = [0.39894228, -0.3988024e-1, -0.362018e-2, 0.163801e-2, -0.1031555e-1, 0.2282967e-1, -0.2895312e-1,
        0.1787654e-1, -0.420059e-2]


def _logbessi01(n, x):
    """log of Abramowitz & Stegun 9.8.1-9.8.4 (order 0 or 1) minus x."""
    small = x < 3.75
    y = np.where(small, (x / 3.75) ** 2, 3.75 / np.maximum(x, 3.75))
    S, L = (_I0S, _I0L) if n == 0 else (_I1S, _I1L)
    p = np.where(small, np.polynomial.polynomial.polyval(y, S), np.polynomial.polynomial.polyval(y, L))
    if n == 1:
        p = np.where(small, p * x, p)
    return np.log(p) + np.where(small, -x, -0.5 * np.log(np.maximum(x, 3.75)))


def _sw64(A, g, t, u):
    """sum over branches of log(bessi(|d|, x)) - x, Miller's recurrence for
    |d| >= 2 started at 2 (|d| + floor(sqrt(40 |d|)))."""
    b = _lengths(g, t)
    keep = np.flatnonzero(g.down >= 0)
    x = b[:, keep] * u[:, None]
    d = np.abs(A[:, keep] - A[:, g.down[keep]])
    term = np.zeros_like(x)
    for n in np.unique(d):
        at = d == n
        xs = x[at]
        if n <= 1:
            term[at] = _logbessi01(int(n), xs)
            continue
        tox = 2.0 / xs
        bip, bi, ans = np.zeros_like(xs), np.ones_like(xs), np.zeros_like(xs)
        lb = np.zeros_like(xs)  # log scale taken out of bi after ans was set
        for j in range(2 * (int(n) + int(math.sqrt(40.0 * n))), 0, -1):
            bim = bip + j * tox * bi
            bip, bi = bi, bim
            big = np.abs(bi) > 1e10
            bi = np.where(big, bi * 1e-10, bi)
            bip = np.where(big, bip * 1e-10, bip)
            if j < n:
                lb = lb + np.where(big, -10.0 * math.log(10.0), 0.0)
            if j == n:
                ans = bip.copy()
                lb = np.zeros_like(xs)
        term[at] = np.log(ans) + lb - np.log(bi) + _logbessi01(0, xs)
    return term.sum(axis=1)


def _work_likelihood(case):
    nch = case["chains"]
    if case["kind"] == "mc3_is":
        n = 2 * case["copies"]
        items, sites = nch * case["loci"], 10
        return {"bytes": items * ((2 * n - 1) * 16 + n * sites + 28), "flops": items * sites * 60}
    if case["kind"] == "sw":
        n = 3 * case["copies"]
        return {"bytes": nch * case["loci"] * ((2 * n - 1) * 20 + 28), "flops": nch * case["loci"] * (2 * n - 2) * 35}
    if case["kind"] == "hky":
        n, S, items = 2 * case["copies"], 60, nch * case["loci"]
        return {"bytes": items * ((n - 1) * S * 20 + (2 * n - 1) * 16 + 28), "flops": items * (n - 1) * S * 28}
    n, S = 96, 80  # mean copies and site patterns of the mixed loci
    hi, si = nch * case["hky"], nch * case["sw"]
    return {"bytes": hi * ((n - 1) * S * 20 + (2 * n - 1) * 16 + 28) + si * ((2 * n - 1) * 20 + 28),
            "flops": hi * (n - 1) * S * 28 + si * (2 * n - 2) * 35}


# ---------------------------------------------------------------- hky_edit
def _edit_inputs(case, seed):
    rng = np.random.default_rng([seed, 21])
    nch = case["chains"]
    g = synth.two_pop_tree(rng, case["copies"], case["copies"], 10.0, 0.2, 1.5)
    kap = float(rng.uniform(2.0, 8.0))
    loc = synth.hky_data(rng, g, case["bases"], float(rng.lognormal(0.0, 0.5)), kap, rng.dirichlet([5] * 4))
    old, new, edits = [], [], []
    for _ in range(nch):
        a = _variants(rng, g, 1, max(1, g.n // 8))[0]
        a.time = _rescaled(a, float(np.exp(rng.normal(0.0, 0.15))))
        e = None
        while e is None:  # small genealogies: a move may not fit at once
            b, e = _moved(rng, a)
            if e is None and g.n < 6:
                e = [int(a.up0[a.root]), int(a.up1[a.root]), -1, -1]
        old.append(a)
        new.append(b)
        edits.append(e)
    u = np.full(nch, float(rng.lognormal(0.0, 0.3)))
    return loc, old, new, np.array(edits, np.int32), u, np.full(nch, kap)


def _prepare_edit(case, seed):
    loc, old, new, edits, u, kap = _edit_inputs(case, seed)
    nch = case["chains"]
    ctx = _context([("hky", loc)], nch)
    ci, li = np.arange(nch, dtype=np.int32), np.zeros(nch, np.int32)
    pack = lambda gs: [np.concatenate([getattr(g, f) for g in gs])  # noqa: E731
                       for f in ("up0", "up1", "down", "time")]
    for c in range(nch):
        ctx.set_pi(c, 0, loc.pi)
    ctx.set_genealogies(ci, li, *pack(old))
    ctx.eval(ci, li, u, kap)
    ctx.commit(ci, li, np.ones(nch, np.uint8))
    return {"kind": "hky_edit", "ctx": ctx, "ci": ci, "li": li, "to": [pack(new), pack(old)], "edits": edits, "u": u,
            "par": kap, "all": np.ones(nch, np.uint8), "pass": 0}


def _run_edit(s):
    ctx = s["ctx"]
    ctx.set_genealogies(s["ci"], s["li"], *s["to"][s["pass"] & 1])  # there and, the next time, back
    s["pass"] += 1
    res, st = ctx.eval(s["ci"], s["li"], s["u"], s["par"], edits=s["edits"])
    ctx.commit(s["ci"], s["li"], s["all"])
    return {"loglik": res, "status": st}


def _exact_edit(case, seed):
    loc, _, new, _, u, kap = _edit_inputs(case, seed)
    return {"loglik": np.array([_hky64(loc, g, g.time[None, :], u[c:c + 1], kap[c:c + 1])[0]
                                for c, g in enumerate(new)]), "status": None}


def _work_edit(case):
    n, S = 2 * case["copies"], 60
    dirty = min(n - 1, 2 + 2 * int(math.log2(n)))
    return {"bytes": case["chains"] * (dirty * S * 60 + (2 * n - 1) * 20 + 32), "flops": case["chains"] * dirty * S * 28}


# ------------------------------------------------------- saved genealogies
def _shape(pops):
    np_ = 2 * pops - 1
    return np_, {2: 2, 3: 8}[pops]


def _saved_rows(seed, G, pops):
    """Saved-genealogy rows of a run whose marginals peak inside the priors
    (theta <= 20, m <= 2), with the prior integrals of every genealogy."""
    np_, nm = _shape(pops)
    off = synth.gsamp_layout(np_, nm, pops - 1)
    gen = torch.Generator(device="cuda").manual_seed(seed * 7 + 3)
    f64 = dict(device="cuda", dtype=torch.float64)
    U = lambda n, lo, hi: lo + (hi - lo) * torch.rand((G, n), generator=gen, **f64)  # noqa: E731
    cc = torch.poisson(torch.full((G, np_), 15.0, **f64), generator=gen).clamp_(min=2.0)
    fc = (cc * U(np_, 1.0, 5.0)).float().double()
    mc = torch.poisson(torch.full((G, nm), 4.0, **f64), generator=gen)
    fm = (mc.clamp(min=0.5) / U(nm, 0.3, 2.0)).float().double()
    q = torch.lgamma(cc - 1) + torch.log(torch.special.gammaincc(cc - 1, 2 * fc / THETA_MAX)) + math.log(2.0) + \
        (1 - cc) * torch.log(fc)
    m = torch.lgamma(mc + 1) + torch.log(torch.special.gammainc(mc + 1, fm * MIG_MAX)) - (mc + 1) * torch.log(fm)
    rows = torch.zeros((G, off["rowlen"]), **f64)
    for name, v in (("cc", cc), ("fc", fc), ("mc", mc), ("fm", fm), ("qi", q), ("mi", m)):
        rows[:, off[name]:off[name] + v.shape[1]] = v
    rows[:, off["pdg"]] = -100.0 + 5.0 * torch.randn(G, generator=gen, **f64)
    rows[:, off["probg"]] = q.sum(1) + m.sum(1)
    rows[:, off["t"]:off["t"] + pops - 1] = U(pops - 1, 0.1, 3.0)
    return rows.float()


def _grid_rows(seed, G, pops):
    """The surface benchmark's rows: cc ~ Poisson(8), fc ~ Gamma(4, 1),
    mc ~ Poisson(1), fm ~ Gamma(2, 1), log normaliser ~ N(-200, 20)."""
    np_, nm = _shape(pops)
    off = synth.gsamp_layout(np_, nm, pops - 1)
    gen = torch.Generator(device="cuda").manual_seed(seed * 7 + 5)
    rows = torch.zeros((G, off["rowlen"]), device="cuda")
    U = lambda n: torch.rand((G, n), generator=gen, device="cuda").clamp_(min=1e-30)  # noqa: E731
    rows[:, off["cc"]:off["cc"] + np_] = torch.poisson(torch.full((G, np_), 8.0, device="cuda"), generator=gen)
    rows[:, off["fc"]:off["fc"] + np_] = -sum(torch.log(U(np_)) for _ in range(4))
    rows[:, off["mc"]:off["mc"] + nm] = torch.poisson(torch.full((G, nm), 1.0, device="cuda"), generator=gen)
    rows[:, off["fm"]:off["fm"] + nm] = -sum(torch.log(U(nm)) for _ in range(2))
    norm = -200.0 + 20.0 * torch.randn(G, generator=gen, device="cuda", dtype=torch.float64)
    rows[:, off["probg"]] = -norm.float()
    return rows, norm


def _surface_inputs(case, seed):
    np_, nm = _shape(case["pops"])
    rng = np.random.default_rng([seed, 31])
    if case["grid"]:
        rows, norm = _grid_rows(seed, case["G"], case["pops"])
    else:
        rows, norm = _saved_rows(seed, case["G"], case["pops"]), None
    x = synth.surface_points(rng, case["P"], np_, nm, THETA_MAX, MIG_MAX)
    # a two-population search runs the full model; three populations the
    # population sizes alone (the grid: the full model with its normaliser)
    model = 0 if case["grid"] or case["pops"] == 2 else 1
    return rows, norm, x, model


def _prepare_surface(case, seed):
    rows, norm, x, model = _surface_inputs(case, seed)
    np_, nm = _shape(case["pops"])
    ctx = api.Context(0)
    ctx.surface_load(rows.cpu().numpy(), np_, nm, case["pops"], None if norm is None else norm.cpu().numpy())
    return {"kind": "surface", "ctx": ctx, "x": x, "model": model}


def _run_surface(s):
    q, ess = s["ctx"].surface_eval(s["x"], s["model"])
    return {"q": q, "ess": ess}


def _exact_surface(case, seed):
    rows, norm, x, model = _surface_inputs(case, seed)
    if case["G"] * case["P"] > 1 << 37:
        return None
    np_, nm = _shape(case["pops"])
    off = synth.gsamp_layout(np_, nm, case["pops"] - 1)
    X = torch.from_numpy(x).cuda()
    phi = torch.cat([math.log(2.0) - torch.log(X[:, :np_]), -2.0 / X[:, :np_], torch.log(X[:, np_:]), -X[:, np_:]], 1)
    use = [True] * 2 * np_ + [model == 0] * 2 * nm
    phi = phi * torch.tensor(use, device="cuda", dtype=torch.float64)
    q, ess = [], []
    step = max(1, (1 << 29) // case["P"])
    best = torch.full((case["P"],), -math.inf, device="cuda", dtype=torch.float64)
    s1, s2 = torch.zeros_like(best), torch.zeros_like(best)
    for a in range(0, case["G"], step):
        r = rows[a:a + step].double()
        if norm is not None:
            bias = norm[a:a + step]
        elif case["pops"] == 2:
            bias = -r[:, off["probg"]]
        else:
            bias = -r[:, off["qi"]:off["qi"] + np_].sum(1)
        st = torch.cat([r[:, off[k]:off[k] + n] for k, n in (("cc", np_), ("fc", np_), ("mc", nm), ("fm", nm))], 1)
        p = torch.addmm(bias[None, :], phi, st.t())
        m = torch.maximum(best, p.max(1).values)
        e = p.sub_(m[:, None]).exp_()
        f = torch.exp(best - m)
        s1 = s1 * f + e.sum(1)
        s2 = s2 * f * f + e.square_().sum(1)
        best = m
    return {"q": (math.log(case["G"]) - best - torch.log(s1)), "ess": s1 * s1 / s2}


def _work_surface(case):
    np_, nm = _shape(case["pops"])
    K = 2 * (np_ + nm) if case["grid"] or case["pops"] == 2 else 2 * np_
    return {"bytes": case["G"] * (K + 2) * 4 + case["P"] * (np_ + nm + 2) * 8, "flops": 2 * K * case["G"] * case["P"]}


def _prepare_saved(case, seed):
    pops = case.get("pops", 3)
    np_, nm = _shape(pops)
    ctx = api.Context(0)
    ctx.surface_load(_saved_rows(seed, case["G"], pops).cpu().numpy(), np_, nm, pops)
    s = {"kind": case["kind"], "ctx": ctx, "points": case["points"]}
    if case["kind"] == "curves":
        s |= {"lo": np.zeros(np_ + nm), "hi": np.concatenate([np.full(np_, THETA_MAX), np.full(nm, MIG_MAX)])}
    else:
        s |= {"terms": _terms(case), "theta": np.full(np_, THETA_MAX), "mig": np.full(nm, MIG_MAX)}
    return s


def _terms(case):
    pm = popmodel.build("((0,1):3,2):4", 3)
    return [(t, m) for t, m, _ in popmodel.popmig_terms(pm)][:case["terms"]]


def _run_saved(s):
    if s["kind"] == "curves":
        x, y = s["ctx"].fillvec(s["lo"], s["hi"], s["points"])
        return {"x": x, "y": y}
    x, y, mx = s["ctx"].popmig_curves(s["terms"], s["theta"], s["mig"], gridsize=s["points"])
    return {"x": x, "y": y, "maxx": mx}


def _exact_curves(case, seed):
    pops = case["pops"]
    np_, nm = _shape(pops)
    off = synth.gsamp_layout(np_, nm, pops - 1)
    r = _saved_rows(seed, case["G"], pops).double()
    xs, ys = [], []
    for p in range(np_ + nm):
        hi = THETA_MAX if p < np_ else MIG_MAX
        x = (torch.arange(case["points"], device="cuda", dtype=torch.float64) + 0.5) * hi / case["points"]
        if p < np_:
            c, f, k = (r[:, off[n] + p] for n in ("cc", "fc", "qi"))
        else:
            c, f, k = (r[:, off[n] + p - np_] for n in ("mc", "fm", "mi"))
        y = []
        for xc in x.split(max(1, (1 << 27) // case["G"])):
            t = torch.outer(math.log(2.0) - torch.log(xc), c) - torch.outer(2.0 / xc, f) if p < np_ else \
                torch.outer(torch.log(xc), c) - torch.outer(xc, f)
            y.append(t.sub_(k[None, :]).exp_().mean(1))
        xs.append(x)
        ys.append(torch.cat(y))
    return {"x": torch.stack(xs), "y": torch.stack(ys)}


def _density_2nm(r, off, th, mi, x):
    """Posterior density of 2NM = theta m / 2 at the points x."""
    cc, fc, q = (r[:, off[n] + th][None, :] for n in ("cc", "fc", "qi"))
    mc, fm, m = (r[:, off[n] + mi][None, :] for n in ("mc", "fm", "mi"))
    out = []
    for xc in x.split(max(1, (1 << 25) // r.shape[0])):
        xc = xc[:, None]
        a = cc + mc
        z = fc + fm * xc
        x1, x2 = 2 * z / THETA_MAX, MIG_MAX * z / xc
        # Gamma(a, x1) - Gamma(a, x2) = gamma(a, x2) - gamma(a, x1): the pair
        # that does not cancel
        up = torch.special.gammaincc(a, x1) - torch.special.gammaincc(a, x2)
        lo = torch.special.gammainc(a, x2) - torch.special.gammainc(a, x1)
        d = torch.where(x1 > a, up, lo)
        t = math.log(2.0) + mc * torch.log(xc) - a * torch.log(z) - q - m + torch.lgamma(a) + torch.log(d)
        e = torch.exp(t)
        out.append(torch.where((t < 700) & (t > -700), e, torch.zeros_like(e)).mean(1))
    return torch.cat(out)


def _exact_popmig(case, seed):
    np_, nm = _shape(3)
    off = synth.gsamp_layout(np_, nm, 2)
    r = _saved_rows(seed, case["G"], 3).double()
    n = case["points"]
    xs, ys, mx = [], [], []
    j = torch.arange(n, device="cuda", dtype=torch.float64) + 0.5
    top = THETA_MAX * MIG_MAX / 2.0
    for th, mi in _terms(case):
        # the curve's range: the largest grid point with a density above 1e-9
        hit = torch.nonzero(_density_2nm(r, off, th, mi, j * top / n) > 1e-9)
        hi = float(j[hit[-1, 0]]) * top / n if len(hit) else top
        xs.append(j * hi / n)
        ys.append(_density_2nm(r, off, th, mi, xs[-1]))
        mx.append(hi)
    return {"x": torch.stack(xs), "y": torch.stack(ys), "maxx": np.array(mx)}


def _work_saved(case):
    if case["kind"] == "curves":
        np_, nm = _shape(case["pops"])
        n = (np_ + nm) * case["points"]
        return {"bytes": case["G"] * (4 * np_ + 3 * nm) * 4 + n * 16, "flops": n * case["G"] * 25}
    n = case["terms"] * case["points"]
    return {"bytes": case["G"] * 37 * 4 + n * 16, "flops": n * case["G"] * 150}


# --------------------------------------------------------------- splittime
def _prepare_splittime(case, seed):
    rng = np.random.default_rng([seed, 41])
    nl, nch = case["loci"], case["chains"]
    pm = popmodel.build("((0,1):3,2):4", 3)
    base, samp, seqs = [], [], []
    for _ in range(min(nl, 25)):
        s = [int(v) for v in rng.integers(4, 61, 3)]
        base.append(synth.sim_im_labeled(rng, s, list(rng.uniform(2.0, 6.0, 5)), 0.3, [(0.6, 0, 1, 3), (1.4, 3, 2, 4)]))
        samp.append(s)
        seqs.append(synth.is_data(rng, base[-1].g, 1.0, min_sites=2))
    pick = [l % len(base) for l in range(nl)]
    ctx = _context([("is", seqs[b]) for b in pick], nch)
    nth, nmg = len(pm.th_cells), len(pm.mg_cells)
    ctx.set_popmodel(pm, [15.0] * nth, [0.0] * nth, [MIG_MAX] * nmg, [0.0] * nmg, [1.0] * nmg)
    cs = splittime.ResidentChainSet(ctx, [[base[b] for b in pick]] * nch, np.tile([0.6, 1.4], (nch, 1)),
                                    np.linspace(1.0, 0.5, nch), np.ones(nl), [samp[b] for b in pick], _rates(rng, nl))
    return {"kind": "splittime", "ctx": ctx, "chains": np.arange(nch, dtype=np.int32), "rng": api.MT19937(seed + 99),
            "period": np.random.default_rng([seed, 42]), "u": np.tile(cs.u, nch), "kappa": np.tile(cs.kappa, nch),
            "tprior": [(0.0, 3.0), (0.0, 6.0)]}


def _run_splittime(s):
    period = s["period"].integers(0, 2, len(s["chains"]))
    acc, pdgsum, probg, newt = s["ctx"].changet_ry1_sweep_mt(s["chains"], period, s["tprior"], s["rng"], s["u"],
                                                            s["kappa"])
    return {"accept": acc, "pdgsum": pdgsum, "probg": probg, "newt": newt, "pdg": s["ctx"].get_pdg()}


# --------------------------------------------------------------- genealogy
def _prepare_genealogy(case, seed):
    rng = np.random.default_rng([seed, 51])
    nl, nch, k = case["loci"], case["chains"], case["copies"]
    hky = case["model"] == "hky"
    if hky:
        tree, npops, tv, splits, theta = "(0,1):2", 2, [1.5], [(1.5, 0, 1, 2)], 10.0
    else:
        tree, npops, tv, splits, theta = "((0,1):3,2):4", 3, [0.8, 1.6], [(0.8, 0, 1, 3), (1.6, 2, 3, 4)], 4.0
    u = _rates(rng, nl)
    kap = rng.uniform(2.0, 8.0, nl)
    base, loci, al, ar = [], [], [], None
    for l in range(nl):
        lg = synth.sim_im_labeled(rng, [k] * npops, [theta] * (2 * npops - 1), 0.0, splits)
        base.append(lg)
        if hky:
            loci.append(("hky", synth.hky_data(rng, lg.g, 1000, float(u[l]), float(kap[l]), rng.dirichlet([5] * 4))))
        else:
            al.append(synth.sw_alleles(rng, lg.g, float(u[l])))
            loci.append(("sw", lg.g.n))
    if not hky:
        ar = np.array([[int(a.min()) - 5, int(a.max()) + 5] for a in al], np.int32)
    ctx = _context(loci, nch)
    pm = popmodel.build(tree, npops, nomig=True)
    th_max, th_min, _, _, _ = popmodel.priors(pm, 30.0, 0.0)
    ctx.set_popmodel(pm, th_max, th_min)
    ci = np.repeat(np.arange(nch, dtype=np.int32), nl)
    li = np.tile(np.arange(nl, dtype=np.int32), nch)
    flat = base * nch
    cat = lambda f: np.concatenate([getattr(g.g, f) for g in flat])  # noqa: E731
    ctx.set_genealogies(ci, li, cat("up0"), cat("up1"), cat("down"), cat("time"), length=np.full(len(flat), -1.0))
    ctx.set_labels(ci, li, flat)
    ctx.set_locus_pops(np.ones(nl), np.full((nl, npops), k, np.int32))
    for c in range(nch):
        for l in range(nl):
            if hky:
                ctx.set_pi(c, l, loci[l][1].pi)
            else:
                ctx.set_alleles(c, l, al[l])
    ctx.set_betas(1.0 / (1.0 + 0.05 * np.arange(nch)))
    return {"kind": "genealogy", "ctx": ctx, "chains": np.arange(nch, dtype=np.int32), "tv": np.tile(tv, (nch, 1)),
            "sweeps": case["sweeps"], "rngs": [api.UgRng(1000 + seed % 100000 * 128 + c) for c in range(nch)],
            "u": np.tile(u, nch), "kappa": np.tile(kap if hky else np.ones(nl), nch), "range": ar}


def _run_genealogy(s):
    acc, top, probg = s["ctx"].updategenealogy_sweep(s["chains"], s["tv"], s["sweeps"], s["rngs"], s["u"], s["kappa"],
                                                     precision=api.PREC_FAST, allele_range=s["range"])
    return {"accepted": acc, "topology": top, "probg": probg, "pdg": s["ctx"].get_pdg()}


def _work_chains(case):
    nl, nch = case["loci"], case["chains"]
    if case["kind"] == "splittime":
        # node times moved there (and back for the rejected half), the events
        # read once for the weights, the branches once for the likelihood
        n = 96
        return {"bytes": nl * nch * (2 * n - 1) * (8 * 3 + 8 + 4 + 8), "flops": nl * nch * (2 * n - 1) * 30}
    n = case["copies"] * (2 if case["model"] == "hky" else 3)
    per = (2 * n - 1) * 36 + (8 * 60 * 60 if case["model"] == "hky" else 400)
    return {"bytes": nl * nch * case["sweeps"] * per, "flops": nl * nch * case["sweeps"] * (n * 40 + 2000)}


# ------------------------------------------------------------------ the API
_LIK = ("mc3_is", "hky", "sw", "mixed")


def prepare(case, seed):
    kind = case["kind"]
    if kind in _LIK:
        return _prepare_likelihood(case, seed)
    return {"hky_edit": _prepare_edit, "surface": _prepare_surface, "curves": _prepare_saved,
            "popmig": _prepare_saved, "splittime": _prepare_splittime, "genealogy": _prepare_genealogy}[kind](case, seed)


def run(state):
    kind = state["kind"]
    if kind in _LIK:
        return _run_likelihood(state)
    return {"hky_edit": _run_edit, "surface": _run_surface, "curves": _run_saved, "popmig": _run_saved,
            "splittime": _run_splittime, "genealogy": _run_genealogy}[kind](state)


def work(case):
    kind = case["kind"]
    if kind in _LIK:
        return _work_likelihood(case)
    return {"hky_edit": _work_edit, "surface": _work_surface, "curves": _work_saved, "popmig": _work_saved,
            "splittime": _work_chains, "genealogy": _work_chains}[kind](case)


def exact(case, seed):
    """The outputs in plain FP64; None for the samplers, whose outputs follow
    from the framework's own draws and decisions."""
    kind = case["kind"]
    if kind in _LIK:
        return _exact_likelihood(case, seed)
    f = {"hky_edit": _exact_edit, "surface": _exact_surface, "curves": _exact_curves, "popmig": _exact_popmig}.get(kind)
    return None if f is None else f(case, seed)
