"""The device's incomplete gamma functions (igamma.cuh: a series of four terms
a division, a fraction without divisions, a test for the function that leaves
the other at log Gamma(a)) against the reference's loops (utilities.cpp:
808-1130) run term for term, the number of terms by its FP64 rule and the sums
in extended precision: at the change from series to fraction (x = a + 1), far
from it on both sides, about the two bounds of the short cut, at the smallest
and largest counts, and where 1,000 terms do not do.

Tolerance: log of the sum + (-x + a log x - gln) + gln is rounded at each step,
the logarithm and the sum of up to 1,000 positive terms to a few 2^-53 of
themselves: 8 2^-53 (a |log x| + x + 2 |gln| + 8).  The functions are shared by
the files compiled without FMA contraction, and so is this."""
import ctypes as C
import math
import os
import subprocess

import numpy as np
import pytest

from ima2p_gb300 import build

pytestmark = pytest.mark.gpu

EPS, FPMIN, ITMAX = 3.0e-7, 1.0e-30, 1000
L = np.longdouble


def series_terms(a, x):
    ap, d = float(a), 1.0 / a
    s = d
    for n in range(1, ITMAX + 1):
        ap += 1.0
        d *= x / ap
        s += d
        if abs(d) < abs(s) * EPS:
            return n
    return 0


def fraction_terms(a, x):
    b = x + 1.0 - a
    c, d = 1.0 / FPMIN, 1.0 / b
    for i in range(1, ITMAX + 1):
        an = -i * (i - a)
        b += 2.0
        d = an * d + b
        d = FPMIN if abs(d) < FPMIN else d
        c = b + an / c
        c = FPMIN if abs(c) < FPMIN else c
        d = 1.0 / d
        if abs(d * c - 1.0) < EPS:
            return i
    return 0


def log_part(a, x, gln):
    """log of gser / gcf's value, or None where 1,000 terms do not do."""
    xl = L(x)
    lead = -xl + L(a) * np.log(xl) - L(gln)
    if x < a + 1.0:
        n = series_terms(a, x)
        ap, d = L(a), L(1) / L(a)
        s = d
        for _ in range(n):
            ap = ap + 1
            d = d * xl / ap
            s = s + d
        return np.log(s) + lead if n else None
    n = fraction_terms(a, x)
    b = xl + 1 - L(a)
    A, Am, B, Bm = L(1), L(0), b, L(1)
    for i in range(1, n + 1):
        an = -L(i) * (L(i) - L(a))
        b = b + 2
        A, Am, B, Bm = b * A + an * Am, A, b * B + an * Bm, B
        A, Am, B, Bm = A / B, Am / B, L(1), Bm / B
    return np.log(A / B) + lead if n else None


def expected(a, x, gln):
    v = log_part(a, x, gln)
    if v is None:
        return None, None
    low = x < a + 1.0  # v is the lower function's share
    with np.errstate(all="ignore"):
        rest = np.log1p(-np.exp(v))
    up, lo = (rest, v) if low else (v, rest)
    return L(gln) + up, L(gln) + lo


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    here = os.path.dirname(os.path.abspath(__file__))
    so = str(tmp_path_factory.mktemp("igamma") / "probe.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, *build.NOFMAD, "-I" + build.CSRC, "-shared", "-o", so,
                    os.path.join(here, "igamma_probe.cu")], check=True)
    lib = C.CDLL(so)
    lf = np.concatenate([[0.0], np.cumsum(np.log(np.arange(1, lib.probe_table(), dtype=np.float64)))])

    def run(a, x):
        a, x = np.ascontiguousarray(a, np.int32), np.ascontiguousarray(x, np.float64)
        up, lo, st = np.zeros(len(a)), np.zeros(len(a)), np.zeros((len(a), 2), np.int32)
        p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
        assert lib.probe(p(lf), len(a), p(a), p(x), p(up), p(lo), p(st)) == 0
        return up, lo, st

    return run, lf


def close(got, want, a, x, gln):
    tol = 8 * 2.0 ** -53 * (a * abs(math.log(x)) + x + 2 * abs(gln) + 8)
    assert abs(L(got) - want) <= tol, (a, x, got, want, tol)


@pytest.mark.parametrize("a", [1, 2, 3, 7, 31, 32, 33, 64, 191, 500, 3000, 20000])
def test_against_the_loops(probe, a):
    run, lf = probe
    edge = a + 1.0
    near = [edge * (1 + s * 2.0 ** -k) for k in (52, 40, 20, 10, 6, 4, 3, 2, 1) for s in (-1, 1)] + [edge]
    far = [edge * f for f in (1e-6, 1e-3, 0.02, 0.1, 0.3, 1.7, 2.5, 4.0, 9.0, 30.0)]
    # the short cut's bounds: a log x - x - gln = -38 and -54
    gln = lf[a - 1]
    cut = []
    for bound in (-38.0, -54.0):
        for lo, hi in ((1e-9, float(a)), (float(a), 50.0 * a + 500.0)):
            f = lambda v: a * math.log(v) - v - gln - bound  # noqa: E731
            if f(lo) * f(hi) < 0:
                for _ in range(80):
                    m = 0.5 * (lo + hi)
                    lo, hi = (m, hi) if f(lo) * f(m) > 0 else (lo, m)
                cut += [lo * (1 - 1e-4), lo * (1 - 1e-9), lo * (1 + 1e-9), lo * (1 + 1e-4)]
    xs = [v for v in near + far + cut if v > 0]
    up, lo, st = run([a] * len(xs), xs)
    for k, x in enumerate(xs):
        wu, wl = expected(a, x, gln)
        if wu is None:  # the sum's own function is refused; the other may have taken the short cut
            assert st[k].any()
            continue
        # where one function is what is left of 1 beside the other, it is
        # compared while it keeps digits
        if wu - L(gln) > -30 or x >= a + 1.0:
            assert st[k, 0] == 0
            if not (x < a + 1.0 and wu - L(gln) < -1):
                close(up[k], wu, a, x, gln)
        if wl - L(gln) > -30 or x < a + 1.0:
            assert st[k, 1] == 0
            if not (x >= a + 1.0 and wl - L(gln) < -1):
                close(lo[k], wl, a, x, gln)


def test_short_cut_is_exact(probe):
    """Where the other function is left at log Gamma(a), the reference's own
    FP64 expression gives log Gamma(a) too."""
    run, lf = probe
    rng = np.random.default_rng(1)
    a = rng.integers(1, 400, 4000)
    x = (a + 1.0) * np.exp(rng.uniform(-9.0, 3.5, 4000))
    up, lo, _ = run(a, x)
    for k in range(len(a)):
        gln = float(lf[a[k] - 1])
        low = x[k] < a[k] + 1.0
        got = up[k] if low else lo[k]
        if got != gln:
            continue
        v = log_part(int(a[k]), float(x[k]), gln)
        if v is not None:
            assert gln + math.log(1.0 - float(np.exp(v))) == pytest.approx(gln, rel=2 ** -52, abs=2 ** -53)


def test_refused(probe):
    run, _ = probe
    up, lo, st = run([0, 5, -1, 5, 200000], [1.0, -1.0, 1.0, 0.0, 200001.0])
    assert st[0, 1] and st[1].all() and st[2].all()   # a = 0 has no lower function; x < 0, a < 0 have none
    assert st[0, 0] == 0 and st[3, 0] == 0
    assert st[4].any()                                # past 1,000 terms, or past the table
