"""The split-time move's arithmetic, bit for bit: times moved by the reference's
expressions (update_t_RY.cpp's beforesplit and aftersplit) with one FP64
rounding a step -- the device divides by a reciprocal and exact remainders --
and a time's two floats, made from its bits."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

from ima2p_gb300 import api, build, popmodel, splittime, synth

pytestmark = pytest.mark.gpu


def moved(t, period, last, o, n, tu, td):
    with np.errstate(all="ignore"):
        below = t * n / o if period == 0 else tu + (t - tu) * (n - tu) / (o - tu)
        above = t + n - o if period == last - 1 else td - (td - n) * (td - t) / (td - o)
    return np.where((t <= o) & (t > tu), below, np.where((t > o) & (t < td), above, t))


@pytest.mark.parametrize("scale", [1.0, 1e-9, 3e5])
def test_band(scale):
    rng = np.random.default_rng(8)
    nch, nl = 40, 3
    pm = popmodel.build("(((0,1):4,2):5,3):6", 4)  # three splits: the first, one between, the last
    gens = [synth.sim_im_labeled(rng, [30] * 4, [4.0] * 7, 0.1, [(0.5, 0, 1, 4), (1.1, 2, 4, 5), (1.7, 3, 5, 6)]) for _ in range(nl)]
    ctx = api.Context(0)
    for g in gens:
        ctx.add_locus_is(synth.is_data(rng, g.g, 1.0, min_sites=1))
    ctx.set_chains(1, nch)
    nth, nmg = len(pm.th_cells), len(pm.mg_cells)
    ctx.set_popmodel(pm, [15.0] * nth, [0.0] * nth, [2.0] * nmg, [0.0] * nmg, [1.0] * nmg)
    splittime.ResidentChainSet(ctx, [gens] * nch, np.tile([0.5, 1.1, 1.7], (nch, 1)), np.ones(nch), np.ones(nl),
                               [[30] * 4] * nl, np.ones(nl))
    lines = [len(g.pop) for g in gens]
    ci, li = np.repeat(np.arange(nch), nl), np.tile(np.arange(nl), nch)
    tu, td = np.array([0.0, 0.5, 1.1]) * scale, np.array([1.1 * scale, 1.7 * scale, 1000000.0])
    split = np.array([0.5, 1.1, 1.7]) * scale
    for period in range(3):
        o = np.full(nch, split[period])
        hi = td[period] if period < 2 else 3.0 * scale
        n = tu[period] + (hi - tu[period]) * rng.uniform(0.001, 0.999, nch)
        t = [np.concatenate([rng.uniform(0.0, 3.0 * scale, lines[l] - 4), tu[period:period + 1], o[:1], [hi, 0.0]])
             for _ in range(nch) for l in range(nl)]
        ctx.set_times(ci, li, np.concatenate(t), length=np.ones(nch * nl))
        ctx.rubber_band(np.arange(nch), np.full(nch, period), o, n, np.full(nch, tu[period]), np.full(nch, td[period]))
        for k in range(nch * nl):
            got, _ = ctx.get_times(ci[k], li[k], lines[li[k]])
            c = ci[k]
            np.testing.assert_array_equal(got, moved(t[k], period, 3, o[c], n[c], tu[period], td[period]))


def test_two_floats(tmp_path):
    so = str(tmp_path / "probe.so")
    subprocess.run([build.nvcc(), *build.ARCH, *build.FLAGS, "-I" + build.CSRC, "-shared", "-o", so,
                    os.path.join(os.path.dirname(os.path.abspath(__file__)), "ff_probe.cu")], check=True)
    rng = np.random.default_rng(2)
    bits = (rng.integers(1023 - 160, 1023 + 140, 1 << 20).astype(np.uint64) << np.uint64(52)) | rng.integers(0, 1 << 52, 1 << 20, dtype=np.uint64)
    # ties, their neighbours and carries into the exponent
    top = rng.integers(0, 1 << 23, 1 << 16, dtype=np.uint64)
    top[:64] = (1 << 23) - 1
    low = np.array([0, 1, (1 << 28) - 1, 1 << 28, (1 << 28) + 1, (1 << 29) - 1], np.uint64)
    e = rng.integers(1023 - 130, 1023 + 129, 1 << 16).astype(np.uint64) << np.uint64(52)
    ties = (e[:, None] | (top[:, None] << np.uint64(29)) | low[None, :]).ravel()
    z = np.concatenate([bits, ties]).view(np.float64)
    z = np.concatenate([z, [0.0, 5e-324, 2.0 ** -126, 2.0 ** 127, 3.4028234663852886e38, 1.0, 1.0 + 2.0 ** -24]])
    z = z[z < 3.4e38]
    out = np.zeros((len(z), 2), np.float32)
    p = lambda v: v.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert C.CDLL(so).probe_round(len(z), p(z), p(out)) == 0
    hi = z.astype(np.float32)
    lo = (z - hi.astype(np.float64)).astype(np.float32)
    np.testing.assert_array_equal(out[:, 0].view(np.uint32), hi.view(np.uint32))
    # a zero remainder may carry either sign
    same = (out[:, 1].view(np.uint32) == lo.view(np.uint32)) | ((out[:, 1] == 0) & (lo == 0))
    assert np.all(same), z[~same][:5]
