"""Trees over prims with values that are not finite (raw build calls accept
them), against a plain restatement of the builder's rule for them: bounds are
minima and maxima that ignore NaN; a bin's bounds are minima and maxima of the
values in the order of their bits (a positive NaN above infinity, a negative
one below -infinity), and a bin whose bound comes out NaN has none; NaN bins as
0 and is never below a plane.  Orders, links and inner bounds match exactly.
Nodes of 3 to 10 prims, 11 and more, and the whole CTA's (over 256)."""
import numpy as np
import pytest

import py_build_ref as ref
from helpers import gpu_build_bl, gpu_build_tl

pytestmark = pytest.mark.gpu

f32, INF, FMAX = np.float32, np.float32(np.inf), ref.F32_MAX
SPECIAL = np.array([np.nan, -np.nan, np.inf, -np.inf, 3e38, -3e38], np.float32)


def _key(v):  # the bits' order, as a signed integer
    i = np.asarray(v, np.float32).view(np.int32).astype(np.int64)
    return np.where(i >= 0, i, i ^ 0x7FFFFFFF)


def _unkey(k):
    return np.where(k >= 0, k, k ^ 0x7FFFFFFF).astype(np.int32).view(np.float32)


def _area(lo, hi):
    d = hi - lo
    return f32(2) * ((d[0] * d[1] + d[0] * d[2]) + d[1] * d[2])


def _split(lo, hi, cen):
    """(axis, position) of the best plane"""
    best, at = FMAX, (0, f32(0))
    cl, ch = np.fmin(FMAX, np.fmin.reduce(cen)), np.fmax(-FMAX, np.fmax.reduce(cen))
    for d in range(3):
        b = np.array([ref.bin_index(v) for v in (cen[:, d] - cl[d]) * (f32(32) / (ch[d] - cl[d]))])
        n = np.bincount(b, minlength=32)
        blo, bhi = np.full((32, 3), INF), np.full((32, 3), -INF)
        for k in np.flatnonzero(n):
            blo[k] = np.fmin(INF, _unkey(np.minimum(_key(INF), _key(lo[b == k]).min(0))))
            bhi[k] = np.fmax(-INF, _unkey(np.maximum(_key(-INF), _key(hi[b == k]).max(0))))
        for p in range(31):
            nl, nr = n[:p + 1].sum(), n[p + 1:].sum()
            al = _area(blo[:p + 1].min(0), bhi[:p + 1].max(0)) if nl else f32(0)
            ar = _area(blo[p + 1:].min(0), bhi[p + 1:].max(0)) if nr else f32(0)
            cost = al * f32(nl) + ar * f32(nr)
            if cost < best:
                best, at = cost, (d, cl[d] + (f32(p) + f32(1)) * ((ch[d] - cl[d]) / f32(32)))
    return at


def _tree(lo, hi, cen):
    """node -> (left, right or prim, parent, bounds of an inner node), and the prim order"""
    n = len(lo)
    order, nodes = list(range(n)), {}

    def node(at, base, first, c, parent):
        if c == 1:
            nodes[at] = (ref.INVALID, order[first], parent, None)
            return
        s = order[first:first + c]
        b = (np.fmin.reduce(lo[s]), np.fmax.reduce(hi[s]))
        if c > 2:  # (two prims without a bound leave their node without one)
            b = (np.fmin(INF, b[0]), np.fmax(-INF, b[1]))
        b = (b[0] - f32(0.0001), b[1] + f32(0.0001))
        nl = 1
        if c > 2:
            d, x = _split(lo[s], hi[s], cen[s])
            nl = ref.partition(order, first, c, lambda p: cen[p, d] < x)
            nl = nl if 0 < nl < c else c // 2
        nodes[at] = (base, base + 1, parent, b)
        node(base, base + 2, first, nl, at)
        node(base + 1, base + 2 * nl, first + nl, c - nl, at)

    node(0, 1, 0, n, ref.INVALID)
    return nodes, order


def _check(got, lo, hi, cen, what):
    nodes, order = got
    for a in (lo, hi):  # (the device's arithmetic gives the positive NaN)
        a[np.isnan(a)] = np.nan
    with np.errstate(all="ignore"):
        want, worder = _tree(lo, hi, cen)
    assert list(order) == worder, what
    for i, (l, r, parent, b) in want.items():
        g = nodes[i]
        assert (g["left"], g["right"], g["parent"]) == (l, r, parent), (what, i)
        if b is not None:
            assert np.array_equal(g["min"], b[0], equal_nan=True), (what, i)
            assert np.array_equal(g["max"], b[1], equal_nan=True), (what, i)


def _spoil(rng, a, rate):
    m = rng.random(a.shape) < rate
    a[m] = rng.choice(SPECIAL, m.sum())
    return a


@pytest.mark.parametrize("rate", [0.01, 0.1, 0.4])
def test_trees_of_values_not_finite(gpu_ctx, rate):
    rng = np.random.default_rng(int(1000 * rate))
    sizes = [3, 4, 5, 7, 10, 11, 12, 33] * 6 + [300]
    ids = [np.arange(n, dtype=np.uint32) for n in sizes]
    tl, bl = [], []
    for n in sizes:
        lo = (rng.random((n, 3)) * 32).astype(np.float32)
        box = _spoil(rng, np.concatenate([lo, lo + (rng.random((n, 3)) * 4).astype(np.float32)], 1), rate)
        both = rng.random((n, 3)) < rate / 2  # no bound at all on an axis
        box[:, :3][both] = box[:, 3:][both] = np.nan
        tl.append(box)
        bl.append(_spoil(rng, (rng.random((n, 9)) * 20).astype(np.float32), rate / 3))
    with np.errstate(all="ignore"):
        got = gpu_build_tl(gpu_ctx, [(a, np.ones(n, np.float32), i, None) for a, n, i in zip(tl, sizes, ids)])
        for a, g in zip(tl, got):
            lo, hi = np.fmin(a[:, :3], a[:, 3:]), np.fmax(a[:, :3], a[:, 3:])
            _check(g, lo, hi, (lo + hi) / f32(2), ("boxes", len(a)))
        got = gpu_build_bl(gpu_ctx, [(a, np.ones(n, np.float32), i) for a, n, i in zip(bl, sizes, ids)])
        for a, g in zip(bl, got):
            v = a.reshape(-1, 3, 3)
            lo, hi = np.fmin.reduce(v, 1), np.fmax.reduce(v, 1)
            _check(g, lo, hi, ((v[:, 0] + v[:, 1]) + v[:, 2]) / f32(3), ("triangles", len(a)))
