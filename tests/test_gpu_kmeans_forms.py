"""The k-means kernel's forms (fbc_kmeans): squared distances below and above 2^32, member counts above
the exact integer distances' range, more borders than a staged tile, points over several blocks of a
cluster, one point, k = 1 and k = every point, no borders; and what it refuses.  Centroids and weights
equal the oracle's restatement of the reference."""
import ctypes as C

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _set(rng, npv, nb, lmax, cmax, groups):
    """Points near a few prototypes, with repeated and equally distant ones among them."""
    proto = rng.integers(0, max(lmax, 1), (groups, nb))
    L = np.clip(proto[rng.integers(0, groups, npv)] + rng.integers(-2, 3, (npv, nb)), 0, lmax).astype(np.float64)
    return L, rng.integers(0, cmax + 1, (npv, nb)).astype(np.int32), rng.integers(1, 9, npv).astype(np.int32)


def _same(got, sets, kfrac):
    for (L, Cn, w), (idx, gw) in zip(sets, got):
        oi, ow = oracle.kmeans_pivots(L, Cn, w, kfrac)
        first = [i for i, x in enumerate(idx.tolist()) if x not in idx.tolist()[:i]]  # the oracle drops repeats
        assert idx[first].tolist() == oi.tolist() and gw[first].tolist() == ow.tolist()


@pytest.mark.parametrize("kfrac", [0.5, 0.05, 1.0])
@pytest.mark.parametrize("npv,nb,lmax,cmax,groups", [
    (1, 3, 100, 2, 1), (2, 0, 0, 0, 1), (33, 5, 50, 3, 4), (300, 40, 3000, 6, 7),
    (400, 20, 1_000_000, 3, 3),        # above 2^32
    (500, 8, 20_000_000, 3, 2),        # members above the exact integers' range
    (120, 700, 900, 4, 5),             # two staged tiles of borders
    (1500, 12, 40, 2, 30)])
def test_forms(fg, kfrac, npv, nb, lmax, cmax, groups):
    rng = np.random.default_rng([npv, nb])
    sets = [_set(rng, npv, nb, lmax, cmax, groups)]
    if kfrac == 0.5:  # with others of other sizes, in one call
        sets += [_set(rng, 7, 9, 30, 1, 2), _set(rng, 210, nb, lmax, cmax, groups)]
    _same(fg.kmeans(sets, kfrac), sets, kfrac)


def test_refusals(fg):
    rng = np.random.default_rng(1)
    good = _set(rng, 20, 4, 50, 2, 3)
    for bad, code in ((0.5, fg.FBC_ERR_INVALID_ARG), (-1.0, fg.FBC_ERR_INVALID_ARG), (2147483648.0, fg.FBC_ERR_INVALID_ARG),
                      (np.nan, fg.FBC_ERR_INVALID_ARG), (94906266.0, fg.FBC_ERR_RANGE)):
        L = good[0].copy()
        L[7, 2] = bad
        for sets in ([(L, *good[1:])], [good, (L, *good[1:]), good]):
            with pytest.raises(fg.FbcError) as e:
                fg.kmeans(sets)
            assert e.value.code == code
    _same(fg.kmeans([good]), [good], 0.5)


def test_vectors_apart(fg):
    """Sets whose vectors do not lie back to back in the caller's arrays (and one before the other)."""
    rng = np.random.default_rng(4)
    sets = [_set(rng, 40, 6, 60, 2, 3), _set(rng, 25, 3, 60, 2, 3)]
    L = np.zeros(1000)
    Cn = np.zeros(1000, np.int32)
    at = np.array([500, 17], np.int64)
    for o, (l, c, _) in zip(at, sets):
        L[o:o + l.size], Cn[o:o + c.size] = l.ravel(), c.ravel()
    off = np.array([0, 40, 65], np.int64)
    nb, k = np.array([6, 3], np.int32), np.array([20, 12], np.int32)
    w = np.concatenate([s[2] for s in sets])
    idx, ow = np.zeros(32, np.int32), np.zeros(32, np.int32)
    p = lambda a: a.ctypes.data_as(C.c_void_p)  # noqa: E731
    assert fg.lib.fbc_kmeans(2, p(off), p(nb), p(at), p(L), p(Cn), p(w), p(k), 0.0, 100, p(idx), p(ow), None) == 0
    _same([(idx[:20], ow[:20]), (idx[20:], ow[20:])], sets, 0.5)
