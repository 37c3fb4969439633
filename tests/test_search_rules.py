"""The sampler's searches by a single thread, restated in binary32: where they call themselves
sure, they must find the place that a scan of every prefix finds."""
import numpy as np
import pytest

F = np.float32


def ks_scan(x):
    """Kogge-Stone inclusive scan along axis 1 (32 places), one rounding per addition."""
    v = x.astype(F).copy()
    off = 1
    while off < v.shape[1]:
        v[:, off:] = (v[:, off:] + v[:, :-off].copy()).astype(F)
        off <<= 1
    return v


def crossing(v, t):
    """The binary search over 32 prefixes: (place, its predecessor's prefix, sure)."""
    n = len(t)
    idx = np.zeros(n, np.int64)
    prev = np.zeros(n, F)
    rows = np.arange(n)
    for h in (16, 8, 4, 2, 1):
        probe = v[rows, idx + h - 1]
        up = ~(t < probe)
        prev = np.where(up, probe, prev)
        idx = idx + np.where(up, h, 0)
    sure = (t < v[rows, idx]) & ~(t < (prev * F(1 + 2.0**-19)).astype(F))
    return idx, prev, sure


def _terms(kind, rng, n):
    if kind == "plain":
        x = rng.random((n, 32))
    elif kind == "skewed":
        x = np.exp(rng.normal(0, 8, (n, 32)))
    elif kind == "sparse":
        x = rng.random((n, 32)) * (rng.random((n, 32)) < 0.2)
    elif kind == "tiny":
        x = np.where(rng.random((n, 32)) < 0.5, 1.0, 1e-9) * rng.random((n, 32))
    else:  # equal terms whose prefixes round
        x = np.repeat(rng.random((n, 1)).astype(F), 32, 1)
    return x.astype(F)


@pytest.mark.parametrize("target", ["uniform", "at a prefix", "near a prefix"])
@pytest.mark.parametrize("kind", ["plain", "skewed", "sparse", "tiny", "equal"])
def test_crossing_is_the_first_prefix_above(kind, target):
    rng = np.random.default_rng(7)
    n = 20000
    v = ks_scan(_terms(kind, rng, n))
    total = v.max(1)
    if target == "uniform":
        t = (rng.random(n).astype(F) * total).astype(F)
    else:
        t = v[np.arange(n), rng.integers(0, 32, n)]
        if target == "near a prefix":
            t = (t * (F(1) + F(2.0**-23) * rng.integers(-40, 41, n).astype(F))).astype(F)
    idx, prev, sure = crossing(v, t)
    above = t[:, None] < v
    first = np.where(above.any(1), above.argmax(1), 32)
    assert (idx[sure] == first[sure]).all()
    has_prev = sure & (idx > 0)
    assert (prev[has_prev] == v[np.arange(n), np.maximum(idx - 1, 0)][has_prev]).all()
    if target == "uniform" and kind in ("plain", "sparse"):
        assert sure[total > 0].mean() > 0.99  # the slow path stays rare


@pytest.mark.parametrize("K", [2049, 4096, 10001])
def test_smoothing_table_search(K):
    """The table of carried round prefixes: a sure target has every entry before the answer at
    or below it and every later one above it, whatever places a search probes."""
    rng = np.random.default_rng(K)
    n_k = rng.integers(0, 200000, K) * (rng.random(K) < 0.7)
    r = (F(1) / (n_k.astype(F) + F(1000.0))).astype(F)
    term = (F(0.1) * (F(0.01) * r).astype(F)).astype(F)
    rounds = -(-K // 32)
    pad = np.zeros(rounds * 32, F)
    pad[:K] = term
    ks = ks_scan(pad.reshape(rounds, 32))
    T = np.empty_like(ks)
    carry = F(0)
    for i in range(rounds):
        T[i] = (carry + ks[i]).astype(F)
        carry = F(carry + ks[i, 31])
    T = T.reshape(-1)[:K]
    x = np.concatenate([(rng.random(20000).astype(F) * T[-1]).astype(F), T[rng.integers(0, K, 5000)]])
    k = np.searchsorted(np.maximum.accumulate(T), x, side="right")
    ok = k < K
    x, k = x[ok], k[ok]
    up = F(1 + 2.0**-20)
    sure = ((x * up).astype(F) < T[k]) & ~((k > 0) & (x < (T[np.maximum(k - 1, 0)] * up).astype(F)))
    lo = np.maximum.accumulate(T)  # largest entry up to a place
    hi = np.minimum.accumulate(T[::-1])[::-1]  # smallest entry from a place on
    assert (hi[k[sure]] > x[sure]).all()
    assert (lo[np.maximum(k[sure] - 1, 0)][k[sure] > 0] <= x[sure][k[sure] > 0]).all()
    assert sure.mean() > 0.5
