"""The sampler's searches by a single thread, compiled for the host from the kernels' own header:
a draw that calls itself sure is the one that the whole warp's scan of every prefix makes, for
targets anywhere, at a prefix and a few units in the last place beside one."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

F = np.float32
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("search") / "search.so")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-fno-fast-math", "-fPIC", "-shared", "-w",
                    "-I" + os.path.join(HERE, "..", "lda_sc20_b200", "csrc"), "-o", so,
                    os.path.join(HERE, "thread_search_host.cpp")], check=True)
    return C.CDLL(so)


def _p(a):
    return C.c_void_p(a.ctypes.data)


def _ks(x):
    """Kogge-Stone inclusive scan along the last axis, one rounding per addition."""
    v = np.array(x, dtype=F)
    off = 1
    while off < v.shape[-1]:
        v[..., off:] = v[..., off:] + v[..., :-off].copy()
        off <<= 1
    return v


def _first(mask):
    return int(np.argmax(mask)) if mask.any() else -1


def _targets(rng, prefixes, n):
    """n targets each: below the total, at a prefix, and up to 40 units beside one."""
    p = np.unique(prefixes[prefixes > 0])
    top = p.max() if len(p) else F(1)
    at = p[rng.integers(0, len(p), n)] if len(p) else np.zeros(n, F)
    near = (at * (F(1) + F(2.0**-23) * rng.integers(-40, 41, n).astype(F))).astype(F)
    return np.concatenate([(rng.random(n).astype(F) * top).astype(F), at, near, [F(0), top, F(2) * top]]).astype(F)


def _call(f, t, *args):
    z, flag = np.zeros(len(t), np.int32), np.zeros(len(t), np.uint8)
    f(C.c_int(len(t)), *args, _p(t), _p(z), _p(flag))
    return z, flag.astype(bool)


def _word(rng, K, kind):
    """A word's column with its max topic zeroed (alpha * column are the draw's terms)."""
    col = rng.random(K) * (1e-4 if kind == "plain" else np.exp(rng.normal(0, 4, K)))
    if kind == "sparse":
        col *= rng.random(K) < 0.05
    if kind == "equal":
        col[:] = 1e-3
    if kind == "lanes":
        col[np.arange(K) % 32 % 3 == 1] = 0.0  # whole lanes of Q without mass
    maxK = int(rng.integers(K))
    col[maxK] = 0.0
    return col.astype(F), maxK


def _lane_partials(col, alpha, K):
    ql = np.zeros(32, F)
    for k in range(K):
        ql[k % 32] = F(float(alpha) * float(col[k]) + float(ql[k % 32]))
    return ql


def _warp_q_draw(col, alpha, K, maxK, ql, qp, tt):
    """The lane by the Q partials' prefixes, then its topics in rounds of 32 with a carry."""
    ls = _first((tt < qp) & (ql > 0))
    if ls < 0:
        pos = np.nonzero(ql > 0)[0]
        ls = int(pos[-1]) if len(pos) else 0
    t2 = F(tt - qp[ls - 1]) if ls > 0 else tt
    n, carry, last = (K - ls + 31) // 32, F(0), -1
    for base in range(0, n, 32):
        key = ls + 32 * np.arange(base, min(base + 32, n))
        ks = _ks(np.pad(alpha * col[key], (0, 32 - len(key))))
        ok = col[key] > 0
        f = _first(ok & (t2 < (carry + ks[:len(key)]).astype(F)))
        if f >= 0:
            return int(key[f])
        if ok.any():
            last = int(key[np.nonzero(ok)[0][-1]])
        carry = F(carry + ks[31])
    return last if last >= 0 else maxK


@pytest.mark.parametrize("kind", ["plain", "skewed", "sparse", "equal"])
def test_crossing(lib, kind):
    rng = np.random.default_rng(3)
    n = 4000
    x = rng.random((n, 32)) if kind != "skewed" else np.exp(rng.normal(0, 8, (n, 32)))
    if kind == "sparse":
        x = x * (rng.random((n, 32)) < 0.2)
    if kind == "equal":
        x[:] = x[:, :1]
    x = x.astype(F)
    v = _ks(x)
    at = v[np.arange(n), rng.integers(0, 32, n)]
    near = (at * (F(1) + F(2.0**-23) * rng.integers(-40, 41, n).astype(F))).astype(F)
    for t in ((rng.random(n).astype(F) * v[:, 31]).astype(F), at, near):
        idx, prev, sure = np.zeros(n, np.int32), np.zeros(n, F), np.zeros(n, np.uint8)
        lib.crossing(n, _p(x), _p(t), _p(idx), _p(prev), _p(sure))
        sure = sure.astype(bool)
        above = t[:, None] < v
        assert (idx == above.argmax(1))[sure].all() and above.any(1)[sure].all()
        assert (prev == np.where(idx > 0, v[np.arange(n), np.maximum(idx - 1, 0)], F(0)))[sure].all()
    assert not sure.all()  # targets beside a prefix are left to the warp


@pytest.mark.parametrize("kind", ["plain", "skewed", "sparse", "equal", "lanes"])
@pytest.mark.parametrize("K", [4, 31, 32, 33, 100, 255, 256])
def test_q_draw(lib, K, kind):
    rng = np.random.default_rng(K)
    alpha = F(50.0 / K)
    for _ in range(3):
        col, maxK = _word(rng, K, kind)
        ql = _lane_partials(col, alpha, K)
        qp = _ks(ql)
        t = _targets(rng, qp, 60)
        qpos = int(sum(1 << i for i in range(32) if ql[i] > 0))
        z, unsure = _call(lib.q_draw, t, C.c_int(K), _p(col), C.c_float(alpha), C.c_int(maxK), _p(qp), C.c_uint(qpos))
        ref = np.array([_warp_q_draw(col, alpha, K, maxK, ql, qp, x) for x in t])
        assert (z == ref)[~unsure].all()
        assert unsure[-2:].all()  # at or above every prefix


@pytest.mark.parametrize("kind", ["plain", "skewed", "sparse", "lanes"])
@pytest.mark.parametrize("K", [2049, 4100])
def test_q_draw_with_the_round_table(lib, K, kind):
    rng = np.random.default_rng(K)
    alpha = F(0.1)
    rounds = ((K + 31) // 32 + 31) // 32
    col, maxK = _word(rng, K, kind)
    ql = _lane_partials(col, alpha, K)
    qp = _ks(ql)
    tab, inner = np.zeros((32, rounds, 2), F), []
    for ls in range(32):
        carry = F(0)
        for r in range(rounds):
            key = np.arange(ls + 1024 * r, min(K, ls + 1024 * (r + 1)), 32)
            ks = _ks(np.pad(alpha * col[key], (0, 32 - len(key))))
            tab[ls, r] = carry, carry + ks.max()
            inner.append((qp[ls - 1] if ls else F(0)) + (carry + ks))  # targets that end beside an inner prefix
            carry = F(carry + ks[31])
    t = np.concatenate([_targets(rng, qp, 100), _targets(rng, np.concatenate(inner).astype(F), 150)])
    qpos = int(sum(1 << i for i in range(32) if ql[i] > 0))
    z, unsure = _call(lib.q_draw_table, t, C.c_int(K), _p(col), C.c_float(alpha), _p(qp), C.c_uint(qpos), _p(tab), C.c_int(rounds))
    ref = np.array([_warp_q_draw(col, alpha, K, maxK, ql, qp, x) for x in t])
    assert (z == ref)[~unsure].all()
    assert unsure.any() and not unsure[:100].all()


def _first_above(T, lo, hi, x):
    """The warp's 32-way search of the smoothing table."""
    if lo >= hi or not x < T[hi - 1]:
        return -1
    while hi - lo > 32:
        step = (hi - lo + 31) >> 5
        ends = np.minimum(lo + (np.arange(32) + 1) * step - 1, hi - 1)
        f = _first(x < T[ends])
        nlo = lo if f == 0 else min(lo + f * step - 1, hi - 1) + 1
        hi, lo = min(lo + (f + 1) * step - 1, hi - 1) + 1, nlo
    return lo + _first(x < T[lo:hi])


@pytest.mark.parametrize("where", ["first", "middle", "own", "last", "before the last"])
@pytest.mark.parametrize("K,nnz", [(2049, 1), (2049, 32), (4097, 20), (4097, 33)])
def test_split_draw(lib, K, nnz, where):
    rng = np.random.default_rng(K + nnz)
    alpha, beta = F(0.1), F(0.01)
    n_k = rng.integers(0, 200000, K) * (rng.random(K) < 0.7)
    r = (F(1) / (n_k.astype(F) + F(1000.0))).astype(F)
    rounds = -(-K // 32)
    ks = _ks(np.pad((alpha * (beta * r)).astype(F), (0, rounds * 32 - K)).reshape(rounds, 32))
    T, carry = np.empty_like(ks), F(0)
    for i in range(rounds):
        T[i] = carry + ks[i]
        carry = F(carry + ks[i, 31])
    T = T.reshape(-1)[:K].copy()
    tend = T[np.minimum(K, 32 * np.arange(rounds) + 32) - 1].copy()
    topics = np.sort(rng.choice(K, nnz, replace=False))
    counts = rng.integers(1, 50, nnz)
    ent = ((topics << 16) | counts).astype(np.uint32)
    maxK = {"first": 0, "middle": K // 2, "own": int(topics[0]), "last": K - 1, "before the last": K - 2}[where]
    term = np.where(topics == maxK, F(0), alpha * (counts.astype(F) * r[topics]).astype(F)).astype(F)
    prefixes, carry = [], F(0)
    for i in range(0, nnz, 32):
        part = _ks(np.pad(term[i:i + 32], (0, 32 - len(term[i:i + 32]))))
        prefixes.append((carry + part).astype(F))
        carry = F(carry + part[31])
    Qw, own = carry, np.concatenate(prefixes)[:nnz]
    wp = prefixes[0].copy()
    one = nnz <= 32
    wok = int(sum(1 << i for i in range(min(nnz, 32)) if term[i] > 0))
    sm = F(alpha * F(beta * r[maxK]))

    def warp(t):
        if t < Qw:
            ok = term > 0
            f = _first(ok & (t < own))
            if f >= 0:
                return int(topics[f])
            if ok.any():
                return int(topics[np.nonzero(ok)[0][-1]])
        t1 = F(t - Qw)
        if maxK > 0 and t1 < T[maxK - 1]:
            return _first_above(T, 0, maxK, t1)
        z = _first_above(T, maxK + 1, K, F(t1 + sm))
        return z if z >= 0 else (K - 2 if maxK == K - 1 else K - 1)

    smooth = np.concatenate([[Qw], Qw + T, Qw + T - sm]).astype(F)
    t = np.concatenate([_targets(rng, own, 60), _targets(rng, smooth, 200)])
    t = t[t < F(Qw + F(T[-1] - sm))]
    z, unsure = _call(lib.split_draw, t, C.c_int(K), C.c_float(alpha), C.c_float(beta), C.c_int(maxK), _p(ent), C.c_uint(nnz),
                      C.c_float(Qw), _p(T), _p(r), _p(wp) if one else C.c_void_p(None), C.c_uint(wok), _p(tend))
    ref = np.array([warp(x) for x in t])
    assert (z == ref)[~unsure].all()
    if not one:
        assert unsure[t < Qw].all()
    assert unsure.any() and not unsure.all()
