"""The allocation-free entry point's tables are of each call's own topic totals, and its launch
shape of the call's own K: calls of different K and totals in turn, through the one scratch
array and the 16 launch shapes they share."""
import numpy as np
import pytest

import lda_sc20_b200 as L
from test_zz_no_alloc import LL_RTOL, _call, _device_io, _state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Ks", [(100, 2048, 100), (2049, 5001, 2049, 64), tuple(range(250, 268))])
def test_calls_of_different_topic_counts_in_turn(Ks):
    torch = pytest.importorskip("torch")
    states = []
    for K in Ks:
        n = 200 + len(states)  # another corpus, and other totals, at each place
        st = _state(K, L.corpus_config("c0", num_docs=n, vocab=900, K=K, num_chunks=1, dense_kind=2, dense_param=30.0))
        states.append((K, st) + _device_io(torch, st, K))
    for _ in range(2):
        for K, st, bufs, sizes, ntiles in states:
            got, ll, status = _call(torch, st, K, bufs, sizes, ntiles)
            assert status == 0
            assert np.array_equal(got, st["z_ref"])
            assert abs(ll - st["ll_ref"]) <= LL_RTOL * abs(st["ll_ref"])
