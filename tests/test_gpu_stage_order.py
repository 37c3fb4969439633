"""Sampling after lda_update_wt without lda_max_topic in between: the statistics stay the
earlier ones, the word columns take the current counts and topic totals.  The reference is the
allocation-free entry point, which is handed both."""
import numpy as np
import pytest

import lda_sc20_b200 as L
from test_zz_no_alloc import LL_RTOL, _call, _device_io

pytestmark = pytest.mark.gpu


# at 4096 topics the entry point's smoothing table follows the current totals, the trainer's the
# last lda_max_topic: draws from it may differ, and alpha leaves next to none of them
@pytest.mark.parametrize("K,alpha,dense", [(64, 0.5, 40.0), (300, 0.1, 40.0), (2048, 0.1, 40.0), (4096, 1e-7, 0.0)])
@pytest.mark.parametrize("before_any_stats", [False, True])
def test_columns_follow_the_last_update_wt(K, alpha, dense, before_any_stats):
    torch = pytest.importorskip("torch")
    corpus = L.Corpus.generate(L.corpus_config("c0", num_docs=300, vocab=700, K=K, num_chunks=1, dense_kind=2,
                                               dense_param=dense))
    tr = L.Trainer(corpus, K=K, alpha=alpha, seed=42)
    if not before_any_stats:
        tr.iterate(3)
        tr.update_wt()
        tr.max_topic()
    rng = np.random.default_rng(K)
    z = (K * rng.random(corpus.num_tokens) ** 3).astype(np.uint16)  # other totals, most of them in few topics
    tr.set_topics(z)
    tr.update_wt()
    tr.update_dt(0)
    tr.sync()
    st = {"corpus": corpus, "tr": tr, "z_before": tr.topics(), "iter": tr.iteration, "n_k": tr.topic_totals(),
          "dwt": tr.dense_wt(), "swt": tr.sparse_wt(), "stats": tr.word_stats(), "rows": tr.doc_rows(),
          "meta": tr.token_meta()}
    q = tr.counters().branch_q
    tr.sample_chunk(0, ll=True)
    ll_ref = tr.perplexity()
    from_table = tr.counters().branch_q - q if K > 2048 else 0
    assert from_table < 10
    bufs, sizes, ntiles = _device_io(torch, st, K)
    got, ll, status = _call(torch, st, K, bufs, sizes, ntiles)
    assert status == 0
    assert (got != tr.topics()).sum() <= from_table
    assert ll == ll_ref or abs(ll - ll_ref) <= LL_RTOL * abs(ll_ref)  # before any statistics both may be -inf
    # and with the statistics formed anew, as a sweep does
    tr.set_topics(z)
    tr.update_wt()
    tr.max_topic()
    tr.update_dt(0)
    tr.sample_chunk(0)
    ref = L.Trainer(corpus, K=K, alpha=alpha, seed=42)
    ref.set_topics(z)
    ref.iteration = tr.iteration
    ref.iterate(1)
    assert np.array_equal(ref.topics(), tr.topics())
