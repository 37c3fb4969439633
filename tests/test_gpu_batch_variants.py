"""The batched sweep's kernels by topic counts and work-list shapes, against plain trainers."""
import numpy as np
import pytest

import lda_sc20_b200 as L
from lda_sc20_b200.batch import Batch

pytestmark = pytest.mark.gpu


def _pairs(models, tuning=None, **kw):
    """Two trainers per (corpus, K): one swept by itself, one in the batch."""
    plain, batched = ([L.Trainer(c, K=K, seed=5 + i, **kw) for i, (c, K) in enumerate(models)] for _ in range(2))
    return plain, batched, Batch(batched, tuning=tuning)


# the sampler's variant and its row slots follow the largest K (256, 512, 1024), the order of a
# model's topics is found 32 topics at a time and kept for 64
@pytest.mark.parametrize("ll", [False, True])
@pytest.mark.parametrize("Ks", [(33, 257, 64), (512, 16), (513, 100), (300, 1024, 31), (1025, 65), (100, 1500, 2048, 2047)])
def test_variants_by_the_largest_topic_count(Ks, ll):
    models = [(L.Corpus.generate(L.corpus_config("c0", num_docs=120 + 40 * i, vocab=300 + 50 * i, K=K, dense_kind=2,
                                                 dense_param=25.0, num_chunks=1 + i % 2, corpus_seed=i)), K)
              for i, K in enumerate(Ks)]
    plain, batched, b = _pairs(models)
    for n in (1, 3):
        got = b.iterate(n, ll=ll)
        for i, t in enumerate(plain):
            ref = t.iterate(n, ll=ll)
            assert np.array_equal(t.topics(), batched[i].topics()), f"K={Ks[i]} with {Ks}"
            if ll:
                assert got[i] == ref
            cp, cb = t.counters(), batched[i].counters()
            assert (cp.tokens, cp.early_accept, cp.branch_max, cp.branch_s, cp.branch_q) == \
                   (cb.tokens, cb.early_accept, cb.branch_max, cb.branch_s, cb.branch_q)


# work items of several tiles: runs of up to 16 sparse words of a few tokens, and of a frequent
# word's neighbouring tiles (its column is kept between them); a batch forms them once it has
# several times the tiles that its warps take at once
@pytest.mark.parametrize("models,vocab,tokens,dense,Ks,items_per_word", [
    (30, 16000, 60000, 50.0, (16, 100, 256), 0.5), (20, 1000, 180000, 500.0, (64, 300), 4)])
def test_items_of_several_tiles(models, vocab, tokens, dense, Ks, items_per_word):
    rng = np.random.default_rng(models)
    off = np.arange(0, tokens + 1, 100, dtype=np.int64)
    pairs = []
    for i in range(models):
        K = Ks[i % len(Ks)]
        words = rng.integers(0, vocab, tokens).astype(np.int32)
        pairs.append((L.Corpus.from_docs(off, words, vocab=vocab, K=K, dense_kind=2, dense_param=dense, topic_seed=i), K))
    plain, batched, b = _pairs(pairs)
    stats_and_docs = models * (-(-vocab // 32) + -(-(len(off) - 1) // 16))
    # one item per tile would be one of the rebuild for each word, and one of the sampler for each
    # 32 tokens of it (2 items a word of the first batch, 7 of the second)
    used = sum(int((c.word_count() > 0).sum()) for c, _ in pairs)
    assert b.stats()[1] - stats_and_docs < items_per_word * used
    got = b.iterate(3, ll=True)
    for i, t in enumerate(plain):
        ref = t.iterate(3, ll=True)
        assert np.array_equal(t.topics(), batched[i].topics()), f"model {i} (K={pairs[i][1]})"
        assert got[i] == ref
