"""Word columns that a warp keeps from one sparse word to the next: words whose topic counts lie
around the put-back limit (an eighth of the topics), followed on the same warps by thousands of
words of a few topics, against the CPU oracle."""
import numpy as np
import pytest

import lda_sc20_b200 as L
from oracle import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dense", [0.0, 20.0])
@pytest.mark.parametrize("K", [64, 250, 1024, 2048])
def test_columns_after_topic_rich_words(K, dense):
    rng = np.random.default_rng(K)
    vocab, rich = 9000, 200
    counts = np.full(vocab, 3)
    counts[:rich] = K // 8 + rng.integers(-1, 2, rich)
    words = np.repeat(np.arange(vocab, dtype=np.int32), counts)
    # a word's topics are distinct, so that it has as many as tokens
    topics = np.concatenate([rng.choice(K, n, replace=False) for n in counts]).astype(np.uint16)
    at = rng.permutation(len(words))
    off = np.unique(np.append(np.arange(0, len(words), 120), len(words))).astype(np.int64)
    c = L.Corpus.from_docs(off, words[at], vocab=vocab, K=K, topics=topics[at], dense_kind=2, dense_param=dense)
    tr = L.Trainer(c, K=K, seed=8)
    o = Oracle(c.tok_word(), c.tok_doc(), c.info.vocab, c.info.num_docs, K, tr.alpha, tr.beta, num_dense=tr.Vd)
    z = c.topics()
    o.rebuild(z)
    tr.update_wt()
    tr.max_topic()
    tr.sync()
    for a, b, name in zip(tr.word_stats(), o.word_stats(), ("top2", "k3", "phi4", "ql")):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), name
    for it in range(2):
        o.iterate(z, 8, it)
        tr.iterate(1)
        assert np.array_equal(tr.topics(), z), f"sweep {it}"
    cnt = tr.counters()
    assert (cnt.word_tiles_dense + cnt.word_tiles_sparse) // 2 > 8 * 5 * 148  # more tiles than resident warps
