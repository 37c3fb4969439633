"""Kernels and dispatch rules at the sizes where they change or can go wrong, against the CPU
oracle: topics and integer state identical, word statistics bit for bit, the FP64
log-likelihood within 1e-9 relative (its summation order differs)."""
import numpy as np
import pytest

import lda_sc20_b200 as L
from lda_sc20_b200.serving import Model, Server
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _oracle(c, tr, K):
    i = c.info
    return Oracle(c.tok_word(), c.tok_doc(), i.vocab, i.num_docs, K, tr.alpha, tr.beta, num_dense=tr.Vd)


# the sampler's variants change at 256, 1024 and 2048 topics, a lane's Q topics at multiples of 32
@pytest.mark.parametrize("ll", [False, True])
@pytest.mark.parametrize("K", [31, 32, 33, 256, 257, 1023, 1025, 2048, 2049, 4097])
def test_topic_counts_at_the_variants_edges(K, ll):
    c = L.Corpus.generate(L.corpus_config("c0", num_docs=300, vocab=700, K=K, num_chunks=2, dense_kind=2,
                                          dense_param=40.0, len_p1=150.0))
    tr = L.Trainer(c, K=K, seed=11)
    o = _oracle(c, tr, K)
    z = c.topics()
    for it in range(3):
        st = o.iterate(z, 11, it, ll=ll)
        tr.iterate(1, ll=ll)
        assert np.array_equal(tr.topics(), z), f"sweep {it}"
        if ll:
            assert abs(tr.loglik()[0] - st.loglik) <= 1e-9 * abs(st.loglik)
    cnt = tr.counters()
    assert cnt.tokens == 3 * len(z)


# doc rows around the row loads' step and batch sizes (32, 64, 96, 128, 256 entries), rows longer
# than a batch, and docs of one token
@pytest.mark.parametrize("K", [200, 1000, 1500, 3000])
def test_doc_rows_around_the_load_batches(K):
    lens = [1, 2, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160, 255, 256, 257, 300, 700]
    rng = np.random.default_rng(5)
    off = np.concatenate([[0], np.cumsum(lens * 6)]).astype(np.int64)
    words = rng.integers(0, 90, off[-1]).astype(np.int32)
    # a doc's topics are distinct as far as K goes, so that its row is as long as the doc
    topics = np.concatenate([rng.permutation(max(K, n))[:n] % K for n in lens * 6]).astype(np.uint16)
    c = L.Corpus.from_docs(off, words, vocab=100, K=K, topics=topics, num_chunks=3, dense_kind=2, dense_param=30.0)
    tr = L.Trainer(c, K=K, seed=3)
    o = _oracle(c, tr, K)
    z = c.topics()
    for it in range(2):
        o.iterate(z, 3, it)
        tr.iterate(1)
        assert np.array_equal(tr.topics(), z), f"sweep {it}"


# words without tokens, words that hold every topic of the order list (no three topics left
# outside), and equal topic totals (ties to the lower topic)
@pytest.mark.parametrize("K", [8, 64, 100, 1024, 2049])
def test_word_statistics_ties_and_empty_words(K):
    D, n = 64, 96
    off = np.arange(D + 1, dtype=np.int64) * n
    words = np.tile(np.arange(n, dtype=np.int32) % 12, D)
    topics = (np.arange(D * n) % K).astype(np.uint16)  # every topic (almost) equally often
    c = L.Corpus.from_docs(off, words, vocab=500, K=K, topics=topics, num_chunks=2, dense_kind=2, dense_param=3.0)
    for nd in (0, -1):
        tr = L.Trainer(c, K=K, seed=1, num_dense=nd)
        if nd == -1:
            tr.Vd = 0
        o = _oracle(c, tr, K)
        o.rebuild(c.topics())
        tr.update_wt()
        tr.max_topic()
        tr.sync()
        for a, b, name in zip(tr.word_stats(), o.word_stats(), ("top2", "k3", "phi4", "ql")):
            assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), (name, nd)


# a word of many more tokens than a word-topic or sampler tile holds, and tiles that end
# inside a group
@pytest.mark.parametrize("K,tokens", [(64, 2048), (64, 2049), (64, 9000), (3000, 513), (3000, 5000)])
def test_frequent_word_over_tile_edges(K, tokens):
    rng = np.random.default_rng(tokens)
    words = np.concatenate([np.zeros(tokens, np.int32), rng.integers(1, 50, 3000).astype(np.int32)])
    rng.shuffle(words)
    off = np.minimum(np.arange(0, len(words) + 200, 200), len(words)).astype(np.int64)
    c = L.Corpus.from_docs(np.unique(off), words, vocab=50, K=K, num_chunks=2, dense_kind=2, dense_param=5.0)
    tr = L.Trainer(c, K=K, seed=2)
    o = _oracle(c, tr, K)
    z = c.topics()
    for it in range(2):
        o.iterate(z, 2, it)
        tr.iterate(1)
        assert np.array_equal(tr.topics(), z)
    o.rebuild(z)
    tr.update_wt()
    tr.sync()
    assert np.array_equal(tr.topic_totals(), o.topic_totals())


# large K: sparse words that hold many of the topics (the lookups and Q draws of topic-rich
# words), around the 32 topics of one round and a 32nd of the topics
@pytest.mark.parametrize("ll", [False, True])
@pytest.mark.parametrize("K,per_word", [(2049, 20), (2049, 40), (2049, 64), (2049, 66), (2049, 600), (4096, 2000)])
def test_topic_rich_sparse_words_at_large_k(K, per_word, ll):
    vocab = 24
    rng = np.random.default_rng(per_word)
    words = np.repeat(np.arange(vocab, dtype=np.int32), per_word)
    rng.shuffle(words)
    off = np.unique(np.append(np.arange(0, len(words), 150), len(words))).astype(np.int64)
    c = L.Corpus.from_docs(off, words, vocab=vocab, K=K, num_chunks=2, dense_kind=2, dense_param=2.0)
    tr = L.Trainer(c, K=K, alpha=0.1, seed=4)
    o = _oracle(c, tr, K)
    z = c.topics()
    for it in range(3):
        st = o.iterate(z, 4, it, ll=ll)
        tr.iterate(1, ll=ll)
        assert np.array_equal(tr.topics(), z), f"sweep {it}"
        if ll:
            assert abs(tr.loglik()[0] - st.loglik) <= 1e-9 * abs(st.loglik)


# more requests than slots and a fragmented token pool: admissions and retirements change the
# request table at nearly every step; rows beyond the 128 entries held in registers
@pytest.mark.parametrize("K,active", [(300, 3), (1024, 5), (1025, 2)])
def test_foldin_admissions_and_long_rows(K, active):
    c = L.Corpus.generate(L.corpus_config("c0", num_docs=200, vocab=600, K=K))
    tr = L.Trainer(c, K=K, seed=42)
    tr.iterate(3)
    o = _oracle(c, tr, K)
    o.rebuild(tr.topics())
    rng = np.random.default_rng(1)
    lens = [1, 700, 33, 128, 129, 5, 257, 64, 900, 2, 31, 400]
    docs = [rng.integers(0, 600, n).astype(np.int32) for n in lens]
    s = Server(Model(tr), sweeps=5, max_active=active, max_tokens=1500, seed=9)
    got = s.run(docs)
    for rid, d in enumerate(docs):
        _, th = o.foldin(d, rid, 9, 5)
        assert np.array_equal(got[rid].view(np.uint32), th.view(np.uint32)), f"request {rid} of {len(d)} tokens"
