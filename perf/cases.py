"""The work that this framework's performance is measured on: training sweeps, batched
training and fold-in serving, each through the calls a user's program makes.

A corpus is drawn on the GPU from the LDA generative process (Zipf word base, Dirichlet
topics and documents) and handed over in document order, as a program with its own
documents does (Corpus.from_docs).  A training case stands for a run in progress: prepare()
sweeps `burn` times from random topics, and a pass is the next `sweeps` sweeps.  Cases with
burn 0 are the start of a run.
"""
import numpy as np
import torch

import lda_sc20_b200 as L
from lda_sc20_b200.batch import Batch
from lda_sc20_b200.serving import Model, Server

# what the fields of a training case mean when it does not say otherwise
TRAIN = dict(kind="train", docs=2000, vocab=5000, mean_len=100.0, sigma=0.0, gen_topics=32, K=64, chunks=1, dense="count",
             alpha=0.0, burn=20, sweeps=1, ll=False, mode="resident")


def _train(name, **kw):
    return dict(TRAIN, name=name, **kw)


def listed():
    return [
        # the smallest training run (the K=64 corpus), the log-likelihood printed every sweep
        # as the command-line driver does: latency and launches count
        _train("small_k64_ll", ll=True),
        # the same corpus, ten sweeps per call without the log-likelihood
        _train("small_k64_x10", sweeps=10),
        # an ordinary run with an odd topic count, uneven documents and three chunks
        _train("mid_k100", docs=9001, vocab=12345, mean_len=181.0, sigma=0.6, gen_topics=40, K=100, chunks=3),
        # the K=1024 corpus at one fifth of its documents (the driver's own setting: K=1024, 8 chunks)
        _train("big_k1024", docs=60000, vocab=60000, mean_len=240.0, sigma=0.6, gen_topics=256, K=1024, chunks=8,
               dense="fraction"),
        # the first sweeps of a K=1024 run, with the log-likelihood of each
        _train("start_k1024_ll", docs=12000, vocab=30000, mean_len=240.0, sigma=0.6, gen_topics=128, K=1024, chunks=8,
               dense="fraction", burn=0, ll=True),
        # more topics than 1024, not a multiple of 32
        _train("mid_k1500", docs=15000, vocab=25000, mean_len=200.0, sigma=0.6, gen_topics=128, K=1500, chunks=4,
               dense="fraction"),
        # the large-K corpus (K=10,000, 8 chunks), scaled down
        _train("big_k10000", docs=40000, vocab=60000, mean_len=250.0, gen_topics=250, K=10000, chunks=8, dense="top",
               alpha=0.1, burn=6),
        # large K streamed through four slots of a device budget
        _train("stream_k4096", docs=16000, vocab=40000, mean_len=250.0, gen_topics=128, K=4096, chunks=8, dense="top",
               alpha=0.1, burn=6, mode="stream"),
        # topics kept in pinned host buffers and copied in and out every sweep, chained
        _train("host_k1024", docs=20000, vocab=40000, mean_len=240.0, sigma=0.6, gen_topics=128, K=1024, chunks=8,
               dense="fraction", sweeps=4, mode="host"),
        # many independent models of uneven size in one launch
        dict(name="batch_48", kind="batch", models=48, docs_lo=100, docs_hi=5000, vocab_lo=1000, vocab_hi=20000,
             mean_len=80.0, gen_topics=16, burn=20, sweeps=4),
        # fold-in of one new document at a time: the latency of a single request
        dict(name="serve_one", kind="serve", requests=1, median_len=150.0, sigma=1.0, sweeps=30, K=1024, vocab=40000),
        # a burst of requests of very different lengths, continuously batched
        dict(name="serve_many", kind="serve", requests=2048, median_len=150.0, sigma=1.0, sweeps=30, K=1024, vocab=40000),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    what = rng.choice(["small", "mid", "mid", "big", "large", "start", "host", "batch", "serve", "serve"])
    if what == "batch":
        return dict(kind="batch", models=rng.randint(5, 40), docs_lo=100, docs_hi=_log(rng, 300, 5000), vocab_lo=1000,
                    vocab_hi=_log(rng, 2000, 20000), mean_len=rng.choice([40.0, 80.0, 117.0]), gen_topics=16, burn=20,
                    sweeps=rng.randint(1, 4))
    if what == "serve":
        return dict(kind="serve", requests=_log(rng, 1, 2000), median_len=float(_log(rng, 30, 300)), sigma=rng.choice([0.3, 1.0]),
                    sweeps=rng.choice([10, 30]), K=rng.choice([64, 100, 300, 1000, 1024]), vocab=_log(rng, 5000, 40000))
    c = dict(TRAIN, vocab=_log(rng, 3000, 40000), mean_len=float(_log(rng, 40, 300)), sigma=rng.choice([0.0, 0.6, 0.9]),
             gen_topics=rng.choice([16, 40, 128]), chunks=rng.randint(1, 8))
    if what == "small":
        tokens, K = _log(rng, 20000, 400000), rng.choice([16, 33, 64, 100])
    elif what == "large":
        tokens, K = _log(rng, 200000, 4000000), rng.choice([2049, 3000, 4096, 7001])
        c.update(dense="top", alpha=0.1, burn=5, mode=rng.choice(["resident", "stream"]), ll=rng.random() < 0.3)
    elif what == "big":
        tokens, K = _log(rng, 3000000, 10000000), rng.choice([256, 777, 1024])
        c.update(dense="fraction", ll=rng.random() < 0.3)
    else:
        tokens, K = _log(rng, 300000, 4000000), rng.choice([50, 128, 256, 500, 1000, 1024, 2000, 2048])
        c.update(dense=rng.choice(["count", "fraction"]), ll=rng.random() < 0.3)
    c.update(K=K, docs=max(c["chunks"], int(tokens / c["mean_len"])))
    if what == "start":
        c.update(burn=0, ll=True, sweeps=1)
    elif what == "host":
        c.update(mode="host", ll=False, sweeps=rng.randint(1, 4))
    elif not c["ll"]:
        c.update(sweeps=rng.randint(1, 3))
    return c


# ------------------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 2654435761 % (1 << 62) + 17)
    return g


def _cdf(shape, g):
    """Cumulative Dirichlet draws, one per row of the Gamma shapes; row i spans [i, i + 1]."""
    x = torch._standard_gamma(shape, generator=g).double().clamp_min_(1e-300)
    x = torch.cumsum(x, 1)
    x /= x[:, -1:].clone()
    x += torch.arange(x.shape[0], device=x.device, dtype=x.dtype)[:, None]
    return x


def _pick(cdf, row, g):
    """One draw from row `row` of the cumulative table for each token."""
    u = torch.rand(row.shape, generator=g, device="cuda", dtype=torch.float64) + row
    n = cdf.shape[1]
    at = torch.searchsorted(cdf.view(-1), u, right=True) - row * n
    return at.clamp_(0, n - 1)


def _words_of_topics(vocab, topics, g):
    z = 1.0 / torch.arange(1, vocab + 1, device="cuda", dtype=torch.float64) ** 1.05
    a = (0.05 * vocab * z / z.sum()).float()
    return _cdf(a.expand(topics, vocab).contiguous(), g)


def _lengths(n, mean, sigma, lo, hi, g):
    if sigma > 0:
        mu = np.log(mean) - 0.5 * sigma * sigma
        x = torch.exp(mu + sigma * torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    else:
        x = torch.poisson(torch.full((n,), mean, device="cuda", dtype=torch.float64), generator=g)
    return x.round().clamp(lo, hi).long()


def _documents(lens, phi, g):
    """The tokens of documents of the given lengths, in document order: (doc of each, word of each)."""
    doc = torch.repeat_interleave(torch.arange(lens.numel(), device="cuda"), lens)
    theta = _cdf(torch.full((lens.numel(), phi.shape[0]), 0.1, device="cuda"), g)
    return doc, _pick(phi, _pick(theta, doc, g), g)


def _corpus_arrays(c, seed):
    g = _gen(seed)
    phi = _words_of_topics(c["vocab"], c["gen_topics"], g)
    # the documents' lengths are the case's: every seed's arrays have the same sizes
    lens = _lengths(c["docs"], c["mean_len"], c["sigma"], 5, 4000, _gen(c["docs"] * 31 + c["vocab"]))
    doc, word = _documents(lens, phi, g)
    topic = torch.randint(0, c["K"], word.shape, generator=g, device="cuda")
    return lens, doc, word, topic


def _corpus(c, lens, word, topic):
    off = torch.zeros(lens.numel() + 1, dtype=torch.int64)
    off[1:] = torch.cumsum(lens, 0).cpu()
    kind, param = {"count": (0, 0.0), "fraction": (1, 0.02), "top": (2, float(c["vocab"] // 50))}[c["dense"]]
    return L.Corpus.from_docs(off.numpy(), word.to(torch.int32).cpu().numpy(), vocab=c["vocab"], K=c["K"],
                              topics=topic.to(torch.int32).cpu().numpy().astype(np.uint16), num_chunks=c["chunks"],
                              dense_kind=kind, dense_param=param)


class _Device:
    """A trainer's topics on the device as torch sees them (no copy); a tensor over it keeps
    it, and so the trainer that owns the memory, alive."""

    def __init__(self, trainer):
        ptr, n = trainer.topics_device()
        self.trainer = trainer
        self.__cuda_array_interface__ = dict(shape=(n,), typestr="<i2", data=(ptr, False), version=3)


def _topics_of(trainer):
    return torch.as_tensor(_Device(trainer), device="cuda")


def _trainer(c, seed):
    lens, _, word, topic = _corpus_arrays(c, seed)
    corpus = _corpus(c, lens, word, topic)
    kw = dict(stream_mode=2, num_streams=4) if c["mode"] == "stream" else {}
    t = L.Trainer(corpus, K=c["K"], alpha=c["alpha"] or None, seed=seed & 0xFFFF, **kw)
    corpus.close()
    if c["burn"]:
        t.iterate(c["burn"])
    return t


# ------------------------------------------------------------------------- the passes

def prepare(case, seed):
    if case["kind"] == "train":
        t = _trainer(case, seed)
        s = dict(kind="train", mode=case["mode"], t=t, sweeps=case["sweeps"], ll=case["ll"], z=_topics_of(t))
        if case["mode"] == "host":
            s["host"] = [torch.from_numpy(t.topics().view(np.int16)).pin_memory() for _ in range(2)]
            s["np"] = [x.numpy().view(np.uint16) for x in s["host"]]
        return s
    if case["kind"] == "batch":
        r = np.random.default_rng(case["models"])  # the models' sizes are the case's
        trainers = []
        for m in range(case["models"]):
            c = dict(TRAIN, docs=int(r.integers(case["docs_lo"], case["docs_hi"] + 1)),
                     vocab=int(r.integers(case["vocab_lo"], case["vocab_hi"] + 1)), mean_len=case["mean_len"],
                     gen_topics=case["gen_topics"], K=int(r.choice([16, 32, 64, 128, 256])), burn=0)
            trainers.append(_trainer(c, seed * 1000 + m))
        b = Batch(trainers)
        b.iterate(case["burn"])
        return dict(kind="batch", b=b, sweeps=case["sweeps"], z=[_topics_of(t) for t in trainers])
    # serving: a model trained for a few sweeps on documents of the same process
    c = dict(TRAIN, docs=6000, vocab=case["vocab"], mean_len=240.0, sigma=0.6, gen_topics=128, K=case["K"], chunks=4,
             dense="fraction", burn=30)
    t = _trainer(c, seed)
    model = Model(t)
    t.close()
    g = _gen(seed + 1)
    lens = _lengths(case["requests"], case["median_len"] * float(np.exp(0.5 * case["sigma"] ** 2)), case["sigma"], 5, 4000,
                    _gen(case["requests"]))
    _, word = _documents(lens, _words_of_topics(case["vocab"], 128, g), g)
    words = word.to(torch.int32).cpu().numpy()
    off = np.concatenate([[0], np.cumsum(lens.cpu().numpy())]).astype(np.int64)
    tokens = max(1 << 16, 1 << int(np.ceil(np.log2(len(words) + 1))))
    server = Server(model, sweeps=case["sweeps"], max_tokens=tokens, seed=seed & 0xFFFF)
    return dict(kind="serve", server=server, model=model, off=off, words=words, n=case["requests"])


def run(state):
    if state["kind"] == "train":
        t = state["t"]
        if state["mode"] == "host":
            bufs = state["np"]
            for _ in range(state["sweeps"]):
                t.iterate_host_async(bufs[0], bufs[1])
                bufs[0], bufs[1] = bufs[1], bufs[0]
                state["host"].reverse()
            t.wait()
            return state["host"][0]
        ll = t.iterate(state["sweeps"], ll=state["ll"])
        return [state["z"], ll] if state["ll"] else [state["z"]]
    if state["kind"] == "batch":
        return state["z"] + [state["b"].iterate(state["sweeps"], ll=True)]
    s = state["server"]
    if state["n"] == 1:
        return s.run([state["words"]])[0]
    return s.replay(state["off"], state["words"], np.zeros(state["n"]), want_theta=True)[1]


def work(case):
    """Per token and sweep: its doc, its place and word in document order, its topic read and
    written (16 bytes), and a multiply-add for each of a few topics of its document."""
    if case["kind"] == "train":
        n = case["docs"] * case["mean_len"] * case["sweeps"]
        extra = 4 * case["K"] * case["sweeps"]
    elif case["kind"] == "batch":
        n = case["models"] * 0.5 * (case["docs_lo"] + case["docs_hi"]) * case["mean_len"] * case["sweeps"]
        extra = 4 * 100 * case["models"] * case["sweeps"]
    else:
        n = case["requests"] * case["median_len"] * float(np.exp(0.5 * case["sigma"] ** 2)) * case["sweeps"]
        extra = 4 * case["K"] * case["requests"]
    return {"bytes": 16.0 * n + extra, "flops": 2.0 * n * 16}


def exact(case, seed):
    """The mean per-token log-likelihood of the starting topics in 64 bits, where a pass
    evaluates it from topics that this file drew; sampled topics have no such value."""
    if case["kind"] != "train" or not case["ll"] or case["burn"] or case["sweeps"] != 1:
        return None
    lens, doc, word, topic = _corpus_arrays(case, seed)
    D, V, K, N = case["docs"], case["vocab"], case["K"], word.numel()
    alpha = float(np.float32(case["alpha"] or 50.0 / K))
    beta = float(np.float32(0.01))
    n_k = torch.bincount(topic, minlength=K).double()
    phi = (torch.bincount(word * K + topic, minlength=V * K).view(V, K).double() + beta) / (n_k + V * beta)
    n_dk = torch.bincount(doc * K + topic, minlength=D * K).view(D, K).int()
    total = torch.zeros((), dtype=torch.float64, device="cuda")
    step = max(1, (1 << 27) // K)
    for i in range(0, N, step):
        d, w = doc[i:i + step], word[i:i + step]
        p = torch.einsum("nk,nk->n", n_dk[d].double() + alpha, phi[w])
        total += torch.log(p / (lens[d].double() + K * alpha)).sum()
    return [None, float(total) / N]
