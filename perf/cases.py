"""The work a user of this package has it do, as cases that can be timed.

A case is a dict of plain values; `prepare` makes what the user's program holds
before the call (a model with its corpus uploaded, documents to infer, counts),
`run` is one pass through the public entry points and returns what the user
reads.  Corpora come from the package's seeded LDA generator with the shapes of
bench.py's workloads and of the tests.

Kinds:
  train   Engine.train(iters) with a log-likelihood point half way and at the
          end (as a user watching convergence asks for), then the state read
          back: assignments, n_kw, n_k and the re-fitted alpha.  `opt` is the
          conditional's option: "one" (plain LDA), "idf" (TermWeight IDF),
          "labels" (LLDA's per-document topic masks).
  model   LDAModel.train(iters) on documents of strings, then ll_per_word and
          every topic's word distribution: the smallest call, where launches
          and host work count.
  infer   Engine.infer of a batch of unseen documents against a trained model.
  serve   the same through Server: submit_batch, then poll until all are done.
  ll      Engine.ll of a given state.
"""
import math

import numpy as np
import torch

import tomotopy_b200 as T

ALPHA, ETA = 0.1, 0.01


def listed():
    return [
        # a first look at a small collection through the tomotopy-style class
        dict(name="model_small", kind="model", K=20, V=2000, N=35000, mean=60.0, sigma=0.6, lo=5, hi=400, iters=10),
        # bench.py's c1: few long documents, k=20 (books, reports)
        dict(name="train_c1", kind="train", opt="one", K=20, V=10000, topics=20, N=1_500_000, mean=1500.0, sigma=0.0, lo=1,
             hi=100000, iters=10),
        # bench.py's c2: a mid-size collection, k=100
        dict(name="train_c2", kind="train", opt="one", K=100, V=50000, topics=100, N=27_500_000, mean=200.0, sigma=0.8,
             lo=10, hi=10000, iters=10),
        # bench.py's c3 (its default), k=1000, on the first 24M tokens of it
        dict(name="train_c3", kind="train", opt="one", K=1000, V=100000, topics=1000, N=24_000_000, mean=100.0, sigma=1.2,
             lo=5, hi=5000, iters=10),
        # an odd number of topics and ragged, mostly short documents (posts, abstracts)
        dict(name="train_k333", kind="train", opt="one", K=333, V=20011, topics=100, N=4_900_001, mean=50.0, sigma=1.0, lo=1,
             hi=2000, iters=10),
        # TermWeight.IDF: float counts, the second model size of bench.py's c5
        dict(name="train_idf_k200", kind="train", opt="idf", K=200, V=50000, topics=200, N=8_000_000, mean=100.0, sigma=1.2,
             lo=5, hi=10000, iters=10),
        # LLDA: every document restricted to its labels
        dict(name="train_labels_k130", kind="train", opt="labels", K=130, V=20000, topics=130, N=4_100_000, mean=100.0,
             sigma=0.8, lo=5, hi=5000, iters=10),
        # one unseen document (an interactive request), bench.py's c4 model
        dict(name="infer_one_k100", kind="infer", K=100, V=10000, topics=20, N=1_500_000, mean=1500.0, sigma=0.0, lo=1,
             hi=100000, n=1, qmean=250.0, qsigma=0.0, qhi=5000, iters=50),
        # a batch of unseen documents, bench.py's c4 model and request lengths
        dict(name="infer_c4", kind="infer", K=100, V=10000, topics=20, N=1_500_000, mean=1500.0, sigma=0.0, lo=1, hi=100000,
             n=4096, qmean=150.0, qsigma=1.0, qhi=5000, iters=50),
        # a batch against a large model, the third model of bench.py's c5
        dict(name="infer_k1000", kind="infer", K=1000, V=100000, topics=1000, N=4_000_000, mean=100.0, sigma=1.2, lo=5,
             hi=10000, n=1024, qmean=100.0, qsigma=1.2, qhi=1500, iters=50),
        # served inference at saturation, the first model of bench.py's c5
        dict(name="serve_k50", kind="serve", K=50, V=20000, topics=50, N=4_000_000, mean=100.0, sigma=1.2, lo=5, hi=10000,
             n=4000, qmean=100.0, qsigma=1.2, qhi=10000, iters=100),
        # the log-likelihood of a large state by itself (model selection, convergence checks)
        dict(name="ll_k400", kind="ll", K=400, V=30000, N=10_000_000, mean=150.0, sigma=0.8, lo=1, hi=5000),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "infer", "infer", "model", "serve", "ll"])
    K = _log_uniform(rng, 8, 1000)
    V = _log_uniform(rng, 2000, 100000)
    mean, sigma = float(_log_uniform(rng, 40, 400)), rng.choice([0.0, 0.5, 0.8, 1.2])
    c = dict(kind=kind, K=K, V=V, topics=max(10, K // 2), mean=mean, sigma=sigma, lo=rng.randint(1, 10), hi=5000,
             iters=10)
    c["N"] = _log_uniform(rng, 200_000, 6_000_000)
    if kind == "train":
        c["opt"] = rng.choice(["one", "one", "idf", "labels"])
    elif kind == "model":
        c.update(K=min(K, 60), V=min(V, 5000), N=rng.randint(5_000, 50_000), mean=60.0, sigma=0.6, hi=400)
    elif kind in ("infer", "serve"):
        c["N"] = min(c["N"], 1_000_000)
        n = _log_uniform(rng, 1, 3000) if kind == "infer" else _log_uniform(rng, 50, 3000)
        c.update(n=n, qmean=float(_log_uniform(rng, 30, 300)), qsigma=rng.choice([0.0, 0.8, 1.0]), qhi=1500,
                 iters=rng.choice([10, 50]))
    return c


def _length(mean, sigma, lo, hi):
    if sigma == 0.0:
        return ("poisson", mean, lo, hi)
    return ("lognormal", math.log(mean), sigma, lo, hi)


def _topics(c):
    return c.get("topics", max(2, c["K"]))


def _mean_length(c):
    m, sg = c["mean"], c["sigma"]
    return min(m if sg == 0.0 else m * math.exp(sg * sg / 2), c["hi"])


def _documents(c, seed):
    """Generated documents, the last one cut, N tokens in all: (doc_off, words)."""
    D = int(1.05 * c["N"] / _mean_length(c)) + 16
    while True:
        off, words = T.synth_corpus(c["V"], _topics(c), D, _length(c["mean"], c["sigma"], c["lo"], c["hi"]), seed=seed)
        if len(words) >= c["N"]:
            break
        D = int(1.3 * D)
    return _cut(off, c["N"]), np.ascontiguousarray(words[:c["N"]])


def _cut(off, N):
    off = off[:int(np.searchsorted(off, N)) + 1].copy()
    off[-1] = N
    return off


def _corpus(c, seed):
    """(doc_off, words, vocabulary order) of a prepared corpus."""
    off, words = _documents(c, seed)
    off, words, _, order = T.prepare_ids(off, words)
    return off, words, order


def _idf(off, words, V):
    """(float)log(D / df) per token, as TermWeight.IDF weighs them."""
    o = off.astype(np.int64)
    first = np.ones(len(words), bool)
    first[1:] = words[1:] != words[:-1]
    first[o[:-1][np.diff(o) > 0]] = True
    df = np.bincount(words[first], minlength=V)[:V]
    idf = np.log((len(off) - 1) / np.maximum(df, 1).astype(np.float64)).astype(np.float32)
    return idf[words]


def _labels(off, K, seed):
    """One to four labels a document: the D x K mask and a z0 inside it."""
    g = np.random.default_rng(seed)
    D = len(off) - 1
    lab = g.integers(0, K, size=(D, 4))
    lab[:, 1:] = np.where(np.arange(1, 4)[None, :] < g.integers(1, 5, size=D)[:, None], lab[:, 1:], lab[:, :1])
    mask = np.zeros((D, K), bool)
    mask[np.arange(D)[:, None], lab] = True
    lens = np.diff(off.astype(np.int64))
    doc = np.repeat(np.arange(D), lens)
    z0 = lab[doc, g.integers(0, 4, size=len(doc))].astype(np.uint16)
    return mask, z0


def _queries(c, order, seed):
    """Unseen documents of the model's generative process: (doc_off, words)."""
    off, w = T.synth_corpus(c["V"], _topics(c), c["n"], _length(c["qmean"], c["qsigma"], 10, c["qhi"]), seed=seed,
                            doc_offset=10_000_000)
    # words the model never saw are out of its vocabulary
    w = np.where(w < len(order), order[np.minimum(w, len(order) - 1)], len(order) + 5).astype(np.uint32)
    return off, w


def _ll_state(c, seed):
    """A corpus with an assignment, from the seed alone (numpy)."""
    g = np.random.default_rng(seed)
    N, K, V = c["N"], c["K"], c["V"]
    D = int(1.3 * N / _mean_length(c)) + 64
    if c["sigma"] == 0.0:
        lens = g.poisson(c["mean"], D)
    else:
        lens = np.round(g.lognormal(math.log(c["mean"]), c["sigma"], D))
    lens = np.clip(lens, c["lo"], c["hi"]).astype(np.int64)
    lens[-1] += max(0, N - int(lens.sum()))
    off = _cut(np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64), N)
    lens = np.diff(off.astype(np.int64))
    D = len(lens)
    words = np.minimum((V * g.random(N) ** 3).astype(np.int64), V - 1).astype(np.uint32)   # skewed, as words are
    doc = np.repeat(np.arange(D), lens)
    words = words[np.lexsort((words, doc))]
    # every document leans on a few topics
    own = g.integers(0, K, size=(D, 8))
    z0 = own[doc, g.integers(0, 8, size=N)].astype(np.uint16)
    return off, words, z0


def prepare(case, seed):
    c = dict(case)
    kind = c["kind"]
    if kind == "ll":
        off, words, z0 = _ll_state(c, seed)
        eng = T.Engine(c["K"], c["V"], alpha=ALPHA, eta=ETA, seed=seed)
        eng.upload(off, words, z0=z0)
        return dict(case=c, eng=eng)
    if kind == "model":
        off, words = _documents(c, seed)
        mdl = T.LDAModel(k=c["K"], alpha=ALPHA, eta=ETA, seed=seed)
        names = ["w%d" % i for i in range(c["V"])]
        for d in range(len(off) - 1):
            mdl.add_doc([names[i] for i in words[int(off[d]):int(off[d + 1])]])
        mdl.train(1)
        return dict(case=c, mdl=mdl)
    off, words, order = _corpus(c, seed)
    V = c["V"]
    if kind == "train":
        eng = T.Engine(c["K"], V, alpha=ALPHA, eta=ETA, seed=seed)
        if c["opt"] == "idf":
            eng.upload(off, words, weights=_idf(off, words, V))
        elif c["opt"] == "labels":
            mask, z0 = _labels(off, c["K"], seed)
            eng.upload(off, words, z0=z0)
            eng.set_doc_topic_mask(mask)
        else:
            eng.upload(off, words)
        return dict(case=c, eng=eng)
    # a trained model, alpha re-fitted on the way
    eng = T.Engine(c["K"], V, alpha=ALPHA, eta=ETA, seed=seed)
    eng.upload(off, words)
    eng.train(10)
    qoff, qwords = _queries(c, order, seed)
    st = dict(case=c, eng=eng, off=qoff, words=qwords, seed=seed)
    if kind == "serve":
        st["srv"] = T.Server(max_slots=8192, token_budget=1 << 25, max_doc_len=1 << 16)
        st["mid"] = st["srv"].add_engine_model(eng)
        eng.close()
    return st


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "train":
        eng = state["eng"]
        ll = eng.train(c["iters"], ll_every=max(1, c["iters"] // 2))
        z, nkw, nk, alpha = eng.state()
        return dict(ll=ll, z=z, nkw=nkw, nk=nk, alpha=alpha)
    if kind == "model":
        mdl = state["mdl"]
        mdl.train(c["iters"])
        phi = np.zeros((c["K"], c["V"]), np.float32)         # (a word of the generator's may not occur)
        for k in range(c["K"]):
            dist = mdl.get_topic_word_dist(k)
            phi[k, :len(dist)] = dist
        return dict(phi=phi, alpha=mdl.alpha, n_k=mdl.get_count_by_topics().astype(np.int64),
                    ll_per_word=mdl.ll_per_word)
    if kind == "infer":
        theta, ll = state["eng"].infer(state["off"], state["words"], iters=c["iters"], seed=state["seed"])
        return dict(theta=theta, ll=ll)
    if kind == "ll":
        docs, rest = state["eng"].ll()
        return dict(docs=docs, rest=rest)
    srv, n = state["srv"], c["n"]
    rids = srv.submit_batch(state["mid"], state["off"], state["words"], iters=c["iters"], seed=state["seed"])
    theta = np.empty((n, c["K"]), np.float32)
    ll = np.empty(n, np.float64)
    done, first = 0, int(rids[0])
    while done < n:
        got = srv.poll_batch(max_n=4096, wait_ms=1000)
        if got is None:
            continue
        rid, _, th, l_, _ = got
        at = (rid - np.uint64(first)).astype(np.int64)       # a batch's ids are consecutive
        theta[at] = th[:, :c["K"]]
        ll[at] = l_
        done += len(rid)
    return dict(theta=theta, ll=ll)


def work(case):
    c = case
    K, V, N = c["K"], c["V"], c["N"]
    D = N / _mean_length(c)
    if c["kind"] == "ll":
        # the counts once; an lgamma (~40 operations) per nonzero count, at most one per token in each table
        return {"bytes": 4.0 * (D * K + K * V + D + K), "flops": 80.0 * N}
    if c["kind"] in ("train", "model"):
        # per sweep: a token's word and assignment read, the assignment written
        # (and its weight read), both count tables read and written once; a
        # multiply-add per topic and draw.  Then the state read.
        wt = 4.0 if c.get("opt") == "idf" else 0.0
        per = (8.0 + wt) * N + 8.0 * D * K + 8.0 * K * V
        return {"bytes": c["iters"] * per + 2.0 * N + 4.0 * K * V, "flops": c["iters"] * 2.0 * K * N}
    n, it = c["n"], c["iters"]
    Q = n * min(c["qmean"] * math.exp(c["qsigma"] ** 2 / 2), c["qhi"])
    # the documents and the used part of the model once, theta and ll written;
    # a multiply-add and the word weight (an add and a multiply) per topic and draw
    return {"bytes": 4.0 * Q + 4.0 * K * min(V, Q) + 4.0 * n * K + 8.0 * n, "flops": it * 4.0 * K * Q}


def exact(case, seed):
    """The log-likelihood of a given state in 64 bits (LDAModel::getLLDocs,
    getLLRest).  The other kinds return samples, whole numbers drawn with the
    package's own random stream, and what follows from them."""
    c = case
    if c["kind"] != "ll":
        return None
    off, words, z0 = _ll_state(c, seed)
    K, V, D = c["K"], c["V"], len(off) - 1
    lens = np.diff(off.astype(np.int64))
    doc = np.repeat(np.arange(D), lens)
    alpha, eta = float(np.float32(ALPHA)), float(np.float32(ETA))

    def lg(x):
        return torch.lgamma(torch.as_tensor(np.asarray(x, dtype=np.float64)))

    ndk = np.bincount(doc * K + z0, minlength=D * K)
    ndk = ndk[ndk > 0]
    nkw = np.bincount(words.astype(np.int64) * K + z0, minlength=V * K)
    nkw = nkw[nkw > 0]
    nk = np.bincount(z0, minlength=K)
    docs = (lg(ndk + alpha) - lg(alpha)).sum() - (lg(lens + K * alpha) - lg(K * alpha)).sum()
    rest = (lg(nkw + eta) - lg(eta)).sum() - (lg(nk + V * eta) - lg(V * eta)).sum()
    return dict(docs=float(docs), rest=float(rest))
