"""Inference kernels of K <= 1024 at the edges of their variants: topic counts
where the lane layout, the scan depth or the column loads change, documents
around the batch of 32 tokens, runs of one word inside a batch, across batches
and to the document's end, weighted counts, word priors, launches that stop and
resume, and a second upload into the same handle.  theta equals the oracle's
bit for bit, ll to 1e-12."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T

pytestmark = pytest.mark.gpu

EDGES = [1, 2, 4, 32, 33, 36, 64, 68, 124, 125, 128, 132, 256, 260, 384, 388, 512, 516, 999, 1000, 1024, 1028]


def model(K, seed, weighted=False, priors=None):
    off, w = T.synth_corpus(300, 8, 60, ("poisson", 60, 1, 400), seed=seed)
    off, w, V, _ = T.prepare_ids(off, w)
    c = O.Corpus(off, w, V)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=seed, optim_interval=0)
    if priors is not None:
        eng.set_word_priors(*priors(c))
    wt = vw = None
    if weighted:
        wt, vw = O.weights_idf(c)
        vw = np.where(np.isfinite(vw) & (vw >= 0), vw, np.float32(1))     # words the corpus lacks
    eng.upload(off, w, weights=wt)
    eng.train(5)
    return eng, c, vw


def documents(V, seed):
    """Lengths around the batch size; runs inside a batch, across batches, at the end."""
    rng = np.random.default_rng(seed)
    docs = [np.sort(rng.integers(0, V, n)) for n in (0, 1, 2, 31, 32, 33, 63, 64, 65, 97)]
    docs.append(np.array([3] * 2 + [5] + [7] * 3 + [9] * 40 + [11, 12, 12]))
    docs.append(np.array([1] * 100))
    docs.append(np.array(list(range(30)) + [40] * 6 + [50] * 29 + [60] * 2))
    docs.append(np.concatenate([np.sort(rng.integers(0, V, 45)), [V, V, V + 3]]))      # unknown words
    docs.append(np.array([V + 1, V + 2]))
    off = np.concatenate([[0], np.cumsum([len(d) for d in docs])]).astype(np.uint64)
    return off, np.concatenate(docs).astype(np.uint32)


@pytest.mark.parametrize("K", EDGES)
def test_infer_edges(K):
    eng, c, _ = model(K, 10 + K)
    off, w = documents(c.V, K)
    theta, ll = eng.infer(off, w, iters=9, seed=3)
    _, nkw, nk, alpha = eng.state()
    for d in range(len(off) - 1):
        ol, _, _, ot = O.infer_doc(K, c.V, alpha, 0.01, nkw, nk, w[off[d]:off[d + 1]], 9, 3, 0)
        np.testing.assert_array_equal(theta[d], ot)
        assert ll[d] == pytest.approx(ol, rel=1e-12, abs=1e-9)


@pytest.mark.parametrize("K", [20, 64, 124, 126, 200, 384, 512, 1000, 1024])
def test_weighted_infer_edges(K):
    eng, c, vw = model(K, 20 + K, weighted=True)
    off, w = documents(c.V, K)
    ws = np.where(w < c.V, vw[np.minimum(w, c.V - 1)], 0).astype(np.float32)
    theta, ll = eng.infer(off, w, iters=9, seed=3, weights=ws)
    _, nkw, nk, alpha = eng.state()
    for d in range(len(off) - 1):
        a, b = int(off[d]), int(off[d + 1])
        ol, _, _, ot = O.infer_doc_w(K, c.V, alpha, 0.01, nkw, nk, w[a:b], ws[a:b], 9, 3, 0)
        np.testing.assert_array_equal(theta[d], ot)
        assert ll[d] == pytest.approx(ol, rel=1e-12, abs=1e-9)


@pytest.mark.parametrize("K", [24, 128, 300, 1000])
def test_prior_infer_edges(K):
    def priors(c):
        rng = np.random.default_rng(K)
        ids = np.sort(rng.choice(c.V, 30, replace=False)).astype(np.uint32)
        pr = rng.uniform(0.01, 0.5, (30, K)).astype(np.float32)
        return ids, pr
    eng, c, _ = model(K, 30 + K, priors=priors)
    st = O.StateP(c, K, 0.1, 0.01, 30 + K, *priors(c))
    off, w = documents(c.V, K)
    theta, ll = eng.infer(off, w, iters=9, seed=3)
    _, nkw, nk, alpha = eng.state()
    for d in range(len(off) - 1):
        ol, _, _, ot = st.infer_doc(nkw, nk, alpha, w[off[d]:off[d + 1]], 9, 3, 0)
        np.testing.assert_array_equal(theta[d], ot)
        assert ll[d] == pytest.approx(ol, rel=1e-12, abs=1e-9)


@pytest.mark.parametrize("K", [50, 200, 1000])
def test_served_in_steps_equals_batch(K):
    eng, c, _ = model(K, 40 + K)
    off, w = documents(c.V, K)
    theta, ll = eng.infer(off, w, iters=9, seed=3)
    srv = T.Server(max_slots=8, token_budget=4096, step_token_sweeps=40, max_doc_len=512)
    mid = srv.add_engine_model(eng)
    n = len(off) - 1
    rids = srv.submit_batch(mid, off, w, iters=9, seed=3)
    got = {}
    while len(got) < n:
        r = srv.poll(wait_ms=20000)
        assert r is not None
        got[r[0]] = r
    for d, rid in enumerate(rids):
        np.testing.assert_array_equal(got[int(rid)][2], theta[d])
        assert got[int(rid)][3] == ll[d]
    srv.close()


def test_infer_after_a_second_upload():
    eng, c, _ = model(40, 7)
    off, w = documents(c.V, 7)
    eng.infer(off, w, iters=3, seed=1)
    eng.upload(c.doc_off, c.words)
    theta, ll = eng.infer(off, w, iters=3, seed=1)
    ref = T.Engine(40, c.V, alpha=0.1, eta=0.01, seed=7, optim_interval=0)
    ref.upload(c.doc_off, c.words)
    t2, l2 = ref.infer(off, w, iters=3, seed=1)
    np.testing.assert_array_equal(theta, t2)
    np.testing.assert_array_equal(ll, l2)
