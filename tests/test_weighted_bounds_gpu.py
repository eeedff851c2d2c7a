"""Inference against weighted counts at the ends of what set_counts_f32 and the
server accept: up to where the fast modes' reciprocals and products hold, and past it.
theta equals the oracle's bit for bit, batched and served."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T
from tomotopy_b200._lib import lib
from tomotopy_b200.engine import _p, check

pytestmark = pytest.mark.gpu

# (n_kw, n_k) of one topic: 2^38 + 1, past 2^39, where products and the bound on them
# cross, past the reciprocals' range, and where 1 / n_k is below the smallest normal float
COUNTS = [(2.0 ** 38 + 2 ** 15, 2.0 ** 38 + 2 ** 15), (3e12, 4e12), (8e15, 8e15), (1e17, 1e16), (3e32, 4e32), (2e38, 2.5e38),
          (3e38, 2.0), (5.0, 3e38)]


def corpus(seed):
    off, w = T.synth_corpus(200, 8, 50, ("poisson", 50, 1, 300), seed=seed)
    off, w, V, _ = T.prepare_ids(off, w)
    return off, w, V


def queries(V, seed):
    rng = np.random.default_rng(seed)
    docs = [np.sort(rng.integers(0, V, n)) for n in (0, 1, 33, 70)] + [np.array([3] * 20 + [4, 5], np.int64)]
    off = np.concatenate([[0], np.cumsum([len(d) for d in docs])]).astype(np.uint64)
    w = np.concatenate(docs).astype(np.uint32)
    return off, w, rng.uniform(0.2, 4, V).astype(np.float32)[w]


@pytest.mark.parametrize("K", [20, 100, 300, 1000])
@pytest.mark.parametrize("big", COUNTS)
def test_large_weighted_counts(K, big):
    off, w, V = corpus(K)
    wt = np.random.default_rng(K).uniform(0.2, 4, V).astype(np.float32)[w]
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=2, optim_interval=0)
    eng.upload(off, w, weights=wt)
    qo, qw, qt = queries(V, K)
    eng.infer(qo, qw, iters=2, seed=3, weights=qt)            # (the bound of the counts before)
    _, nkw, nk, alpha = eng.state()
    nkw[3, 2], nk[2] = big
    check(lib.tmt_set_counts_f32(eng.h, _p(nkw), _p(nk)), eng.h)
    theta, _ = eng.infer(qo, qw, iters=5, seed=3, weights=qt)
    srv = T.Server(max_slots=8, token_budget=4096, max_doc_len=512)
    rids = srv.submit_batch(srv.add_engine_model(eng), qo, qw, iters=5, seed=3, weights=qt)
    got = {}
    while len(got) < len(rids):
        r = srv.poll(wait_ms=20000)
        assert r is not None
        got[r[0]] = r[2]
    srv.close()
    for d in range(len(qo) - 1):
        a, b = int(qo[d]), int(qo[d + 1])
        _, _, _, ot = O.infer_doc_w(K, V, alpha, 0.01, nkw, nk, qw[a:b], qt[a:b], 5, 3, 0)
        np.testing.assert_array_equal(theta[d], ot)
        np.testing.assert_array_equal(got[int(rids[d])], ot)


def test_served_counts_below_zero():
    """The server takes weighted counts as they are; a negative or non-finite n_kw has to be seen."""
    K = 50
    off, w, V = corpus(1)
    rng = np.random.default_rng(1)
    nkw = (rng.integers(0, 5, (V, K)) * 0.5).astype(np.float32)
    nk = (nkw.sum(axis=0) + 10).astype(np.float32)
    nkw[::3, 4] = -2.0
    qo, qw, qt = queries(V, 9)
    alpha = np.full(K, 0.1, np.float32)
    srv = T.Server(max_slots=8, token_budget=4096, max_doc_len=512)
    rids = srv.submit_batch(srv.add_model(K, V, alpha, 0.01, nkw, nk), qo, qw, iters=5, seed=3, weights=qt)
    for _ in rids:
        rid, _, th, _, _ = srv.poll(wait_ms=20000)
        d = int(rid - rids[0])
        a, b = int(qo[d]), int(qo[d + 1])
        _, _, _, ot = O.infer_doc_w(K, V, alpha, 0.01, nkw, nk, qw[a:b], qt[a:b], 5, 3, 0)
        np.testing.assert_array_equal(th, ot)
    srv.close()
