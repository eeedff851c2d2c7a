"""Batches whose documents are taken up longest first (many documents, some much
longer than the mean) give what the documents give one at a time, and a model of
2^22 tokens and more, whose counts are looked at, what the oracle gives."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [20, 300])
@pytest.mark.parametrize("longest", [90, 4095, 4096, 9001])
def test_ordered_batch_equals_single_documents(K, longest):
    off, w = T.synth_corpus(300, 8, 60, ("poisson", 60, 1, 400), seed=K)
    off, w, V, _ = T.prepare_ids(off, w)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=2, optim_interval=0)
    eng.upload(off, w)
    eng.train(3)
    rng = np.random.default_rng(longest)
    lens = rng.integers(0, 12, 2500)
    lens[[3, 1100, 2499]] = longest, longest - 1, longest // 2
    qo = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    qw = rng.integers(0, V + 2, int(qo[-1])).astype(np.uint32)
    keys = rng.integers(0, 1 << 40, len(lens)).astype(np.uint64)
    theta, ll = eng.infer(qo, qw, iters=2, seed=7, doc_keys=keys)
    for d in [0, 1, 2, 3, 4, 1099, 1100, 1101, 2498, 2499]:
        t1, l1 = eng.infer(np.array([0, lens[d]], np.uint64), qw[int(qo[d]):int(qo[d + 1])], iters=2, seed=7,
                           doc_keys=keys[d:d + 1])
        np.testing.assert_array_equal(theta[d], t1[0])
        assert ll[d] == l1[0]
    assert np.isfinite(theta).all() and np.allclose(theta.sum(axis=1), 1, atol=1e-5)


def test_model_of_many_tokens():
    K = 20
    off, w = T.synth_corpus(400, 8, 22000, ("poisson", 200, 1, 900), seed=1)
    off, w, V, _ = T.prepare_ids(off, w)
    assert len(w) >= 1 << 22
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=2, optim_interval=0)
    eng.upload(off, w)
    rng = np.random.default_rng(1)
    q = np.sort(rng.integers(0, V, 120)).astype(np.uint32)
    for _ in range(2):
        eng.train(1)
        for _ in range(2):                   # (the second call of a state does not look again)
            theta, _ = eng.infer(np.array([0, len(q)], np.uint64), q, iters=5, seed=3)
        _, nkw, nk, alpha = eng.state()
        np.testing.assert_array_equal(theta[0], O.infer_doc(K, V, alpha, 0.01, nkw, nk, q, 5, 3, 0)[3])
