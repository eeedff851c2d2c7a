"""The shared-row sweep kernel (K in 513..1024, and larger launches from K = 257)
at the edges of its variants: every block count per lane, a partial last block,
16-bit and 32-bit count rows, weighted counts, masks and per-document alphas, word
priors, words outside the vocabulary.  z and every count equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T

pytestmark = pytest.mark.gpu


def corpus(seed, V=300, D=60, mean=60):
    off, w = T.synth_corpus(V, 10, D, ("lognormal", float(np.log(mean)), 1.0, 1, 900), seed=seed)
    off, w, V, _ = T.prepare_ids(off, w)
    w = w.copy()
    w[::31] = V + 1
    return off, w, V


def assert_same(eng, st):
    z, nkw, nk, _ = eng.state()
    np.testing.assert_array_equal(z, st.z)
    np.testing.assert_array_equal(nk, st.nk)
    np.testing.assert_array_equal(nkw, st.nkw)
    np.testing.assert_array_equal(eng.doc_topic(), st.ndk)


@pytest.mark.parametrize("K", [513, 640, 641, 768, 769, 896, 897, 1021, 1024])
def test_block_counts_bitexact(K):
    off, w, V = corpus(seed=K)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=2, optim_interval=0, sweep_groups=2)
    eng.upload(off, w)
    st = O.State(O.Corpus(off, w, V), K, 0.1, 0.01, 2)
    eng.train(3)
    st.doc_live_sweeps(3, groups=2)
    assert_same(eng, st)


@pytest.mark.parametrize("K", [257, 384, 385, 512])
def test_many_documents_bitexact(K):
    # 16 documents an SM and more in the launch: this kernel instead of the register rows
    off, w, V = corpus(seed=K, D=2600, mean=6)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=3, optim_interval=0, sweep_groups=1)
    eng.upload(off, w)
    st = O.State(O.Corpus(off, w, V), K, 0.1, 0.01, 3)
    eng.train(2)
    st.doc_live_sweeps(2, groups=1)
    assert_same(eng, st)


@pytest.mark.parametrize("K", [600, 1024])
def test_weighted_bitexact(K):
    off, w, V = corpus(seed=50 + K)
    c = O.Corpus(off, w, V)
    wt = O.weights_idf(c)[0]
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=4, optim_interval=0, sweep_groups=2)
    eng.upload(off, w, weights=wt)
    st = O.StateW(c, K, 0.1, 0.01, 4, wt)
    eng.train(3)
    st.doc_live_sweeps(3, groups=2)
    assert_same(eng, st)


@pytest.mark.parametrize("K", [700, 1000])
def test_masks_alphas_bitexact(K):
    off, w, V = corpus(seed=80 + K)
    D = len(off) - 1
    rng = np.random.default_rng(K)
    mask = rng.random((D, K)) < 0.2
    mask[np.arange(D), rng.integers(0, K, D)] = True
    z0 = np.zeros(len(w), np.uint16)
    for d in range(D):
        z0[off[d]:off[d + 1]] = rng.choice(np.flatnonzero(mask[d]), int(off[d + 1] - off[d]))
    z0[w >= V] = 0xFFFF
    rows = rng.uniform(0.05, 0.5, (4, K)).astype(np.float32)
    doc_row = rng.integers(0, 4, D).astype(np.uint32)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=5, optim_interval=0, sweep_groups=2)
    eng.upload(off, w, z0=z0)
    eng.set_doc_topic_mask(mask)
    eng.set_doc_alpha(rows, doc_row)
    st = O.StateM(O.Corpus(off, w, V), K, 0.1, 0.01, 5, z0, mask=mask, alpha_rows=rows, doc_row=doc_row)
    eng.train(3)
    st.doc_live_sweeps(3, groups=2)
    assert_same(eng, st)


def test_word_priors_bitexact():
    off, w, V = corpus(seed=7)
    K = 530
    rng = np.random.default_rng(1)
    ids = np.sort(rng.choice(V, 20, replace=False)).astype(np.uint32)
    pri = rng.uniform(0.01, 0.5, (20, K)).astype(np.float32)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=6, optim_interval=0, sweep_groups=2)
    eng.set_word_priors(ids, pri)
    eng.upload(off, w)
    st = O.StateP(O.Corpus(off, w, V), K, 0.1, 0.01, 6, ids, pri)
    eng.train(3)
    st.doc_live_sweeps(3, groups=2)
    assert_same(eng, st)


@pytest.mark.parametrize("n", [65535, 65536])
def test_count_row_width_bitexact(n):
    rng = np.random.default_rng(n)
    V, K = 40, 520
    w = np.concatenate([np.sort(rng.integers(0, V, n)), np.arange(30)]).astype(np.uint32)
    off = np.array([0, n, n + 30], np.uint64)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=7, optim_interval=0, sweep_groups=1)
    eng.upload(off, w, z0=np.zeros(len(w), np.uint16))     # every token on topic 0: its count is the length
    st = O.State(O.Corpus(off, w, V), K, 0.1, 0.01, 7, z0=np.zeros(len(w), np.uint16))
    eng.train(1)
    st.doc_live_sweeps(1, groups=1)
    assert_same(eng, st)
