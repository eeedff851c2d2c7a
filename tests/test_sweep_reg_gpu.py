"""The register-row sweep kernel (K <= 512) at the edges of its variants: the
topic counts where the lane layout or the scan depth changes, batches with
words outside the vocabulary (none, some or all tokens of a batch of 32
sampled), every split step class, and the documents it leaves to the general
kernel (2^24 tokens or more).  z and every count equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T

pytestmark = pytest.mark.gpu

EDGES = [2, 4, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257, 384, 385, 511, 512, 513]


def gappy_corpus(seed, V=400, D=70):
    off, w = T.synth_corpus(V, 10, D, ("lognormal", float(np.log(80)), 1.0, 1, 1500), seed=seed)
    off, w, V, _ = T.prepare_ids(off, w)
    w = w.copy()
    o = off.astype(np.int64)
    w[::29] = V + 1                                    # scattered
    d = int(np.argmax(np.diff(o)))
    w[o[d] + 40:o[d] + 115] = V + 7                    # two whole batches, then sampled words again
    s = int(np.argmin(np.diff(o)))
    w[o[s]:o[s + 1]] = V                               # a document without sampled words
    return off, w, V


def assert_same(eng, st):
    z, nkw, nk, _ = eng.state()
    np.testing.assert_array_equal(z, st.z)
    np.testing.assert_array_equal(nk, st.nk)
    np.testing.assert_array_equal(nkw, st.nkw)
    np.testing.assert_array_equal(eng.doc_topic(), st.ndk)


@pytest.mark.parametrize("K", EDGES)
def test_topic_count_edges_bitexact(K):
    off, w, V = gappy_corpus(seed=100 + K)
    step = (16, 5, 40, 32, 1)[K % 5]
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=2, optim_interval=0, sweep_groups=2)
    eng.set_doc_split(150, step)
    eng.upload(off, w)
    st = O.State(O.Corpus(off, w, V), K, 0.1, 0.01, 2)
    eng.train(3)
    st.doc_live_sweeps(3, groups=2, split_min=150, split_step=step)
    assert_same(eng, st)


@pytest.mark.parametrize("K", [32, 128, 200, 300, 500])
def test_weighted_edges_bitexact(K):
    off, w, V = gappy_corpus(seed=200 + K)
    c = O.Corpus(off, w, V)
    wt = O.weights_idf(c)[0]
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=3, optim_interval=0, sweep_groups=2)
    eng.upload(off, w, weights=wt)
    st = O.StateW(c, K, 0.1, 0.01, 3, wt)
    eng.train(3)
    st.doc_live_sweeps(3, groups=2)
    assert_same(eng, st)


@pytest.mark.parametrize("K", [64, 200, 300, 500])
def test_masked_split_edges_bitexact(K):
    off, w, V = gappy_corpus(seed=300 + K)
    D = len(off) - 1
    rng = np.random.default_rng(K)
    mask = rng.random((D, K)) < 0.3
    mask[np.arange(D), rng.integers(0, K, D)] = True
    z0 = np.zeros(len(w), np.uint16)
    for d in range(D):
        z0[off[d]:off[d + 1]] = rng.choice(np.flatnonzero(mask[d]), int(off[d + 1] - off[d]))
    z0[w >= V] = 0xFFFF
    rows = rng.uniform(0.05, 0.5, (4, K)).astype(np.float32)
    doc_row = rng.integers(0, 4, D).astype(np.uint32)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=4, optim_interval=0, sweep_groups=2)
    eng.set_doc_split(150, 16)
    eng.upload(off, w, z0=z0)
    eng.set_doc_topic_mask(mask)
    eng.set_doc_alpha(rows, doc_row)
    st = O.StateM(O.Corpus(off, w, V), K, 0.1, 0.01, 4, z0, mask=mask, alpha_rows=rows, doc_row=doc_row)
    eng.train(3)
    st.doc_live_sweeps(3, groups=2, split_min=150, split_step=16)
    assert_same(eng, st)


@pytest.mark.parametrize("split_min", [0, 2 ** 32 - 1])
def test_documents_past_float_counts_bitexact(split_min):
    n, V, K = (1 << 24) + 77, 50, 3
    rng = np.random.default_rng(1)
    w = np.sort(rng.integers(0, V, n)).astype(np.uint32)
    off = np.array([0, n, n + 40], np.uint64)
    w = np.concatenate([w, np.arange(40, dtype=np.uint32)])
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=5, optim_interval=0, sweep_groups=1)
    eng.set_doc_split(split_min)
    eng.upload(off, w)
    st = O.State(O.Corpus(off, w, V), K, 0.1, 0.01, 5)
    eng.train(1)
    st.doc_live_sweeps(1, groups=1, split_min=split_min)
    assert_same(eng, st)
