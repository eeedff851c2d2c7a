"""Documents of 2^24 tokens and more in the register-row kernel, whose counts are no
longer exact as floats: every block count per lane, split and whole documents,
masks and per-document alphas, weights.  Every token starts on one topic, so
its count passes 2^24 (but with `known` below 1, the part of the tokens whose word is
in the vocabulary: the oracle takes a minute for all of them at K = 500).  z and every
count equal the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T

pytestmark = pytest.mark.gpu

N = (1 << 24) + 77
NEVER = 2 ** 32 - 1


def corpus(V=50, known=1.0):
    rng = np.random.default_rng(1)
    w = np.sort(rng.integers(0, V, N)).astype(np.uint32)
    if known < 1:
        w[rng.random(N) >= known] = V + 3
    off = np.array([0, N, N + 40], np.uint64)
    return off, np.concatenate([w, np.arange(40, dtype=np.uint32)]), V


def assert_same(eng, st):
    z, nkw, nk, _ = eng.state()
    np.testing.assert_array_equal(z, st.z)
    np.testing.assert_array_equal(nk, st.nk)
    np.testing.assert_array_equal(nkw, st.nkw)
    np.testing.assert_array_equal(eng.doc_topic(), st.ndk)


@pytest.mark.parametrize("K,split_min,known", [(40, NEVER, 1.0), (130, 0, 1.0), (130, NEVER, 0.05), (300, 0, 0.05),
                                               (300, NEVER, 0.05), (500, 0, 0.05), (500, NEVER, 0.05)])
def test_integer_counts_bitexact(K, split_min, known):
    off, w, V = corpus(known=known)
    z0 = np.full(len(w), K - 2, np.uint16)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=5, optim_interval=0, sweep_groups=1)
    eng.set_doc_split(split_min)
    eng.upload(off, w, z0=z0)
    st = O.State(O.Corpus(off, w, V), K, 0.1, 0.01, 5, z0=z0)
    eng.train(1)
    st.doc_live_sweeps(1, groups=1, split_min=split_min)
    assert_same(eng, st)


def test_masks_alphas_bitexact():
    off, w, V = corpus()
    K = 70
    rng = np.random.default_rng(2)
    mask = rng.random((2, K)) < 0.5
    mask[:, 7] = True
    z0 = np.full(len(w), 7, np.uint16)
    rows = rng.uniform(0.05, 0.5, (2, K)).astype(np.float32)
    doc_row = np.array([1, 0], np.uint32)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=5, optim_interval=0, sweep_groups=1)
    eng.upload(off, w, z0=z0)
    eng.set_doc_topic_mask(mask)
    eng.set_doc_alpha(rows, doc_row)
    st = O.StateM(O.Corpus(off, w, V), K, 0.1, 0.01, 5, z0, mask=mask, alpha_rows=rows, doc_row=doc_row)
    eng.train(1)
    st.doc_live_sweeps(1, groups=1)
    assert_same(eng, st)


def test_weighted_counts_bitexact():
    off, w, V = corpus()
    K = 40
    wt = np.random.default_rng(3).uniform(0.2, 3, V).astype(np.float32)[w]
    z0 = np.full(len(w), 3, np.uint16)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=5, optim_interval=0, sweep_groups=1)
    eng.upload(off, w, z0=z0, weights=wt)
    st = O.StateW(O.Corpus(off, w, V), K, 0.1, 0.01, 5, wt, z0=z0)
    eng.train(1)
    st.doc_live_sweeps(1, groups=1)
    assert_same(eng, st)
