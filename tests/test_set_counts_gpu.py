"""Counts set from outside (tmt_set_counts) that do not contain the uploaded
documents' assignments: sweeps then take tokens off cells that never held them, so
n_kw turns negative.  Sweeps and inference on such a state, and inference at the
count where the kernels' conversions change, equal the oracle bit for bit."""
import math

import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T
from tomotopy_b200._lib import lib
from tomotopy_b200.engine import _p, check

pytestmark = pytest.mark.gpu


def corpus(seed, V=250, D=60):
    off, w = T.synth_corpus(V, 8, D, ("poisson", 60, 1, 400), seed=seed)
    off, w, V, _ = T.prepare_ids(off, w)
    return O.Corpus(off, w, V)


def unseen(V, seed):
    rng = np.random.default_rng(seed)
    docs = [np.sort(rng.integers(0, V, n)) for n in (0, 1, 31, 64, 97, 150)]
    docs.append(np.array([1] * 40 + [2, 3, 3], np.int64))
    off = np.concatenate([[0], np.cumsum([len(d) for d in docs])]).astype(np.uint64)
    return off, np.concatenate(docs).astype(np.uint32)


def set_counts(eng, nkw, nk):
    check(lib.tmt_set_counts(eng.h, _p(nkw), _p(nk)), eng.h)


def assert_infers(eng, K, V, nkw, nk, alpha, seed):
    off, w = unseen(V, seed)
    theta, ll = eng.infer(off, w, iters=6, seed=3)
    for d in range(len(off) - 1):
        ol, _, _, ot = O.infer_doc(K, V, alpha, 0.01, nkw, nk, w[off[d]:off[d + 1]], 6, 3, 0)
        np.testing.assert_array_equal(theta[d], ot)
        if np.isfinite(ol):
            # differences of lgammas: each within 4 ulp here, 1 in the oracle, two
            # of the largest count's size in each of the two cells that can be large
            tol = 1e-9 + 4 * 5 * np.spacing(math.lgamma(max(2, nkw.max(), nk.max())))
            assert ll[d] == pytest.approx(ol, rel=1e-12, abs=tol)


@pytest.mark.parametrize("K", [20, 100, 300, 600, 1000, 1100])
def test_sweeps_and_inference_on_foreign_counts(K):
    c = corpus(K)
    eng = T.Engine(K, c.V, alpha=0.1, eta=0.01, seed=2, optim_interval=0, sweep_groups=2)
    eng.upload(c.doc_off, c.words)
    st = O.State(c, K, 0.1, 0.01, 2)
    rng = np.random.default_rng(K)
    nkw = (rng.integers(0, 4, (c.V, K)) * (rng.random((c.V, K)) < 0.3)).astype(np.int32)
    nk = (nkw.sum(axis=0) + 2 * len(c.words)).astype(np.int32)      # stays positive
    set_counts(eng, nkw, nk)
    st.nkw, st.nk = nkw.copy(), nk.copy()
    assert_infers(eng, K, c.V, nkw, nk, st.alpha, K)
    for step in (0, 2):
        eng.train(2)
        st.doc_live_sweeps(2, start_step=step, groups=2)
        z, gkw, gk, _ = eng.state()
        np.testing.assert_array_equal(z, st.z)
        np.testing.assert_array_equal(gkw, st.nkw)
        np.testing.assert_array_equal(gk, st.nk)
        assert (gkw < 0).any() and (gk > 0).all()
        assert_infers(eng, K, c.V, gkw, gk, st.alpha, K + step)
    # counts without negative ones again
    set_counts(eng, nkw, nk)
    assert_infers(eng, K, c.V, nkw, nk, st.alpha, K)


@pytest.mark.parametrize("K", [20, 130, 1000])
@pytest.mark.parametrize("top", [-1, 0, 1, 6, (1 << 23) + 3, 1 << 30])
def test_inference_around_exact_counts(K, top):
    """The largest count with the longest document (150 tokens) added: 2^23 + top."""
    c = corpus(7)
    eng = T.Engine(K, c.V, alpha=0.1, eta=0.01, seed=2, optim_interval=0)
    eng.upload(c.doc_off, c.words)
    _, nkw, nk, alpha = eng.state()
    big = (1 << 23) - 150 + top
    nkw[3, 2], nk[2] = big, big
    set_counts(eng, nkw, nk)
    assert_infers(eng, K, c.V, nkw, nk, alpha, K)


def test_only_a_word_count_is_large():
    """n_k says nothing about n_kw once counts are set."""
    K, c = 20, corpus(8)
    eng = T.Engine(K, c.V, alpha=0.1, eta=0.01, seed=2, optim_interval=0)
    eng.upload(c.doc_off, c.words)
    _, nkw, nk, alpha = eng.state()
    nkw[3, 2] = (1 << 23) + 5
    set_counts(eng, nkw, nk)
    assert_infers(eng, K, c.V, nkw, nk, alpha, 1)
