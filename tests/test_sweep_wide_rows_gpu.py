"""The shared-row sweep kernel (K in 513..1024) on what reaches it by another way than a
plain corpus: documents that share a row (the token pipeline starts anew for each
of a row's documents), rows and masked documents of 65,536 tokens and more, and
corpora sharded across ranks (the count deltas go to exchange buffers).  z and
every count equal the oracle's, or one engine's, bit for bit."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T
from test_shard_gpu import corpus as shard_corpus, run_sharded, run_single

pytestmark = pytest.mark.gpu


def assert_same(eng, st):
    z, nkw, nk, _ = eng.state()
    np.testing.assert_array_equal(z, st.z)
    np.testing.assert_array_equal(nk, st.nk)
    np.testing.assert_array_equal(nkw, st.nkw)
    np.testing.assert_array_equal(eng.doc_topic(), st.ndk)


@pytest.mark.parametrize("K,R", [(520, 9), (600, 150), (1000, 40), (1024, 300)])
def test_shared_rows_bitexact(K, R):
    off, w = T.synth_corpus(600, 15, 300, ("lognormal", float(np.log(20)), 0.9, 0, 150), seed=K)
    off, w, V, _ = T.prepare_ids(off, w)
    w = w.copy()
    w[::29] = V + 1
    rows = np.random.default_rng(K).integers(0, R, len(off) - 1).astype(np.uint32)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=3, optim_interval=0, sweep_groups=2)
    eng.upload(off, w)
    eng.set_doc_rows(rows, R)
    st = O.StateR(O.Corpus(off, w, V), K, 0.1, 0.01, 3, rows, R)
    for step in (0, 2):
        eng.train(2)
        st.doc_live_sweeps(2, start_step=step, groups=2)
        assert_same(eng, st)


@pytest.mark.parametrize("extra", [0, 1])
def test_shared_row_of_many_tokens_bitexact(extra):
    """Three documents below 65,536 tokens whose row holds 65,535 + extra, all on one topic."""
    rng = np.random.default_rng(extra)
    V, K = 40, 520
    lens = [30000, 35000, 535 + extra, 30]
    w = np.concatenate([np.sort(rng.integers(0, V, n)) for n in lens]).astype(np.uint32)
    off = np.concatenate([[0], np.cumsum(lens)]).astype(np.uint64)
    rows = np.array([0, 0, 0, 1], np.uint32)
    z0 = np.full(len(w), 5, np.uint16)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=7, optim_interval=0, sweep_groups=1)
    eng.upload(off, w, z0=z0)
    eng.set_doc_rows(rows, 2)
    st = O.StateR(O.Corpus(off, w, V), K, 0.1, 0.01, 7, rows, 2, z0=z0)
    eng.train(1)
    st.doc_live_sweeps(1, groups=1)
    assert_same(eng, st)


def test_masked_document_of_many_tokens_bitexact():
    rng = np.random.default_rng(3)
    V, K, n = 40, 700, 65536
    w = np.concatenate([np.sort(rng.integers(0, V, n)), np.arange(30)]).astype(np.uint32)
    off = np.array([0, n, n + 30], np.uint64)
    mask = np.zeros((2, K), bool)
    mask[0, [3, 130, 699]] = True
    mask[1, [0, 3]] = True
    z0 = np.full(len(w), 3, np.uint16)
    rows = rng.uniform(0.05, 0.5, (2, K)).astype(np.float32)
    doc_row = np.array([1, 0], np.uint32)
    eng = T.Engine(K, V, alpha=0.1, eta=0.01, seed=7, optim_interval=0, sweep_groups=1)
    eng.upload(off, w, z0=z0)
    eng.set_doc_topic_mask(mask)
    eng.set_doc_alpha(rows, doc_row)
    st = O.StateM(O.Corpus(off, w, V), K, 0.1, 0.01, 7, z0, mask=mask, alpha_rows=rows, doc_row=doc_row)
    eng.train(2)
    st.doc_live_sweeps(2, groups=1)
    assert_same(eng, st)


@pytest.mark.parametrize("K,groups,cuts", [(520, 3, [0, 150, 400]), (1000, 1, [0, 90, 260, 400])])
def test_sharded_equals_one_gpu(K, groups, cuts):
    off, w, V = shard_corpus()
    ref = run_single(off, w, V, K, 3, groups, 0)
    out, _ = run_sharded(off, w, V, K, cuts, 3, groups, 0)
    np.testing.assert_array_equal(np.concatenate([o[0] for o in out]), ref[0])
    np.testing.assert_array_equal(np.concatenate([o[4] for o in out]), ref[4])
    for o in out:
        np.testing.assert_array_equal(o[1], ref[1])
        np.testing.assert_array_equal(o[2], ref[2])
        assert o[5][1] == ref[5][1]


@pytest.mark.parametrize("K", [520, 1000])
def test_sharded_alpha_optimisation(K):
    """Several blocks of topics in the optimiser, their sums reduced over the ranks: FP64
    sums in another order, so a topic's alpha can round to the next float.  A step adds
    digamma(alpha) for every document (D, an ulp or two of 1 / alpha each) to a sum of
    at least nz / alpha: D / nz x 2e-7 in each of ten steps, 1e-4 with nz / D > 0.02."""
    off, w, V = shard_corpus()
    ref = run_single(off, w, V, K, 1, 2, 1)
    out, _ = run_sharded(off, w, V, K, [0, 200, 400], 1, 2, 1, ll=False)
    np.testing.assert_array_equal(np.concatenate([o[0] for o in out]), ref[0])   # drawn before the first step
    assert (ref[4] > 0).mean(axis=0).min() > 0.02
    for o in out:
        np.testing.assert_allclose(o[3], ref[3], rtol=1e-4)
        np.testing.assert_array_equal(o[3], out[0][3])
