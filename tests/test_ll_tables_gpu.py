"""The log-likelihood's tables of small counts, at the edges of their sizes: corpora
too small for any table, and states whose counts and lengths lie inside and past
every table, with asymmetric alpha, before and after an optimisation step."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T

pytestmark = pytest.mark.gpu


def assert_ll(eng, st):
    ld, lr = eng.ll()
    od, orr = st.ll_f64()
    assert ld == pytest.approx(od, rel=1e-11, abs=1e-7)
    assert lr == pytest.approx(orr, rel=1e-11, abs=1e-7)


@pytest.mark.parametrize("D", [1, 5, 64, 65])
@pytest.mark.parametrize("K", [1, 2, 3, 4, 7])
def test_tiny_corpora(K, D):
    """One block of the optimiser's partial sums (D <= 64) holds fewer than four
    numbers at K < 4: no room for tables."""
    off, w = T.synth_corpus(40, 4, D, ("poisson", 12, 1, 60), seed=K + D)
    off, w, V, _ = T.prepare_ids(off, w)
    alpha = (0.05 * (np.arange(K) + 1)).astype(np.float32)
    eng = T.Engine(K, V, alpha=alpha, eta=0.01, seed=3, optim_interval=0)
    eng.upload(off, w)
    st = O.State(O.Corpus(off, w, V), K, alpha, 0.01, 3)
    assert_ll(eng, st)
    ll = eng.train(4, ll_every=2)
    st.doc_live_sweeps(4, groups=8)
    assert ll[-1] == pytest.approx(sum(st.ll_f64()), rel=1e-11, abs=1e-7)


@pytest.mark.parametrize("K,V,D", [(20, 9000, 45000), (65, 6000, 12000), (300, 3000, 2500), (1001, 800, 700)])
def test_tables_and_counts_past_them(K, V, D):
    """More than 2^20 counts; document counts past 1024, word counts and lengths past 4096."""
    off, w = T.synth_corpus(V, 10, D, ("poisson", 14, 1, 80), seed=K)
    rng = np.random.default_rng(K)
    long = np.sort(np.concatenate([np.full(5000, 7), rng.integers(0, V, 900)])).astype(np.uint32)
    off = np.concatenate([off, off[-1:] + np.uint64(len(long))])
    w = np.concatenate([w, long])
    off, w, V, _ = T.prepare_ids(off, w)
    z0 = rng.integers(0, K, len(w)).astype(np.uint16)
    z0[int(off[-2]):] = K - 1                           # the long document's tokens on one topic
    alpha = rng.uniform(0.02, 0.7, K).astype(np.float32)
    eng = T.Engine(K, V, alpha=alpha, eta=0.01, seed=3, optim_interval=1, burn_in=0)
    eng.upload(off, w, z0=z0)
    c = O.Corpus(off, w, V)
    st = O.State(c, K, alpha, 0.01, 3, z0=z0)
    assert (c.D + V) * K > 1 << 20 and st.ndk.max() > 1024 and st.nkw.max() > 4096 and c.doc_len.max() > 4096
    assert_ll(eng, st)
    eng.train(1)
    z, _, _, a = eng.state()
    assert_ll(eng, O.State(c, K, a, 0.01, 3, z0=z))
