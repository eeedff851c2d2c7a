"""The alpha optimiser's kernels where a launch has several blocks of topics (64
and 256 topics a block), a short last block, and tiles of one document or many,
against the oracle's ten fixed-point iterations.

A topic's numerator sums digamma(n + alpha) - digamma(alpha) over the documents.
The float digammas of device and oracle differ by an ulp or two, in all D documents
alike, 2e-7 |digamma(alpha)| each; the sum is at least nz / alpha with nz
the documents that hold the topic, and |digamma(alpha)| about 1 / alpha: relative to
it D / nz x 2e-7, and ten times that after ten iterations.  With nz / D > 0.02 that is 1e-4,
and twice that is allowed; the test checks nz."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T
from tomotopy_b200._lib import lib
from tomotopy_b200.engine import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weighted", [False, True])
@pytest.mark.parametrize("K", [2, 63, 64, 65, 130, 256, 257, 520, 1000])
def test_one_step_matches_oracle(K, weighted):
    off, w = T.synth_corpus(500, 12, 300, ("poisson", max(60, K), 1, 3000), seed=K)
    off, w, V, _ = T.prepare_ids(off, w)
    c = O.Corpus(off, w, V)
    rng = np.random.default_rng(K)
    alpha = rng.uniform(0.05, 0.6, K).astype(np.float32)
    z0 = rng.integers(0, K, len(w)).astype(np.uint16)
    eng = T.Engine(K, V, alpha=alpha, eta=0.01, seed=5, optim_interval=1, burn_in=0)
    if weighted:
        wt = rng.uniform(0.5, 2.0, V).astype(np.float32)[w]
        eng.upload(off, w, z0=z0, weights=wt)
    else:
        eng.upload(off, w, z0=z0)
    for _ in range(2):                       # (the block counter is left as a second step needs it)
        eng.train(1)
        z, _, _, a = eng.state()
        st = O.StateW(c, K, alpha, 0.01, 5, wt, z0=z) if weighted else O.State(c, K, alpha, 0.01, 5, z0=z)
        assert (st.ndk > 0).mean(axis=0).min() > 0.02
        if weighted:
            st.ndk = eng.doc_topic()         # (the sums' rounding follows the sweeps' order)
        st.optimize_alpha()
        np.testing.assert_allclose(a, st.alpha, rtol=2e-4)
        alpha = a
