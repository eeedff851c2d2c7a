"""Inference at the edges of the widths above 512 topics (blocks of four topics a lane
5 to 8), plain, weighted and with word priors, 16-byte and element column loads.
theta equals the oracle's bit for bit, ll to 1e-12."""
import numpy as np
import pytest

import oracle as O
from test_infer_reg_gpu import documents, model

pytestmark = pytest.mark.gpu

EDGES = [513, 516, 639, 640, 641, 768, 769, 772, 895, 896, 897, 900, 1021]


@pytest.mark.parametrize("K", EDGES)
def test_plain_and_priors(K):
    def priors(c):
        rng = np.random.default_rng(K)
        ids = np.sort(rng.choice(c.V, 25, replace=False)).astype(np.uint32)
        return ids, rng.uniform(0.005, 0.3, (25, K)).astype(np.float32)

    for pri in (None, priors):
        eng, c, _ = model(K, 5 + K, priors=pri)
        off, w = documents(c.V, K)
        theta, ll = eng.infer(off, w, iters=5, seed=3)
        _, nkw, nk, alpha = eng.state()
        st = O.StateP(c, K, 0.1, 0.01, 5 + K, *pri(c)) if pri else None
        for d in range(len(off) - 1):
            doc = w[off[d]:off[d + 1]]
            if pri:
                ol, _, _, ot = st.infer_doc(nkw, nk, alpha, doc, 5, 3, 0)
            else:
                ol, _, _, ot = O.infer_doc(K, c.V, alpha, 0.01, nkw, nk, doc, 5, 3, 0)
            np.testing.assert_array_equal(theta[d], ot)
            assert ll[d] == pytest.approx(ol, rel=1e-12, abs=1e-9)


@pytest.mark.parametrize("K", [513, 640, 641, 768, 896, 897])
def test_weighted(K):
    eng, c, vw = model(K, 20 + K, weighted=True)
    off, w = documents(c.V, K)
    wt = np.where(w < c.V, vw[np.minimum(w, c.V - 1)], 0).astype(np.float32)
    theta, ll = eng.infer(off, w, iters=5, seed=3, weights=wt)
    _, nkw, nk, alpha = eng.state()
    for d in range(len(off) - 1):
        a, b = int(off[d]), int(off[d + 1])
        ol, _, _, ot = O.infer_doc_w(K, c.V, alpha, 0.01, nkw, nk, w[a:b], wt[a:b], 5, 3, 0)
        np.testing.assert_array_equal(theta[d], ot)
        assert ll[d] == pytest.approx(ol, rel=1e-12, abs=1e-9)
