"""Inference at the ends of what the fast modes take (launch_infer_reg_g): V eta around
1e-30 and 1e30, and alphas so large that a product of weights could pass the
float range.  On both sides of each line theta equals the oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
import tomotopy_b200 as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K", [20, 130, 300, 1000])
@pytest.mark.parametrize("alpha,veta", [(0.1, 0.9e-30), (0.1, 1.1e-30), (0.1, 1e-37), (0.1, 0.9e30), (0.1, 1.1e30),
                                        (1e23, 1.0), (1e26, 1.0), (1e-30, 1.0)])
def test_ends_of_the_fast_modes(K, alpha, veta):
    off, w = T.synth_corpus(250, 8, 60, ("poisson", 60, 1, 400), seed=K)
    off, w, V, _ = T.prepare_ids(off, w)
    eta = veta / V
    eng = T.Engine(K, V, alpha=alpha, eta=eta, seed=2, optim_interval=0)
    eng.upload(off, w)
    _, nkw, nk, al = eng.state()
    rng = np.random.default_rng(K)
    docs = [np.sort(rng.integers(0, V, n)) for n in (0, 1, 31, 64, 97, 150)] + [np.array([1] * 40 + [2, 3, 3])]
    qo = np.concatenate([[0], np.cumsum([len(d) for d in docs])]).astype(np.uint64)
    qw = np.concatenate(docs).astype(np.uint32)
    theta, _ = eng.infer(qo, qw, iters=6, seed=3)
    for d in range(len(docs)):
        ot = O.infer_doc(K, V, al, eta, nkw, nk, qw[int(qo[d]):int(qo[d + 1])], 6, 3, 0)[3]
        np.testing.assert_array_equal(theta[d], ot)
