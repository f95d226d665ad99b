"""GPU: a log-domain fit's bits do not depend on the other problems of the call.

wdl_fit_weights_log gives a problem between 1 and 16 CTAs, by how many problems share
the GPU; many L-BFGS steps would amplify a sum's other rounding.  Weights, losses and
counts after many iterations are compared bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,K,loss", [(5, 3, 1, 2), (16, 16, 3, 1), (32, 31, 3, 2), (33, 47, 2, 4), (64, 65, 4, 2),
                                        (100, 129, 2, 2), (130, 60, 3, 4)])
def test_fit_bits_alone_and_among_many(W, H, K, loss):
    from wassersteindictionarylearning_b200 import CudaLogSignArrayGaussian2DKernel
    from wassersteindictionarylearning_b200.batch import fit_device
    from wassersteindictionarylearning_b200.synthetic import blob_histograms
    side = max(W, H)
    prob = dict(W=W, H=H, K=K, L=6, loss_type=loss, atoms=blob_histograms(K, W, H, seed=1).reshape(-1),
                observed=blob_histograms(1, W, H, seed=2).reshape(-1))
    fill = dict(prob, W=16, H=16, loss_type=2, observed=blob_histograms(1, 16, 16, seed=3).reshape(-1),
                atoms=blob_histograms(K, 16, 16, seed=4).reshape(-1))
    k = CudaLogSignArrayGaussian2DKernel(2.0, side, side, precision="fp32")
    out = [fit_device(k, [prob] + [fill] * n, lbfgs_iterations=25, log_domain=True)[0] for n in (0, 8, 20, 60, 400)]
    k.close()
    for w, f, st, ev in out[1:]:
        assert np.array_equal(w, out[0][0]) and np.array_equal(f, out[0][1])
        assert np.array_equal(st, out[0][2]) and np.array_equal(ev, out[0][3])
