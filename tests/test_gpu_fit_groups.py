"""GPU: log-domain weight fits on clusters of every size.

wdl_fit_weights_log gives a problem more CTAs when few problems share the GPU.
The elementwise steps and log-sum-exp passes do not depend on the split; only the
FP64 dot products' order of summation does, so one evaluation's loss and the
weights after one accepted step agree to FP64 summation rounding (taken as 1e-9,
far above N * 2^-53 for these grids), alone and among many."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,K", [(5, 3, 1), (17, 16, 2), (32, 31, 3), (33, 47, 2), (64, 65, 4), (100, 129, 2)])
def test_fit_alone_and_among_many(W, H, K):
    from wassersteindictionarylearning_b200 import CudaLogSignArrayGaussian2DKernel
    from wassersteindictionarylearning_b200.batch import fit_device
    from wassersteindictionarylearning_b200.synthetic import blob_histograms
    side = max(W, H)
    prob = dict(W=W, H=H, K=K, L=4, loss_type=2, atoms=blob_histograms(K, W, H, seed=1).reshape(-1),
                observed=blob_histograms(1, W, H, seed=2).reshape(-1))
    filler = dict(prob, W=16, H=16, observed=blob_histograms(1, 16, 16, seed=3).reshape(-1),
                  atoms=blob_histograms(K, 16, 16, seed=4).reshape(-1))
    k = CudaLogSignArrayGaussian2DKernel(2.0, max(side, 16), max(side, 16), precision="fp32")
    out = []
    for n in (0, 20, 400):  # fillers: the problem's group shrinks from 16 CTAs to its class's least
        (w, f, st, ev) = fit_device(k, [prob] + [filler] * n, lbfgs_iterations=1, log_domain=True)[0]
        out.append((w[0], f[0], st[0], ev[0]))
    k.close()
    for w, f, st, ev in out[1:]:
        assert (st, ev) == out[0][2:]
        assert abs(f - out[0][1]) <= 1e-9 * abs(out[0][1])
        assert np.max(np.abs(w - out[0][0])) <= 1e-9
