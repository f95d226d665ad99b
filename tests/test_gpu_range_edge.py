"""GPU: the iteration at which a kernel-domain scaling first leaves the FP32 range.

On these dictionaries phi passes the largest FP32 number while a, conv_b and every
earlier phi are still finite, so at one iteration count (23 or 24 of the counts
below) phi = inf is the only sign of the overflow.  A histogram then comes back
NaN in its barycenter and loss; before that iteration both are near the FP64
result.  The bound on a finite result: a pass sums some 20 positive terms, so four
passes of at most 26 iterations add at most 26 * 4 * 20 * 2^-24 = 1.2e-4 to a
pixel's relative error, and subnormal b (of pixels that hardly count beside
others) some more: 1e-3, where a saturated phi costs 6e-3 or more."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,gamma,seed", [(64, 4.0, 5), (32, 2.0, 6)])
@pytest.mark.parametrize("L", range(20, 27))
def test_first_overflow_is_reported(W, gamma, seed, L):
    from wassersteindictionarylearning_b200 import CudaGaussian2DKernel
    from wassersteindictionarylearning_b200._lib import check, dptr, lib
    from wassersteindictionarylearning_b200.synthetic import blob_histograms
    K, P, N = 5, 2, W * W
    atoms = np.ascontiguousarray(blob_histograms(K, W, W, 1, n_blobs=(1, 3), seed=seed))
    obs = np.ascontiguousarray(blob_histograms(P, W, W, 1, n_blobs=(1, 3), seed=101))
    w = np.full((P, K), 1.0 / K)
    out = {}
    for prec in ("fp32", "fp64"):
        k = CudaGaussian2DKernel(gamma, W, W, precision=prec)
        bary = np.empty(P * N)
        check(lib().wdl_barycenter(k.ctx, P, K, L, dptr(atoms), dptr(w), dptr(bary)), k.ctx)
        la, bary2, loss = np.empty(P * K), np.empty(P * N), np.empty(P)
        check(lib().wdl_gradient_both(k.ctx, P, K, L, 2, dptr(atoms), dptr(w), dptr(obs), None, dptr(la),
                                      None, dptr(bary2), dptr(loss), None), k.ctx)
        k.close()
        assert np.array_equal(bary, bary2, equal_nan=True)
        out[prec] = (bary.reshape(P, N), loss, la.reshape(P, K))
    bary, loss, la = out["fp32"]
    ref, loss_ref, _ = out["fp64"]
    assert np.all(np.isfinite(ref))
    for p in range(P):
        if np.isnan(bary[p]).any():
            assert np.all(np.isnan(bary[p])) and np.isnan(loss[p]) and np.all(np.isnan(la[p]))
        else:
            assert np.max(np.abs(bary[p] - ref[p]) / ref[p]) < 1e-3
            slack = 2 * np.sum(np.abs(ref[p] - obs.reshape(P, N)[p]) * 1e-3 * ref[p]) + np.sum((1e-3 * ref[p]) ** 2)
            assert abs(loss[p] - loss_ref[p]) < slack
    assert np.isnan(bary).any() == (L >= {64: 23, 32: 24}[W])
