"""GPU: the operator inside evaluations on grids around the line below which it runs as
dense passes.

The Wasserstein loss applies the operator on its own, 101 times; its value, gradients
and the barycenters against the FP64 oracle on both sides of each line (sizes, the
two types, volumes by their factor's width)."""
import numpy as np
import pytest

from conftest import rel, rel_scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("W,H,D,gamma", [
    (1, 9, 1, 2.0), (32, 32, 1, 2.0), (33, 32, 1, 2.0), (48, 48, 1, 40.0), (49, 48, 1, 40.0), (24, 64, 1, 9.0),
    (65, 24, 1, 9.0), (64, 50, 1, 40.0), (12, 10, 9, 4.0), (20, 17, 40, 2.0), (48, 7, 8, 60.0)])
def test_wasserstein_loss_around_the_line(oracle, W, H, D, gamma, precision):
    from wassersteindictionarylearning_b200 import (CudaGaussian2DKernel, CudaGaussian3DKernel, Problem,
                                                    WassersteinRegression)
    from wassersteindictionarylearning_b200.synthetic import init_atoms, init_weights, scale_dictionary, to_variables
    P, K, L, loss, N = 2, 3, 3, 3, W * H * D
    # observations near the barycenters' own values: the loss's scalings stay in FP32's range
    obs = init_atoms(P, N, seed=7)
    atoms, w, sd = init_atoms(K, N, seed=8), init_weights(P, K, seed=9), scale_dictionary(N, P)
    x, PK = to_variables(w, atoms, sd), P * K
    k = (CudaGaussian3DKernel(gamma, W, H, D, precision=precision) if D > 1 else
         CudaGaussian2DKernel(gamma, W, H, precision=precision))
    reg = WassersteinRegression(Problem(np.ones((K, N)), obs, k, None, P), L, loss, sd)
    f, g = reg.evaluate_both(x)
    k.close()
    f_ref, g_ref, bary_ref = oracle.evaluate_both(W, H, D, gamma, P, K, L, loss, sd, x, obs, want_bary=True)
    assert rel(reg.last_barycenters, bary_ref) < (1e-10 if precision == "fp64" else 1e-5)
    # gamma times logarithms of the loss's scalings, summed with masses of 1 and 1: a
    # scaling's relative error is at most 101 applications' roundings of some 40 terms
    # (FP64 has the summation order's 1e-10 to keep, as everywhere)
    assert abs(f - f_ref) <= P * gamma * (1e-10 if precision == "fp64" else 2 * 101 * 40 * 2.0 ** -24)
    if precision == "fp64":  # FP32's are differences of such logarithms
        assert rel(g[PK:], g_ref[PK:]) < 1e-9
        scale = oracle.weight_gradient_scale(W, H, D, gamma, P, K, L, loss, sd, x, obs)
        assert rel_scaled(g[:PK], g_ref[:PK], scale) < 1e-10
