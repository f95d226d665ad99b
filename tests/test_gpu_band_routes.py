"""GPU: CUDA-core evaluations on both sides of each line between the fused banded
kernels and separate kernels around the operator.

The fused kernels issue about half the launches, which tells the routes apart (an
iteration: 2 against 4 or more, on volumes 4 against 8).  Loss, gradients and barycenters
against the FP64 oracle at the parity tolerances on both."""
import numpy as np
import pytest

from conftest import rel, rel_scaled

pytestmark = pytest.mark.gpu

# (W, H, D, K, gamma, fused for FP32, for FP64)
CASES = [(16, 16, 1, 3, 2.0, False, True), (8, 16, 1, 4, 2.0, False, True), (8, 16, 1, 5, 2.0, False, False),
         (17, 16, 1, 9, 2.0, False, True), (31, 33, 1, 3, 2.0, False, True),
         (32, 32, 1, 3, 2.0, True, True), (32, 32, 1, 32, 2.0, True, True), (64, 20, 1, 24, 2.0, True, True),
         (64, 20, 1, 25, 2.0, False, False), (64, 20, 1, 12, 50.0, True, True), (64, 20, 1, 13, 50.0, True, False),
         (64, 20, 1, 16, 50.0, True, False), (64, 20, 1, 17, 50.0, False, False), (65, 4, 1, 25, 2.0, True, True),
         (128, 5, 1, 24, 2.0, False, False), (128, 5, 1, 16, 2.0, True, True), (100, 9, 1, 33, 2.0, False, False),
         (8, 8, 8, 2, 2.0, False, False), (16, 9, 8, 4, 2.0, False, True), (16, 16, 16, 3, 2.0, False, True),
         (17, 16, 16, 3, 2.0, True, True), (40, 11, 10, 16, 2.0, True, True), (40, 11, 10, 17, 2.0, False, False),
         (40, 33, 7, 12, 60.0, True, True), (40, 33, 7, 13, 60.0, False, False), (32, 13, 11, 20, 60.0, True, True),
         (32, 13, 11, 21, 60.0, True, False), (32, 13, 11, 25, 60.0, False, False)]


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("W,H,D,K,gamma,f32,f64", CASES)
def test_evaluation_on_both_routes(oracle, W, H, D, K, gamma, f32, f64, precision):
    from wassersteindictionarylearning_b200 import (CudaGaussian2DKernel, CudaGaussian3DKernel, Problem,
                                                    WassersteinRegression)
    from wassersteindictionarylearning_b200._lib import lib
    from wassersteindictionarylearning_b200.synthetic import make_problem, to_variables
    P, L, loss = 2, 4, 2
    cfg, obs, atoms, w = make_problem(None, seed=K, P=P, W=W, H=H, D=D, K=K, L=L, gamma=gamma, loss=loss)
    x, sd, PK = to_variables(w, atoms, cfg["scale_dic"]), cfg["scale_dic"], P * K
    k = (CudaGaussian3DKernel(gamma, W, H, D, precision=precision) if D > 1 else
         CudaGaussian2DKernel(gamma, W, H, precision=precision))
    reg = WassersteinRegression(Problem(np.ones((K, W * H * D)), obs, k, None, P), L, loss, sd)
    f, g = reg.evaluate_both(x)
    launches = lib().wdl_launch_count(k.ctx)
    k.close()
    # banded: (2 L + 2 L) launches, (8 L) on volumes, and at most 16 around them; separate: at
    # least 4 L + 6 (L - 1), on volumes 6 more for each pair of applications
    assert (launches <= (8 if D > 1 else 4) * L + 16) == (f32 if precision == "fp32" else f64), launches
    f_ref, g_ref, bary_ref = oracle.evaluate_both(W, H, D, gamma, P, K, L, loss, sd, x, obs, want_bary=True)
    tol = 1e-10 if precision == "fp64" else 1e-5
    assert rel(reg.last_barycenters, bary_ref) < tol
    assert abs(f - f_ref) <= tol * abs(f_ref)
    assert rel(g[PK:], g_ref[PK:]) < tol
    scale = oracle.weight_gradient_scale(W, H, D, gamma, P, K, L, loss, sd, x, obs)
    assert rel_scaled(g[:PK], g_ref[:PK], scale) < tol
