"""GPU: evaluations of tensor-core contexts above one tile, on both sides of the line
between the FP32 band sums and the tensor-core axis passes.

The axis passes leave an autotuner entry per pass shape, the band sums none, which
tells the routes apart.  Wide factors (sums of more than 72 taps on lines above 48)
take the axis passes, in evaluate_both and in barycenters; results at the
tensor-core targets of the operator (split BF16: barycenter and loss 1e-4, gradients
1e-3; TF32: 3e-3 and 2e-2), on the band sums at FP32's 1e-5."""
import numpy as np
import pytest

from conftest import rel, rel_scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D,gamma,axes", [
    (200, 152, 1, 25.0, False), (200, 152, 1, 40.0, True), (200, 152, 1, 300.0, True), (136, 131, 1, 400.0, True),
    (24, 20, 16, 400.0, False), (48, 40, 33, 100.0, False), (56, 40, 33, 100.0, True), (20, 64, 18, 25.0, False)])
@pytest.mark.parametrize("precision", ["split_bf16", "tf32"])
def test_evaluation_on_both_routes(oracle, W, H, D, gamma, axes, precision):
    from wassersteindictionarylearning_b200 import (CudaGaussian2DKernel, CudaGaussian3DKernel, Problem,
                                                    WassersteinBarycenter, WassersteinRegression)
    from wassersteindictionarylearning_b200._lib import lib
    from wassersteindictionarylearning_b200.synthetic import make_problem, to_variables
    P, K, L, loss = 2, 3, 4, 2
    cfg, obs, atoms, w = make_problem(None, seed=4, P=P, W=W, H=H, D=D, K=K, L=L, gamma=gamma, loss=loss)
    x, sd, PK = to_variables(w, atoms, cfg["scale_dic"]), cfg["scale_dic"], P * K
    f_ref, g_ref, bary_ref = oracle.evaluate_both(W, H, D, gamma, P, K, L, loss, sd, x, obs, want_bary=True)
    scale = oracle.weight_gradient_scale(W, H, D, gamma, P, K, L, loss, sd, x, obs)
    k = (CudaGaussian3DKernel(gamma, W, H, D, precision=precision) if D > 1 else
         CudaGaussian2DKernel(gamma, W, H, precision=precision))
    prob = Problem(np.ones((K, W * H * D)), obs, k, None, P)
    reg = WassersteinRegression(prob, L, loss, sd)
    f, g = reg.evaluate_both(x)
    assert (lib().wdl_autotune_count(k.ctx) > 0) == axes
    t_bary, t_grad = (1e-5, 1e-5) if not axes else (1e-4, 1e-3) if precision == "split_bf16" else (3e-3, 2e-2)
    assert rel(reg.last_barycenters, bary_ref) < t_bary
    assert abs(f - f_ref) <= t_bary * abs(f_ref)
    assert rel(g[PK:], g_ref[PK:]) < t_grad
    assert rel_scaled(g[:PK], g_ref[:PK], scale) < t_grad
    k.close()
    # barycenters alone, from the normalised atoms and weights
    k = (CudaGaussian3DKernel(gamma, W, H, D, precision=precision) if D > 1 else
         CudaGaussian2DKernel(gamma, W, H, precision=precision))
    ref = oracle.barycenter(W, H, D, gamma, K, L, np.asarray(atoms).reshape(K, -1), np.asarray(w).reshape(P, K)[0])
    bary = WassersteinBarycenter(Problem(np.asarray(atoms).reshape(K, -1), obs, k), L).compute_barycenter(
        np.asarray(w).reshape(P, K)[0])
    assert rel(bary, ref) < t_bary
    assert (lib().wdl_autotune_count(k.ctx) > 0) == axes
    k.close()
