"""GPU: evaluate_both on grids whose workspace has an odd size.

The FP64 staging of evaluate_both lies behind the workspace in one allocation;
with an odd number of pixels the workspace ends off an 8-byte boundary, so these
cases check that the staging is aligned (against the FP64 oracle)."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,P,precision,log", [(31, 27, 1, "fp32", False), (31, 27, 3, "fp64", False),
                                                 (31, 27, 3, "fp64", True), (15, 9, 1, "fp32", True)])
def test_evaluate_on_odd_grids(oracle, W, H, P, precision, log):
    from wassersteindictionarylearning_b200 import (CudaGaussian2DKernel, CudaLogSignArrayGaussian2DKernel,
                                                    Problem, WassersteinRegression)
    from wassersteindictionarylearning_b200.synthetic import make_problem, to_variables
    K, L, gamma = 3, 5, 2.0
    cfg, obs, atoms, w = make_problem(None, seed=2, P=P, W=W, H=H, K=K, L=L, gamma=gamma, loss=2)
    x = to_variables(w, atoms, cfg["scale_dic"])
    k = (CudaLogSignArrayGaussian2DKernel if log else CudaGaussian2DKernel)(gamma, W, H, precision=precision)
    reg = WassersteinRegression(Problem(np.ones((K, W * H)), obs, k, None, P), L, 2, cfg["scale_dic"])
    f, g = reg.evaluate_both(x)
    f_ref, g_ref = oracle.evaluate_both(W, H, 1, gamma, P, K, L, 2, cfg["scale_dic"], x, obs, log_domain=log)
    tol = 1e-10 if precision == "fp64" else 1e-5
    assert abs(f - f_ref) <= tol * abs(f_ref)
    assert rel(g[P * K:], g_ref[P * K:]) < tol
    k.close()
