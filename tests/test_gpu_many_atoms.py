"""GPU: evaluations with more atoms than one banded block or one fused reverse step holds.

From 33 atoms on the reverse steps run as separate kernels (in the kernel and the log
domain), above 64 every CUDA-core evaluation does.  Grids of a few to a few hundred
pixels make the segments of their dot products smaller than a block, just as long
and longer; against the FP64 oracle at the parity tolerances."""
import numpy as np
import pytest

from conftest import rel, rel_scaled

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("log", [False, True])
@pytest.mark.parametrize("W,H,P,K", [(5, 3, 1, 33), (16, 13, 2, 65), (32, 32, 1, 40), (70, 40, 1, 65), (101, 61, 2, 33)])
def test_many_atoms(oracle, W, H, P, K, log, precision):
    from wassersteindictionarylearning_b200 import (CudaGaussian2DKernel, CudaLogSignArrayGaussian2DKernel, Problem,
                                                    WassersteinRegression)
    from wassersteindictionarylearning_b200.synthetic import make_problem, to_variables
    L, gamma = 3, 2.0
    cfg, obs, atoms, w = make_problem(None, seed=K, P=P, W=W, H=H, K=K, L=L, gamma=gamma, loss=2)
    x, sd, PK = to_variables(w, atoms, cfg["scale_dic"]), cfg["scale_dic"], P * K
    k = (CudaLogSignArrayGaussian2DKernel if log else CudaGaussian2DKernel)(gamma, W, H, precision=precision)
    reg = WassersteinRegression(Problem(np.ones((K, W * H)), obs, k, None, P), L, 2, sd)
    f, g = reg.evaluate_both(x)
    k.close()
    f_ref, g_ref = oracle.evaluate_both(W, H, 1, gamma, P, K, L, 2, sd, x, obs, log_domain=log)
    tol = 1e-10 if precision == "fp64" else 1e-5
    assert abs(f - f_ref) <= tol * abs(f_ref)
    assert rel(g[PK:], g_ref[PK:]) < tol
    scale = oracle.weight_gradient_scale(W, H, 1, gamma, P, K, L, 2, sd, x, obs)
    assert rel_scaled(g[:PK], g_ref[:PK], scale) < tol
