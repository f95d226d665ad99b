"""GPU: banded launches whose line buffers end just under 48 KB of shared memory.

A launch gets 48 KB without asking for more, and the kernel's static arrays count
towards it: these sizes take between 47.4 and 48 KB for their lines.  The limit
belongs to a kernel for the rest of a process, so a size that needs more would
hide the smaller one's refusal: each list runs in a process of its own, and in it
each kernel (by type, atom count and pass) meets the size at the limit first."""
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, rel

pytestmark = pytest.mark.gpu

# (precision, W, H, K): bwd lines at the limit for FP64 K = 5, 9 and FP32 K = 6, 18; fwd ones
# for FP64 K = 33 and FP32 K = 17
LISTS = [[("fp64", 49, 12, 5), ("fp64", 64, 9, 9), ("fp32", 225, 7, 6), ("fp32", 64, 10, 18)],
         [("fp64", 65, 8, 33), ("fp32", 155, 6, 17)]]


def _run(cases):
    from oracle.oracle import OracleLib
    from wassersteindictionarylearning_b200 import CudaGaussian2DKernel, Problem, WassersteinRegression
    from wassersteindictionarylearning_b200.synthetic import make_problem, to_variables
    orc = OracleLib()
    for precision, W, H, K in cases:
        P, L, gamma = 2, 3, 2.0
        cfg, obs, atoms, w = make_problem(None, seed=K, P=P, W=W, H=H, K=K, L=L, gamma=gamma, loss=2)
        x = to_variables(w, atoms, cfg["scale_dic"])
        k = CudaGaussian2DKernel(gamma, W, H, precision=precision)
        reg = WassersteinRegression(Problem(np.ones((K, W * H)), obs, k, None, P), L, 2, cfg["scale_dic"])
        f, g = reg.evaluate_both(x)
        k.close()
        f_ref, g_ref = orc.evaluate_both(W, H, 1, gamma, P, K, L, 2, cfg["scale_dic"], x, obs)
        tol = 1e-10 if precision == "fp64" else 1e-5
        assert abs(f - f_ref) <= tol * abs(f_ref), (precision, W, H, K)
        assert rel(g[P * K:], g_ref[P * K:]) < tol, (precision, W, H, K)


@pytest.mark.parametrize("i", range(len(LISTS)))
def test_lines_just_under_the_default_limit(i):
    code = f"import sys; sys.path[:0] = [{ROOT!r}, {os.path.dirname(__file__)!r}]\n" \
           f"import test_gpu_smem_limit as t; t._run(t.LISTS[{i}])"
    r = subprocess.run([sys.executable, "-c", code], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
