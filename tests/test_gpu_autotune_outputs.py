"""GPU: the autotuner's record tells the log-domain forms apart, and the forms agree on
operands that are not finite (a first call ends with the one-output form's result,
profiling keeps four outputs per thread)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_recorded_forms():
    from wassersteindictionarylearning_b200 import CudaGaussian3DKernel, CudaLogSignArrayGaussian2DKernel
    from wassersteindictionarylearning_b200._lib import check, lib
    seen = []
    # a few small FP64 images, where one output per thread is far ahead, and a stack that fills the GPU
    for W, H, n, precision in ((61, 84, 6, "fp64"), (96, 96, 300, "fp32")):
        k = CudaLogSignArrayGaussian2DKernel(1.0, W, H, precision=precision)
        k.log_convolve(np.log(np.random.default_rng(0).random(n * W * H) + 1e-3), n)
        key, choice, ms = (C.c_longlong * 6)(), C.c_int(), C.c_float()
        for i in range(lib().wdl_autotune_count(k.ctx)):
            check(lib().wdl_autotune_entry(k.ctx, i, key, C.byref(choice), C.byref(ms)), k.ctx)
            out = lib().wdl_autotune_outputs(k.ctx, i)
            assert out == 4 or (out == 1 and choice.value == 8)
            seen.append((n, out))
        assert lib().wdl_autotune_outputs(k.ctx, -1) < 0
        assert lib().wdl_autotune_outputs(k.ctx, lib().wdl_autotune_count(k.ctx)) < 0
        k.close()
    assert (6, 1) in seen and (300, 4) in seen and (300, 1) not in seen
    k = CudaGaussian3DKernel(2.0, 20, 18, 10, precision="split_bf16")
    k.convolve(np.ones(20 * 18 * 10), 1)
    assert lib().wdl_autotune_count(k.ctx) > 0
    assert all(lib().wdl_autotune_outputs(k.ctx, i) == 0 for i in range(lib().wdl_autotune_count(k.ctx)))
    k.close()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("W,H", [(1, 5), (9, 14), (37, 66)])
def test_forms_agree_on_values_that_are_not_finite(W, H, precision):
    from wassersteindictionarylearning_b200 import CudaLogSignArrayGaussian2DKernel
    from wassersteindictionarylearning_b200._lib import lib
    n = 5
    rng = np.random.default_rng(W)
    u = 20.0 * rng.standard_normal((n, W * H))
    u[0, rng.random(W * H) < 0.5] = -np.inf  # logarithms of exact zeros
    u[1] = -np.inf
    u[2, W * H // 2] = np.inf
    u[3, W * H // 3] = np.nan
    u[4, 0], u[4, -1] = np.inf, np.nan
    signs = rng.integers(0, 256, (n * W * H + 7) // 8).astype(np.uint8)
    outs = []
    for plain in (0, 1):
        k = CudaLogSignArrayGaussian2DKernel(0.7, W, H, precision=precision)
        lib().wdl_set_profiling(k.ctx, plain)
        sg = signs.copy()
        outs.append((k.log_convolve(u.reshape(-1), n), k.log_convolve_signArray(u.reshape(-1), sg, n), sg))
        k.close()
    for a, b in zip(*outs):
        assert np.array_equal(a, b, equal_nan=True)
