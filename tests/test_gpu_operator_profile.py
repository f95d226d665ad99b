"""GPU: wdl_conv_profile counts the operator's own calls, one application per image."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", ["fp32", "fp64", "split_bf16"])
@pytest.mark.parametrize("W,H,D", [(24, 17, 1), (12, 10, 9)])
def test_operator_calls_are_counted(W, H, D, precision):
    from wassersteindictionarylearning_b200 import CudaGaussian2DKernel, CudaGaussian3DKernel
    from wassersteindictionarylearning_b200._lib import lib
    n = 5
    u = np.random.default_rng(0).random(n * W * H * D)
    k = (CudaGaussian3DKernel(2.0, W, H, D, precision=precision) if D > 1 else
         CudaGaussian2DKernel(2.0, W, H, precision=precision))
    lib().wdl_set_profiling(k.ctx, 1)
    ms, calls, images = C.c_double(), C.c_longlong(), C.c_double()
    for i in (1, 2):
        k.convolve(u, n)
        lib().wdl_conv_profile(k.ctx, C.byref(ms), C.byref(calls), C.byref(images))
        assert ms.value > 0 and calls.value == i and images.value == i * n
    k.close()
