"""GPU: FP32 band sums of narrow factors over data of a very wide spread.

At gamma 0.5 and 1 the FP32 factor ends 7 and 10 pixels from the centre; values
2^170 apart within a block would ask for more than that.  Against the dense
product with the FP32 factor, in FP64: positive terms, so the bound is the
roundings on an output's way (at most 2 * 21 taps, conversion and factor included)
and the part left out."""
import numpy as np
import pytest

from test_gpu_band import _dense, _factors, _kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D,n", [(128, 128, 1, 2), (129, 40, 1, 1), (40, 35, 33, 1)])
@pytest.mark.parametrize("gamma", [0.005, 0.5, 1.0, 2.0])
def test_wide_spread_on_narrow_factors(W, H, D, n, gamma):
    rng = np.random.default_rng(W)
    u = np.exp2(rng.uniform(-85.0, 85.0, n * W * H * D)).astype(np.float32).astype(np.float64)
    k = _kernel(W, H, D, gamma, "fp32")
    out = k.convolve(u, n)
    k.close()
    ref = _dense(u, [f.astype(np.float32).astype(np.float64) for f in _factors(W, H, D, gamma)], W, H, D)
    bound = 80 * 2.0 ** -24 + 3 * 2.0 ** -40
    assert np.all(np.abs(out - ref) <= bound * ref), float(np.max(np.abs(out - ref) / ref))
