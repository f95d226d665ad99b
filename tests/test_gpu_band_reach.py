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


@pytest.mark.parametrize("W,H,gamma", [(200, 24, 0.5), (200, 24, 25.0), (133, 61, 4.0), (24, 90, 2.0)])
@pytest.mark.parametrize("values", [(np.inf,), (np.inf, -np.inf), (np.nan,), (np.inf, np.nan, np.inf)])
def test_not_finite_meets_the_zeros(W, H, gamma, values):
    """Infinite within the reach of an infinity (NaN where two of other signs meet), NaN
    where a zero of the factor meets it, the neighbouring lines untouched."""
    rng = np.random.default_rng(W + len(values))
    u = (rng.random((2, H, W)) + 0.5).astype(np.float32)
    for i, v in enumerate(values):  # rows on their own and together, first and last columns among them
        u[1, (7 * i) % 14, (0, W // 2 - 1, W - 1)[i]] = v
    F = [f.astype(np.float32) for f in _factors(W, H, 1, gamma)]
    k = _kernel(W, H, 1, gamma, "fp32")
    out = k.convolve(u.astype(np.float64).reshape(-1), 2).reshape(2, H, W)
    k.close()
    with np.errstate(invalid="ignore"):
        t = np.stack([(F[0] * u[1, y][:, None]).sum(0) for y in range(H)])
        ref = np.stack([(F[1] * t[:, x][:, None]).sum(0) for x in range(W)], axis=1)
    assert np.allclose(out[0], _dense(u[0].astype(np.float64), F, W, H, 1).reshape(H, W), rtol=1e-5, atol=0)
    assert np.array_equal(np.isnan(out[1]), np.isnan(ref))
    assert np.array_equal(np.isposinf(out[1]), np.isposinf(ref))
    assert np.array_equal(np.isneginf(out[1]), np.isneginf(ref))
    ok = np.isfinite(ref)
    assert np.allclose(out[1][ok], ref[ok], rtol=1e-5, atol=0)
