"""GPU: the banded CUDA-core operator and evaluation at the sizes their blocks
treat specially.

The operator sums only the taps that reach a line's rounding, in groups of eight
outputs, two FP32 lines at a time: lines of one to a few values, lengths around
multiples of 8 and 4, odd numbers of lines, factors wider than the zero padding
around a line, and inputs over many orders of magnitude, against the dense FP64
product.  With positive inputs every output is a sum of positive terms, so its
relative error is at most the number of roundings on its way (one per tap of each
axis, the conversion, the factor's own rounding) times the unit roundoff, plus
the part left out (2^-40 per axis in FP32, 2^-60 in FP64).  Values that are not
finite must end where the dense product puts them."""
import numpy as np
import pytest

from conftest import rel, rel_scaled

pytestmark = pytest.mark.gpu

EPS = {"fp32": 2.0 ** -24, "fp64": 2.0 ** -53}


def _factors(W, H, D, gamma):
    out = []
    for n in (W, H, D)[: 3 if D > 1 else 2]:
        i = np.arange(n, dtype=np.float64)
        out.append(np.maximum(1e-250, np.exp(-(i[:, None] - i[None, :]) ** 2 / gamma)))
    return out


def _dense(u, F, W, H, D):
    u = u.reshape(-1, D, H, W)
    u = np.einsum("ndhk,kw->ndhw", u, F[0])
    u = np.einsum("ndkw,kh->ndhw", u, F[1])
    if D > 1:
        u = np.einsum("nkhw,kd->ndhw", u, F[2])
    return u.reshape(-1)


def _kernel(W, H, D, gamma, precision):
    from wassersteindictionarylearning_b200 import CudaGaussian2DKernel, CudaGaussian3DKernel
    if D > 1:
        return CudaGaussian3DKernel(gamma, W, H, D, precision=precision)
    return CudaGaussian2DKernel(gamma, W, H, precision=precision)


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("W,H,D,n,gamma,spread", [
    (1, 7, 1, 2, 2.0, 1.0), (8, 1, 1, 1, 2.0, 1.0), (3, 17, 1, 3, 0.05, 1.0), (9, 8, 1, 2, 1.0, 8.0),
    (33, 31, 1, 2, 2.0, 15.0), (64, 65, 1, 1, 25.0, 1.0), (127, 36, 1, 2, 4.0, 8.0), (200, 23, 1, 1, 300.0, 8.0),
    (20, 12, 1, 1, 1e6, 1.0), (520, 40, 1, 1, 2.0, 15.0), (7, 10, 9, 2, 2.0, 8.0), (18, 5, 33, 1, 9.0, 1.0)])
def test_operator_edges(W, H, D, n, gamma, spread, precision):
    rng = np.random.default_rng(W * 1000 + H)
    u = np.exp(spread * rng.standard_normal(n * W * H * D))
    if precision == "fp32":
        u = u.astype(np.float32).astype(np.float64)
    k = _kernel(W, H, D, gamma, precision)
    out = k.convolve(u, n)
    k.close()
    ref = _dense(u, _factors(W, H, D, gamma), W, H, D)
    rounds = sum((W, H, D)[: 3 if D > 1 else 2]) + 8
    bound = rounds * EPS[precision] + 3 * (2.0 ** -40 if precision == "fp32" else 2.0 ** -60)
    # FP32's own range: results below its smallest normal number are rounded absolutely
    floor = 1e-36 if precision == "fp32" else 0.0
    assert np.all(np.abs(out - ref) <= bound * ref + floor), float(np.max(np.abs(out - ref) / ref))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_operator_with_zeros(precision):
    """Exact zeros (empty background) next to values, signed."""
    W, H = 70, 45
    rng = np.random.default_rng(5)
    u = np.where(rng.random(2 * W * H) < 0.9, 0.0, rng.standard_normal(2 * W * H))
    if precision == "fp32":
        u = u.astype(np.float32).astype(np.float64)
    k = _kernel(W, H, 1, 2.0, precision)
    out = k.convolve(u, 2)
    k.close()
    F = _factors(W, H, 1, 2.0)
    scale = _dense(np.abs(u), F, W, H, 1)
    bound = (W + H + 8) * EPS[precision] + 2.0 ** (-39 if precision == "fp32" else -59)
    # a zero keeps the whole FP32 band or FP64 line: results far from any value count too
    assert np.all(np.abs(out - _dense(u, F, W, H, 1)) <= bound * scale + (1e-36 if precision == "fp32" else 0.0))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_operator_not_finite(precision, value):
    """A value that is not finite meets the factor's zeros as in the dense product."""
    W, H = 90, 37
    rng = np.random.default_rng(6)
    u = rng.random((2, H, W)) + 0.5
    u[1, 11, 40] = value
    dt = np.float32 if precision == "fp32" else np.float64
    F = [f.astype(dt) for f in _factors(W, H, 1, 2.0)]
    k = _kernel(W, H, 1, 2.0, precision)
    out = k.convolve(u.reshape(-1), 2).reshape(2, H, W)
    k.close()
    with np.errstate(invalid="ignore"):
        t = np.stack([(F[0] * u[1, y].astype(dt)[:, None]).sum(0) for y in range(H)])
        ref = np.stack([(F[1] * t[:, x][:, None]).sum(0) for x in range(W)], axis=1)
    assert np.all(np.isfinite(out[0]))
    assert np.array_equal(np.isnan(out[1]), np.isnan(ref))
    assert np.array_equal(np.isposinf(out[1]), np.isposinf(ref))
    assert np.array_equal(np.isneginf(out[1]), np.isneginf(ref))


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
@pytest.mark.parametrize("W,H,D,P,K,L,gamma", [
    (13, 9, 1, 1, 1, 4, 2.0), (30, 21, 1, 2, 7, 5, 1.0), (24, 17, 1, 3, 8, 4, 4.0), (18, 20, 1, 2, 9, 4, 2.0),
    (40, 33, 1, 1, 11, 3, 30.0), (11, 13, 7, 2, 3, 4, 2.0)])
def test_evaluation_edges(oracle, W, H, D, P, K, L, gamma, precision):
    """Atom counts with and without a kernel of their own, odd rows and columns, a volume."""
    from wassersteindictionarylearning_b200 import Problem, WassersteinRegression
    from wassersteindictionarylearning_b200.synthetic import make_problem, to_variables
    cfg, obs, atoms, w = make_problem(None, seed=K, P=P, W=W, H=H, D=D, K=K, L=L, gamma=gamma, loss=2)
    x = to_variables(w, atoms, cfg["scale_dic"])
    k = _kernel(W, H, D, gamma, precision)
    reg = WassersteinRegression(Problem(np.ones((K, W * H * D)), obs, k, None, P), L, 2, cfg["scale_dic"])
    f, g = reg.evaluate_both(x)
    k.close()
    f_ref, g_ref = oracle.evaluate_both(W, H, D, gamma, P, K, L, 2, cfg["scale_dic"], x, obs)
    tol = 1e-10 if precision == "fp64" else 1e-5
    assert abs(f - f_ref) <= tol * abs(f_ref)
    assert rel(g[P * K:], g_ref[P * K:]) < tol
    scale = oracle.weight_gradient_scale(W, H, D, gamma, P, K, L, 2, cfg["scale_dic"], x, obs)
    assert rel_scaled(g[: P * K], g_ref[: P * K], scale) < tol


@pytest.mark.parametrize("precision", ["fp32", "fp64"])
def test_profile_counts_the_applications(precision):
    """wdl_conv_profile of an evaluation, in operator applications per atom and histogram:
    2 per iteration; in the reverse pass 2 per round and recursion, but 1 for the
    dictionary and none for the weights in the last round."""
    import ctypes as C
    from wassersteindictionarylearning_b200 import Problem, WassersteinRegression
    from wassersteindictionarylearning_b200._lib import lib
    from wassersteindictionarylearning_b200.synthetic import make_problem, to_variables
    P, K, L = 2, 3, 4
    cfg, obs, atoms, w = make_problem(None, seed=1, P=P, W=24, H=17, K=K, L=L, gamma=2.0, loss=2)
    k = _kernel(24, 17, 1, 2.0, precision)
    lib().wdl_set_profiling(k.ctx, 1)
    reg = WassersteinRegression(Problem(np.ones((K, 24 * 17)), obs, k, None, P), L, 2, cfg["scale_dic"])
    reg.evaluate_both(to_variables(w, atoms, cfg["scale_dic"]))
    ms, n, apps = C.c_double(), C.c_longlong(), C.c_double()
    lib().wdl_conv_profile(k.ctx, C.byref(ms), C.byref(n), C.byref(apps))
    k.close()
    assert ms.value > 0 and n.value > 0 and apps.value == (2 * L + (2 * L - 1) + 2 * (L - 1)) * P * K
