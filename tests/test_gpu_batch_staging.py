"""GPU: many-problem calls around the sizes that decide how their arrays travel.

Arrays of 128 KB and more go up from the caller's memory, smaller ones through the
context's staging buffer, results come back through another; both are kept up to
32 MB.  One context runs small, boundary, large and again small calls: losses, weight
gradients and atom gradients of every problem against the FP64 oracle at the
split-BF16 targets."""
import numpy as np
import pytest

from conftest import rel, rel_scaled

pytestmark = pytest.mark.gpu

GAMMA = 4.0


def _problem(i, W, H, K, L, P, mode):
    from wassersteindictionarylearning_b200.synthetic import blob_histograms, init_atoms, init_weights
    return dict(W=W, H=H, K=K, L=L, P=P, mode=mode, loss_type=2, atoms=init_atoms(K, W * H, seed=i).reshape(-1),
                weights=init_weights(P, K, seed=i + 1).reshape(-1),
                observed=blob_histograms(P, W, H, seed=i + 2).reshape(-1))


def _check(oracle, probs, outs):
    for pr, o in zip(probs, outs):
        W, H, K, L, P = (pr[k] for k in ("W", "H", "K", "L", "P"))
        N = W * H
        atoms, w, obs = pr["atoms"].reshape(K, N), pr["weights"].reshape(P, K), pr["observed"].reshape(P, N)
        dic = np.zeros(K * N)
        for p in range(P):
            if pr["mode"] == "barycenter":
                ref = oracle.barycenter(W, H, 1, GAMMA, K, L, atoms, w[p])
                assert rel(o["bary"][p * N:(p + 1) * N], ref) < 1e-4
                continue
            la, d, bary = oracle.gradient_both(W, H, 1, GAMMA, K, L, 2, atoms, w[p], obs[p])
            scale = oracle.gradient_both_scale(W, H, 1, GAMMA, K, L, 2, atoms, w[p], obs[p])
            assert rel_scaled(o["la"][p * K:(p + 1) * K], la, scale) < 1e-3
            f, _ = oracle.loss(2, W, H, 1, GAMMA, bary, obs[p])
            assert abs(o["loss"][p] - f) <= 1e-4 * abs(f)
            dic += d
        if pr["mode"] == "both":
            assert rel(o["dic"], dic) < 1e-3


def test_calls_of_every_size_on_one_context(oracle):
    from wassersteindictionarylearning_b200 import CudaGaussian2DKernel
    from wassersteindictionarylearning_b200.batch import batch_run
    k = CudaGaussian2DKernel(GAMMA, 128, 128, precision="split_bf16")
    small = [_problem(1, 9, 7, 2, 3, 1, "both"), _problem(2, 16, 12, 3, 5, 2, "weights"),
             _problem(3, 8, 20, 2, 4, 1, "barycenter")]
    # 4 x 64 x 64 and 1 x 128 x 128 doubles are 128 KB
    line = [_problem(10, 64, 64, 4, 3, 1, "both"), _problem(11, 63, 65, 4, 4, 4, "both"),
            _problem(12, 128, 128, 1, 2, 1, "both"), _problem(13, 128, 127, 1, 2, 1, "weights"),
            _problem(14, 65, 64, 4, 2, 1, "barycenter"), _problem(15, 20, 10, 2, 6, 82, "weights")]
    large = [_problem(20, 128, 128, 5, 2, 1, "both"), _problem(21, 128, 128, 3, 3, 4, "both")]
    for probs in (small, line, large, small, line):
        _check(oracle, probs, batch_run(k, probs))
    many = [large[0]] * 64  # 42 MB of results: given back after the call
    outs = batch_run(k, many)
    _check(oracle, many[:1] * 3, [outs[0], outs[31], outs[63]])
    _check(oracle, small, batch_run(k, small))
    k.close()
