"""The calls whose time matters to a user of this framework, through its public
entry points: the separable operator, dictionary learning's objective
(evaluate_both) in every arithmetic and both domains, the projection and
barycenter requests of a serving loop, many uneven problems in one launch, and
weight fits in the log domain.  Sizes are those of the repository's named
workloads, tests and bench, plus odd ones of the same ranges.
"""
import ctypes
import math
import random

import numpy as np
import torch

from wassersteindictionarylearning_b200 import (CudaGaussian2DKernel, CudaGaussian3DKernel,
                                                CudaLogSignArrayGaussian2DKernel, Problem,
                                                WassersteinBarycenter)
from wassersteindictionarylearning_b200._lib import check, dptr, lib
from wassersteindictionarylearning_b200.batch import batch_run, fit_device

TV, QUADRATIC, KL = 1, 2, 4


def listed():
    return [
        # one step of a host program that drives the KernelType operator itself
        # on a handful of small device images: latency and launches
        dict(name="conv64_fp32", kind="conv", W=64, H=64, D=1, n=4, gamma=2.0, precision="fp32"),
        # the operator on a stack of odd-sized volumes in the reference's arithmetic
        dict(name="conv3d_odd_fp64", kind="conv", W=45, H=51, D=38, n=6, gamma=2.0, precision="fp64"),
        # plain 2-D dictionary learning, one objective evaluation (16 histograms on 64x64)
        dict(name="dict64_fp32", kind="evaluate", domain="kernel", W=64, H=64, D=1, P=16, K=4, L=25,
             gamma=2.0, loss=QUADRATIC, precision="fp32"),
        # the batched workload's plain FP32 form (64 histograms on 128x128)
        dict(name="batched128_fp32", kind="evaluate", domain="kernel", W=128, H=128, D=1, P=64, K=5,
             L=100, gamma=1.0, loss=KL, precision="fp32"),
        # the same on the tensor cores: the bench's headline
        dict(name="batched128_split", kind="evaluate", domain="kernel", W=128, H=128, D=1, P=64, K=5,
             L=100, gamma=1.0, loss=KL, precision="split_bf16"),
        # the grid of the reference's bundled images, above the fused kernel's tile
        dict(name="images272_split", kind="evaluate", domain="kernel", W=272, H=240, D=1, P=8, K=4,
             L=50, gamma=25.0, loss=QUADRATIC, precision="split_bf16"),
        # small regularisation, log domain, 256x256
        dict(name="log256_fp32", kind="evaluate", domain="log", W=256, H=256, D=1, P=16, K=8, L=100,
             gamma=0.5, loss=QUADRATIC, precision="fp32"),
        # a small odd-sized log-domain evaluation in the reference's arithmetic
        dict(name="log_odd_fp64", kind="evaluate", domain="log", W=61, H=84, D=1, P=2, K=3, L=20,
             gamma=1.0, loss=TV, precision="fp64"),
        # one evaluation of one served projection request (weights only, host
        # buffers); these dictionaries need FP64
        dict(name="serve_project161_fp64", kind="project", W=161, H=161, D=1, P=1, K=5, L=50, gamma=2.0,
             loss=QUADRATIC, precision="fp64"),
        # one served barycenter request on a volume
        dict(name="serve_bary48c_fp64", kind="barycenter", W=48, H=48, D=48, P=1, K=5, L=50, gamma=2.0,
             precision="fp64"),
        # many uneven independent problems in one launch
        dict(name="batch_uneven_split", kind="batch", count=24, mix=3, gamma=2.0, precision="split_bf16"),
        # weight fits onto fixed blob dictionaries, log domain, L-BFGS on the device
        dict(name="fit_uneven_log_fp32", kind="fit", count=12, mix=5, gamma=2.0, iterations=4,
             precision="fp32"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["conv", "conv", "evaluate", "evaluate", "evaluate", "evaluate", "log", "log", "project",
                       "project", "barycenter", "barycenter", "batch", "fit"])
    if kind == "conv":
        precision = rng.choice(["fp32", "fp64", "split_bf16"])
        if rng.random() < 0.3:
            W, H, D = (_log_int(rng, 24, 64) for _ in range(3))
        else:
            W, H, D = _log_int(rng, 32, 300), _log_int(rng, 32, 300), 1
        return dict(kind=kind, W=W, H=H, D=D, n=_log_int(rng, 1, 64), gamma=rng.choice([1.0, 2.0, 4.0, 25.0]),
                    precision=precision)
    if kind in ("evaluate", "log"):
        precision = rng.choice(["fp32", "fp32", "split_bf16", "fp64"] if kind == "evaluate" else
                               ["fp32", "fp32", "fp64"])
        big = 288 if kind == "evaluate" and precision != "fp64" else 256
        W = _log_int(rng, 40, big)
        H = W if rng.random() < 0.4 else _log_int(rng, 40, big)
        # rows of any length, but a number of them that keeps P * K * W * H a multiple of 4
        # (P * W * H of 2), the only sizes whose FP64 staging evaluate_both aligns
        H += -H % 4
        K, L, P = rng.randint(2, 8), _log_int(rng, 10, 100), _log_int(rng, 1, 64)
        most = {("evaluate", "fp32"): 2.5e8, ("evaluate", "fp64"): 1.5e8, ("evaluate", "split_bf16"): 3e8,
                ("log", "fp32"): 4e8, ("log", "fp64"): 2e7}[kind, precision]
        P = max(1, min(P, int(most / (K * L * W * H))))
        if kind == "evaluate":
            gamma = 25.0 if W > 200 else rng.choice([1.0, 2.0, 4.0])
        else:
            gamma = rng.choice([0.5, 1.0, 2.0])
        loss = rng.choice([TV, QUADRATIC, KL] if precision == "fp64" else [QUADRATIC, KL])
        return dict(kind="evaluate", domain="kernel" if kind == "evaluate" else "log", W=W, H=H, D=1, P=P,
                    K=K, L=L, gamma=gamma, loss=loss, precision=precision)
    if kind in ("project", "barycenter"):
        if rng.random() < 0.25:
            W = H = D = rng.randint(36, 56)
        else:
            W, D = rng.randint(64, 256), 1
            H = W
        c = dict(kind=kind, W=W, H=H, D=D, P=rng.randint(1, 4), K=rng.randint(3, 6), L=rng.randint(30, 60),
                 gamma=2.0, precision="fp64")
        if kind == "project":
            c["loss"] = rng.choice([QUADRATIC, KL])
        return c
    if kind == "batch":
        return dict(kind=kind, count=_log_int(rng, 4, 32), mix=rng.randint(0, 999),
                    gamma=rng.choice([1.0, 2.0, 4.0]), precision="split_bf16")
    return dict(kind=kind, count=_log_int(rng, 4, 12), mix=rng.randint(0, 999), gamma=rng.choice([1.0, 2.0]),
                iterations=rng.randint(2, 4), precision="fp32")


# ---------------------------------------------------------------- inputs ----------------
def _blobs(gen, n, W, H, D, blobs, std, floor=1e-6):
    """n histograms (n, D*H*W): mixtures of anisotropic Gaussian blobs, a floor, sum 1."""
    dev, f64 = gen.device, torch.float64
    dims = 3 if D > 1 else 2
    side = torch.tensor([W, H, D][:dims], dtype=f64, device=dev)
    axes = [torch.arange(s, dtype=f64, device=dev) + 0.5 for s in ([W, H, D][:dims])]
    grid = torch.stack(torch.meshgrid(*axes[::-1], indexing="ij")[::-1], dim=-1).reshape(-1, dims)
    out = torch.zeros(n, grid.shape[0], dtype=f64, device=dev)
    uni = lambda *s: torch.rand(*s, generator=gen, dtype=f64, device=dev)  # noqa: E731
    count = torch.randint(blobs[0], blobs[1] + 1, (n, 1), generator=gen, device=dev)
    mix = -torch.log(uni(n, blobs[1]) + 1e-12) * (torch.arange(blobs[1], device=dev) < count)
    mix = mix / mix.sum(1, keepdim=True)
    for b in range(blobs[1]):
        centre = (0.2 + 0.6 * uni(n, dims)) * side
        s = (std[0] + (std[1] - std[0]) * uni(n, dims)) * side
        q, r = torch.linalg.qr(torch.randn(n, dims, dims, generator=gen, dtype=f64, device=dev))
        q = q * torch.sign(torch.diagonal(r, dim1=1, dim2=2))[:, None, :]
        for i in range(n):
            z = ((grid - centre[i]) @ q[i]) / s[i]
            out[i] += mix[i, b] / s[i].prod() * torch.exp(-0.5 * (z * z).sum(-1))
    out = out / (2 * math.pi) ** (dims / 2) + floor
    return out / out.sum(1, keepdim=True)


def _init_atoms(gen, K, N):
    """Atoms as dictionary learning starts them: uniform with a small perturbation."""
    a = 1.0 + 0.1 * torch.rand(K, N, generator=gen, dtype=torch.float64, device=gen.device)
    return a / a.sum(1, keepdim=True)


def _weights(gen, P, K):
    w = torch.rand(P, K, generator=gen, dtype=torch.float64, device=gen.device) + 1e-3
    return w / w.sum(1, keepdim=True)


def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + salt)
    return g


_STREAM = None


def _stream():
    """The one stream of a program that runs its device calls one after the other."""
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def _kernel(c, log=False):
    if log:
        return CudaLogSignArrayGaussian2DKernel(c["gamma"], c["W"], c["H"], precision=c["precision"])
    if c.get("D", 1) > 1:
        return CudaGaussian3DKernel(c["gamma"], c["W"], c["H"], c["D"], precision=c["precision"])
    return CudaGaussian2DKernel(c["gamma"], c["W"], c["H"], precision=c["precision"])


def _shapes(c):
    """The uneven problems of a case: (side, K, L, P, mode), fixed by the case itself."""
    rng = random.Random(1000 * c["mix"] + c["count"])
    if c["kind"] == "batch":
        return [dict(W=rng.choice([32, 48, 61, 64, 96, 109, 128]), H=rng.choice([32, 48, 57, 64, 96, 128]),
                     K=rng.randint(3, 8), L=rng.randint(10, 40), P=rng.randint(1, 4), loss_type=rng.choice([2, 4]),
                     mode=rng.choice(["both", "weights", "barycenter"])) for _ in range(c["count"])]
    out = []
    for _ in range(c["count"]):
        side = rng.choice([32, 48, 64, 96])
        out.append(dict(W=side, H=side, K=rng.randint(3, 8), L=rng.randint(25, 50), P=1, loss_type=2))
    return out


def _histograms(c, gen, P, W, H, D):
    sharp = c.get("domain") == "log"
    return _blobs(gen, P, W, H, D, (1, 3) if sharp else (2, 5), (0.01, 0.04) if sharp else (0.03, 0.12))


def _data(c, seed):
    """The inputs of a case as FP64 tensors on the GPU."""
    gen = _gen(seed)
    W, H, D = c["W"], c["H"], c.get("D", 1)
    N = W * H * D
    if c["kind"] == "conv":  # scalings as the iteration holds them: positive, over a few orders of magnitude
        return dict(u=torch.exp(1.5 * torch.randn(c["n"], N, generator=gen, dtype=torch.float64, device="cuda")))
    P, K = c["P"], c["K"]
    if c["kind"] == "evaluate":
        scale = N / P / 100.0
        atoms, w = _init_atoms(gen, K, N), _weights(gen, P, K)
        return dict(x=torch.cat([torch.log(w).reshape(-1) * scale, torch.log(atoms).reshape(-1)]), scale=scale,
                    observed=_histograms(c, gen, P, W, H, D))
    # a served request: a resident dictionary of blobs
    return dict(atoms=_blobs(gen, K, W, H, D, (1, 3), (0.03, 0.12)), weights=_weights(gen, P, K),
                observed=_blobs(gen, P, W, H, D, (1, 3), (0.03, 0.12)))


def prepare(case, seed):
    c = dict(case)
    s = dict(case=c)
    if c["kind"] in ("batch", "fit"):
        gen = _gen(seed)
        probs = []
        for q in _shapes(c):
            N = q["W"] * q["H"]
            if c["kind"] == "batch":
                atoms = _init_atoms(gen, q["K"], N)
            else:
                atoms = _blobs(gen, q["K"], q["W"], q["H"], 1, (1, 3), (0.03, 0.12))
            p = dict(q, atoms=atoms.cpu().numpy().reshape(-1), weights=_weights(gen, q["P"], q["K"]).cpu().numpy(),
                     observed=_blobs(gen, q["P"], q["W"], q["H"], 1, (1, 3), (0.03, 0.12)).cpu().numpy().reshape(-1))
            probs.append(p)
        side = 128 if c["kind"] == "batch" else max(q["W"] for q in probs)
        s["kernel"] = _kernel(dict(c, W=side, H=side), log=c["kind"] == "fit")
        s["problems"] = probs
        return s
    s["kernel"] = _kernel(c, log=c.get("domain") == "log")
    d = _data(c, seed)
    out64 = lambda n: torch.empty(n, dtype=torch.float64, device="cuda")  # noqa: E731
    if c["kind"] == "conv":
        s["u"], s["out"] = d["u"], torch.empty_like(d["u"])
    elif c["kind"] == "evaluate":
        s.update(d)
        s["g"], s["f"] = out64(d["x"].numel()), out64(1)
    else:  # the serving loop's requests are host buffers
        s.update({k: np.ascontiguousarray(v.cpu().numpy().reshape(-1)) for k, v in d.items()})
        if c["kind"] == "project":
            s["la"], s["loss"] = np.empty(c["P"] * c["K"]), np.empty(c["P"])
        else:
            prob = Problem(s["atoms"], s["observed"], s["kernel"])
            s["bary"] = WassersteinBarycenter(prob, c["L"])
    torch.cuda.synchronize()
    return s


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    c, kern = s["case"], s["kernel"]
    kind, wide = c["kind"], c["precision"] == "fp64"
    if kind == "conv":
        st = _stream()
        check(lib().wdl_convolve_device(kern.ctx, _ptr(s["u"]), _ptr(s["out"]), c["n"],
                                        ctypes.c_void_p(st.cuda_stream)), kern.ctx)
        with torch.cuda.stream(st):  # a program in FP32 keeps its results in FP32
            return s["out"] if wide else s["out"].float()
    if kind == "evaluate":
        st = _stream()
        check(lib().wdl_evaluate_both_device(kern.ctx, c["P"], c["K"], c["L"], c["loss"], s["scale"], _ptr(s["x"]),
                                             _ptr(s["g"]), s["g"].numel(), _ptr(s["observed"]), _ptr(s["f"]), None,
                                             None, None, ctypes.c_void_p(st.cuda_stream)), kern.ctx)
        with torch.cuda.stream(st):
            return dict(g=s["g"], f=s["f"]) if wide else dict(g=s["g"].float(), f=s["f"].float())
    if kind == "project":
        check(lib().wdl_gradient_both(kern.ctx, c["P"], c["K"], c["L"], c["loss"], dptr(s["atoms"]),
                                      dptr(s["weights"]), dptr(s["observed"]), None, dptr(s["la"]), None, None,
                                      dptr(s["loss"]), None), kern.ctx)
        return dict(la=s["la"], loss=s["loss"])
    if kind == "barycenter":
        return s["bary"].compute_barycenter(s["weights"].reshape(c["P"], c["K"]))
    if kind == "batch":
        outs = batch_run(kern, s["problems"])
        # one array for each kind of result, problem after problem
        return {k: np.concatenate([o[k] for o in outs if k in o]).astype(np.float32)
                for k in ("la", "dic", "bary", "loss") if any(k in o for o in outs)}
    outs = fit_device(kern, s["problems"], lbfgs_iterations=c["iterations"], log_domain=True)
    return dict(weights=np.concatenate([o[0].reshape(-1) for o in outs]).astype(np.float32),
                loss=np.concatenate([o[1] for o in outs]).astype(np.float32))


# ---------------------------------------------------------------- cost ------------------
def _application(W, H, D, gamma, eps):
    """Flops of the separable Gaussian on one image: the taps above the arithmetic's rounding."""
    reach = math.ceil(math.sqrt(gamma * -math.log(eps)))
    taps = sum(min(n, 2 * reach + 1) for n in ([W, H, D] if D > 1 else [W, H]))
    return 2.0 * taps * W * H * D


def _evaluation(W, H, D, P, K, L, gamma, size, dic=True, back=True):
    """(bytes, flops) of one evaluation: inputs and outputs in FP64, and the iterate store
    (conv_b and phi of every iteration) written once and read once."""
    N = W * H * D
    eps = 2.0 ** -53 if size == 8 else 2.0 ** -24
    apps = 2 * L + ((2 * L - 1 if dic else 0) + 2 * (L - 1) if back else 0)
    flops = P * K * (apps * _application(W, H, D, gamma, eps) + 10.0 * N * L)
    bytes_ = 8.0 * (2 * (P * K + K * N) + P * N) + (4.0 * L * P * K * N * size if back else 0)
    return bytes_, flops


def work(case):
    c = case
    size = 8 if c["precision"] == "fp64" else 4
    if c["kind"] == "conv":
        N = c["W"] * c["H"] * c["D"]
        f = c["n"] * _application(c["W"], c["H"], c["D"], c["gamma"], 2.0 ** -53 if size == 8 else 2.0 ** -24)
        return dict(bytes=16.0 * c["n"] * N, flops=f)
    if c["kind"] in ("batch", "fit"):
        b = f = 0.0
        for q in _shapes(c):
            times = 1 if c["kind"] == "batch" else c["iterations"] + 1
            mode = q.get("mode", "weights")
            db, df = _evaluation(q["W"], q["H"], 1, q["P"], q["K"], q["L"], c["gamma"], size, mode == "both",
                                 mode != "barycenter")
            b, f = b + times * db, f + times * df
        return dict(bytes=b, flops=f)
    b, f = _evaluation(c["W"], c["H"], c["D"], c["P"], c["K"], c["L"], c["gamma"], size, c["kind"] == "evaluate",
                       c["kind"] != "barycenter")
    return dict(bytes=b, flops=f)


# ---------------------------------------------------------------- 64 bits ---------------
def _factors(W, H, D, gamma, floor):
    out = []
    for n in ([W, H, D] if D > 1 else [W, H]):
        i = torch.arange(n, dtype=torch.float64, device="cuda")
        out.append(torch.exp(-(i[:, None] - i[None, :]) ** 2 / gamma).clamp_min(floor))
    return out


def _conv(u, F):
    """Separable Gaussian of (..., [D,] H, W)."""
    u = torch.matmul(torch.matmul(F[1], u), F[0])
    if len(F) == 3:
        u = torch.tensordot(F[2], u, dims=([1], [u.dim() - 3])).movedim(0, -3)
    return u


def _forward(atoms, lam, F, L, keep):
    """Bregman projections of P histograms: barycenters and, with keep, the stored iterates."""
    b = torch.ones(lam.shape[:2] + atoms.shape[1:], dtype=torch.float64, device="cuda")
    w = lam.reshape(lam.shape[:2] + (1,) * (atoms.dim() - 1))
    tape = [b]
    for _ in range(L):
        cb = _conv(b, F)
        phi = _conv(atoms / cb, F)
        bary = torch.exp((w * torch.log(phi.clamp_min(1e-250))).sum(1))
        b = bary[:, None] / phi
        if keep:
            tape += [cb, phi, b]
    return bary, tape


def _gradient(atoms, lam, obs, F, L, loss):
    """(raw weight gradient, raw atom gradient summed over P, losses)."""
    bary, tape = _forward(atoms, lam, F, L, True)
    w = lam.reshape(lam.shape[:2] + (1,) * (atoms.dim() - 1))
    axes = tuple(range(1, bary.dim()))
    if loss == TV:
        f, n = 0.5 * (bary - obs).abs().sum(axes), torch.where(bary > obs, 0.5, -0.5).double()
    elif loss == QUADRATIC:
        f, n = ((bary - obs) ** 2).sum(axes), 2 * (bary - obs)
    else:
        lr = torch.log((bary / obs).clamp_min(1e-250))
        f, n = (bary * lr - bary + obs).sum(axes), lr
    gw = n * bary
    v = r = 0.0
    la, dic = torch.zeros_like(lam), torch.zeros_like(atoms)
    for s in range(L, 0, -1):
        cb, phi, b = tape[3 * s - 2:3 * s + 1]
        la += (torch.log(phi) * gw[:, None]).sum(tuple(range(2, phi.dim())))
        c = _conv((w * n[:, None] - v) * b, F)
        dic += (c / cb).sum(0)
        if s > 1:
            phi0, b0 = tape[3 * s - 4], tape[3 * s - 3]
            u = _conv((w * gw[:, None] - r) / phi, F)
            v = _conv(-atoms * c / (cb * cb), F) / phi0
            r = _conv(-atoms * u / (cb * cb), F) * b0
            n, gw = v.sum(1), r.sum(1)
    return la, dic, f


def exact(case, seed):
    c = dict(case)
    if c["kind"] == "fit":  # the path of an optimiser has no closed form
        return None
    if c["kind"] == "batch":
        return None
    W, H, D = c["W"], c["H"], c["D"]
    shape = (D, H, W) if D > 1 else (H, W)
    # the log domain's operator has no floor under its factor
    F = _factors(W, H, D, c["gamma"], 0.0 if c.get("domain") == "log" else 1e-250)
    d = _data(c, seed)
    if c["kind"] == "conv":
        return _conv(d["u"].reshape((c["n"],) + shape), F).reshape(c["n"], -1)
    P, K, L = c["P"], c["K"], c["L"]
    if c["kind"] == "evaluate":
        x, scale = d["x"], d["scale"]
        lam = torch.softmax(x[:P * K].reshape(P, K) / scale, 1)
        atoms = torch.softmax(x[P * K:].reshape(K, -1), 1)
    else:
        lam, atoms = d["weights"], d["atoms"]
    img = atoms.reshape((K,) + shape)
    if c["kind"] == "barycenter":
        bary, _ = _forward(img, lam, F, L, False)
        return bary.reshape(-1) if P == 1 else bary.reshape(P, -1)
    las, fs, dic = [], [], 0.0
    per = max(1, int(2e9 / (3 * L * K * atoms.shape[1])))  # histograms at a time: the iterates of all may be large
    for p in range(0, P, per):
        obs = d["observed"][p:p + per].reshape((-1,) + shape)
        la, g, f = _gradient(img, lam[p:p + per], obs, F, L, c["loss"])
        las.append(la)
        fs.append(f)
        dic = dic + g.reshape(K, -1)
    la, f = torch.cat(las), torch.cat(fs)
    if not bool(torch.isfinite(la).all() & torch.isfinite(dic).all()):
        return None  # outside the range of the direct form (the log domain's own range is wider)
    if c["kind"] == "project":
        return dict(la=la.reshape(-1), loss=f)
    gl = (la - (lam * la).sum(1, keepdim=True)) * lam / scale
    ga = (dic - (atoms * dic).sum(1, keepdim=True)) * atoms
    return dict(g=torch.cat([gl.reshape(-1), ga.reshape(-1)]), f=f.sum().reshape(1))
