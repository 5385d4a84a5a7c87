"""Performance cases of the primal-dual TV / TGV^2 engine: what its users have it do, over the range they do it.

A case is a dict of plain values. ``prepare`` makes its inputs on the GPU and the handles a program keeps,
``run`` is one pass through the package's public entry points, ``exact`` is the same result in 64 bits by
plain torch, ``work`` the bytes and operations a pass cannot do without. Kinds of case:

  denoise   TvOptimizer / TgvOptimizer on a real or complex image
  mri       a with-operator solve (TGV-MRI, TGV, TV) with a Cartesian or the sampling operator
  radial    the same with the radial operator
  batch     many Cartesian solves of mixed shapes advanced together (BatchSolver)
  ops       one forward and one adjoint of a Cartesian operator on dense k-space
  rad_ops   one forward and one adjoint of a radial operator
  train     one training step of the warm-start network (loss, gradients, Adam update)
  predict   inference of the warm-start network
"""
import math
import os
import random
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "primal-dual-toolbox_gb300"))

import primaldualtoolbox as pdt  # noqa: E402
from primaldualtoolbox.warmstart import WarmStartNet  # noqa: E402

DEV = "cuda"
C64, C128, F32, F64 = torch.complex64, torch.complex128, torch.float32, torch.float64
BATCH_SIZES = [(192, 192), (256, 256), (320, 320), (640, 368)]


def listed():
    return [
        # a thumbnail or a patch: a few microseconds an iteration, latency and launches count
        dict(name="denoise_tv_64x48_it101", kind="denoise", opt="tv", dtype="f32", H=64, W=48, iters=101),
        # the denoising benchmark (ROF, lambda 10, 500 -> 501 iterations) and TGV on the same image
        dict(name="denoise_tv_512x512_it501", kind="denoise", opt="tv", dtype="f32", H=512, W=512, iters=501),
        dict(name="denoise_tgv_512x512_it501", kind="denoise", opt="tgv", dtype="f32", H=512, W=512, iters=501),
        # a large complex image whose state lives in HBM
        dict(name="denoise_tgv_4096x4096_c64_it21", kind="denoise", opt="tgv", dtype="c64", H=4096, W=4096, iters=21),
        # the benchmark reconstruction: 15 coils, readout oversampling removed, 4x random lines, 1001 iterations
        dict(name="mri_roos_15c_640x368_it1001", kind="mri", opt="tgv_mri", op="roos", C=15, H=640, W=368, accel=4.0,
             mask="random", iters=1001),
        # an odd, ragged matrix, the plain operator and the data weight Lambda
        dict(name="mri_8c_231x175_it101", kind="mri", opt="tgv_op", op="plain", C=8, H=231, W=175, accel=3.0,
             mask="regular", iters=101),
        # the single-coil sampling operator with a two-dimensional random mask
        dict(name="mri_sampling_256x256_it101", kind="mri", opt="tgv_mri", op="sampling", C=1, H=256, W=256, accel=3.0,
             mask="points", iters=101),
        # mixed reconstructions of one study solved together
        dict(name="batch_16_mixed_it41", kind="batch", problems=16, specs=3000, iters=41),
        # the radial slice: 256 x 256, 12 coils, 64 spokes x 512 samples, width 3 on a 1.5x grid
        dict(name="radial_12c_256_it201", kind="radial", opt="tgv_mri", C=12, N=256, spokes=64, osf=1.5, kw=3, iters=201),
        # single operator calls, as a user's own iteration makes them
        dict(name="ops_roos_15c_640x368", kind="ops", op="roos", C=15, H=640, W=368, accel=4.0, mask="random"),
        # the warm-start network: a training step on its configuration, and inference on the benchmark's image
        dict(name="train_4x320x320", kind="train", B=4, H=320, W=320),
        dict(name="predict_1x320x368", kind="predict", B=1, H=320, W=368),
    ]


def _log(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _matrix(rng, lo, hi):
    """An acquisition matrix size: between lo and hi, without a prime factor above 13."""
    n = _log(rng, lo, hi)
    while True:
        rest = n
        for p in (2, 3, 5, 7, 11, 13):
            while rest % p == 0:
                rest //= p
        if rest == 1:
            return n
        n -= 1


def draw(rng):
    kind = rng.choice(["denoise", "denoise", "denoise", "mri", "mri", "mri", "radial", "batch", "ops", "rad_ops", "train",
                       "predict"])
    if kind == "denoise":
        H, W = _log(rng, 33, 4096), _log(rng, 33, 4096)
        most = 131e6 * (1 if rng.random() < 0.5 else 0.25) / (H * W)  # pixel iterations up to the 512 x 512 case's
        return dict(kind=kind, opt=rng.choice(["tv", "tgv"]), dtype=rng.choice(["f32", "f32", "c64"]), H=H, W=W,
                    iters=max(8, min(501, int(most))))
    if kind in ("mri", "ops"):
        op = rng.choice(["roos", "plain", "plain", "sampling"]) if kind == "mri" else rng.choice(["roos", "plain"])
        C = 1 if op == "sampling" else _log(rng, 2, 24)
        H, W = _matrix(rng, 40, 640), _matrix(rng, 40, 384)
        if op == "roos":
            H = 2 * _matrix(rng, 20, 320)
        mask = "points" if op == "sampling" or rng.random() < 0.15 else rng.choice(["random", "regular"])
        d = dict(kind=kind, op=op, C=C, H=H, W=W, accel=round(rng.uniform(2, 8), 2), mask=mask)
        if kind == "mri":
            d.update(opt=rng.choice(["tgv_mri", "tgv_mri", "tgv_op", "tv_op"]),
                     iters=max(11, min(_log(rng, 21, 201), int(2e8 / (C * H * W)))))
        return d
    if kind in ("radial", "rad_ops"):
        N = 8 * _matrix(rng, 6, 32)
        d = dict(kind=kind, C=_log(rng, 1, 12), N=N, spokes=rng.randint(16, 64), osf=rng.choice([1.25, 1.5, 2.0]),
                 kw=rng.choice([3, 3, 4, 5]))
        if kind == "radial":
            d.update(opt=rng.choice(["tgv_mri", "tv_op"]), iters=_log(rng, 21, 81))
        return d
    if kind == "batch":
        return dict(kind=kind, problems=rng.randint(2, 12), specs=rng.randint(0, 1 << 20), iters=_log(rng, 11, 41))
    B = rng.randint(1, 4)
    return dict(kind=kind, B=B, H=_log(rng, 48, 368), W=_log(rng, 48, 368))


# -----------------------------------------------------------------------------------------------------
# Inputs
# -----------------------------------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _grid(H, W):
    y = (torch.arange(H, device=DEV, dtype=F32) - (H - 1) / 2) / max(1.0, H / 2)
    x = (torch.arange(W, device=DEV, dtype=F32) - (W - 1) / 2) / max(1.0, W / 2)
    return torch.meshgrid(y, x, indexing="ij")


def _shapes(seed, H, W, n=20):
    """A piecewise constant image of n random ellipses and rectangles, intensities U(0, 1)."""
    r = random.Random(int(seed))
    Y, X = _grid(H, W)
    img = torch.zeros(H, W, device=DEV)
    for _ in range(n):
        cy, cx, ry, rx = r.uniform(-1, 1), r.uniform(-1, 1), r.uniform(0.06, 0.5), r.uniform(0.06, 0.5)
        val, th, ellipse = r.uniform(0, 1), r.uniform(0, math.pi), r.random() < 0.5
        dy, dx = Y - cy, X - cx
        a, b = (dx * math.cos(th) + dy * math.sin(th)) / rx, (dy * math.cos(th) - dx * math.sin(th)) / ry
        img[(a * a + b * b <= 1) if ellipse else (torch.maximum(a.abs(), b.abs()) <= 1)] = val
    return img


def _phantom(seed, H, W):
    """A piecewise constant complex image inside an oval, with a smooth random phase."""
    r = random.Random(int(seed) + 7)
    Y, X = _grid(H, W)
    mag = torch.where((X / 0.72) ** 2 + (Y / 0.92) ** 2 <= 1, 0.2 + _shapes(seed, H, W, 10), torch.zeros_like(X))
    phase = sum(r.uniform(-1, 1) * (X / 1.5) ** i * (Y / 1.5) ** j for i in range(3) for j in range(3 - i))
    return torch.polar(mag, math.pi * phase)


def _coils(seed, C, H, W):
    """Gaussian blobs on a ring with random linear phase, normalised to sum |c|^2 = 1."""
    r = random.Random(int(seed) + 13)
    Y, X = _grid(H, W)
    out = torch.empty(C, H, W, dtype=C64, device=DEV)
    for c in range(C):
        a = 2 * math.pi * c / C + r.uniform(-0.1, 0.1)
        mag = torch.exp(-((X - 0.55 * math.cos(a)) ** 2 + (Y - 0.55 * math.sin(a)) ** 2) / (2 * 0.45 ** 2))
        out[c] = torch.polar(mag, r.uniform(0, 2 * math.pi) + r.uniform(-1, 1) * X + r.uniform(-1, 1) * Y)
    return out / torch.linalg.vector_norm(out, dim=0, keepdim=True)


def _noise(g, *shape):
    return torch.randn(*shape, generator=g, dtype=C64, device=DEV)


def _mask(kind, seed, H, W, accel):
    """Phase-encode lines (28 central ones, the others random or regular) or random points; float32 (H, W)."""
    r = random.Random(int(seed) + 29)
    m = torch.zeros(H, W, device=DEV)
    mid = min(28, max(2, W // 8))
    lines = set(range(W // 2 - mid // 2, W // 2 - mid // 2 + mid))
    total = max(mid, round(W / accel))
    if kind == "regular":
        lines |= set(range(0, W, int(accel)))
    elif kind == "random":
        lines |= set(r.sample(sorted(set(range(W)) - lines), total - len(lines)))
    else:
        g = _gen(seed + 31)
        m[torch.rand(H, W, generator=g, device=DEV) < 1 / accel] = 1
        m[H // 2 - min(8, H // 4):H // 2 + min(8, H // 4), W // 2 - min(8, W // 4):W // 2 + min(8, W // 4)] = 1
        return m
    m[:, sorted(lines)] = 1
    return m


def _y0(H):
    return int(np.float32(H) * np.float32(0.25) + np.float32(1))


def _fwd(u, sens, mask, op):
    """mask . fftshift(fft2(ifftshift(pad(u) . sens))) / sqrt(W H), the operators' shift conventions."""
    H, W = mask.shape
    if op == "roos":
        full = torch.zeros(H, W, dtype=u.dtype, device=DEV)
        full[_y0(H):_y0(H) + H // 2] = u
        u = full
    x = u[None] if sens is None else u[None] * sens
    k = torch.fft.fft2(torch.roll(x, ((H + 1) // 2, (W + 1) // 2), (-2, -1)), norm="ortho")
    return torch.roll(k, (H // 2, W // 2), (-2, -1)) * mask


def _adj(k, sens, mask, op):
    H, W = mask.shape
    x = torch.fft.ifft2(torch.roll(k * mask, ((H + 1) // 2, (W + 1) // 2), (-2, -1)), norm="ortho")
    x = torch.roll(x, (H // 2, W // 2), (-2, -1))
    x = x[0] if sens is None else (x * sens.conj()).sum(0)
    return x[_y0(H):_y0(H) + H // 2] if op == "roos" else x


def _mri_data(case, seed):
    """Coil maps, mask, noisy k-space of a phantom (noise 1e-3 of the largest value) and alpha1."""
    H, W, op = case["H"], case["W"], case["op"]
    shape_seed = 1000 * H + 10 * W + case["C"]  # the sampled lines belong to the protocol, the data to the seed
    mask = _mask(case["mask"], shape_seed, H, W, case["accel"])
    sens = None if op == "sampling" else _coils(seed, case["C"], H, W)
    truth = _phantom(seed, H // 2 if op == "roos" else H, W)
    k = _fwd(truth, sens, mask, op)
    k = (k + mask * 1e-3 * k.abs().max() * _noise(_gen(seed), *k.shape)).to(C64)
    if op == "sampling":
        k = k[0].contiguous()
    return dict(sens=sens, mask=mask, f=k.contiguous(), alpha1=0.05 * float(truth.abs().max()))


def _specs(case):
    r = random.Random(case["specs"])
    out = []
    for i in range(case["problems"]):
        H, W = BATCH_SIZES[r.randrange(len(BATCH_SIZES))]
        out.append(dict(kind="mri", opt="tgv_mri", op="plain", C=r.randint(8, 32), H=H, W=W, accel=float(r.randint(2, 8)),
                        mask=r.choice(["random", "regular"]), iters=case["iters"]))
    return out


def _trajectory(case):
    """(2, Ns) golden-angle trajectory, rows [imag k, real k], and density weights sqrt|k|."""
    ang = np.arange(case["spokes"]) * np.pi * (np.sqrt(5) - 1) / 2
    r = (np.arange(2 * case["N"]) - case["N"]) / (2 * case["N"])
    k = (r[:, None] * np.exp(1j * ang[None, :])).ravel()
    return np.array([k.imag, k.real]).astype(np.float32), np.sqrt(np.abs(k)).astype(np.float32)[None, :]


def _radial_data(case, seed):
    """Coil maps and noisy radial samples of a phantom (the exact non-uniform transform, weighted)."""
    N, C = case["N"], case["C"]
    traj, dcf = _trajectory(case)
    sens = _coils(seed, C, N, N)
    img = _phantom(seed, N, N)[None] * sens
    t = torch.from_numpy(traj).to(DEV, F64)
    x = torch.arange(N, device=DEV, dtype=F64) - N // 2
    ex = torch.polar(torch.ones((), device=DEV, dtype=F64), -2 * math.pi * t[0][:, None] * x).to(C64)  # (Ns, x)
    ey = torch.polar(torch.ones((), device=DEV, dtype=F64), -2 * math.pi * t[1][:, None] * x).to(C64)  # (Ns, y)
    f = torch.stack([((ey @ img[c]) * ex).sum(1) for c in range(C)]) * (torch.from_numpy(dcf).to(DEV) / N)
    f = f + 0.01 * f.abs().max() * _noise(_gen(seed), C, f.shape[1])
    return dict(traj=traj, dcf=dcf, sens=sens, f=f.to(C64).contiguous(), alpha1=0.02)


def _image(case, seed):
    H, W = case["H"], case["W"]
    if case["dtype"] == "f32":
        return _shapes(seed, H, W) + 0.1 * torch.randn(H, W, generator=_gen(seed), device=DEV)
    return _phantom(seed, H, W) + 0.1 * _noise(_gen(seed), H, W)


LAYERS = [(2, 32)] + [(32, 32)] * 6 + [(32, 8)]  # input and output channels; weights are stored [tap][out][in]


def _params(seed):
    """Network weights of an ordinary size: residual branches small, biases near zero."""
    r = np.random.default_rng(int(seed) + 5)
    out = []
    for n, (ci, co) in enumerate(LAYERS):
        gain = (1.0, 0.25, 0.1)[(n > 0) + (n == 7)]
        w = gain * math.sqrt(2 / (9 * ci)) * r.standard_normal((9, co, ci))
        if n == 7:
            w[:, 6:] = 0  # two padding channels
        out += [w.ravel(), 0.01 * r.standard_normal(co) * (np.arange(co) < 6 if n == 7 else 1)]
    return np.concatenate(out).astype(np.float32)


def _net_data(case, seed):
    B, H, W = case["B"], case["H"], case["W"]
    clean = torch.stack([_phantom(seed + 101 * b, H, W) for b in range(B)])
    g = _gen(seed)
    k = torch.fft.fft2(clean, norm="ortho") * (torch.rand(1, 1, W, generator=g, device=DEV) < 0.4)
    u0 = torch.fft.ifft2(k, norm="ortho") + 0.01 * _noise(g, B, H, W)
    vt = torch.stack([torch.roll(clean, -1, d) - clean for d in (2, 1)], 1) * 0.5
    return u0.to(C64).contiguous(), clean.contiguous(), vt.contiguous()


# -----------------------------------------------------------------------------------------------------
# Handles and passes
# -----------------------------------------------------------------------------------------------------
def _set(prm, case, alpha1):
    prm.max_iter = case["iters"] - 1
    if case["opt"] == "tgv_mri":
        prm.reduction = 0.01
    else:
        prm.Lambda = 2.0
    if case["opt"] != "tv_op":
        prm.alpha1, prm.alpha0 = alpha1, 2 * alpha1


def _cart_op(case, d):
    op = {"roos": pdt.mri.MriCartesianRemoveROOSOperator, "plain": pdt.mri.MriCartesianOperator,
          "sampling": pdt.mri.MriSamplingOperator}[case["op"]]()
    if d["sens"] is not None:
        op.setCoilSens(d["sens"])
    op.setMask(d["mask"])
    return op


def _solver(case, op, alpha1):
    m = pdt.mri
    if case.get("op") in ("roos", "plain"):
        cls = {"tgv_mri": m.TgvMriOptimizer_2c3c, "tgv_op": m.TgvOptimizer_2c3c, "tv_op": m.TvOptimizerWithOp_2c3c}
    else:
        cls = {"tgv_mri": m.TgvMriOptimizer_2c2c, "tgv_op": m.TgvOptimizer_2c2c, "tv_op": m.TvOptimizer_2c2c}
    opt = cls[case["opt"]]()
    _set(opt.getParameters(), case, alpha1)
    opt.setOperator(op)
    return opt


def _radial_op(case, d):
    op = pdt.mri.MriRadialOperator({"osf": case["osf"], "sector_width": 8, "kernel_width": case["kw"], "img_dim": case["N"]})
    op.setTrajectory(d["traj"])
    op.setDcf(d["dcf"])
    op.setCoilSens(d["sens"])
    return op


def _image_shape(case):
    if "N" in case:
        return case["N"], case["N"]
    return (case["H"] // 2 if case.get("op") == "roos" else case["H"]), case["W"]


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind == "denoise":
        f = _image(case, seed)
        d, dt = pdt.denoising, case["dtype"]
        opt = {"tvf32": d.TvOptimizer_2f, "tvc64": d.TvOptimizer_2c, "tgvf32": d.TgvOptimizer_2f,
               "tgvc64": d.TgvOptimizer_2c}[case["opt"] + dt]()
        p = opt.getParameters()
        p.Lambda, p.max_iter = 10.0, case["iters"] - 1
        if case["opt"] == "tgv":
            p.alpha0, p.alpha1 = 2.0, 1.0
        s.update(opt=opt, f=f, u=torch.empty_like(f), stream=torch.cuda.Stream())
    elif kind in ("mri", "radial"):
        d = _mri_data(case, seed) if kind == "mri" else _radial_data(case, seed)
        op = _cart_op(case, d) if kind == "mri" else _radial_op(case, d)
        u0 = torch.empty(_image_shape(case), dtype=C64, device=DEV)
        op.adjoint(d["f"], out=u0)  # lays out the operator's plan, as a program does that keeps it
        s.update(op=op, opt=_solver(case, op, d["alpha1"]), f=d["f"], u0=u0, u=torch.empty_like(u0),
                 stream=torch.cuda.Stream())
    elif kind == "batch":
        s.update(items=[], stream=torch.cuda.Stream())
        for i, spec in enumerate(_specs(case)):
            d = _mri_data(spec, seed + 17 * i)
            op = _cart_op(spec, d)
            u0 = torch.empty(_image_shape(spec), dtype=C64, device=DEV)
            op.adjoint(d["f"], out=u0)
            s["items"].append((op, _solver(spec, op, d["alpha1"]), d["f"], u0, torch.empty_like(u0)))
        s["batch"] = pdt.batch.BatchSolver([it[1] for it in s["items"]])
    elif kind in ("ops", "rad_ops"):
        d = _mri_data(case, seed) if kind == "ops" else _radial_data(case, seed)
        op = _cart_op(case, d) if kind == "ops" else _radial_op(case, d)
        u = _phantom(seed + 1, *_image_shape(case))
        s.update(op=op, x=u.contiguous(), f=d["f"], k=torch.empty_like(d["f"]), u=torch.empty_like(u),
                 stream=torch.cuda.Stream())
        op.adjoint(s["f"], out=s["u"])
    else:
        net = WarmStartNet(seed=0)
        net.set_params(_params(seed))
        u0, ut, vt = _net_data(case, seed)
        s.update(net=net, u0=u0, ut=ut, vt=vt, u=torch.empty_like(u0), v=torch.empty_like(vt), stream=torch.cuda.Stream())
    torch.cuda.synchronize()  # the streams that run() uses start after the inputs are there
    return s


def _start_solve(op, opt, f, u0, st):
    """A fresh solve from the zero-filled image, as a program makes it slice by slice."""
    opt.setNoisyData(f, stream=st)
    op.adjoint(f, out=u0, stream=st)
    if hasattr(opt, "setInput0"):
        opt.setInput0(u0, stream=st)
    else:
        opt.setInput0UV(u0, stream=st)


def run(s):
    kind, st = s["case"]["kind"], s["stream"]
    if kind == "denoise":
        s["opt"].setNoisyData(s["f"], stream=st)
        s["opt"].setInput0UV(s["f"], stream=st)
        s["opt"].solve(stream=st)
        return s["opt"].getResult(out=s["u"], stream=st)
    if kind in ("mri", "radial"):
        _start_solve(s["op"], s["opt"], s["f"], s["u0"], st)
        s["opt"].solve(stream=st)
        return s["opt"].getResult(out=s["u"], stream=st)
    if kind == "batch":
        for op, opt, f, u0, _ in s["items"]:
            _start_solve(op, opt, f, u0, st)
        s["batch"].solve(stream=st)
        return [opt.getResult(out=u, stream=st) for _, opt, _, _, u in s["items"]]
    if kind in ("ops", "rad_ops"):
        s["op"].forward(s["x"], out=s["k"], stream=st)
        s["op"].adjoint(s["f"], out=s["u"], stream=st)
        return [s["k"], s["u"]]
    if kind == "train":
        loss = s["net"].train_step(s["u0"], s["ut"], s["vt"], lr=1e-5, stream=st)
        return [loss, s["net"].grads()]
    s["net"].predict(s["u0"], s["u"], s["v"], stream=st)
    return [s["u"], s["v"]]


# -----------------------------------------------------------------------------------------------------
# The bytes and operations of a pass
# -----------------------------------------------------------------------------------------------------
def _fft(n):
    return 5.0 * n * math.log2(max(2, n))


def _mri_work(c):
    H, W = c["H"], c["W"]
    Hi, C, pix = _image_shape(c)[0], c["C"], 8.0
    points = c["mask"] == "points"
    mid = min(28, max(2, W // 8))
    ns = W if points else max(mid, round(W / c["accel"])) if c["mask"] == "random" else min(W, mid + -(-W // int(c["accel"])))
    share = 1 / c["accel"] if points else ns / W
    sens = 0 if c["op"] == "sampling" else C * Hi * W * pix
    # an operator and its adjoint: transforms along both axes for a mask of points, along the lines alone
    # where whole lines are sampled; the coil products
    one = C * (2 * Hi * _fft(W) + (2 * ns * _fft(H) if points else 0) + 16.0 * Hi * W)
    return sens, share * C * H * W * pix, one, ns


def work(case):
    kind = case["kind"]
    if kind == "denoise":
        n, k = case["H"] * case["W"], 1 if case["dtype"] == "f32" else 2
        return {"bytes": 2.0 * n * 4 * k, "flops": case["iters"] * n * k * (22.0 if case["opt"] == "tv" else 65.0)}
    if kind == "mri":
        sens, data, one, _ = _mri_work(case)
        n = math.prod(_image_shape(case))
        side = 130.0 if case["opt"] != "tv_op" else 44.0
        return {"bytes": sens + data + 4.0 * case["H"] * case["W"] + 8.0 * n, "flops": case["iters"] * (one + side * n)}
    if kind == "batch":
        w = [work(c) for c in _specs(case)]
        return {k: sum(x[k] for x in w) for k in ("bytes", "flops")}
    if kind == "ops":
        sens, data, _, ns = _mri_work(case)
        Hi, W = _image_shape(case)
        dense = 8.0 * case["C"] * case["H"] * W
        return {"bytes": sens + data + dense + 4.0 * case["H"] * W + 16.0 * Hi * W,
                "flops": 2 * case["C"] * (Hi * _fft(W) + ns * _fft(case["H"]) + 8.0 * Hi * W)}
    if kind in ("radial", "rad_ops"):
        N, C = case["N"], case["C"]
        G, Ns = math.ceil(case["osf"] * N), 2 * N * case["spokes"]
        one = C * (2 * (N + G) * _fft(G) + 8.0 * case["kw"] ** 2 * Ns + 24.0 * N * N)
        bytes_ = 8.0 * C * N * N + 12.0 * Ns + 8.0 * C * Ns * (2 if kind == "rad_ops" else 1) + 16.0 * N * N
        return {"bytes": bytes_, "flops": one if kind == "rad_ops" else case["iters"] * (one + 130.0 * N * N)}
    n = case["B"] * case["H"] * case["W"]
    macs = 9.0 * sum(a * b for a, b in LAYERS)
    if kind == "predict":
        return {"bytes": n * 8.0 * 4, "flops": 2 * n * macs}
    return {"bytes": n * 8.0 * 4 + 4.0 * 58000 * 8, "flops": 6 * n * macs}


# -----------------------------------------------------------------------------------------------------
# The same results in 64 bits
# -----------------------------------------------------------------------------------------------------
def _d(x, dim):
    """Forward difference, zero in the last row or column."""
    out = torch.zeros_like(x)
    n = x.shape[dim]
    out.narrow(dim, 0, n - 1).copy_(x.narrow(dim, 1, n - 1) - x.narrow(dim, 0, n - 1))
    return out


def _dt(x, dim):
    """Minus its adjoint (the divergence of one component)."""
    n = x.shape[dim]
    out = x.clone()
    out.narrow(dim, n - 1, 1).zero_()
    out.narrow(dim, 1, n - 1).sub_(x.narrow(dim, 0, n - 1))
    return out


def _proj(n2, alpha):
    return 1 / torch.clamp(torch.sqrt(n2) / alpha, min=1)


def _abs2(x):
    return x.real ** 2 + x.imag ** 2 if x.is_complex() else x * x


def _dual(p, q, ub, vb, sigma, a0, a1, tgv):
    a = [p[0] + sigma * (_d(ub, 1) - (vb[0] if tgv else 0)), p[1] + sigma * (_d(ub, 0) - (vb[1] if tgv else 0))]
    s = _proj(_abs2(a[0]) + _abs2(a[1]), a1)
    p = [a[0] * s, a[1] * s]
    if tgv:
        e = [q[0] + sigma * _d(vb[0], 1), q[1] + sigma * _d(vb[1], 0),
             q[2] + sigma * 0.5 * (_d(vb[0], 0) + _d(vb[1], 1))]
        s = _proj(_abs2(e[0]) + _abs2(e[1]) + 2 * _abs2(e[2]), a0)
        q = [x * s for x in e]
    return p, q


def _vstep(v, p, q, tau):
    vn = [v[0] + tau * (_dt(q[0], 1) + _dt(q[2], 0) + p[0]), v[1] + tau * (_dt(q[1], 0) + _dt(q[2], 1) + p[1])]
    return vn, [2 * vn[0] - v[0], 2 * vn[1] - v[1]]


def _zeros(u, n):
    return [torch.zeros_like(u) for _ in range(n)]


def _denoise64(f, opt, iters, lam=10.0, a0=2.0, a1=1.0):
    tgv = opt == "tgv"
    tau = sigma = 1 / math.sqrt(12.0 if tgv else 8.0)
    u = ub = f
    p, q, v = _zeros(f, 2), _zeros(f, 3), _zeros(f, 2)
    vb = v
    for _ in range(iters):
        if not tgv:
            p, q = _dual(p, q, ub, vb, sigma, a0, 1.0, False)
        un = (u + tau * (_dt(p[0], 1) + _dt(p[1], 0) + lam * f)) / (1 + tau * lam)
        u, ub = un, 2 * un - u
        if tgv:
            v, vb = _vstep(v, p, q, tau)
            p, q = _dual(p, q, ub, vb, sigma, a0, a1, True)
    return u


def _solve64(case, f, fwd, adj, alpha1):
    opt, K = case["opt"], case["iters"] - 1
    tgv, tau, sigma = opt != "tv_op", 1 / 16 if opt == "tgv_mri" else 1 / 8, 1 / 8
    lam, red = (1.0, 0.01) if opt == "tgv_mri" else (2.0, 1.0)
    u = ub = adj(f)
    r = torch.zeros_like(f)
    p, q, v = _zeros(u, 2), _zeros(u, 3), _zeros(u, 2)
    vb = v
    for k in range(K + 1):
        a1 = alpha1 * red ** (k / K) if tgv else 1.0
        p, q = _dual(p, q, ub, vb, sigma, 2 * a1, a1, tgv)
        r = (r + sigma * (fwd(ub) - f)) / (1 + sigma * lam)
        un = u + tau * (_dt(p[0], 1) + _dt(p[1], 0) - adj(r))
        u, ub = un, 2 * un - u
        if tgv:
            v, vb = _vstep(v, p, q, tau)
    return u


def _cart64(case, d):
    sens, mask = None if d["sens"] is None else d["sens"].to(C128), d["mask"].to(F64)
    f = d["f"].to(C128)
    f = f[None] if sens is None else f
    return f, lambda u: _fwd(u, sens, mask, case["op"]), lambda k: _adj(k, sens, mask, case["op"])


def _radial64(case, d):
    """Kaiser-Bessel gridding on the oversampled grid (beta of Beatty et al. 2005), taps and transforms in 64 bits."""
    N, C, kw, osf = case["N"], case["C"], case["kw"], case["osf"]
    G = math.ceil(osf * N - 1e-9)
    G += G & 1
    beta = math.pi * math.sqrt(max((kw / osf * (osf - 0.5)) ** 2 - 0.8, 1e-12))
    t = torch.from_numpy(d["traj"]).to(DEV, F64) * G
    g0 = torch.ceil(t - kw / 2)
    taps = g0[..., None] + torch.arange(kw, device=DEV)
    z = 2 * (taps - t[..., None]) / kw
    wt = torch.where(z.abs() <= 1, torch.special.i0(beta * torch.sqrt(torch.clamp(1 - z * z, min=0))), torch.zeros_like(z))
    g = torch.remainder(taps, G).long()
    cells = (g[1][:, :, None] * G + g[0][:, None, :]).reshape(t.shape[1], -1)  # row ky, column kx
    w = (wt[1][:, :, None] * wt[0][:, None, :]).reshape(t.shape[1], -1)
    m = (torch.arange(N, device=DEV, dtype=F64) - N // 2) * math.pi * kw / G
    s2 = beta * beta - m * m
    s1 = torch.sqrt(s2.abs())
    deap = kw * torch.where(s2 > 0, torch.sinh(s1), torch.sin(s1)) / s1
    dcf, sens = torch.from_numpy(d["dcf"]).to(DEV, F64), d["sens"].to(C128)
    scale = sens / (N * deap[:, None] * deap[None, :])
    at = torch.remainder(torch.arange(N, device=DEV) - N // 2, G)

    def fwd(u):
        grid = torch.zeros(C, G, G, dtype=C128, device=DEV)
        grid[:, at[:, None], at[None, :]] = u * scale
        F = torch.fft.fft2(grid).reshape(C, -1)
        return (F[:, cells.reshape(-1)].reshape(C, *cells.shape) * w).sum(-1) * dcf

    def adj(k):
        grid = torch.zeros(C, G * G, dtype=C128, device=DEV)
        grid.index_add_(1, cells.reshape(-1), ((k * dcf)[..., None] * w).reshape(C, -1))
        x = torch.fft.ifft2(grid.reshape(C, G, G), norm="forward")
        return (x[:, at[:, None], at[None, :]] * scale.conj()).sum(0)

    return d["f"].to(C128), fwd, adj


def _net64(params, x):
    o, h = 0, x
    for n, (ci, co) in enumerate(LAYERS):
        w = params[o:o + 9 * co * ci].reshape(3, 3, co, ci).permute(2, 3, 0, 1)
        o += 9 * co * ci
        z = torch.nn.functional.conv2d(h, w, params[o:o + co], padding=1)
        o += co
        h = torch.relu(z) if n == 0 else h + torch.relu(z) if n < 7 else z
    return h


def exact(case, seed):
    kind = case["kind"]
    if kind == "denoise":
        f = _image(case, seed)
        return _denoise64(f.to(F64 if case["dtype"] == "f32" else C128), case["opt"], case["iters"])
    if kind in ("mri", "radial"):
        d = _mri_data(case, seed) if kind == "mri" else _radial_data(case, seed)
        return _solve64(case, *(_cart64(case, d) if kind == "mri" else _radial64(case, d)), d["alpha1"])
    if kind == "batch":
        out = []
        for i, c in enumerate(_specs(case)):
            d = _mri_data(c, seed + 17 * i)
            out.append(_solve64(c, *_cart64(c, d), d["alpha1"]))
        return out
    if kind in ("ops", "rad_ops"):
        d = _mri_data(case, seed) if kind == "ops" else _radial_data(case, seed)
        f, fwd, adj = _cart64(case, d) if kind == "ops" else _radial64(case, d)
        return [fwd(_phantom(seed + 1, *_image_shape(case)).to(C128)), adj(f)]
    u0, ut, vt = (x.to(C128) for x in _net_data(case, seed))
    s = u0.abs().amax((1, 2))[:, None, None, None]
    params = torch.from_numpy(_params(seed)).to(DEV, F64).requires_grad_(kind == "train")
    o = _net64(params, torch.stack([u0.real, u0.imag], 1) / s)
    if kind == "predict":
        c = torch.complex(o[:, 0:6:2], o[:, 1:6:2]) * s
        return [u0 + c[:, 0], c[:, 1:]]
    target = torch.cat([(ut - u0)[:, None], vt], 1) / s
    diff = o[:, :6] - torch.view_as_real(target).permute(0, 1, 4, 2, 3).flatten(1, 2)
    loss = (diff * diff).sum() / (u0.numel())
    loss.backward()
    return [float(loss.detach()), params.grad]
