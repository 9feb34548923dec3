"""The calls whose speed is tracked: single operators of the registration path
and whole registrations, from the smallest grids to the largest.

Every case goes through the package's public entry points on device tensors,
as a program that embeds the library does.  Inputs are random fields made from
the seed alone (nothing of this package computes them):

* ``_velocity``: band-limited velocities, Fourier modes 1 <= |k| <= 6 of
  amplitude 1/|k|^2 scaled to an RMS (the spectrum of the benchmark's recipe,
  whose RMS is 0.3; a solve starts from rest and grows towards it);
* ``_rough``: full-band fields with a power-law spectrum: images with edges
  (power 2), image forces and residuals (power 1), Krylov directions of noisy
  images (power 2: a force divided by the regularisation symbol);
* ``_images``: a template of smooth-edged regions in [0, 1] and the reference
  it becomes under a velocity, transported in float64.

Whole registrations use the seminorms: the counts and the velocity of a solve
with the full H1 / H2 norms follow single-precision roundoff, those with the
seminorms do not (they repeat to a few 1e-7 when a transform's rounding
changes).
"""
import math

import torch

import claire_b200 as cb

TWO_PI = 2.0 * math.pi


# ---------------------------------------------------------------------------
# cases
# ---------------------------------------------------------------------------
def _grid(n1, n2=None, n3=None):
    return {"n1": n1, "n2": n2 or n1, "n3": n3 or n1}


def listed():
    brain = _grid(128, 150, 128)  # the grid of the example brain images
    return [
        # one image warped by a given map on the smallest grid in production
        # use: a call of a few microseconds, bound by latency and launches
        {"name": "warp_64", "kind": "interp", "dof": 1, "rms": 0.3, "nt": 4, **_grid(64)},
        # an image (or label map) carried along a known velocity: characteristic
        # plus nt time steps, on the ragged brain grid
        {"name": "transport_brain", "kind": "transport", "rms": 0.3, "nt": 4, "flag": "state", **brain},
        # a velocity at the foot points of the adjoint characteristic, three
        # components at one map (every Hessian application does this)
        {"name": "velocity_at_feet_192", "kind": "interp", "dof": 3, "rms": 0.1, "nt": 8, **_grid(192)},
        # one time step of an image stored in bfloat16 on the largest grid
        {"name": "warp_bf16_256", "kind": "interp16", "dof": 1, "rms": 0.3, "nt": 8, **_grid(256)},
        # the preconditioner, once per Krylov iteration, mid-size grid
        {"name": "precond_h2s_96", "kind": "inverse", "norm": "h2s", "beta": 1e-3, **_grid(96)},
        # the regularisation operator on the largest grid
        {"name": "reg_h1s_256", "kind": "reggrad", "norm": "h1s", "beta": 1e-2, **_grid(256)},
        # the projection of the default (relaxed Stokes) model on the brain grid
        {"name": "leray_brain", "kind": "leray", "model": "relaxedstokes", "beta": 1e-2, **brain},
        # first derivatives: the gradient of an image and the divergence of a
        # velocity at the benchmark's size
        {"name": "derivatives_128", "kind": "derivs", **_grid(128)},
        # a whole registration of one brain pair with the default options
        # (H1 seminorm, relaxed Stokes); pairs like these take four
        # Gauss-Newton iterations
        {"name": "register_brain", "kind": "register", "batch": 1, "norm": "default", "beta": 1e-2, "nt": 4,
         "maxit": 4, "rms": 0.3, "bf16": False, **brain},
        # a batch of small registrations, as a pool of the server runs them
        {"name": "register_64_x32", "kind": "register", "batch": 32, "norm": "h1s", "beta": 1e-2, "nt": 4, "maxit": 3,
         "rms": 0.3, "bf16": False, **_grid(64)},
        # the benchmark's size, time steps and batch: the first two
        # Gauss-Newton iterations of eight registrations
        {"name": "register_128_x8", "kind": "register", "batch": 8, "norm": "h1s", "beta": 1e-2, "nt": 8, "maxit": 2,
         "rms": 0.3, "bf16": False, **_grid(128)},
        # the largest problem, images in bfloat16: the first Gauss-Newton iteration
        {"name": "register_bf16_256", "kind": "register", "batch": 1, "norm": "h2s", "beta": 1e-2, "nt": 8, "maxit": 1,
         "rms": 0.3, "bf16": True, **_grid(256)},
    ]


# Lengths with a transform on every axis; x1 and x2 also take 150.
_SIDES = (32, 48, 64, 96, 128, 192, 256)


def _draw_grid(rng, most):
    """A grid of at most `most` points: cubic half of the time, each axis of
    its own otherwise."""
    while True:
        if rng.random() < 0.5:
            g = _grid(rng.choice(_SIDES))
        else:
            g = _grid(rng.choice(_SIDES + (150,)), rng.choice(_SIDES + (150,)), rng.choice(_SIDES))
        if g["n1"] * g["n2"] * g["n3"] <= most:
            return g


def draw(rng):
    """One more case: an operator on any supported grid up to 256^3, or a
    registration of up to 16.8 million points in all."""
    kind = rng.choice(["interp", "interp16", "transport", "inverse", "reggrad", "leray", "derivs", "register"])
    rms = round(10.0 ** rng.uniform(-1.7, -0.52), 4)  # 0.02 .. 0.3
    nt = rng.choice([4, 8])
    beta = round(10.0 ** rng.uniform(-3.0, -2.0), 5)
    if kind == "register":
        g = _draw_grid(rng, 128 * 150 * 128)
        n = g["n1"] * g["n2"] * g["n3"]
        batch = max(1, min(32, int(2.0 ** rng.uniform(0, math.log2(max(2.0, 8 * 128 ** 3 / n))))))
        bf16 = rng.random() < 0.25
        # the state of a bfloat16 solve is rounded at every time step: past the
        # first iteration its velocity carries that rounding
        return {"kind": kind, "batch": batch, "norm": rng.choice(["default", "h1s", "h2s"]), "beta": beta, "nt": nt,
                "maxit": 1 if bf16 else rng.choice([1, 2]), "rms": min(rms, 0.2), "bf16": bf16, **g}
    g = _draw_grid(rng, 256 ** 3)
    if kind == "transport":
        return {"kind": kind, "rms": rms, "nt": nt, "flag": rng.choice(["state", "adjoint"]), **g}
    if kind in ("interp", "interp16"):
        return {"kind": kind, "dof": rng.choice([1, 3]) if kind == "interp" else 1, "rms": rms, "nt": nt, **g}
    if kind == "inverse":
        return {"kind": kind, "norm": rng.choice(["h1s", "h2s", "h1", "h2"]), "beta": beta, **g}
    if kind == "reggrad":
        return {"kind": kind, "norm": rng.choice(["h1s", "h1"]), "beta": beta, **g}
    if kind == "leray":
        return {"kind": kind, "model": rng.choice(["stokes", "relaxedstokes"]), "beta": beta, **g}
    return {"kind": kind, **g}


def _shape(c):
    return int(c["n1"]), int(c["n2"]), int(c["n3"])


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _wave(shape, half, keep_nyquist=True):
    """Signed wavenumbers of the three axes, broadcastable, float64."""
    ks = []
    for a, n in enumerate(shape):
        m = n // 2 + 1 if (half and a == 2) else n
        k = torch.arange(m, device="cuda", dtype=torch.float64)
        k = torch.where(k > n // 2, k - n, k)
        if not keep_nyquist and n % 2 == 0:
            k[n // 2] = 0.0
        ks.append(k.reshape([-1 if i == a else 1 for i in range(3)]))
    return ks


def _rough(gen, shape, fields, power):
    """Random real fields with amplitude |k|^-power (mean included), unit RMS."""
    out = torch.empty((fields,) + shape, device="cuda", dtype=torch.float32)
    k1, k2, k3 = _wave(shape, True)
    kk = (k1 * k1 + k2 * k2 + k3 * k3).float().clamp_min(1.0) ** (-0.5 * power)
    for f in range(fields):
        w = torch.randn(shape, device="cuda", generator=gen)
        x = torch.fft.irfftn(torch.fft.rfftn(w) * kk, s=shape)
        out[f] = x / x.square().mean().sqrt()
    return out


def _velocity(gen, shape, rms):
    """Random velocity with modes 1 <= |k| <= 6, amplitude 1/|k|^2, and this RMS."""
    v = torch.empty((3,) + shape, device="cuda", dtype=torch.float32)
    k1, k2, k3 = _wave(shape, True)
    kk = k1 * k1 + k2 * k2 + k3 * k3
    band = torch.where((kk >= 1.0) & (kk <= 36.0), 1.0 / kk.clamp_min(1.0), torch.zeros_like(kk)).float()
    for f in range(3):
        w = torch.randn(shape, device="cuda", generator=gen)
        v[f] = torch.fft.irfftn(torch.fft.rfftn(w) * band, s=shape)
    return v * (rms / v.square().mean().sqrt())


def _displacement(gen, shape, rms, nt):
    """A backward map over one time step, in grid units."""
    v = _velocity(gen, shape, rms)
    for a in range(3):
        v[a] *= -shape[a] / (TWO_PI * nt)
    return v


def _images(gen, shape, rms, nt):
    """(reference, template): smooth-edged regions in [0, 1] and their image
    under a velocity, transported in float64."""
    t = _rough(gen, shape, 1, 2.5)[0].double()
    m = torch.sigmoid(4.0 * t)
    mT = m.float().contiguous()
    disp = _velocity(gen, shape, rms).double()
    for a in range(3):
        disp[a] *= -shape[a] / (TWO_PI * nt)
    for _ in range(nt):
        m = _cubic(m, disp)
    return m.clamp(0.0, 1.0).float().contiguous(), mT


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    shape, kind = _shape(case), case["kind"]
    s = {"kind": kind}
    if kind in ("interp", "interp16"):
        s["disp"] = _displacement(gen, shape, case["rms"], case["nt"])
        f = _rough(gen, shape, case["dof"], 2.0)
        if case["dof"] == 1:
            f = f[0].contiguous()
        s["f"] = f.to(torch.bfloat16) if kind == "interp16" else f
    elif kind == "transport":
        s["sl"], s["flag"], s["nt"] = cb.SemiLagrangian(case["nt"]), case["flag"], case["nt"]
        s["v"] = _velocity(gen, shape, case["rms"])
        s["m"] = torch.sigmoid(4.0 * _rough(gen, shape, 1, 2.5)[0]).contiguous()
    elif kind == "inverse":
        s["op"] = cb.Preconditioner(case["norm"], case["beta"], 1e-4)
        s["x"] = _rough(gen, shape, 3, 1.0)
    elif kind == "reggrad":
        s["op"] = cb.Regularization(case["norm"], case["beta"], 1e-4)
        s["x"] = _rough(gen, shape, 3, 2.0)
    elif kind == "leray":
        s["model"], s["beta"] = case["model"], (case["beta"], 1e-4, 1e-4)
        s["b"] = _rough(gen, shape, 3, 1.0)
        s["work"] = torch.empty_like(s["b"])
    elif kind == "derivs":
        s["m"] = _rough(gen, shape, 1, 2.0)[0].contiguous()
        s["v"] = _rough(gen, shape, 3, 2.0)
    elif kind == "register":
        argv = ["-nx", "x".join(str(n) for n in shape), "-nt", str(case["nt"]), "-maxit", str(case["maxit"])]
        if case["norm"] != "default":
            argv += ["-regnorm", case["norm"]]
        argv += ["-beta", repr(case["beta"])] + (["-bf16images"] if case["bf16"] else [])
        s["images"] = [_images(gen, shape, case["rms"], case["nt"]) for _ in range(case["batch"])]
        s["bf16"] = case["bf16"]
        s["ci"] = cb.CLAIREInterface(cb.RegOpt(argv), nbatch=case["batch"])
        s["zero"] = torch.zeros((3,) + shape, device="cuda")
        s["v"] = [torch.empty((3,) + shape, device="cuda") for _ in range(case["batch"])]
        s["m1"] = [torch.empty(shape, device="cuda") for _ in range(case["batch"])]
    else:
        raise ValueError(kind)
    torch.cuda.synchronize()  # a context's own stream reads what was made on torch's
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "interp":
        return cb.SemiLagrangian.Interpolate(s["f"], s["disp"])
    if kind == "interp16":
        return cb.SemiLagrangian.InterpolateBF16(s["f"], s["disp"])
    if kind == "transport":
        disp = s["sl"].ComputeTrajectory(s["v"], s["flag"])
        m = s["m"]
        for _ in range(s["nt"]):
            m = s["sl"].Interpolate(m, disp)
        return disp, m
    if kind == "inverse":
        return s["op"].MatVec(s["x"])
    if kind == "reggrad":
        return s["op"].EvaluateGradient(s["x"])
    if kind == "leray":
        s["work"].copy_(s["b"])  # the projection is in place: the caller keeps its body force
        return cb.leray(s["work"], s["model"], s["beta"])
    if kind == "derivs":
        return cb.fft_grad(s["m"]), cb.fft_div(s["v"])
    # a registration: images and the zero initial guess in, velocities and
    # transported templates out
    ci = s["ci"]
    for b, (mR, mT) in enumerate(s["images"]):
        ci.set_images(mR, mT, b)
        ci.SetInitialGuess(s["zero"], b)
    ci.Run()
    for b in range(len(s["images"])):
        ci.GetSolution(b, out=s["v"][b])
        ci.GetFinalState(b, out=s["m1"][b])
    m1 = torch.stack(s["m1"])
    return torch.stack(s["v"]), m1.to(torch.bfloat16) if s["bf16"] else m1  # in the images' storage type


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    n1, n2, n3 = _shape(case)
    n, kind = n1 * n2 * n3, case["kind"]
    tap = 2 * 84.0  # multiply-adds of one tricubic point (64 + 16 + 4)
    fft = 2.5 * n * math.log2(n)  # one real 3D transform
    if kind == "interp":
        d = case["dof"]
        return {"bytes": 4.0 * n * (2 * d + 3), "flops": tap * d * n}
    if kind == "interp16":
        return {"bytes": n * (2 * 2 + 12.0), "flops": tap * n}
    if kind == "transport":
        # the velocity in, the map out; every step reads the map and the image
        return {"bytes": 4.0 * n * (6 + 5 * case["nt"]), "flops": tap * n * (3 + case["nt"])}
    if kind in ("inverse", "reggrad", "leray"):
        return {"bytes": 24.0 * n, "flops": 6 * fft}
    if kind == "derivs":
        return {"bytes": 32.0 * n, "flops": 8 * fft}
    nt, b = case["nt"], case["batch"]
    img = 2 if case["bf16"] else 4
    # Hessian application and Krylov update: velocity at the feet, sources,
    # nt - 1 incremental and nt adjoint steps, body force, preconditioner
    # and the regulariser's transform, vector updates
    krylov = 36 + 4 * (6 + 7 * nt) + 24 * (2 * nt - 1) + 4 * (4 * (nt + 1) + 3) + 48 + 72
    objective = 24 + nt * (12 + 2 * img) + 2 * img + 12
    gradient = 24 + 16 * (nt + 1) + 16 + 24 + 24 * nt + 4 * (4 * (nt + 1) + 3) + 24
    cache = 3 * nt * 8 + 12
    gn = case["maxit"]
    steps = gn * (3 * krylov + objective + gradient + cache) + objective + gradient
    gathers = gn * (3 * (2 * nt + 2) + 2 * nt + 4 + 3 * nt) + 2 * nt + 4
    ffts = gn * (3 * 12 + 12 + 6 * (nt + 1)) + 6 * (nt + 1)
    return {"bytes": float(n) * b * steps, "flops": b * (tap * n * gathers + fft * ffts)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _cubic(f, disp):
    """Periodic tricubic Lagrange interpolation of f at i + disp (grid units), float64."""
    shape = f.shape
    idx, wts = [], []
    for a in range(3):
        i = torch.arange(shape[a], device=f.device, dtype=torch.float64)
        q = i.reshape([-1 if k == a else 1 for k in range(3)]) + disp[a].double()
        fl = torch.floor(q)
        s = q - fl
        idx.append(fl.long() - 1)
        wts.append([-s * (s - 1) * (s - 2) / 6, (s + 1) * (s - 1) * (s - 2) / 2, -(s + 1) * s * (s - 2) / 2,
                    (s + 1) * s * (s - 1) / 6])
    flat = f.double().reshape(-1)
    out = torch.zeros(shape, device=f.device, dtype=torch.float64)
    for a in range(4):
        ia = torch.remainder(idx[0] + a, shape[0]) * shape[1]
        for b in range(4):
            ib = (ia + torch.remainder(idx[1] + b, shape[1])) * shape[2]
            w = wts[0][a] * wts[1][b]
            for c in range(4):
                out += w * wts[2][c] * flat[ib + torch.remainder(idx[2] + c, shape[2])]
    return out


def _fft3(x):
    return torch.fft.rfftn(x.double(), dim=(-3, -2, -1))


def _ifft3(x, shape):
    return torch.fft.irfftn(x, s=shape, dim=(-3, -2, -1))


def exact(case, seed):
    kind, shape = case["kind"], _shape(case)
    if kind == "register":
        return None
    s = prepare(case, seed)
    if kind in ("interp", "interp16"):
        f = s["f"].double()
        if case["dof"] == 1:
            return _cubic(f, s["disp"])
        return torch.stack([_cubic(f[k], s["disp"]) for k in range(3)])
    if kind == "transport":
        sign = 1.0 if case["flag"] == "state" else -1.0
        v = s["v"].double()
        scale = torch.tensor([sign * shape[a] / (TWO_PI * case["nt"]) for a in range(3)], device="cuda",
                             dtype=torch.float64).reshape(3, 1, 1, 1)
        first = -scale * v
        disp = torch.stack([-0.5 * scale[k] * (v[k] + _cubic(v[k], first)) for k in range(3)])
        m = s["m"].double()
        for _ in range(case["nt"]):
            m = _cubic(m, disp)
        return disp, m
    k1, k2, k3 = _wave(shape, True, keep_nyquist=False)
    kap = k1 * k1 + k2 * k2 + k3 * k3
    hd = TWO_PI ** 3 / (shape[0] * shape[1] * shape[2])
    if kind in ("inverse", "reggrad"):
        b0, b1 = case["beta"], 1e-4
        sym = {"h1s": kap, "h2s": kap * kap, "h1": kap + b1, "h2": kap * kap + b1}[case["norm"]] * b0
        if kind == "reggrad":
            g = hd * sym
        else:
            if case["norm"] in ("h1s", "h2s"):
                sym = torch.where(kap == 0.0, torch.full_like(sym, b0), sym)
            g = 1.0 / sym
        return torch.stack([_ifft3(_fft3(s["x"][k]) * g, shape) for k in range(3)])
    if kind == "leray":
        b = s["b"].double()
        x = [_fft3(b[k]) for k in range(3)]
        ks = (k1, k2, k3)
        kd = k1 * x[0] + k2 * x[1] + k3 * x[2]
        if case["model"] == "stokes":
            l1, l2, l3 = _wave(shape, True)
            kl, c = l1 * l1 + l2 * l2 + l3 * l3, 1.0
        else:
            kl, c = kap, 1.0 / (case["beta"] / (1e-4 * (kap + 1.0)) + 1.0)
        inv = torch.where(kl == 0.0, torch.full_like(kl, -1.0), -1.0 / kl.clamp_min(1e-30))
        return torch.stack([b[a] + _ifft3(ks[a] * (c * inv * kd), shape) for a in range(3)])
    m, v = _fft3(s["m"]), [_fft3(s["v"][a]) for a in range(3)]
    ks = (k1, k2, k3)
    grad = torch.stack([_ifft3(1j * ks[a] * m, shape) for a in range(3)])
    return grad, _ifft3(1j * (k1 * v[0] + k2 * v[1] + k3 * v[2]), shape)
