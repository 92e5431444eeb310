"""The work that users of this library have it do, as timed cases.

Every case is one call sequence through the public Python entry points (`Context`,
`rtm_multi`, `lsrtm.cgls`, `nn.UNet`, `nn.Ops`) with CUDA tensors in and out.  Grids,
time steps, absorbing widths and network shapes are those of the repository's own
workloads, tests and smoke run; only the number of time steps per pass is cut, since
a pass repeats the same step thousands of times.

`exact` restates the modelling passes, the linearised modelling and the network in
plain torch in 64 bits.  Migration images, gradients of the Born operators and CG
results have none: an image divides two wavefields where the source field peaks and
is not a smooth function of its inputs, and the adjoint's value is its transpose.
"""
from __future__ import annotations

import importlib
import math
import random

import numpy as np
import torch

PKG = "2d_and_3d_elastic_reverse_time_migration_b200"
ertm = importlib.import_module(PKG)
nn = importlib.import_module(PKG + ".nn")
lsrtm = importlib.import_module(PKG + ".lsrtm")

DEV = "cuda:0"
LEVELS = (16, 32, 64, 128)


def listed():
    return [
        # the smallest modelling call: a 2D quick look (the learned workload's 128 x 64
        # interior with 20-cell layers), where launches and latency count
        dict(name="model2d_small", kind="model", nx=168, ny=1, nz=104, order=8, boundary="cpml", pml=20, nt=240),
        # the 2D RTM shot of the plain workload: 600 x 300 interior, 40-cell C-PML
        dict(name="rtm2d_shot", kind="rtm", nx=680, ny=1, nz=380, order=8, boundary="cpml", pml=40, nt=240),
        # a long 2D line in the parity scheme (12th order, cubic sponge), ragged sizes
        dict(name="model2d_line_o12", kind="model", nx=1471, ny=1, nz=803, order=12, boundary="cubic", pml=40, nt=90),
        # a small 3D modelling pass with odd extents (test- and smoke-sized work and up)
        dict(name="model3d_odd", kind="model", nx=151, ny=133, nz=117, order=8, boundary="cpml", pml=15, nt=80),
        # the headline: one 3D RTM shot on 480 x 480 x 380 cells, 40-cell C-PML
        dict(name="rtm3d_shot", kind="rtm", nx=480, ny=480, nz=380, order=8, boundary="cpml", pml=40, nt=45),
        # several aperture windows of a shared 3D model in one launch per step
        dict(name="rtm3d_windows", kind="multi", shots=5, wmin=64, wmax=192, nz=280, order=8, pml=40, nt=36, geo=7),
        # linearised modelling of a shot group on the viscoelastic LSRTM grid
        dict(name="born_forward_gsls", kind="born_fwd", nx=880, nz=480, shots=10, nm=3, order=8, pml=40, nt=100),
        # the adjoint (migration) of the learned workload's 512 x 256 patch geometry, elastic
        dict(name="born_adjoint_patch", kind="born_adj", nx=592, nz=336, shots=8, nm=0, order=8, pml=40, nt=240,
             every=100),
        # CG iterations on the small LSRTM geometry that training pairs are made on
        dict(name="lsrtm_cg_small", kind="cgls", nx=168, nz=104, shots=6, nm=0, order=8, pml=20, nt=200, every=100,
             iters=2),
        # the preconditioner inside CG: one image through the network
        dict(name="unet_infer", kind="unet_fwd", n=1, h=256, w=512),
        # one training batch: loss and all gradients
        dict(name="unet_train", kind="unet_grad", n=16, h=256, w=512),
        # one 3x3 layer on its own, forward and both gradients, ragged image
        dict(name="conv_layer_odd", kind="conv", n=5, h=61, w=107, ci=32, co=48),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["model", "model", "rtm", "rtm", "multi", "born_fwd", "born_adj", "cgls", "unet_fwd",
                       "unet_grad", "conv"])
    if kind in ("model", "rtm"):
        two_d = rng.random() < 0.5
        order = rng.choice([8, 8, 12])
        boundary = rng.choice(["cpml", "cpml", "cubic" if two_d else "cos"])
        if two_d:
            return dict(kind=kind, nx=_log(rng, 120, 1600), ny=1, nz=_log(rng, 90, 850), order=order,
                        boundary=boundary, pml=rng.randint(10, 40), nt=rng.randint(60, 240))
        hi = 400 if kind == "rtm" else 220
        return dict(kind=kind, nx=_log(rng, 64, hi), ny=_log(rng, 64, hi), nz=_log(rng, 64, min(hi, 300)),
                    order=order, boundary=boundary, pml=rng.randint(8, 24), nt=rng.randint(24, 45))
    if kind == "multi":
        return dict(kind=kind, shots=rng.randint(2, 6), wmin=64, wmax=rng.randint(80, 192), nz=rng.randint(120, 280),
                    order=8, pml=rng.randint(12, 40), nt=rng.randint(24, 36), geo=rng.randint(1, 10 ** 6))
    if kind in ("born_fwd", "born_adj"):
        c = dict(kind=kind, nx=_log(rng, 160, 880), nz=_log(rng, 100, 480), shots=rng.randint(1, 10),
                 nm=rng.choice([0, 0, 1, 2, 3]), order=rng.choice([8, 8, 12]), pml=rng.randint(20, 40),
                 nt=rng.randint(60, 160))
        if kind == "born_adj":
            c["every"] = rng.choice([40, 100, 200])
        return c
    if kind == "cgls":
        return dict(kind=kind, nx=_log(rng, 140, 400), nz=_log(rng, 90, 220), shots=rng.randint(2, 8),
                    nm=rng.choice([0, 0, 3]), order=8, pml=20, nt=rng.randint(80, 200), every=100, iters=2)
    if kind in ("unet_fwd", "unet_grad"):
        n = 1 if kind == "unet_fwd" else _log(rng, 1, 16)
        return dict(kind=kind, n=n, h=8 * _log(rng, 8, 32), w=8 * _log(rng, 8, 64))
    return dict(kind="conv", n=rng.randint(1, 16), h=_log(rng, 16, 256), w=_log(rng, 16, 512),
                ci=8 * _log(rng, 1, 16), co=8 * _log(rng, 2, 16))


# ---- inputs -----------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def ricker(f0, dt):
    """Ricker wavelet, peak at 1.2 / f0 (float32 numpy)."""
    n = int(2.4 / f0 / dt) + 1
    t = (np.arange(n) - n // 2) * dt
    a = (math.pi * f0 * t) ** 2
    return ((1 - 2 * a) * np.exp(-a)).astype(np.float32)


def _earth(seed, nx, ny, nz, vmax):
    """Layers of seeded depth with gentle lateral structure: (vp, vs, rho), (nz, ny, nx)."""
    r = random.Random(seed)
    z = torch.linspace(0, 1, nz, device=DEV).view(nz, 1, 1)
    x = torch.linspace(0, 1, nx, device=DEV).view(1, 1, nx)
    y = torch.linspace(0, 1, ny, device=DEV).view(1, ny, 1)
    vp = torch.full((nz, ny, nx), 1900.0, device=DEV)
    tops = sorted(r.uniform(0.12, 0.95) for _ in range(5))
    for top in tops:
        dip = top + 0.04 * torch.sin(2 * math.pi * (r.uniform(0.5, 2) * x + r.uniform(0, 1) * y + r.random()))
        vp += (vmax - 1900.0) / 5 * torch.sigmoid((z - dip) * 60)
    lens = ((x - r.uniform(0.3, 0.7)) ** 2 + (y - 0.5) ** 2 * (ny > 1) + (z - 0.5) ** 2) / 0.02
    vp *= 1 + r.uniform(0.03, 0.08) * torch.exp(-lens)
    vs = vp / math.sqrt(3)
    rho = 310 * vp.sqrt().sqrt()
    return vp.contiguous(), vs.contiguous(), rho.contiguous()


def _spread(c):
    """(h, dt in ms, wavelet frequency, fastest layer) of the 2D and 3D workloads"""
    return (5.0, 0.5, 15.0, 3200.0) if c.get("ny", 1) == 1 else (10.0, 0.8, 10.0, 3800.0)


def _boundary(c):
    if c.get("boundary", "cubic") == "cpml":
        return dict(boundary=ertm.BOUNDARY_CPML)
    if c.get("boundary") == "cos":
        return dict(boundary=ertm.BOUNDARY_SPONGE_COS, sponge_coef=60.0)
    return dict(boundary=ertm.BOUNDARY_SPONGE_CUBIC, sponge_coef=150.0)


def _config(c, nx, ny, nz, nt):
    h, dt, _, _ = _spread(c if "ny" in c else dict(ny=ny))
    p, py = c["pml"], c["pml"] if ny > 1 else 0
    extra = dict(checkpoint_every=c["every"]) if "every" in c else {}
    if c.get("nm"):
        extra.update(visco_nmech=c["nm"], visco_qp=100.0, visco_qs=50.0, visco_f0=15.0)
    return ertm.Config(nx=nx, ny=ny, nz=nz, dx=h, dy=h, dz=h, dt_ms=dt, nt=nt, src_steps=2 * nt // 3,
                       order=c["order"], pml=(p, p, py, py, p, p), **_boundary(c), **extra)


def _shot(c, seed, nx, ny, nz):
    """Source just below the top absorbing layer, receivers across the interior."""
    r, p = random.Random(seed + 1), c["pml"]
    _, dt, f0, _ = _spread(c if "ny" in c else dict(ny=ny))
    w = ricker(2.5 * f0, dt / 1e3)
    sx = r.randint(p + 2, nx - p - 3)
    if ny == 1:
        return ertm.Shot(sx, 0, p + 3, wavelet=w, rx0=p, nrx=nx - 2 * p, rz=p + 2)
    sy = r.randint(p + 2, ny - p - 3)
    return ertm.Shot(sx, sy, p + 3, wavelet=w, rx0=p, nrx=(nx - 2 * p + 1) // 2, drx=2, ry0=p,
                     nry=(ny - 2 * p + 1) // 2, dry=2, rz=p + 2)


def _record(seed, nt, nrec):
    """Observed data: band-limited arrivals (3, nt, nrec)."""
    t = torch.randn((3, nt, nrec), generator=_gen(seed), device=DEV)
    k = torch.exp(-0.5 * (torch.arange(-8, 9, device=DEV) / 3.0) ** 2)
    t = torch.nn.functional.conv1d(t.transpose(1, 2).reshape(-1, 1, nt), k.view(1, 1, -1), padding=8)
    return (1e-3 * t.view(3, nrec, nt).transpose(1, 2)).contiguous()


def _windows(c):
    r = random.Random(c["geo"])
    return [(r.randint(c["wmin"], c["wmax"]) + 2 * c["pml"], r.randint(c["wmin"], c["wmax"]) + 2 * c["pml"],
             c["nt"] - r.randint(0, c["nt"] // 3)) for _ in range(c["shots"])]


def _line_shots(c, seed):
    """Shots evenly spaced along a 2D line, every surface cell a receiver."""
    p, nx = c["pml"], c["nx"]
    w = ricker(25.0, 5e-4)
    off = random.Random(seed).randint(0, 3)
    xs = np.linspace(p + 4, nx - p - 8, c["shots"]).round().astype(int) + off
    return [ertm.Shot(int(x), 0, p + 3, wavelet=w, rx0=p, nrx=nx - 2 * p, rz=p + 2) for x in xs]


def _reflectivity(seed, nx, nz):
    """Relative perturbations of (vp, vs, rho): (nz, 1, nx) each, smooth and a few per cent."""
    g = _gen(seed)
    n = torch.randn((3, 1, nz, nx), generator=g, device=DEV)
    k = torch.exp(-0.5 * (torch.arange(-6, 7, device=DEV) / 2.0) ** 2)
    k = k / k.sum()
    n = torch.nn.functional.conv2d(n, k.view(1, 1, 1, -1), padding=(0, 6))
    n = torch.nn.functional.conv2d(n, k.view(1, 1, -1, 1), padding=(6, 0))
    return tuple((0.1 * n[q].reshape(nz, 1, nx)).contiguous() for q in range(3))


def _layers():
    """name -> (rows, K) of the network's parameters"""
    out, cin = {}, 8
    for l, c in enumerate(LEVELS):
        out[f"e{l}a"], out[f"e{l}b"] = (c, 9 * cin), (c, 9 * c)
        cin = c
    for l in (2, 1, 0):
        c = LEVELS[l]
        out[f"u{l}"], out[f"d{l}a"], out[f"d{l}b"] = (4 * c, LEVELS[l + 1]), (c, 18 * c), (c, 9 * c)
    out["out"] = (16, 9 * LEVELS[0])
    return out


def _weights(seed):
    """He-initialised weights that the BF16 kernels hold exactly, and small biases."""
    r = np.random.default_rng(seed)
    sd = {}
    for name, (rows, k) in _layers().items():
        w = torch.from_numpy(r.standard_normal((rows, k)) * (2.0 / k) ** 0.5).to(torch.bfloat16).float().numpy()
        if name == "e0a":
            w.reshape(rows, 9, 8)[:, :, 3:] = 0
        sd[name] = (w, (0.05 * r.standard_normal(rows // 4 if name[0] == "u" else rows)).astype(np.float32))
    return sd


def _images(seed, n, h, w):
    """RMS-normalised smooth images (n, h, w, 3): gradients as the network sees them."""
    x = torch.randn((3 * n, 1, h, w), generator=_gen(seed), device=DEV)
    k = torch.exp(-0.5 * (torch.arange(-4, 5, device=DEV) / 1.5) ** 2)
    x = torch.nn.functional.conv2d(x, k.view(1, 1, -1, 1), padding=(4, 0))
    x = torch.nn.functional.conv2d(x, k.view(1, 1, 1, -1), padding=(0, 4))
    return (x / x.square().mean().sqrt()).view(n, 3, h, w).permute(0, 2, 3, 1).contiguous()


def _conv_inputs(c, seed):
    g = _gen(seed)
    n, h, w, ci, co = c["n"], c["h"], c["w"], c["ci"], c["co"]
    bf = torch.bfloat16
    x = torch.randn((n, h, w, ci), generator=g, device=DEV).relu().to(bf)
    wt = (torch.randn((co, 9, ci), generator=g, device=DEV) * (2.0 / (9 * ci)) ** 0.5).to(bf)
    b = 0.1 * torch.randn(co, generator=g, device=DEV)
    dy = torch.randn((n, h, w, co), generator=g, device=DEV).to(bf)
    return x, wt, b, dy


# ---- a pass -----------------------------------------------------------------------

def prepare(case, seed):
    c, kind = case, case["kind"]
    s = dict(c=c)
    if kind in ("model", "rtm"):
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        ctx = ertm.Context(_config(c, nx, ny, nz, c["nt"]))
        shot = _shot(c, seed, nx, ny, nz)
        ctx.set_model(ertm.TRUE_MODEL if kind == "model" else ertm.MIGRATION_MODEL,
                      *_earth(seed, nx, ny, nz, _spread(c)[3]))
        s.update(ctx=ctx, shot=shot)
        if kind == "model":
            s["out"] = torch.zeros((3, c["nt"], shot.nrec), device=DEV)
        else:
            s["data"] = _record(seed, c["nt"], shot.nrec)
            s["img"] = [torch.zeros((nz, ny, nx), device=DEV) for _ in range(3)]
    elif kind == "multi":
        s.update(ctx=[], shots=[], data=[], img=[])
        for q, (nx, ny, nt) in enumerate(_windows(c)):
            ctx = ertm.Context(_config(dict(c, boundary="cpml", ny=ny), nx, ny, c["nz"], nt))
            ctx.set_model(ertm.MIGRATION_MODEL, *_earth(seed + q, nx, ny, c["nz"], 3800.0))
            shot = _shot(dict(c, ny=ny), seed + q, nx, ny, c["nz"])
            s["ctx"].append(ctx)
            s["shots"].append(shot)
            s["data"].append(_record(seed + q, nt, shot.nrec))
            s["img"].append(tuple(torch.zeros((c["nz"], ny, nx), device=DEV) for _ in range(3)))
    elif kind in ("born_fwd", "born_adj", "cgls"):
        nx, nz = c["nx"], c["nz"]
        ctx = ertm.Context(_config(c, nx, 1, nz, c["nt"]))
        ctx.set_model(ertm.MIGRATION_MODEL, *_earth(seed, nx, 1, nz, 3200.0))
        shots = _line_shots(c, seed)
        nrec = shots[0].nrec
        s.update(ctx=ctx, shots=shots)
        if kind == "born_fwd":
            s["r"] = _reflectivity(seed, nx, nz)
            s["out"] = torch.zeros((c["shots"], 3, c["nt"], nrec), device=DEV)
        else:
            s["data"] = torch.stack([_record(seed + q, c["nt"], nrec) for q in range(c["shots"])])
            s["g"] = [torch.zeros((nz, 1, nx), device=DEV) for _ in range(3)]
    elif kind in ("unet_fwd", "unet_grad"):
        net = nn.UNet(DEV)
        net.load_state_dict(_weights(seed))
        s.update(net=net, x=_images(seed, c["n"], c["h"], c["w"]))
        if kind == "unet_grad":
            s["t"] = _images(seed + 1, c["n"], c["h"], c["w"])
    else:
        n, h, w, ci, co = c["n"], c["h"], c["w"], c["ci"], c["co"]
        x, wt, b, dy = _conv_inputs(c, seed)
        s.update(ops=nn.Ops(DEV), x=x, w=wt, b=b, dy=dy, y=torch.zeros_like(dy), dx=torch.zeros_like(x),
                 wf=torch.zeros((ci, 9, co), dtype=torch.bfloat16, device=DEV))
        s["ops"].flip3(wt, s["wf"], co, ci)
    torch.cuda.synchronize()
    return s


def run(s):
    c = s["c"]
    kind = c["kind"]
    if kind == "model":
        return s["ctx"].forward_together_using_real_model(s["shot"], out=s["out"])
    if kind == "rtm":
        return s["ctx"].rtm_shot(s["shot"], s["data"], *s["img"])
    if kind == "multi":
        return ertm.rtm_multi(s["ctx"], s["shots"], s["data"], s["img"])
    if kind == "born_fwd":
        return s["ctx"].born_forward_shots(s["shots"], *s["r"], out=s["out"])
    if kind == "born_adj":
        return s["ctx"].born_adjoint_shots(s["shots"], s["data"], *s["g"])
    if kind == "cgls":
        r = lsrtm.cgls(s["ctx"], s["shots"], list(s["data"]), niter=c["iters"])
        return [r.m, r.misfit]
    if kind == "unet_fwd":
        return s["net"].forward(s["x"])
    if kind == "unet_grad":
        loss = s["net"].loss_grad(s["x"], s["t"])
        return [loss, {k: (p.g, p.bg) for k, p in s["net"].params.items()}]
    o, n, h, w = s["ops"], c["n"], c["h"], c["w"]
    x, y, dy, dx = (nn.act(s[k], n, h, w) for k in ("x", "y", "dy", "dx"))
    o.conv(x, s["w"], s["b"], y)
    dw = torch.zeros((c["co"], 9, c["ci"]), device=DEV)
    db = torch.zeros(c["co"], device=DEV)
    o.conv_wgrad(x, dy, dw)
    o.bias_grad(dy, db)
    o.conv_dgrad(dy, s["wf"], dx, mask=x)
    return [s["y"], dw, db, s["dx"]]


def work(case):
    """Compulsory traffic and arithmetic.  Per cell and time step a pass reads and writes
    every wavefield and reads the model once (3D 84 B, 2D 52 B)."""
    c, kind = case, case["kind"]
    taps = 2 * (c.get("order", 8) // 2)
    if kind in ("model", "rtm"):
        two_d = c["ny"] == 1
        cells, steps = c["nx"] * c["ny"] * c["nz"], c["nt"] + (2 * c["nt"] // 3 if kind == "rtm" else 0)
        der = (8 if two_d else 18) + ((2 if two_d else 3) if kind == "rtm" else 0)
        return dict(bytes=cells * steps * (52 if two_d else 84), flops=cells * steps * (der * 1.5 * taps + 40))
    if kind == "multi":
        cs = sum(nx * ny * c["nz"] * (nt + 2 * nt // 3) for nx, ny, nt in _windows(c))
        return dict(bytes=84 * cs, flops=cs * (21 * 1.5 * taps + 40))
    if kind in ("born_fwd", "born_adj", "cgls"):
        cs = c["nx"] * c["nz"] * c["nt"] * c["shots"]
        fwd = 8 * 2 * (5 + 3 * c["nm"])                 # background and scattered state, read and written
        adj = 2 * 8 * (5 + 3 * c["nm"]) + 8 * (5 + 3 * c["nm"]) + 32 + 24
        ffl, afl = 16 * 1.5 * taps + 80 + 36 * c["nm"], 24 * 1.5 * taps + 120 + 54 * c["nm"]
        nf, na = dict(born_fwd=(1, 0), born_adj=(0, 1), cgls=(c.get("iters", 0), c.get("iters", 0) + 1))[kind]
        return dict(bytes=cs * (nf * fwd + na * adj), flops=cs * (nf * ffl + na * afl))
    if kind in ("unet_fwd", "unet_grad"):
        flops = act = 0
        for name, (rows, k) in _layers().items():
            l = int(name[1]) if name[0] in "edu" and name != "out" else 0
            pix = c["n"] * (c["h"] >> l) * (c["w"] >> l)
            if name[0] == "u":
                pix //= 4
            flops += 2 * pix * rows * k
            act += 2 * pix * (rows + (k if name[0] == "u" else k // 9))
        return dict(bytes=act if kind == "unet_fwd" else 3 * act, flops=flops * (1 if kind == "unet_fwd" else 3))
    pix, ci, co = c["n"] * c["h"] * c["w"], c["ci"], c["co"]
    return dict(bytes=2 * pix * (2 * ci + 2 * co) + 2 * pix * ci, flops=3 * 2 * pix * co * 9 * ci)


# ---- 64-bit restatement -----------------------------------------------------------

def _taylor(R):
    """staggered first-derivative weights c_1 .. c_R"""
    m, n = np.meshgrid(np.arange(R), np.arange(R), indexing="ij")
    e = np.zeros(R)
    e[0] = 1
    return np.linalg.solve((2.0 * n + 1) ** (2.0 * m + 1), e)


def _diff(f, axis, plus, cf):
    """D+ (half a cell up) or D- (half a cell down) of f along axis, zero outside."""
    R, n = len(cf), f.shape[axis]
    pad = [0, 0] * f.dim()
    i = 2 * (f.dim() - 1 - axis)
    pad[i] = pad[i + 1] = R
    q = torch.nn.functional.pad(f, pad)
    out = torch.zeros_like(f)
    for k in range(1, R + 1):
        hi, lo = (k, 1 - k) if plus else (k - 1, -k)
        out += cf[k - 1] * (q.narrow(axis, R + hi, n) - q.narrow(axis, R + lo, n))
    return out


def _cpml(n, w, stagger, h, vmax, dts, rc=1e-3, f0=10.0):
    """C-PML recursion coefficients (a, b) of one axis, kappa = 1"""
    a, b = np.zeros(n), np.ones(n)
    for q in range(n):
        p, dist = q + 0.5 * stagger, 0.0
        if w > 0 and p < w - 1:
            dist = (w - 1) - p
        elif w > 0 and p > n - w:
            dist = p - (n - w)
        if dist <= 0:
            continue
        x = dist / w
        d = -3.0 * vmax * math.log(rc) / (2.0 * w * h) * x * x
        al = max(0.0, math.pi * f0 * (1 - x))
        b[q] = math.exp(-(d + al) * dts)
        a[q] = d * (b[q] - 1) / (d + al)
    return a, b


def _sponge(n, w, kind, coef):
    v = np.zeros(n)
    for i in range(w):
        x = (w - 1.0 - i) / (w - 1.0)
        t = coef * (1 - math.cos(3.1415926 / 2 * x)) if kind == "cos" else coef * x ** 3
        v[i] += t
        v[n - 1 - i] += t
    return v


class _Medium:
    """Grid operators and absorbing layers of a case, 64 bits, volumes (shots, nz, ny, nx)."""

    def __init__(self, c, nx, ny, nz, vp, vs, rho):
        h, dt, _, _ = _spread(dict(ny=ny))
        dt = float(np.float32(dt) / np.float32(1000))
        self.dt, self.two_d = dt, ny == 1
        self.cf = [float(np.float32(v / h)) for v in np.float32(_taylor(c["order"] // 2))]
        d = lambda a: torch.as_tensor(a, dtype=torch.float64, device=DEV)
        vp, vs, rho = (v.double() for v in (vp, vs, rho))
        self.M, self.U, self.b = rho * vp * vp, rho * vs * vs, 1 / rho
        self.psi, self.prof = {}, None
        self.g1 = self.g2 = torch.ones((), dtype=torch.float64, device=DEV)
        dims, view = (nz, ny, nx), ((-1, 1, 1), (1, -1, 1), (1, 1, -1))
        if c.get("boundary", "cubic") == "cpml":
            vmax = float(vp.max())
            self.prof = {}
            for ax in range(3):
                w = 0 if dims[ax] == 1 else c["pml"]
                for half in (0, 1):
                    a, b = _cpml(dims[ax], w, 0 if not half else (1 if ax == 0 else -1), h, vmax, dt)
                    self.prof[ax, half] = (d(a).view(view[ax]), d(b).view(view[ax]))
        else:
            at = torch.zeros(dims, dtype=torch.float64, device=DEV)
            for ax in range(3):
                if dims[ax] > 1:
                    at += d(_sponge(dims[ax], c["pml"], c.get("boundary", "cubic"),
                                    60.0 if c.get("boundary") == "cos" else 150.0)).view(view[ax])
            self.g1, self.g2 = 1 / (1 + at * dt / 2), 1 - at * dt / 2

    def der(self, key, f, ax, plus, half):
        """derivative along ax (0 z, 1 y, 2 x), through its memory variable under C-PML"""
        v = _diff(f, f.dim() - 3 + ax, plus, self.cf)
        if self.prof is None:
            return v
        a, b = self.prof[ax, half]
        p = a * v + (b * self.psi[key] if key in self.psi else 0)
        self.psi[key] = p
        return v + p


def _exact_model(c, seed):
    nx, ny, nz, nt = c["nx"], c["ny"], c["nz"], c["nt"]
    shot = _shot(c, seed, nx, ny, nz)
    m = _Medium(c, nx, ny, nz, *_earth(seed, nx, ny, nz, _spread(c)[3]))
    z = lambda: torch.zeros((nz, ny, nx), dtype=torch.float64, device=DEV)
    vx, vy, vz, xx, yy, zz, xy, xz, yz = (z() for _ in range(9))
    out = torch.zeros((3, nt, shot.nrec), dtype=torch.float64, device=DEV)
    ys = slice(shot.ry0, shot.ry0 + (shot.nry - 1) * shot.dry + 1, shot.dry)
    xs = slice(shot.rx0, shot.rx0 + (shot.nrx - 1) * shot.drx + 1, shot.drx)
    L, D, dt = m.M - 2 * m.U, m.der, m.dt
    up = lambda f, inc: m.g1 * (m.g2 * f + dt * inc)
    for it in range(nt):
        if it < len(shot.wavelet):
            for f in (xx, zz) if ny == 1 else (xx, yy, zz):
                f[shot.sz, shot.sy, shot.sx] += float(shot.wavelet[it])
        exx, ezz = D("exx", vx, 2, True, 0), D("ezz", vz, 0, False, 0)
        exz = D("dzvx", vx, 0, True, 1) + D("dxvz", vz, 2, False, 1)
        eyy = 0.0
        if ny > 1:
            eyy = D("eyy", vy, 1, True, 0)
            xy = up(xy, m.U * (D("dyvx", vx, 1, False, 1) + D("dxvy", vy, 2, False, 1)))
            yz = up(yz, m.U * (D("dzvy", vy, 0, True, 1) + D("dyvz", vz, 1, False, 1)))
            yy = up(yy, m.M * eyy + L * (exx + ezz))
        xx, zz, xz = up(xx, m.M * exx + L * (eyy + ezz)), up(zz, m.M * ezz + L * (exx + eyy)), up(xz, m.U * exz)
        ax = D("dxtxx", xx, 2, False, 1) + D("dztxz", xz, 0, False, 0)
        az = D("dxtxz", xz, 2, True, 0) + D("dztzz", zz, 0, True, 1)
        if ny > 1:
            ax = ax + D("dytxy", xy, 1, True, 0)
            az = az + D("dytyz", yz, 1, True, 0)
            vy = up(vy, m.b * (D("dxtxy", xy, 2, True, 0) + D("dytyy", yy, 1, False, 1) + D("dztyz", yz, 0, False, 0)))
        vx, vz = up(vx, m.b * ax), up(vz, m.b * az)
        for q, f in enumerate((vx, vy, vz)):
            out[q, it] = f[shot.rz, ys, xs].reshape(-1)
    return out


def _exact_born(c, seed):
    nx, nz, nt, nm = c["nx"], c["nz"], c["nt"], c["nm"]
    shots = _line_shots(c, seed)
    ns, nrec = len(shots), shots[0].nrec
    m = _Medium(c, nx, 1, nz, *_earth(seed, nx, 1, nz, 3200.0))
    rp, rs, rr = (r.double() for r in _reflectivity(seed, nx, nz))
    dM, dU = m.M * (rr + 2 * rp), m.U * (rr + 2 * rs)
    tp = ts = 0.0
    ra, rb = [], []
    if nm:
        f0 = 15.0
        tau = [1 / (2 * math.pi * f0 * 10 ** (2 * (l + 0.5) / nm - 1)) for l in range(nm)]
        wv = 2 * math.pi * f0 / 4 * 16 ** (np.arange(32) / 31)
        S = sum(wv * t / (1 + (wv * t) ** 2) for t in tau)
        tp, ts = 0.01 * S.sum() / (S * S).sum(), 0.02 * S.sum() / (S * S).sum()
        for t in tau:
            q = m.dt / (2 * t)
            ra.append((1 - q) / (1 + q))
            rb.append(-2 * q / (1 + q))
    kp, ks = 1 + nm * tp, 1 + nm * ts
    z = lambda: torch.zeros((ns, nz, 1, nx), dtype=torch.float64, device=DEV)
    bg, sc = [z() for _ in range(5)], [z() for _ in range(5)]          # vx vz xx zz xz
    mb, ms = [[z() for _ in range(nm)] for _ in range(3)], [[z() for _ in range(nm)] for _ in range(3)]
    iso = lambda p, u, e: (p * e[0] + (p - 2 * u) * e[1], p * e[1] + (p - 2 * u) * e[0], u * e[2])
    D, dt = m.der, m.dt
    strain = lambda f: (D("", f[0], 2, True, 0), D("", f[1], 0, False, 0),
                        D("", f[0], 0, True, 0) + D("", f[1], 2, False, 0))
    acc = lambda f: (m.b * (D("", f[2], 2, False, 0) + D("", f[4], 0, False, 0)),
                     m.b * (D("", f[4], 2, True, 0) + D("", f[3], 0, True, 0)))
    out = torch.zeros((ns, 3, nt, nrec), dtype=torch.float64, device=DEV)
    for it in range(nt):
        for q, sh in enumerate(shots):
            if it < len(sh.wavelet):
                for f in (bg[2], bg[3]):
                    f[q, sh.sz, 0, sh.sx] += float(sh.wavelet[it])
        e0, e = strain(bg), strain(sc)
        E0, E, dE = iso(m.M * kp, m.U * ks, e0), iso(m.M * kp, m.U * ks, e), iso(dM * kp, dU * ks, e0)
        F0, F, dF = iso(m.M * tp, m.U * ts, e0), iso(m.M * tp, m.U * ts, e), iso(dM * tp, dU * ts, e0)
        for q in range(3):
            for l in range(nm):
                mb[q][l] = ra[l] * mb[q][l] + rb[l] * F0[q]
                ms[q][l] = ra[l] * ms[q][l] + rb[l] * (F[q] + dF[q])
            bg[2 + q] = m.g1 * (m.g2 * bg[2 + q] + dt * (E0[q] + sum(mb[q])))
            sc[2 + q] = m.g1 * (m.g2 * sc[2 + q] + dt * (E[q] + dE[q] + sum(ms[q])))
        a0, a = acc(bg), acc(sc)
        for q in range(2):
            bg[q] = m.g1 * (m.g2 * bg[q] + dt * a0[q])
            sc[q] = m.g1 * (m.g2 * sc[q] + dt * (a[q] - rr * a0[q]))
        p = c["pml"]
        out[:, 0, it], out[:, 2, it] = sc[0][:, p + 2, 0, p:nx - p], sc[1][:, p + 2, 0, p:nx - p]
    return out


def _net64(w, x):
    """The U-Net on (n, h, w, 3) in 64 bits; w: name -> (weight, bias)."""
    F = torch.nn.functional

    def conv(t, name, relu=True):
        k, b = w[name]
        k = k.view(k.shape[0], 3, 3, -1).permute(0, 3, 1, 2)
        t = F.conv2d(t, k[:, :t.shape[1]], b, padding=1)
        return t.relu() if relu else t

    def up(t, name):
        k, b = w[name]
        k = k.view(2, 2, -1, k.shape[1]).permute(3, 2, 0, 1)
        return F.conv_transpose2d(t, k, b, stride=2).relu()

    t, skips = x.permute(0, 3, 1, 2), []
    for l in range(4):
        t = conv(conv(t, f"e{l}a"), f"e{l}b")
        if l < 3:
            skips.append(t)
            t = F.max_pool2d(t, 2)
    for l in (2, 1, 0):
        t = conv(conv(torch.cat([up(t, f"u{l}"), skips[l]], 1), f"d{l}a"), f"d{l}b")
    return conv(t, "out", False)[:, :3].permute(0, 2, 3, 1)


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "model":
        return _exact_model(c, seed)
    if kind == "born_fwd":
        return _exact_born(c, seed)
    if kind in ("unet_fwd", "unet_grad"):
        w = {k: tuple(torch.from_numpy(v).double().to(DEV) for v in p) for k, p in _weights(seed).items()}
        x = _images(seed, c["n"], c["h"], c["w"]).double()
        if kind == "unet_fwd":
            with torch.no_grad():
                return _net64(w, x)
        for p in w.values():
            for v in p:
                v.requires_grad_()
        t, total = _images(seed + 1, c["n"], c["h"], c["w"]).double(), 0.0
        for q in range(c["n"]):                          # one image at a time: memory
            loss = (_net64(w, x[q:q + 1]) - t[q:q + 1]).square().sum() / t.numel()
            loss.backward()
            total += loss.detach()
        return [total.view(1), {k: (p[0].grad, p[1].grad) for k, p in w.items()}]
    if kind == "conv":
        x, wt, b, dy = (v.double() for v in _conv_inputs(c, seed))
        k = wt.view(c["co"], 3, 3, c["ci"]).permute(0, 3, 1, 2).contiguous().requires_grad_()
        xi = x.permute(0, 3, 1, 2).contiguous().requires_grad_()
        y = torch.nn.functional.conv2d(xi, k, b, padding=1)
        y.backward(dy.permute(0, 3, 1, 2))
        return [y.detach().relu().permute(0, 2, 3, 1).contiguous(),
                k.grad.permute(0, 2, 3, 1).reshape(c["co"], 9, c["ci"]), dy.sum((0, 1, 2)),
                (xi.grad.permute(0, 2, 3, 1) * (x > 0)).contiguous()]
    return None
