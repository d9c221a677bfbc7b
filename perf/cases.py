"""Timed cases of the reconstruction path, through the Python binding's entry points.

Every case is one call (or, for a reconstruction, the one call) that a program
on top of this library makes with its data already on the GPU: the operators
F and F^H, the brute-force and Toeplitz reconstructions, the Toeplitz set-up
steps (Q and F^H d by gridding) and the warm start's network.  `listed()` holds
one case of each; `draw()` gives others of the same ranges.

Inputs are seeded and synthetic: variable-density spirals (stacked along kz in
3-D) with centric-out timing, Gaussian-bump coil maps of unit root-sum-of-
squares, smooth field maps of up to 50 Hz, ellipse phantoms.  Toeplitz cases
that start from a given Q take the kernel of such a trajectory's sampling
density, cut into time segments.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TWO_PI = 2.0 * math.pi


def _package():
    """The package directory impatient-mri_b200/ as the module impatient_mri_b200."""
    name = "impatient_mri_b200"
    if name not in sys.modules:
        path = os.path.join(os.getcwd(), "impatient-mri_b200")
        if not os.path.isdir(path):
            path = os.path.join(_ROOT, "impatient-mri_b200")
        spec = importlib.util.spec_from_file_location(
            name, os.path.join(path, "__init__.py"), submodule_search_locations=[path])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[name] = mod
        spec.loader.exec_module(mod)
    return sys.modules[name]


# ------------------------------------------------------------------ the cases


def listed():
    return [
        # One F of the smallest configuration (64x64, one coil, 4 x 1024 spiral), as a custom
        # solver or a simulation loop calls it: launches and host work count.
        dict(name="ft_64x64", kind="ft", nx=64, ny=64, nz=1, coils=1, inter=4, read=1024),
        # One F^H of a ragged problem: odd image sides, three coils, a sample count that is no
        # multiple of anything.
        dict(name="ift_97x90_c3", kind="ift", nx=97, ny=90, nz=1, coils=3, inter=7, read=1429),
        # One F^H with the many-coil arrays of the multi-slice configuration (32 ring coils).
        dict(name="ift_192x192_c32", kind="ift", nx=192, ny=192, nz=1, coils=32, inter=16,
             read=2048),
        # The 3-D brute-force configuration (64x64x16, 4 coils, 16 kz x 4 x 1024, field map) with
        # the finite-difference penalty and the default number of CG iterations.
        dict(name="bruteforce_64x64x16", kind="bf", nx=64, ny=64, nz=16, coils=4, inter=4,
             read=1024, cg=8),
        # The batched multi-slice solver: slices of one volume with their own spirals, field maps
        # and sample counts, 32 coils.
        dict(name="batch_4x160x160_c32", kind="batch", nx=160, ny=160, nz=1, coils=32, inter=14,
             read=1024, slices=4, cg=3),
        # Q of a 3-D trajectory by gridding on the doubled grid (L = 8, oversampling 2 as in the
        # 3-D Toeplitz configuration), once per trajectory.
        dict(name="q_128x128x32", kind="q", nx=128, ny=128, nz=32, inter=8, read=2048, segs=8,
             os_q=2.0),
        # F^H d by gridding, once per slice: every coil, the default 12 time segments.
        dict(name="fhd_256x256_c16", kind="fhd", nx=256, ny=256, nz=1, coils=16, inter=16,
             read=4096, segs=12, os_fh=1.5),
        # The headline: Toeplitz CG from a starting image, 512x512, 32 coils, no field map (one
        # segment), 20 updates.
        dict(name="cg_512x512_c32", kind="tcg", nx=512, ny=512, nz=1, coils=32, segs=0, cg=20),
        # The 3-D Toeplitz configuration (256x256x32, 4 coils, L = 8), a short CG with the
        # finite-difference penalty.
        dict(name="recon_256x256x32_c4", kind="trecon", nx=256, ny=256, nz=32, coils=4, segs=8,
             cg=4),
        # A 2-D reconstruction at a clinical matrix size that is no power of two, field map, the
        # default number of CG iterations.
        dict(name="recon_240x240_c8", kind="trecon", nx=240, ny=240, nz=1, coils=8, segs=6, cg=8),
        # The warm start's network on one image (serving).
        dict(name="unet_forward_512_b1", kind="unet", size=512, batch=1, train=False),
        # Loss and gradients of the network on a training batch of eight.
        dict(name="unet_gradients_512_b8", kind="unet", size=512, batch=8, train=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _side(rng, lo, hi, step):
    """An image side in [lo, hi]: a power of two in two cases out of five, else a multiple of
    `step`."""
    if rng.random() < 0.4:
        p = [1 << b for b in range(4, 11) if lo <= (1 << b) <= hi]
        if p:
            return rng.choice(p)
    return min(hi, max(lo, step * int(round(_log_int(rng, lo, hi) / step))))


def draw(rng):
    kind = rng.choice(["ft", "ift", "ift", "bf", "batch", "q", "fhd", "tcg", "trecon", "trecon",
                       "unet"])
    if kind in ("ft", "ift"):
        nz = rng.choice([1, 1, 1, 12])
        n = _log_int(rng, 32, 64 if nz > 1 else 200)
        nx, ny = n + rng.randrange(0, 9), n
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, coils=_log_int(rng, 1, 32),
                    inter=rng.randrange(2, 17), read=_log_int(rng, 256, 2048 if nz == 1 else 256))
    if kind == "bf":
        nz = rng.choice([1, 1, 8])
        n = _log_int(rng, 32, 128 if nz == 1 else 48)
        return dict(kind=kind, nx=n, ny=n, nz=nz, coils=_log_int(rng, 1, 8),
                    inter=rng.randrange(2, 9), read=_log_int(rng, 256, 1024), cg=rng.randrange(3, 9))
    if kind == "batch":
        n = _log_int(rng, 48, 128)
        return dict(kind=kind, nx=n, ny=n, nz=1, coils=_log_int(rng, 1, 32),
                    inter=rng.randrange(4, 13), read=_log_int(rng, 256, 1024),
                    slices=rng.randrange(2, 7), cg=3)
    if kind == "q":
        if rng.random() < 0.5:
            return dict(kind=kind, nx=_side(rng, 48, 128, 8), ny=_side(rng, 48, 128, 8),
                        nz=rng.choice([8, 16, 24]), inter=rng.randrange(4, 9),
                        read=_log_int(rng, 512, 2048), segs=rng.randrange(0, 9),
                        os_q=rng.choice([1.25, 1.5, 2.0]))
        return dict(kind=kind, nx=_side(rng, 64, 512, 8), ny=_side(rng, 64, 512, 8), nz=1,
                    inter=rng.randrange(4, 17), read=_log_int(rng, 512, 4096),
                    segs=rng.randrange(0, 13), os_q=rng.choice([1.25, 1.5, 2.0]))
    if kind == "fhd":
        if rng.random() < 0.3:
            return dict(kind=kind, nx=_side(rng, 48, 128, 8), ny=_side(rng, 48, 128, 8),
                        nz=rng.choice([8, 16, 24]), coils=_log_int(rng, 1, 8),
                        inter=rng.randrange(4, 9), read=_log_int(rng, 512, 2048),
                        segs=rng.randrange(0, 9), os_fh=rng.choice([1.5, 2.0]))
        return dict(kind=kind, nx=_side(rng, 64, 512, 8), ny=_side(rng, 64, 512, 8), nz=1,
                    coils=_log_int(rng, 1, 32), inter=rng.randrange(4, 17),
                    read=_log_int(rng, 512, 4096), segs=rng.randrange(0, 13),
                    os_fh=rng.choice([1.5, 2.0]))
    if kind == "tcg":
        return dict(kind=kind, nx=_side(rng, 64, 512, 8), ny=_side(rng, 64, 512, 8), nz=1,
                    coils=_log_int(rng, 1, 32), segs=0, cg=rng.randrange(4, 13))
    if kind == "trecon":
        if rng.random() < 0.4:
            return dict(kind=kind, nx=_side(rng, 48, 192, 8), ny=_side(rng, 48, 192, 8),
                        nz=rng.choice([8, 16, 24, 32]), coils=_log_int(rng, 1, 8),
                        segs=rng.randrange(1, 9), cg=rng.randrange(3, 6))
        return dict(kind=kind, nx=_side(rng, 64, 384, 8), ny=_side(rng, 64, 384, 8), nz=1,
                    coils=_log_int(rng, 1, 16), segs=rng.randrange(0, 9),
                    cg=rng.randrange(4, 9))
    return dict(kind="unet", size=8 * _log_int(rng, 8, 64), batch=rng.randrange(1, 5),
                train=rng.random() < 0.5)


# ------------------------------------------------------------------ the inputs


def _gen(seed, salt):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, salt])


def _axis(n):
    return (np.arange(n) - n // 2) / n


def _shape(case):
    """Image shape in voxel order: 2-D (x, y) with y fastest, 3-D (y, x, z) with z fastest."""
    if case["nz"] == 1:
        return (case["nx"], case["ny"])
    return (case["ny"], case["nx"], case["nz"])


def _coords(case):
    """Axis coordinates of the voxel grid as broadcastable float64 CUDA tensors."""
    shape = _shape(case)
    out = []
    for a, n in enumerate(shape):
        v = torch.as_tensor(_axis(n), device="cuda")
        out.append(v.reshape([n if b == a else 1 for b in range(len(shape))]))
    return out


def _positions(case):
    c = [x.expand(_shape(case)).reshape(-1).float().contiguous() for x in _coords(case)]
    if case["nz"] == 1:
        return c[0], c[1], torch.zeros_like(c[0])
    return c[1], c[0], c[2]


def _trajectory(case, rng, inter=None):
    """(kx, ky, kz, t): a variable-density spiral, repeated over the kz levels in 3-D."""
    inter = case["inter"] if inter is None else inter
    read = case["read"]
    kmax = min(case["nx"], case["ny"]) / 2 - 0.05
    s = np.arange(read) / read
    turns = max(kmax / inter, 1.0)
    th = TWO_PI * (turns * s[None, :] + np.arange(inter)[:, None] / inter) + rng.uniform(0, TWO_PI)
    r = kmax * s[None, :] ** 1.5
    kx = (r * np.cos(th)).ravel().astype(np.float32)
    ky = (r * np.sin(th)).ravel().astype(np.float32)
    t = np.tile(s * 0.010, inter).astype(np.float32)
    nz = case["nz"]
    kz = np.repeat(np.arange(-(nz // 2), nz - nz // 2, dtype=np.float32), kx.size)
    if nz > 1:
        kx, ky, t = np.tile(kx, nz), np.tile(ky, nz), np.tile(t, nz)
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32)).cuda()
    return dev(kx), dev(ky), dev(kz), dev(t)


def _field_map(case, rng):
    co = _coords(case)
    f = sum(rng.uniform(-1, 1) * c ** 2 + rng.uniform(-0.5, 0.5) * c for c in co)
    d2 = sum((c - rng.uniform(-0.2, 0.2)) ** 2 for c in co)
    f = f + rng.uniform(0.5, 1.0) * torch.exp(-d2 / 0.02)
    f = f / f.abs().max().clamp_min(1e-12)
    return (TWO_PI * 50.0 * f).reshape(-1).float().contiguous()


def _coil_maps(case, rng):
    """[C][N] complex64, unit root-sum-of-squares (one coil: ones)."""
    C = case["coils"]
    n = math.prod(_shape(case))
    if C == 1:
        return torch.ones(1, n, dtype=torch.complex64, device="cuda")
    co = _coords(case)
    maps = []
    for c in range(C):
        a = TWO_PI * c / C
        centre = [0.5 * math.cos(a), 0.5 * math.sin(a), 0.0]
        g = torch.exp(-sum((x - m) ** 2 for x, m in zip(co, centre)) / 0.32)
        ph = sum(rng.uniform(-1.0, 1.0) * x for x in co) * math.pi
        maps.append(torch.polar(g, ph).reshape(-1))
    maps = torch.stack(maps)
    return (maps / maps.abs().square().sum(0).sqrt()).to(torch.complex64)


def _phantom(case, rng):
    co = _coords(case)
    shape = _shape(case)
    img = torch.zeros(shape, dtype=torch.float64, device="cuda")
    for _ in range(8):
        q = sum(((c - rng.uniform(-0.25, 0.25)) / rng.uniform(0.1, 0.3)) ** 2 for c in co)
        img += rng.uniform(0.1, 1.0) * (q <= 1.0)
    ph = sum(rng.uniform(-1.0, 1.0) * c for c in co) * math.pi
    return torch.polar(img, ph.expand(shape)).reshape(-1).to(torch.complex64)


def _segments(case, t):
    """(tau, t0) of the time segmentation."""
    t0, t1 = float(t[0]), float(t[-1])
    L = case["segs"]
    return ((t1 - t0) / L if L > 0 else t1 - t0), t0


def _density_q(case, rng, tau, t0):
    """Q_l (complex128 [L+1][2N grid], centre at n for each axis) of a variable-density
    trajectory's sampling density: spectrum ~ 1/sqrt-radius density over the sampled disc with a
    seeded ripple, cut into the Hanning time segments of centric-out timing."""
    shape = tuple(2 * n for n in _shape(case))
    fr = [torch.fft.fftfreq(n, device="cuda", dtype=torch.float64) * 2 for n in shape]
    fr = [v.reshape([-1 if b == a else 1 for b in range(len(shape))]) for a, v in enumerate(fr)]
    rad = torch.sqrt(fr[0] ** 2 + fr[1] ** 2)
    rad = rad.expand(shape) if len(shape) == 2 else (rad + 0 * fr[2]).expand(shape)
    dens = 1.0 / (0.05 + rad) ** 0.5 * (1.0 + 0.2 * torch.cos(
        rng.uniform(4, 9) * math.pi * fr[0] + rng.uniform(0, 6)) * torch.cos(
            rng.uniform(4, 9) * math.pi * fr[1]))
    dens = dens * torch.sigmoid((1.0 - rad) * 40.0)
    time = t0 + 0.010 * rad.clamp_max(1.0) ** (1.0 / 1.5)
    axes = tuple(range(len(shape)))
    for l in range(case["segs"] + 1):
        if case["segs"] == 0:
            w = dens
        else:
            x = time - tau * l - t0
            w = torch.where(x.abs() < tau, 0.5 + 0.5 * torch.cos(math.pi * x / tau), 0.0 * x) * dens
        yield torch.fft.fftshift(torch.fft.ifftn(w.to(torch.complex128), dim=axes), dim=axes)


def _he_params(rng):
    parts = []
    for ci, co, k in _UNET:
        parts.append(rng.standard_normal(co * k * k * ci) * math.sqrt(2.0 / (k * k * ci)))
        parts.append(rng.standard_normal(co) * 0.05)
    return np.concatenate(parts).astype(np.float32)


def _unet_images(rng, batch, n):
    """[batch][2][n*n] float32: smooth complex images of unit RMS with a noise floor."""
    ax = torch.as_tensor(_axis(n), device="cuda").reshape(-1, 1)
    out = torch.zeros(batch, 2, n, n, dtype=torch.float64, device="cuda")
    for b in range(batch):
        img = torch.zeros(n, n, dtype=torch.float64, device="cuda")
        for _ in range(8):
            q = ((ax - rng.uniform(-0.25, 0.25)) / rng.uniform(0.05, 0.3)) ** 2 + (
                (ax.T - rng.uniform(-0.25, 0.25)) / rng.uniform(0.05, 0.3)) ** 2
            img += rng.uniform(0.1, 1.0) * torch.sigmoid((1.0 - q) * 8.0)
        ph = math.pi * (rng.uniform(-1, 1) * ax + rng.uniform(-1, 1) * ax.T)
        out[b, 0], out[b, 1] = img * torch.cos(ph), img * torch.sin(ph)
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 30)))
    out += 0.02 * torch.randn(out.shape, generator=g, device="cuda", dtype=torch.float64)
    out /= out.square().mean().sqrt()
    return out.reshape(batch, 2, n * n).float().contiguous()


# (cin, cout, kernel size) of the network's convolutions, in parameter order
_UNET = [(16, 32, 3), (32, 32, 3), (32, 64, 3), (64, 64, 3), (64, 128, 3), (128, 128, 3),
         (128, 256, 3), (256, 256, 3), (256, 128, 1), (256, 128, 3), (128, 128, 3), (128, 64, 1),
         (128, 64, 3), (64, 64, 3), (64, 32, 1), (64, 32, 3), (32, 32, 3), (32, 16, 1)]


def _noise(rng, shape):
    g = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 30)))
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float32)


def _inputs(case, seed):
    """The case's input tensors by name, from the seed alone."""
    rng = _gen(seed, 1)
    kind = case["kind"]
    d = {}
    if kind == "unet":
        d["params"] = _he_params(rng)
        d["x"] = _unet_images(rng, case["batch"], case["size"])
        d["target"] = _unet_images(rng, case["batch"], case["size"])
        return d
    if kind == "batch":
        tr = [_trajectory(case, rng, inter=case["inter"] + (s % 3) - (1 if s == 1 else 0))
              for s in range(case["slices"])]
        # ragged: the later slices lose a few samples of their last readout
        tr = [tuple(a[:a.numel() - 13 * s].contiguous() for a in k) for s, k in enumerate(tr)]
        d["off"] = np.concatenate([[0], np.cumsum([k[0].numel() for k in tr])]).astype(int).tolist()
        for i, nm in enumerate(("kx", "ky", "kz", "t")):
            d[nm] = torch.cat([k[i] for k in tr]).contiguous()
        d["fm"] = torch.cat([_field_map(case, rng) for _ in range(case["slices"])]).contiguous()
    elif kind in ("tcg", "trecon"):
        d["t"] = torch.as_tensor(np.linspace(0.0, 0.010, 4096, endpoint=False,
                                             dtype=np.float32)).cuda()
    else:
        d["kx"], d["ky"], d["kz"], d["t"] = _trajectory(case, rng)
    if kind == "q":
        return d
    n = math.prod(_shape(case))
    if kind != "batch":
        d["fm"] = torch.zeros(n, device="cuda") if case.get("segs") == 0 else _field_map(case, rng)
    sens = _coil_maps(case, rng)
    d["sens"] = sens
    d["sr"], d["si"] = sens.real.contiguous().reshape(-1), sens.imag.contiguous().reshape(-1)
    if kind in ("ft", "ift", "bf", "batch"):
        d["ix"], d["iy"], d["iz"] = _positions(case)
    if kind == "ft":
        x = _phantom(case, rng)
        d["xr"], d["xi"] = x.real.contiguous(), x.imag.contiguous()
    elif kind in ("ift", "fhd", "bf", "batch"):
        m = d["t"].numel()
        # decaying k-space: amplitude falls with the time into the readout (the radius)
        slices = [(0, m)] if kind != "batch" else list(zip(d["off"][:-1], d["off"][1:]))
        parts = []
        for a, b in slices:
            amp = n * 0.2 / (1.0 + 60.0 * (d["t"][a:b] / 0.010) ** 1.5)
            parts.append((_noise(rng, (2, case["coils"], b - a)) * amp).reshape(2, -1))
        kd = torch.cat(parts, dim=1)
        d["kr"], d["ki"] = kd[0].contiguous(), kd[1].contiguous()
    elif kind in ("tcg", "trecon"):
        tau, t0 = _segments(case, d["t"])
        shape = _shape(case)
        g = math.prod(2 * v for v in shape)
        L1 = case["segs"] + 1
        d["qr"] = torch.empty(L1 * g, device="cuda")
        d["qi"] = torch.empty(L1 * g, device="cuda")
        for l, q in enumerate(_density_q(case, rng, tau, t0)):
            d["qr"][l * g:(l + 1) * g] = q.real.reshape(-1).float()
            d["qi"][l * g:(l + 1) * g] = q.imag.reshape(-1).float()
        xt = _phantom(case, rng)
        b = _aha(case, d, xt, torch.complex64)
        b = b + 0.01 * b.abs().square().mean().sqrt() * torch.complex(_noise(rng, (n,)),
                                                                       _noise(rng, (n,)))
        d["br"], d["bi"] = b.real.contiguous(), b.imag.contiguous()
        if kind == "tcg":
            x0 = 0.5 * xt + 0.02 * torch.complex(_noise(rng, (n,)), _noise(rng, (n,)))
            d["x0r"], d["x0i"] = x0.real.contiguous(), x0.imag.contiguous()
    return d


# the finite-difference weight of the iterative cases, relative to the operator's scale
_LAM_TOEP = 1e-2


def _bf_lam(case):
    return 1e-3 * case["inter"] * case["read"] * case["nz"]


def prepare(case, seed):
    imp = _package()
    d = _inputs(case, seed)
    kind = case["kind"]
    st = dict(case=case, imp=imp, d=d, ctx=imp.Context(0))
    n = 0 if kind == "unet" else math.prod(_shape(case))
    z = lambda m: torch.zeros(m, device="cuda")
    if kind == "ft":
        st["yr"], st["yi"] = (z(case["coils"] * d["t"].numel()) for _ in range(2))
    elif kind in ("ift", "fhd", "trecon", "tcg"):
        st["yr"], st["yi"] = z(n), z(n)
    elif kind == "bf":
        st["yr"], st["yi"] = z(n), z(n)
        st["opts"] = imp.bf_options(cg_num=case["cg"], fd_penalizer=_bf_lam(case),
                                    use_z=int(case["nz"] > 1),
                                    dims=(case["nx"], case["ny"], case["nz"]))
    elif kind == "batch":
        st["yr"], st["yi"] = z(case["slices"] * n), z(case["slices"] * n)
        st["opts"] = imp.bf_options(cg_num=case["cg"], fd_penalizer=_bf_lam(case),
                                    dims=(case["nx"], case["ny"], 1))
    elif kind == "q":
        g = (8 if case["nz"] > 1 else 4) * n * (case["segs"] + 1)
        st["yr"], st["yi"] = z(g), z(g)
    if kind in ("q", "fhd", "tcg", "trecon"):
        st["opts"] = imp.toeplitz_options(
            cg_num=case.get("cg", 8), ntime_segs=case["segs"], gridOS_Q=case.get("os_q", 1.125),
            gridOS_FH=case.get("os_fh", 1.5),
            fd_penalizer=_LAM_TOEP if kind in ("tcg", "trecon") else None)
    if kind == "unet":
        st["net"] = imp.UNet(st["ctx"], case["batch"], case["size"], case["size"], seed=0)
        st["net"].set_params(torch.as_tensor(d["params"]).cuda())
        st["out"] = torch.zeros_like(d["x"])
        st["grads"] = torch.zeros(d["params"].size, device="cuda")
    torch.cuda.synchronize()
    return st


def run(st):
    case, imp, d, ctx = st["case"], st["imp"], st["d"], st["ctx"]
    kind = case["kind"]
    if kind == "unet":
        if case["train"]:
            loss, grads = st["net"].gradients(d["x"], d["target"], st["grads"])
            return grads, loss
        return st["net"].forward(d["x"], st["out"])
    yr, yi, C = st["yr"], st["yi"], case.get("coils", 1)
    m = d["t"].numel()
    n = math.prod(_shape(case))
    dims = (case["nx"], case["ny"], case["nz"])
    z = int(case["nz"] > 1)
    if kind == "ft":
        geo = (d["kx"], d["ky"], d["kz"], d["ix"], d["iy"], d["iz"], d["fm"], d["t"], m, n)
        if C == 1:
            imp.ftGpu(ctx, yr, yi, d["xr"], d["xi"], *geo, use_z=z)
        else:
            imp.parallelFtGpu(ctx, yr, yi, d["xr"], d["xi"], *geo, d["sr"], d["si"], C, use_z=z)
    elif kind == "ift":
        geo = (d["kx"], d["ky"], d["kz"], d["ix"], d["iy"], d["iz"], d["fm"], d["t"], m, n)
        if C == 1:
            imp.iftGpu(ctx, yr, yi, d["kr"], d["ki"], *geo, use_z=z)
        else:
            imp.parallelIftGpu(ctx, yr, yi, d["kr"], d["ki"], *geo, d["sr"], d["si"], C, use_z=z)
    elif kind == "bf":
        yr.zero_()
        yi.zero_()
        imp.bruteForceGpu(ctx, st["opts"], yr, yi, d["kr"], d["ki"], d["kx"], d["ky"], d["kz"],
                          d["ix"], d["iy"], d["iz"], d["fm"], d["t"], d["sr"], d["si"], m, n, C, 1)
    elif kind == "batch":
        yr.zero_()
        yi.zero_()
        imp.bruteForceBatch(ctx, st["opts"], yr, yi, d["kr"], d["ki"], d["kx"], d["ky"], d["kz"],
                            d["t"], d["off"], d["ix"], d["iy"], d["iz"], d["fm"], d["sr"], d["si"],
                            n, C)
    elif kind == "q":
        imp.toeplitz_q(ctx, st["opts"], yr, yi, d["kx"], d["ky"], d["kz"], d["t"], m, *dims)
    elif kind == "fhd":
        imp.toeplitz_fhd(ctx, st["opts"], yr, yi, d["kr"], d["ki"], d["kx"], d["ky"], d["kz"],
                         d["t"], d["fm"], d["sr"], d["si"], m, C, *dims)
    elif kind == "trecon":
        imp.toeplitz_recon(ctx, st["opts"], yr, yi, d["br"], d["bi"], d["qr"], d["qi"], d["t"], m,
                           d["fm"], d["sr"], d["si"], C, *dims)
    elif kind == "tcg":
        yr.copy_(d["x0r"])
        yi.copy_(d["x0i"])
        imp.toeplitz_cg(ctx, st["opts"], yr, yi, d["br"], d["bi"], d["qr"], d["qi"], d["t"], m,
                        d["fm"], d["sr"], d["si"], C, *dims, tol=0.0, max_iter=case["cg"])
    return yr, yi


# ------------------------------------------------------------------ the work and its accuracy


def work(case):
    kind = case["kind"]
    if kind == "unet":
        h = case["size"]
        lv = [0, 0, 1, 1, 2, 2, 3, 3, 3, 2, 2, 2, 1, 1, 1, 0, 0, 0]
        macs = sum((h >> l) ** 2 * ci * co * k * k for (ci, co, k), l in zip(_UNET, lv))
        par = sum(ci * co * k * k + co for ci, co, k in _UNET)
        px = case["batch"] * 2 * h * h * 4
        if case["train"]:
            return dict(bytes=2 * px + 8 * par, flops=6 * macs * case["batch"])
        return dict(bytes=2 * px + 4 * par, flops=2 * macs * case["batch"])
    n, C = math.prod(_shape(case)), case.get("coils", 1)
    three = case["nz"] > 1
    if kind in ("ft", "ift", "bf", "batch"):
        m = case["inter"] * case["read"] * case["nz"] * case.get("slices", 1)
        applies = 1 if kind in ("ft", "ift") else 1 + 2 * (case["cg"] - 1)
        s = case.get("slices", 1)
        pair = 2 * ((4 if three else 3) + 4 * C)
        return dict(bytes=4 * (4 * m + 2 * C * m + s * 3 * n + 3 * n + 2 * C * n),
                    flops=pair * m * n * applies)
    g = (8 if three else 4) * n
    L1 = case["segs"] + 1
    if kind in ("q", "fhd"):
        m = case["inter"] * case["read"] * case["nz"]
        os = case["os_q"] if kind == "q" else case["os_fh"]
        dim = 3 if three else 2
        taps = (4 * os + 1) ** dim
        cells = (g if kind == "q" else n) * os ** dim
        fft = 5 * cells * math.log2(cells)
        if kind == "q":
            # a sample lies in at most two segments
            return dict(bytes=16 * m + 8 * g * L1, flops=2 * 2 * 2 * m * taps + L1 * fft)
        return dict(bytes=16 * m + 8 * C * m + 8 * C * n + 12 * n,
                    flops=C * (2 * 2 * 2 * m * taps + L1 * fft))
    # pruned forward and inverse transforms of the doubled grid per segment, coil and application
    part = (1 / 4 + 1 / 2 + 1) / 3 if three else (1 / 2 + 1) / 2
    apps = case["cg"] + 1
    return dict(bytes=8 * g * L1 + 8 * C * n + 4 * n + 8 * n * 3,
                flops=apps * L1 * C * (2 * 5 * g * math.log2(g) * part + 6 * g))


def tolerance(case):
    """About four times the distance between the FP32 (or BF16) path and the same in 64 bits."""
    kind = case["kind"]
    if kind in ("ft", "ift"):
        return {"rel": 1e-5}
    if kind in ("q", "fhd"):
        # the nearly real Q's imaginary part and the oversampled grids' cancelling edges
        return {"rel": 1e-4}
    if kind in ("bf", "batch"):
        return {"rel": 5e-5}
    if kind in ("tcg", "trecon"):
        return {"rel": 2e-5}
    # BF16 activations through 18 layers
    return {"rel": 4e-2} if case["train"] else {"rel": 2e-2}


# ------------------------------------------------------------------ the same in 64 bits


def _aha(case, d, p, ctype):
    """A^H A p = sum_l conj(e_l) sum_c conj(S_c) crop(ifft(Qf_l fft(pad(e_l S_c p))))."""
    shape = _shape(case)
    two = tuple(2 * v for v in shape)
    axes = tuple(range(len(shape)))
    g = math.prod(two)
    rtype = torch.float64 if ctype == torch.complex128 else torch.float32
    tau, t0 = _segments(case, d["t"])
    out = torch.zeros(shape, dtype=ctype, device="cuda")
    fm = d["fm"].double().reshape(shape)
    sens = d["sens"].to(ctype).reshape((case["coils"],) + shape)
    p = p.to(ctype).reshape(shape)
    crop = tuple(slice(0, v) for v in shape)
    for l in range(case["segs"] + 1):
        q = torch.complex(d["qr"][l * g:(l + 1) * g].to(rtype),
                          d["qi"][l * g:(l + 1) * g].to(rtype)).reshape(two)
        qf = torch.fft.fftn(torch.fft.ifftshift(q, dim=axes), dim=axes)
        ph = -fm * (tau * l + t0)
        e = torch.polar(torch.ones_like(ph), ph).to(ctype)
        for c in range(case["coils"]):
            f = torch.fft.fftn(sens[c] * e * p, s=two, dim=axes)
            out += (sens[c] * e).conj() * torch.fft.ifftn(qf * f, dim=axes)[crop]
    return out.reshape(-1)


def _dhd(case, x):
    """D^H D x: periodic first differences along every image axis."""
    shape = _shape(case)
    v = x.reshape(shape)
    out = torch.zeros_like(v)
    for a in range(len(shape)):
        out += 2 * v - torch.roll(v, 1, a) - torch.roll(v, -1, a)
    return out.reshape(-1)


def _toep_exact(case, d, L0):
    b = torch.complex(d["br"].double(), d["bi"].double())
    x = torch.zeros_like(b) if L0 is None else L0
    op = lambda v: _aha(case, d, v, torch.complex128) + _LAM32 * _dhd(case, v)
    r = b - op(x)
    p = r.clone()
    best, rb = x.clone(), float(r.abs().square().sum())
    beta = rb
    if L0 is None:
        best = torch.zeros_like(b)
    for _ in range(case["cg"]):
        q = op(p)
        alpha = beta / float((p.conj() * q).real.sum())
        x = x + alpha * p
        r = r - alpha * q
        bn = float(r.abs().square().sum())
        if bn < rb:
            rb, best = bn, x.clone()
        p = r + (bn / beta) * p
        beta = bn
    return best


_LAM32 = float(np.float32(_LAM_TOEP))


def _nudft(case, k, pos, fm, t, v, adjoint):
    """F ([N][C] -> [M][C]) or F^H ([M][C] -> [N][C]) in complex128, in blocks of samples."""
    z = case["nz"] > 1
    kk = torch.stack([k[0], k[1], k[2] if z else 0 * k[2]]).double()
    pp = torch.stack([pos[0], pos[1], pos[2]]).double()
    n, m = pp.shape[1], kk.shape[1]
    out = torch.zeros(n if adjoint else m, v.shape[1], dtype=torch.complex128, device="cuda")
    blk = max(1, (1 << 27) // n)
    w = fm.double()[None, :]
    for a in range(0, m, blk):
        ph = TWO_PI * (kk[:, a:a + blk].T @ pp) + t[a:a + blk].double()[:, None] * w
        if adjoint:
            e = torch.polar(torch.ones_like(ph), ph)
            out += e.T @ v[a:a + blk]
        else:
            e = torch.polar(torch.ones_like(ph), -ph)
            out[a:a + blk] = e @ v
    return out


def _bf_exact(case, d, sl):
    n, C = math.prod(_shape(case)), case["coils"]
    a, b = (0, d["t"].numel()) if sl is None else (d["off"][sl], d["off"][sl + 1])
    k = (d["kx"][a:b], d["ky"][a:b], d["kz"][a:b])
    t = d["t"][a:b]
    fm = d["fm"] if sl is None else d["fm"][sl * n:(sl + 1) * n]
    pos = (d["ix"], d["iy"], d["iz"])
    S = d["sens"].to(torch.complex128).T
    kd = torch.complex(d["kr"][C * a:C * b].double(), d["ki"][C * a:C * b].double())
    y = kd.reshape(C, b - a).T
    lam = float(np.float32(_bf_lam(case)))
    x = torch.zeros(n, dtype=torch.complex128, device="cuda")
    af = torch.zeros_like(y)
    dirn, old = torch.zeros_like(x), 0.0
    for _ in range(case["cg"] - 1):
        g = (S.conj() * _nudft(case, k, pos, fm, t, y - af, True)).sum(1) - lam * _dhd(case, x)
        gg = float(g.abs().square().sum())
        dirn = g + (gg / old if old else 0.0) * dirn
        old = gg
        q = _nudft(case, k, pos, fm, t, S * dirn[:, None], False)
        den = float(q.abs().square().sum()) + lam * float((dirn.conj() * _dhd(case, dirn)).real.sum())
        alpha = float((dirn.conj() * g).real.sum()) / den
        af = af + alpha * q
        x = x + alpha * dirn
    return x


def _i0(x):
    """The modified Bessel function by the Abramowitz-Stegun polynomials 9.8.1 and 9.8.2, which
    define the gridding kernel."""
    y = (x / 3.75) ** 2
    small = 1.0 + y * (3.5156229 + y * (3.0899424 + y * (1.2067492 + y * (0.2659732 + y * (
        0.360768e-1 + y * 0.45813e-2)))))
    u = 3.75 / x.clamp_min(3.75)
    big = torch.exp(x) / torch.sqrt(x.clamp_min(3.75)) * (0.39894228 + u * (0.1328592e-1 + u * (
        0.225319e-2 + u * (-0.157565e-2 + u * (0.916281e-2 + u * (-0.2057706e-1 + u * (
            0.2635537e-1 + u * (-0.1647633e-1 + u * 0.392377e-2))))))))
    return torch.where(x < 3.75, small, big)


def _grid_exact(img, os, kscale, beta_after, k, w, data):
    """Images [img x, img y(, img z)][C] of Kaiser-Bessel gridding (width 4) of data [M][C]
    weighted by w: unnormalised inverse FFT, crop, deapodisation."""
    f32 = np.float32
    if img[2] == 1:
        osr = f32(2.0) * f32(np.ceil(f32(f32(os) * f32(img[0])) / f32(2.0))) / f32(img[0])
    else:
        osr = f32(4.0) * f32(np.ceil(f32(f32(os) * f32(img[2])) / f32(4.0))) / f32(img[2])
    beat = lambda o: math.pi * math.sqrt((o - 0.5) ** 2 * 64.0 / (o * o) - 0.8)
    beta = beat(float(osr)) if beta_after else beat(float(f32(os)))
    dim = 2 if img[2] == 1 else 3
    gs = [int(np.ceil(f32(osr * f32(v)))) for v in img[:dim]]
    for a in range(2):
        gs[a] += gs[a] % 2
    osd = float(osr)
    keep = w != 0
    val = w[keep, None] * data[keep]
    axes = []
    reach = int(math.ceil(2.0 * osd)) + 1
    for a in range(dim):
        c = osd * (kscale * k[a][keep].double() + 0.5 * img[a])
        base = torch.floor(c).long()
        ent = []
        for o in range(-reach, reach + 1):
            i = base + o
            dist = (c - i).abs() / osd
            arg = 1.0 - 0.25 * dist * dist
            ww = torch.where((dist <= 2.0) & (i >= 0) & (i < gs[a]),
                             _i0(beta * torch.sqrt(arg.clamp_min(0.0))) / 4.0, torch.zeros_like(c))
            ent.append((i.clamp(0, gs[a] - 1), ww))
        axes.append(ent)
    C = data.shape[1]
    grid = torch.zeros(math.prod(gs), 2 * C, dtype=torch.float64, device="cuda")
    v2 = torch.view_as_real(val).reshape(-1, 2 * C)
    for ix, wx in axes[0]:
        for iy, wy in axes[1]:
            if dim == 2:
                grid.index_add_(0, ix * gs[1] + iy, v2 * (wx * wy)[:, None])
            else:
                base, wxy = (ix * gs[1] + iy) * gs[2], wx * wy
                for iz, wz in axes[2]:
                    grid.index_add_(0, base + iz, v2 * (wxy * wz)[:, None])
    grid = torch.view_as_complex(grid.reshape(gs + [C, 2]))
    ax = tuple(range(dim))
    im = torch.fft.fftshift(torch.fft.ifftn(torch.fft.ifftshift(grid, dim=ax), dim=ax,
                                            norm="forward"), dim=ax)
    for a in range(dim):
        o = gs[a] // 2 - img[a] // 2
        im = im.narrow(a, o, img[a])
        u = (torch.arange(img[a], device="cuda", dtype=torch.float64) - 0.5 * img[a]) / img[a]
        e = (math.pi * 4.0 * u) ** 2 - beta * beta
        s = torch.sqrt(e.abs())
        kb = torch.where(e > 0, torch.sin(s) / s, torch.sinh(s) / s)
        im = im / kb.reshape([-1 if b == a else 1 for b in range(im.dim())]) / osd
    return im


def _hanning(t, tau, l, t0):
    x = t.double() - tau * l - t0
    return torch.where(x.abs() < tau, 0.5 + 0.5 * torch.cos(math.pi * x / tau), torch.zeros_like(x))


def _unet_exact(case, d):
    """The network in float64 (no rounding to BF16 anywhere)."""
    F = torch.nn.functional
    B, n = case["batch"], case["size"]
    p = torch.as_tensor(d["params"]).cuda().double()
    leaves, off = [], 0
    for ci, co, k in _UNET:
        w = p[off:off + co * k * k * ci].reshape(co, k, k, ci).permute(0, 3, 1, 2).contiguous()
        off += co * k * k * ci
        leaves.append((w.requires_grad_(case["train"]),
                       p[off:off + co].clone().requires_grad_(case["train"])))
        off += co

    def conv(i, h, relu=True):
        w, b = leaves[i]
        # the border padding and the 64-bit sums as one matrix product per kernel tap
        k = _UNET[i][2]
        hp = F.pad(h, (k // 2,) * 4)
        y = b.reshape(1, -1, 1, 1)
        for dy in range(k):
            for dx in range(k):
                y = y + torch.einsum("oc,bchw->bohw", w[:, :, dy, dx],
                                     hp[:, :, dy:dy + h.shape[2], dx:dx + h.shape[3]])
        return F.relu(y) if relu else y

    def net(img):
        x = torch.zeros(1, 16, n, n, dtype=torch.float64, device="cuda")
        x[:, :2] = img.double().reshape(1, 2, n, n)
        up = lambda h: F.interpolate(h, scale_factor=2, mode="nearest")
        s1 = conv(1, conv(0, x))
        s2 = conv(3, conv(2, F.max_pool2d(s1, 2)))
        s3 = conv(5, conv(4, F.max_pool2d(s2, 2)))
        m = conv(7, conv(6, F.max_pool2d(s3, 2)))
        f = conv(10, conv(9, torch.cat([s3, up(conv(8, m, False))], 1)))
        f = conv(13, conv(12, torch.cat([s2, up(conv(11, f, False))], 1)))
        f = conv(16, conv(15, torch.cat([s1, up(conv(14, f, False))], 1)))
        return conv(17, f, False)[:, :2].reshape(1, 2, n * n)

    if not case["train"]:
        return torch.cat([net(d["x"][b]) for b in range(B)])
    total = 0.0
    for b in range(B):  # one image at a time: the tape of a batch would not fit
        loss = (net(d["x"][b]) - d["target"][b].double()).square().sum() / d["x"].numel()
        loss.backward()
        total += float(loss.detach())
    grads = torch.cat([torch.cat([w.grad.permute(0, 2, 3, 1).reshape(-1), v.grad])
                       for w, v in leaves])
    return grads, total


def exact(case, seed):
    kind = case["kind"]
    d = _inputs(case, seed)
    if kind == "unet":
        return _unet_exact(case, d)
    split = lambda v: (v.real.reshape(-1), v.imag.reshape(-1))
    C = case.get("coils", 1)
    if kind in ("ft", "ift"):
        k, pos = (d["kx"], d["ky"], d["kz"]), (d["ix"], d["iy"], d["iz"])
        S = d["sens"].to(torch.complex128).T
        if kind == "ft":
            x = torch.complex(d["xr"].double(), d["xi"].double())
            return split(_nudft(case, k, pos, d["fm"], d["t"], S * x[:, None], False).T)
        y = torch.complex(d["kr"].double(), d["ki"].double()).reshape(C, -1).T.contiguous()
        return split((S.conj() * _nudft(case, k, pos, d["fm"], d["t"], y, True)).sum(1))
    if kind == "bf":
        return split(_bf_exact(case, d, None))
    if kind == "batch":
        return split(torch.cat([_bf_exact(case, d, s) for s in range(case["slices"])]))
    if kind in ("q", "fhd"):
        tau, t0 = _segments(case, d["t"])
        three = case["nz"] > 1
        k = (d["kx"], d["ky"], d["kz"])
        order = (1, 0, 2) if three else (0, 1)
        img = [case["nx"], case["ny"], case["nz"]]
        one = torch.ones(d["t"].numel(), 1, dtype=torch.complex128, device="cuda")
        if kind == "q":
            img = [2 * case["nx"], 2 * case["ny"], 2 * case["nz"] if three else 1]
            qs = [_grid_exact(img, case["os_q"], 2.0, True, k, _hanning(d["t"], tau, l, t0),
                              one)[..., 0].permute(order).reshape(-1)
                  for l in range(case["segs"] + 1)]
            return split(torch.cat(qs))
        y = torch.complex(d["kr"].double(), d["ki"].double()).reshape(C, -1).T.contiguous()
        S = d["sens"].to(torch.complex128).T
        acc = torch.zeros(math.prod(img), dtype=torch.complex128, device="cuda")
        for l in range(case["segs"] + 1):
            im = _grid_exact(img, case["os_fh"], 1.0, False, k, _hanning(d["t"], tau, l, t0), y)
            im = im.permute(order + (im.dim() - 1,)).reshape(-1, C)
            ph = d["fm"].double() * (tau * l + t0)
            acc += torch.polar(torch.ones_like(ph), ph) * (S.conj() * im).sum(1)
        return split(acc)
    if kind == "tcg":
        return split(_toep_exact(case, d, torch.complex(d["x0r"].double(), d["x0i"].double())))
    return split(_toep_exact(case, d, None))
