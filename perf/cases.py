"""Workloads of the framework, each one pass through its public entry points.

The cases are what users of the package run: projecting maps (matching, training with gradients,
several maps at once), reconstructing maps from images, fitting a map and its orientations to central
slices, inserting slices (plain, CTF-weighted, many volumes of uneven size), and sampling and splatting
subvolumes at arbitrary coordinates.  ``listed()`` names twelve of them; ``draw()`` gives others of the
same families over the same ranges of sizes and options.

A case is a dict of plain values.  ``kind`` selects the family; ``d`` is the box size, ``n`` the number
of rotations, slices, images or subvolumes.  Options, where a family has them:

    pad         pad factor of the real-space wrappers
    fmax        fftfreq_max (0: none)
    grad        also the backward pass: gradients of every differentiable input
    f64         float64 volume (projection), float64 rotation matrices (elsewhere)
    c128        complex128 slices (insertion)
    det         deterministic insertion / volume gradient
    channels    maps sharing one set of rotations (0: the single-map function)

Volumes are sums of Gaussian blobs with white noise, slices and images noise under a falling amplitude
envelope as experimental spectra have, rotations uniform on SO(3), all made on the GPU from the seed.
"""

import math

import torch
import torch.nn.functional as F

from teamtomo_b200.batched import (
    ctf_params,
    extract_central_slices_rfft_3d_batched,
    insert_central_slices_rfft_3d_batched,
)
from teamtomo_b200.losses import central_slice_mse
from teamtomo_b200.torch_fourier_slice import (
    backproject_2d_to_3d,
    backproject_2d_to_3d_multichannel,
    extract_central_slices_rfft_3d,
    insert_central_slices_rfft_3d,
    project_3d_to_2d,
    project_3d_to_2d_multichannel,
)
from teamtomo_b200.torch_image_interpolation import insert_into_image_3d, sample_image_3d

DEV = "cuda"


def listed():
    return [
        # one small map at a hundred orientations: the interactive call, bound by latency and launches
        {"name": "project_small", "kind": "project", "d": 64, "n": 100, "pad": 2.0, "fmax": 0.0, "grad": False,
         "f64": False, "channels": 0},
        # a training step that goes through the projection operator: gradients of map and orientations
        {"name": "project_train", "kind": "project", "d": 90, "n": 256, "pad": 2.0, "fmax": 0.0, "grad": True,
         "f64": False, "channels": 0},
        # projections of two half maps with the same orientations
        {"name": "project_half_maps", "kind": "project", "d": 160, "n": 400, "pad": 2.0, "fmax": 0.0, "grad": False,
         "f64": False, "channels": 2},
        # reconstruction from a particle stack
        {"name": "backproject_stack", "kind": "backproject", "d": 128, "n": 10000, "pad": 2.0, "fmax": 0.0,
         "channels": 0},
        # a handful of slices up to a resolution limit: the smallest call on the Fourier-space functions
        {"name": "extract_few", "kind": "extract", "d": 96, "n": 8, "fmax": 0.37, "grad": False, "f64": True,
         "det": False},
        # slices of a 256 box at 4096 orientations with gradients of volume and orientations
        {"name": "extract_fit", "kind": "extract", "d": 256, "n": 4096, "fmax": 0.0, "grad": True, "f64": False,
         "det": False},
        # the insertion of as many slices
        {"name": "insert_full", "kind": "insert", "d": 256, "n": 4096, "fmax": 0.0, "grad": False, "c128": False,
         "det": False},
        # one step of map and pose refinement with the fused loss
        {"name": "mse_refine", "kind": "mse", "d": 162, "n": 3000, "fmax": 0.43, "f64": True},
        # CTF-weighted extraction and insertion of several particles classes of uneven box size
        {"name": "batched_ctf", "kind": "batched", "boxes": "64,96,128,160,200,256",
         "counts": "2000,1500,1200,700,800,500", "extract": True},
        # CTF-weighted insertion of a large box at full scale
        {"name": "insert_ctf_large", "kind": "batched", "boxes": "320", "counts": "8192", "extract": False},
        # rotated subvolumes sampled from a tomogram, with gradients of tomogram and positions
        {"name": "sample_subvolumes", "kind": "sample", "dz": 200, "dy": 400, "dx": 400, "d": 64, "n": 64,
         "dtype": "float32", "channels": 1, "grad": True, "nearest": False},
        # planes of complex Fourier samples splatted at explicit coordinates
        {"name": "splat_planes", "kind": "splat", "d": 192, "n": 500, "dtype": "complex64", "grad": False,
         "nearest": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["project", "project", "backproject", "extract", "extract", "insert", "insert", "mse",
                       "batched", "sample", "splat"])
    fmax = rng.choice([0.0, 0.0, round(rng.uniform(0.2, 0.49), 3) + 0.0003])
    if kind == "project":
        d = _log_int(rng, 24, 160)
        channels = rng.choice([0, 0, 0, 1, 2, 3])
        grad = rng.random() < 0.4
        pad = rng.choice([1.0, 1.5, 2.0, 2.0])
        n = _log_int(rng, 1, max(2, min(2000, 40_000_000 // (d * d * 4 * max(channels, 1)))))
        return {"kind": kind, "d": d, "n": n, "pad": pad, "fmax": fmax, "grad": grad,
                "f64": rng.random() < 0.15, "channels": channels}
    if kind == "backproject":
        d = _log_int(rng, 24, 160)
        channels = rng.choice([0, 0, 1, 2])
        pad = rng.choice([1.0, 1.5, 2.0, 2.0])
        n = _log_int(rng, 8, max(16, min(10000, 160_000_000 // (d * d * max(channels, 1)))))
        return {"kind": kind, "d": d, "n": n, "pad": pad, "fmax": fmax, "channels": channels}
    if kind in ("extract", "insert", "mse"):
        d = _log_int(rng, 24, 320)
        n = _log_int(rng, 1, max(2, min(8192, 200_000_000 // (d * (d // 2 + 1)))))
        if kind == "extract":
            return {"kind": kind, "d": d, "n": n, "fmax": fmax, "grad": rng.random() < 0.6,
                    "f64": rng.random() < 0.3, "det": rng.random() < 0.15}
        if kind == "insert":
            c128 = rng.random() < 0.12
            return {"kind": kind, "d": d, "n": n // 4 + 1 if c128 else n, "fmax": fmax, "grad": rng.random() < 0.35,
                    "c128": c128, "det": not c128 and rng.random() < 0.2}
        return {"kind": kind, "d": d, "n": n, "fmax": fmax, "f64": rng.random() < 0.3}
    if kind == "batched":
        boxes = [_log_int(rng, 24, 288) for _ in range(rng.randint(1, 8))]
        counts = [_log_int(rng, 1, max(2, min(4000, 30_000_000 // (b * (b // 2 + 1))))) for b in boxes]
        return {"kind": kind, "boxes": ",".join(map(str, boxes)), "counts": ",".join(map(str, counts)),
                "extract": rng.random() < 0.7}
    dtype = rng.choice(["float32", "float32", "complex64"])
    nearest = rng.random() < 0.15
    grad = not nearest and rng.random() < 0.5
    if kind == "sample":
        d = _log_int(rng, 12, 96)
        return {"kind": kind, "dz": _log_int(rng, 40, 240), "dy": _log_int(rng, 60, 400),
                "dx": _log_int(rng, 60, 400), "d": d, "n": _log_int(rng, 1, max(2, min(400, 16_000_000 // d**3))),
                "dtype": dtype, "channels": rng.choice([1, 1, 1, 2, 3]), "grad": grad, "nearest": nearest}
    d = _log_int(rng, 24, 256)
    return {"kind": kind, "d": d, "n": _log_int(rng, 1, max(2, min(1000, 12_000_000 // (d * (d // 2 + 1))))),
            "dtype": dtype, "grad": grad, "nearest": nearest}


# ------------------------------------------------------------------ inputs


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _blobs(g, shape, blobs=20):
    """Gaussian blobs (sigma 2 to 6 voxels of a 64 box) in the middle of the box, with white noise."""
    scale = min(shape) / 64
    sigma = (2 + 4 * torch.rand(blobs, generator=g, device=DEV)) * scale
    axes = []
    for n in shape:
        centre = n / 2 + (torch.rand(blobs, generator=g, device=DEV) - 0.5) * 0.6 * n
        x = torch.arange(n, device=DEV, dtype=torch.float32)
        axes.append(torch.exp(-((x - centre[:, None]) ** 2) / (2 * sigma[:, None] ** 2)))
    vol = torch.einsum("bz,by,bx->zyx", *axes)
    return vol + 0.01 * torch.randn(shape, generator=g, device=DEV)


def _rfft_volume(vol):
    dft = torch.fft.rfftn(torch.fft.fftshift(vol, dim=(-3, -2, -1)), dim=(-3, -2, -1))
    return torch.fft.fftshift(dft, dim=(-3, -2)).contiguous()


def _rotations(g, n, f64=False):
    """Uniform on SO(3), from unit quaternions."""
    q = torch.randn((n, 4), generator=g, device=DEV, dtype=torch.float64)
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], dim=1).reshape(n, 3, 3)
    return R if f64 else R.to(torch.float32)


def _spectra(g, n, d, scale=1.0, dtype=torch.complex64):
    """Noise slices (n, d, d//2+1) under a falling amplitude envelope (rows fftshifted)."""
    ky = torch.arange(d, device=DEV, dtype=torch.float32) - d // 2
    kx = torch.arange(d // 2 + 1, device=DEV, dtype=torch.float32)
    k = torch.sqrt(ky[:, None] ** 2 + kx**2)
    env = scale * (0.05 + 10.0 / (1.0 + k) ** 1.5)
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    out = torch.empty((n, d, d // 2 + 1, 2), device=DEV, dtype=real)
    out.normal_(generator=g)
    out *= env[:, :, None]
    return torch.view_as_complex(out)


def _ctf(g, n):
    defocus = 0.5 + 2.5 * torch.rand(n, generator=g, device=DEV)
    astigmatism = 0.05 * torch.rand(n, generator=g, device=DEV)
    angle = 180.0 * torch.rand(n, generator=g, device=DEV)
    return ctf_params(defocus.cpu(), astigmatism.cpu(), angle.cpu(), n=n, device=DEV)


def _box_grid(d):
    ax = torch.arange(d, device=DEV, dtype=torch.float32) - d // 2
    return torch.stack(torch.meshgrid(ax, ax, ax, indexing="ij"), dim=-1)


def _ints(text):
    return [int(x) for x in str(text).split(",")]


def _inputs(case, seed):
    """The tensors of a case, from the seed alone."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "project":
        d, n, c = case["d"], case["n"], case["channels"]
        vol = torch.stack([_blobs(g, (d, d, d)) for _ in range(max(c, 1))])
        vol = (vol if c else vol[0]).to(torch.float64 if case["f64"] else torch.float32)
        s = {"volume": vol, "R": _rotations(g, n)}
        if case["grad"]:
            odd = int((d * (case["pad"] - 1.0)) // 2) * 2 + d
            w = 2 * (odd // 2) - (odd - d)  # an odd padded box gives images one column narrower
            s["G"] = torch.randn((n, c, d, w) if c else (n, d, w), generator=g, device=DEV).to(vol.dtype)
        return s
    if kind == "backproject":
        d, n, c = case["d"], case["n"], case["channels"]
        shape = (n, c, d, d) if c else (n, d, d)
        blob = _blobs(g, (max(1, min(n, 8)), d, d), blobs=12)
        images = torch.randn(shape, generator=g, device=DEV)
        images += 3.0 * (blob[torch.arange(n, device=DEV) % blob.shape[0]][:, None] if c
                         else blob[torch.arange(n, device=DEV) % blob.shape[0]])
        return {"images": images, "R": _rotations(g, n)}
    if kind == "extract":
        d, n = case["d"], case["n"]
        s = {"volume": _rfft_volume(_blobs(g, (d, d, d))), "R": _rotations(g, n, case["f64"])}
        if case["grad"]:
            s["G"] = _spectra(g, n, d, 1e-3)
        return s
    if kind == "insert":
        d, n = case["d"], case["n"]
        dt = torch.complex128 if case["c128"] else torch.complex64
        s = {"images": _spectra(g, n, d, dtype=dt), "R": _rotations(g, n)}
        if case["grad"]:
            s["G"] = _rfft_volume(_blobs(g, (d, d, d))).to(dt)
        return s
    if kind == "mse":
        d, n = case["d"], case["n"]
        return {"volume": _rfft_volume(_blobs(g, (d, d, d))), "R": _rotations(g, n, case["f64"]),
                "targets": _spectra(g, n, d, d)}
    if kind == "batched":
        boxes, counts = _ints(case["boxes"]), _ints(case["counts"])
        s = {"R": [_rotations(g, n) for n in counts], "ctf": [_ctf(g, n) for n in counts],
             "images": [_spectra(g, n, b) for b, n in zip(boxes, counts)]}
        if case["extract"]:
            s["volumes"] = [_rfft_volume(_blobs(g, (b, b, b))) for b in boxes]
        return s
    dtype = getattr(torch, case["dtype"])
    if kind == "sample":
        shape, d, n, c = (case["dz"], case["dy"], case["dx"]), case["d"], case["n"], case["channels"]
        vol = torch.stack([_blobs(g, shape, blobs=8) for _ in range(c)])
        if dtype == torch.complex64:
            vol = torch.complex(vol, torch.randn(vol.shape, generator=g, device=DEV))
        size = torch.tensor(shape, device=DEV, dtype=torch.float32)
        centre = torch.rand((n, 3), generator=g, device=DEV) * (size - 1)
        R = _rotations(g, n)
        coords = torch.einsum("nij,zyxj->nzyxi", R, _box_grid(d)) + centre[:, None, None, None]
        s = {"image": vol if c > 1 else vol[0], "coords": coords.contiguous()}
        if case["grad"]:
            lead = tuple(coords.shape[:-1])
            G = torch.randn(lead + ((c,) if c > 1 else ()), generator=g, device=DEV)
            s["G"] = torch.complex(G, G.flip(0)) if dtype == torch.complex64 else G
        return s
    # planes of a half-transform at random orientations, redirected into its stored half
    d, n = case["d"], case["n"]
    y = torch.arange(d, device=DEV, dtype=torch.float32) - d // 2
    x = torch.arange(d // 2 + 1, device=DEV, dtype=torch.float32)
    R = _rotations(g, n)
    p = y[None, :, None, None] * R[:, None, None, :, 1] + x[None, None, :, None] * R[:, None, None, :, 2]
    p = torch.where(p[..., 2:] < 0, -p, p)
    coords = p + torch.tensor([d // 2, d // 2, 0], device=DEV, dtype=torch.float32)
    vals = _spectra(g, n, d)
    s = {"values": vals if dtype == torch.complex64 else vals.real.contiguous(), "coords": coords.contiguous(),
         "shape": (d, d, d // 2 + 1)}
    if case["grad"]:
        G = torch.randn(s["shape"], generator=g, device=DEV)
        s["G"] = torch.complex(G, G.flip(0)) if dtype == torch.complex64 else G
    return s


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    for key in {"project": ("volume", "R"), "extract": ("volume", "R"), "insert": ("images",),
                "sample": ("image", "coords"), "splat": ("values",)}.get(case["kind"], ()):
        if case["grad"]:
            s[key].requires_grad_(True)
    if case["kind"] == "mse":
        s["volume"].requires_grad_(True)
        s["R"].requires_grad_(True)
    return s


# --------------------------------------------------------------------- run


def run(s):
    case = s["case"]
    kind = case["kind"]
    fmax = case.get("fmax") or None
    d = case.get("d")
    if kind == "project":
        fn = project_3d_to_2d_multichannel if case["channels"] else project_3d_to_2d
        out = fn(s["volume"], s["R"], pad_factor=case["pad"], fftfreq_max=fmax)
        return _with_grads(out, s, ("volume", "R"))
    if kind == "backproject":
        fn = backproject_2d_to_3d_multichannel if case["channels"] else backproject_2d_to_3d
        return {"out": fn(s["images"], s["R"], pad_factor=case["pad"], fftfreq_max=fmax)}
    if kind == "extract":
        out = extract_central_slices_rfft_3d(s["volume"], (d, d, d), s["R"], fftfreq_max=fmax,
                                             deterministic=case["det"])
        return _with_grads(out, s, ("volume", "R"))
    if kind == "insert":
        out, weights = insert_central_slices_rfft_3d(s["images"], (d, d, d), s["R"], fftfreq_max=fmax,
                                                     deterministic=case["det"])
        return _with_grads(out, s, ("images",), weights=weights)
    if kind == "mse":
        loss = central_slice_mse(s["volume"], (d, d, d), s["R"], s["targets"], fftfreq_max=fmax)
        gv, gr = torch.autograd.grad(loss, [s["volume"], s["R"]])
        return {"out": loss.detach(), "volume": gv, "R": gr}
    if kind == "batched":
        r = {"inserted": insert_central_slices_rfft_3d_batched(s["images"], s["R"], ctf=s["ctf"])}
        if case["extract"]:
            r["slices"] = extract_central_slices_rfft_3d_batched(s["volumes"], s["R"], ctf=s["ctf"])
        return r
    mode = "nearest" if case["nearest"] else "trilinear"
    if kind == "sample":
        return _with_grads(sample_image_3d(s["image"], s["coords"], mode), s, ("image", "coords"))
    image = torch.zeros(s["shape"], dtype=s["values"].dtype, device=DEV)
    out, weights = insert_into_image_3d(s["values"], s["coords"], image, interpolation=mode)
    return _with_grads(out, s, ("values",), weights=weights)


def _with_grads(out, s, names, **more):
    r = {"out": out.detach(), **more}
    if s["case"]["grad"]:
        for name, g in zip(names, torch.autograd.grad(out, [s[k] for k in names], grad_outputs=s["G"])):
            r[name] = g
    return r


# -------------------------------------------------------------------- work


def _fft_flops(points, transform):
    """A real transform of ``points`` points in sub-transforms of ``transform`` points."""
    return 2.5 * points * math.log2(max(2, transform))


def work(case):
    """Every input read once and every output written once; operations per slice pixel or point: its
    position (about 30) and a trilinear sum over eight corners."""
    kind = case["kind"]
    d, n = case.get("d", 0), case.get("n", 0)
    pixels, voxels = n * d * (d // 2 + 1), d * d * (d // 2 + 1)
    if kind in ("project", "backproject"):
        c = max(case["channels"], 1)
        size = 8 if case.get("f64") else 4
        e = d + 2 * int((d * (case["pad"] - 1.0)) // 2)
        bytes_ = c * size * (d**3 + n * d * d) + 36 * n
        flops = c * (_fft_flops(e**3, e**3) + n * _fft_flops(e * e, e * e)) + n * e * (e // 2 + 1) * (30 + 32 * c)
        if case.get("grad"):
            bytes_, flops = 2 * bytes_, 2.5 * flops
        return {"bytes": bytes_, "flops": flops}
    if kind == "extract":
        k = 2 if case["grad"] else 1
        return {"bytes": k * (8 * voxels + 8 * pixels + 36 * n), "flops": pixels * (190 if case["grad"] else 62)}
    if kind == "insert":
        size = 16 if case["c128"] else 8
        k = 1 + int(case["grad"])
        return {"bytes": k * size * (voxels + pixels) + size // 2 * voxels, "flops": pixels * 80 * k}
    if kind == "mse":
        return {"bytes": 16 * voxels + 8 * pixels + 72 * n, "flops": pixels * 170}
    if kind == "batched":
        k = 2 if case["extract"] else 1
        bytes_ = flops = 0
        for b, m in zip(_ints(case["boxes"]), _ints(case["counts"])):
            px, vx = m * b * (b // 2 + 1), b * b * (b // 2 + 1)
            bytes_ += k * 8 * (px + vx) + 4 * vx
            flops += px * 120 * k
        return {"bytes": bytes_, "flops": flops}
    size = 4 if case["dtype"] == "float32" else 8
    k = 2 if case["grad"] else 1
    if kind == "sample":
        points, vox, c = n * d**3, case["dz"] * case["dy"] * case["dx"], case["channels"]
        return {"bytes": k * (12 * points + size * c * (points + vox)),
                "flops": points * (20 + 4 * size * c) * (2.5 if k == 2 else 1)}
    return {"bytes": 12 * pixels + k * size * (pixels + voxels) + 4 * voxels, "flops": pixels * (20 + 6 * size) * k}


# ------------------------------------------- the same results in 64 bits

CHUNK = 3_000_000  # slice pixels worked on at a time


def _freqs(h, w):
    qy = torch.fft.fftshift(torch.fft.fftfreq(h, dtype=torch.float64, device=DEV))
    return qy, torch.fft.rfftfreq(w, dtype=torch.float64, device=DEV)


def _keep(qy, qx, fmax):
    q = torch.sqrt(qy[:, None] ** 2 + qx**2)
    return torch.ones_like(q, dtype=torch.bool) if not fmax else q <= fmax


def _plane(R, qy, qx):
    """Rotated zyx frequencies of a central slice: three (n, h, w) arrays; R acts on zyx vectors."""
    return [R[:, i, 1, None, None] * qy[:, None] + R[:, i, 2, None, None] * qx for i in range(3)]


def _array_coords(p, shape):
    d, h, w = shape
    return [(p[0] + 0.5) / (1 - 1 / d) * (d - 1), (p[1] + 0.5) / (1 - 1 / h) * (h - 1), p[2] * 2 * (w // 2)]


def _corners(c, dims):
    """Index and weight of the eight corners of points c inside an array of shape ``dims``."""
    lo = [torch.floor(x.detach()).clamp(0, n - 1) for x, n in zip(c, dims)]
    t = [x - f for x, f in zip(c, lo)]
    for k in range(8):
        bits = (k >> 2 & 1, k >> 1 & 1, k & 1)
        at = [(f.long() + b).clamp(max=n - 1) for f, b, n in zip(lo, bits, dims)]
        w = 1.0
        for x, b in zip(t, bits):
            w = w * (x if b else 1 - x)
        yield (at[0] * dims[1] + at[1]) * dims[2] + at[2], w


def _inside(c, dims):
    ok = torch.ones_like(c[0], dtype=torch.bool)
    for x, n in zip(c, dims):
        ok &= (x >= 0) & (x <= n - 1)
    return ok


def _slices64(vol, shape, R, fmax):
    """Central slices of a complex128 volume (d, h, w); R (n, 3, 3) acting on zyx vectors."""
    dims = vol.shape
    qy, qx = _freqs(shape[1], shape[2])
    p = _plane(R, qy, qx)
    px = p[2].detach()
    r11, r12 = R.detach()[:, 2, 2, None, None], R.detach()[:, 2, 1, None, None]
    tie = torch.where(r11.abs() <= 1e-7, r12 < 0, r11 < 0).expand_as(px)
    conj = torch.where(px.abs() < 1e-8, tie, px < -1e-8)
    c = _array_coords([torch.where(conj, -x, x) for x in p], shape)
    ok = _inside(c, dims) & _keep(qy, qx, fmax)
    flat = torch.view_as_real(vol).reshape(-1, 2)
    c = [torch.where(ok, x, 0.0) for x in c]
    out = 0.0
    for at, w in _corners(c, dims):
        out = out + flat.index_select(0, at.reshape(-1)).reshape(*at.shape, 2) * w[..., None]
    out = torch.where(ok[..., None], out, 0.0)
    out = torch.stack([out[..., 0], torch.where(conj, -out[..., 1], out[..., 1])], dim=-1)
    return torch.view_as_complex(out)


def _chunks(n, pixels):
    step = max(1, CHUNK // pixels)
    return [slice(i, min(n, i + step)) for i in range(0, n, step)]


def _zyx64(R, tolerance):
    R = R.detach().to(torch.float32).to(torch.float64).flip((-2, -1))
    return torch.where(R.abs() < 1e-8, 0.0, R) if tolerance else R


def _insert64(images, d, R, fmax, ctf=None, G=None):
    """Insertion of (n, d, d//2+1) slices into a d box: (volume, weights), or the gradient of the slices
    for the volume's gradient G."""
    shape, dims = (d, d, d), (d, d, d // 2 + 1)
    qy, qx = _freqs(d, d)
    keep = _keep(qy, qx, fmax) & ~((qx == 0) & (qy[:, None] < 0))
    acc = torch.zeros((d * d * dims[2], 3), dtype=torch.float64, device=DEV)
    if G is not None:
        flat = torch.zeros_like(acc[:, :2]).requires_grad_(True)
        vol, _ = _friedel(torch.cat([flat, acc[:, 2:]], dim=1), dims)
        (gflat,) = torch.autograd.grad(vol, flat, grad_outputs=G.to(torch.complex128))
        grads = []
    for part in _chunks(R.shape[0], d * dims[2]):
        p = _plane(R[part], qy, qx)
        conj = p[2] < 0
        c = _array_coords([torch.where(conj, -x, x) for x in p], shape)
        ok = _inside(c, dims) & keep
        c = [torch.where(ok, x, 0.0) for x in c]
        if G is not None:
            g = 0.0
            for at, w in _corners(c, dims):
                g = g + gflat.index_select(0, at.reshape(-1)).reshape(*at.shape, 2) * w[..., None]
            g = torch.where(ok[..., None], g, 0.0)
            g[..., 1] = torch.where(conj, -g[..., 1], g[..., 1])
            grads.append(torch.view_as_complex(g))
            continue
        data = images[part].to(torch.complex128)
        unit = torch.ones_like(c[0])
        if ctf is not None:
            v = _ctf64(ctf[part], qy, qx)
            data, unit = data * v, v * v
        data = torch.stack([data.real, torch.where(conj, -data.imag, data.imag), unit], dim=-1)
        data = torch.where(ok[..., None], data, 0.0)
        for at, w in _corners(c, dims):
            acc.index_add_(0, at.reshape(-1), (data * w[..., None]).reshape(-1, 3))
    return torch.cat(grads) if G is not None else _friedel(acc, dims)


def _friedel(acc, dims):
    """Adds the Friedel mates of the x = 0 plane, but the one at the origin."""
    d, h, w = dims
    a = acc.reshape(d, h, w, 3)
    z, y = torch.arange(d, device=DEV), torch.arange(h, device=DEV)
    zm, ym = (d - z) % d, (h - y) % h
    mate = a[:, :, 0][zm][:, ym] * torch.tensor([1.0, -1.0, 1.0], dtype=torch.float64, device=DEV)
    origin = ((zm == d // 2)[:, None] & (ym == h // 2))[..., None]
    plane = a[:, :, 0] + torch.where(origin, 0.0, mate)
    a = torch.cat([plane[:, :, None], a[:, :, 1:]], dim=2)
    return torch.complex(a[..., 0], a[..., 1]), a[..., 2]


def _ctf64(rows, qy, qx):
    """-sin(chi) of each row of CTF parameters on the slice grid."""
    r = rows.to(torch.float64)[:, :, None, None].unbind(1)
    defocus, astig, angle, kv, cs, amplitude, phase, pixel = r
    volts = kv * 1e3
    h, c, m0, e = 6.62607015e-34, 299792458.0, 9.1093837015e-31, 1.602176634e-19
    lam = h * c / torch.sqrt(e * volts * (2 * m0 * c * c + e * volts)) * 1e10
    y, x = qy[:, None] / pixel, qx / pixel
    s2 = y * y + x * x
    norm = torch.sqrt(s2 + torch.finfo(torch.float32).eps)
    th = torch.deg2rad(angle)
    dot = torch.sqrt(astig) * (y / norm * torch.sin(th) + x / norm * torch.cos(th))
    df = (defocus - astig + 2 * dot * dot) * 1e4
    chi = (-math.pi * lam * s2 * df + math.pi / 2 * cs * 1e7 * lam**3 * s2 * s2
           - torch.deg2rad(phase) - torch.atan(amplitude / torch.sqrt(1 - amplitude**2)))
    return -torch.sin(chi)


def _sinc2(shape):
    f = [torch.fft.fftshift(torch.fft.fftfreq(n, dtype=torch.float64, device=DEV)) for n in shape]
    r = torch.sqrt(f[0][:, None, None] ** 2 + f[1][:, None] ** 2 + f[2] ** 2)
    return torch.sinc(r) ** 2


def _irfftn(x, dims):
    """Complex transforms of the leading axes, then a real one that takes its first and last bins as real."""
    x = torch.fft.ifftn(x, dim=tuple(range(-dims, -1)))
    edge = torch.zeros(x.shape[-1], dtype=torch.bool, device=DEV)
    edge[0] = edge[-1] = True
    return torch.fft.irfft(torch.where(edge, torch.complex(x.real, torch.zeros_like(x.real)), x), dim=-1)


def _project64(vol, R, pad, fmax):
    """Projections of one float64 map, a chunk of rotations at a time: a generator of (rows, images)."""
    d = vol.shape[-1]
    p = int((d * (pad - 1.0)) // 2)
    e = d + 2 * p
    x = F.pad(vol, [p] * 6) * _sinc2((e, e, e))
    dft = torch.fft.fftshift(torch.fft.rfftn(torch.fft.fftshift(x, dim=(0, 1, 2)), dim=(0, 1, 2)), dim=(0, 1))
    for part in _chunks(R.shape[0], e * (e // 2 + 1)):
        s = torch.fft.ifftshift(_slices64(dft, (e, e, e), R[part], fmax), dim=-2)
        image = torch.fft.ifftshift(_irfftn(s, 2), dim=(-2, -1))
        yield part, image[:, p : image.shape[1] - p, p : image.shape[2] - p]


def _backproject64(images, R, pad, fmax):
    d = images.shape[-1]
    p = int((d * (pad - 1.0)) // 2)
    e = d + 2 * p
    vol = wts = 0.0
    for part in _chunks(R.shape[0], 8 * e * (e // 2 + 1)):
        x = torch.fft.fftshift(F.pad(images[part].to(torch.float64), [p] * 4), dim=(-2, -1))
        v, w = _insert64(torch.fft.fftshift(torch.fft.rfftn(x, dim=(-2, -1)), dim=-2), e, R[part], fmax)
        vol, wts = vol + v, wts + w
    real = torch.fft.ifftshift(_irfftn(torch.fft.ifftshift(vol / wts.clamp(min=1.0), dim=(0, 1)), 3), dim=(0, 1, 2))
    real = real / _sinc2(real.shape)
    return real[tuple(slice(p, m - p) for m in real.shape)]


def _undo(gR, R):
    """The gradient of the caller's matrices from that of the zyx ones."""
    return torch.where(R.detach().abs() < 1e-8, 0.0, gR.flip((-2, -1)).to(torch.float64))


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case["kind"]
    fmax = case.get("fmax") or None
    if fmax:
        fmax = float(torch.tensor(fmax, dtype=torch.float32))
    d = case.get("d")
    if kind == "project":
        return _exact_project(case, s, fmax)
    if kind == "backproject":
        R = _zyx64(s["R"], False)
        images = s["images"] if case["channels"] else s["images"][:, None]
        vols = [_backproject64(images[:, ch], R, case["pad"], fmax) for ch in range(images.shape[1])]
        return {"out": torch.stack(vols) if case["channels"] else vols[0]}
    if kind in ("extract", "mse"):
        grad = kind == "mse" or case["grad"]
        vol = s["volume"].to(torch.complex128)
        R = _zyx64(s["R"], True)
        out, gv, gr, loss = [], torch.zeros_like(vol), [], 0.0
        total = case["n"] * d * (d // 2 + 1)
        for part in _chunks(case["n"], d * (d // 2 + 1)):
            v, r = vol.clone().requires_grad_(grad), R[part].clone().requires_grad_(grad)
            x = _slices64(v, (d, d, d), r, fmax)
            if kind == "mse":
                one = (x - s["targets"][part].to(torch.complex128)).abs().square().sum() / total
                loss = loss + one.detach()
                a, b = torch.autograd.grad(one, [v, r])
            else:
                out.append(x.detach())
                if not grad:
                    continue
                a, b = torch.autograd.grad(x, [v, r], grad_outputs=s["G"][part].to(torch.complex128))
            gv += a
            gr.append(b)
        res = {"out": loss if kind == "mse" else torch.cat(out)}
        if grad:
            res["volume"], res["R"] = gv, _undo(torch.cat(gr), s["R"])
        return res
    if kind == "insert":
        R = _zyx64(s["R"], False)
        vol, wts = _insert64(s["images"], d, R, fmax)
        res = {"out": vol, "weights": wts}
        if case["grad"]:
            res["images"] = _insert64(None, d, R, fmax, G=s["G"])
        return res
    if kind == "batched":
        boxes = _ints(case["boxes"])
        res = {"inserted": [_insert64(im, b, _zyx64(R, False), None, ctf)
                            for im, b, R, ctf in zip(s["images"], boxes, s["R"], s["ctf"])]}
        if case["extract"]:
            res["slices"] = []
            for vol, b, R, ctf in zip(s["volumes"], boxes, s["R"], s["ctf"]):
                qy, qx = _freqs(b, b)
                v, R = vol.to(torch.complex128), _zyx64(R, True)
                res["slices"].append(torch.cat([
                    _slices64(v, (b, b, b), R[part], None) * _ctf64(ctf[part], qy, qx)
                    for part in _chunks(R.shape[0], b * (b // 2 + 1))]))
        return res
    return _exact_sample(case, s) if kind == "sample" else _exact_splat(case, s)


def _exact_project(case, s, fmax):
    c, grad = case["channels"], case["grad"]
    vols = s["volume"].to(torch.float64).reshape(-1, *s["volume"].shape[-3:])
    R = _zyx64(s["R"], True)
    outs, gvs, gR = [], [], torch.zeros_like(R)
    for ch in range(vols.shape[0]):
        v, r = vols[ch].clone().requires_grad_(grad), R.clone().requires_grad_(grad)
        parts, gv = [], torch.zeros_like(vols[ch])
        for part, image in _project64(v, r, case["pad"], fmax):
            parts.append(image.detach())
            if grad:
                G = (s["G"][part, ch] if c else s["G"][part]).to(torch.float64)
                a, b = torch.autograd.grad(image, [v, r], grad_outputs=G, retain_graph=True)
                gv += a
                gR += b
        outs.append(torch.cat(parts))
        gvs.append(gv)
    res = {"out": torch.stack(outs, dim=1) if c else outs[0]}
    if grad:
        res["volume"] = torch.stack(gvs) if c else gvs[0]
        res["R"] = _undo(gR, s["R"])
    return res


def _wide(t):
    return torch.view_as_real(t.to(torch.complex128)) if t.is_complex() else t.to(torch.float64)[..., None]


def _narrow(t, like):
    return torch.view_as_complex(t.contiguous()) if like.is_complex() else t[..., 0]


def _exact_sample(case, s):
    multi = s["image"].ndim == 4
    image = _wide(s["image"] if multi else s["image"][None])  # (c, d, h, w, e)
    dims, grad = image.shape[1:4], case["grad"]
    flat = image.permute(1, 2, 3, 0, 4).reshape(-1, image.shape[0] * image.shape[4])
    coords = s["coords"].to(torch.float64).reshape(-1, 3)
    G = _wide(s["G"]).reshape(coords.shape[0], -1) if grad else None
    outs, gc, gi = [], [], torch.zeros_like(flat)
    for part in _chunks(coords.shape[0], image.shape[0]):
        x, v = coords[part].clone().requires_grad_(grad), flat
        c = list(x.unbind(1))
        ok = _inside(c, dims)
        if case["nearest"]:
            at = [torch.round(t).long().clamp(0, n - 1) for t, n in zip(c, dims)]
            o = v.index_select(0, (at[0] * dims[1] + at[1]) * dims[2] + at[2])
            outs.append(torch.where(ok[:, None], o, 0.0))
            continue
        o = 0.0
        kept = [torch.where(ok, t, 0.0) for t in c]
        for at, w in _corners(kept, dims):
            o = o + v.index_select(0, at) * w[:, None]
            if grad:
                gi.index_add_(0, at, torch.where(ok[:, None], G[part] * w.detach()[:, None], 0.0))
        o = torch.where(ok[:, None], o, 0.0)
        outs.append(o.detach())
        if grad:
            (g,) = torch.autograd.grad(o, x, grad_outputs=G[part])
            # a coordinate on the border of its axis is clipped there
            edge = (coords[part] <= 0) | (coords[part] >= torch.tensor(dims, device=DEV) - 1)
            gc.append(torch.where(edge, 0.0, g))
    lead, e = s["coords"].shape[:-1], image.shape[4]
    out = _narrow(torch.cat(outs).reshape(*lead, image.shape[0], e), s["image"])
    res = {"out": out if multi else out[..., 0]}
    if grad:
        g = _narrow(gi.reshape(*dims, image.shape[0], e).permute(3, 0, 1, 2, 4), s["image"])
        res["image"] = g if multi else g[0]
        res["coords"] = torch.cat(gc).reshape(s["coords"].shape)
    return res


def _exact_splat(case, s):
    dims = s["shape"]
    vals, coords = _wide(s["values"]), s["coords"].to(torch.float64).reshape(-1, 3)
    vals = vals.reshape(coords.shape[0], -1)
    acc = torch.zeros((math.prod(dims), vals.shape[1] + 1), dtype=torch.float64, device=DEV)
    G = _wide(s["G"]).reshape(acc.shape[0], -1) if case["grad"] else None
    grads = []
    for part in _chunks(coords.shape[0], 1):
        c = list(coords[part].unbind(1))
        ok = _inside(c, dims)
        c = [torch.where(ok, t, 0.0) for t in c]
        x = torch.cat([vals[part], torch.ones_like(vals[part][:, :1])], dim=1)
        x = torch.where(ok[:, None], x, 0.0)
        if case["nearest"]:
            at = [torch.round(t).long() for t in c]
            acc.index_add_(0, (at[0] * dims[1] + at[1]) * dims[2] + at[2], x)
            continue
        g = 0.0
        for at, w in _corners(c, dims):
            acc.index_add_(0, at, x * w[:, None])
            if G is not None:
                g = g + G.index_select(0, at) * w[:, None]
        if G is not None:
            grads.append(torch.where(ok[:, None], g, 0.0))
    acc = acc.reshape(*dims, -1)
    res = {"out": _narrow(acc[..., :-1], s["values"]), "weights": acc[..., -1]}
    if G is not None:
        res["values"] = _narrow(torch.cat(grads).reshape(*s["values"].shape, -1), s["values"])
    return res
