"""Representative calls of this package, with their inputs, for timing and comparing.

Nine kinds of work, each through the entry point that a user's program calls:

  image     ``trace_to_image``: rays through an optical column onto a detector
            (outgoing rays, pixel indices and the hit image)
  grad      ``run_to_end`` under autograd, and its backward pass: gradients of
            the detector positions with respect to rays and column parameters
  scan      ``scan_images``: a 4D-STEM scan, one detector image per position
  field     ``make_gaussian_image``: Gaussian beamlets after a column
  input     ``evaluate_gaussian_input_image``: beamlets in their own plane
  backward  ``make_gaussian_image`` under autograd, and its backward pass
  sweep     ``BatchedTrace.value_and_grad``: many columns in one launch
  fit       ``StemFit.loss_grad``: the 4D-STEM calibration loss and gradient
  transfer  ``transfer_rays``: rays through a stack of transfer matrices

Every input is synthetic and follows from the case and the seed.
"""
import math
import random

import numpy as np
import torch

import temgymcore_gb300 as tg

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # the quick-start call: 65,536 rays, a lens and a 256 x 256 detector;
        # a call of this size is mostly launches and host time
        {"name": "image_quickstart", "kind": "image", "rays": 65536, "parts": 2, "h": 256, "w": 256, "pixels": True},
        # a large bundle through a longer column onto a larger camera, with a
        # ray count that no vector width divides
        {"name": "image_column", "kind": "image", "rays": 8_000_023, "parts": 8, "h": 512, "w": 512, "pixels": True},
        # calibrating a column: gradients of detector positions with respect
        # to every ray and to the column's parameters
        {"name": "grad_column", "kind": "grad", "rays": 2_097_152, "parts": 5},
        # the 4D-STEM shadow-image benchmark: 64 x 64 positions x 1,024 rays,
        # a small disc on a 256 x 256 camera
        {"name": "scan_64x64", "kind": "scan", "rows": 64, "cols": 64, "rays": 1024, "h": 256, "w": 256,
         "disc": 9.0, "xy": False},
        # the same experiment with a long camera length: the disc covers much
        # of the camera, and takes more rays to fill it
        {"name": "scan_wide", "kind": "scan", "rows": 40, "cols": 36, "rays": 10_000, "h": 192, "w": 192,
         "disc": 80.0, "xy": False},
        # aperture diffraction from round beamlets (the separable field)
        {"name": "field_round", "kind": "field", "beams": 16384, "h": 512, "w": 512, "astigmatic": False},
        # the same with astigmatic beamlets
        {"name": "field_astigmatic", "kind": "field", "beams": 16384, "h": 512, "w": 512, "astigmatic": True},
        # a small image decomposed into a few hundred beams, odd sizes
        {"name": "input_small", "kind": "input", "beams": 300, "h": 90, "w": 121, "astigmatic": True},
        # fitting beam amplitudes, positions and a lens to a measured field
        {"name": "backward_round", "kind": "backward", "beams": 8192, "h": 384, "w": 384, "astigmatic": False},
        # the batched sweep benchmark: 512 columns of 2 to 12 components,
        # 1,000 to 260,000 rays each, forward and gradient
        {"name": "sweep_512", "kind": "sweep", "models": 512, "low": 1000, "high": 260_000},
        # the calibration benchmark: 32 x 32 positions x 1,024 rays
        {"name": "fit_32x32", "kind": "fit", "rows": 32, "cols": 32, "rays": 1024},
        # rays through the 16 step matrices of an eight-component column
        {"name": "transfer_16", "kind": "transfer", "rays": 1_048_576, "planes": 16},
    ]


def _between(rng, low, high):
    """A whole number, spread over the logarithm of the range."""
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng):
    kind = rng.choice(["image", "image", "grad", "scan", "scan", "field", "input", "backward", "sweep", "fit",
                       "transfer"])
    if kind == "image":
        return {"kind": kind, "rays": _between(rng, 1000, 8_000_000), "parts": rng.randint(2, 8),
                "h": _between(rng, 64, 512), "w": _between(rng, 64, 512), "pixels": rng.random() < 0.7}
    if kind == "grad":
        return {"kind": kind, "rays": _between(rng, 1000, 3_000_000), "parts": rng.randint(2, 5)}
    if kind == "scan":
        h, w = _between(rng, 64, 256), _between(rng, 64, 256)
        rays = _between(rng, 200, 10_000)
        side = math.sqrt(min(4096, 14_000_000 / rays, 4096 * 65536 / (h * w)))
        rows, cols = _between(rng, 4, max(5, int(side))), _between(rng, 4, max(5, int(side)))
        return {"kind": kind, "rows": rows, "cols": cols, "rays": rays, "h": h, "w": w,
                "disc": round(min(h, w) * math.exp(rng.uniform(math.log(0.03), math.log(0.45))), 2),
                "xy": rng.random() < 0.3}
    if kind in ("field", "input"):
        return {"kind": kind, "beams": _between(rng, 64, 16384), "h": _between(rng, 64, 512),
                "w": _between(rng, 64, 512), "astigmatic": rng.random() < 0.5}
    if kind == "backward":
        return {"kind": kind, "beams": _between(rng, 64, 8192), "h": _between(rng, 64, 384),
                "w": _between(rng, 64, 384), "astigmatic": rng.random() < 0.4}
    if kind == "sweep":
        return {"kind": kind, "models": _between(rng, 4, 512), "low": 1000, "high": _between(rng, 2000, 260_000)}
    if kind == "fit":
        return {"kind": kind, "rows": _between(rng, 4, 32), "cols": _between(rng, 4, 32),
                "rays": _between(rng, 64, 1024)}
    return {"kind": kind, "rays": _between(rng, 1000, 1_000_000), "planes": 2 * rng.randint(1, 8)}


# ------------------------------------------------------------------ inputs

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _uniform(g, n, low, high, dtype=torch.float32):
    return torch.rand(n, generator=g, device=DEV, dtype=dtype) * (high - low) + low


def _normal(g, n, sigma, dtype=torch.float32):
    return torch.randn(n, generator=g, device=DEV, dtype=dtype) * sigma


def _ray_bundle(g, n):
    """x, y ~ U(-1, 1) mm, slopes ~ N(0, 1 mrad)."""
    return [_uniform(g, n, -1e-3, 1e-3), _uniform(g, n, -1e-3, 1e-3), _normal(g, n, 1e-3), _normal(g, n, 1e-3)]


# what stands between the source and the detector, in this order
_ORDER = ("scanner", "descanner", "lens", "deflector", "rotator", "lens", "aperture")
_DESCAN = ("pxo_pxi", "pxo_pyi", "pyo_pxi", "pyo_pyi", "sxo_pxi", "sxo_pyi", "syo_pxi", "syo_pyi")


def _column(parts, seed):
    """A column of ``parts`` components as plain descriptions; the last one is
    the detector's plane.  Two parts: the quick-start lens and detector."""
    r = random.Random(int(seed) * 7919 + parts)
    if parts == 2:
        return [{"kind": "lens", "z": 0.5, "focal_length": 0.2 * r.uniform(0.95, 1.05)}, {"kind": "detector", "z": 1.0}]
    spec, z = [], 0.0
    pos = (r.uniform(-2e-4, 2e-4), r.uniform(-2e-4, 2e-4))
    kinds = _ORDER[:parts - 1] if parts > 3 else ("lens", "deflector")[:parts - 1]
    for kind in kinds:
        z += r.uniform(0.05, 0.2)
        c = {"kind": kind, "z": z}
        if kind == "scanner":
            c |= {"scan_pos_x": pos[0], "scan_pos_y": pos[1]}
        elif kind == "descanner":
            c |= {"scan_pos_x": pos[0], "scan_pos_y": pos[1],
                  "descan": [(1.0 if i in (0, 3) else 0.0) + r.gauss(0.0, 1e-2) for i in range(8)]}
        elif kind == "lens":
            c["focal_length"] = r.uniform(0.4, 1.5)
        elif kind == "deflector":
            c |= {"def_x": r.gauss(0.0, 2e-4), "def_y": r.gauss(0.0, 2e-4)}
        elif kind == "rotator":
            c["angle"] = r.uniform(-90.0, 90.0)
        else:
            c |= {"radius": r.uniform(0.9e-3, 1.3e-3)}
        spec.append(c)
    return spec + [{"kind": "detector", "z": z + r.uniform(0.1, 0.3)}]


def _components(spec, h, w):
    """The package's components for a column's descriptions."""
    out = []
    for c in spec:
        kw = {k: v for k, v in c.items() if k not in ("kind", "descan")}
        if c["kind"] == "detector":
            px = 2.56e-3 / min(h, w)
            out.append(tg.Detector(pixel_size=(px, px), shape=(h, w), **kw))
        elif c["kind"] == "descanner":
            out.append(tg.Descanner(descan_error=tg.DescanError(**dict(zip(_DESCAN, c["descan"]))), **kw))
        else:
            out.append({"scanner": tg.Scanner, "lens": tg.Lens, "deflector": tg.Deflector, "rotator": tg.Rotator,
                        "aperture": tg.Aperture, "biprism": tg.Biprism}[c["kind"]](**kw))
    return out


def _leaf_spec(spec, make):
    """The column with its optical parameters (focal lengths, deflections,
    descan errors, the detector's z) as ``make(value)``; and those, in order."""
    out, leaves = [], []

    def leaf(v):
        leaves.append(make(v))
        return leaves[-1]

    for c in spec:
        c = dict(c)
        if c["kind"] == "lens":
            c["focal_length"] = leaf(c["focal_length"])
        elif c["kind"] == "deflector":
            c |= {"def_x": leaf(c["def_x"]), "def_y": leaf(c["def_y"])}
        elif c["kind"] == "descanner":
            c["descan"] = [leaf(v) for v in c["descan"]]
        elif c["kind"] == "detector":
            c["z"] = leaf(c["z"])
        out.append(c)
    return out, leaves


def _stem(case, seed):
    """A 4D-STEM geometry: scan step, rotation, descan error, and the camera's
    pixel such that the bright-field disc has the case's radius in pixels."""
    r = random.Random(int(seed) * 104729 + 1)
    conv, length = 5e-3, 0.1
    return {"conv": conv, "length": length, "defocus": 1e-6, "step": 1e-9, "rotation": r.uniform(0.0, 360.0),
            "descan": [(1.0 if i in (0, 3) else 0.0) + r.gauss(0.0, 1e-3) for i in range(8)],
            "px": conv * length / case["disc"]}


def _stem_model(case, s):
    z = s["defocus"]
    shape = (case["rows"], case["cols"])
    return [tg.PointSource(z=0.0),
            tg.ScanGrid(z=z, pixel_size=(s["step"], s["step"]), shape=shape, rotation=s["rotation"]),
            tg.Scanner(z=z, scan_pos_x=0.0, scan_pos_y=0.0),
            tg.Descanner(z=z, scan_pos_x=0.0, scan_pos_y=0.0,
                         descan_error=tg.DescanError(**dict(zip(_DESCAN, s["descan"])))),
            tg.Detector(z=z + s["length"], pixel_size=(s["px"], s["px"]), shape=(case["h"], case["w"]))]


def _stem_bundle(case, s, g):
    """Slopes that fill the convergence disc."""
    n = case["rays"]
    rad = s["conv"] * torch.sqrt(torch.rand(n, generator=g, device=DEV))
    phi = _uniform(g, n, 0.0, 2.0 * math.pi)
    return torch.zeros(n, device=DEV), torch.zeros(n, device=DEV), rad * torch.cos(phi), rad * torch.sin(phi)


def _beams(case, seed):
    """Beamlets on a golden-angle spiral: a 50 nm aperture at 200 keV (waist 1 nm)
    for the detector field; an image's disc at 500 nm for the input plane."""
    g, n, r = _gen(seed), case["beams"], random.Random(int(seed) * 31 + 5)
    inp = case["kind"] == "input"
    px = 1e-5 if inp else 5.12e-3 / max(case["h"], case["w"])
    radius = 0.2 * min(case["h"], case["w"]) * px if inp else 5e-8
    i = torch.arange(n, device=DEV, dtype=F64)
    rad = radius * torch.sqrt((i + 0.5) / n)
    phi = i * (math.pi * (3.0 - math.sqrt(5.0))) + r.uniform(0.0, 2.0 * math.pi)
    waist = math.sqrt(math.pi * radius ** 2 / n) if inp else 1e-9
    wxy = torch.full((n, 2), waist, device=DEV, dtype=F64)
    theta = torch.zeros(n, device=DEV, dtype=F64)
    if case["astigmatic"]:
        wxy[:, 1] = waist * _uniform(g, n, 0.5, 1.5, F64)
        theta = _uniform(g, n, 0.0, math.pi, F64)
    amp = _uniform(g, n, 0.5, 1.0, F64) * torch.exp(1j * _uniform(g, n, 0.0, 2.0 * math.pi, F64))
    slope = 1e-4 if inp else 0.0
    return {"x": rad * torch.cos(phi), "y": rad * torch.sin(phi),
            "dx": _normal(g, n, slope, F64), "dy": _normal(g, n, slope, F64), "z": 0.0,
            "pathlength": (0.0 if inp else 1.0) + _normal(g, n, 1e-6, F64), "amplitude": amp.to(torch.complex64),
            "waist_xy": wxy, "radii_of_curv": torch.full((n, 2), math.inf, device=DEV, dtype=F64),
            "wavelength": 500e-9 if inp else 1.97e-12, "theta": theta}, px, g


def _grid(case, px, z):
    return tg.Detector(z=z, pixel_size=(px, px), shape=(case["h"], case["w"]))


def _sweep(case, seed):
    """Columns of 2 to 12 lenses, deflectors, biprisms and apertures (their
    makeup and ray counts follow from the case, their settings from the seed),
    and how many rays each has."""
    makeup, r = random.Random(case["models"]), random.Random(int(seed) * 15485863 + case["models"])
    specs, counts = [], []
    for _ in range(case["models"]):
        spec, z = [], 0.0
        for _ in range(makeup.randint(2, 12)):
            z += r.uniform(0.01, 0.1)
            kind = makeup.choice(("lens", "deflector", "biprism", "aperture"))
            c = {"kind": kind, "z": z}
            if kind == "lens":
                c["focal_length"] = 10.0 ** r.uniform(-2.0, 0.0)
            elif kind == "deflector":
                c |= {"def_x": r.gauss(0.0, 1e-3), "def_y": r.gauss(0.0, 1e-3)}
            elif kind == "biprism":
                c["def_x"] = r.gauss(0.0, 1e-3)
            else:
                c["radius"] = r.uniform(5e-4, 5e-3)
            spec.append(c)
        specs.append(spec)
        counts.append(_between(makeup, case["low"], case["high"]))
    return specs, counts


def _sweep_rays(g, n):
    return _ray_bundle(g, n) + [_normal(g, n, 1e-3), _normal(g, n, 1e-3)]


def _fit_theta(seed):
    """The nominal 21 parameters (lens, distances, scan, descan matrix), and the
    true ones 1 % away, which the measured positions follow."""
    r = random.Random(int(seed) * 6700417 + 3)
    descan = [(1.0 if i % 5 == 0 else 0.0) + r.gauss(0.0, 1e-3) for i in range(16)]
    theta = [0.2, 0.05, 0.95, 37.0, 1e-5] + descan
    return theta, [v * (1.0 + r.gauss(0.0, 0.01)) for v in theta]


def _fit_detector(case, rays, t):
    """Detector (x, y) of every position and ray for the parameters ``t``, float64."""
    x, y, dx, dy = rays
    rows, cols, gap = case["rows"], case["cols"], 0.45
    u = (torch.arange(rows, device=DEV, dtype=F64) - 0.5 * (rows - 1)).repeat_interleave(cols)[:, None]
    v = (torch.arange(cols, device=DEV, dtype=F64) - 0.5 * (cols - 1)).repeat(rows)[:, None]
    f, defocus, length, rot, step, m = t[0], t[1], t[2], t[3] * (math.pi / 180.0), t[4], t[5:].reshape(4, 4)
    sx = step * (torch.cos(rot) * v - torch.sin(rot) * u)
    sy = -step * (torch.cos(rot) * u + torch.sin(rot) * v)
    x2, y2 = x + dx * defocus + m[0, 0] * sx + m[0, 1] * sy, y + dy * defocus + m[1, 0] * sx + m[1, 1] * sy
    dx2, dy2 = dx + m[2, 0] * sx + m[2, 1] * sy, dy + m[3, 0] * sx + m[3, 1] * sy
    x3, y3 = x2 + dx2 * gap, y2 + dy2 * gap
    return x3 + (dx2 - x3 / f) * (length - gap), y3 + (dy2 - y3 / f) * (length - gap)


def _matrices(case, seed):
    """(planes, 5, 5) float64: the step matrices of a column, free space then
    component, with a rotated scan and descan among them."""
    r = random.Random(int(seed) * 27644437 + case["planes"])
    out = []
    for i in range(case["planes"]):
        m = np.eye(5)
        if i % 2 == 0:
            m[0, 2] = m[1, 3] = r.uniform(0.02, 0.3)
        elif i % 4 == 1:
            m[2, 0] = m[3, 1] = -1.0 / r.uniform(0.2, 1.0)
        elif i % 8 == 3:
            angle = r.uniform(-1.0, 1.0)
            c, s = math.cos(angle), math.sin(angle)
            m[:2, :2] = m[2:4, 2:4] = [[c, -s], [s, c]]
        else:
            m[:4, 4] = [r.gauss(0.0, 1e-4) for _ in range(4)]
        out.append(m)
    return np.stack(out)


def prepare(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind == "image":
        x, y, dx, dy = _ray_bundle(g, case["rays"])
        model = _components(_column(case["parts"], seed), case["h"], case["w"])
        return {"case": case, "ray": tg.Ray(x=x, y=y, dx=dx, dy=dy, z=0.0, pathlength=0.0), "model": model}
    if kind == "grad":
        rays = [v.requires_grad_(True) for v in _ray_bundle(g, case["rays"])]
        spec, leaves = _leaf_spec(_column(case["parts"], seed),
                                  lambda v: torch.tensor(v, dtype=F64, requires_grad=True))
        up = (_normal(g, case["rays"], 1.0), _normal(g, case["rays"], 1.0))
        ray = tg.Ray(x=rays[0], y=rays[1], dx=rays[2], dy=rays[3], z=0.0, pathlength=0.0)
        return {"case": case, "ray": ray, "model": _components(spec, 256, 256), "leaves": rays + leaves, "up": up}
    if kind == "scan":
        s = _stem(case, seed)
        x, y, dx, dy = _stem_bundle(case, s, g)
        return {"case": case, "ray": tg.Ray(x=x, y=y, dx=dx, dy=dy, z=0.0, pathlength=0.0),
                "model": _stem_model(case, s)}
    if kind == "input":
        b, px, _ = _beams(case, seed)
        return {"case": case, "rays": tg.GaussianRay(**b), "grid": _grid(case, px, 0.0)}
    if kind in ("field", "backward"):
        b, px, gb = _beams(case, seed)
        f = 0.5
        state = {"case": case}
        if kind == "backward":
            for k in ("amplitude", "x", "y"):
                b[k] = b[k].detach().requires_grad_(True)
            f = torch.tensor(f, dtype=F64, requires_grad=True)
            state["leaves"] = [b["amplitude"], b["x"], b["y"], f]
            n = (case["h"], case["w"])
            state["up"] = torch.complex(_normal(gb, n, 1.0), _normal(gb, n, 1.0))
        state["rays"] = tg.GaussianRay(**b)
        state["model"] = [tg.Lens(z=0.5, focal_length=f), _grid(case, px, 1.0)]
        return state
    if kind == "sweep":
        specs, counts = _sweep(case, seed)
        return {"case": case, "trace": tg.BatchedTrace([_components(s, 1, 1) for s in specs], counts),
                "rays": _sweep_rays(g, sum(counts))}
    if kind == "fit":
        x, y, dx, dy = _ray_bundle(g, case["rays"])
        theta, true = _fit_theta(seed)
        measured = _fit_detector(case, [v.to(F64) for v in (x, y, dx, dy)], torch.tensor(true, dtype=F64, device=DEV))
        return {"case": case, "fit": tg.StemFit(tg.Ray(x=x, y=y, dx=dx, dy=dy, z=0.0, pathlength=0.0), case["rows"],
                                                case["cols"], 0.45, theta, measured)}
    x, y, dx, dy = (v.to(F64) for v in _ray_bundle(g, case["rays"]))
    return {"case": case, "rays": torch.stack([x, y, dx, dy, torch.ones_like(x)], dim=1).contiguous(),
            "matrices": _matrices(case, seed)}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "image":
        out, pix, img = tg.trace_to_image(state["ray"], state["model"], want_pixels=case["pixels"])
        rays = [out.x, out.y, out.dx, out.dy, out.pathlength]
        return rays + ([pix.y, pix.x] if case["pixels"] else []) + [img]
    if kind == "grad":
        out = tg.run_to_end(state["ray"], state["model"])
        grads = torch.autograd.grad((out.x, out.y), state["leaves"], state["up"])
        return [out.x.detach(), out.y.detach(), *grads]
    if kind == "scan":
        r = tg.scan_images(state["ray"], state["model"], return_xy=case["xy"])
        return list(r) if case["xy"] else [r]
    if kind == "field":
        return [tg.make_gaussian_image(state["rays"], state["model"])]
    if kind == "input":
        return [tg.evaluate_gaussian_input_image(state["rays"], state["grid"])]
    if kind == "backward":
        image = tg.make_gaussian_image(state["rays"], state["model"])
        return [image.detach(), *torch.autograd.grad(image, state["leaves"], state["up"])]
    if kind == "sweep":
        loss, raw = state["trace"].value_and_grad(*state["rays"])
        return [loss, raw, *state["trace"].last_outputs]
    if kind == "fit":
        return [state["fit"].loss_grad()]
    return [tg.transfer_rays(state["rays"], state["matrices"])]


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    """Bytes: each input and output once.  Floating-point operations: the
    arithmetic of the formulas (a ray step about 10, a beam and pixel about 16
    with a running product; a round beam's pixels as one complex product of
    its row and column factors)."""
    kind, n = case["kind"], case.get("rays", 0)
    if kind == "image":
        hw = case["h"] * case["w"]
        return {"bytes": n * (16 + 24 + (8 if case["pixels"] else 0)) + 8 * hw, "flops": n * (20 * case["parts"] + 20)}
    if kind == "grad":  # forward: 16 in, x, y, dx, dy, pathlength out; backward: 16 + 8 in, 16 out
        return {"bytes": n * (16 + 24 + 24 + 16), "flops": n * 60 * case["parts"]}
    if kind == "scan":
        p = case["rows"] * case["cols"]
        return {"bytes": 4 * p * case["h"] * case["w"] + 16 * n + (8 * p * n if case["xy"] else 0),
                "flops": p * n * 60}
    if kind in ("field", "input", "backward"):
        b, px = case["beams"], case["h"] * case["w"]
        per = 16 if case["astigmatic"] else 8
        byte, flops = b * 88 + 8 * px, b * px * per
        if kind == "backward":  # six complex moments of each beam's product with the upstream gradient
            byte, flops = byte + 8 * px + b * 24, flops + b * px * (3 * per)
        return {"bytes": byte, "flops": flops}
    if kind == "sweep":
        _, counts = _sweep(case, 1)
        return {"bytes": 49 * sum(counts), "flops": 120 * sum(counts)}
    if kind == "fit":
        r = case["rows"] * case["cols"] * n
        return {"bytes": 8 * r + 16 * n, "flops": 60 * r}
    return {"bytes": n * 40 * (1 + case["planes"]), "flops": n * 50 * case["planes"]}


# ------------------------------------------------------------------ the same in 64 bits

def _walk(spec, x, y, dx, dy, dist=None):
    """A column in float64: (x, y, dx, dy, pathlength, rays that every aperture passes)."""
    z, pl = 0.0, torch.zeros_like(x)
    alive = torch.ones_like(x, dtype=torch.bool)
    for i, c in enumerate(spec):
        d = c["z"] - z if dist is None else dist[i]
        z = c["z"]
        x, y, pl = x + dx * d, y + dy * d, pl + d
        kind = c["kind"]
        if kind == "lens":
            f = c["focal_length"]
            pl = pl - (x * x + y * y) / (2 * f)
            dx, dy = dx - x / f, dy - y / f
        elif kind == "scanner":
            x, y = x + c["scan_pos_x"], y + c["scan_pos_y"]
        elif kind == "descanner":
            px, py, e = c["scan_pos_x"], c["scan_pos_y"], c["descan"]
            x, y = x + (e[0] * px + e[1] * py - px), y + (e[2] * px + e[3] * py - py)
            dx, dy = dx + (e[4] * px + e[5] * py), dy + (e[6] * px + e[7] * py)
        elif kind == "deflector":
            pl = pl + dx * x + dy * y
            dx, dy = dx + c["def_x"], dy + c["def_y"]
        elif kind == "biprism":
            pl = pl + dx * x + dy * y
            dx = dx + c["def_x"] * torch.sign(x.detach())
        elif kind == "rotator":
            a = math.radians(c["angle"])
            co, si = math.cos(a), math.sin(a)
            x, y, dx, dy = x * co - y * si, x * si + y * co, dx * co - dy * si, dx * si + dy * co
        elif kind == "aperture":
            alive = alive & (x * x + y * y < c["radius"] ** 2)
    return x, y, dx, dy, pl, alive


def _exact_sweep(case, seed):
    specs, counts = _sweep(case, seed)
    cols = [v.to(F64) for v in _sweep_rays(_gen(seed), sum(counts))]
    losses, raws, outs, at = [], [], [], 0
    for spec, n in zip(specs, counts):
        x, y, dx, dy, tx, ty = (v[at:at + n] for v in cols)
        at += n
        zs = [0.0] + [c["z"] for c in spec]
        dist = [torch.tensor(b - a, dtype=F64, device=DEV, requires_grad=True) for a, b in zip(zs, zs[1:])]
        lspec, where = [], []  # (leaf, row, column) of the per-step sums
        for i, c in enumerate(spec):
            c = dict(c)
            where.append((dist[i], 2 * i, 0))
            for j, k in enumerate({"lens": ("focal_length",), "deflector": ("def_x", "def_y"),
                                   "biprism": ("def_x",)}.get(c["kind"], ())):
                c[k] = torch.tensor(c[k], dtype=F64, device=DEV, requires_grad=True)
                where.append((c[k], 2 * i + 1, j))
            lspec.append(c)
        o = _walk(lspec, x, y, dx, dy, dist)
        loss = torch.where(o[5], (o[0] - tx) ** 2 + (o[1] - ty) ** 2, 0.0).sum()
        got = torch.autograd.grad(loss, [w[0] for w in where], allow_unused=True)
        raw = torch.zeros((2 * len(spec), 4), dtype=F64, device=DEV)
        for (_, row, col), v in zip(where, got):
            if v is not None:
                raw[row, col] = v
        losses.append(loss.detach())
        raws.append(raw)
        outs.append([v.detach() for v in o[:5]])
    whole = [torch.cat([o[i] for o in outs]) for i in range(5)]
    return [torch.stack(losses), torch.cat(raws), *whole, None]


def _exact_fit(case, seed):
    rays = [v.to(F64) for v in _ray_bundle(_gen(seed), case["rays"])]
    theta, true = (torch.tensor(t, dtype=F64, device=DEV) for t in _fit_theta(seed))
    tx, ty = (t.to(torch.float32).to(F64) for t in _fit_detector(case, rays, true))
    theta.requires_grad_(True)
    ox, oy = _fit_detector(case, rays, theta)
    loss = ((ox - tx) ** 2 + (oy - ty) ** 2).sum()
    return [torch.cat([loss.detach().reshape(1), torch.autograd.grad(loss, theta)[0]])]


def _product(a, b):
    """a * b = p + e exactly (Dekker 1971), float64."""
    def split(v):
        c = 134217729.0 * v
        hi = c - (c - v)
        return hi, v - hi
    p = a * b
    (ah, al), (bh, bl) = split(a), split(b)
    return p, ((ah * bh - p) + ah * bl + al * bh) + al * bl


def _reduced(k, pl):
    """k * pathlength modulo 2 pi, from the exact product."""
    k = torch.full_like(pl, k)
    p, e = _product(k, pl)
    n = torch.round(p / (2.0 * math.pi))
    q, f = _product(n, torch.full_like(pl, 2.0 * math.pi))
    return (p - q) + ((e - f) - n * 2.4492935982947064e-16)


def _beam_forms(b, f=None):
    """Per beam, float64: the phase (k / 2) (S s s + L s + c) of a position s
    relative to an origin, that origin, and the complex factor in front.
    ``f``: the focal length of the lens half way to the detector (None: the
    beams' own plane)."""
    k = 2.0 * math.pi / b["wavelength"]
    q = b["wavelength"] / (math.pi * b["waist_xy"] ** 2)
    co, si = torch.cos(b["theta"]), torch.sin(b["theta"])
    # i (R diag(q) R^T): flat wavefronts
    Q = 1j * torch.stack([co * co * q[:, 0] + si * si * q[:, 1], co * si * (q[:, 0] - q[:, 1]),
                          si * si * q[:, 0] + co * co * q[:, 1]])
    x, y, dx, dy = b["x"], b["y"], b["dx"], b["dy"]
    pl = b["pathlength"].detach()
    front = b["amplitude"].to(torch.complex128) * torch.exp(1j * _reduced(k, pl))
    zero = torch.zeros_like(x.detach())
    if f is None:
        return k, Q, 2 * dx, 2 * dy, zero, (x, y), front
    # free space 0.5, the lens, free space 0.5: scalar A, B, C, D
    A, B, C, D = 1 - 0.5 / f, 1 - 0.25 / f, -1 / f, 1 - 0.5 / f
    m00, m11, m01 = A + B * Q[0], A + B * Q[2], B * Q[1]
    det = m00 * m11 - m01 * m01
    # (A + B Q)^-1 (C + D Q), symmetric
    n00, n11, n01 = C + D * Q[0], C + D * Q[2], D * Q[1]
    S = [(m11 * n00 - m01 * n01) / det, (m11 * n01 - m01 * n11) / det, (m00 * n11 - m01 * n01) / det]
    # P = Q1 (B (A Q1 + B))^-1 with Q1 = Q^-1; Q1 (A Q1 + B)^-1 = (A + B Q)^-1
    P = [m11 / det / B, -m01 / det / B, m00 / det / B]
    rx, ry = A * x + B * dx, A * y + B * dy
    Lx = 2 * (P[0] * rx + P[1] * ry) - 2 * x / B
    Ly = 2 * (P[1] * rx + P[2] * ry) - 2 * y / B
    c = (A / B) * (x * x + y * y) - (P[0] * rx * rx + 2 * P[1] * rx * ry + P[2] * ry * ry)
    return k, S, Lx, Ly, c, (zero, zero), front / torch.sqrt(det)


def _positions(case, px):
    """x of each column and y of each row, metres (y points up)."""
    h, w = case["h"], case["w"]
    return ((torch.arange(w, device=DEV, dtype=F64) - 0.5 * (w - 1)) * px,
            -(torch.arange(h, device=DEV, dtype=F64) - 0.5 * (h - 1)) * px)


def _field_sum(case, px, forms, lo, hi):
    """The field of the beams lo..hi, (h, w) complex128."""
    k, S, Lx, Ly, c, origin, front = forms
    s = slice(lo, hi)
    one = lambda v: v[s, None]  # noqa: E731
    X, Y = (p - one(o) for p, o in zip(_positions(case, px), origin))
    col = 0.5 * k * (one(S[0]) * X * X + one(Lx) * X)
    row = 0.5 * k * (one(S[2]) * Y * Y + one(Ly) * Y + one(c))
    if not case["astigmatic"]:
        return (one(front) * torch.exp(1j * row)).T @ torch.exp(1j * col)
    cross = k * S[1][s, None, None] * Y[:, :, None] * X[:, None, :]
    return (front[s, None, None] * torch.exp(1j * (row[:, :, None] + col[:, None, :] + cross))).sum(0)


def _exact_field(case, seed):
    b, px, g = _beams(case, seed)
    n = case["beams"]
    per = n if not case["astigmatic"] else max(1, 60_000_000 // (case["h"] * case["w"]))
    if case["kind"] != "backward":
        forms = _beam_forms(b, None if case["kind"] == "input" else 0.5)
        return [sum(_field_sum(case, px, forms, i, min(n, i + per)) for i in range(0, n, per))]
    amp = b["amplitude"].to(torch.complex128).requires_grad_(True)
    x, y = b["x"].detach().requires_grad_(True), b["y"].detach().requires_grad_(True)
    f = torch.tensor(0.5, dtype=F64, device=DEV, requires_grad=True)
    size = (case["h"], case["w"])
    up = torch.complex(_normal(g, size, 1.0), _normal(g, size, 1.0)).to(torch.complex128)
    per, image, grads = max(1, per // 8) if case["astigmatic"] else n, 0.0, None
    for i in range(0, n, per):
        part = _field_sum(case, px, _beam_forms({**b, "amplitude": amp, "x": x, "y": y}, f), i, min(n, i + per))
        got = torch.autograd.grad(part, [amp, x, y, f], up)
        grads = got if grads is None else [p + q for p, q in zip(grads, got)]
        image = image + part.detach()
    return [image, *grads]


def exact(case, seed):
    kind, g = case["kind"], _gen(seed)
    if kind == "image":
        o = _walk(_column(case["parts"], seed), *(v.to(F64) for v in _ray_bundle(g, case["rays"])))
        return [*o[:5]] + [None] * (3 if case["pixels"] else 1)
    if kind == "grad":
        rays = [v.to(F64).requires_grad_(True) for v in _ray_bundle(g, case["rays"])]
        spec, leaves = _leaf_spec(_column(case["parts"], seed),
                                  lambda v: torch.tensor(v, dtype=F64, device=DEV, requires_grad=True))
        up = [_normal(g, case["rays"], 1.0).to(F64) for _ in range(2)]
        o = _walk(spec, *rays)
        return [o[0].detach(), o[1].detach(), *torch.autograd.grad((o[0], o[1]), rays + leaves, up,
                                                                   materialize_grads=True, allow_unused=True)]
    if kind == "scan":
        if not case["xy"]:
            return None
        s = _stem(case, seed)
        _, _, dx, dy = (v.to(F64) for v in _stem_bundle(case, s, g))
        rows, cols, a = case["rows"], case["cols"], math.radians(s["rotation"])
        u = (torch.arange(rows, device=DEV, dtype=F64) - 0.5 * (rows - 1)).repeat_interleave(cols)[:, None]
        v = (torch.arange(cols, device=DEV, dtype=F64) - 0.5 * (cols - 1)).repeat(rows)[:, None]
        px, py = s["step"] * (math.cos(a) * v - math.sin(a) * u), -s["step"] * (math.cos(a) * u + math.sin(a) * v)
        e, zs, ln = s["descan"], s["defocus"], s["length"]
        x = dx * zs + e[0] * px + e[1] * py + (dx + e[4] * px + e[5] * py) * ln
        y = dy * zs + e[2] * px + e[3] * py + (dy + e[6] * px + e[7] * py) * ln
        return [None, torch.stack([x, y], dim=1)]
    if kind in ("field", "input", "backward"):
        return _exact_field(case, seed)
    if kind == "sweep":
        return _exact_sweep(case, seed)
    if kind == "fit":
        return _exact_fit(case, seed)
    x, y, dx, dy = (v.to(F64) for v in _ray_bundle(g, case["rays"]))
    m, total = torch.from_numpy(_matrices(case, seed)).to(DEV), None
    out = []
    for t in m.flip(0):
        total = t if total is None else t @ total
        out.append(total)
    return [torch.einsum("mij,nj->nmi", torch.stack(out), torch.stack([x, y, dx, dy, torch.ones_like(x)], dim=1))]
