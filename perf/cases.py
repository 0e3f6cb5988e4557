"""The calls that programs built on this package make, at the sizes they make
them: correlation frames of several sizes, subset shapes, interpolants and
solvers, the tracking routine, the objective's adjoint, strain and image
preprocessing.

A case is a dict of plain values; prepare() makes its inputs and the context a
program keeps, run() makes one pass, work() counts what a pass cannot do
without, exact() evaluates in 64 bits what has a value there.
"""
import ctypes
import math

import numpy as np
import torch

from dice_b200 import abi
from dice_b200 import synthetic as syn
from dice_b200.schema import Schema

DEV = "cuda"
INTERP = {"bilinear": abi.BILINEAR, "bicubic": abi.BICUBIC, "keys": abi.KEYS_FOURTH}


def listed():
    return [
        # a live extensometer: a handful of subsets followed on 8-bit camera
        # frames in host memory, the field rows read back each frame; latency counts
        {"name": "extensometer_9", "kind": "probe", "w": 512, "h": 512, "n": 9, "subset": 31, "interp": "keys",
         "pixel": "u8"},
        # a small full field: the 512^2 pair, 21 px subsets every 10 px
        {"name": "frame_512_21px", "kind": "frame", "w": 512, "h": 512, "subset": 21, "step": 10, "interp": "keys",
         "tol": 1e-5, "pixel": "f32", "filter": 0, "field": "shift", "frame": 1},
        # the headline: one frame of the 2048^2 sequence, 158,404 31 px
        # subsets, each starting from the frame before
        {"name": "frame_2048_31px", "kind": "frame", "w": 2048, "h": 2048, "subset": 31, "step": 5,
         "interp": "keys", "tol": 1e-5, "pixel": "f32", "filter": 0, "field": "wave", "frame": 4},
        # a dense field over a crack: small subsets every 4 px, some of which fail
        {"name": "crack_4096_21px", "kind": "frame", "w": 4096, "h": 4096, "subset": 21, "step": 4,
         "interp": "keys", "tol": 1e-4, "pixel": "f32", "filter": 0, "field": "crack", "frame": 3},
        # coarse speckle wants large subsets
        {"name": "frame_2048_61px", "kind": "frame", "w": 2048, "h": 2048, "subset": 61, "step": 20,
         "interp": "keys", "tol": 1e-4, "pixel": "f32", "filter": 0, "field": "wave", "frame": 2},
        # 16-bit camera frames, low-pass filtered, the cheaper interpolant
        {"name": "bicubic_1024_25px", "kind": "frame", "w": 1024, "h": 1024, "subset": 25, "step": 6,
         "interp": "bicubic", "tol": 1e-4, "pixel": "u16", "filter": 7, "field": "wave", "frame": 5},
        # arbitrary-shape subsets (circles, polygons) with the quadratic shape function
        {"name": "quadratic_shapes", "kind": "shapes", "w": 2048, "h": 2048, "n": 6000, "solver": "quadratic"},
        # thin subsets, whose gradients are too poor: Nelder-Mead
        {"name": "simplex_thin", "kind": "shapes", "w": 2048, "h": 2048, "n": 2400, "solver": "simplex"},
        # tracked parts that occlude each other: shapes, obstructions, blocking subsets
        {"name": "tracking_900", "kind": "tracking", "w": 2048, "h": 2048, "side": 30, "spacing": 60},
        # a displacement model fitted through the objective: value and both derivatives
        {"name": "adjoint_1024_25px", "kind": "adjoint", "w": 1024, "h": 1024, "subset": 25, "step": 7,
         "objective": 0, "image": True},
        # strain from the subset field after a frame
        {"name": "strain_158k", "kind": "strain", "nx": 398, "ny": 398, "step": 5, "window": 41},
        # a large frame filtered and differentiated on the device
        {"name": "filter_4096", "kind": "filter", "w": 4096, "h": 4096, "mask": 7, "smooth": True},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["probe", "frame", "frame", "frame", "shapes", "shapes", "tracking", "adjoint", "strain",
                       "filter"])
    if kind == "probe":
        s = _log(rng, 300, 1400)
        return {"kind": kind, "w": s, "h": s + rng.randrange(0, 90), "n": _log(rng, 1, 40),
                "subset": rng.choice([15, 21, 31, 41, 51]), "interp": rng.choice(["bilinear", "bicubic", "keys"]),
                "pixel": rng.choice(["u8", "u16", "f32"])}
    if kind == "frame":
        s = _log(rng, 300, 2100)
        subset = rng.choice([11, 15, 21, 27, 31, 35, 41, 51, 61])
        return {"kind": kind, "w": s, "h": max(300, s - rng.randrange(0, 97)), "subset": subset,
                "step": rng.randrange(5, 5 + subset // 2), "interp": rng.choice(["keys", "keys", "bicubic", "bilinear"]),
                "tol": rng.choice([1e-3, 1e-4, 1e-5]), "pixel": rng.choice(["u8", "u16", "f32"]),
                "filter": rng.choice([0, 0, 5, 7, 9]), "field": rng.choice(["shift", "wave", "crack"]),
                "frame": rng.randrange(1, 9)}
    if kind == "shapes":
        return {"kind": kind, "w": rng.randrange(900, 2300), "h": rng.randrange(900, 2300), "n": _log(rng, 60, 6000),
                "solver": rng.choice(["quadratic", "affine", "simplex"])}
    if kind == "tracking":
        return {"kind": kind, "w": 2048, "h": 2048, "side": rng.randrange(3, 40), "spacing": rng.randrange(38, 51)}
    if kind == "adjoint":
        s = _log(rng, 200, 1300)
        return {"kind": kind, "w": s, "h": s + rng.randrange(0, 70), "subset": rng.choice([15, 21, 25, 31, 41]),
                "step": rng.randrange(6, 15), "objective": rng.choice([0, 1]), "image": rng.choice([True, True, False])}
    if kind == "strain":
        step = rng.randrange(3, 11)
        return {"kind": kind, "nx": _log(rng, 20, 600), "ny": _log(rng, 20, 600), "step": step,
                "window": step * rng.randrange(4, 10) + rng.randrange(0, 3)}
    return {"kind": kind, "w": _log(rng, 200, 4600), "h": _log(rng, 200, 4000), "mask": rng.choice([5, 7, 9, 11, 13]),
            "smooth": rng.choice([True, False])}


# ---- inputs -----------------------------------------------------------------
def _field(kind, k, h):
    """Displacement field of frame k: (X, Y) -> (u, v)."""
    if kind == "shift":
        return lambda X, Y: (torch.full_like(X, 0.37 * k), torch.full_like(Y, -0.41 * k))
    if kind == "crack":
        return syn.config5_field(h, 2.0 * k / 8, 0.003 * k / 8)
    return syn.config2_field(k, 10)


def _pixels(img, pixel):
    """The image as a camera of that depth gives it (a CUDA tensor)."""
    if pixel == "u8":
        return img.clamp(0, 255).round().to(torch.uint8)
    if pixel == "u16":
        return img.clamp(0, 65535).round().to(torch.int32).to(torch.uint16)
    return img


def _speckle(w, h, seed, pixel, big):
    lo, hi = (20.0, 230.0) if pixel == "u8" else (1000.0, 64000.0)
    r = (3.0, 5.0) if big else (2.0, 4.0)
    ref = syn.speckle_image(w, h, seed=seed, r_min=r[0], r_max=r[1], grey_lo=lo, grey_hi=hi, blur_sigma=0.8,
                            device=DEV)
    return ref, (1.0 if pixel == "u8" else 50.0), (255.0 if pixel == "u8" else 65535.0)


def _at(field, cx, cy):
    u, v = field(torch.from_numpy(np.asarray(cx, np.float64)), torch.from_numpy(np.asarray(cy, np.float64)))
    return u.numpy(), v.numpy()


def _state(**kw):
    torch.cuda.synchronize()
    return kw


def _frame(case, seed):
    w, h, pixel = case["w"], case["h"], case["pixel"]
    ref, noise, top = _speckle(w, h, seed, pixel, case["subset"] > 24)
    field = _field(case["field"], case["frame"], h)
    deff = syn.warp_image(ref, field, noise_sigma=noise, seed=seed + 7, clip=(0.0, top))
    p = abi.default_params(subset_size=case["subset"], enable_rotation=1, enable_normal_strain=1,
                           enable_shear_strain=1, fast_solver_tolerance=case["tol"], interpolation=INTERP[case["interp"]])
    if case["filter"]:
        p.gauss_filter_images = 1
        p.gauss_filter_mask_size = case["filter"]
    cx, cy = syn.grid_points(w, h, case["subset"], case["step"])
    f = syn.init_fields(cx, cy)
    # the frame before has been solved
    f[:, abi.F_DISP_X], f[:, abi.F_DISP_Y] = (a.astype(np.float32) for a in _at(_field(case["field"], case["frame"] - 1, h),
                                                                                cx, cy))
    s = Schema(p, stream=torch.cuda.current_stream())
    s.set_ref_image(_pixels(ref, pixel))
    s.set_fields(f)
    f = torch.from_numpy(f).to(DEV)
    return _state(s=s, rows=f, deff=_pixels(deff, pixel).contiguous(), out=torch.empty_like(f))


def _run_frame(st):
    s = st["s"]
    s.load_fields(st["rows"])
    s.set_def_image(st["deff"])
    s.execute_correlation()
    s.store_fields(st["out"])
    return st["out"]


def _probe(case, seed):
    w, h, pixel = case["w"], case["h"], case["pixel"]
    ref, noise, top = _speckle(w, h, seed, pixel, False)
    deff = syn.warp_image(ref, _field("shift", 1, h), noise_sigma=noise, seed=seed + 7, clip=(0.0, top))
    p = abi.default_params(subset_size=case["subset"], enable_rotation=1, enable_normal_strain=1,
                           enable_shear_strain=1, fast_solver_tolerance=1e-4, interpolation=INTERP[case["interp"]])
    rng = np.random.default_rng(seed)
    m = case["subset"] + 8
    f = syn.init_fields(rng.integers(m, w - m, case["n"]).astype(np.float64),
                        rng.integers(m, h - m, case["n"]).astype(np.float64))
    s = Schema(p, stream=torch.cuda.current_stream())
    s.set_ref_image(_pixels(ref, pixel).cpu().numpy())
    s.set_fields(f)
    return _state(s=s, rows=f, deff=_pixels(deff, pixel).cpu().numpy())


def _run_probe(st):
    s = st["s"]
    s.load_fields(st["rows"])
    s.set_def_image(st["deff"])
    s.execute_correlation()
    return s.fields()


_BANK = {}


def _bank():
    """Pixel offsets of 96 circles, ellipses and convex polygons: (kind, dx, dy) each."""
    if not _BANK:
        cx, cy, offs, px, py, kind, _ = syn.mixed_subsets(400, 400, 96, seed=33)
        for i in range(96):
            a, b = offs[i], offs[i + 1]
            _BANK[i] = (int(kind[i]), (px[a:b] - int(cx[i])).astype(np.int32), (py[a:b] - int(cy[i])).astype(np.int32))
    return _BANK


def _shapes(case, seed):
    w, h, n = case["w"], case["h"], case["n"]
    ref, noise, top = _speckle(w, h, seed, "u8", False)
    field = syn.config3_field(w, h)
    deff = syn.warp_image(ref, field, noise_sigma=noise, seed=seed + 7, clip=(0.0, top))
    rng = np.random.default_rng(seed)
    thin = case["solver"] == "simplex"
    bank = [b for b in _bank().values() if (b[0] == 1) == thin]
    pick = rng.integers(0, len(bank), n)
    cx, cy = rng.integers(70, w - 70, n), rng.integers(70, h - 70, n)
    offs = np.zeros(n + 1, np.int64)
    offs[1:] = np.cumsum([len(bank[k][1]) for k in pick])
    px = np.concatenate([bank[k][1] for k in pick]) + np.repeat(cx, np.diff(offs))
    py = np.concatenate([bank[k][2] for k in pick]) + np.repeat(cy, np.diff(offs))
    quad = case["solver"] == "quadratic"
    u, v = (np.round(a) for a in _at(field, cx, cy))
    f = syn.init_fields(cx.astype(np.float64), cy.astype(np.float64), quadratic=quad)
    if quad:
        p = abi.default_params(shape_function=abi.QUADRATIC_SF, subset_size=0, fast_solver_tolerance=1e-3)
        f[:, abi.F_QUAD_A + 5], f[:, abi.F_QUAD_A + 11] = u, v
    else:
        p = abi.default_params(subset_size=0, enable_rotation=1, fast_solver_tolerance=1e-3)
        f[:, abi.F_DISP_X], f[:, abi.F_DISP_Y] = u, v
    s = Schema(p, stream=torch.cuda.current_stream())
    s.set_ref_image(ref)
    s.set_fields(f)
    s.set_subset_pixels(offs.astype(np.int32), px.astype(np.int32), py.astype(np.int32))
    if thin:
        s.set_force_simplex(np.ones(n, np.uint8))
    f = torch.from_numpy(f).to(DEV)
    return _state(s=s, rows=f, deff=deff, out=torch.empty_like(f))


def _tracking(case, seed):
    w, h, side, step = case["w"], case["h"], case["side"], case["spacing"]
    ref, noise, top = _speckle(w, h, seed, "f32", True)
    deff = syn.warp_image(ref, syn.config2_field(1, 10), noise_sigma=noise, seed=seed + 7, clip=(0.0, top))
    rng = np.random.default_rng(seed)
    shapes, vx, vy, cx, cy, blockers = [], [], [], [], [], []
    x0, y0 = (w - (side - 1) * step) // 2, (h - (side - 1) * step) // 2
    for j in range(side):
        for i in range(side):
            k, x, y = len(cx), x0 + i * step, y0 + j * step
            cx.append(float(x))
            cy.append(float(y))
            if rng.random() < 0.5:
                shapes.append(abi.rectangle(k, x, y, int(rng.integers(29, 41)), int(rng.integers(29, 41))))
            else:
                m = int(rng.integers(5, 8))
                ang = np.sort(rng.uniform(0, 2 * np.pi, m))
                rad = rng.uniform(14, 20, m)
                shapes.append(abi.polygon(k, len(vx), m))
                vx += list(np.round(x + rad * np.cos(ang)).astype(int))
                vy += list(np.round(y + rad * np.sin(ang)).astype(int))
            if rng.random() < 0.3:
                shapes.append(abi.rectangle(k, x + int(rng.integers(-6, 7)), y + int(rng.integers(-6, 7)),
                                            int(rng.integers(5, 10)), int(rng.integers(5, 10)),
                                            role=abi.ROLE_OBSTRUCTED))
            blockers.append(([k + 1] if i + 1 < side else []) + ([k - 1] if i > 0 and k % 10 == 0 else []))
    p = abi.default_params(subset_size=0, enable_rotation=1, correlation_routine=abi.TRACKING_ROUTINE,
                           override_force_simplex=1, fast_solver_tolerance=1e-3)
    f = syn.init_fields(np.asarray(cx), np.asarray(cy))
    s = Schema(p, stream=torch.cuda.current_stream())
    s.set_ref_image(ref)
    s.set_fields(f)
    s.set_subset_shapes(shapes, np.asarray(vx or [0], np.int32), np.asarray(vy or [0], np.int32))
    s.set_blocking(blockers)
    f = torch.from_numpy(f).to(DEV)
    return _state(s=s, rows=f, deff=deff, out=torch.empty_like(f))


def _adjoint(case, seed):
    w, h = case["w"], case["h"]
    ref, noise, top = _speckle(w, h, seed, "u8", False)
    field = syn.config2_field(8, 10)
    deff = syn.warp_image(ref, field, noise_sigma=noise, seed=seed + 7, clip=(0.0, top))
    p = abi.default_params(subset_size=case["subset"], enable_rotation=1, enable_normal_strain=1, enable_shear_strain=1)
    cx, cy = syn.grid_points(w, h, case["subset"], case["step"])
    rng = np.random.default_rng(seed)
    f = syn.init_fields(cx, cy)
    # a fit on its way: near the field, with its first derivatives off
    u, v = _at(field, cx, cy)
    f[:, abi.F_DISP_X] = (u + rng.normal(0, 0.1, len(cx))).astype(np.float32)
    f[:, abi.F_DISP_Y] = (v + rng.normal(0, 0.1, len(cx))).astype(np.float32)
    f[:, abi.F_ROT_Z:abi.F_SHEAR_XY + 1] = rng.normal(0, 2e-3, (len(cx), 4)).astype(np.float32)
    weights = torch.from_numpy(rng.uniform(0.5, 1.5, len(cx))).to(DEV)
    s = Schema(p, stream=torch.cuda.current_stream())
    s.set_ref_image(ref)
    s.set_fields(f)
    s.set_def_image(deff)
    return _state(s=s, rows=torch.from_numpy(f).to(DEV), weights=weights, ref=ref, deff=deff, case=dict(case))


def _run_adjoint(st):
    d = torch.zeros_like(st["deff"]) if st["case"]["image"] else None
    value, dparams = st["s"].adjoint(st["rows"], st["weights"], objective=st["case"]["objective"], ddef=d)
    return {"value": value, "dparams": dparams, "ddef": d} if d is not None else {"value": value, "dparams": dparams}


def _strain_rows(case, seed):
    nx, ny, step = case["nx"], case["ny"], case["step"]
    X, Y = np.meshgrid(30.0 + step * np.arange(nx), 30.0 + step * np.arange(ny))
    f = syn.init_fields(X.ravel(), Y.ravel())
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(100, 160, 2)
    f[:, abi.F_DISP_X] = (0.5 * np.sin(2 * np.pi * f[:, 0] / a) + 0.002 * f[:, 0] + rng.normal(0, 0.01, len(f))).astype(np.float32)
    f[:, abi.F_DISP_Y] = (0.3 * np.cos(2 * np.pi * f[:, 1] / b) + 0.002 * f[:, 1] + rng.normal(0, 0.01, len(f))).astype(np.float32)
    f[:, abi.F_SIGMA] = np.where(rng.random(len(f)) < 0.01, -1.0, 0.01)   # a few subsets failed
    return f


def _strain(case, seed):
    f = _strain_rows(case, seed)
    s = Schema(abi.default_params(subset_size=21), stream=torch.cuda.current_stream())
    s.set_fields(f)
    return _state(s=s, window=case["window"],
                  out=torch.empty((len(f), abi.VSG_STRIDE), dtype=torch.float64, device=DEV))


def _run_strain(st):
    s = st["s"]
    abi.check(s.lib.dicegpu_vsg_strain(s.ctx, st["window"], ctypes.c_void_p(st["out"].data_ptr()), 1), "vsg_strain")
    return st["out"]


def _filter(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    img = 100.0 + 900.0 * torch.rand((case["h"], case["w"]), generator=g, device=DEV)
    img = syn.gaussian_blur(img, 1.0).contiguous()
    return _state(img=img, low=torch.empty_like(img), gx=torch.empty_like(img), gy=torch.empty_like(img),
                  mask=case["mask"], method=abi.CONVOLUTION_5_POINT if case["smooth"] else abi.FINITE_DIFFERENCE,
                  lib=abi.load_library())


def _run_filter(st):
    h, w = st["img"].shape
    p = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    abi.check(st["lib"].dicegpu_gauss_filter(w, h, p(st["img"]), p(st["low"]), st["mask"], stream), "gauss_filter")
    abi.check(st["lib"].dicegpu_image_gradients(w, h, p(st["low"]), p(st["gx"]), p(st["gy"]), st["method"], stream),
              "image_gradients")
    return {"low": st["low"], "gx": st["gx"], "gy": st["gy"]}


_PREPARE = {"probe": _probe, "frame": _frame, "shapes": _shapes, "tracking": _tracking, "adjoint": _adjoint,
            "strain": _strain, "filter": _filter}
_RUN = {"probe": _run_probe, "frame": _run_frame, "shapes": _run_frame, "tracking": _run_frame,
        "adjoint": _run_adjoint, "strain": _run_strain, "filter": _run_filter}


def prepare(case, seed):
    st = _PREPARE[case["kind"]](case, 1 + seed % 1000003)
    st["kind"] = case["kind"]
    return st


def run(state):
    return _RUN[state["kind"]](state)


# ---- work ---------------------------------------------------------------------
# Per pixel and pass: map, weights, interpolation, residuals and products of an
# affine Gauss-Newton iteration, of a quadratic one, and of a gamma evaluation.
_GN, _QUAD, _GAMMA = 390.0, 640.0, 200.0


def work(case):
    kind = case["kind"]
    if kind == "filter":
        n = case["w"] * case["h"]
        taps = case["mask"] ** 2 + (2 * 25 if case["smooth"] else 0) + 8
        return {"bytes": 16.0 * n, "flops": 2.0 * taps * n}
    if kind == "strain":
        n = case["nx"] * case["ny"]
        near = math.pi * (case["window"] / (2.0 * case["step"])) ** 2
        return {"bytes": (5 + 8) * 8.0 * n, "flops": n * (near * 24.0 + 150.0)}
    px = {"u8": 1, "u16": 2}.get(case.get("pixel"), 4)
    image = float(case["w"] * case["h"])
    if kind == "adjoint":
        n = len(syn.grid_points(case["w"], case["h"], case["subset"], case["step"])[0])
        pixels = n * case["subset"] ** 2
        return {"bytes": image * (8 + (4 if case["image"] else 0)) + n * (6 + 1 + 1 + 12) * 8.0,
                "flops": pixels * (_GAMMA + 280.0 + (80.0 if case["image"] else 0.0))}
    if kind == "shapes":
        n, pixels = case["n"], case["n"] * (754.0 if case["solver"] == "simplex" else 760.0)
        per = {"quadratic": 4 * _QUAD, "affine": 4 * _GN, "simplex": 60 * _GAMMA}[case["solver"]]
    elif kind == "tracking":
        n = case["side"] ** 2
        pixels, per = n * 840.0, 4 * _GN
    elif kind == "probe":
        n = case["n"]
        pixels, per = n * case["subset"] ** 2, 4 * _GN
    else:
        n = len(syn.grid_points(case["w"], case["h"], case["subset"], case["step"])[0])
        pixels, per = n * case["subset"] ** 2, 4 * _GN
    # the deformed frame and the reference, the rows read and written; four
    # Gauss-Newton iterations and the final gamma, or 60 gamma evaluations
    return {"bytes": image * (px + 4) + n * 512.0, "flops": pixels * (per + _GAMMA)}


# ---- 64-bit values ----------------------------------------------------------------
def exact(case, seed):
    # A correlation frame has no value in 64 bits: its rows are an iterated
    # float solve's, whose last steps and stopping are decided by the float
    # spacing of the coordinates, with iteration counts and status among them.
    kind, seed = case["kind"], 1 + seed % 1000003
    if kind == "filter":
        return _exact_filter(case, seed)
    if kind == "strain":
        return _exact_strain(case, seed)
    if kind == "adjoint":
        return _exact_adjoint(case, seed)
    return None


_MASK = {5: (0.0014, 0.1574, 0.62825), 7: (0.006, 0.0606, 0.2418, 0.3831), 9: (0.0007, 0.0108, 0.0748, 0.2384, 0.3505),
         11: (0.0001, 0.0017, 0.0168, 0.087, 0.2328, 0.3231),
         13: (0.0001, 0.0012, 0.0085, 0.038, 0.1109, 0.2108, 0.2611)}


def _exact_filter(case, seed):
    img = _filter(case, seed)["img"].double()
    h, w = img.shape
    m, r = case["mask"], case["mask"] // 2
    k = torch.tensor(_MASK[m] + _MASK[m][-2::-1], dtype=torch.float64)
    low = img.clone()
    e = r + 1
    acc = torch.zeros((h - 2 * e, w - 2 * e), dtype=torch.float64, device=img.device)
    for i in range(m):
        for j in range(m):
            acc += float(k[i] * k[j]) * img[e - r + j:h - e - r + j, e - r + i:w - e - r + i]
    low[e:h - e, e:w - e] = acc

    def slope(a):   # along the last axis
        n = a.shape[-1]
        d = torch.empty_like(a)
        d[..., :2] = a[..., 1:3] - a[..., :2]
        d[..., n - 2:] = a[..., n - 2:] - a[..., n - 3:n - 1]
        d[..., 2:n - 2] = (a[..., :n - 4] - 8 * a[..., 1:n - 3] + 8 * a[..., 3:n - 1] - a[..., 4:]) / 12
        return d
    out = [slope(low), slope(low.t()).t()]
    if case["smooth"]:
        b = [0.0625, 0.25, 0.375, 0.25, 0.0625]
        for q in range(2):
            g, o = out[q], out[q].clone()
            o[2:h - 2, 2:w - 2] = sum(b[i] * b[j] * g[i:h - 4 + i, j:w - 4 + j] for i in range(5) for j in range(5))
            out[q] = o
    return {"low": low, "gx": out[0].contiguous(), "gy": out[1].contiguous()}


def _exact_strain(case, seed):
    f = _strain_rows(case, seed)
    nx, ny, step = case["nx"], case["ny"], case["step"]
    grid = lambda c: torch.from_numpy(f[:, c].astype(np.float32)).to(DEV).double().reshape(ny, nx)  # noqa: E731
    u, v, valid = grid(abi.F_DISP_X), grid(abi.F_DISP_Y), grid(abi.F_SIGMA) >= 0
    r2 = (case["window"] / 2.0) ** 2 + 1e-5
    R = int(math.sqrt(r2) / step) + 1
    pad = lambda t: torch.nn.functional.pad(t, (R, R, R, R))  # noqa: E731
    pu, pv, ok = pad(u * valid), pad(v * valid), pad(valid.double())
    m = torch.zeros((12, ny, nx), dtype=torch.float64, device=DEV)
    for j in range(-R, R + 1):
        for i in range(-R, R + 1):
            dx, dy = float(i * step), float(j * step)
            if dx * dx + dy * dy >= r2:
                continue
            cut = lambda t: t[R + j:R + j + ny, R + i:R + i + nx]  # noqa: E731
            a, b, c = cut(ok), cut(pu), cut(pv)
            for q, t in enumerate((a, a * dx, a * dy, a * dx * dx, a * dx * dy, a * dy * dy, b, b * dx, b * dy, c, c * dx,
                                   c * dy)):
                m[q] += t
    A = torch.stack([m[0], m[1], m[2], m[1], m[3], m[4], m[2], m[4], m[5]], -1).reshape(ny, nx, 3, 3)
    good = valid & (m[0] >= 3)
    det = torch.linalg.det(A)
    good &= det > 1e-6 * step ** 4
    A = torch.where(good[..., None, None], A, torch.eye(3, dtype=torch.float64, device=DEV))
    cu = torch.linalg.solve(A, m[6:9].permute(1, 2, 0)[..., None])[..., 0]
    cv = torch.linalg.solve(A, m[9:12].permute(1, 2, 0)[..., None])[..., 0]
    ux, uy, vx, vy = cu[..., 1], cu[..., 2], cv[..., 1], cv[..., 2]
    rows = [ux + 0.5 * (ux * ux + vx * vx), vy + 0.5 * (uy * uy + vy * vy), 0.5 * (uy + vx + ux * uy + vx * vy), ux, uy, vx, vy]
    rows = [torch.where(good, t, torch.zeros_like(t)) for t in rows] + [m[0]]
    return torch.stack(rows, -1).reshape(-1, 8)


def _keys(s):
    s = s.abs()
    return torch.where(s < 1, (4.0 / 3 * s - 7.0 / 3) * s * s + 1,
                       torch.where(s < 2, ((-7.0 / 12 * s + 3) * s - 59.0 / 12) * s + 2.5,
                                   ((s / 12 - 2.0 / 3) * s + 1.75) * s - 1.5))


def _dkeys(s):
    a = s.abs()
    d = torch.where(a < 1, (4 * a - 14.0 / 3) * a,
                    torch.where(a < 2, (-1.75 * a + 6) * a - 59.0 / 12, (0.25 * a - 4.0 / 3) * a + 1.75))
    return d * torch.sign(s)


def _exact_adjoint(case, seed):
    st = _adjoint(case, seed)
    ref, deff, rows, sd = st["ref"].double(), st["deff"].double(), st["rows"], st["weights"]
    h, w = deff.shape
    half = case["subset"] // 2
    o = torch.arange(-half, half + 1, device=DEV, dtype=torch.float64)
    dy, dx = (t.reshape(1, -1) for t in torch.meshgrid(o, o, indexing="ij"))
    n = rows.shape[0]
    value = torch.empty(n, dtype=torch.float64, device=DEV)
    dparams = torch.zeros((n, 12), dtype=torch.float64, device=DEV)
    ddef = torch.zeros(h * w, dtype=torch.float64, device=DEV)
    for b in range(0, n, 4000):
        f = rows[b:b + 4000]
        cx, cy, u, v, t, ex, ey, g = (f[:, c:c + 1] for c in range(8))
        Dx, Dy = (1 + ex) * dx + g * dy, (1 + ey) * dy + g * dx
        c, s = torch.cos(t), torch.sin(t)
        X, Y = c * Dx - s * Dy + u + cx, s * Dx + c * Dy + v + cy
        rx, ry = torch.floor(X + 0.5), torch.floor(Y + 0.5)
        live = ((rx >= 4) & (rx < w - 4) & (ry >= 4) & (ry < h - 4)).double()
        ix, iy = torch.floor(X).clamp(2, w - 4), torch.floor(Y).clamp(2, h - 4)
        F = ref.reshape(-1)[((cy + dy) * w + cx + dx).long()]
        G, gx, gy = torch.zeros_like(X), torch.zeros_like(X), torch.zeros_like(X)
        at = [((iy + m - 2) * w + ix + k - 2).long() for m in range(6) for k in range(6)]
        wx = [_keys(X - ix - k + 2) for k in range(6)]
        wy = [_keys(Y - iy - k + 2) for k in range(6)]
        dwx = [_dkeys(X - ix - k + 2) for k in range(6)]
        dwy = [_dkeys(Y - iy - k + 2) for k in range(6)]
        for m in range(6):
            for k in range(6):
                I = deff.reshape(-1)[at[6 * m + k]]
                G += wy[m] * wx[k] * I
                gx += wy[m] * dwx[k] * I
                gy += dwy[m] * wx[k] * I
        cnt = live.sum(1, keepdim=True)
        Ft, Gt = (F - (F * live).sum(1, keepdim=True) / cnt) * live, (G - (G * live).sum(1, keepdim=True) / cnt) * live
        ff, gg, S = (Ft * Ft).sum(1, keepdim=True), (Gt * Gt).sum(1, keepdim=True), (Ft * Gt).sum(1, keepdim=True)
        if case["objective"] == 0:
            value[b:b + 4000] = (2 - 2 * S / (gg * ff).sqrt())[:, 0]
            lam = -2 / (gg * ff).sqrt() * Ft + 2 * S / (gg * (gg * ff).sqrt()) * Gt
        else:
            value[b:b + 4000] = (gg + ff - 2 * S)[:, 0]
            lam = 2 * (Gt - Ft)
        lam = lam * sd[b:b + 4000, None]
        r = (gx, gy, gx * (-s * Dx - c * Dy) + gy * (c * Dx - s * Dy), gx * dx * c + gy * dx * s,
             -gx * dy * s + gy * dy * c, gx * (c * dy - s * dx) + gy * (s * dy + c * dx))
        for i in range(6):
            dparams[b:b + 4000, i] = (lam * r[i]).sum(1)
        if case["image"]:
            for m in range(6):
                for k in range(6):
                    ddef.index_add_(0, at[6 * m + k].reshape(-1), (lam * wy[m] * wx[k]).reshape(-1))
    out = {"value": value, "dparams": dparams}
    return dict(out, ddef=ddef.reshape(h, w)) if case["image"] else out
