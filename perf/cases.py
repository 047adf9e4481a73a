"""Workloads of the library, each one pass through its public entry points.

A case is a dict of plain values. Its "kind" says which call it is:

  evaluate   one metric evaluation (Mattes, mean squares or correlation; value and
             derivative, or the value alone): what an optimizer calls at every step
  bspline    one Mattes value and derivative through a B-spline transform
  pyramid    one level of the multi-resolution schedule (smooth, shrink, resample)
  register   a whole multi-resolution registration, from two images to parameters
  batch      a batch of small registrations: objects built, optimised, destroyed
  train      training steps of the learned initialiser, and the gradients they leave
  gemm       the tensor-core product behind the initialiser's layers, by itself

Images are blob phantoms (a ramp, Gaussian blobs and noise; the moving image is the
same phantom under a rigid pose with noise of its own), made on the GPU from a seed.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "sitk-rs_b200"))

EPS = float(np.finfo(np.float64).eps)
DEV = "cuda"


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------

def _evaluate(size, **kw):
    case = dict(kind="evaluate", nx=size[0], ny=size[1], nz=size[2], sx=1.0, sy=1.0, sz=1.0, metric="mattes",
                transform="affine", bins=32, sampling="none", percentage=1.0, storage="f32", masks=False,
                derivative=True)
    case.update(kw)
    return case


def listed():
    return [
        # the smallest level of a pyramid, or a thumbnail pair: latency and launches count
        _evaluate((64, 64, 64), name="mattes_64_affine", bins=50),
        # the finest level of a rigid registration, sampled: the everyday call
        _evaluate((256, 256, 256), name="mattes_256_versor", transform="versor", sampling="random", percentage=0.1),
        # a line search asks for the value alone; odd sizes, both masks, regular sampling, anisotropic voxels
        _evaluate((181, 217, 179), name="mattes_masked_value", transform="euler", sampling="regular", percentage=0.25,
                  bins=50, sx=0.9, sy=1.1, sz=1.3, masks=True, derivative=False),
        # a large scan with the moving volume stored in 16 bits
        _evaluate((512, 512, 512), name="mattes_512_bf16", transform="euler", sampling="random", percentage=0.2,
                  bins=64, storage="bf16"),
        # same-modality registration, every voxel of an odd-sized, anisotropic scan
        _evaluate((240, 239, 155), name="mean_squares_full", metric="mean_squares", transform="affine", sx=0.9, sy=0.9,
                  sz=1.5),
        # the same with intensities that differ by gain and offset, sampled
        _evaluate((256, 256, 256), name="correlation_256", metric="correlation", transform="versor", sampling="random",
                  percentage=0.1),
        # deformable registration on an 8x8x8 mesh
        dict(name="bspline_256_mesh8", kind="bspline", nx=256, ny=256, nz=256, mx=8, my=8, mz=8, bins=32,
             sampling="random", percentage=0.1),
        # a coarse level of the schedule; images that fill the card's caches and no even sizes
        dict(name="pyramid_250", kind="pyramid", nx=251, ny=256, nz=243, sigma=2.0, factor=4, sx=1.0, sy=0.9, sz=1.1),
        # a whole three-level rigid registration of a full-size pair
        dict(name="register_256", kind="register", nx=256, ny=256, nz=256, levels=3, bins=32, percentage=0.1,
             transform="versor", iterations=60),
        # a study's worth of small pairs of uneven sizes
        dict(name="batch_24", kind="batch", pairs=24, smallest=48, largest=112, bins=50, percentage=0.2, iterations=50),
        # four batches of an epoch
        dict(name="train_64", kind="train", batch=64, steps=4),
        # a product as large as the layers' together
        dict(name="gemm_4096", kind="gemm", m=4096, n=4096, k=4096, pad=0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sampling(rng):
    return rng.choice([("none", 1.0), ("regular", round(rng.uniform(0.05, 0.6), 3)),
                       ("random", round(rng.uniform(0.05, 0.6), 3))])


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "bspline", "pyramid", "register", "batch", "train", "gemm"])
    if kind == "evaluate":
        edge = _log(rng, 40, 300)
        size = [max(32, int(edge * rng.uniform(0.7, 1.1))) for _ in range(3)]
        s, p = _sampling(rng)
        return _evaluate(size, metric=rng.choice(["mattes", "mattes", "mean_squares", "correlation"]),
                         transform=rng.choice(["affine", "euler", "versor", "translation"]),
                         bins=rng.choice([16, 32, 50, 64, 100]), sampling=s, percentage=p,
                         storage=rng.choice(["f32", "bf16"]), masks=rng.random() < 0.3, derivative=rng.random() < 0.7,
                         sx=round(rng.uniform(0.6, 1.5), 2), sy=round(rng.uniform(0.6, 1.5), 2),
                         sz=round(rng.uniform(0.8, 2.5), 2))
    if kind == "bspline":
        edge = _log(rng, 64, 256)
        s, p = rng.choice([("regular", 0.25), ("random", 0.1), ("random", round(rng.uniform(0.05, 0.3), 3))])
        return dict(kind=kind, nx=edge, ny=max(48, int(edge * rng.uniform(0.7, 1.0))),
                    nz=max(48, int(edge * rng.uniform(0.6, 1.0))), mx=rng.randint(3, 14), my=rng.randint(3, 14),
                    mz=rng.randint(3, 14), bins=rng.choice([32, 50]), sampling=s, percentage=p)
    if kind == "pyramid":
        edge = _log(rng, 48, 256)
        return dict(kind=kind, nx=edge, ny=max(20, int(edge * rng.uniform(0.5, 1.1))),
                    nz=max(20, int(edge * rng.uniform(0.3, 1.1))), sigma=rng.choice([1.0, 2.0, 3.5]),
                    factor=rng.choice([1, 2, 3, 4]), sx=round(rng.uniform(0.6, 1.5), 2), sy=1.0,
                    sz=round(rng.uniform(0.8, 2.5), 2))
    if kind == "register":
        edge = _log(rng, 64, 240)
        return dict(kind=kind, nx=edge, ny=max(48, int(edge * rng.uniform(0.7, 1.0))),
                    nz=max(48, int(edge * rng.uniform(0.7, 1.0))), levels=rng.choice([2, 3]),
                    bins=rng.choice([32, 50]), percentage=round(rng.uniform(0.05, 0.3), 3),
                    transform=rng.choice(["versor", "euler", "affine"]), iterations=rng.randint(20, 60))
    if kind == "batch":
        lo = rng.randint(32, 64)
        return dict(kind=kind, pairs=rng.randint(3, 24), smallest=lo, largest=lo + rng.randint(8, 48),
                    bins=rng.choice([32, 50]), percentage=round(rng.uniform(0.1, 0.3), 3),
                    iterations=rng.randint(20, 50))
    if kind == "train":
        return dict(kind=kind, batch=_log(rng, 5, 64), steps=rng.randint(1, 4))
    # the layers' own shapes (tall, narrow, or deep in K), general ones and odd ones
    shape = rng.choice(["layer", "general", "general"])
    if shape == "layer":
        m, n, k = rng.choice([(4096, 16, 56), (512, 32, 432), (64, 64, 864), (8, 128, 1728), (1, 256, 1024)])
        b = rng.randint(3, 64)
        m, n, k = rng.choice([(m * b, n, k), (n, k, m * b), (m * b, k, n)])
    else:
        m, n, k = _log(rng, 64, 4096), _log(rng, 16, 4096), _log(rng, 48, 4096)
        if rng.random() < 0.7:
            k = (k + 7) // 8 * 8
    return dict(kind=kind, m=m, n=n, k=k, pad=rng.choice([0, 0, 8, 16]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) * 7919 + 13)


def _uniform(g, lo, hi, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo


def _rotation(angles):
    cx, cy, cz = torch.cos(angles).unbind()
    sx, sy, sz = torch.sin(angles).unbind()
    one, zero = torch.ones_like(cx), torch.zeros_like(cx)
    rx = torch.stack([one, zero, zero, zero, cx, -sx, zero, sx, cx]).reshape(3, 3)
    ry = torch.stack([cy, zero, sy, zero, one, zero, -sy, zero, cy]).reshape(3, 3)
    rz = torch.stack([cz, -sz, zero, sz, cz, zero, zero, zero, one]).reshape(3, 3)
    return rz @ rx @ ry


def _phantom(size, spacing, centres, sigma, amplitude, ramp, noise, g):
    """A ramp, Gaussian blobs (physical centres) and noise on an (nz, ny, nx) grid with its origin at zero."""
    at = [torch.arange(size[d], device=DEV, dtype=torch.float64) * spacing[d] for d in range(3)]
    e = [torch.exp(-0.5 * ((at[d][None, :] - centres[:, d:d + 1]) / sigma[:, None]) ** 2).float() for d in range(3)]
    yz = (amplitude.float()[:, None, None] * e[2][:, :, None] * e[1][:, None, :]).reshape(len(sigma), -1)
    vol = (yz.t() @ e[0]).reshape(size[2], size[1], size[0])
    span = sum((size[d] - 1) * spacing[d] for d in range(3)) + 1e-9
    vol += 20.0
    for d, shape in ((0, (1, 1, -1)), (1, (1, -1, 1)), (2, (-1, 1, 1))):
        vol += (40.0 * ramp[d] * at[d] / span).float().reshape(shape)
    vol += noise * torch.randn(vol.shape, generator=g, device=DEV)
    return vol


def _pair(size, spacing, seed, blobs=40, shift=3.0, turn=0.05):
    """Fixed and moving volumes, the rigid pose between them (angles, translation) and the centre it turns about."""
    g = _gen(seed)
    extent = torch.tensor([(size[d] - 1) * spacing[d] for d in range(3)], device=DEV, dtype=torch.float64)
    centres = _uniform(g, 0.0, 1.0, blobs, 3) * extent
    small = float(extent.min())
    sigma = _uniform(g, 0.03, 0.1, blobs) * max(small, 40.0)
    amplitude = _uniform(g, 50.0, 200.0, blobs)
    angles = _uniform(g, -turn, turn, 3)
    offset = _uniform(g, -shift, shift, 3)
    centre = extent / 2
    moved = (centres - centre) @ _rotation(angles).t() + centre + offset
    fixed = _phantom(size, spacing, centres, sigma, amplitude, (1.0, 0.5, 0.25), 5.0, g)
    moving = _phantom(size, spacing, moved, sigma, amplitude, (1.0, 0.5, 0.25), 5.0, g)
    return fixed, moving, angles.cpu().numpy(), offset.cpu().numpy(), centre.cpu().numpy()


def _pose(kind, seed, angles, offset, centre):
    """Parameters near the pose between the images, as an optimizer meets them on its way: (parameters, centre)."""
    r = np.random.Generator(np.random.PCG64(seed))
    a = angles + r.uniform(-0.02, 0.02, 3)
    t = offset + r.uniform(-1.0, 1.0, 3)
    if kind == "translation":
        return t, None
    if kind == "euler":
        return np.concatenate([a, t]), centre
    if kind == "versor":
        return np.concatenate([np.sin(a / 2.0), t]), centre
    m = _rotation(torch.tensor(a, device=DEV)).cpu().numpy() + r.uniform(-0.02, 0.02, (3, 3))
    return np.concatenate([m.ravel(), t]), centre


def _transform(kind, p, centre):
    import sitk_b200 as sb
    if kind == "translation":
        return sb.TranslationTransform(p)
    if kind == "euler":
        return sb.Euler3DTransform(p[:3], p[3:], centre)
    if kind == "versor":
        return sb.VersorRigid3DTransform(p[:3], p[3:], centre)
    return sb.AffineTransform(p[:9].reshape(3, 3), p[9:], centre)


def _image(volume, spacing):
    import sitk_b200 as sb
    torch.cuda.synchronize()
    nz, ny, nx = volume.shape
    return sb.DeviceImage.from_device_ptr(volume.data_ptr(), (nx, ny, nz), spacing)


def _masks(case, seed):
    """An ellipsoid of the fixed image (1 inside) and a box of the moving one with a hole in it, on the host."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    z, y, x = np.meshgrid(np.linspace(-1, 1, nz), np.linspace(-1, 1, ny), np.linspace(-1, 1, nx), indexing="ij",
                          sparse=True)
    r = np.random.Generator(np.random.PCG64(seed + 5))
    a = r.uniform(0.8, 0.95, 3)
    fixed = ((x / a[0]) ** 2 + (y / a[1]) ** 2 + (z / a[2]) ** 2 <= 1.0)
    moving = (np.abs(x) < 0.95) & (np.abs(y) < 0.97) & (z > -0.9) & ((x - 0.3) ** 2 + y ** 2 + z ** 2 > 0.02)
    return fixed.astype(np.float32), np.ascontiguousarray(moving.astype(np.uint8))


def _geometry(case):
    return ((case["nx"], case["ny"], case["nz"]),
            (case.get("sx", 1.0), case.get("sy", 1.0), case.get("sz", 1.0)))


_STRATEGY = {"none": 0, "regular": 1, "random": 2}


def _evaluate_inputs(case, seed):
    size, spacing = _geometry(case)
    fixed, moving, angles, offset, centre = _pair(size, spacing, seed)
    p, c = _pose(case["transform"], seed, angles, offset, centre)
    masks = _masks(case, seed) if case["masks"] else (None, None)
    return fixed, moving, masks, p, c


def _bspline_inputs(case, seed):
    size, spacing = _geometry(case)
    fixed, moving, _, _, _ = _pair(size, spacing, seed, shift=1.0, turn=0.01)
    n = (case["mx"] + 3) * (case["my"] + 3) * (case["mz"] + 3)
    coef = np.random.Generator(np.random.PCG64(seed)).normal(0.0, 0.8, 3 * n)
    return fixed, moving, coef


CHANNELS = (2, 16, 32, 64, 128)
LAYERS = tuple((CHANNELS[i + 1], 27 * CHANNELS[i]) for i in range(4)) + ((256, 1024), (12, 256))


def _train_inputs(case, seed):
    """Per step: normalised inputs and encoded targets; and the weights the steps start from."""
    g = _gen(seed)
    b, steps = case["batch"], case["steps"]
    x = torch.randn((steps, b, 32, 32, 32, 2), generator=g, device=DEV)
    t = torch.rand((steps, b, 12), generator=g, device=DEV) * 0.5 + 0.5
    weights = []
    for i, (o, k) in enumerate(LAYERS):
        bound = math.sqrt(6.0 / k) * (0.1 if i == 5 else 1.0)
        w = (torch.rand((o, k), generator=g, device=DEV) * 2 - 1) * bound
        weights.append((w, 0.05 * torch.randn((o,), generator=g, device=DEV)))
    return x, t, weights


def _gemm_inputs(case, seed):
    g = _gen(seed)
    a = torch.randn((case["m"], case["k"] + case["pad"]), generator=g, device=DEV).to(torch.bfloat16)
    b = torch.randn((case["n"], case["k"] + case["pad"]), generator=g, device=DEV).to(torch.bfloat16)
    return a, b


LEARNING_RATE = 1e-4


def prepare(case, seed):
    import sitk_b200 as sb
    kind = case["kind"]
    if kind == "evaluate":
        size, spacing = _geometry(case)
        fixed, moving, masks, p, c = _evaluate_inputs(case, seed)
        f, m = _image(fixed, spacing), _image(moving, spacing)
        cls = {"mattes": sb.DeviceMattesMetric, "mean_squares": sb.DeviceMeanSquaresMetric,
               "correlation": sb.DeviceCorrelationMetric}[case["metric"]]
        kw = dict(bins=case["bins"]) if case["metric"] == "mattes" else {}
        metric = cls.from_device_sampled(f, m, fixed_mask=masks[0], moving_mask=masks[1],
                                         strategy=_STRATEGY[case["sampling"]], percentage=case["percentage"],
                                         seed=seed, moving_storage=case["storage"], **kw)
        f.free()
        m.free()
        return {"kind": kind, "metric": metric, "transform": _transform(case["transform"], p, c),
                "derivative": case["derivative"]}
    if kind == "bspline":
        from sitk_b200.transforms import BSplineTransform
        size, spacing = _geometry(case)
        fixed, moving, coef = _bspline_inputs(case, seed)
        f, m = _image(fixed, spacing), _image(moving, spacing)
        metric = sb.DeviceMattesMetric.from_device_sampled(f, m, bins=case["bins"], seed=seed,
                                                           strategy=_STRATEGY[case["sampling"]],
                                                           percentage=case["percentage"])
        t = BSplineTransform.from_image_domain(f.geo, (case["mx"], case["my"], case["mz"]))
        t.set_parameters(coef)
        f.free()
        m.free()
        return {"kind": kind, "metric": metric, "transform": t}
    if kind in ("pyramid", "register"):
        size, spacing = _geometry(case)
        fixed, moving, angles, offset, centre = _pair(size, spacing, seed)
        return {"kind": kind, "case": dict(case), "fixed": _image(fixed, spacing), "moving": _image(moving, spacing),
                "seed": seed}
    if kind == "batch":
        r = np.random.Generator(np.random.PCG64(seed))
        state = {"kind": kind, "case": dict(case), "fixed": [], "moving": [], "centres": [], "seed": seed}
        for i in range(case["pairs"]):
            n = int(r.integers(case["smallest"], case["largest"] + 1))
            fixed, moving, _, _, centre = _pair((n, n, n), (1.0, 1.0, 1.0), seed * 100 + i, blobs=20)
            state["fixed"].append(_image(fixed, (1.0, 1.0, 1.0)))
            state["moving"].append(_image(moving, (1.0, 1.0, 1.0)))
            state["centres"].append(centre)
        return state
    if kind == "train":
        from sitk_b200.initnet import InitNet
        x, t, weights = _train_inputs(case, seed)
        net = InitNet(seed=seed, max_batch=case["batch"])
        for i, (w, b) in enumerate(weights):
            net.set(i, w.cpu().numpy(), b.cpu().numpy())
        return {"kind": kind, "net": net, "x": x, "t": t}
    a, b = _gemm_inputs(case, seed)
    vp, ci = ctypes.c_void_p, ctypes.c_int
    call = sb._lib.load().mi_gemm_bf16_tn
    call.argtypes = [vp, ci, ci, ci, vp, ci, vp, ci, vp, ci]
    call.restype = ci
    torch.cuda.synchronize()
    return {"kind": kind, "call": call, "ctx": sb.default_context(), "a": a, "b": b, "k": case["k"],
            "c": torch.empty((case["m"], case["n"]), device=DEV)}


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------

class _Volume:
    """A device image handed on as a tensor, without a copy; the image lives as long as the tensor."""

    def __init__(self, image):
        nx, ny, nz = image.size
        self.image = image
        self.__cuda_array_interface__ = {"shape": (nz, ny, nx), "typestr": "<f4", "strides": None, "version": 3,
                                         "data": (image.device_ptr(), False)}


def run(state):
    kind = state["kind"]
    if kind == "evaluate":
        if not state["derivative"]:
            return {"value": state["metric"].value(state["transform"])}
        r = state["metric"].evaluate(state["transform"])
        return {"value": r.value, "derivative": r.derivative, "valid": r.valid_points}
    if kind == "bspline":
        r = state["metric"].evaluate(state["transform"])
        return {"value": r.value, "derivative": r.derivative, "valid": r.valid_points}
    if kind == "pyramid":
        from sitk_b200.metric import pyramid_level
        c = state["case"]
        level = pyramid_level(state["fixed"], state["moving"], c["sigma"], c["factor"])
        return [torch.as_tensor(_Volume(v), device=DEV) for v in level]
    if kind == "register":
        from sitk_b200.registration import centered_initialize, register_multilevel
        c = state["case"]
        centre, t = centered_initialize(state["fixed"], state["moving"])
        start = {"versor": np.zeros(6), "euler": np.zeros(6),
                 "affine": np.concatenate([np.eye(3).ravel(), np.zeros(3)])}[c["transform"]]
        start[-3:] = t
        levels = c["levels"]
        r = register_multilevel(state["fixed"], state["moving"], _transform(c["transform"], start, centre),
                                shrink_factors=[2 ** (levels - 1 - i) for i in range(levels)],
                                smoothing_sigmas=[float(levels - 1 - i) for i in range(levels)], bins=c["bins"],
                                percentage=c["percentage"], seed=state["seed"], iterations=c["iterations"])
        return {"parameters": r.params, "values": [v.value for v in r.levels], "valid": [v.valid_points for v in r.levels],
                "iterations": [v.iterations for v in r.levels]}
    if kind == "batch":
        from sitk_b200.registration import BatchRegistration
        c, n = state["case"], state["case"]["pairs"]
        batch = BatchRegistration(state["fixed"], state["moving"], bins=c["bins"], kind=0, centers=state["centres"],
                                  strategy=2, percentage=c["percentage"], seeds=[state["seed"] + i for i in range(n)])
        start = np.tile(np.concatenate([np.eye(3).ravel(), np.zeros(3)]), (n, 1))
        p, r = batch.register(start, iterations=c["iterations"], autotune=False)
        batch.close()
        return {"parameters": p, "values": np.array([v.value for v in r]),
                "valid": np.array([v.valid_points for v in r]), "iterations": np.array([v.iterations for v in r])}
    if kind == "train":
        net = state["net"]
        losses = [net.train_step(x, t, LEARNING_RATE) for x, t in zip(state["x"], state["t"])]
        return {"losses": losses, "gradients": [net.get(i, grads=True) for i in range(len(LAYERS))]}
    a, b, c = state["a"], state["b"], state["c"]
    status = state["call"](state["ctx"].handle, a.shape[0], b.shape[0], state["k"], a.data_ptr(), a.shape[1], b.data_ptr(),
                           b.shape[1], c.data_ptr(), c.shape[1])
    if status:
        raise RuntimeError("mi_gemm_bf16_tn: status %d" % status)
    return c


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def _sample_count(case):
    n = case["nx"] * case["ny"] * case["nz"]
    if case["sampling"] == "random":
        return int(n * case["percentage"])
    if case["sampling"] == "regular":
        s = max(1, math.ceil(1.0 / case["percentage"]))
        return (n + s - 1) // s
    return n


def work(case):
    kind = case["kind"]
    if kind in ("evaluate", "bspline"):
        n, s = case["nx"] * case["ny"] * case["nz"], _sample_count(case)
        word = 2 if case.get("storage") == "bf16" else 4
        # per sample its fixed value (and voxel, where it is drawn), and the part of the moving volume its cells touch
        b = s * (4 if case["sampling"] == "none" else 8) + word * min(n, 8 * s)
        flops = s * (60 if case.get("derivative", True) else 40)
        if kind == "bspline":
            nper = (case["mx"] + 3) * (case["my"] + 3) * (case["mz"] + 3)
            b += 2 * 3 * nper * 8
            flops = s * (2 * 3 * 64 * 2 + 100)  # the displacement's 64 x 3 products, and the derivative's
        return {"bytes": b, "flops": flops}
    if kind == "pyramid":
        n = case["nx"] * case["ny"] * case["nz"]
        level = n // case["factor"] ** 3
        return {"bytes": 4 * (2 * n + n + level), "flops": 2 * n * 3 * 32 + 40 * level}
    if kind == "register":
        n, b, f = case["nx"] * case["ny"] * case["nz"], 0.0, 0.0
        for i in range(case["levels"]):
            s = int(n // 8 ** (case["levels"] - 1 - i) * case["percentage"])
            b += 12 * n + 10 * (8 * s + 4 * min(n, 8 * s))  # the level's images, and ten evaluations on it
            f += 2 * n * 3 * 32 + 10 * 60 * s
        return {"bytes": b, "flops": f}
    if kind == "batch":
        n = ((case["smallest"] + case["largest"]) / 2) ** 3
        s = n * case["percentage"]
        return {"bytes": case["pairs"] * (8 * n + 20 * (8 * s + 4 * min(n, 8 * s))), "flops": case["pairs"] * 20 * 60 * s}
    if kind == "train":
        b, f = case["batch"], 0.0
        rows = [b * 16 ** 3, b * 8 ** 3, b * 4 ** 3, b * 2 ** 3, b, b]
        for i, ((o, k), r) in enumerate(zip(LAYERS, rows)):
            f += 2.0 * r * o * k * (3 if i else 2)  # forward, weight gradient, input gradient (not of the first layer)
        weights = sum(o * k for o, k in LAYERS)
        acts = sum(r * o for (o, _), r in zip(LAYERS, rows))
        return {"bytes": case["steps"] * (b * 32 ** 3 * 2 * 4 + 2 * 2 * acts + 7 * 4 * weights), "flops": case["steps"] * f}
    m, n, k = case["m"], case["n"], case["k"]
    return {"bytes": 2 * (m * k + n * k) + 4 * m * n, "flops": 2.0 * m * n * k}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------

def _splitmix(seed, count, voxels):
    i = np.arange(1, count + 1, dtype=np.uint64)
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + i * np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return (z % np.uint64(voxels)).astype(np.int64)


def _samples(case, seed, fixed_mask):
    n, count = case["nx"] * case["ny"] * case["nz"], _sample_count(case)
    if case["sampling"] == "random":
        flat = torch.from_numpy(_splitmix(seed, count, n)).to(DEV)
    elif case["sampling"] == "regular":
        flat = torch.arange(count, device=DEV) * max(1, math.ceil(1.0 / case["percentage"]))
    else:
        flat = torch.arange(n, device=DEV)
    if fixed_mask is not None:
        flat = flat[torch.from_numpy(fixed_mask).to(DEV).reshape(-1)[flat] != 0]
    return flat


def _affine_map(kind, p, centre):
    """The matrix and translation about the centre, differentiable in p."""
    if kind == "translation":
        return torch.eye(3, device=DEV, dtype=torch.float64), p, torch.zeros(3, device=DEV, dtype=torch.float64)
    c = torch.tensor(centre, device=DEV)
    if kind == "euler":
        return _rotation(p[:3]), p[3:], c
    if kind == "versor":
        x, y, z = p[:3].unbind()
        w = torch.sqrt(1.0 - x * x - y * y - z * z)
        m = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - z * w), 2 * (x * z + y * w),
                         2 * (x * y + z * w), 1 - 2 * (x * x + z * z), 2 * (y * z - x * w),
                         2 * (x * z - y * w), 2 * (y * z + x * w), 1 - 2 * (x * x + y * y)])
        return m.reshape(3, 3), p[3:], c
    return p[:9].reshape(3, 3), p[9:], c


def _sample_moving(moving, mask, y, size, spacing):
    """Which points lie inside, the trilinear value and the physical gradient (points as three vectors)."""
    c = [y[d] / spacing[d] for d in range(3)]
    ok = torch.ones_like(c[0], dtype=torch.bool)
    for d in range(3):
        ok &= (c[d] >= -0.5) & (c[d] < size[d] - 0.5)
    if mask is not None:
        r = [torch.floor(c[d] + 0.5).clamp(0, size[d] - 1).long() for d in range(3)]
        ok &= torch.from_numpy(mask).to(DEV).reshape(-1)[r[0] + size[0] * (r[1] + size[1] * r[2])] != 0
    lo = [torch.floor(v) for v in c]
    fr = [v - w for v, w in zip(c, lo)]
    value, grad = torch.zeros_like(c[0]), [torch.zeros_like(c[0]) for _ in range(3)]
    flat = moving.reshape(-1)
    for corner in range(8):
        bit = [(corner >> d) & 1 for d in range(3)]
        at = [(lo[d] + bit[d]).clamp(0, size[d] - 1).long() for d in range(3)]
        v = flat[at[0] + size[0] * (at[1] + size[1] * at[2])].double()
        w = [fr[d] if bit[d] else 1.0 - fr[d] for d in range(3)]
        value += w[0] * w[1] * w[2] * v
        for d in range(3):
            a, b = [w[e] for e in range(3) if e != d]
            grad[d] += (1.0 if bit[d] else -1.0) * a * b * v
    return ok, value, [grad[d] / spacing[d] for d in range(3)]


def _b3(u):
    a = u.abs()
    inner = (4.0 - 6.0 * a * a + 3.0 * a * a * a) / 6.0
    return torch.where(a < 1.0, inner, torch.where(a < 2.0, (2.0 - a) ** 3 / 6.0, torch.zeros_like(a)))


def _b3_slope(u):
    a, s = u.abs(), torch.sign(u)
    return torch.where(a < 1.0, s * (-2.0 * a + 1.5 * a * a), torch.where(a < 2.0, -0.5 * s * (2.0 - a) ** 2,
                                                                          torch.zeros_like(a)))


def _mattes(fv, ok, mv, moving_range, bins):
    """-MI, the count of valid samples, which they are, and each one's weight of its moving gradient."""
    lo, hi = moving_range
    fs, ms = float(fv.max() - fv.min()) / (bins - 4), (hi - lo) / (bins - 4)
    ok = ok & (mv >= lo) & (mv <= hi)
    fi = torch.trunc(fv / fs - (float(fv.min()) / fs - 2.0)).clamp(2, bins - 3).long()[ok]
    term = (mv / ms - (lo / ms - 2.0))[ok]
    mi = torch.trunc(term).clamp(2, bins - 3)
    joint = torch.zeros(bins * bins, device=DEV, dtype=torch.float64)
    for t in range(-1, 3):
        joint.index_add_(0, fi * bins + (mi + t).long(), _b3(mi + t - term))
    joint = joint.reshape(bins, bins)
    total, n = joint.sum(), int(ok.sum())
    jp, fm = joint / total, torch.bincount(fi, minlength=bins).double() / total
    mm = jp.sum(0)
    take = (jp > EPS) & (mm > EPS)[None, :] & (fm > EPS)[:, None]
    ratio = torch.where(take, torch.log(torch.where(take, jp / mm[None, :].clamp_min(EPS), torch.ones_like(jp))),
                        torch.zeros_like(jp))
    lf = torch.log(fm.clamp_min(1e-300))[:, None]
    value = -float(torch.where(take, jp * (ratio - lf), torch.zeros_like(jp)).sum())
    weight = torch.zeros_like(term)
    table = ratio.reshape(-1)
    for t in range(-1, 3):
        weight += _b3_slope(mi + t - term) * table[fi * bins + (mi + t).long()]
    return value, n, ok, weight / (ms * n)


def _contract(weight, grad, x, kind, p, centre):
    """The derivative by the parameters of a sum whose derivative by each mapped point is weight times grad."""
    with torch.enable_grad():
        q = torch.tensor(p, device=DEV, dtype=torch.float64, requires_grad=True)
        m, t, c = _affine_map(kind, q, centre)
        g = torch.stack([weight * v for v in grad])
        moment = g @ torch.stack([x[d] - c[d] for d in range(3)]).t()
        loss = (m * moment.detach()).sum() + (t * g.sum(1).detach()).sum()
        return torch.autograd.grad(loss, q)[0].cpu().numpy()


def _exact_evaluate(case, seed):
    size, spacing = _geometry(case)
    fixed, moving, masks, p, centre = _evaluate_inputs(case, seed)
    if case["storage"] == "bf16":
        moving = moving.to(torch.bfloat16).float()
    flat = _samples(case, seed, masks[0])
    at = [flat % size[0], (flat // size[0]) % size[1], flat // (size[0] * size[1])]
    x = [a.double() * s for a, s in zip(at, spacing)]
    m, t, c = _affine_map(case["transform"], torch.tensor(p, device=DEV, dtype=torch.float64), centre)
    y = [sum(m[d, e] * (x[e] - c[e]) for e in range(3)) + c[d] + t[d] for d in range(3)]
    fv = fixed.reshape(-1)[flat].double()
    ok, mv, grad = _sample_moving(moving, masks[1], y, size, spacing)
    if case["metric"] == "mattes":
        seen = moving if masks[1] is None else moving[torch.from_numpy(masks[1]).to(DEV) != 0]
        value, n, ok, weight = _mattes(fv, ok, mv, (float(seen.min()), float(seen.max())), case["bins"])
    else:
        f, v = fv[ok], mv[ok]
        n = int(ok.sum())
        if case["metric"] == "mean_squares":
            value, weight = float(((v - f) ** 2).mean()), 2.0 * (v - f) / n
        else:
            f, v = f - f.mean(), v - v.mean()
            sff, smm, sfm = (f * f).sum(), (v * v).sum(), (f * v).sum()
            value = -float(sfm * sfm / (sff * smm))
            weight = -2.0 * sfm / (sff * smm) * (f - sfm / smm * v)
    if not case["derivative"]:
        return {"value": value}
    d = _contract(weight, [g[ok] for g in grad], [v[ok] for v in x], case["transform"], p, centre)
    return {"value": value, "derivative": d, "valid": None}


def _exact_bspline(case, seed):
    size, spacing = _geometry(case)
    fixed, moving, coef = _bspline_inputs(case, seed)
    flat = _samples(case, seed, None)
    at = [flat % size[0], (flat // size[0]) % size[1], flat // (size[0] * size[1])]
    mesh = (case["mx"], case["my"], case["mz"])
    grid = [v + 3 for v in mesh]
    nper = grid[0] * grid[1] * grid[2]
    x = [a.double() * s for a, s in zip(at, spacing)]
    start, w, inside = [], [], torch.ones_like(x[0], dtype=torch.bool)
    for d in range(3):
        # the domain's first plane lies on the edge of the valid region, as its index rounds
        width = size[d] * spacing[d] / mesh[d]
        u = (x[d] + width) * (1.0 / width)
        inside &= u >= 1.0
        u = u.clamp_min(1.0)
        s = torch.floor(u - 1.0)
        start.append(s.long())
        w.append([_b3(u - s - t) for t in range(4)])
    disp = [torch.zeros_like(x[0]) for _ in range(3)]
    c = torch.tensor(coef, device=DEV)

    def support():
        for t in range(64):
            i, j, k = t & 3, (t >> 2) & 3, t >> 4
            yield (start[0] + i) + grid[0] * ((start[1] + j) + grid[1] * (start[2] + k)), w[0][i] * w[1][j] * w[2][k]

    for q, weight in support():
        for d in range(3):
            disp[d] += torch.where(inside, weight * c[d * nper + q], torch.zeros_like(weight))
    ok, mv, grad = _sample_moving(moving, None, [a + b for a, b in zip(x, disp)], size, spacing)
    fv = fixed.reshape(-1)[flat].double()
    value, n, ok, weight = _mattes(fv, ok, mv, (float(moving.min()), float(moving.max())), case["bins"])
    out = torch.zeros(3 * nper, device=DEV, dtype=torch.float64)
    g = [weight * v[ok] for v in grad]
    for q, s in support():
        s = torch.where(inside, s, torch.zeros_like(s))[ok]
        for d in range(3):
            out.index_add_(0, d * nper + q[ok], s * g[d])
    return {"value": value, "derivative": out.cpu().numpy(), "valid": None}


def _recursive_gaussian(v, sigma):
    """The fourth-order recursive Gaussian along the first axis (sigma in voxels), its border values extended."""
    w1, l1, w2, l2, a1, b1, a2, b2 = 0.6681, -1.3932, 2.0787, -1.3732, 1.3530, 1.8151, -0.3531, 0.0902
    c1, c2, s1, s2 = math.cos(w1 / sigma), math.cos(w2 / sigma), math.sin(w1 / sigma), math.sin(w2 / sigma)
    e1, e2 = math.exp(l1 / sigma), math.exp(l2 / sigma)
    d = [-2 * (e2 * c2 + e1 * c1), 4 * c2 * c1 * e1 * e2 + e1 * e1 + e2 * e2,
         -2 * c1 * e1 * e2 * e2 - 2 * c2 * e2 * e1 * e1, e1 * e1 * e2 * e2]
    n = [a1 + a2, e2 * (b2 * s2 - (a2 + 2 * a1) * c2) + e1 * (b1 * s1 - (a1 + 2 * a2) * c1),
         ((a1 + a2) * c2 * c1 - b1 * c2 * s1 - b2 * c1 * s2) * 2 * e1 * e2 + a2 * e1 * e1 + a1 * e2 * e2,
         e2 * e1 * e1 * (b2 * s2 - a2 * c2) + e1 * e2 * e2 * (b1 * s1 - a1 * c1)]
    sd = 1.0 + sum(d)
    alpha = 2 * sum(n) / sd - n[0]
    n = [q / alpha for q in n]
    m = [n[1] - d[0] * n[0], n[2] - d[1] * n[0], n[3] - d[2] * n[0], -d[3] * n[0]]

    def sweep(order, taps, lag):
        total = sum(taps)
        edge = v[order[0]]
        back = [edge] * 4
        outs = [edge * (total / sd)] * 4
        got = [None] * len(order)
        for i in order:
            if not lag:
                back = [v[i]] + back[:3]
            new = sum(t * b for t, b in zip(taps, back)) - sum(q * o for q, o in zip(d, outs))
            outs = [new] + outs[:3]
            got[i] = new
            if lag:
                back = [v[i]] + back[:3]
        return torch.stack(got)

    index = list(range(v.shape[0]))
    return sweep(index, n, False) + sweep(index[::-1], m, True)


def _exact_pyramid(case, seed):
    size, spacing = _geometry(case)
    fixed, moving, _, _, _ = _pair(size, spacing, seed)
    smooth = []
    for v in (fixed, moving):
        v = v.double()
        for d in range(3):
            v = _recursive_gaussian(v.transpose(0, 2 - d).contiguous(), case["sigma"] / spacing[d]).transpose(0, 2 - d)
        smooth.append(v)
    f = case["factor"]
    if f == 1:
        return [smooth[0].contiguous(), smooth[1].contiguous()]
    # the level is drawn from the smoothed image as it is held, in 32 bits
    level = smooth[0].float().double()
    for d in range(3):
        n = max(size[d] // f, 1)
        c = torch.arange(n, device=DEV, dtype=torch.float64) * f + ((size[d] - 1) / 2.0 - f * (n - 1) / 2.0)
        lo = torch.floor(c)
        fr = (c - lo).reshape([-1 if 2 - d == k else 1 for k in range(3)])
        a, b = lo.clamp(0, size[d] - 1).long(), (lo + 1).clamp(0, size[d] - 1).long()
        level = level.index_select(2 - d, a) * (1.0 - fr) + level.index_select(2 - d, b) * fr
    return [level.contiguous(), smooth[1].contiguous()]


def _exact_train(case, seed):
    x, t, weights = _train_inputs(case, seed)
    x, t = x.double(), t.double()
    params = [v.double() for pair in weights for v in pair]
    m1, m2 = [torch.zeros_like(v) for v in params], [torch.zeros_like(v) for v in params]
    losses, grads = [], []
    for step in range(case["steps"]):
        with torch.enable_grad():
            p = [v.detach().requires_grad_() for v in params]
            a = x[step].permute(0, 4, 1, 2, 3)
            for i in range(4):
                w = p[2 * i].reshape(-1, 3, 3, 3, CHANNELS[i]).permute(0, 4, 1, 2, 3)
                cols = torch.nn.functional.pad(a, (1, 1, 1, 1, 1, 1)).unfold(2, 3, 2).unfold(3, 3, 2).unfold(4, 3, 2)
                a = torch.relu(torch.einsum("bczyxijk,ocijk->bozyx", cols, w) + p[2 * i + 1].reshape(1, -1, 1, 1, 1))
            a = a.permute(0, 2, 3, 4, 1).reshape(a.shape[0], -1)
            a = torch.relu(a @ p[8].t() + p[9]) @ p[10].t() + p[11]
            loss = ((a - t[step]) ** 2).mean()
            grads = torch.autograd.grad(loss, p)
        losses.append(float(loss))
        for i, g in enumerate(grads):
            m1[i] = 0.9 * m1[i] + 0.1 * g
            m2[i] = 0.999 * m2[i] + 0.001 * g * g
            params[i] = params[i] - LEARNING_RATE * (m1[i] / (1 - 0.9 ** (step + 1))) / (
                torch.sqrt(m2[i] / (1 - 0.999 ** (step + 1))) + 1e-8)
    return {"losses": losses, "gradients": [(grads[2 * i], grads[2 * i + 1]) for i in range(len(LAYERS))]}


def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "evaluate":
            return _exact_evaluate(case, seed)
        if kind == "bspline":
            return _exact_bspline(case, seed)
        if kind == "pyramid":
            return _exact_pyramid(case, seed)
        if kind == "train":
            return _exact_train(case, seed)
        if kind == "gemm":
            a, b = _gemm_inputs(case, seed)
            return a[:, :case["k"]].double() @ b[:, :case["k"]].double().t()
    return None  # an optimizer's path: each step depends on the last one's rounding
