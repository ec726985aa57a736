"""The work that this package is timed on: its filters on device-resident images, through the itkg Python API.

A case is a dict of plain values; `kind` says which filter, the rest its sizes (reference axis order, axis 0
fastest) and options.  Sizes and options come from the package's own configurations, tests and benchmark.

  image       GaussianFilter on a 2-D f32 image (1 component, or the 3 of VecPixel<f32, 3>): one small call
  photo       u8 -> f32 cast, GaussianFilter, round and clamp to u8: the blur_png program on a decoded image
  volume      GaussianFilter on a 3-D f32 volume, in either rounding
  ct          GaussianFilter on an i16 CT-like volume with anisotropic spacing, stored as f32, bf16 or f16
  wide        GaussianFilter on a 3-D f32 volume with a large sigma (radius above 12)
  u8_volume   GaussianFilter<Image<u8, 3>>: the pixel type's own u8 arithmetic
  unsharp     UnsharpMaskFilter on a 3-D f32 volume
  recursive   RecursiveGaussianFilter on a 3-D f32 volume (f64 recursions)
  vjp         gaussian_vjp: the gradient with respect to a volume and to sigma
  scale_loss  multi-scale squared-error loss of one volume with its gradients
  batch       Batch: forward + VJP of many ragged volumes, planned once, replayed
"""
from __future__ import annotations

import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "itk-rs_gb300"))

import itkg  # noqa: E402

ROUNDING = {"reference": itkg.ROUND_REFERENCE, "fma": itkg.ROUND_FMA}
STORAGE = {"f32": itkg.F32, "bf16": itkg.BF16, "f16": itkg.F16, "i16": itkg.I16, "u8": itkg.U8}
TORCH = {itkg.F32: torch.float32, itkg.BF16: torch.bfloat16, itkg.F16: torch.float16, itkg.I16: torch.int16,
         itkg.U8: torch.uint8}
BYTES = {"f32": 4, "bf16": 2, "f16": 2, "i16": 2, "u8": 1}


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # The smallest call: one 512 x 512 image at sigma 1.5, where the call itself counts (a viewer, a tracker).
        {"name": "image_512", "kind": "image", "nx": 512, "ny": 512, "components": 1, "sigma": 1.5, "rounding": "fma"},
        # The blur_png program on a photograph of odd sides, already on the device; the API's default rounding.
        {"name": "photo_1601x1067", "kind": "photo", "nx": 1601, "ny": 1067, "components": 1, "sigma": 3.0,
         "rounding": "reference"},
        # The benchmark's forward: 256^3, sigma 2, fused multiply-adds.
        {"name": "volume_256", "kind": "volume", "nx": 256, "ny": 256, "nz": 256, "sigma": 2.0, "rounding": "fma"},
        # A scan of odd sides in the default (reference) rounding, what a first-time user gets.
        {"name": "volume_reference_odd", "kind": "volume", "nx": 197, "ny": 233, "nz": 189, "sigma": 1.5,
         "rounding": "reference"},
        # The largest single image: CT, i16 in, bf16 out, sigma in millimetres and anisotropic spacing.
        {"name": "ct_512", "kind": "ct", "nx": 512, "ny": 512, "nz": 384, "sigma": 1.5, "sx": 0.7, "sz": 2.5,
         "out": "bf16", "rounding": "fma"},
        # A background / scale-space level: sigma 8 (radius 24) on a mid-size volume.
        {"name": "wide_sigma8", "kind": "wide", "nx": 192, "ny": 192, "nz": 192, "sigma": 8.0, "rounding": "fma"},
        # An 8-bit volume filtered as it is stored.
        {"name": "u8_volume", "kind": "u8_volume", "nx": 250, "ny": 250, "nz": 161, "sigma": 2.0},
        # Sharpening in the default rounding.
        {"name": "unsharp_192", "kind": "unsharp", "nx": 192, "ny": 192, "nz": 192, "sigma": 1.5, "amount": 0.5,
         "threshold": 0.01, "rounding": "reference"},
        # The recursive Gaussian in the default rounding, odd sides.
        {"name": "recursive_odd", "kind": "recursive", "nx": 161, "ny": 193, "nz": 145, "sigma": 4.0,
         "rounding": "reference"},
        # One volume's gradient, as a training step of a single sample takes it.
        {"name": "vjp_odd", "kind": "vjp", "nx": 181, "ny": 217, "nz": 163, "sigma": 2.0},
        # The multi-scale loss with all its gradients: one sample of the benchmark's eight.
        {"name": "scale_loss_192", "kind": "scale_loss", "nx": 192, "ny": 192, "nz": 192, "levels": 4},
        # A training batch of ragged volumes, forward and backward, as one graph.
        {"name": "batch_16", "kind": "batch", "volumes": 16, "shapes": 7, "longest": 320},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _sides(rng, n, lo, hi, most):
    """n sides in lo..hi with at most `most` elements in all."""
    while True:
        s = [_log_int(rng, lo, hi) for _ in range(n)]
        if math.prod(s) <= most:
            return s


def draw(rng: random.Random):
    kind = rng.choice(["image", "photo", "volume", "volume", "ct", "wide", "u8_volume", "unsharp", "recursive", "vjp",
                       "scale_loss", "batch"])
    sigma = round(rng.uniform(0.5, 4.0), 3)
    rounding = rng.choice(["reference", "fma"])
    if kind in ("image", "photo"):
        nx, ny = _sides(rng, 2, 64, 1024 if kind == "image" else 2400, 1 << 22)
        return {"kind": kind, "nx": nx, "ny": ny, "components": rng.choice([1, 3]), "sigma": sigma, "rounding": rounding}
    if kind == "batch":
        return {"kind": kind, "volumes": rng.randint(4, 16), "shapes": rng.randint(100, 1 << 20),
                "longest": rng.randint(96, 256)}
    if kind == "ct":
        nx, ny, nz = _sides(rng, 3, 64, 512, 512 * 512 * 256)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "sigma": round(rng.uniform(0.5, 2.5), 3),
                "sx": round(rng.uniform(0.5, 1.0), 3), "sz": round(rng.uniform(1.0, 3.0), 3),
                "out": rng.choice(["f32", "bf16", "f16"]), "rounding": rounding}
    if kind == "wide":
        nx, ny, nz = _sides(rng, 3, 48, 256, 192**3)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "sigma": round(rng.uniform(4.1, 8.0), 3), "rounding": rounding}
    if kind == "scale_loss":
        nx, ny, nz = _sides(rng, 3, 48, 256, 192**3)
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "levels": rng.randint(1, 4)}
    most = {"volume": 256**3, "u8_volume": 250 * 250 * 161, "unsharp": 192**3, "recursive": 161 * 193 * 145,
            "vjp": 192**3}[kind]
    nx, ny, nz = _sides(rng, 3, 32, 320, most)
    c = {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "sigma": sigma}
    if kind in ("volume", "unsharp", "recursive"):
        c["rounding"] = rounding
    if kind == "unsharp":
        c.update(sigma=round(rng.uniform(0.5, 3.0), 3), amount=round(rng.uniform(0.2, 1.5), 2),
                 threshold=rng.choice([0.0, 0.01, 0.05]))
    if kind == "recursive":
        c["sigma"] = round(rng.uniform(0.6, 8.0), 3)
    return c


def _batch_items(case):
    """(size, sigma) of every volume of a batch case: sides U{32..longest}, sigma U[0.5, 4]."""
    r = random.Random(case["shapes"])
    return [(tuple(r.randint(32, case["longest"]) for _ in range(3)), r.uniform(0.5, 4.0)) for _ in range(case["volumes"])]


def _scales(case):
    return [1.0, 2.0, 4.0, 8.0][:case["levels"]]


def _size(case):
    return tuple(case[k] for k in ("nx", "ny", "nz") if k in case)


def _spacing(case):
    return (case["sx"], case["sx"], case["sz"]) if case["kind"] == "ct" else (1.0,) * len(_size(case))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
class _Memory:
    """A DeviceImage's buffer as the CUDA array interface sees it (the pitched rows included)."""

    CODE = {itkg.F32: "<f4", itkg.I16: "<i2", itkg.U8: "|u1", itkg.BF16: "<i2", itkg.F16: "<f2"}

    def __init__(self, dev):
        self.dev = dev
        D, c = dev.dim, dev.components
        item = int(self.CODE[dev.dtype][2])
        shape = tuple(reversed(dev.region.size)) + ((c,) if c > 1 else ())
        strides = tuple(dev.c.pitch[d] for d in reversed(range(D))) + ((item,) if c > 1 else ())
        self.__cuda_array_interface__ = {"shape": shape, "strides": strides, "typestr": self.CODE[dev.dtype],
                                         "data": (dev.c.data, False), "version": 3}


def _tensor(dev):
    """The image as a tensor of shape ([nz,] ny, nx[, components]) over the same memory."""
    return torch.as_tensor(_Memory(dev), device="cuda").view(TORCH[dev.dtype])


def _device_image(values, dtype=itkg.F32, components=1, spacing=None):
    size = tuple(reversed(values.shape[:-1] if components > 1 else values.shape))
    dev = itkg.DeviceImage(itkg.Region((0,) * len(size), size), dtype, components, spacing)
    _tensor(dev).copy_(values)
    return dev


def _empty_like(dev, dtype=itkg.F32):
    return itkg.DeviceImage(dev.region, dtype, dev.components, dev.spacing)


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _uniform(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float64)


def _blobs(size, g, noise=0.05, blobs=32):
    """A sum of Gaussian blobs (amplitude U[0.5, 2], std U[4, 24] voxels) plus N(0, noise), f32."""
    amp, sd = _uniform(g, 0.5, 2.0, blobs, 1), _uniform(g, 4.0, 24.0, blobs, 1)
    axes = []
    for n in reversed(size):
        centre = _uniform(g, 0.0, float(n), blobs, 1)
        axes.append(torch.exp(-0.5 * ((torch.arange(n, device="cuda") - centre) / sd) ** 2).float())
    axes[0] = axes[0] * amp.float()
    plane = axes[-1] if len(axes) == 1 else (axes[-2][:, :, None] * axes[-1][:, None, :]).reshape(blobs, -1)
    v = axes[0].t() @ plane if len(axes) == 3 else plane.reshape(blobs, size[1], size[0]).mul(amp.float()[..., None]).sum(0)
    v = v.reshape(tuple(reversed(size)))
    return v + noise * torch.randn(v.shape, generator=g, device="cuda")


def _ct(size, g, ellipsoids=12):
    """Air (-1000) with ellipsoids of constant value U[-1000, 1500], plus N(0, 20), as i16."""
    shape = tuple(reversed(size))
    grid = torch.meshgrid(*(torch.arange(n, device="cuda", dtype=torch.float32) for n in shape), indexing="ij")
    v = torch.full(shape, -1000.0, device="cuda")
    par = torch.cat([_uniform(g, 0.2, 0.8, ellipsoids, 3), _uniform(g, 0.05, 0.35, ellipsoids, 3),
                     _uniform(g, -1000.0, 1500.0, ellipsoids, 1)], 1).tolist()
    for c0, c1, c2, a0, a1, a2, value in par:
        d = sum(((x - c * n) / (a * n)) ** 2 for x, c, a, n in zip(grid, (c0, c1, c2), (a0, a1, a2), shape))
        v.masked_fill_(d <= 1, value)
    v += 20.0 * torch.randn(shape, generator=g, device="cuda")
    return v.round().clamp(-32768, 32767).to(torch.int16)


def _photo(case, g):
    """An 8-bit image: smooth shapes and grain, 0..255."""
    v = torch.stack([_blobs(_size(case), g) for _ in range(case["components"])], -1)
    v = (v * 90.0 + 12.0).round().clamp(0, 255).to(torch.uint8)
    return v if case["components"] > 1 else v[..., 0]


def _inputs(case, seed):
    """The case's input tensors, from the seed alone."""
    g, kind = _generator(seed), case["kind"]
    if kind == "batch":
        return [(_blobs(size, g), _blobs(size, g)) for size, _ in _batch_items(case)]
    if kind == "image":
        shape = tuple(reversed(_size(case))) + ((3,) if case["components"] == 3 else ())
        return torch.rand(shape, generator=g, device="cuda")
    if kind == "photo":
        return _photo(case, g)
    if kind == "ct":
        return _ct(_size(case), g)
    if kind == "u8_volume":
        return (_blobs(_size(case), g) * 60.0 + 10.0).round().clamp(0, 255).to(torch.uint8)
    if kind in ("vjp", "scale_loss"):
        return _blobs(_size(case), g), _blobs(_size(case), g)
    return _blobs(_size(case), g)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    """Images on the device, the filter node or plan over them, and the output images a program keeps."""
    kind = case["kind"]
    values = _inputs(case, seed)
    s = {"kind": kind}
    if kind == "batch":
        items = _batch_items(case)
        s["batch"] = itkg.Batch()
        s["sigma_bar"] = torch.zeros(len(items), dtype=torch.float64, device="cuda")
        s["out"] = []
        for i, ((x, target), (_, sigma)) in enumerate(zip(values, items)):
            dx, dy = _device_image(x), _device_image(x - target)
            y = s["batch"].add(dx, sigma)
            xbar = s["batch"].add_vjp(dx, dy, sigma, sigma_bar_dev=s["sigma_bar"].data_ptr() + 8 * i)
            s["out"] += [_tensor(y), _tensor(xbar)]
        s["out"].append(s["sigma_bar"])
        torch.cuda.synchronize()
        s["batch"].plan()
        return s
    if kind == "vjp":
        x, target = values
        s.update(x=_device_image(x), ybar=_device_image(x - target), sigma=case["sigma"])
        s["xbar"] = _empty_like(s["x"])
        s["out"] = _tensor(s["xbar"])
        return s
    if kind == "scale_loss":
        s.update(x=_device_image(values[0]), target=_device_image(values[1]), sigmas=_scales(case))
        s["xbar"] = _empty_like(s["x"])
        s["out"] = _tensor(s["xbar"])
        return s
    dtype = {"photo": itkg.U8, "ct": itkg.I16, "u8_volume": itkg.U8}.get(kind, itkg.F32)
    s["image"] = img = _device_image(values, dtype, case.get("components", 1), _spacing(case))
    s["request"] = img.largest_region()
    rounding = ROUNDING[case.get("rounding", "reference")]
    if kind == "recursive":
        s["filter"] = itkg.RecursiveGaussianFilter(img, case["sigma"], rounding=rounding)
        return s
    out_dtype = {"photo": itkg.U8, "u8_volume": itkg.U8, "ct": STORAGE[case.get("out", "f32")]}.get(kind, itkg.F32)
    s["out_dtype"], s["out_image"] = out_dtype, _empty_like(img, out_dtype)
    s["out"] = _tensor(s["out_image"])
    if kind == "unsharp":
        s["filter"] = itkg.UnsharpMaskFilter(img, case["sigma"], case["amount"], case["threshold"], rounding=rounding)
    else:
        src = itkg.CastFilter(img, itkg.F32) if kind in ("photo", "ct") else img
        s["filter"] = itkg.GaussianFilter(src, case["sigma"], rounding=rounding)
    return s


def run(state):
    kind = state["kind"]
    if kind == "batch":
        state["batch"].run()
        return state["out"]
    if kind == "vjp":
        _, sigma_bar = itkg.vjp(state["x"], state["ybar"], state["sigma"], xbar=state["xbar"])
        return {"xbar": state["out"], "sigma_bar": sigma_bar}
    if kind == "scale_loss":
        loss, _, sigma_bar = itkg.scale_stack_loss_vjp(state["x"], state["target"], state["sigmas"], xbar=state["xbar"])
        return {"loss": loss, "xbar": state["out"], "sigma_bar": sigma_bar}
    if kind == "recursive":
        return _tensor(state["filter"].generate_region(state["request"]))
    state["filter"].generate_region(state["request"], out_dtype=state["out_dtype"], out=state["out_image"])
    return state["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _radii(sigma, spacing):
    return [math.ceil(3.0 * sigma / s) for s in spacing]


def _taps(case, sigma=None):
    """Kernel taps per element, all axes of the separable filter added."""
    sp = _spacing(case) if "nx" in case else (1.0,) * 3
    return sum(2 * r + 1 for r in _radii(case["sigma"] if sigma is None else sigma, sp))


def work(case):
    kind = case["kind"]
    if kind == "batch":
        n = [(math.prod(size), _taps(case, sigma)) for size, sigma in _batch_items(case)]
        # forward: x in, y out; VJP: x and ybar in, xbar out; the VJP's passes are the adjoint's and their derivatives'
        return {"bytes": 20.0 * sum(v for v, _ in n), "flops": sum(v * t * (2.0 + 16.0 / 3.0) for v, t in n)}
    n = math.prod(_size(case)) * case.get("components", 1)
    if kind == "scale_loss":
        return {"bytes": 12.0 * n, "flops": sum(n * _taps(case, s) * (2.0 + 16.0 / 3.0) for s in _scales(case))}
    if kind == "vjp":
        return {"bytes": 12.0 * n, "flops": n * _taps(case) * 16.0 / 3.0}
    if kind == "recursive":
        return {"bytes": 8.0 * n, "flops": 42.0 * n}  # 4 products and 3 sums, forwards and backwards, on 3 axes
    item = {"photo": 1 + 1, "u8_volume": 1 + 1, "ct": 2 + BYTES[case.get("out", "f32")]}.get(kind, 4 + 4)
    return {"bytes": float(item * n), "flops": 2.0 * n * _taps(case)}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
def _kernel64(sigma, r):
    """The normalised weights of radius r at sigma pixels, and their derivative with respect to sigma."""
    t = np.arange(-r, r + 1, dtype=np.float64)
    e = np.exp(-0.5 * (t / sigma) ** 2)
    w = e / e.sum()
    de = e * t * t / sigma**3
    return w, (de - w * de.sum()) / e.sum()


def _along(v, axis, w):
    """Clamped convolution of v with w along a dimension, taps as shifted slices."""
    r, n = (len(w) - 1) // 2, v.shape[axis]
    at = torch.arange(-r, n + r, device=v.device).clamp_(0, n - 1)
    p = v.index_select(axis, at)
    out = torch.zeros_like(v)
    for k, c in enumerate(w.tolist()):
        out.add_(p.narrow(axis, k, n), alpha=c)
    return out


def _along_t(v, axis, w):
    """The adjoint of _along."""
    r, n = (len(w) - 1) // 2, v.shape[axis]
    shape = list(v.shape)
    shape[axis] += 2 * r
    p = torch.zeros(shape, dtype=v.dtype, device=v.device)
    for k, c in enumerate(w.tolist()):
        p.narrow(axis, k, n).add_(v, alpha=c)
    at = torch.arange(-r, n + r, device=v.device).clamp_(0, n - 1)
    return torch.zeros_like(v).index_add_(axis, at, p)


def _gauss64(v, kernels):
    """kernels: per reference axis; dimension D - 1 - axis of the tensor."""
    for a, (w, _) in enumerate(kernels):
        v = _along(v, len(kernels) - 1 - a, w)
    return v


def _vjp64(x, ybar, kernels):
    """G^T ybar and <ybar, dG/dsigma x> (one sigma for all axes, spacing 1)."""
    last = len(kernels) - 1
    xbar = ybar
    for a in reversed(range(len(kernels))):
        xbar = _along_t(xbar, last - a, kernels[a][0])
    y, dy = x, torch.zeros_like(x)
    for a, (w, d) in enumerate(kernels):
        y, dy = _along(y, last - a, w), _along(dy, last - a, w) + _along(y, last - a, d)
    return xbar, float((ybar * dy).sum())


def _kernels64(sigma, spacing):
    return [_kernel64(sigma / s, r) for s, r in zip(spacing, _radii(sigma, spacing))]


def _recursive64(v, sigma):
    """Young and van Vliet's recursive Gaussian (Signal Processing 44, 1995), each line forwards and backwards from
    the steady state of its first sample."""
    q = 0.98711 * sigma - 0.96330 if sigma >= 2.5 else 3.97156 - 4.14554 * math.sqrt(1 - 0.26891 * sigma)
    b0 = 1.57825 + 2.44413 * q + 1.4281 * q**2 + 0.422205 * q**3
    a = ((2.44413 * q + 2.85619 * q**2 + 1.26661 * q**3) / b0, -(1.4281 * q**2 + 1.26661 * q**3) / b0, 0.422205 * q**3 / b0)
    B = 1 - sum(a)
    for axis in reversed(range(v.dim())):
        v = v.movedim(axis, 0).contiguous()
        for order in (range(v.shape[0]), range(v.shape[0] - 1, -1, -1)):
            y1 = y2 = y3 = v[order[0]].clone()
            for i in order:
                y1, y2, y3 = B * v[i] + a[0] * y1 + a[1] * y2 + a[2] * y3, y1, y2
                v[i] = y1
        v = v.movedim(0, axis)
    return v


def exact(case, seed):
    kind = case["kind"]
    values = _inputs(case, seed)
    if kind in ("photo", "u8_volume"):
        return None  # bytes
    if kind == "batch":
        outs, bars = [], []
        for (x, target), (size, sigma) in zip(values, _batch_items(case)):
            k = _kernels64(sigma, (1.0,) * 3)
            xbar, bar = _vjp64(x.double(), (x - target).double(), k)
            outs += [_gauss64(x.double(), k), xbar]
            bars.append(bar)
        return outs + [torch.tensor(bars, dtype=torch.float64)]
    if kind == "vjp":
        x, target = values
        xbar, bar = _vjp64(x.double(), (x - target).double(), _kernels64(case["sigma"], _spacing(case)))
        return {"xbar": xbar, "sigma_bar": bar}
    if kind == "scale_loss":
        x, target = values[0].double(), values[1].double()
        loss, total, bars = 0.0, torch.zeros_like(x), []
        for s in _scales(case):
            k = _kernels64(s, _spacing(case))
            d = _gauss64(x, k) - target
            loss += float((d * d).sum())
            xbar, bar = _vjp64(x, 2 * d, k)
            total += xbar
            bars.append(bar)
        return {"loss": loss, "xbar": total, "sigma_bar": bars}
    x = values.double()
    if kind == "recursive":
        return _recursive64(x, case["sigma"])
    if kind == "image" and case["components"] == 3:
        return torch.stack([_gauss64(x[..., c], _kernels64(case["sigma"], (1.0, 1.0))) for c in range(3)], -1)
    y = _gauss64(x, _kernels64(case["sigma"], _spacing(case)))
    if kind == "unsharp":
        d = x - y
        return torch.where(d.abs() > case["threshold"], x + case["amount"] * d, x)
    return y
