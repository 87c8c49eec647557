"""The measured cases of this framework: what its users have it do, at the sizes they do it.

`listed()` names the cases, `draw(rng)` gives more of the same ranges, `prepare(case, seed)`
makes a user's inputs and plans on the GPU, `run(state)` is one pass through the public entry
points, `work(case)` the bytes and operations the pass cannot do without, and
`exact(case, seed)` the same outputs in 64 bits by plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import iane_gb300 as g
from iane_gb300 import abi, learned
from iane_gb300._lib import check, lib

DEV = "cuda"
EPS = 1e-6
LAYERS = {name: (ci, co, relu) for name, ci, co, relu in learned.LAYERS}
SKIPS = {"d2a": (64, 32), "d1a": (32, 16)}  # layers that read an upsampled and a skip tensor


def listed():
    return [
        # one small image filtered on its own, as in an interactive tool: latency and launches
        # (the reference's 2-D configuration: 512 x 512, normalised 7 x 7 Gaussian, mirror)
        {"name": "conv2d_f32_512", "op": "conv", "shape": "512x512", "kernel": "7x7", "src": "f32", "taps": "f32",
         "dst": "f32", "border": "mirror", "pad": 0},
        # a camera frame: the reference's own convolution benchmark
        {"name": "conv2d_u8_frame", "op": "conv", "shape": "1920x2560", "kernel": "9x9", "src": "u8", "taps": "f32",
         "dst": "u8", "border": "clamp", "pad": 0},
        # a ragged volume under a dense 3-D kernel (rows no multiple of 16 bytes)
        {"name": "conv3d_f32_ragged", "op": "conv", "shape": "61x187x253", "kernel": "5x7x7", "src": "f32",
         "taps": "f32", "dst": "f32", "border": "clamp", "pad": 0},
        # smoothing of a large volume: the separable benchmark
        {"name": "separable_512", "op": "separable", "shape": "512x512x512", "kernel": "7x7x7", "border": "mirror"},
        # clean-up of a camera frame before segmentation
        {"name": "opening_u8_frame", "op": "morphology", "shape": "1920x2560", "radius": "2x2", "dtype": "u8",
         "kind": "opening", "border": "zero"},
        # erosion of a volume with the 5 x 5 x 5 box
        {"name": "erode_f32_volume", "op": "morphology", "shape": "256x384x384", "radius": "2x2x2", "dtype": "f32",
         "kind": "erode", "border": "zero"},
        # one prepared Wiener restoration of a camera frame (the reference's example)
        {"name": "wiener_u8_frame", "op": "wiener", "shape": "1920x2560", "kernel": "9x9", "src": "u8", "dst": "u8"},
        # Richardson-Lucy of a microscopy volume, 50 iterations: the framework's headline
        {"name": "rl3d_f32", "op": "rl", "shape": "64x256x256", "kernel": "7x15x15", "sigma": "1x2x2",
         "iterations": 50, "precision": "f32"},
        # the same on the tensor cores
        {"name": "rl3d_bf16", "op": "rl", "shape": "64x256x256", "kernel": "9x9x9", "sigma": "2.5x2.5x2.5",
         "iterations": 50, "precision": "bf16"},
        # a night's worth of uneven 2-D exposures, each with its own PSF, in one launch
        {"name": "rl_batch_256", "op": "rl_batch", "count": 256, "side_lo": 64, "side_hi": 1024, "iterations": 30,
         "pick": 0},
        # one layer of a training step of the warm-start network: the decoder's widest, on the
        # 64^3 training volumes -- forward, input gradient and weight gradient
        {"name": "cnn_train_layer", "op": "cnn_layer", "layer": "d1a", "shape": "64x64x64"},
        # the warm start of a whole volume: the network's inference
        {"name": "cnn_infer_volume", "op": "cnn_infer", "shape": "64x256x256", "sigma": 2.0},
    ]


# ---------------------------------------------------------------------------------------------
# more cases of the same ranges


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, lo, hi):
    return 2 * rng.randint(lo // 2, hi // 2) + 1


def _dims(values):
    return "x".join(str(v) for v in values)


def draw(rng):
    op = rng.choice(["conv", "conv", "separable", "morphology", "morphology", "wiener", "rl", "rl", "rl_batch",
                     "cnn_layer", "cnn_layer", "cnn_infer"])
    border = rng.choice(["clamp", "zero", "mirror"])
    if op == "conv":
        if rng.random() < 0.6:
            shape, kernel = [_log(rng, 96, 4096), _log(rng, 96, 4096)], [_odd(rng, 3, 15)] * 2
            src = rng.choice(["u8", "u8", "u16", "i16", "f32", "f32", "f32"])
        else:
            shape = [_log(rng, 16, 128), _log(rng, 48, 384), _log(rng, 48, 384)]
            kernel = [_odd(rng, 3, 9) for _ in range(3)]
            src = rng.choice(["u16", "f32", "f32", "f32"])
        dst = src if rng.random() < 0.7 else "f32"
        # whole-number kernels (difference operators) on whole-number images give whole numbers
        taps = "i32" if src != "f32" and rng.random() < 0.3 else "f32"
        return {"op": op, "shape": _dims(shape), "kernel": _dims(kernel), "src": src, "taps": taps,
                "dst": "i32" if taps == "i32" else dst, "border": border, "pad": rng.choice([0, 0, 0, 3, 16])}
    if op == "separable":
        if rng.random() < 0.5:
            shape = [_log(rng, 128, 4096), _log(rng, 128, 4096)]
        else:
            shape = [_log(rng, 24, 400), _log(rng, 64, 512), _log(rng, 64, 512)]
        k = _odd(rng, 3, 15)
        return {"op": op, "shape": _dims(shape), "kernel": _dims([k] * len(shape)), "border": border}
    if op == "morphology":
        if rng.random() < 0.5:
            shape = [_log(rng, 128, 4096), _log(rng, 128, 4096)]
        else:
            shape = [_log(rng, 16, 300), _log(rng, 64, 400), _log(rng, 64, 400)]
        r = rng.randint(1, 3)
        radius = [r] * len(shape) if rng.random() < 0.7 else [rng.randint(1, 4) for _ in shape]
        return {"op": op, "shape": _dims(shape), "radius": _dims(radius), "border": border,
                "dtype": rng.choice(["u8", "u8", "u16", "i16", "f32", "f32"]),
                "kind": rng.choice(["erode", "dilate", "opening", "closing"])}
    if op == "wiener":
        return {"op": op, "shape": _dims([_log(rng, 128, 2600), _log(rng, 128, 2600)]),
                "kernel": _dims([_odd(rng, 3, 15)] * 2), "src": rng.choice(["u8", "u8", "f32"]),
                "dst": rng.choice(["u8", "f32"])}
    if op == "rl":
        shape = [_log(rng, 16, 64), _log(rng, 64, 256), _log(rng, 64, 256)]
        if rng.random() < 0.5:
            k, s = [_odd(rng, 5, 7), *[_odd(rng, 7, 15)] * 2], [1.0, 2.0, 2.0]
            precision = "f32"
        else:
            k = [_odd(rng, 5, 11)] * 3
            s = [round(rng.uniform(1.0, 2.5), 2)] * 3
            precision = "bf16"
        return {"op": op, "shape": _dims(shape), "kernel": _dims(k), "sigma": _dims(s),
                "iterations": rng.randint(8, 40), "precision": precision}
    if op == "rl_batch":
        return {"op": op, "count": _log(rng, 8, 128), "side_lo": 64, "side_hi": rng.choice([256, 512, 1024]),
                "iterations": rng.randint(5, 30), "pick": rng.randint(1, 1 << 20)}
    if op == "cnn_layer":
        edges = [4 * _log(rng, 6, 20) for _ in range(3)]
        return {"op": op, "layer": rng.choice([n for n in LAYERS if n not in ("e1a", "head")]), "shape": _dims(edges)}
    return {"op": op, "shape": _dims([4 * _log(rng, 4, 16), 4 * _log(rng, 12, 64), 4 * _log(rng, 12, 64)]),
            "sigma": round(rng.uniform(1.0, 3.0), 2)}


# ---------------------------------------------------------------------------------------------
# inputs

_DTYPES = {"u8": torch.uint8, "u16": torch.uint16, "i16": torch.int16, "i32": torch.int32, "f32": torch.float32}
_SIZES = {"u8": 1, "u16": 2, "i16": 2, "i32": 4, "f32": 4}


def _nums(text, kind=int):
    return tuple(kind(v) for v in text.split("x"))


def _gen(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    return gen


def _image(shape, dtype, seed, pad=0):
    """Uniform samples: [0, 1) for f32, the whole range for bytes, 12 bits for 16-bit sensors
    (signed: around zero). `pad` elements follow each row (a crop of a wider frame)."""
    full = (*shape[:-1], shape[-1] + pad)
    gen = _gen(seed)
    if dtype == "f32":
        t = torch.rand(full, generator=gen, device=DEV)
    else:
        lo, hi = {"u8": (0, 256), "u16": (0, 4096), "i16": (-2048, 2048)}[dtype]
        t = torch.randint(lo, hi, full, generator=gen, device=DEV, dtype=torch.int32)
        t = t.to(torch.int16).view(torch.uint16) if dtype == "u16" else t.to(_DTYPES[dtype])
    return t[..., :shape[-1]]


def _gaussian(shape, sigma):
    grids = np.meshgrid(*[np.arange(n, dtype=np.float64) - n // 2 for n in shape], indexing="ij")
    k = np.exp(-0.5 * sum((x / s) ** 2 for x, s in zip(grids, sigma)))
    return torch.from_numpy((k / k.sum()).astype(np.float32)).to(DEV)


def _kernel(case, seed):
    shape = _nums(case["kernel"])
    if case.get("taps") == "i32":
        return torch.randint(-8, 9, shape, generator=_gen(seed + 7919), device=DEV, dtype=torch.int32)
    return _gaussian(shape, [max(0.5, n / 4.67) for n in shape])


def _blur(vol, psf, pad_to=1):
    """Zero-border convolution by FFT in 64 bits."""
    size = [-(-(n + k - 1) // pad_to) * pad_to for n, k in zip(vol.shape, psf.shape)]
    f = torch.fft.rfftn(vol.double(), s=size) * torch.fft.rfftn(psf.double(), s=size)
    out = torch.fft.irfftn(f, s=size)
    return out[tuple(slice(k // 2, k // 2 + n) for n, k in zip(vol.shape, psf.shape))]


def _volume(shape, psf, seed):
    """Poisson counts of a blurred phantom: ellipsoids of radii 2-20 and intensities 50-1000 on
    a background of 10, 200 of them per 256 x 256 x 64 voxels."""
    rng = np.random.default_rng(seed)
    vol = torch.full(shape, 10.0, dtype=torch.float32, device=DEV)
    axes = [torch.arange(n, dtype=torch.float32, device=DEV) for n in shape]
    for _ in range(max(4, int(200 * math.prod(shape) / (256 * 256 * 64)))):
        centre, radii = [rng.uniform(0, n) for n in shape], [rng.uniform(2.0, 20.0) for _ in shape]
        value = rng.uniform(50.0, 1000.0)
        box = tuple(slice(max(0, int(c - r)), min(n, int(c + r) + 2)) for c, r, n in zip(centre, radii, shape))
        d = [((a[b] - c) / r) ** 2 for a, b, c, r in zip(axes, box, centre, radii)]
        vol[box] += value * (d[0][:, None, None] + d[1][None, :, None] + d[2][None, None, :] <= 1.0)
    return torch.poisson(_blur(vol, psf).clamp_min(0.0).float(), generator=_gen(seed + 1))


def _batch(case, seed):
    """Sparse point sources on a smooth background, blurred by each image's own PSF, with
    Poisson noise. The sizes and PSFs are the case's; the seed makes the images."""
    shapes = np.random.default_rng(case["pick"])
    lo, hi = math.log(case["side_lo"]), math.log(case["side_hi"])
    rng, gen = np.random.default_rng(seed), _gen(seed)
    images, psfs = [], []
    for _ in range(case["count"]):
        ny, nx = (int(round(math.exp(shapes.uniform(lo, hi)))) for _ in range(2))
        k, sigma = int(shapes.integers(1, 16)) * 2 + 1, float(shapes.uniform(0.5, 5.0))
        y = torch.arange(ny, dtype=torch.float32, device=DEV)[:, None]
        x = torch.arange(nx, dtype=torch.float32, device=DEV)[None, :]
        s = float(rng.uniform(0.2, 0.6)) * max(nx, ny)
        img = float(rng.uniform(5, 40)) * torch.exp(
            -((x - float(rng.uniform(0, nx))) ** 2 + (y - float(rng.uniform(0, ny))) ** 2) / (2 * s * s)) + 5.0
        points = torch.rand((ny, nx), generator=gen, device=DEV)
        img = torch.where(points < 0.002, img + 200.0 + points * 2.4e6, img)
        psf = _gaussian((k, k), (sigma, sigma))
        images.append(torch.poisson(_blur(img, psf, 128).clamp_min(0.0).float(), generator=gen))
        psfs.append(psf)
    return images, psfs


def _packed(images):
    """One buffer with a place for each image (64-element aligned), and those places."""
    at, places = 0, []
    for i in images:
        places.append(at)
        at += -(-i.numel() // 64) * 64
    flat = torch.zeros(at, dtype=images[0].dtype, device=DEV)
    return flat, [flat[p:p + i.numel()].view(i.shape) for p, i in zip(places, images)]


def _layer(case):
    """(name, inputs of the two tensors, outputs, relu, volume) of a layer at its own level."""
    name = case["layer"]
    ci, co, relu = LAYERS[name]
    c0, c1 = SKIPS.get(name, (ci, 0))
    step = {"e1": 1, "d1": 1, "he": 1, "e2": 2, "d2": 2, "e3": 4}[name[:2]]
    return name, c0, c1, co, relu, tuple(n // step for n in _nums(case["shape"]))


def _activation(c, shape, gen):
    """A ReLU activation in the network's layout (octets, D, H, W, 8): about half of it zero."""
    x = torch.randn((c // 8, *shape, 8), generator=gen, device=DEV)
    return x.clamp_min(0.0).to(torch.bfloat16)


def _layer_inputs(case, seed):
    name, c0, c1, co, relu, shape = _layer(case)
    gen = _gen(seed)
    ci = c0 + c1
    x0 = _activation(c0, shape, gen)
    x1 = _activation(c1, shape, gen) if c1 else None
    w = (torch.randn((co, ci, 27), generator=gen, device=DEV) * math.sqrt(2.0 / (27 * ci))).to(torch.bfloat16)
    bias = torch.randn(co, generator=gen, device=DEV) * 0.1
    dy = torch.randn((co // 8, *shape, 8), generator=gen, device=DEV) * 1e-3
    dy = (dy * (torch.rand(dy.shape, generator=gen, device=DEV) < 0.5)).to(torch.bfloat16)  # behind the ReLU
    return x0, x1, w, bias, dy


def prepare(case, seed):
    op = case["op"]
    st = {"case": case, "op": op}
    if op == "conv":
        shape = _nums(case["shape"])
        st["src"] = _image(shape, case["src"], seed, case["pad"])
        st["kernel"] = _kernel(case, seed)
        st["dst"] = torch.empty(shape, dtype=_DTYPES[case["dst"]], device=DEV)
    elif op == "separable":
        shape, k = _nums(case["shape"]), _nums(case["kernel"])
        st["src"] = _image(shape, "f32", seed)
        st["taps"] = [_gaussian((n,), (n / 4.67,)) for n in reversed(k)]
        st["dst"] = torch.empty_like(st["src"])
    elif op == "morphology":
        st["src"] = _image(_nums(case["shape"]), case["dtype"], seed)
        st["dst"] = torch.empty_like(st["src"])
        st["radius"] = _nums(case["radius"])
        if case["kind"] in ("opening", "closing"):  # a program that repeats it keeps its scratch
            image = -(-st["src"].numel() * _SIZES[case["dtype"]] // 256) * 256
            st["scratch"] = torch.empty(2 * image, dtype=torch.uint8, device=DEV)
    elif op == "wiener":
        shape = _nums(case["shape"])
        st["src"] = _image(shape, case["src"], seed)
        st["plan"] = g.Wiener(_kernel(case, seed), shape, 0.002)
        st["dst"] = torch.empty(shape, dtype=_DTYPES[case["dst"]], device=DEV)
        st["scratch"] = torch.empty(st["plan"].scratch_bytes, dtype=torch.uint8, device=DEV)
    elif op == "rl":
        shape = _nums(case["shape"])
        psf = _gaussian(_nums(case["kernel"]), _nums(case["sigma"], float))
        st["observed"] = _volume(shape, psf, seed)
        st["plan"] = g.RichardsonLucy(psf, shape, precision=case["precision"])
        st["estimate"] = torch.empty_like(st["observed"])
        st["scratch"] = torch.empty(st["plan"].scratch_bytes, dtype=torch.uint8, device=DEV)
    elif op == "rl_batch":
        st["observed"], psfs = _batch(case, seed)
        st["plan"] = g.RichardsonLucyBatch(psfs, [tuple(i.shape) for i in st["observed"]])
        st["all"], st["estimates"] = _packed(st["observed"])
        st["scratch"] = torch.empty(st["plan"].scratch_bytes, dtype=torch.uint8, device=DEV)
    elif op == "cnn_layer":
        name, c0, c1, co, relu, shape = _layer(case)
        x0, x1, w, bias, dy = _layer_inputs(case, seed)
        ci = c0 + c1
        vol = math.prod(shape)
        st.update(x0=x0, x1=x1, w=w, bias=bias, dy=dy, y=torch.zeros_like(dy), flipped=torch.empty_like(w),
                  dx=torch.zeros((ci // 8, *shape, 8), dtype=torch.bfloat16, device=DEV),
                  dw=torch.zeros(w.shape, dtype=torch.float32, device=DEV),
                  db=torch.zeros(co, dtype=torch.float32, device=DEV), vol=vol)
        need = lib().iane_gb_cnn_wgrad_scratch_bytes(c0, c1, *shape, co)
        st["scratch"] = torch.empty(int(need), dtype=torch.uint8, device=DEV)
    elif op == "cnn_infer":
        shape = _nums(case["shape"])
        sigma = float(case["sigma"])
        psf = _gaussian((learned.psf_extent(sigma),) * 3, (sigma,) * 3)
        observed = _volume(shape, psf, seed)
        st["observed"] = observed / observed.mean()
        st["net"] = learned.load_default(DEV)
    return st


# ---------------------------------------------------------------------------------------------
# one pass


def _p(t):
    return None if t is None else t.data_ptr()


def run(st):
    case, op = st["case"], st["op"]
    if op == "conv":
        return g.convolve(st["src"], st["kernel"], st["dst"], case["border"])
    if op == "separable":
        return g.convolve_separable(st["src"], st["taps"], st["dst"], case["border"])
    if op == "morphology":
        return g.morphology(st["src"], st["dst"], st["radius"], case["kind"], case["border"],
                            scratch=st.get("scratch"))
    if op == "wiener":
        return st["plan"].run(st["src"], st["dst"], scratch=st["scratch"])
    if op == "rl":
        return st["plan"].run(st["observed"], st["estimate"], case["iterations"], EPS, init=abi.RL_INIT_MEAN,
                              scratch=st["scratch"])
    if op == "rl_batch":
        st["plan"].run(st["observed"], st["estimates"], case["iterations"], EPS, init=abi.RL_INIT_MEAN,
                       scratch=st["scratch"])
        return st["all"]
    if op == "cnn_layer":
        # what a training step does for the layer, through the C ABI
        name, c0, c1, co, relu, s = _layer(case)
        ci = c0 + c1
        stream = torch.cuda.current_stream().cuda_stream
        x0, x1, w, dy, dx, wt = (st[k] for k in ("x0", "x1", "w", "dy", "dx", "flipped"))
        check(lib().iane_gb_cnn_conv3(_p(x0), c0, _p(x1), c1, *s, _p(w), _p(st["bias"]), co, _p(st["y"]), None, None,
                                      1 if relu else 0, None, stream))
        st["dw"].zero_()
        st["db"].zero_()
        check(lib().iane_gb_cnn_conv3_wgrad(_p(x0), c0, _p(x1), c1, *s, _p(dy), co, _p(st["dw"]), _p(st["db"]),
                                            _p(st["scratch"]), st["scratch"].numel(), stream))
        check(lib().iane_gb_cnn_flip(_p(w), co, ci, _p(wt), stream))
        # the ReLU of the layer below is part of the input gradient where the input is its output
        mask = x0 if c1 == 0 else None
        for at, n in ([(0, ci)] if ci <= 64 else [(0, c0), (c0, c1)]):  # up to 64 channels a call
            check(lib().iane_gb_cnn_conv3(_p(dy), co, None, 0, *s, wt.data_ptr() + 2 * at * co * 27, None, n,
                                          dx.data_ptr() + 2 * at * st["vol"], None, None, 0, _p(mask), stream))
        return {"y": st["y"], "dx": dx, "dw": st["dw"], "db": st["db"]}
    return st["net"].forward(st["observed"], case["sigma"], tensor_cores=True)


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without


def work(case):
    op = case["op"]
    if op == "rl_batch":
        shapes = np.random.default_rng(case["pick"])
        lo, hi = math.log(case["side_lo"]), math.log(case["side_hi"])
        nbytes = flops = 0
        for _ in range(case["count"]):
            ny, nx = (int(round(math.exp(shapes.uniform(lo, hi)))) for _ in range(2))
            k, _s = int(shapes.integers(1, 16)) * 2 + 1, shapes.uniform(0.5, 5.0)
            nbytes += 8 * nx * ny
            flops += 2 * case["iterations"] * 2 * nx * ny * k * k
        return {"bytes": nbytes, "flops": flops}
    n = math.prod(_nums(case["shape"]))
    if op == "conv":
        return {"bytes": n * (_SIZES[case["src"]] + _SIZES[case["dst"]]), "flops": 2 * n * math.prod(_nums(case["kernel"]))}
    if op == "separable":
        return {"bytes": 8 * n, "flops": 2 * n * sum(_nums(case["kernel"]))}
    if op == "morphology":
        passes = 2 if case["kind"] in ("opening", "closing") else 1
        return {"bytes": 2 * n * _SIZES[case["dtype"]], "flops": passes * n * sum(2 * r for r in _nums(case["radius"]))}
    if op == "wiener":
        # two real transforms of 2.5 n log2 n and the spectral product; the filter is read once
        return {"bytes": n * (_SIZES[case["src"]] + _SIZES[case["dst"]]) + 4 * n, "flops": int(5 * n * math.log2(n) + 3 * n)}
    if op == "rl":
        return {"bytes": 8 * n, "flops": 2 * case["iterations"] * 2 * n * math.prod(_nums(case["kernel"]))}
    if op == "cnn_layer":
        name, c0, c1, co, relu, s = _layer(case)
        v, ci = math.prod(s), c0 + c1
        # read x and dy, write y and dx; the weights and their gradient
        return {"bytes": v * 2 * (2 * ci + 2 * co) + 27 * ci * co * (2 + 4), "flops": 3 * 2 * 27 * ci * co * v}
    flops = sum(2 * 27 * ci * co / {"1": 1, "2": 8, "3": 64}.get(name[1], 1) for name, (ci, co, _) in LAYERS.items())
    return {"bytes": 8 * n, "flops": int(n * flops)}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits


def _indices(n, r, border):
    """Source index of the positions -r .. n + r - 1 (-1: the zero sample)."""
    i = torch.arange(-r, n + r, device=DEV)
    if border == "clamp":
        return i.clamp(0, n - 1)
    if border == "mirror":
        m = i % (2 * n)
        return torch.where(m < n, m, 2 * n - 1 - m)
    return torch.where((i >= 0) & (i < n), i, torch.full_like(i, -1))


def _padded(x, radii, border):
    for axis, r in enumerate(radii):
        idx = _indices(x.shape[axis], r, border)
        y = x.index_select(axis, idx.clamp_min(0))
        if border == "zero":
            view = [1] * x.dim()
            view[axis] = -1
            y = y * (idx >= 0).view(view)
        x = y
    return x


def _convolve64(src, kernel, border):
    radii = [k // 2 for k in kernel.shape]
    p = _padded(src.double(), radii, border)
    out = torch.zeros(src.shape, dtype=torch.float64, device=DEV)
    taps = kernel.double().cpu().numpy()
    for q in np.ndindex(*kernel.shape):
        at = tuple(slice(k - 1 - i, k - 1 - i + n) for i, k, n in zip(q, kernel.shape, src.shape))
        out.add_(p[at], alpha=float(taps[q]))
    return out


def _rl64(observed, psf, iterations, pad_to=1):
    """The Richardson-Lucy loop from the flat start: guarded ratio, adjoint, edge correction."""
    obs = observed.double()
    size = [-(-(n + k - 1) // pad_to) * pad_to for n, k in zip(obs.shape, psf.shape)]
    crop = tuple(slice(k // 2, k // 2 + n) for n, k in zip(obs.shape, psf.shape))
    forward = torch.fft.rfftn(psf.double(), s=size)
    adjoint = torch.fft.rfftn(psf.double().flip(list(range(psf.dim()))), s=size)

    def conv(x, spec):
        return torch.fft.irfftn(torch.fft.rfftn(x, s=size) * spec, s=size)[crop]

    sens = conv(torch.ones_like(obs), adjoint).clamp_min(EPS)
    est = torch.full_like(obs, max(float(obs.mean()), EPS))
    for _ in range(iterations):
        ratio = obs / conv(est, forward).clamp_min(EPS)
        est = est * conv(ratio, adjoint) / sens
    return est


def _planar(x, c):
    """(octets, D, H, W, 8) -> (C, D, H, W) in 64 bits."""
    return x.double().permute(0, 4, 1, 2, 3).reshape(-1, *x.shape[1:4])[:c]


def _octets(x):
    return x.reshape(x.shape[0] // 8, 8, *x.shape[1:]).permute(0, 2, 3, 4, 1).contiguous()


def _taps3(x):
    """The 27 shifted copies of a zero-padded (C, D, H, W) volume, as (C, V) matrices."""
    d, h, w = x.shape[1:]
    p = torch.nn.functional.pad(x, (1, 1, 1, 1, 1, 1))
    for t in range(27):
        tx, ty, tz = t % 3, t // 3 % 3, t // 9
        yield t, p[:, tz:tz + d, ty:ty + h, tx:tx + w].reshape(x.shape[0], -1)


def _conv3_64(x, w, bias=None):
    out = torch.zeros((w.shape[0], math.prod(x.shape[1:])), dtype=torch.float64, device=DEV)
    if bias is not None:
        out += bias.double()[:, None]
    for t, m in _taps3(x):
        out += w[:, :, t].double() @ m
    return out.view(w.shape[0], *x.shape[1:])


def exact(case, seed):
    op = case["op"]
    if op in ("morphology", "conv", "wiener") and case.get("dst", case.get("dtype")) != "f32":
        return None  # whole numbers
    if op == "morphology":
        return None  # selects among its inputs: the same bits, or wrong
    if op == "conv":
        src = _image(_nums(case["shape"]), case["src"], seed, case["pad"])
        return _convolve64(src.to(torch.int32) if case["src"] == "u16" else src, _kernel(case, seed), case["border"])
    if op == "separable":
        x, rank = _image(_nums(case["shape"]), "f32", seed).double(), len(_nums(case["shape"]))
        for axis, n in enumerate(_nums(case["kernel"])):
            x = _convolve64(x, _gaussian((n,), (n / 4.67,)).view([-1 if a == axis else 1 for a in range(rank)]),
                            case["border"])
        return x
    if op == "wiener":
        shape, psf = _nums(case["shape"]), _kernel(case, seed).double()
        padded = torch.zeros(shape, dtype=torch.float64, device=DEV)
        padded[:psf.shape[0], :psf.shape[1]] = psf
        padded = padded.roll([-(k // 2) for k in psf.shape], (0, 1))
        h = torch.fft.rfft2(padded)
        spec = torch.fft.rfft2(_image(shape, case["src"], seed).double()) * h.conj() / (h.abs() ** 2 + 0.002)
        return torch.fft.irfft2(spec, s=shape)
    if op == "rl":
        psf = _gaussian(_nums(case["kernel"]), _nums(case["sigma"], float))
        return _rl64(_volume(_nums(case["shape"]), psf, seed), psf, case["iterations"])
    if op == "rl_batch":
        images, psfs = _batch(case, seed)
        flat, views = _packed([o.double() for o in images])
        for o, k, v in zip(images, psfs, views):
            v.copy_(_rl64(o, k, case["iterations"], 128))
        return flat
    if op == "cnn_layer":
        name, c0, c1, co, relu, s = _layer(case)
        x0, x1, w, bias, dy = _layer_inputs(case, seed)
        x = _planar(x0, c0) if x1 is None else torch.cat([_planar(x0, c0), _planar(x1, c1)])
        gy = _planar(dy, co)
        y = _conv3_64(x, w, bias)
        y = y.clamp_min(0.0) if relu else y
        dx = _conv3_64(gy, w.transpose(0, 1).flip(2).contiguous())
        dx = torch.where(x > 0, dx, torch.zeros_like(dx)) if c1 == 0 else dx
        dw = torch.empty((co, c0 + c1, 27), dtype=torch.float64, device=DEV)
        for t, m in _taps3(x):
            dw[:, :, t] = gy.view(co, -1) @ m.T
        return {"y": _octets(y), "dx": _octets(dx), "dw": dw, "db": gy.reshape(co, -1).sum(1)}
    st = prepare(case, seed)
    net, x = st["net"], st["observed"].double()

    def layer(name, v):
        ci, co, relu = LAYERS[name]
        out = _conv3_64(v, net.w16(name).view(co, ci, 27), net.bias(name))
        return out.clamp_min(0.0) if relu else out

    def pool(v):
        return torch.nn.functional.avg_pool3d(v[None], 2)[0]

    def up(v):
        return v.repeat_interleave(2, 1).repeat_interleave(2, 2).repeat_interleave(2, 3)

    e1 = layer("e1b", layer("e1a", torch.stack([x, torch.full_like(x, case["sigma"] / 3.0)])))
    e2 = layer("e2b", layer("e2a", pool(e1)))
    v = layer("e3c", layer("e3b", layer("e3a", pool(e2))))
    v = layer("d2b", layer("d2a", torch.cat([up(v), e2])))
    v = layer("d1b", layer("d1a", torch.cat([up(v), e1])))
    return x[None] + layer("head", v)
