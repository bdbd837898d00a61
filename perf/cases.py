"""Performance cases: what a program does with the library, through its public entry points.

A case is a dict of plain values. `call` says which entry points it goes through:

  measure   one ImageProximity measure of a resident image and template
  find      a measure, then the index reduction of its map (the reference's way to locate a part)
  track     a host frame is sent, the best match of a template is returned (ocipProximityIndx)
  fft       an FFT-named measure (templates of any size, tensor path)
  batch     every image against every template, one prepared batch
  gradient  SqrDistance and CrossCorr_Norm, then the gradients of both
  integral  the Integral and the SqrIntegral table of one image

and the other entries give the path (plain, auto, tensor), pixel type and sizes.
"""
import math

import numpy as np
import torch

from openclipp_b200 import ocip

_PATHS = {"plain": ocip.PATH_PLAIN, "auto": ocip.PATH_AUTO, "tensor": ocip.PATH_TENSOR}
_TYPES = {"u8": np.uint8, "u16": np.uint16, "f32": np.float32, "f64": np.float64}
# Types torch can hold the raw bits of an image in (it has few operations on unsigned 16-bit).
_RAW = {"u8": torch.uint8, "u16": torch.int16, "f32": torch.float32, "f64": torch.float64}
_SIDES = (8, 12, 16, 24, 32, 48, 64)  # template sides of the batches


def listed():
    return [
        # Part search on a small camera image with the drop-in defaults: latency and launches.
        {"name": "plain_u8_512_t16", "call": "measure", "path": "plain", "type": "u8",
         "measure": "CrossCorr_Norm", "w": 512, "h": 512, "ch": 1, "tw": 16, "th": 16},
        # A video loop: each VGA frame comes from the host, only the position goes back.
        {"name": "track_u8_640x480_t24", "call": "track", "path": "auto", "type": "u8",
         "measure": "CrossCorr_Norm", "w": 640, "h": 480, "ch": 1, "tw": 24, "th": 24},
        # The reference's flow on an odd-sized float image: map, then the place of its minimum.
        {"name": "find_f32_1021x767_t31", "call": "find", "path": "plain", "type": "f32",
         "measure": "SqrDistance_Norm", "w": 1021, "h": 767, "ch": 1, "tw": 31, "th": 31},
        # An HD frame with a ragged template, 8-bit scores exact on either kind of kernel.
        {"name": "auto_u8_1920x1080_t48x40", "call": "measure", "path": "auto", "type": "u8",
         "measure": "CrossCorr_Norm", "w": 1920, "h": 1080, "ch": 1, "tw": 48, "th": 40},
        # Sum of absolute differences, the usual 8-bit block matching measure.
        {"name": "abs_u8_1920x1080_t31", "call": "measure", "path": "plain", "type": "u8",
         "measure": "AbsDistance", "w": 1920, "h": 1080, "ch": 1, "tw": 31, "th": 31},
        # The large single image, the measure most used for matching, on tensor cores.
        {"name": "f32_4096_t31_ccnorm", "call": "measure", "path": "tensor", "type": "f32",
         "measure": "CrossCorr_Norm", "w": 4096, "h": 4096, "ch": 1, "tw": 31, "th": 31},
        # The same image with the measure that has no product form.
        {"name": "f32_4096_t31_abs", "call": "measure", "path": "plain", "type": "f32",
         "measure": "AbsDistance", "w": 4096, "h": 4096, "ch": 1, "tw": 31, "th": 31},
        # A 4K four-channel 16-bit image with the largest one-tile template.
        {"name": "u16_3840x2160x4_t64", "call": "measure", "path": "tensor", "type": "u16",
         "measure": "SqrDistance_Norm", "w": 3840, "h": 2160, "ch": 4, "tw": 64, "th": 64},
        # A large template, which the reference serves with its FFT entry points.
        {"name": "fft_f32_2048x1536_t200x120", "call": "fft", "path": "plain", "type": "f32",
         "measure": "CrossCorrFFT_Norm", "w": 2048, "h": 1536, "ch": 1, "tw": 200, "th": 120},
        # Many templates of uneven sizes over a set of images.
        {"name": "batch_u8_6x1024_10t", "call": "batch", "path": "tensor", "type": "u8",
         "measure": "SqrDistance", "w": 1024, "h": 1024, "ch": 1, "images": 6, "templates": 10},
        # Template refinement: forward maps and gradients of one image and template.
        {"name": "gradient_f32_1024_t32", "call": "gradient", "path": "tensor", "type": "f32",
         "measure": "", "w": 1024, "h": 1024, "ch": 1, "tw": 32, "th": 32},
        # Both tables behind normalised measures, the library's pure memory path.
        {"name": "integral_f32_4096", "call": "integral", "path": "plain", "type": "f32",
         "measure": "", "w": 4096, "h": 4096, "ch": 1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: images of 256 to 4096 a side, templates of 8 to 64 (up to
    256 for the FFT names), sizes mostly odd; kept below the largest listed case's cost."""
    call = rng.choice(["measure"] * 5 + ["find", "track", "fft", "batch", "gradient", "integral"])
    w, h = _log(rng, 256, 4096), _log(rng, 256, 4096)
    tw, th = rng.randint(8, 64), rng.randint(8, 64)
    c = {"call": call, "path": "tensor", "type": "f32", "measure": "", "w": w, "h": h, "ch": 1}
    product = ["SqrDistance", "SqrDistance_Norm", "CrossCorr", "CrossCorr_Norm"]
    if call == "integral":
        c.update(path="plain", type=rng.choice(["u8", "u16", "f32"]))
        return c
    if call == "batch":
        c.update(type=rng.choice(["u8", "u8", "f32"]), measure=rng.choice(product),
                 w=_log(rng, 256, 1024), h=_log(rng, 256, 1024),
                 images=rng.randint(2, 6), templates=rng.randint(2, 10))
        return c
    c.update(tw=tw, th=th)
    if call == "fft":
        c.update(path="plain", measure=rng.choice(["SqrDistanceFFT", "SqrDistanceFFT_Norm",
                                                   "CrossCorrFFT", "CrossCorrFFT_Norm"]),
                 w=_log(rng, 256, 2048), h=_log(rng, 256, 1536),
                 tw=rng.randint(40, 200), th=rng.randint(40, 120))
    elif call == "gradient":
        c.update(w=_log(rng, 256, 2048), h=_log(rng, 256, 2048))
    elif call == "track":
        c.update(path="auto", type="u8", w=_log(rng, 256, 1920), h=_log(rng, 256, 1080),
                 measure=rng.choice(["SqrDistance", "SqrDistance_Norm", "CrossCorr_Norm"]))
    elif call == "find" and rng.random() < 0.5:
        # The position is a whole number: the well-conditioned measure for float images.
        c.update(type="f32", measure="CrossCorr_Norm")
    elif call == "measure" and rng.random() < 0.5:
        c.update(type=rng.choice(["u8", "u16", "f32", "f32"]), measure=rng.choice(product))
        c.update(ch=rng.choice([1, 1, 1, 3, 4]))
        while c["w"] * c["h"] * c["ch"] * tw * th > 1.3e11:
            c.update(w=int(c["w"] * 0.8), h=int(c["h"] * 0.8))
    else:
        c.update(path="plain", type=rng.choice(["u8", "u8", "u16", "f32", "f32", "f64"]),
                 measure=rng.choice(product + ["AbsDistance"]))
        if call == "find" and c["measure"] == "CrossCorr":
            c.update(measure="CrossCorr_Norm")  # a plain product finds the brightest place
    if c["path"] == "plain" and call in ("measure", "find"):
        # Taps of the CUDA-core kernels: 8-bit and float sources, then the double-precision ones.
        most = 1.0e10 if c["type"] in ("u8", "f32") else 2.0e9
        if c["type"] == "u8" and c["measure"] != "AbsDistance" and c["tw"] * c["th"] > 258:
            most = 2.0e9
        while c["w"] * c["h"] * c["tw"] * c["th"] > most:
            k = max(("w", "h", "tw", "th"), key=lambda n: c[n] / (1 if n in ("w", "h") else 1 / 32))
            c[k] = max(8, int(c[k] * 0.8))
    return c


# ---- Inputs -------------------------------------------------------------------------------------

def _field(g, h, w):
    """Smooth blobs plus noise: 200 Gaussians of sigma 4..40 and amplitude 0..1, noise 0..0.05."""
    dev = g.device
    u = torch.rand(4, 200, generator=g, device=dev)
    sig = 4 + 36 * u[2]
    gy = torch.exp(-0.5 * ((torch.arange(h, device=dev)[None] - u[0][:, None] * h) / sig[:, None]) ** 2)
    gx = torch.exp(-0.5 * ((torch.arange(w, device=dev)[None] - u[1][:, None] * w) / sig[:, None]) ** 2)
    return (gy * u[3][:, None]).T @ gx + 0.05 * torch.rand(h, w, generator=g, device=dev)


def _source(g, c):
    """(source, template makers): pixel values as the tensor type that holds their bits."""
    h, w, ch = c["h"], c["w"], c["ch"]
    planes = []
    for _ in range(ch):
        f = _field(g, h, w)
        if c["type"] in ("u8", "u16"):
            f = f * (200.0 / f.max()) + torch.rand(h, w, generator=g, device=f.device) * 55
        planes.append(f)
    v = torch.stack(planes, -1)
    if c["type"] == "u8":
        return v.round().clamp(0, 255)
    if c["type"] == "u16":
        return (v * 257).round().clamp(0, 65535)
    return v


def _template(g, c, src, tw, th):
    """A crop of the source with noise, in the source's range."""
    at = torch.rand(2, generator=g, device=g.device).tolist()
    y, x = int(at[0] * (c["h"] - th)), int(at[1] * (c["w"] - tw))
    t = src[y:y + th, x:x + tw]
    n = torch.randn(t.shape, generator=g, device=g.device)
    if c["type"] == "u8":
        return (t + 4 * n).round().clamp(0, 255)
    if c["type"] == "u16":
        return (t + 1028 * n).round().clamp(0, 65535)
    return t + 0.02 * n


def _inputs(c, seed):
    """Sources, templates and upstream gradients of a case, as float or double values."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    srcs = [_source(g, c) for _ in range(c.get("images", 1))]
    if c["call"] == "batch":
        pick = torch.rand(c["templates"], generator=g, device=g.device).tolist()
        # Template sides go round the list, so that every seed has the same work.
        sides = [_SIDES[j % len(_SIDES)] for j in range(c["templates"])]
        tpls = [_template(g, c, srcs[int(p * len(srcs))], s, s) for p, s in zip(pick, sides)]
    elif "tw" in c:
        tpls = [_template(g, c, srcs[0], c["tw"], c["th"])]
    else:
        tpls = []
    ups = []
    if c["call"] == "gradient":
        ups = [torch.randn(c["h"], c["w"], 1, generator=g, device=g.device) for _ in range(2)]
    kind = torch.float64 if c["type"] == "f64" else torch.float32
    return [s.to(kind) for s in srcs], [t.to(kind) for t in tpls], ups


class _Rows:
    """An image's device rows as a CUDA array; keeps the image (a tensor made from it keeps this)."""

    def __init__(self, img, kind):
        self.img = img
        ptr, pitch = img.device_ptr()
        d = img.desc
        item = np.dtype(kind).itemsize
        self.__cuda_array_interface__ = {
            "shape": (d.Height, d.Width * d.Channels), "typestr": np.dtype(kind).str,
            "data": (ptr, False), "strides": (pitch, item), "version": 2}


def _view(img, kind):
    return torch.as_tensor(_Rows(img, kind), device="cuda")


class _State:
    """What a program keeps between calls: its images, its programs, its context."""

    def __init__(self, case, ctx):
        self.case, self.ctx = case, ctx
        self.fill, self.programs = [], []

    def upload(self, value, kind):
        img = ocip.Image(shape=tuple(value.shape), dtype=_TYPES[kind])
        self.fill.append((img, value, kind))
        return img

    def result(self, shape, kind=np.float32):
        img = ocip.Image(shape=shape, dtype=kind)
        return img, _view(img, kind)

    def finish(self):
        self.ctx.finish()
        for img, value, kind in self.fill:
            if kind == "u16":
                value = torch.where(value > 32767, value - 65536, value)
            raw = np.int16 if kind == "u16" else _TYPES[kind]
            _view(img, raw).copy_(value.to(_RAW[kind]).reshape(value.shape[0], -1))
        torch.cuda.synchronize()
        self.fill = []

    def __del__(self):
        # An image is released with the last reference to it: results outlive the state.
        for p in self.programs:
            p.release()


_contexts = {}


def _context(path):
    if path not in _contexts:
        _contexts[path] = ocip.Context(torch.cuda.current_device())
        _contexts[path].set_path(_PATHS[path])
    _contexts[path].make_current()
    return _contexts[path]


def prepare(case, seed):
    c = dict(case)
    torch.cuda.init()
    s = _State(c, _context(c["path"]))
    srcs, tpls, ups = _inputs(c, seed)
    shape = (c["h"], c["w"], c["ch"])
    if c["call"] == "track":
        s.frame = srcs[0].to(torch.uint8).reshape(c["h"], c["w"]).cpu().numpy()
        s.src = ocip.Image(s.frame)
    else:
        s.srcs = [s.upload(v, c["type"]) for v in srcs]
        s.src = s.srcs[0]
    s.tpls = [s.upload(v, c["type"]) for v in tpls]
    kind = np.float64 if c["type"] == "f64" else np.float32
    if c["call"] in ("measure", "find", "fft"):
        s.dst, s.out = s.result(shape, kind)
    if c["call"] == "find":
        s.programs.append(ocip.prepare_statistics(s.dst))
    elif c["call"] == "fft":
        s.programs.append(ocip.prepare_proximity_fft(s.src, s.tpls[0]))
    elif c["call"] == "integral":
        s.programs.append(ocip.prepare_integral(s.src))
        s.sum, s.sum_out = s.result(shape, np.float64)
        s.sqr, s.sqr_out = s.result(shape, np.float64)
    elif c["call"] == "gradient":
        s.up = [s.upload(v, "f32") for v in ups]
        s.fwd = [s.result(shape) for _ in range(2)]
        s.gs, s.gs_out = s.result(shape)
        s.gt, s.gt_out = s.result((c["th"], c["tw"], 1))
    elif c["call"] == "batch":
        s.dsts = [s.result(shape) for _ in range(len(srcs) * len(tpls))]
    s.finish()
    if c["call"] == "batch":
        s.programs.append(ocip.prepare_batch(c["measure"], s.srcs, s.tpls, [d for d, _ in s.dsts]))
    torch.cuda.synchronize()
    return s


def run(s):
    c = s.case
    s.ctx.make_current()
    call = c["call"]
    if call in ("measure", "find"):
        ocip.check(ocip.proximity(c["measure"], s.src, s.tpls[0], s.dst), c["measure"])
        if call == "measure":
            return s.out
        rc, v, x, y = ocip.index_reduce(_best(c["measure"]), s.programs[0], s.dst)
        ocip.check(rc, "index reduction")
        return s.out, v, x, y
    if call == "track":
        s.src.send()
        rc, v, x, y = ocip.proximity_index(c["measure"], _best(c["measure"]), s.src, s.tpls[0])
        ocip.check(rc, "ocipProximityIndx")
        return v, x, y
    if call == "fft":
        fn = getattr(ocip.lib, "ocip" + c["measure"])
        ocip.check(fn(s.programs[0].handle, s.src.handle, s.tpls[0].handle, s.dst.handle),
                   c["measure"])
        return s.out
    if call == "integral":
        ocip.integral(s.programs[0], s.src, s.sum)
        ocip.integral(s.programs[0], s.src, s.sqr, sqr=True)
        return s.sum_out, s.sqr_out
    if call == "batch":
        ocip.check(s.programs[0].run(), "ocipRunProximityBatch")
        return [v for _, v in s.dsts]
    ocip.sqr_distance(s.src, s.tpls[0], s.fwd[0][0])
    ocip.cross_corr_norm(s.src, s.tpls[0], s.fwd[1][0])
    ocip.check(ocip.proximity_backward(s.src, s.tpls[0], s.up[0], s.up[1], s.fwd[1][0], s.gs, s.gt),
               "ocipProximityBackward")
    return s.fwd[0][1], s.fwd[1][1], s.gs_out, s.gt_out


def _best(measure):
    return "MaxIndx" if measure.startswith("CrossCorr") else "MinIndx"


# ---- Work ---------------------------------------------------------------------------------------

def work(case):
    """Bytes: each source, template and gradient map read once, each result written once.
    Flops: two per template pixel and output (one product sum per map; the energies add up from
    running sums), the adjoint's two correlations counted as well. A large template's product sums
    need no more than a transform of the image, of the template and of their product."""
    c = case
    px = c["w"] * c["h"] * c["ch"]
    size = np.dtype(_TYPES[c["type"]]).itemsize
    out = 8 if c["type"] == "f64" else 4
    if c["call"] == "integral":
        return {"bytes": px * (size + 16), "flops": 5 * px}
    if c["call"] == "batch":
        sides = [_SIDES[j % len(_SIDES)] for j in range(c["templates"])]
        taps = sum(t * t for t in sides)
        pairs = c["images"] * c["templates"]
        return {"bytes": px * size * c["images"] + taps * size + px * out * pairs,
                "flops": 2 * px * taps * c["images"]}
    taps = c["tw"] * c["th"]
    if c["call"] == "track":
        return {"bytes": px * size + taps * size, "flops": 2 * px * taps}
    if c["call"] == "gradient":
        return {"bytes": px * 4 * 6 + taps * 8, "flops": 6 * px * taps}
    flops = 2 * px * taps
    if c["call"] == "fft":
        n = (c["w"] + c["tw"]) * (c["h"] + c["th"])
        flops = min(flops, 7.5 * n * math.log2(n))
    return {"bytes": px * (size + out) + taps * size * c["ch"], "flops": flops}


# ---- Values in 64 bits --------------------------------------------------------------------------

def _windows(src, tw, th, ax, ay):
    """The source padded with zeros so that [h:h+H, w:w+W] is the window element (w, h)."""
    h, w = src.shape[:2]
    p = torch.zeros((h + th - 1, w + tw - 1) + tuple(src.shape[2:]), dtype=torch.float64,
                    device=src.device)
    p[ay:ay + h, ax:ax + w] = src
    return p


def _correlate(src, t, ax, ay):
    """sum_{w,h} src(x + w - ax, y + h - ay) t(w, h), per channel."""
    th, tw = t.shape[:2]
    h, w = src.shape[:2]
    p = _windows(src, tw, th, ax, ay)
    acc = torch.zeros(src.shape, dtype=torch.float64, device=src.device)
    tl = t.tolist()
    for j in range(th):
        for i in range(tw):
            for k in range(src.shape[2]):
                acc[..., k].add_(p[j:j + h, i:i + w, k], alpha=tl[j][i][k])
    return acc


def _box(src, tw, th, ax, ay):
    """Window sums."""
    h, w = src.shape[:2]
    p = _windows(src, tw, th, ax, ay)
    rows = torch.zeros((h + th - 1, w) + tuple(src.shape[2:]), dtype=torch.float64, device=src.device)
    for i in range(tw):
        rows += p[:, i:i + w]
    acc = torch.zeros(src.shape, dtype=torch.float64, device=src.device)
    for j in range(th):
        acc += rows[j:j + h]
    return acc


def _map(measure, s, t):
    th, tw = t.shape[:2]
    ax, ay = tw // 2, th // 2
    if measure == "AbsDistance":
        h, w = s.shape[:2]
        p = _windows(s, tw, th, ax, ay)
        acc = torch.zeros(s.shape, dtype=torch.float64, device=s.device)
        for j in range(th):
            for i in range(tw):
                acc += (p[j:j + h, i:i + w] - t[j, i]).abs_()
        return acc
    v = _correlate(s, t, ax, ay)
    if measure == "CrossCorr":
        return v
    es, et = _box(s * s, tw, th, ax, ay), (t * t).sum((0, 1))
    if measure.startswith("SqrDistance"):
        v = es - 2 * v + et
    return v / (es * et).sqrt() if measure.endswith("_Norm") else v


def _gradients(s, t, up):
    """Maps and gradients of sum up0 * SqrDistance + sum up1 * CrossCorr_Norm."""
    th, tw = t.shape[:2]
    h, w = s.shape[:2]
    ax, ay = tw // 2, th // 2
    es, et = _box(s * s, tw, th, ax, ay), (t * t).sum()
    cc = _correlate(s, t, ax, ay)
    n = cc / (es * et).sqrt()
    m = -2 * up[0] + up[1] / (es * et).sqrt()
    p = 2 * up[0] - up[1] * n / es
    gs = _correlate(m, t.flip(0, 1), tw - 1 - ax, th - 1 - ay)
    gs += s * _box(p, tw, th, tw - 1 - ax, th - 1 - ay)
    win = _windows(s, tw, th, ax, ay)
    gt = torch.stack([torch.stack([(m * win[j:j + h, i:i + w]).sum() for i in range(tw)])
                      for j in range(th)])[..., None]
    gt = gt + t * (2 * up[0].sum() - (up[1] * n).sum() / et)
    return es - 2 * cc + et, n, gs, gt


def exact(case, seed):
    c = dict(case)
    srcs, tpls, ups = _inputs(c, seed)
    srcs, tpls, ups = ([v.double() for v in x] for x in (srcs, tpls, ups))
    rows = lambda v: v.reshape(v.shape[0], -1)  # noqa: E731
    if c["call"] == "integral":
        return tuple(rows(v.cumsum(0).cumsum(1)) for v in (srcs[0], srcs[0] ** 2))
    if c["call"] == "batch":
        return [rows(_map(c["measure"], s, t)) for s in srcs for t in tpls]
    if c["call"] == "gradient":
        return tuple(rows(v) for v in _gradients(srcs[0], tpls[0], ups))
    v = rows(_map(c["measure"].replace("FFT", ""), srcs[0], tpls[0]))
    if c["call"] in ("measure", "fft"):
        return v
    best = float(v.max() if _best(c["measure"]) == "MaxIndx" else v.min())
    return (v, best, None, None) if c["call"] == "find" else (best, None, None)
