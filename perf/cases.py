"""Performance cases of the codec, through its public Python entry points.

A pass is what a user's program does with a field already in GPU memory: one
compression (a relative bound is resolved on the field first) or one decode,
of a single field or of a batch of chunks. Archives are byte streams and
decodes are defined bit for bit by the archive format, so every output has to
stay exactly what it was; `exact` gives the decode in 64-bit arithmetic.

Relative bounds are rounded to the sample type: the strict check of the format
refuses a field that has a sample between a bound and the bound's rounding.
"""
import math

import numpy as np
import torch

import waltz_b200

# Listed cases. "op": compress or decompress. "data": "smooth" (random field of
# spectrum |k|^(-11/3), what a resolved turbulence or climate variable looks
# like to a wavelet), "spikes" (the same with 1 % of the samples at +-50:
# detector hits, masks), "front" (|k|^(-5/3) and a sharp layer along z).
# "rel": bound relative to the value range; "abs": absolute bound. Sizes are
# (z, y, x).
_LISTED = [
    # a small block, as of an adaptive mesh or an interactive viewer: latency
    {"name": "enc_f32_64", "op": "compress", "dtype": "f32", "z": 64, "y": 64, "x": 64,
     "data": "smooth", "rel": 1e-3, "form": "plain"},
    {"name": "dec_f32_64", "op": "decompress", "dtype": "f32", "z": 64, "y": 64, "x": 64,
     "data": "smooth", "rel": 1e-3, "form": "plain"},
    # a field whose sides are multiples of nothing: staggered or cropped grids
    {"name": "enc_f32_181x257x333", "op": "compress", "dtype": "f32", "z": 181, "y": 257, "x": 333,
     "data": "smooth", "rel": 1e-3, "form": "plain"},
    {"name": "dec_f32_181x257x333", "op": "decompress", "dtype": "f32", "z": 181, "y": 257, "x": 333,
     "data": "smooth", "rel": 1e-3, "form": "plain"},
    # the snapshot of a large simulation cube: the headline workload
    {"name": "enc_f32_512", "op": "compress", "dtype": "f32", "z": 512, "y": 512, "x": 512,
     "data": "smooth", "rel": 1e-3, "form": "plain"},
    {"name": "dec_f32_512", "op": "decompress", "dtype": "f32", "z": 512, "y": 512, "x": 512,
     "data": "smooth", "rel": 1e-3, "form": "plain"},
    # wide and shallow (atmosphere levels, detector stacks); the form left to
    # the library, which takes the tensor-core one
    {"name": "enc_f32_64x1024x1024_auto", "op": "compress", "dtype": "f32", "z": 64, "y": 1024, "x": 1024,
     "data": "spikes", "rel": 1e-3, "form": "auto"},
    {"name": "dec_f32_64x1024x1024_auto", "op": "decompress", "dtype": "f32", "z": 64, "y": 1024, "x": 1024,
     "data": "spikes", "rel": 1e-3, "form": "auto"},
    # double precision, an absolute bound, the plane schedule in the plain form
    {"name": "enc_f64_96x256x384", "op": "compress", "dtype": "f64", "z": 96, "y": 256, "x": 384,
     "data": "front", "abs": 1e-4, "form": "plain"},
    {"name": "dec_f64_96x256x384", "op": "decompress", "dtype": "f64", "z": 96, "y": 256, "x": 384,
     "data": "front", "abs": 1e-4, "form": "plain"},
    # a chunked dataset: many uneven chunks a call, each with its own range
    {"name": "enc_batch_512", "op": "compress", "dtype": "f32", "chunks": 512, "lo": 32, "hi": 128, "step": 16,
     "data": "smooth", "rel": 1e-3},
    {"name": "dec_batch_512", "op": "decompress", "dtype": "f32", "chunks": 512, "lo": 32, "hi": 128, "step": 16,
     "data": "smooth", "rel": 1e-3},
]


def listed():
    return [dict(c) for c in _LISTED]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a near-cube, a shallow field or a batch, of any sides."""
    op = rng.choice(["compress", "decompress"])
    kind = rng.choice(["cube", "cube", "plane", "plane", "batch"])
    rel = 10.0 ** rng.uniform(-4.5, -2.0)
    if kind == "batch":
        step = rng.choice([1, 8, 16])
        return {"op": op, "dtype": rng.choice(["f32", "f32", "f64"]), "chunks": _log_int(rng, 16, 256),
                "lo": 32 // step * step, "hi": 112 // step * step, "step": step, "data": "smooth", "rel": rel}
    dtype = rng.choice(["f32", "f32", "f64"])
    most = (1 << 26) if dtype == "f32" else (1 << 25)
    if kind == "cube":
        side = _log_int(rng, 48, 384)
        dims = [max(40, int(side * rng.uniform(0.75, 1.3))) for _ in range(3)]
    else:
        dims = [_log_int(rng, 16, 128), _log_int(rng, 128, 1024), _log_int(rng, 128, 1024)]
    if rng.random() < 0.4:  # grids of whole tiles are common too
        dims = [max(16, d // 16 * 16) for d in dims]
    while dims[0] * dims[1] * dims[2] > most:
        dims[dims.index(max(dims))] //= 2
    case = {"op": op, "dtype": dtype, "z": dims[0], "y": dims[1], "x": dims[2],
            "data": rng.choice(["smooth", "spikes", "front"]), "form": rng.choice(["plain", "plain", "auto"])}
    if case["data"] == "front":
        case["abs"] = 10.0 ** rng.uniform(-3.5, -2.0)
    else:
        case["rel"] = rel
    return case


# ------------------------------------------------------------------ inputs
def _spectral(shape, gen, slope):
    white = torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64)
    spec = torch.fft.rfftn(white)
    nz, ny, nx = shape
    kz = torch.fft.fftfreq(nz, d=1.0 / nz, device="cuda", dtype=torch.float64)
    ky = torch.fft.fftfreq(ny, d=1.0 / ny, device="cuda", dtype=torch.float64)
    kx = torch.fft.rfftfreq(nx, d=1.0 / nx, device="cuda", dtype=torch.float64)
    k2 = kz[:, None, None] ** 2 + ky[None, :, None] ** 2 + kx[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    k2.pow_(slope / 4.0)
    k2[0, 0, 0] = 0.0
    spec.mul_(k2)
    field = torch.fft.irfftn(spec, s=shape)
    return (field - field.mean()).div_(field.std())


def _field(case, seed):
    shape = (case["z"], case["y"], case["x"])
    gen = torch.Generator(device="cuda").manual_seed(seed)
    f = _spectral(shape, gen, -5.0 / 3.0 if case["data"] == "front" else -11.0 / 3.0)
    if case["data"] == "spikes":
        hit = torch.rand(shape, generator=gen, device="cuda") < 0.01
        sign = torch.rand(shape, generator=gen, device="cuda") < 0.5
        f = torch.where(hit, torch.where(sign, -50.0, 50.0).to(f.dtype), f)
    elif case["data"] == "front":
        z = torch.arange(shape[0], device="cuda", dtype=torch.float64)
        f = f + 10.0 * torch.tanh((z - shape[0] / 2) / 2.0)[:, None, None]
    return f.to(_dtype(case)).contiguous()


def _shapes(case):
    """The chunking of a batch: fixed for a dataset, whatever its contents."""
    gen = torch.Generator().manual_seed(case["chunks"])
    sides = torch.arange(case["lo"], case["hi"] + 1, case["step"])
    picks = torch.randint(len(sides), (case["chunks"], 3), generator=gen)
    return [tuple(int(v) for v in sides[p]) for p in picks]


def _chunks(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    spans = 10.0 ** (5.0 * torch.rand(case["chunks"], generator=torch.Generator().manual_seed(seed)) - 2.0)
    fields = []
    for shape, span in zip(_shapes(case), spans.tolist()):
        f = _spectral(shape, gen, -11.0 / 3.0)
        lo, hi = torch.aminmax(f)
        fields.append(((f - lo) * (span / (hi - lo))).to(_dtype(case)).contiguous())
    return fields


def _dtype(case):
    return torch.float32 if case["dtype"] == "f32" else torch.float64


def _held(case, bound):
    return float(np.float32(bound)) if case["dtype"] == "f32" else float(bound)


def _bound(case, field):
    if "abs" in case:
        return _held(case, case["abs"])
    lo, hi = torch.aminmax(field)
    return _held(case, case["rel"] * (float(hi) - float(lo)))


def prepare(case, seed):
    if "chunks" in case:
        fields = _chunks(case, seed)
        bounds = [_bound(case, f) for f in fields]
        size = fields[0].element_size()
        room = sum(waltz_b200.compressed_capacity(f.numel(), size) + 16 for f in fields)
        out = torch.zeros(room, dtype=torch.uint8, device="cuda")  # kept by the program from batch to batch
        if case["op"] == "compress":
            return {"case": case, "fields": fields, "bounds": bounds, "out": out}
        archives = [a.clone() for a in waltz_b200.compress_batch(fields, bounds, out=out)]
        shapes = [tuple(f.shape) for f in fields]
        frame = torch.empty(sum(f.numel() for f in fields), dtype=_dtype(case), device="cuda")
        return {"case": case, "archives": archives, "shapes": shapes, "out": frame}
    field = _field(case, seed)
    if case["op"] == "compress":
        # where the program collects its archives
        record = torch.zeros(field.numel() * field.element_size() * 5 // 4 + (1 << 16), dtype=torch.uint8, device="cuda")
        return {"case": case, "field": field, "record": record}
    archive = waltz_b200.compress_tensor(field, _bound(case, field), form=case["form"]).clone()
    return {"case": case, "archive": archive, "shape": tuple(field.shape)}


def run(state):
    case = state["case"]
    if "chunks" in case:
        out = state["out"]
        if case["op"] == "compress":
            archives = waltz_b200.compress_batch(state["fields"], state["bounds"], out=out)
            return {"sizes": np.array([a.numel() for a in archives]), "archives": out}
        waltz_b200.decompress_batch(state["archives"], state["shapes"], _dtype(case), out=out)
        return out
    if case["op"] == "compress":
        field, record = state["field"], state["record"]
        bound = case["abs"] if "abs" in case else waltz_b200.rel_to_abs_bound(field, case["rel"])
        archive = waltz_b200.compress_tensor(field, _held(case, bound), form=case["form"])
        record[:archive.numel()].copy_(archive)
        return {"size": archive.numel(), "record": record}
    return waltz_b200.decompress_tensor(state["archive"], state["shape"], _dtype(case))


# ------------------------------------------------------- what a pass needs
def work(case):
    """The field and its archive (taken as a quarter of it: these data
    compress three- to fivefold) once each; the lifting of three axes, seven
    operations per sample and axis and 8/7 over the levels, in the direction
    the call has (a compression also reconstructs, to find its repairs)."""
    width = 4 if case["dtype"] == "f32" else 8
    if "chunks" in case:
        n = sum(math.prod(shape) for shape in _shapes(case))
    else:
        n = case["z"] * case["y"] * case["x"]
    passes = 2 if case["op"] == "compress" else 1
    return {"bytes": int(n * width * 1.25), "flops": int(n * 24 * passes)}


def tolerance(case):
    """The format fixes every byte of an archive and every bit of a decode."""
    return "exact"


# --------------------------------------------------- the decode in 64 bits
_A, _B, _G, _D, _K = (-1.586134342059924, -0.052980118572961, 0.882911075530934, 0.443506852043971,
                      1.1496043988602418)


def _levels(n):
    count = 0
    while n > 8 and count < 5:
        n -= n // 2
        count += 1
    return count


def _after(e, odds):   # the even sample to the right of each odd one, reflected at the end
    return torch.cat([e[1:], e[-1:]])[:odds]


def _before(o, evens):  # sum of the odd samples on both sides of each even one
    left = torch.cat([o[:1], o])[:evens]
    right = torch.cat([o, o[-1:]])[:evens]
    return left + right


def _lift(box, axis, inverse):
    x = box.movedim(axis, 0)
    n = x.shape[0]
    h = n - n // 2
    if inverse:
        e, o = x[:h] / _K, x[h:] * -_K
        e = e - _D * _before(o, h)
        o = o - _G * (e[:n - h] + _after(e, n - h))
        e = e - _B * _before(o, h)
        o = o - _A * (e[:n - h] + _after(e, n - h))
        y = torch.empty_like(x)
        y[0::2], y[1::2] = e, o
    else:
        e, o = x[0::2].clone(), x[1::2].clone()
        o = o + _A * (e[:n - h] + _after(e, n - h))
        e = e + _B * _before(o, h)
        o = o + _G * (e[:n - h] + _after(e, n - h))
        e = e + _D * _before(o, h)
        y = torch.cat([e * _K, o / -_K])
    return y.movedim(0, axis)


def _steps(shape):
    """(axes, box) of every analysis step: all axes level by level where they
    have the same number of levels, else all of z, then y and x."""
    nz, ny, nx = shape
    lz, lxy = _levels(nz), _levels(min(nx, ny))
    steps, box = [], [nz, ny, nx]

    def add(axes, count):
        for _ in range(count):
            steps.append((axes, tuple(box)))
            for a in axes:
                box[a] -= box[a] // 2
    if lz == lxy:
        add((1, 2, 0), lz)
    else:
        add((0,), lz)
        box[0] = nz
        add((1, 2), lxy)
    return steps


def _decoded(field, bound):
    c = field.to(torch.float64, copy=True)
    steps = _steps(tuple(c.shape))
    for axes, (bz, by, bx) in steps:
        for axis in axes:
            c[:bz, :by, :bx] = _lift(c[:bz, :by, :bx], axis, False)
    quantum = 1.5 * bound
    c = torch.round(c / quantum) * quantum
    for axes, (bz, by, bx) in reversed(steps):
        for axis in reversed(axes):
            c[:bz, :by, :bx] = _lift(c[:bz, :by, :bx], axis, True)
    original = field.to(torch.float64)
    return torch.where((c - original).abs() > bound, original, c)


def exact(case, seed):
    """A decode's samples; archives have no 64-bit value."""
    if case["op"] == "compress":
        return None
    if "chunks" in case:
        return torch.cat([_decoded(f, _bound(case, f)).reshape(-1) for f in _chunks(case, seed)])
    field = _field(case, seed)
    return _decoded(field, _bound(case, field))
