"""The workloads this framework is timed on, through its public entry points.

Twelve listed cases and a generator of more of the same ranges: plain batched
transforms (short calls, power-of-two, smooth and long axes), half-precision
2-D transforms, real 2-D transforms, the FFT convolution of image batches, a
differentiable 3-D convolution, batches of uneven lengths, lengths with large
primes, map hooks, and reductions.  Shapes are those of the benchmark
configurations and the tests, or generic ones (full-HD frames, 1500-point
rows).
"""

from __future__ import annotations

import math

import numpy as np
import torch

import vkdispatch_gb300 as vd
import vkdispatch_gb300.autograd as ag
import vkdispatch_gb300.codegen as vc
from vkdispatch_gb300.batch import BatchPlan

_DTYPES = {"complex64": torch.complex64, "complex128": torch.complex128}
_HALF = {"bf16": vd.complexbf16, "fp16": vd.complex32}


def listed():
    return [
        # a small batch, host data already on the device: launches and latency count
        {"name": "roundtrip_256x1024", "kind": "roundtrip", "rows": 256, "n": 1024},
        # the same transform at HBM scale
        {"name": "fft_1024", "kind": "fft", "outer": 32768, "n": 1024, "inner": 1, "dtype": "complex64",
         "inverse": False},
        # a smooth length that is not a power of two, the kind an application arrives with
        {"name": "fft_1500", "kind": "fft", "outer": 16001, "n": 1500, "inner": 1, "dtype": "complex64",
         "inverse": True},
        # a long axis (spectrometers, long records)
        {"name": "fft_65536", "kind": "fft", "outer": 384, "n": 65536, "inner": 1, "dtype": "complex64",
         "inverse": False},
        # the mixed-precision 2-D transform: 16-bit storage, fp32 butterflies
        {"name": "fft2_bf16_16384", "kind": "half2", "images": 1, "h": 16384, "w": 16384, "type": "bf16"},
        # real frames to half spectra and back
        {"name": "rfft2_1080x1920", "kind": "rfft2", "images": 16, "h": 1080, "w": 1920},
        # the image convolution of the benchmark: one kernel spectrum per image
        {"name": "convolve2dr_64x512x512", "kind": "convolve2dr", "images": 64, "h": 512, "w": 512,
         "broadcast": False},
        # a learnable 3-D convolution, forward and backward
        {"name": "conv_train_256", "kind": "conv_train", "d": 256, "h": 256, "w": 256},
        # many transforms of uneven lengths in one launch, forward and inverse
        {"name": "uneven_1024_items", "kind": "uneven", "items": 1024, "points": 1 << 26, "mix": 3},
        # a prime length: the user's record is what it is
        {"name": "fft_prime_1009", "kind": "fft", "outer": 4096, "n": 1009, "inner": 1, "dtype": "complex64",
         "inverse": False},
        # map hooks: cross-correlation of a padded region, columns
        {"name": "padded_correlation_600", "kind": "padded", "outer": 16, "rows": 1024, "cols": 600, "inner": 512},
        # row sums
        {"name": "reduce_rows_65536", "kind": "reduce", "rows": 1024, "n": 65536, "op": "add", "type": "float32"},
    ]


# ---------------------------------------------------------------------------
# drawn cases
# ---------------------------------------------------------------------------
def _smooth(primes, lo, hi):
    out = [1]
    for p in primes:
        more = []
        for v in out:
            while v <= hi:
                more.append(v)
                v *= p
        out = more
    return sorted(v for v in out if v >= lo)


_SMOOTH13 = _smooth((2, 3, 5, 7, 11, 13), 2, 1 << 17)
_SMOOTH7 = _smooth((2, 3, 5, 7), 16, 65536)


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _near(rng, table, lo, hi):
    """An entry of a sorted table, spread over the logarithm of [lo, hi]; a power of two one time in three."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    if rng.random() < 1 / 3:
        p = 1 << int(round(math.log2(x)))
        if lo <= p <= hi:
            return p
    return min((v for v in table if lo <= v <= hi), key=lambda v: abs(math.log(v / x)))


def draw(rng):
    kind = rng.choice(["roundtrip", "fft", "fft", "fft", "half2", "rfft2", "convolve2dr", "conv_train", "uneven",
                       "prime", "padded", "reduce"])
    if kind == "roundtrip":
        n = _near(rng, _SMOOTH13, 16, 4096)
        return {"kind": kind, "rows": max(1, _log(rng, 1 << 10, 1 << 20) // n), "n": n}
    if kind == "fft":
        dtype = "complex128" if rng.random() < 0.15 else "complex64"
        n = _near(rng, _SMOOTH13, 16, 4096 if dtype == "complex128" else 1 << 17)
        points = _log(rng, 1 << 14, 1 << (23 if dtype == "complex128" else 25))
        inner = 1 if rng.random() < 0.6 else min(_log(rng, 2, 512), max(2, points // n))
        return {"kind": kind, "outer": max(1, points // (n * inner)), "n": n, "inner": inner, "dtype": dtype,
                "inverse": rng.random() < 0.5}
    if kind == "prime":
        while True:
            n = _log(rng, 17, 16381)
            if n not in _SMOOTH13:
                break
        inner = 1 if rng.random() < 0.7 else _log(rng, 2, 64)
        return {"kind": "fft", "outer": max(1, _log(rng, 1 << 14, 1 << 22) // (n * inner)), "n": n, "inner": inner,
                "dtype": "complex64", "inverse": rng.random() < 0.5}
    if kind == "half2":
        t = rng.choice(["bf16", "fp16"])
        hi = 16384 if t == "bf16" else 1024  # unscaled fp16 spectra of larger images leave the type's range
        h, w = _near(rng, _SMOOTH13, 64, hi), _near(rng, _SMOOTH13, 64, hi)
        return {"kind": kind, "images": max(1, _log(rng, 1 << 16, 1 << 24) // (h * w)), "h": h, "w": w, "type": t}
    if kind == "rfft2":
        h, w = _near(rng, _SMOOTH13, 32, 2048), _near(rng, [v for v in _SMOOTH13 if v % 2 == 0], 32, 2048)
        return {"kind": kind, "images": max(1, _log(rng, 1 << 14, 1 << 25) // (h * w)), "h": h, "w": w}
    if kind == "convolve2dr":
        h, w = _near(rng, _SMOOTH13, 64, 1024), _near(rng, [v for v in _SMOOTH13 if v % 2 == 0], 64, 1024)
        return {"kind": kind, "images": max(1, _log(rng, 1 << 16, 1 << 24) // (h * w)), "h": h, "w": w,
                "broadcast": rng.random() < 0.5}
    if kind == "conv_train":
        return {"kind": kind, "d": _near(rng, _SMOOTH13, 8, 256), "h": _near(rng, _SMOOTH13, 8, 256),
                "w": _near(rng, _SMOOTH13, 8, 256)}
    if kind == "uneven":
        points = _log(rng, 1 << 21, 1 << 26)
        return {"kind": kind, "items": _log(rng, 8, max(8, points >> 16)), "points": points,
                "mix": rng.randrange(1 << 20)}
    if kind == "padded":
        cols, inner = _near(rng, _SMOOTH13, 16, 2048), _log(rng, 1, 512)
        return {"kind": kind, "outer": max(1, _log(rng, 1 << 14, 1 << 23) // (cols * inner)),
                "rows": cols + _log(rng, 1, cols), "cols": cols, "inner": inner}
    t = rng.choice(["float32", "float32", "int32", "complex64"])
    total = _log(rng, 1 << 10, 1 << 26)
    n = _log(rng, 16, total)
    return {"kind": "reduce", "rows": max(1, min(16384, total // n)), "n": n,
            "op": "add" if t == "complex64" else rng.choice(["add", "max"]) if t == "float32" else "max", "type": t}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _crandn(shape, gen, dtype=torch.complex64):
    real = torch.float64 if dtype == torch.complex128 else torch.float32
    return torch.view_as_complex(torch.randn(tuple(shape) + (2,), generator=gen, device="cuda", dtype=real))


def _half_input(case, seed):
    t = torch.bfloat16 if case["type"] == "bf16" else torch.float16
    out = torch.empty((case["images"], case["h"], case["w"], 2), dtype=t, device="cuda")
    gen = _gen(seed)
    flat = out.view(-1)
    step = 1 << 26  # in pieces: the fp32 values of the largest image need not all exist at once
    for i in range(0, flat.numel(), step):
        m = min(step, flat.numel() - i)
        flat[i:i + m] = torch.randn(m, generator=gen, device="cuda")
    return out


def _gaussian_spectrum(h, w):
    """Half spectrum of a normalised 31 x 31 Gaussian (sigma 5), zero-padded to h x w."""
    i = torch.arange(31, dtype=torch.float64, device="cuda") - 15
    g = torch.exp(-i * i / 50.0)
    k = torch.outer(g, g)
    pad = torch.zeros((h, w), dtype=torch.float64, device="cuda")
    pad[:31, :31] = k / k.sum()
    return torch.fft.rfft2(pad).to(torch.complex64)


def _uneven_items(case):
    """(offset, length, count) items: 7-smooth lengths, log-uniform in [16, 65536]."""
    rng = np.random.default_rng(case["mix"])
    logs = np.log(np.array(_SMOOTH7, dtype=np.float64))
    u = rng.uniform(math.log(16), math.log(65536), case["items"])
    lengths = [_SMOOTH7[int(np.argmin(np.abs(logs - x)))] for x in u]
    share = max(1, case["points"] // case["items"])
    items, off = [], 0
    for n in lengths:
        c = max(1, int(round(share / n)))
        items.append((off, n, c))
        off += n * c
    return items, off


def _padded_maps(case):
    """The maps of a transform over the first `cols` rows of axis 1."""
    full = (case["outer"], case["rows"], case["inner"])
    trimmed = (case["outer"], case["cols"], case["inner"])

    def remap(io_index):
        return vc.unravel_index(vc.ravel_index(io_index, trimmed).to_register(), full)

    @vd.map
    def input_map(inb: vc.Buffer[vc.c64]):
        op = vd.fft.read_op()
        op.read_from_buffer(inb, io_index=remap(op.io_index))

    @vd.map
    def output_map(outb: vc.Buffer[vc.c64]):
        op = vd.fft.write_op()
        op.write_to_buffer(outb, io_index=remap(op.io_index))

    @vd.map
    def kernel_map(spectrum: vc.Buffer[vc.c64]):
        op = vd.fft.read_op()
        k = vc.new_register(vc.c64)
        op.read_from_buffer(spectrum, register=k)
        op.register[:] = vc.mult_complex(op.register, k.conjugate())

    return input_map, output_map, kernel_map


@vd.reduce.map_reduce(vd.reduce.SubgroupAdd)
def _magnitude_sum(buffer: vc.Buff[vd.complex64]) -> vd.float32:
    v = buffer[vd.reduce.mapped_io_index()]
    return vc.sqrt(v.real * v.real + v.imag * v.imag)


@vd.reduce.map_reduce(vd.reduce.SubgroupAdd, axes=[1])
def _magnitude_rows(buffer: vc.Buff[vd.complex64]) -> vd.float32:
    v = buffer[vd.reduce.mapped_io_index()]
    return vc.sqrt(v.real * v.real + v.imag * v.imag)


@vd.reduce.reduce(0, axes=[1])
def _add_f32(a: vc.f32, b: vc.f32) -> vc.f32:
    return a + b


@vd.reduce.reduce("-inf", axes=[1])
def _max_f32(a: vc.f32, b: vc.f32) -> vc.f32:
    return vc.max(a, b)


@vd.reduce.reduce(-(1 << 31), axes=[1])
def _max_i32(a: vc.i32, b: vc.i32) -> vc.i32:
    return vc.max(a, b)


_REDUCERS = {("add", "float32"): _add_f32, ("max", "float32"): _max_f32, ("max", "int32"): _max_i32,
             ("add", "complex64"): _magnitude_rows}


def _inputs(case, seed):
    """The case's input tensors, a dict."""
    g = _gen(seed)
    kind = case["kind"]
    if kind == "roundtrip":
        return {"x": _crandn((case["rows"], case["n"]), g)}
    if kind == "fft":
        shape = (case["outer"], case["n"]) + ((case["inner"],) if case["inner"] > 1 else ())
        return {"x": _crandn(shape, g, _DTYPES[case["dtype"]])}
    if kind == "half2":
        return {"x": _half_input(case, seed)}
    if kind == "rfft2":
        return {"x": torch.randn((case["images"], case["h"], case["w"]), generator=g, device="cuda")}
    if kind == "convolve2dr":
        return {"x": torch.rand((case["images"], case["h"], case["w"]), generator=g, device="cuda") * 2 - 1}
    if kind == "conv_train":
        shape = (case["d"], case["h"], case["w"])
        return {"x": _crandn(shape, g), "khat": _crandn(shape, g) * 0.1,
                "w": torch.rand(shape, generator=g, device="cuda")}
    if kind == "uneven":
        return {"x": _crandn((_uneven_items(case)[1],), g)}
    if kind == "padded":
        phase = torch.rand((case["outer"], case["cols"], case["inner"]), generator=g, device="cuda") * (2 * math.pi)
        # a spectrum of unit modulus: repeated passes over one buffer stay in range
        return {"x": _crandn((case["outer"], case["rows"], case["inner"]), g),
                "spectrum": torch.polar(torch.ones_like(phase), phase)}
    shape = (case["rows"], case["n"])
    if case["type"] == "complex64":
        return {"x": _crandn(shape, g)}
    if case["type"] == "int32":
        return {"x": torch.randint(-(1 << 31), (1 << 31) - 1, shape, generator=g, device="cuda", dtype=torch.int32)}
    return {"x": torch.randn(shape, generator=g, device="cuda")}


# ---------------------------------------------------------------------------
# the cases' interface
# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    t = _inputs(case, seed)
    s = {"case": case, **t}
    if kind in ("roundtrip", "padded"):
        s["buf"] = vd.from_cuda_array(t["x"], var_type=vd.complex64)
    if kind == "half2":
        b = vd.Buffer((case["images"], case["h"], case["w"]), _HALF[case["type"]])
        b.tensor.copy_(t["x"])
        del s["x"]
        s["buf"] = b
    if kind == "convolve2dr":
        shape = (case["images"], case["h"], case["w"])
        b = vd.RFFTBuffer(shape)
        real = torch.view_as_real(b.tensor).reshape(shape[0], shape[1], -1)
        real.zero_()
        real[..., : case["w"]] = t["x"]
        spec = _gaussian_spectrum(case["h"], case["w"])
        kb = vd.RFFTBuffer((1 if case["broadcast"] else case["images"],) + shape[1:])
        kb.tensor.copy_(spec.expand(kb.tensor.shape))
        s.update(buf=b, ker=kb, image=real[..., : case["w"]])
        del s["x"]
    if kind == "uneven":
        items, _ = _uneven_items(case)
        s["fwd"], s["inv"] = BatchPlan(items), BatchPlan(items, inverse=True)
        s["ws"] = s["fwd"].make_workspace()
    if kind == "padded":
        s["maps"] = _padded_maps(case)
        s["kbuf"] = vd.from_cuda_array(t["spectrum"], var_type=vd.complex64)
    if kind == "reduce":
        vt = {"float32": vd.float32, "int32": vd.int32, "complex64": vd.complex64}[case["type"]]
        s["buf"] = vd.from_cuda_array(t["x"], var_type=vt)
        s["reducer"] = _REDUCERS[(case["op"], case["type"])]
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "roundtrip":
        vd.fft.fft(s["buf"])
        vd.fft.ifft(s["buf"])
        total = _magnitude_sum(s["buf"])
        return [s["x"], total.tensor.reshape(-1)[:1]]
    if kind == "fft":
        f = vd.torch_fft.ifft if case["inverse"] else vd.torch_fft.fft
        return f(s["x"], dim=1)
    if kind == "half2":
        vd.fft.fft2(s["buf"])
        vd.fft.ifft2(s["buf"])
        return s["buf"].tensor
    if kind == "rfft2":
        y = vd.torch_fft.rfft2(s["x"])
        return [y, vd.torch_fft.irfft2(y, s=(case["h"], case["w"]))]
    if kind == "convolve2dr":
        vd.fft.convolve2DR(s["buf"], s["ker"])
        return s["image"]
    if kind == "conv_train":
        x, k = s["x"].detach().requires_grad_(True), s["khat"].detach().requires_grad_(True)
        loss = ag.conv_weighted_sqnorm(x, k, s["w"])
        loss.backward()
        return [loss.detach(), x.grad, k.grad]
    if kind == "uneven":
        s["fwd"](s["x"], s["ws"])
        s["inv"](s["x"], s["ws"])
        return s["x"]
    if kind == "padded":
        im, om, km = s["maps"]
        vd.fft.convolve(s["buf"], s["buf"], s["kbuf"], buffer_shape=(case["outer"], case["cols"], case["inner"]),
                        axis=1, input_map=im, output_map=om, kernel_map=km)
        return s["x"]
    return s["reducer"](s["buf"]).tensor.reshape(-1)[: case["rows"]]


def exact(case, seed):
    kind = case["kind"]
    t = _inputs(case, seed)
    x = t["x"]
    if kind == "roundtrip":
        y = x.to(torch.complex128)
        return [y, y.abs().sum().reshape(1)]
    if kind == "fft":
        f = torch.fft.ifft if case["inverse"] else torch.fft.fft
        return f(x.to(torch.complex128), dim=1)
    if kind == "half2":
        return x.double()
    if kind == "rfft2":
        x = x.double()
        return [torch.fft.rfft2(x), x]
    if kind == "convolve2dr":
        k = _gaussian_spectrum(case["h"], case["w"]).to(torch.complex128)
        return torch.fft.irfft2(torch.fft.rfft2(x.double()) * k.conj(), s=(case["h"], case["w"]))
    if kind == "conv_train":
        xa = x.to(torch.complex128).requires_grad_(True)
        ka = t["khat"].to(torch.complex128).requires_grad_(True)
        y = torch.fft.ifftn(torch.fft.fftn(xa) * ka.conj())
        loss = (t["w"].double() * (y.real ** 2 + y.imag ** 2)).sum()
        loss.backward()
        return [loss.detach(), xa.grad.resolve_conj(), ka.grad.resolve_conj()]
    if kind == "uneven":
        return x.to(torch.complex128)
    if kind == "padded":
        y = x.to(torch.complex128)
        c = case["cols"]
        y[:, :c] = torch.fft.ifft(torch.fft.fft(y[:, :c], dim=1) * t["spectrum"].to(torch.complex128).conj(), dim=1)
        return y
    if case["type"] == "complex64":
        return x.to(torch.complex128).abs().sum(dim=1)
    if case["op"] == "max":
        return x.amax(dim=1) if case["type"] == "int32" else x.double().amax(dim=1)
    return x.double().sum(dim=1)


def work(case):
    kind = case["kind"]

    def fft_flops(points, length):
        return 5.0 * points * math.log2(max(2, length))

    if kind == "roundtrip":
        p = case["rows"] * case["n"]
        return {"bytes": 16 * p, "flops": 2 * fft_flops(p, case["n"]) + 4 * p}
    if kind == "fft":
        p = case["outer"] * case["n"] * case["inner"]
        return {"bytes": (32 if case["dtype"] == "complex128" else 16) * p, "flops": fft_flops(p, case["n"])}
    if kind == "half2":
        p = case["images"] * case["h"] * case["w"]
        return {"bytes": 8 * p, "flops": 2 * fft_flops(p, case["h"] * case["w"])}
    if kind == "rfft2":
        p = case["images"] * case["h"] * case["w"]
        half = case["images"] * case["h"] * (case["w"] // 2 + 1)
        return {"bytes": 8 * p + 8 * half, "flops": fft_flops(p, case["h"] * case["w"])}
    if kind == "convolve2dr":
        p = case["images"] * case["h"] * case["w"]
        ker = (1 if case["broadcast"] else case["images"]) * case["h"] * (case["w"] // 2 + 1)
        return {"bytes": 8 * p + 8 * ker, "flops": fft_flops(p, case["h"] * case["w"]) + 3 * p}
    if kind == "conv_train":
        p = case["d"] * case["h"] * case["w"]
        return {"bytes": 36 * p, "flops": 4 * fft_flops(p, p) + 24 * p}
    if kind == "uneven":
        items, p = _uneven_items(case)
        return {"bytes": 16 * p, "flops": 2 * sum(fft_flops(n * c, n) for _, n, c in items)}
    if kind == "padded":
        p = case["outer"] * case["cols"] * case["inner"]
        return {"bytes": 24 * p, "flops": 2 * fft_flops(p, case["cols"]) + 6 * p}
    p = case["rows"] * case["n"]
    return {"bytes": (8 if case["type"] == "complex64" else 4) * p + 4 * case["rows"],
            "flops": (4 if case["type"] == "complex64" else 1) * p}
