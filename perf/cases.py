"""Workloads of the batched 1D transform library, for timing its device path.

Each case is a dict of plain values; ``family`` says which kind of call it is.
``prepare`` builds the plans and the device buffers a program keeps between
calls, ``run`` enqueues one pass on torch's current stream, ``work`` gives the
bytes and operations a pass cannot do without and ``exact`` the same outputs
in 64 bits from torch's own FFT.  Data are uniform in [-1, 1) (fixed point:
uniform in [-2^(B-2), 2^(B-2))), made from the seed alone.
"""
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "perf-libs-fft_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import plfft  # noqa: E402

_DCT_DST = {"dct2": 1, "dct3": 2, "dct4": 3, "dst2": 5, "dst3": 6, "dst4": 7}


def listed():
    return [
        # a handful of short transforms per call: a streaming filter or a
        # per-symbol demodulator, where the launch is the cost
        dict(name="c2c_small_n256_b16", family="c2c", n=256, batch=16, direction=-1),
        # the library's headline batch (bench.py's default workload)
        dict(name="c2c_n1024_b4096", family="c2c", n=1024, batch=4096, direction=-1),
        # decimal lengths: sample rates, OFDM grids, images that are no power of two
        dict(name="c2c_n1000_b16384", family="c2c", n=1000, batch=16384, direction=-1),
        # lengths given by the data and not chosen: a prime (Rader) and a
        # length with a large prime factor (Bluestein)
        dict(name="c2c_n1009_n1031_b8192", family="awkward", n=1009, n_b=1031, batch=8192, direction=-1),
        # long transforms (spectrometers, convolution by FFT), beyond one SM
        dict(name="c2c_n1m_b64", family="c2c", n=1 << 20, batch=64, direction=-1),
        # real signal to spectrum and back, normalised: spectral filtering
        dict(name="r2c_c2r_n4096_b8192", family="real", n=4096, batch=8192),
        # the same at a decimal length
        dict(name="r2c_c2r_n1000_b16384", family="real", n=1000, batch=16384),
        # DCT-II of frames: audio and image coding
        dict(name="dct2_n1024_b4096", family="r2r", kind="dct2", n=1024, batch=4096),
        # fixed-point frames of a DSP front end
        dict(name="q15_n256_b16384", family="fixed", kind="c2c", bits=16, n=256, batch=16384, direction=-1),
        # thousands of transforms of uneven length in one grouped execution
        dict(name="grouped_4000", family="grouped", count=4000, low=16, high=65536, draw_seed=2026),
        # double precision 2-D transform: unit-stride rows, then strided columns
        dict(name="fft2d_fp64_2048x2048", family="fft2d", rows=2048, cols=2048, direction=-1),
        # half-precision storage, forward and back (normalised)
        dict(name="fp16_n1024_b4096", family="half", n=1024, batch=4096),
    ]


# ---------------------------------------------------------------------------
# lengths
# ---------------------------------------------------------------------------
def _smooth(n, top):
    for p in (2, 3, 5, 7, 11, 13):
        while p <= top and n % p == 0:
            n //= p
    return n == 1


def _prime(n):
    return n > 1 and all(n % d for d in range(2, int(math.isqrt(n)) + 1))


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _smooth_len(rng, lo, hi, top=13):
    n = hi + 1
    while n > hi:
        n = _log_int(rng, lo, hi)
        while not _smooth(n, top):
            n += 1
    return n


def group_lengths(count, low, high, seed):
    """Log-uniform lengths: 60% powers of two, 20% 7-smooth, 10% primes,
    10% with a large prime factor; sorted."""
    rng = random.Random(seed)
    out = []
    for _ in range(count):
        u = rng.random()
        n = _log_int(rng, low, high)
        if u < 0.6:
            n = min(1 << round(math.log2(n)), high)
        elif u < 0.8:
            while not _smooth(n, 7):
                n -= 1
        elif u < 0.9:
            while not _prime(n):
                n -= 1
        else:
            while _smooth(n, 13) or _prime(n):
                n += 1
            n = n if n <= high else 4 * 17
        out.append(max(1, n))
    return sorted(out)


def draw(rng):
    family = rng.choice(["pow2", "smooth", "awkward", "long", "real", "r2r", "fixed", "grouped", "fft2d", "half"])
    direction = rng.choice([-1, 1])

    def batch(n, top):
        # at least one member, in all 2^10 .. `top` elements, odd counts too
        total = math.exp(rng.uniform(math.log(1 << 10), math.log(top)))
        return max(1, int(total / n))

    if family == "pow2":
        n = 1 << rng.randint(4, 13)
        return dict(family="c2c", n=n, batch=batch(n, 1 << 24), direction=direction)
    if family == "smooth":
        n = _smooth_len(rng, 12, 16384)
        return dict(family="c2c", n=n, batch=batch(n, 1 << 24), direction=direction)
    if family == "awkward":
        n = _log_int(rng, 17, 4000)
        while not _prime(n):
            n += 1
        m = _log_int(rng, 17, 4000)
        while _smooth(m, 13) or _prime(m):
            m += 1
        return dict(family="awkward", n=n, n_b=m, batch=batch(max(n, m), 1 << 23), direction=direction)
    if family == "long":
        n = 1 << rng.randint(14, 20) if rng.random() < 0.6 else _smooth_len(rng, 16385, 1 << 20, 7)
        return dict(family="c2c", n=n, batch=batch(n, 1 << 26), direction=direction)
    if family == "real":
        n = 1 << rng.randint(6, 14) if rng.random() < 0.4 else _smooth_len(rng, 24, 8192, 13)
        return dict(family="real", n=n, batch=batch(n, 1 << 24))
    if family == "r2r":
        n = 1 << rng.randint(6, 13) if rng.random() < 0.6 else _smooth_len(rng, 24, 4096, 7)
        return dict(family="r2r", kind=rng.choice(sorted(_DCT_DST)), n=n, batch=batch(n, 1 << 24))
    if family == "fixed":
        n = 1 << rng.randint(3, 12)
        return dict(family="fixed", kind=rng.choice(["c2c", "r2c", "c2r"]), bits=rng.choice([16, 16, 8]), n=n,
                    batch=batch(n, 1 << 22), direction=direction)
    if family == "grouped":
        return dict(family="grouped", count=_log_int(rng, 64, 3000), low=16, high=65536,
                    draw_seed=rng.randrange(1 << 30))
    if family == "fft2d":
        return dict(family="fft2d", rows=_smooth_len(rng, 64, 3000, 7), cols=_smooth_len(rng, 64, 3000, 7),
                    direction=direction)
    n = 1 << rng.randint(6, 13) if rng.random() < 0.6 else _smooth_len(rng, 24, 8192, 7)
    return dict(family="half", n=n, batch=batch(n, 1 << 23))


# ---------------------------------------------------------------------------
# inputs and plans
# ---------------------------------------------------------------------------
def _uniform(shape, seed, dtype):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(shape, generator=g, device="cuda", dtype=dtype).mul_(2).sub_(1)


def _fixed_types(case):
    """element type, scalars in and scalars out of one member"""
    n, h = case["n"], case["n"] // 2 + 1
    dt = torch.int16 if case["bits"] == 16 else torch.int8
    return {"c2c": (dt, 2 * n, 2 * n), "r2c": (dt, n, 2 * h), "c2r": (dt, 2 * h, n)}[case["kind"]]


def _inputs(case, seed):
    f = case["family"]
    if f == "c2c":
        return _uniform((case["batch"], case["n"], 2), seed, torch.float32)
    if f == "awkward":
        return (_uniform((case["batch"], case["n"], 2), seed, torch.float32),
                _uniform((case["batch"], case["n_b"], 2), seed + 1, torch.float32))
    if f in ("real", "r2r"):
        return _uniform((case["batch"], case["n"]), seed, torch.float32)
    if f == "fixed":
        dt, nin, _ = _fixed_types(case)
        top = 1 << (case["bits"] - 2)
        g = torch.Generator(device="cuda").manual_seed(seed)
        return torch.randint(-top, top, (case["batch"], nin), generator=g, device="cuda", dtype=torch.int32).to(dt)
    if f == "grouped":
        total = sum(group_lengths(case["count"], case["low"], case["high"], case["draw_seed"]))
        return _uniform((total, 2), seed, torch.float32)
    if f == "fft2d":
        return _uniform((case["rows"], case["cols"], 2), seed, torch.float64)
    return _uniform((case["batch"], case["n"], 2), seed, torch.float32).to(torch.float16)


def prepare(case, seed):
    f = case["family"]
    x = _inputs(case, seed)
    s = {"family": f, "x": x}
    if f == "c2c":
        s["plan"] = plfft.make_plan("c2c", case["n"], case["batch"], direction=case["direction"])
        s["y"] = torch.empty_like(x)
    elif f == "awkward":
        s["plans"] = [plfft.make_plan("c2c", n, case["batch"], direction=case["direction"])
                      for n in (case["n"], case["n_b"])]
        s["y"] = [torch.empty_like(t) for t in x]
    elif f == "real":
        n, b = case["n"], case["batch"]
        s["fwd"] = plfft.make_plan("r2c", n, b)
        s["inv"] = plfft.make_plan("c2r", n, b, scale=1.0 / n)
        s["spec"] = torch.empty((b, n // 2 + 1, 2), device="cuda", dtype=torch.float32)
        s["y"] = torch.empty_like(x)
    elif f == "r2r":
        s["plan"] = plfft.make_plan("r2r", case["n"], case["batch"], r2r_kind=_DCT_DST[case["kind"]])
        s["y"] = torch.empty_like(x)
    elif f == "fixed":
        dt, _, nout = _fixed_types(case)
        s["plan"] = plfft.make_plan(case["kind"], case["n"], case["batch"], direction=case["direction"],
                                    data_type=plfft.DataType.Q15 if case["bits"] == 16 else plfft.DataType.Q7)
        s["y"] = torch.empty((case["batch"], nout), device="cuda", dtype=dt)
    elif f == "grouped":
        lengths = np.array(group_lengths(case["count"], case["low"], case["high"], case["draw_seed"]), np.int64)
        off = np.concatenate([[0], np.cumsum(lengths)[:-1]])
        s["group"] = plfft.Group(lengths, off, off)
        s["y"] = torch.empty_like(x)
    elif f == "fft2d":
        r, c = case["rows"], case["cols"]
        s["row_plan"] = plfft.make_plan("c2c", c, r, direction=case["direction"], data_type=plfft.DataType.FP64)
        s["col_plan"] = plfft.make_plan("c2c", r, c, istride=c, idist=1, ostride=c, odist=1,
                                        direction=case["direction"], data_type=plfft.DataType.FP64)
        s["mid"] = torch.empty_like(x)
        s["y"] = torch.empty_like(x)
    else:
        n, b = case["n"], case["batch"]
        s["fwd"] = plfft.make_plan("c2c", n, b, direction=-1, data_type=plfft.DataType.FP16, scale=1.0 / math.sqrt(n))
        s["inv"] = plfft.make_plan("c2c", n, b, direction=1, data_type=plfft.DataType.FP16, scale=1.0 / math.sqrt(n))
        s["spec"] = torch.empty_like(x)
        s["y"] = torch.empty_like(x)
    return s


def run(s):
    st = torch.cuda.current_stream().cuda_stream
    f, x, y = s["family"], s["x"], s["y"]
    if f in ("c2c", "r2r", "fixed"):
        s["plan"].execute_async(x.data_ptr(), y.data_ptr(), stream=st)
        return y
    if f == "awkward":
        for plan, a, b in zip(s["plans"], x, y):
            plan.execute_async(a.data_ptr(), b.data_ptr(), stream=st)
        return y
    if f in ("real", "half"):
        s["fwd"].execute_async(x.data_ptr(), s["spec"].data_ptr(), stream=st)
        s["inv"].execute_async(s["spec"].data_ptr(), y.data_ptr(), stream=st)
        return [s["spec"], y]
    if f == "grouped":
        s["group"].execute_async(x.data_ptr(), y.data_ptr(), stream=st)
        return y
    s["row_plan"].execute_async(x.data_ptr(), s["mid"].data_ptr(), stream=st)
    s["col_plan"].execute_async(s["mid"].data_ptr(), y.data_ptr(), stream=st)
    return [s["mid"], y]


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _c2c_flops(n):
    return 5.0 * n * math.log2(max(n, 2))


def work(case):
    f = case["family"]
    if f == "grouped":
        lengths = group_lengths(case["count"], case["low"], case["high"], case["draw_seed"])
        return {"bytes": 16 * sum(lengths), "flops": sum(_c2c_flops(n) for n in lengths)}
    if f == "fft2d":
        r, c = case["rows"], case["cols"]
        # each of the two transforms is a call of its own: 32 bytes an element
        return {"bytes": 64 * r * c, "flops": r * _c2c_flops(c) + c * _c2c_flops(r)}
    n, b = case["n"], case["batch"]
    if f == "c2c":
        return {"bytes": 16 * n * b, "flops": b * _c2c_flops(n)}
    if f == "awkward":
        return {"bytes": 16 * b * (n + case["n_b"]), "flops": b * (_c2c_flops(n) + _c2c_flops(case["n_b"]))}
    if f == "real":
        return {"bytes": 2 * b * (4 * n + 8 * (n // 2 + 1)), "flops": b * _c2c_flops(n)}
    if f == "r2r":
        return {"bytes": 8 * n * b, "flops": 0.5 * b * _c2c_flops(n)}
    if f == "fixed":
        _, nin, nout = _fixed_types(case)
        ops = _c2c_flops(n) * (1.0 if case["kind"] == "c2c" else 0.5)
        return {"bytes": b * (nin + nout) * case["bits"] // 8, "flops": b * ops}
    return {"bytes": 2 * 8 * n * b, "flops": 2 * b * _c2c_flops(n)}


# ---------------------------------------------------------------------------
# the same outputs in 64 bits
# ---------------------------------------------------------------------------
def _fft(x, direction):
    """Unnormalised transform of the last axis, complex128."""
    n = x.shape[-1]
    return torch.fft.fft(x) if direction < 0 else torch.fft.ifft(x) * n


def _cplx(x):
    return torch.view_as_complex(x.to(torch.float64).contiguous())


def _chunked(fn, x, rows):
    return torch.cat([fn(x[i:i + rows]) for i in range(0, x.shape[0], rows)])


def _c2c_exact(x, direction, scale=1.0):
    rows = max(1, (1 << 24) // x.shape[1])
    return _chunked(lambda t: torch.view_as_real(_fft(_cplx(t), direction) * scale), x, rows)


def _dct_dst(kind, x):
    """FFTW-convention DCT / DST II, III, IV through a complex transform of 2n points."""
    n = x.shape[1]
    x = x.to(torch.float64)
    j = torch.arange(n, device=x.device, dtype=torch.float64)

    def phase(t):
        return torch.polar(torch.ones_like(t), -math.pi * t)

    def padded(z, at=0):
        out = torch.zeros((z.shape[0], 2 * n), device=z.device, dtype=torch.complex128)
        out[:, at:at + n] = z
        return torch.fft.fft(out)

    if kind == "dct2":
        return 2 * (phase(j / (2 * n)) * padded(x)[:, :n]).real
    if kind == "dst2":
        return -2 * (phase((j + 1) / (2 * n)) * padded(x)[:, 1:n + 1]).imag
    if kind == "dct3":
        w = torch.ones_like(j)
        w[0] = 0.5
        return 2 * padded(x * w * phase(j / (2 * n)))[:, :n].real
    if kind == "dst3":
        w = torch.ones_like(j)
        w[-1] = 0.5
        return -2 * padded(x * w * phase((j + 1) / (2 * n)), 1)[:, :n].imag
    z = phase((2 * j + 1) / (4 * n)) * padded(x * phase(j / (2 * n)))[:, :n]
    return 2 * z.real if kind == "dct4" else -2 * z.imag


def exact(case, seed):
    f = case["family"]
    if f == "fixed":
        return None  # whole numbers
    x = _inputs(case, seed)
    if f == "c2c":
        return _c2c_exact(x, case["direction"])
    if f == "awkward":
        return [_c2c_exact(t, case["direction"]) for t in x]
    if f == "real":
        # the inverse is of the spectrum as written: it is x up to rounding
        rows = max(1, (1 << 24) // x.shape[1])
        spec = _chunked(lambda t: torch.view_as_real(torch.fft.rfft(t.to(torch.float64))), x, rows)
        return [spec, x.to(torch.float64)]
    if f == "r2r":
        rows = max(1, (1 << 24) // (2 * x.shape[1]))
        return _chunked(lambda t: _dct_dst(case["kind"], t), x, rows)
    if f == "grouped":
        lengths = group_lengths(case["count"], case["low"], case["high"], case["draw_seed"])
        out = torch.empty(x.shape, device=x.device, dtype=torch.float64)
        at = 0
        i = 0
        while i < len(lengths):  # sorted: equal lengths lie side by side
            n = lengths[i]
            k = i
            while k < len(lengths) and lengths[k] == n:
                k += 1
            span = n * (k - i)
            z = _cplx(x[at:at + span].reshape(k - i, n, 2))
            out[at:at + span] = torch.view_as_real(_fft(z, -1)).reshape(span, 2)
            at += span
            i = k
        return out
    if f == "fft2d":
        z = _fft(_cplx(x), case["direction"])
        return [torch.view_as_real(z), torch.view_as_real(_fft(z.t(), case["direction"]).t().contiguous())]
    # FP16: the spectrum is rounded to 16 bits before the inverse
    root = 1.0 / math.sqrt(case["n"])
    return [_c2c_exact(x, -1, root), x.to(torch.float64)]
