"""Mixed-radix tile engine: C2C in FP32, FP64 and FP16 and the one-pass real
transforms, at the lengths where tiles, stages and layouts change."""
import numpy as np
import pytest

import oracle
import plfft
from helpers import gather, seeded_complex, seeded_real, span, to_dev

pytestmark = pytest.mark.gpu

# one stage (2, 13, 16), two, three, four; primes of the radix menu; a tile of
# many transforms and of one; the longest two- and one-buffer tiles (7128, 8788);
# 8000 and beyond: the tile kernel or two passes
LENGTHS = [2, 13, 16, 18, 121, 169, 210, 360, 1000, 1001, 1155, 2187, 4000, 6561, 7128, 8000, 8788, 12000, 14336]


@pytest.mark.parametrize("n", LENGTHS)
@pytest.mark.parametrize("direction", [-1, 1])
def test_c2c_fp32(n, direction):
    import torch

    hm = 37 if n <= 4000 else 3  # a ragged last tile
    # unit stride with padded members, members interleaved, both sides mixed
    for is_, id_, os_, od in [(1, n + 1, 1, n), (hm + 2, 1, hm + 2, 1), (1, n, hm, 1), (hm, 1, 2, 2 * n + 1)]:
        x = seeded_complex(span(hm, id_, n, is_), n)
        y = torch.full((span(hm, od, n, os_),), 7.0, dtype=torch.complex64, device="cuda")
        plan = plfft.make_plan("c2c", n, hm, is_, id_, os_, od, direction=direction, scale=0.5)
        plan.execute(to_dev(x).data_ptr(), y.data_ptr())
        got = y.cpu().numpy()
        ref = 0.5 * oracle.c2c(gather(x, hm, id_, n, is_).astype(np.complex128), direction, method="fft")
        assert oracle.rel_l2(gather(got, hm, od, n, os_), ref) <= oracle.fp32_tol(n), plan.describe()
        touched = np.zeros(got.size, bool)
        touched[(np.arange(hm)[:, None] * od + np.arange(n)[None, :] * os_).ravel()] = True
        assert np.all(got[~touched] == 7.0), "wrote outside the members"


# which of them the engine holds in one pass
@pytest.mark.parametrize("n,buffers", [(4095, "one-buffer"), (6561, ""), (7128, "two-buffers"), (8788, "one-buffer"),
                                       (6720, None), (8000, None), (8190, None)])
def test_c2c_reach(n, buffers):
    d = plfft.make_plan("c2c", n, 37).describe()
    assert d.startswith("(c2c-mix") == (buffers is not None) and (not buffers or buffers in d), d


# members interleaved at an even pitch: two numbers to an aligned 16-byte word,
# an odd last member, the same bases one element further, and in place
@pytest.mark.parametrize("n", [2, 13, 16, 30, 169, 1000, 4095])
@pytest.mark.parametrize("pitch,hm", [(38, 37), (40, 37), (2, 2), (4, 3)])
@pytest.mark.parametrize("offset", [0, 1])
def test_c2c_fp32_pairs(n, pitch, hm, offset):
    import torch

    m = span(hm, 1, n, pitch)
    x = seeded_complex(m + offset, n)
    plan = plfft.make_plan("c2c", n, hm, pitch, 1, pitch, 1, alias=plfft.IoAlias.MAY_ALIAS)
    ref = oracle.c2c(gather(x[offset:], hm, 1, n, pitch).astype(np.complex128), -1, method="fft" if n > 16 else "auto")
    touched = np.zeros(m + offset, bool)
    touched[offset + (np.arange(hm)[:, None] + np.arange(n)[None, :] * pitch).ravel()] = True
    d = to_dev(x)
    for dst in (torch.full((m + offset + 2,), 7.0, dtype=torch.complex64, device="cuda"), d):
        before = dst.cpu().numpy()[: m + offset]
        plan.execute(d.data_ptr() + 8 * offset, dst.data_ptr() + 8 * offset)
        got = dst.cpu().numpy()
        assert oracle.rel_l2(gather(got[offset:], hm, 1, n, pitch), ref) <= oracle.fp32_tol(n), plan.describe()
        assert np.array_equal(got[: m + offset][~touched], before[~touched]), "wrote outside the members"
        assert np.all(got[m + offset:] == 7.0), "wrote behind the members"


# in place with equal layouts, dense and interleaved, several CTAs
@pytest.mark.parametrize("n,hm", [(18, 5001), (1000, 301), (4095, 37), (8788, 5)])
@pytest.mark.parametrize("dense", [True, False])
@pytest.mark.parametrize("kind", ["FP32", "FP64", "FP16"])
def test_c2c_in_place(n, hm, dense, kind):
    if (kind == "FP64" and n == 8788) or (kind == "FP16" and n > 4096):
        n = 7168 if kind == "FP64" else 4000
    s, d = (1, n) if dense else (hm, 1)
    rng = np.random.default_rng(n)
    real = {"FP32": np.float32, "FP64": np.float64, "FP16": np.float16}[kind]
    x = rng.uniform(-1, 1, 2 * n * hm).astype(real)
    plan = plfft.make_plan("c2c", n, hm, s, d, s, d, data_type=plfft.DataType[kind], scale=n**-0.5,
                           alias=plfft.IoAlias.MAY_ALIAS)
    buf = to_dev(x)
    plan.execute(buf.data_ptr(), buf.data_ptr())
    z = gather(x.astype(np.float64).view(np.complex128), hm, d, n, s)
    got = gather(buf.cpu().numpy().astype(np.float64).view(np.complex128), hm, d, n, s)
    tol = {"FP32": oracle.fp32_tol(n), "FP64": 8 * np.log2(n) * 2.0**-53, "FP16": 2.0**-11 + oracle.fp32_tol(n)}[kind]
    assert oracle.rel_l2(got, np.fft.fft(z) * n**-0.5) <= tol, plan.describe()


# lengths of one radix: stored from shared memory, or from 14 points on a dense
# batch as two stages
@pytest.mark.parametrize("n,radices", [(5, "5"), (8, "8"), (12, "12"), (13, "13"), (14, "7x2"), (15, "5x3"), (16, "4x4")])
def test_c2c_short(n, radices):
    import torch

    hm = 1001
    for (s, d), want in [((1, n), radices), ((1, n + 1), radices), ((hm + 1, 1), str(n))]:
        for dt, ct in [(plfft.DataType.FP32, np.complex64), (plfft.DataType.FP64, np.complex128)]:
            x = seeded_complex(span(hm, d, n, s), n).astype(ct)
            y = torch.full((x.size,), 7.0, dtype=to_dev(x).dtype, device="cuda")
            plan = plfft.make_plan("c2c", n, hm, s, d, s, d, data_type=dt)
            assert "radices=%s)" % want in plan.describe(), plan.describe()
            plan.execute(to_dev(x).data_ptr(), y.data_ptr())
            got = y.cpu().numpy()
            ref = oracle.c2c(gather(x, hm, d, n, s).astype(np.complex128), -1)
            assert oracle.rel_l2(gather(got, hm, d, n, s), ref) <= oracle.fp32_tol(n), plan.describe()
            touched = np.zeros(got.size, bool)
            touched[(np.arange(hm)[:, None] * d + np.arange(n)[None, :] * s).ravel()] = True
            assert np.all(got[~touched] == 7.0), "wrote outside the members"


# n <= 4096 (one pass), one-buffer and two-buffer tiles, a two-pass length;
# 2^-53 per rounding, 8 log2 n of them
@pytest.mark.parametrize("n", [2, 13, 64, 143, 1000, 2048, 4096, 5000, 8192, 30000])
@pytest.mark.parametrize("strided", [False, True])
def test_c2c_fp64(n, strided):
    import torch

    hm = 9
    is_, id_ = (hm + 1, 1) if strided else (1, n)
    rng = np.random.default_rng(n)
    m = span(hm, id_, n, is_)
    x = rng.uniform(-1, 1, m) + 1j * rng.uniform(-1, 1, m)
    for direction in (-1, 1):
        plan = plfft.make_plan("c2c", n, hm, is_, id_, is_, id_, direction=direction, data_type=plfft.DataType.FP64)
        y = torch.zeros(m, dtype=torch.complex128, device="cuda")
        plan.execute(to_dev(x).data_ptr(), y.data_ptr())
        xl = torch.from_numpy(gather(x, hm, id_, n, is_))
        ref = (torch.fft.fft(xl) if direction < 0 else torch.fft.ifft(xl) * n).numpy()
        tol = 8 * max(1.0, np.log2(n)) * 2.0**-53
        assert oracle.rel_l2(gather(y.cpu().numpy(), hm, id_, n, is_), ref) <= tol, plan.describe()


# binary16 buffers on 4-byte and on odd 2-byte boundaries, strided and dense:
# one rounding of the output (2^-11) on top of FP32
@pytest.mark.parametrize("n", [2, 16, 64, 100, 128, 512, 1000, 1024, 2048, 4096, 8192])
@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("strided", [False, True])
def test_c2c_fp16(n, offset, strided):
    import torch

    hm = 21
    s, d = (hm, 1) if strided else (1, n)
    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, 2 * n * hm + offset).astype(np.float16)
    y = torch.zeros(x.size, dtype=torch.float16, device="cuda")
    plan = plfft.make_plan("c2c", n, hm, s, d, s, d, data_type=plfft.DataType.FP16, scale=n**-0.5)
    dx = to_dev(x)
    plan.execute(dx.data_ptr() + 2 * offset, y.data_ptr() + 2 * offset)
    z = x[offset:].astype(np.float64).view(np.complex128)
    ref = oracle.c2c(gather(z, hm, d, n, s), -1, method="fft") * n**-0.5
    got = y.cpu().numpy()[offset:].astype(np.float64).view(np.complex128)
    assert oracle.rel_l2(gather(got, hm, d, n, s), ref) <= 2.0**-11 + oracle.fp32_tol(n), plan.describe()


REAL_LENGTHS = [4, 6, 26, 28, 30, 32, 100, 242, 1000, 2002, 4374, 8000, 20000]
R2R = [plfft.R2RKind.DCT_2, plfft.R2RKind.DCT_3, plfft.R2RKind.DCT_4, plfft.R2RKind.DST_2, plfft.R2RKind.DST_3,
       plfft.R2RKind.DST_4, plfft.R2RKind.DHT, plfft.R2RKind.R2HC, plfft.R2RKind.HC2R]


@pytest.mark.parametrize("n", REAL_LENGTHS)
@pytest.mark.parametrize("pad", [0, 1])
def test_r2c_c2r(n, pad):
    import torch

    hm, h = 11, n // 2 + 1
    x = seeded_real(span(hm, n + pad, n, 1), n)
    f = plfft.make_plan("r2c", n, hm, 1, n + pad, 1, h + pad)
    y = torch.full((span(hm, h + pad, h, 1),), 7.0, dtype=torch.complex64, device="cuda")
    f.execute(to_dev(x).data_ptr(), y.data_ptr())
    xl = gather(x, hm, n + pad, n, 1).astype(np.float64)
    spec = gather(y.cpu().numpy(), hm, h + pad, h, 1)
    assert oracle.rel_l2(spec, np.fft.rfft(xl)) <= oracle.fp32_tol(n), f.describe()
    b = plfft.make_plan("c2r", n, hm, 1, h + pad, 1, n + pad, scale=1.0 / n)
    z = torch.full((x.size,), 7.0, dtype=torch.float32, device="cuda")
    b.execute(y.data_ptr(), z.data_ptr())
    got = z.cpu().numpy()
    assert oracle.rel_l2(gather(got, hm, n + pad, n, 1), xl) <= 2 * oracle.fp32_tol(n), b.describe()
    if pad:
        assert np.all(got[np.arange(hm - 1) * (n + 1) + n] == 7.0), "wrote between the members"


@pytest.mark.parametrize("n", [6, 26, 28, 30, 32, 100, 1000, 2002])
@pytest.mark.parametrize("kind", R2R)
def test_r2r(n, kind):
    import torch

    hm = 7
    for pad in (0, 1):
        x = seeded_real(span(hm, n + pad, n, 1), n)
        plan = plfft.make_plan("r2r", n, hm, 1, n + pad, 1, n + pad, r2r_kind=kind)
        y = torch.zeros(x.size, dtype=torch.float32, device="cuda")
        plan.execute(to_dev(x).data_ptr(), y.data_ptr())
        ref = oracle.r2r(gather(x, hm, n + pad, n, 1).astype(np.float64), int(kind))
        got = gather(y.cpu().numpy(), hm, n + pad, n, 1)
        assert oracle.rel_l2(got, ref) <= oracle.fp32_tol(2 * n), plan.describe()


# in-place layouts whose outputs do not lie on their own member's inputs read
# the whole batch before the first write
def test_r2c_in_place_dense():
    import torch

    n, hm = 1000, 5
    h = n // 2 + 1
    x = seeded_real(hm * n, 3)
    buf = torch.zeros(hm * 2 * h, dtype=torch.float32, device="cuda")
    buf[: hm * n] = to_dev(x)
    plan = plfft.make_plan("r2c", n, hm, 1, n, 1, h, alias=plfft.IoAlias.MAY_ALIAS)
    plan.execute(buf.data_ptr(), buf.data_ptr())
    got = buf.cpu().numpy().view(np.complex64).reshape(hm, h)
    assert oracle.rel_l2(got, np.fft.rfft(x.reshape(hm, n).astype(np.float64))) <= oracle.fp32_tol(n), plan.describe()


# In place with outputs away from their own member's inputs: batches of several
# CTAs (and of the two or more members that shared one), whose members a CTA
# may write while another has yet to read them.  Kind, length, members, input
# and output (stride, distance).
MOVED = [("c2c", 360, 16, (1, 360), (16, 1)), ("c2c", 360, 700, (1, 360), (700, 1)),
         ("c2c", 1000, 600, (600, 1), (1, 1001)), ("c2c", 1024, 300, (1, 1024), (300, 1)),
         ("c2c", 1031, 200, (1, 1031), (200, 1)), ("c2c", 12000, 5, (1, 12000), (5, 1)),
         ("r2c", 1000, 1500, (1, 1000), (1, 501)), ("c2r", 1000, 1500, (1, 501), (1, 1000)),
         ("r2c", 4096, 2, (1, 4096), (1, 2049)), ("c2r", 4096, 300, (1, 2049), (1, 4096)),
         ("dct2", 1000, 900, (1, 1000), (1, 1001)), ("dct2", 1024, 900, (1, 1024), (1, 1025))]
MOVED64 = [("c2c", 1000, 300, (1, 1000), (300, 1)), ("c2c", 5000, 40, (1, 5000), (40, 1)),
           ("c2c", 8192, 40, (40, 1), (1, 8192)), ("r2c", 1000, 300, (1, 1000), (1, 501))]


def _moved(kind, n, hm, i, o, dtype, adjoint):
    """one execution in a buffer of its own and one in place, as the output spans' members"""
    import torch

    h = n // 2 + 1
    nin, ci = (h, 2) if kind == "c2r" else (n, 2 if kind == "c2c" else 1)
    nout, co = (h, 2) if kind == "r2c" else (n, 2 if kind == "c2c" else 1)
    args = (hm, i[0], i[1], o[0], o[1])
    kw = dict(data_type=plfft.DataType.FP32 if dtype == torch.float32 else plfft.DataType.FP64)
    if kind == "dct2":
        kw["r2r_kind"] = plfft.R2RKind.DCT_2
    plans = [plfft.make_plan("r2r" if kind == "dct2" else kind, n, *args, alias=a, **kw)
             for a in (plfft.IoAlias.NO_ALIAS, plfft.IoAlias.MAY_ALIAS)]
    if adjoint:
        (nin, ci, i), (nout, co, o) = (nout, co, o), (nin, ci, i)
    si, so = ci * span(hm, i[1], nin, i[0]), co * span(hm, o[1], nout, o[0])
    x = torch.rand(si, generator=torch.Generator().manual_seed(n), dtype=dtype).cuda()
    run = [(p.execute_adjoint if adjoint else p.execute) for p in plans]
    y = torch.zeros(so, dtype=dtype, device="cuda")
    run[0](x.data_ptr(), y.data_ptr())
    buf = torch.zeros(max(si, so), dtype=dtype, device="cuda")
    buf[:si] = x
    run[1](buf.data_ptr(), buf.data_ptr())
    apart = torch.zeros(so, dtype=dtype, device="cuda")  # the same plan on two buffers
    run[1](x.data_ptr(), apart.data_ptr())
    torch.cuda.synchronize()
    ctype = {1: None, 2: np.complex64 if dtype == torch.float32 else np.complex128}[co]
    pick = lambda t: gather(t.cpu().numpy()[:so].view(ctype) if ctype else t.cpu().numpy()[:so], hm, o[1], nout, o[0])
    return pick(y), pick(buf), pick(apart), plans[1]


# the same schedule on the same numbers: equal up to how a CTA's members are
# grouped, one FP32 (FP64) rounding chain
@pytest.mark.parametrize("kind,n,hm,i,o", MOVED)
def test_in_place_moved_members(kind, n, hm, i, o):
    import torch

    ref, got, apart, plan = _moved(kind, n, hm, i, o, torch.float32, False)
    assert oracle.rel_l2(got, ref) <= oracle.fp32_tol(n), plan.describe()
    assert oracle.rel_l2(apart, ref) <= oracle.fp32_tol(n), plan.describe()


@pytest.mark.parametrize("kind,n,hm,i,o", MOVED64)
def test_in_place_moved_members_fp64(kind, n, hm, i, o):
    import torch

    ref, got, apart, plan = _moved(kind, n, hm, i, o, torch.float64, False)
    tol = 8 * np.log2(n) * 2.0**-53
    assert oracle.rel_l2(got, ref) <= tol, plan.describe()
    assert oracle.rel_l2(apart, ref) <= tol, plan.describe()


# the adjoint of such a plan, in place
@pytest.mark.parametrize("kind,n,hm,i,o", MOVED)
def test_adjoint_in_place_moved_members(kind, n, hm, i, o):
    import torch

    ref, got, apart, plan = _moved(kind, n, hm, i, o, torch.float32, True)
    assert oracle.rel_l2(got, ref) <= oracle.fp32_tol(n), plan.describe()
    assert oracle.rel_l2(apart, ref) <= oracle.fp32_tol(n), plan.describe()


# Rader and Bluestein convolutions over the listed lengths between the powers
# of two: the first and last n of each, dense and interleaved, odd batches
@pytest.mark.parametrize("n", [263, 317, 383, 521, 577, 641, 761, 1031, 1151, 1153, 1279, 1531, 1223])
@pytest.mark.parametrize("direction", [-1, 1])
def test_conv_list(n, direction):
    import torch

    for hm in (1, 7):
        for s, d in [(1, n + 1), (hm + 1, 1)]:
            x = seeded_complex(span(hm, d, n, s), n)
            y = torch.zeros(x.size, dtype=torch.complex64, device="cuda")
            plan = plfft.make_plan("c2c", n, hm, s, d, s, d, direction=direction)
            plan.execute(to_dev(x).data_ptr(), y.data_ptr())
            ref = oracle.c2c(gather(x, hm, d, n, s).astype(np.complex128), direction, method="fft")
            got = gather(y.cpu().numpy(), hm, d, n, s)
            assert oracle.rel_l2(got, ref) <= oracle.fp32_tol(n), plan.describe()


# which of them a batch takes: the ends of each rule
@pytest.mark.parametrize("n,hm,listed", [(313, 1024, True), (313, 1025, False), (277, 1025, False), (331, 1024, True),
                                         (331, 1025, False), (383, 1025, True), (521, 148, False), (521, 149, True),
                                         (601, 149, True), (641, 149, True), (563, 3, True), (677, 3, True)])
def test_conv_list_batches(n, hm, listed):
    import torch

    x = seeded_complex(hm * n, n)
    y = torch.zeros(x.size, dtype=torch.complex64, device="cuda")
    plan = plfft.make_plan("c2c", n, hm)
    assert (" list)" in plan.describe()) == listed, plan.describe()
    plan.execute(to_dev(x).data_ptr(), y.data_ptr())
    ref = oracle.c2c(x.reshape(hm, n).astype(np.complex128), -1, method="fft")
    assert oracle.rel_l2(y.cpu().numpy().reshape(hm, n), ref) <= oracle.fp32_tol(n), plan.describe()


# short lengths of 11 and 13 in small batches: direct sums
@pytest.mark.parametrize("n,hm,sums", [(11, 31, False), (11, 32, True), (11, 1000, True), (11, 1001, False), (26, 32, True),
                                       (26, 1001, False), (33, 64, False)])
def test_fp64_short(n, hm, sums):
    import torch

    rng = np.random.default_rng(n)
    x = rng.uniform(-1, 1, n * hm) + 1j * rng.uniform(-1, 1, n * hm)
    y = torch.zeros(n * hm, dtype=torch.complex128, device="cuda")
    plan = plfft.make_plan("c2c", n, hm, data_type=plfft.DataType.FP64)
    assert ("direct sums" in plan.describe()) == sums, plan.describe()
    plan.execute(to_dev(x).data_ptr(), y.data_ptr())
    tol = 8 * np.log2(n) * 2.0**-53
    assert oracle.rel_l2(y.cpu().numpy().reshape(hm, n), np.fft.fft(x.reshape(hm, n))) <= tol, plan.describe()


# small batches inside a real transform: the tile kernel where the engine's
# first two radices are long ones
@pytest.mark.parametrize("n,hm,inner", [(143, 12, "c2c-tile"), (143, 13, "c2c-mix"), (225, 1, "c2c-tile"), (429, 4, "c2c-tile"),
                                        (847, 3, "c2c-mix"), (33, 1, "c2c-mix"), (81, 1, "c2c-mix"), (675, 1, "c2c-mix")])
def test_real_small_batches(n, hm, inner):
    import torch

    h = n // 2 + 1
    x = seeded_real(hm * n, n)
    y = torch.zeros(hm * h, dtype=torch.complex64, device="cuda")
    plan = plfft.make_plan("r2c", n, hm)
    assert inner in plan.describe(), plan.describe()
    plan.execute(to_dev(x).data_ptr(), y.data_ptr())
    ref = np.fft.rfft(x.reshape(hm, n).astype(np.float64))
    assert oracle.rel_l2(y.cpu().numpy().reshape(hm, h), ref) <= oracle.fp32_tol(n), plan.describe()


# two passes over interleaved members: lanes along the members from eight of
# them, a short last chunk (600000 x 23), an odd pitch, in place, one side dense
@pytest.mark.parametrize("n,hm", [(12000, 7), (12000, 8), (13312, 37), (16250, 64), (600000, 23)])
@pytest.mark.parametrize("direction", [-1, 1])
def test_four_step_members(n, hm, direction):
    import torch

    for i, o in [((hm, 1), (hm, 1)), ((hm + 1, 1), (hm + 2, 1)), ((1, n), (hm, 1))]:
        x = torch.randn(span(hm, i[1], n, i[0]), dtype=torch.complex64, device="cuda",
                        generator=torch.Generator("cuda").manual_seed(n))
        plan = plfft.make_plan("c2c", n, hm, *i, *o, direction=direction, alias=plfft.IoAlias.MAY_ALIAS, scale=0.5)
        assert ("member lanes" in plan.describe()) == (hm >= 8 and i[0] > 1), plan.describe()
        y = torch.full((span(hm, o[1], n, o[0]),), 7.0, dtype=torch.complex64, device="cuda")
        xl = torch.as_strided(x, (hm, n), (i[1], i[0])).to(torch.complex128)
        ref = 0.5 * (torch.fft.fft(xl) if direction < 0 else torch.fft.ifft(xl) * n)
        for dst in (y, x) if i == o else (y,):  # the second: in place
            plan.execute(x.data_ptr(), dst.data_ptr())
            got = torch.as_strided(dst, (hm, n), (o[1], o[0]))
            assert float((got - ref).norm() / ref.norm()) <= oracle.fp32_tol(n), plan.describe()
        untouched = torch.ones(y.numel(), dtype=torch.bool, device="cuda")
        torch.as_strided(untouched, (hm, n), (o[1], o[0])).fill_(False)
        assert bool((y[untouched] == 7.0).all()), "wrote outside the members"


# long Rader and Bluestein transforms in place: element 0 of a member is an
# output that other CTAs once read as the input
@pytest.mark.parametrize("n,hm", [(12289, 1), (12289, 9), (40961, 3), (9001, 9)])
def test_long_convolution_in_place(n, hm):
    for s, d in [(1, n), (hm, 1)]:
        x = seeded_complex(n * hm, n)
        plan = plfft.make_plan("c2c", n, hm, s, d, s, d, alias=plfft.IoAlias.MAY_ALIAS)
        buf = to_dev(x)
        plan.execute(buf.data_ptr(), buf.data_ptr())
        ref = np.fft.fft(gather(x, hm, d, n, s).astype(np.complex128))
        assert oracle.rel_l2(gather(buf.cpu().numpy(), hm, d, n, s), ref) <= oracle.fp32_tol(n), plan.describe()
