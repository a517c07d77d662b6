"""The bound that the linear RgbaF16 synthesis' integer mismatch rests on: over every float y in [0, 1] the PQ segment
table (csrc/fg_formats.cu pqApprox) is within kPqTol / 2 of the level the series gives (fmtPq255), roundings included.
The table is the library's own; the series is restated here in single float32 operations and first checked, bit for bit,
against the library's level of every half value."""
import ctypes
import os
import re

import pytest
import torch

import build
import framegen as fg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def built():
    build.build()
    return fg.lib()


def f32(x):
    return torch.tensor(x, dtype=torch.float32, device="cuda")


def log2(x):
    b = x.view(torch.int32)
    e = ((b >> 23) & 255) - 127
    m = ((b & 0x7FFFFF) | 0x3F800000).view(torch.float32)
    big = m > f32(float.fromhex("0x1.6a09e6p+0"))
    m = torch.where(big, m * 0.5, m)
    e = torch.where(big, e + 1, e)
    s = (m - 1.0) / (m + 1.0)
    z = s * s
    p = f32(float.fromhex("0x1.484b14p-2"))
    for c in ("0x1.a61762p-2", "0x1.2776c6p-1", "0x1.ec709ep-1", "0x1.715476p+1"):
        p = p * z
        p = p + f32(float.fromhex(c))
    q = s * p
    return e.float() + q


def exp2(x):
    n = torch.floor(x)
    g = x - n
    g = g - 0.5
    p = f32(float.fromhex("0x1.ffcbfcp-17"))
    for c in ("0x1.430912p-13", "0x1.5d87fep-10", "0x1.3b2ab6p-7", "0x1.c6b08ep-5", "0x1.ebfbe0p-3", "0x1.62e430p-1", "0x1p+0"):
        p = p * g
        p = p + f32(float.fromhex(c))
    p = p * f32(float.fromhex("0x1.6a09e6p+0"))
    r = p * ((n.clamp(-126, 127).int() + 127) << 23).view(torch.float32)
    return torch.where(x >= -126.0, r, torch.zeros_like(r))


def level(y):
    """fmtPq255 at y = v kWhite, y in [0, 1]"""
    tiny = float.fromhex("0x1p-126")
    p = torch.where(y >= tiny, exp2(f32(0.1593017578125) * log2(y.clamp(min=tiny))), torch.zeros_like(y))
    num = f32(18.8515625) * p
    num = num + 0.8359375
    den = f32(18.6875) * p
    den = den + 1.0
    l = log2(num / den)
    return exp2(f32(78.84375) * l) * 255.0


def source(name):
    src = open(os.path.join(build.HERE, "csrc", "fg_formats.cu")).read()
    return re.search(rf"\b{name} = ([^;,]+)[;,]", src).group(1)


@pytest.mark.parametrize("nits", [80.0, 203.0, 10000.0])
def test_the_restated_series(built, nits):
    k = f32(nits) / f32(10000.0)
    tab = torch.empty(65536, dtype=torch.float32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    f = getattr(built, "_ZN3fgk13launchPqTableEPffP11CUstream_st")
    assert f(ctypes.c_void_p(tab.data_ptr()), ctypes.c_float(float(k)), ctypes.c_void_p(stream)) == 0
    h = torch.arange(65536, dtype=torch.int32, device="cuda").to(torch.int16).view(torch.float16).float()
    y = torch.nan_to_num(h * k, nan=0.0, posinf=1.0, neginf=0.0).clamp(0.0, 1.0)
    assert torch.equal(level(y).view(torch.int32), tab.view(torch.int32))


def test_every_float(built):
    tol, shift, octaves = float(source("kPqTol").rstrip("f")), int(source("kPqShift")), int(source("kPqOctaves"))
    segs = (octaves << (23 - shift)) + 1
    base = (127 - octaves) << 23
    seg = torch.empty((segs, 2), dtype=torch.float32, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    f = getattr(built, "_ZN3fgk16launchPqSegmentsEP6float2P11CUstream_st")
    assert f(ctypes.c_void_p(seg.data_ptr()), ctypes.c_void_p(stream)) == 0
    worst, step = 0.0, 1 << 25
    for b0 in range(0, 0x3F800001, step):
        bits = torch.arange(b0, min(b0 + step, 0x3F800001), dtype=torch.int32, device="cuda")
        y = bits.view(torch.float32)
        t = seg[((bits.clamp(min=base) - base) >> shift).long()]
        a = (y.double() * t[:, 0].double() + t[:, 1].double()).float()   # one rounding, as the kernel's fused multiply-add
        worst = max(worst, float((a.double() - level(y).double()).abs().max()))
    # two levels' errors and the roundings of their two differences and of m -+ kPqTol, half an ulp below 256 each
    assert 2 * worst + 4 * 2.0 ** -17 < tol, worst
    assert worst > tol / 4   # (the series and the table were compared at all)
