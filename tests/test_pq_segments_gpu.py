"""Linear RgbaF16's mismatch from the PQ segment table: the pixels the table cannot decide take the exact level. Contents
that stress the choice, against the oracle: flat pairs whose level difference lies within the table's tolerance of an
integer (every region pixel undecided), and frames of extreme halves (0, subnormal, negative, past the white level)."""
import numpy as np
import pytest

import oracle
from test_formats_gpu import check_frames

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


def near_integer_pair(side, white, tol=0.003):
    """two halves whose PQ level difference is an integer from above (side 1) or below (-1), within tol"""
    halves = np.arange(0x2800, 0x4900, 7, dtype=np.uint16).view(np.float16).astype(np.float32)
    lv = np.array([oracle.pq255(v, white) for v in halves])
    for i in range(0, len(lv), 3):
        d = np.abs(lv - lv[i])
        f = d - np.rint(d)
        ok = (np.rint(d) >= 3) & (np.rint(d) <= 9) & (np.abs(f) <= tol) & (f * side > 0)
        if ok.any():
            return halves[i], halves[int(np.argmax(ok))]
    raise AssertionError("no pair found")


@pytest.mark.parametrize("name,white", [("f16_linear", 80.0), ("f16_linear_203", 203.0)])
@pytest.mark.parametrize("side", [1, -1])
def test_undecided_everywhere(name, white, side):
    va, vc = near_integer_pair(side, white)
    a, c = (np.full((70, 131, 4), v, np.float16) for v in (va, vc))
    a[..., 3] = c[..., 3] = 1.0
    s = oracle.Settings(sceneCutSad=250.0, trustLow=2.0, trustHigh=10.0, globalFallback=1.0)
    check_frames(name, a, c, [0.5, 0.25], settings=s)


@pytest.mark.parametrize("fs", [1, 2])
def test_extreme_halves(fs):
    rng = np.random.default_rng(12)
    pool = np.array([0x0000, 0x8000, 0x0001, 0x03FF, 0x0400, 0xBC00, 0x3C00, 0x57D0, 0x57D1, 0x5640, 0x7BFF, 0x1400, 0x2E66],
                    np.uint16)
    base = pool[rng.integers(0, len(pool), (24, 40, 3))]
    a = np.full((96, 160, 4), 0x3C00, np.uint16)
    a[..., :3] = np.repeat(np.repeat(base, 4, 0), 4, 1)
    c = np.roll(a, (3, -2), (0, 1))
    s = oracle.Settings(sceneCutSad=250.0, globalFallback=1.0, flowScale=fs)
    check_frames("f16_linear", a.view(np.float16), c.view(np.float16), [0.5, float(np.float32(1 / 3))], settings=s)
