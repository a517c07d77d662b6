"""The synthesis tiles at the line between interior tiles (no clamps, flowScale 2's fixed row pattern) and the others,
against the oracle, in every format: frames whose middle 58 x 58 tile just is or just is not interior, vectors that take
the taps of a middle tile to the border on each side, odd sizes, the other flow scales."""
import numpy as np
import pytest

import oracle
import workloads
from test_estimate_q_gpu import moved
from test_formats_gpu import check
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu
T13 = float(np.float32(1 / 3))
FORMATS = ["rgb10_argb", "f16_linear", "f16_encoded", "nv12_709_limited", "p010_2020_limited"]
OPEN = oracle.Settings(globalFallback=1.0, sceneCutSad=250.0)


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


def run(fmt, p, c, ts, settings=None):
    if fmt == "rgba8":
        check_against_oracle(p, c, ts, settings)
    else:
        check(fmt, p, c, ts, settings=settings)


@pytest.mark.parametrize("fmt", ["rgba8"] + FORMATS)
@pytest.mark.parametrize("W,H", [(121, 122), (122, 122), (123, 121), (124, 125)])
def test_still_pair_around_the_line(fmt, W, H):
    """a still pair: the middle tile is interior from 122 px on"""
    p, _ = workloads.pan_pair(W, H, seed=W + 3 * H)
    run(fmt, p, p, [0.5, 0.25, T13])


@pytest.mark.parametrize("fmt", ["rgba8"] + FORMATS)
@pytest.mark.parametrize("dx,dy", [(30, 0), (-30, 0), (0, 30), (0, -30), (7, -5)])
def test_moving_pair(fmt, dx, dy):
    p, c = moved(300, 186, dx, dy, 9)
    run(fmt, p, c, [0.25, T13], OPEN)


@pytest.mark.parametrize("fmt", ["rgba8", "nv12_709_limited", "f16_linear"])
@pytest.mark.parametrize("fs", [1, 4])
def test_other_flow_scales(fmt, fs):
    p, c, _ = workloads.flow_pair(240, 200, seed=fs)
    run(fmt, p, c, [0.5, T13], oracle.Settings(flowScale=fs))


@pytest.mark.parametrize("W,H", [(986, 986), (1044, 986)])
def test_one_wave_and_more(W, H):
    """289 and 306 tiles: the 8-bit kernel's forms for grids of at most 2 CTAs per SM and for larger ones"""
    p, c, _ = workloads.flow_pair(W, H, seed=W)
    check_against_oracle(p, c, [0.5, 0.25, T13])
