"""The estimate's integer passes (csrc/fg_estimate_q.cu) against the oracle at the sizes where they can go wrong: flow
fields at and around the pixel-field tile (60 x 32) and its 8-row runs, block counts at both sides of the integer
search's threshold (2048 blocks) on level 0 and level 1, radii 1 and 2, sub-pixel refinement off, vectors whose taps
leave the frame on every side, every flow scale, and the float level 0 that recordTrace makes from the pair planes."""
import numpy as np
import pytest

import oracle
import workloads
from test_formats_gpu import check
from test_parity_gpu import check_against_oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


def moved(W, H, dx, dy, seed):
    """a texture moved by whole pixels, the uncovered part fresh: vectors near the border point out of the frame"""
    rng = np.random.default_rng(seed)
    t = workloads.value_noise(H + 2 * abs(dy), W + 2 * abs(dx), np.random.Generator(np.random.PCG64(seed)))
    y, x = abs(dy), abs(dx)
    f = [workloads._to_rgba(t[y + s * dy:y + s * dy + H, x + s * dx:x + s * dx + W]) for s in (0, -1)]
    f[1][:4, :4, :3] = rng.integers(0, 256, (4, 4, 3))
    return f


@pytest.mark.parametrize("W,H", [(118, 62), (120, 64), (122, 66), (121, 65), (16, 18), (130, 127), (240, 142)])
def test_pixel_field_tile_edges(W, H):
    p, c, _ = workloads.flow_pair(W, H, seed=W * H)
    check_against_oracle(p, c, [0.5])


@pytest.mark.parametrize("dx,dy", [(40, 0), (-40, 0), (0, 28), (0, -28), (-36, 24)])
def test_vectors_leaving_the_frame(dx, dy):
    p, c = moved(246, 150, dx, dy, 5)
    check_against_oracle(p, c, [0.25], oracle.Settings(globalFallback=1.0, sceneCutSad=250.0))


@pytest.mark.parametrize("W,H", [(512, 256), (513, 257), (509, 300)])   # 2048 blocks, 2145, 2432
@pytest.mark.parametrize("R", [1, 2])
def test_search_threshold(W, H, R):
    p, c, _ = workloads.flow_pair(W, H, seed=W + R)
    check_against_oracle(p, c, [0.5], oracle.Settings(flowScale=1, searchRadius=R))


@pytest.mark.parametrize("settings", [oracle.Settings(flowScale=1), oracle.Settings(flowScale=1, subpixel=False),
                                      oracle.Settings(flowScale=1, searchRadius=1, searchPenalty=0.0)],
                         ids=["r2", "nosubpix", "r1"])
def test_two_integer_levels(settings):
    """1003 x 565 at flowScale 1: 8946 blocks on level 0, 2268 on level 1"""
    p, c, _ = workloads.flow_pair(1003, 565, seed=31)
    check_against_oracle(p, c, [0.5], settings)


def test_flow_scale_4():
    """16 px cells (multiples of 1/16 level), 2400 blocks on level 0"""
    p, c, _ = workloads.flow_pair(1600, 1536, seed=8)
    check_against_oracle(p, c, [0.5], oracle.Settings(flowScale=4))


@pytest.mark.parametrize("name", ["rgb10_abgr", "f16_linear", "nv12_709_limited", "p010_2020_limited"])
def test_formats_integer_levels(name):
    p, c, _ = workloads.flow_pair(515, 301, seed=77)
    check(name, p, c, [0.5], settings=oracle.Settings(flowScale=1))
