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


def test_vectors_wider_apart_than_the_window():
    """halves of a frame moving 26 px apart from each other: tiles whose vectors differ by more than the staged window"""
    W, H = 256, 176
    a = workloads.value_noise(H, W + 64, np.random.Generator(np.random.PCG64(3)))
    p = workloads._to_rgba(a[:, 32:32 + W])
    c = np.concatenate([workloads._to_rgba(a[:, 32 + 26:32 + 26 + W // 2]), workloads._to_rgba(a[:, 32 + W // 2 - 26:32 + W - 26])], axis=1)
    check_against_oracle(p, c, [0.5], oracle.Settings(flowScale=1, globalFallback=1.0, sceneCutSad=250.0))


def test_still_and_uniform_motion():
    """every neighbour's vector the own block's: candidates left out; and a still frame with one moving sprite"""
    p, c, _ = workloads.flow_pair(300, 200, seed=2)
    check_against_oracle(p, p, [0.5])
    q = p.copy()
    q[80:112, 100:140] = np.roll(p, 9, axis=1)[80:112, 100:140]
    check_against_oracle(p, q, [0.25])


@pytest.mark.parametrize("W,H,fs", [(16, 16, 4), (17, 16, 2), (64, 64, 1), (200, 120, 2), (1032, 1024, 1), (4096, 3744, 1)])
def test_scene_cut_mean(W, H, fs):
    """numpy's pairwise mean of the SADs: 1 block, a few, one leaf, several, many leaves, more than fit shared memory"""
    import framegen as fg
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(W)
    f = torch.randint(0, 256, (2, H, W, 4), generator=g, dtype=torch.uint8, device="cuda")
    it = fg.Interpolator()
    assert it.init(W, H, fg.VK_R8G8B8A8_UNORM, settings=fg.Settings(flowScale=fs)), it.init_error()
    it.begin_frame()
    assert it.record_estimate(f[0], f[1])
    tr = fg.read_trace(it)
    assert tr["sads"].size == -(-round(W / fs) // 8) * -(-round(H / fs) // 8)   # (sizes round half to even)
    assert np.float32(tr["sad"]) == tr["sads"].mean(dtype=np.float32)
    assert tr["sadSum256"] == int(np.rint(tr["sads"].ravel() * np.float32(256)).astype(np.int64).sum()) & 0xFFFFFFFF
    it.close()
