"""recordTrace where the float level 0 of the luma is not the latest record's: after a change of flow scale or size before
the next estimate, and after the replay of a graph whose estimate was followed by one that kept another form of level 0."""
import numpy as np
import pytest
import torch

import framegen as fg
import workloads
from gpu_util import to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


def pair(W, H, seed):
    p, c, _ = workloads.flow_pair(W, H, seed=seed)
    return to_dev(p), to_dev(c)


def interpolator(W, H, settings):
    I = fg.Interpolator()
    assert I.init(W, H, fg.VK_R8G8B8A8_UNORM, settings=settings), I.init_error()
    return I


def estimate(I, p, c, stream=None):
    I.begin_frame()
    assert I.record_estimate(p, c, stream=stream), I.last_error()


# 1024 x 1024 at flowScale 2: 4096 blocks, so radius 2 searches the pair planes and level 0 is written as pair planes
# only; radius 3 has it written as float too
@pytest.mark.parametrize("first,later", [(2, 3), (3, 2)])
def test_replayed_estimate(first, later):
    W = H = 1024
    I = interpolator(W, H, fg.Settings(searchRadius=first))
    a, b = pair(W, H, 1), pair(W, H, 2)
    estimate(I, *a)
    want = fg.read_trace(I)
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            estimate(I, *a, stream=s)
    assert I.set_settings(fg.Settings(searchRadius=later))
    estimate(I, *b)
    other = fg.read_trace(I)
    assert not np.array_equal(other["luma"][0][0], want["luma"][0][0])
    torch.cuda.synchronize()
    g.replay()
    torch.cuda.synchronize()
    got = fg.read_trace(I)
    for k in range(2):
        for l in range(len(want["luma"])):
            assert np.array_equal(got["luma"][l][k], want["luma"][l][k]), (l, k)
    assert np.array_equal(got["pf"], want["pf"])
    del g


@pytest.mark.parametrize("how", ["flow scale", "size", "same planes"])
def test_trace_before_the_next_estimate(how):
    """a new layout holds zeros, whether it keeps pair planes (heights not of the form 4 k + 3 at flowScale 4) or not"""
    W, H = 1024, 1023
    I = interpolator(W, H, fg.Settings(flowScale=2 if how != "size" else 4, searchRadius=2))
    if how == "size":
        assert I.resize(2048, 2048)
        estimate(I, *pair(2048, 2048, 3))
        assert I.resize(W, H)
    else:
        estimate(I, *pair(W, H, 3))
        assert I.reconfigure(fg.Settings(flowScale=4 if how == "flow scale" else 1))
    tr = fg.read_trace(I)
    for planes in tr["luma"]:
        assert not planes[0].any() and not planes[1].any()
    assert tr["err"] == 0 and not tr["pf"].any()
    p, c = pair(W, H, 3)
    estimate(I, p, c)   # and the layout works
    J = interpolator(W, H, I.settings())
    estimate(J, p, c)
    x, y = fg.read_trace(I), fg.read_trace(J)
    assert np.array_equal(x["luma"][0][0], y["luma"][0][0]) and np.array_equal(x["pf"], y["pf"])
