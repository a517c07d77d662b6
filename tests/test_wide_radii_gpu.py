"""Radii 7 .. 12 (the runtime-radius search) on levels below and above the block count that changes its launch, recorded
directly and replayed from a graph, against the oracle."""
import numpy as np
import pytest
import torch

import framegen as fg
import oracle
import workloads
from gpu_util import assert_estimate_equal, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


# level 0 at flowScale 2: 32 x 64 = 2048 blocks, 33 x 63 = 2079 blocks
@pytest.mark.parametrize("W,H", [(512, 1024), (528, 1008)])
@pytest.mark.parametrize("radius,top", [(2, 7), (2, 12), (7, 12), (12, 9)])
def test_radii(W, H, radius, top):
    kw = dict(searchRadius=radius, searchRadiusTop=top)
    p, c, _ = workloads.flow_pair(W, H, seed=radius + top)
    a, b = to_dev(p), to_dev(c)
    I = fg.Interpolator()
    assert I.init(W, H, fg.VK_R8G8B8A8_UNORM, settings=fg.Settings(**kw)), I.init_error()
    I.begin_frame()
    assert I.record_estimate(a, b), I.last_error()
    want = oracle.estimate(p, c, oracle.Settings(**kw))
    assert_estimate_equal(fg.read_trace(I), want)
    q, r = to_dev(np.ascontiguousarray(p[::-1])), to_dev(np.ascontiguousarray(c[::-1]))
    I.begin_frame()
    assert I.record_estimate(q, r), I.last_error()
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(s):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            I.begin_frame()
            assert I.record_estimate(a, b, stream=s), I.last_error()
    g.replay()
    torch.cuda.synchronize()
    assert_estimate_equal(fg.read_trace(I), want)
    del g
    I.close()
