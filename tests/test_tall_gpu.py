"""Frames of more than 65535 block rows: 16 x 524304 at flowScale 1 has 65538, past a grid's second dimension."""
import numpy as np
import pytest

import framegen as fg
import oracle
from gpu_util import assert_estimate_equal, to_dev

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


@pytest.mark.parametrize("kw", [dict(searchRadiusTop=2), dict(searchRadiusTop=1), dict(searchRadiusTop=6),
                                dict(searchRadiusTop=2, subpixel=False)], ids=["r2", "r1", "r6", "nosubpix"])
def test_block_rows_past_a_grid_dimension(kw):
    W, H = 16, 524304
    rng = np.random.default_rng(5)
    p = rng.integers(0, 256, (H, W, 4), dtype=np.uint8)
    c = np.roll(p, 2, axis=0)
    I = fg.Interpolator()
    assert I.init(W, H, fg.VK_R8G8B8A8_UNORM, settings=fg.Settings(flowScale=1, **kw)), I.init_error()
    I.begin_frame()
    a, b = to_dev(p), to_dev(c)
    assert I.record_estimate(a, b), I.last_error()
    assert_estimate_equal(fg.read_trace(I), oracle.estimate(p, c, oracle.Settings(flowScale=1, **kw)))
    assert I.record_synth(a, b, a.clone(), 0.5), I.last_error()
    I.close()
