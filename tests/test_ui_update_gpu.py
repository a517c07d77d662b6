"""CrosshairV2's state update on the GPU where its staged 22 x 14 pixel windows have edges: boxes at the frame's corners
(the 7x7 median's taps are clamped to the frame), boxes over the whole frame, work rectangles that are not multiples of
the 16 x 8 CTA. The frames hold still, so the local contrast is found at every pixel of the box; every state word and
mask byte equals the oracle's (oracle/ui_v2.py): integers, no tolerance."""
import numpy as np
import pytest
import torch

import framegen as fg
import ui_v2
from test_ui_v2_gpu import oracle_words, v2_settings

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


@pytest.mark.parametrize("W,H,bw,bh,ox,oy", [(64, 48, 16, 16, -24, -16), (64, 48, 14, 12, 25, 18), (65, 49, 17, 9, 3, -2),
                                             (66, 50, 64, 48, 0, 0), (64, 48, 30, 14, 0, 0)])
def test_update_at_tile_and_frame_edges(W, H, bw, bh, ox, oy):
    s = v2_settings(uiBoxWidth=bw, uiBoxHeight=bh, uiBoxOffsetX=ox, uiBoxOffsetY=oy)
    rng = np.random.default_rng(W * 1000 + bw)
    still = rng.integers(0, 256, (H, W, 4), dtype=np.uint8)
    I = fg.Interpolator()
    assert I.init(W, H, fg.VK_R8G8B8A8_UNORM, settings=s), I.init_error()
    st = ui_v2.State(s, W, H)
    assert fg.work_rect(s, W, H) == st.work
    for k in range(4):
        f = still.copy()
        f[rng.random((H, W)) < 0.1] ^= 0x80   # some pixels of each frame move
        d = torch.from_numpy(f).cuda()
        assert I.record_observe(d)
        st.update(f)
        want_mask = st.mask()
        got = fg.read_ui(I, d, s, W, H)
        for name, want in zip(("w0", "w1", "w2"), oracle_words(st)):
            assert np.array_equal(got[name], want), f"frame {k}: state word {name} differs"
        assert np.array_equal(got["mask"], want_mask), f"frame {k}: mask differs"
    I.close()
