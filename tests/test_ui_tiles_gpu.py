"""CrosshairV2's synthesis tiles: a tile whose taps cannot touch a mask's rectangle skips the rejection. A small overlay is
moved pixel by pixel over the borders of a 58 x 58 tile, across and down, on a panning background (the taps reach 1/4,
1/2 and 3/4 of the pan to either side): every distance between a tile's taps and the rectangle comes up, the first pixel
that touches and the last that does not among them. Every output byte is the oracle's, which tests every tap."""
import numpy as np
import pytest
import torch

import framegen as fg
import oracle
import ui_v2
from test_ui_v2_fmt_gpu import SPECS, dev, empty_like, host, same
from test_ui_v2_gpu import grain_scene, oracle_settings, v2_settings

pytestmark = pytest.mark.gpu
T = 58                       # tile side (csrc/fg_device.h kSyT, kSyTH)
W = H = 3 * T


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


def background():
    if not hasattr(background, "f"):
        background.f = grain_scene(W, H, 4, pan=(14, -10), plus=False)[0]
    return background.f


@pytest.mark.parametrize("axis", [0, 1], ids=["across", "down"])
@pytest.mark.parametrize("name", ["rgba8", "rgb10", "f16_linear", "nv12", "p010"])
def test_overlay_over_a_tile_border(name, axis):
    rgba8 = name == "rgba8"
    vk, spec, conv, extra = (fg.VK_R8G8B8A8_UNORM, None, lambda f: f, {}) if rgba8 else SPECS[name]
    shown = 0
    for off in [s * k for k in range(T // 2 - 14, T // 2 + 9) for s in (-1, 1)]:   # the centre tile ends at +-29
        ox, oy = (off, 3) if axis == 0 else (3, off)
        s = v2_settings(uiBoxWidth=6, uiBoxHeight=6, uiBoxOffsetX=ox, uiBoxOffsetY=oy, uiStillFrames=2, uiEstimateFill=True,
                        uiContrastThreshold=0.0, globalFallback=1.0, sceneCutSad=255.0)
        x0, y0, w, h = (int(v) for v in fg.box_rect(s, W, H))
        rgba = [f.copy() for f in background()]
        for f in rgba:
            f[y0:y0 + h, x0:x0 + w, :3] = (0, 255, 255)
        frames = [conv(f) for f in rgba]
        I = fg.Interpolator()
        assert I.init(W, H, vk, settings=s, **extra), I.init_error()
        st = ui_v2.State(s, W, H)
        d = [dev(f) for f in frames]
        masks = []
        for f, g in zip(frames, d):
            assert I.record_observe(g)
            st.update(f) if rgba8 else st.update(f, spec=spec)
            masks.append(st.mask())
        assert (masks[-1] == 255).any()
        I.begin_frame()
        assert I.record_estimate(d[-2], d[-1])
        ui = ((masks[-2], st.work), (masks[-1], st.work))
        os_ = oracle_settings(s)
        if rgba8:
            est = oracle.estimate(frames[-2], frames[-1], settings=os_, ui_fill=ui)
        else:
            est = oracle.estimate_fmt(frames[-2], frames[-1], spec, settings=os_, ui_fill=ui)
        for t in (0.5, 0.25):
            o = empty_like(d[0])
            assert I.record_synth(d[-2], d[-1], o, t), I.last_error()
            if rgba8:
                ref, plain = (oracle.synth(frames[-2], frames[-1], est, t, settings=os_, ui=u)[0] for u in (ui, None))
            else:
                ref, plain = (oracle.synth_fmt(frames[-2], frames[-1], est, t, spec, settings=os_, ui=u)[0] for u in (ui, None))
            shown += not same(ref, plain)
            if rgba8:
                ui_v2.patch(ref, frames[-1], masks[-1], st.work)
            else:
                ui_v2.patch_fmt(ref, frames[-1], masks[-1], st.work, spec)
            torch.cuda.synchronize()
            assert same(host(o, ref), ref), f"offset {ox}, {oy}, t={t}"
        I.close()
    assert shown > 60, shown   # the rejection changes the frame
