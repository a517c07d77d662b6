"""The synthesis' forms by grid: at most 2 CTAs per SM (the latency form) and more, at 289 and 306 tiles of 58 x 58 (B200 has
148 SMs; up to 148 tiles ask for another split of the L1 at flowScale 1), in every format and flow scale, plain and with
the overlay protection, against the oracle; and the mask test of a tap's pixels, which reads whole words, with masks
whose rows end at every place of a word."""
import numpy as np
import pytest
import torch

import framegen as fg
import oracle
import ui_v2
import workloads
from test_synth_tiles_gpu import FORMATS, T13, run
from test_ui_v2_fmt_gpu import SPECS, dev, empty_like, host, same
from test_ui_v2_gpu import grain_scene, oracle_settings, v2_settings

pytestmark = pytest.mark.gpu
SIZES = [(986, 986), (1044, 986), (696, 696), (232, 2146)]   # 289, 306, 144 and 148 tiles


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


@pytest.mark.parametrize("fmt", ["rgba8"] + FORMATS)
@pytest.mark.parametrize("fs", [1, 2, 4])
@pytest.mark.parametrize("W,H", SIZES)
def test_one_wave_and_more(W, H, fs, fmt):
    p, c, _ = workloads.flow_pair(W, H, seed=W + fs)
    run(fmt, p, c, [0.5, T13], oracle.Settings(flowScale=fs))


def protected(name, W, H, box, offset, ts, **kw):
    rgba8 = name == "rgba8"
    vk, spec, conv, extra = (fg.VK_R8G8B8A8_UNORM, None, lambda f: f, {}) if rgba8 else SPECS[name]
    s = v2_settings(uiBoxWidth=box[0], uiBoxHeight=box[1], uiBoxOffsetX=offset[0], uiBoxOffsetY=offset[1], uiStillFrames=2,
                    uiEstimateFill=True, uiContrastThreshold=0.0, globalFallback=1.0, sceneCutSad=255.0, **kw)
    x0, y0, w, h = (int(v) for v in fg.box_rect(s, W, H))
    rgba = grain_scene(W, H, 4, pan=(14, -10), plus=False)[0]
    for f in rgba:
        if name in ("nv12", "p010"):   # a whole patch, 2 px wider: a chroma texel of the box holds nothing that moves
            f[y0 - 2:y0 + h + 2, x0 - 2:x0 + w + 2, :3] = (0, 255, 255)
        else:   # dots: a tap's pixels are partly marked
            f[y0:y0 + h:2, x0:x0 + w:2, :3] = (0, 255, 255)
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
    est = oracle.estimate(frames[-2], frames[-1], settings=os_, ui_fill=ui) if rgba8 else \
        oracle.estimate_fmt(frames[-2], frames[-1], spec, settings=os_, ui_fill=ui)
    for t in ts:
        o = empty_like(d[0])
        assert I.record_synth(d[-2], d[-1], o, t), I.last_error()
        if rgba8:
            ref = oracle.synth(frames[-2], frames[-1], est, t, settings=os_, ui=ui)[0]
            ui_v2.patch(ref, frames[-1], masks[-1], st.work)
        else:
            ref = oracle.synth_fmt(frames[-2], frames[-1], est, t, spec, settings=os_, ui=ui)[0]
            ui_v2.patch_fmt(ref, frames[-1], masks[-1], st.work, spec)
        torch.cuda.synchronize()
        assert same(host(o, ref), ref), (box, offset, t)
    I.close()


@pytest.mark.parametrize("name", ["rgba8", "rgb10", "f16_linear", "f16_encoded", "nv12", "p010"])
@pytest.mark.parametrize("fs", [1, 2])
@pytest.mark.parametrize("W,H", [SIZES[1], SIZES[2]])
def test_protected_one_wave_and_more(W, H, fs, name):
    protected(name, W, H, (90, 70), (20, -14), [0.5, T13], flowScale=fs)


@pytest.mark.parametrize("name", ["rgba8", "nv12"])
@pytest.mark.parametrize("width", [1, 2, 3, 4, 5, 6, 7, 9])
def test_mask_rows_of_every_width(name, width):
    for off in range(4):
        protected(name, 174, 174, (width, 3 + off), (off, -off), [0.5, 0.25])
