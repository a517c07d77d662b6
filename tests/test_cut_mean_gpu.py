"""The tickets of the scene-cut mean and of the global medians: the CTA that comes last has to see what every other one
wrote. Long chains of estimates of two alternating pairs, nothing waited for in between, each result copied out on the
stream and compared with the pair's own."""
import pytest
import torch

import framegen as fg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def built():
    import build
    build.build()


# leaves of at most 128 SADs: 1, 16 (two CTAs of 8 warps), 128, 2048 (more than the shared memory of a CTA holds)
@pytest.mark.parametrize("W,H,fs", [(64, 64, 1), (192, 400, 1), (1024, 600, 1), (4096, 3840, 1)])
def test_chains_of_estimates(W, H, fs):
    g = torch.Generator(device="cuda")
    g.manual_seed(W + H)
    f = torch.randint(0, 256, (3, H, W, 4), generator=g, dtype=torch.uint8, device="cuda")
    f[2, :H // 2] = f[1, :H // 2]
    pairs = [(f[0], f[1]), (f[1], f[2])]
    I = fg.Interpolator()
    assert I.init(W, H, fg.VK_R8G8B8A8_UNORM, settings=fg.Settings(flowScale=fs)), I.init_error()
    want = []
    for p, c in pairs:
        I.begin_frame()
        assert I.record_estimate(p, c)
        tr = fg.read_trace(I)
        assert tr["sads"].mean(dtype="float32") == tr["sad"]
        want.append((tr["sadSum256"], tr["meds"].copy(), tr["sad"]))
    assert want[0][0] != want[1][0]
    n = 200 if W < 4096 else 40
    got = torch.zeros((n, 2), dtype=torch.int32, device="cuda")
    for i in range(n):
        I.begin_frame()
        assert I.record_estimate(*pairs[i & 1])
        assert I.record_debug_counters(got[i])
    s = got[:, 1].cpu().numpy().astype("uint32")
    assert [int(v) for v in s] == [want[i & 1][0] for i in range(n)]
    tr = fg.read_trace(I)
    assert tr["sad"] == want[1][2] and (tr["meds"] == want[1][1]).all()
