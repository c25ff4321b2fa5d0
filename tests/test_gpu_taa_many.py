"""Frames most of whose pixels are disoccluded (a fast pan, a camera that jumps): pixels one a lane, chosen by how many lie
in blocks of many, beside those in blocks of few; and the motion test that a common motion decides. Against the oracle,
bit for bit, NaN == NaN."""
import numpy as np
import pytest

from tests import taa_cases
from tests.test_gpu_taa_taps import _check

pytestmark = pytest.mark.gpu


def _frame(W, H, kind, motion):
    rng = np.random.default_rng(W + H)
    fr = taa_cases.frame(W, H, W, 0)
    out = np.zeros((H, W), bool)
    if kind == "all":
        out[:] = True
    elif kind == "columns":  # not a multiple of the blocks of 32 x 4 pixels, and some pixels apart
        out[:, : W * 5 // 8 + 5] = True
        out[rng.integers(0, H, 60), rng.integers(0, W, 60)] = True
    elif kind == "mixed":  # blocks of all shares
        out = rng.random((H, W)) < np.repeat(np.repeat(rng.random((H // 4 + 1, W // 32 + 1)) * 1.6, 4, 0), 32, 1)[:H, :W]
    fr["motion"][out] = np.array([-1.5, 0.25], np.float32) + np.float32(motion) * rng.random((int(out.sum()), 2)).astype(np.float32)
    return fr


# above 85,120 disoccluded pixels in warps of many on 152 SMs
@pytest.mark.parametrize("W,H", [(525, 331), (1003, 190)])
@pytest.mark.parametrize("kind", ["all", "columns", "mixed"])
@pytest.mark.parametrize("motion", [0.0, 0.06, 0.2])
def test_many_disoccluded(vxl, ctx, W, H, kind, motion):
    want = _check(vxl, ctx, _frame(W, H, kind, motion), W, H)
    assert (want[3:, :, 3] == 1.0).mean() > 0.4


@pytest.mark.parametrize("image", ["light", "color", "normal", "material", "depth", "motion"])
@pytest.mark.parametrize("value", [np.nan, np.inf, 3e38, -2e19])
def test_wild_values(vxl, ctx, image, value):
    W, H = 431, 211
    fr = _frame(W, H, "all", 0.0)
    rng = np.random.default_rng(1)
    for _ in range(30):
        fr[image][int(rng.integers(3, H)), int(rng.integers(0, W)), int(rng.integers(0, fr[image].shape[2]))] = value
    _check(vxl, ctx, fr, W, H)


@pytest.mark.parametrize("base", [0.06, -2.0, 200.0, 1e6])
@pytest.mark.parametrize("scale", [0.0, 0.034, 0.036, 0.07, 0.2])
def test_common_motion(vxl, ctx, base, scale):
    """Motions around one that is not zero, within the skipping bound and beyond it."""
    W, H = 431, 211
    fr = taa_cases.frame(W, H, 8, 0)
    sign = np.where((np.arange(W)[None, :] // 9 + np.arange(H)[:, None] // 6) % 2 == 0, 1.0, -1.0)
    fr["motion"] = np.ascontiguousarray(base + (sign * scale)[..., None] * [1.0, 1.0], np.float32)
    fr["color"][:] = 0.5  # every tap counts
    fr["material"][:] = 0.25
    fr["normal"][:] = [0.0, 1.0, 0.0]
    fr["depth"][:] = 0.05
    _check(vxl, ctx, fr, W, H)


@pytest.mark.parametrize("W,H", [(97, 45), (431, 211)])
def test_captured(vxl, ctx, W, H):
    """Replays of a captured call on new inputs, whose launches follow one another as the call's own do."""
    import torch

    import oracle
    from tests.gpu_util import dev, same_bits
    from tests.test_gpu_taa import KEYS

    frames = [_frame(W, H, kind, 0.05) for kind in ("columns", "all", "mixed")]
    d = [dev(frames[0][k]) for k in KEYS]
    out = torch.empty(W * H * 4, dtype=torch.float32, device="cuda")
    vxl.light_taa(ctx, *d, W, H, out)  # sizes the workspace
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        vxl.light_taa(ctx, *d, W, H, out, stream=torch.cuda.current_stream())
    got = []
    for fr in frames:
        for t, k in zip(d, KEYS):
            t.copy_(dev(fr[k]))
        g.replay()
        got.append(out.clone())
    torch.cuda.synchronize()
    for fr, o in zip(frames, got):
        want = oracle.taa(*[fr[k] for k in KEYS])
        assert same_bits(o.cpu().numpy().reshape(H, W, 4), want).all()
