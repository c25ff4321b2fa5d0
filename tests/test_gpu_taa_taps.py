"""The shortened taps of the temporal accumulation (one texel for four that agree, no normal and material where the
colour rules a tap out, no motion where none can matter) against the oracle, bit for bit, NaN == NaN: values that are
not finite or far too large in every image, motion around the skipping bound, taps that reach far, images of one texel."""
import numpy as np
import pytest

import oracle
from tests import taa_cases
from tests.gpu_util import dev, same_bits
from tests.test_gpu_taa import KEYS

pytestmark = pytest.mark.gpu


def _check(vxl, ctx, fr, W, H):
    import torch

    out = torch.empty(W * H * 4, dtype=torch.float32, device="cuda")
    d = [dev(fr[k]) for k in KEYS]
    vxl.light_taa(ctx, *d, W, H, out)
    torch.cuda.synchronize()
    got, want = out.cpu().numpy().reshape(H, W, 4), oracle.taa(*[fr[k] for k in KEYS])
    assert same_bits(got, want).all(), np.argwhere(~same_bits(got, want))[:5]
    return want


@pytest.mark.parametrize("W,H", [(1, 1), (2, 3), (33, 9), (64, 16), (600, 5)])
def test_sizes(vxl, ctx, W, H):
    _check(vxl, ctx, taa_cases.frame(W, H, W, 0), W, H)


@pytest.mark.parametrize("image", ["light", "last", "color", "normal", "material", "depth", "motion", "noise"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 3e38, -2e19, -0.0])
def test_wild_values(vxl, ctx, image, value):
    W, H = 97, 45
    rng = np.random.default_rng(4)
    fr = taa_cases.frame(W, H, 6, 3)
    for k in range(20):
        y, x = int(rng.integers(3, H)), int(rng.integers(0, W))
        fr[image][y, x, int(rng.integers(0, fr[image].shape[2]))] = value
    _check(vxl, ctx, fr, W, H)


@pytest.mark.parametrize("scale", [0.01, 0.0349, 0.0351, 0.08, 0.3])
@pytest.mark.parametrize("reach", [0.0, 1.2, 1.3, 40.0, -300.0])
def test_motion_and_reach(vxl, ctx, scale, reach):
    W, H = 150, 70
    rng = np.random.default_rng(int(scale * 1e4))
    fr = taa_cases.frame(W, H, 8, 0)
    # half the image moves one way, half the other, in patches, so that neighbours differ by up to twice the scale
    sign = np.where((np.arange(W)[None, :] // 9 + np.arange(H)[:, None] // 6) % 2 == 0, 1.0, -1.0)
    fr["motion"] = np.ascontiguousarray((sign * scale)[..., None] * [1.0, 1.0], np.float32)
    fr["motion"][:, 80:] *= np.float32(0.2)
    fr["last"][..., 3] = reach
    fr["color"][:] = 0.5  # every tap counts
    fr["material"][:] = 0.25
    fr["normal"][:] = [0.0, 1.0, 0.0]
    fr["depth"][:] = 0.05 + 1e-5 * rng.random((H, W, 1))
    _check(vxl, ctx, fr, W, H)


def test_negative_depth(vxl, ctx):
    W, H = 70, 33
    fr = taa_cases.frame(W, H, 3, 0)
    fr["depth"][:] = -1e-3  # 1 / depth scales the spiral
    _check(vxl, ctx, fr, W, H)


@pytest.mark.parametrize("W,H,band", [(400, 171, 0), (347, 199, 40), (1024, 70, 3)])
def test_frames_of_one_lane_a_pixel(vxl, ctx, W, H, band):
    """Above 68,096 pixels on this GPU (152 SMs): one lane a pixel, and the edge in blocks of 128, several pixels each
    for the wide band."""
    rng = np.random.default_rng(W)
    fr = taa_cases.frame(W, H, W, band)
    fr["motion"][H // 2:, W // 2:] *= np.float32(30.0)  # above the bound in a quarter of the frame
    fr["last"][: H // 3, :, 3] = 3.0
    for image, value in (("material", np.nan), ("depth", np.inf), ("color", -2e19), ("light", np.nan)):
        fr[image][int(rng.integers(3, H)), int(rng.integers(0, W)), 0] = value
    _check(vxl, ctx, fr, W, H)
