"""Small frames of grids whose trace layout is the wide one (bit addresses beyond 32 bits): the 2-, 4- and 8-pixel tiles
that such frames run there, at odd pixel counts. Every output bit for bit as the oracle's."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import empty, export_r8, same_bits

pytestmark = pytest.mark.gpu
KEYS = ("shadow", "ao", "ao_vis", "spec", "spec_t")
N = 1040


@pytest.fixture(scope="module")
def world(vxl, ctx):
    G = vxl.Grid(ctx, N, N, N)
    G.scene_noise(4, 0.6, 1.0 / 32.0, 8)
    G.scene_boxes(4, 300, 4, 48)
    assert G.describe().trace_wide == 1
    return G, export_r8(G)


# on 152 SMs: 2 pixels below 7,782 pixels from 16 rays a pixel on, 4 below 29,184 from 8 on, 8 below 194,560 (136,192
# with fewer than 10 rays)
@pytest.mark.parametrize("W,H,n_ao,n_spec", [(1, 1, 16, 1), (13, 7, 28, 2), (101, 77, 16, 1), (101, 77, 8, 1), (181, 161, 8, 1),
                                             (181, 161, 24, 2), (251, 160, 4, 1), (3, 1, 1, 0)])
@pytest.mark.parametrize("light", [(0.3, 0.8, 0.5), (0.0, 0.8, -0.6)])
def test_small_frame_of_a_wide_grid(vxl, ctx, world, W, H, n_ao, n_spec, light):
    import torch

    G, r8 = world
    cam, tgt = np.array([0.5 * N, 0.9 * N, 0.05 * N], np.float32), np.array([0.5 * N, 0.3 * N, 0.6 * N], np.float32)
    pos, nrm, rough = empty(W * H * 3, torch.float32), empty(W * H * 3, torch.float32), empty(W * H, torch.float32)
    vxl.scene_gbuffer(ctx, G, cam, tgt, W, H, W, pos, nrm, rough)
    kw = dict(light_dir=light, cam_pos=cam, n_ao=n_ao, ao_len=48.0, n_spec=n_spec, seed=W + n_ao)
    outs = {k: empty(W * H, torch.float32) for k in KEYS}
    vxl.trace_occlusion(ctx, G, pos, nrm, rough, W * H, vxl.make_params(**kw), width=W, height=H, **outs)
    torch.cuda.synchronize()
    want = oracle.occlusion(r8, pos.cpu().numpy(), nrm.cpu().numpy(), rough.cpu().numpy(), oracle.make_params(**kw))
    if W * H > 1000:
        assert len(np.unique(want["ao"])) > n_ao and (light[0] == 0.0 or 0.02 < (want["shadow"] == 0.0).mean() < 0.98)
    for k in KEYS:
        assert same_bits(outs[k].cpu().numpy(), want[k]).all(), k
