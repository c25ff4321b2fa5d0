"""Frames whose tiles the occlusion kernels choose smaller than 16 pixels (down to 2), on the trace layout, its wide form
and in a batch: odd pixel counts around the tiles, few and many rays a pixel, shadow rays in the literal form. Every
output bit for bit as the oracle's."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import empty, export_r8, same_bits

pytestmark = pytest.mark.gpu
KEYS = ("shadow", "ao", "ao_vis", "spec", "spec_t")


def _view(vxl, ctx, G, W, H, seed):
    import torch

    n = G.ny
    cam = np.array([0.5 * G.nx, 1.3 * n, -0.3 * n], np.float32)
    tgt = np.array([0.5 * G.nx, 0.4 * n, 0.5 * G.nz], np.float32)
    pos, nrm, rough = empty(W * H * 3, torch.float32), empty(W * H * 3, torch.float32), empty(W * H, torch.float32)
    vxl.scene_gbuffer(ctx, G, cam, tgt, W, H, seed, pos, nrm, rough)
    return cam, pos, nrm, rough


def _want(G, pos, nrm, rough, kw):
    return oracle.occlusion(export_r8(G), pos.cpu().numpy(), nrm.cpu().numpy(), rough.cpu().numpy(), oracle.make_params(**kw))


@pytest.mark.parametrize("W,H", [(1, 1), (3, 1), (13, 7), (61, 53), (161, 91), (251, 160)])
@pytest.mark.parametrize("n_ao,n_spec,light", [(8, 1, (0.3, 0.8, 0.5)), (16, 2, (0.0, 1.0, 0.0)), (28, 2, (0.3, 0.8, 0.5)),
                                               (1, 0, (0.2, 0.9, -0.1))])
def test_small_frame(vxl, ctx, W, H, n_ao, n_spec, light):
    import torch

    G = vxl.Grid(ctx, 96, 64, 80)
    G.scene_noise(3, 0.55, 1.0 / 32.0, 8)
    cam, pos, nrm, rough = _view(vxl, ctx, G, W, H, W)
    kw = dict(light_dir=light, cam_pos=cam, n_ao=n_ao, ao_len=24.0, n_spec=n_spec, seed=W + n_ao)
    outs = {k: empty(W * H, torch.float32) for k in KEYS}
    vxl.trace_occlusion(ctx, G, pos, nrm, rough, W * H, vxl.make_params(**kw), width=W, height=H, **outs)
    torch.cuda.synchronize()
    want = _want(G, pos, nrm, rough, kw)
    for k in KEYS:
        assert same_bits(outs[k].cpu().numpy(), want[k]).all(), k


@pytest.mark.parametrize("W,H", [(9, 5), (101, 67), (251, 160)])
def test_small_frame_of_a_wide_grid(vxl, ctx, W, H):
    import torch

    G = vxl.Grid(ctx, 1040, 128, 1040)
    G.scene_noise(4, 0.6, 1.0 / 32.0, 8)
    if not G.describe().trace_words:
        pytest.skip("no trace layout")
    cam, pos, nrm, rough = _view(vxl, ctx, G, W, H, 5)
    kw = dict(light_dir=(0.3, 0.8, 0.5), cam_pos=cam, n_ao=8, ao_len=32.0, n_spec=1, seed=W)
    outs = {k: empty(W * H, torch.float32) for k in KEYS}
    vxl.trace_occlusion(ctx, G, pos, nrm, rough, W * H, vxl.make_params(**kw), width=W, height=H, **outs)
    torch.cuda.synchronize()
    want = _want(G, pos, nrm, rough, kw)
    for k in KEYS:
        assert same_bits(outs[k].cpu().numpy(), want[k]).all(), k


@pytest.mark.parametrize("count,n_ao", [(3, 8), (3, 20), (70, 16)])
def test_small_batch(vxl, ctx, count, n_ao):
    import torch

    items = []
    for i in range(count):
        G = vxl.Grid(ctx, 64, 48, 56)
        G.scene_noise(10 + i, 0.55, 1.0 / 32.0, 8)
        W, H = 17 + i % 7, 5 + i % 3
        cam, pos, nrm, rough = _view(vxl, ctx, G, W, H, i)
        kw = dict(light_dir=(0.3, 0.8, 0.5), cam_pos=cam, n_ao=n_ao, ao_len=24.0, n_spec=1, seed=i)
        items.append(dict(grid=G, npix=W * H, width=W, height=H, params=vxl.make_params(**kw), pos=pos, nrm=nrm,
                          rough=rough, kw=kw, **{k: empty(W * H, torch.float32) for k in KEYS}))
    vxl.Batch(ctx, [{k: v for k, v in it.items() if k != "kw"} for it in items]).run()
    torch.cuda.synchronize()
    for it in items[::7] if count > 7 else items:
        want = _want(it["grid"], it["pos"], it["nrm"], it["rough"], it["kw"])
        for k in KEYS:
            assert same_bits(it[k].cpu().numpy(), want[k]).all(), k
