"""A tile shape that the caller sets is the one that runs, on small frames too (seen in a batch's tile count), and the
default chooses; the batched kernel in each tile, the 16 pixels of every large batch among them, against the oracle."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import empty, export_r8, same_bits

pytestmark = pytest.mark.gpu
KEYS = ("shadow", "ao", "ao_vis", "spec", "spec_t")


def _items(vxl, ctx, sizes, n_ao=8):
    import torch

    items = []
    for i, (W, H) in enumerate(sizes):
        G = vxl.Grid(ctx, 64, 48, 56)
        G.scene_noise(20 + i, 0.55, 1.0 / 32.0, 8)
        cam, tgt = np.array([32, 62, -14], np.float32), np.array([32, 19, 28], np.float32)
        pos, nrm, rough = empty(W * H * 3, torch.float32), empty(W * H * 3, torch.float32), empty(W * H, torch.float32)
        vxl.scene_gbuffer(ctx, G, cam, tgt, W, H, i, pos, nrm, rough)
        kw = dict(light_dir=(0.3, 0.8, 0.5), cam_pos=cam, n_ao=n_ao, ao_len=24.0, n_spec=1, seed=i)
        items.append(dict(grid=G, npix=W * H, width=W, height=H, params=vxl.make_params(**kw), pos=pos, nrm=nrm,
                          rough=rough, kw=kw, **{k: empty(W * H, torch.float32) for k in KEYS}))
    return items


def _tiles(vxl, ctx, items):
    b = vxl.Batch(ctx, [{k: v for k, v in it.items() if k != "kw"} for it in items])
    n = b.info()[0]
    b.run()
    b.close()
    return n


def _match(items):
    import torch

    torch.cuda.synchronize()
    for it in items:
        want = oracle.occlusion(export_r8(it["grid"]), it["pos"].cpu().numpy(), it["nrm"].cpu().numpy(),
                                it["rough"].cpu().numpy(), oracle.make_params(**it["kw"]))
        for k in KEYS:
            assert same_bits(it[k].cpu().numpy(), want[k]).all(), k


# as one call sets it: the tile alone, with its shape, or among other knobs
@pytest.mark.parametrize("knobs", [dict(tile_px=16), dict(tile_px=16, tile_w=16), dict(tile_px=8, tile_w=8),
                                   dict(tile_px=32, tile_w=32), dict(tile_px=8, kstep=8, leap=2, order=1, tile_w=8, grab=1)])
def test_a_chosen_tile_is_kept(vxl, knobs):
    ctx = vxl.Context(0)
    items = _items(vxl, ctx, [(61, 53), (17, 9), (1, 1)])
    default = ctx.get_tuning()
    free = _tiles(vxl, ctx, items)
    assert free > sum(-(-it["npix"] // 16) for it in items)  # the default runs smaller tiles here
    ctx.set_tuning(**knobs)
    px = knobs["tile_px"]
    assert ctx.get_tuning()["tile_px"] == px
    assert _tiles(vxl, ctx, items) == sum(-(-it["npix"] // px) for it in items)
    _match(items)
    ctx.set_tuning(grab=1)  # says nothing of the tile
    assert _tiles(vxl, ctx, items) == sum(-(-it["npix"] // px) for it in items)
    ctx.set_tuning(**default)
    assert _tiles(vxl, ctx, items) == free


def test_large_batches_run_16_pixels(vxl):
    ctx = vxl.Context(0)
    items = _items(vxl, ctx, [(417, 311), (401, 307), (3, 5)])
    assert _tiles(vxl, ctx, items) == sum(-(-it["npix"] // 16) for it in items)
    _match(items)


@pytest.mark.parametrize("n_ao,size,px", [(4, (251, 160), 8), (4, (400, 301), 16), (8, (251, 160), 8), (8, (400, 301), 8),
                                          (16, (101, 50), 2)])
def test_default_tiles(vxl, n_ao, size, px):
    """The measured choice by pixels and rays a pixel, for the 152 SMs that it was measured on."""
    import torch

    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("measured on 152 SMs")
    items = _items(vxl, ctx := vxl.Context(0), [size], n_ao)
    assert _tiles(vxl, ctx, items) == -(-items[0]["npix"] // px)
    _match(items)
