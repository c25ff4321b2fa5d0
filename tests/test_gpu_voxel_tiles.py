"""The voxelizer's tiles and levels against the oracle: models around the edges
of every tile shape, placements scaled beyond the bricks a block gathers, and
crowds of mixed ops whose order matters."""
import numpy as np
import pytest

import oracle
from tests import vox_cases
from tests.gpu_util import dev, export_r8

pytestmark = pytest.mark.gpu

# (sx, sy, sz) around the tile shapes 16x8x8, 8x16x8, 8x8x16, 32x4x8, 16x4x16 and 4x16x16
SHAPES = [(1, 1, 1), (1, 40, 3), (4, 16, 16), (4, 17, 33), (5, 16, 8), (8, 33, 9), (9, 8, 8), (16, 8, 8), (17, 9, 17), (48, 7, 25),
          (8, 8, 16), (7, 8, 31), (32, 4, 8), (31, 3, 24), (64, 4, 9), (16, 4, 16), (15, 4, 32), (33, 12, 16)]


def check(vxl, ctx, n, models, insts, noalloc=False):
    import torch

    dms = [dev(m) for m in models]
    mdesc = [(d.data_ptr(),) + m.shape[::-1] for m, d in zip(models, dms)]
    S = n // 2
    G = vxl.Grid(ctx, n, n, n)
    want = np.zeros((S, S, S), np.uint8)
    aabb0 = np.tile(np.array([S - 1, S - 1, S - 1, 0, 0, 0], np.int32), (len(insts), 1))
    got_aabb = dev(aabb0)
    if noalloc:
        vxl.voxelize_noalloc(G.describe(), mdesc, insts, got_aabb)
    else:
        vxl.voxelize(ctx, G, mdesc, insts, got_aabb)
    torch.cuda.synchronize()
    for k, (M, mi, op) in enumerate(insts):
        oracle.voxelize_model(want, models[mi], M, op, aabb0[k])
    assert want.any()
    assert np.array_equal(export_r8(G), want)
    assert np.array_equal(got_aabb.cpu().numpy(), aabb0)


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_tile_shapes(vxl, ctx, shape, noalloc):
    rng = np.random.default_rng(sum(shape))
    model = vox_cases.random_model(rng, *shape)
    model.flat[0] = 200
    insts = [(vox_cases.world_matrix(rng, 0.5, 8.0), 0, vxl.OP_SET) for _ in range(3)]
    insts.append((vox_cases.world_matrix(rng, -1.0, 0.5), 0, vxl.OP_SET))  # partly outside
    check(vxl, ctx, 100, [model], insts, noalloc)


@pytest.mark.parametrize("scale", [0.25, 1.7, 4.0])
def test_scaled(vxl, ctx, scale):
    rng = np.random.default_rng(int(scale * 100))
    model = vox_cases.random_model(rng, 20, 18, 11)
    insts = []
    for _ in range(4):
        m = vox_cases.world_matrix(rng, 1.0, 9.0).reshape(4, 4).copy()
        m[:3, :3] *= np.float32(scale)
        insts.append((m.reshape(16), 0, vxl.OP_SET))
    check(vxl, ctx, 128, [model], insts)


@pytest.mark.parametrize("count", [2, 70, 1500])
def test_crowded_order(vxl, ctx, count):
    """Sets and clears on top of one another, past one ordering segment at 1500."""
    rng = np.random.default_rng(count)
    models = [vox_cases.random_model(rng, *s) for s in ((7, 9, 8), (12, 5, 17))]
    insts = []
    for i in range(count):
        op = vxl.OP_SET if rng.random() < 0.6 or i == 0 else vxl.OP_CLEAR
        insts.append((vox_cases.world_matrix(rng, 0.0, 4.0), int(rng.integers(0, 2)), op))
    check(vxl, ctx, 48, models, insts)
