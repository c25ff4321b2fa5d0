"""The bounds of placements whose cells leave the range of an int, where a conversion saturates (and makes NaN 0): they
hold every mapped voxel, however the voxels are shared out over warps and blocks."""
import numpy as np
import pytest

from tests import vox_cases
from tests.gpu_util import dev

pytestmark = pytest.mark.gpu
F = np.float32


def _bounds(model, m):
    """min and max cell of the set voxels: ivec3((o + x*dx + y*dy + z*dz) * 10) in float32."""
    z, y, x = (a.astype(F) for a in np.nonzero(model >= 16))
    with np.errstate(all="ignore"):
        d = m * F(0.1)
        w = [((m[12 + a] + d[a] * x) + d[4 + a] * y) + d[8 + a] * z for a in range(3)]
        c = [np.where(np.isnan(v), F(0), v * F(10.0)) for v in w]
        c = [np.where(v >= F(2.0 ** 31), 2 ** 31 - 1, np.where(v < F(-2.0 ** 31), -2 ** 31, np.clip(v, F(-2e9), F(2e9)).astype(np.int64)))
             for v in c]
    return np.array([v.min() for v in c] + [v.max() for v in c], np.int64)


@pytest.mark.parametrize("noalloc", [False, True])
@pytest.mark.parametrize("shape", [(3, 2, 2), (20, 18, 11), (40, 3, 70)])
def test_far_placements(vxl, ctx, shape, noalloc):
    import torch

    rng = np.random.default_rng(sum(shape))
    model = vox_cases.random_model(rng, *shape)
    mats = []
    for value in (np.inf, -np.inf, 1e20, -1e20):
        for at in (0, 5, 10, 12, 13, 14):
            m = vox_cases.world_matrix(rng, 0.5, 6.0).copy()
            m[at] = value
            mats.append(m)
    for scale in (3e7, 6e7, 1.5e8):  # some voxels beyond 2^31 cells, some not
        m = vox_cases.world_matrix(rng, 0.5, 6.0).reshape(4, 4).copy()
        m[:3, :3] *= F(scale)
        mats.append(m.reshape(16))
    start = np.tile(np.array([49, 49, 49, 0, 0, 0], np.int32), (len(mats), 1))
    got, d = dev(start), dev(model)
    G = vxl.Grid(ctx, 100, 100, 100)
    mdesc, insts = [(d.data_ptr(),) + model.shape[::-1]], [(m, 0, vxl.OP_SET) for m in mats]
    if noalloc:
        vxl.voxelize_noalloc(G.describe(), mdesc, insts, got)
    else:
        vxl.voxelize(ctx, G, mdesc, insts, got)
    torch.cuda.synchronize()
    b = np.array([_bounds(model, np.asarray(m, F)) for m in mats])
    want = np.concatenate([np.minimum(b[:, :3], 49), np.maximum(b[:, 3:], 0)], 1)
    assert np.array_equal(got.cpu().numpy(), want), np.argwhere(got.cpu().numpy() != want)[:5]
