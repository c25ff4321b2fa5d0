"""Primary visibility where a box's entry depth is computed less exactly than its hits' depths: scenes far from the origin,
whose coordinates are rounded, and placements that are nearly flat or sheared, whose inverses are. Such boxes are walked
all the same. Bit for bit the oracle's."""
import numpy as np
import pytest

import oracle
from tests.test_gpu_primary import _assert_same, _run_primary, _volumes

pytestmark = pytest.mark.gpu


def _scene(rng, off, scale, flat, shear):
    from voxelengine_gb300 import scenes

    vols = _volumes(8, 5, 4, 40)
    worlds, vol_of = [], []
    for _ in range(150):
        vi = int(rng.integers(0, 5))
        R = scenes.rotation_matrix(rng) * scale * 10.0 ** rng.uniform(flat, 0.0, 3)
        if shear:
            R[:, 0] = R[:, 1] + R[:, 0] * 10.0 ** rng.uniform(-4.0, 0.0)
        m = np.eye(4)
        m[:3, :3] = R
        m[:3, 3] = off + scale * rng.uniform(0.0, 5.0, 3) - R @ (0.05 * np.array(vols[vi].shape[::-1]))
        worlds.append(m.T.astype(np.float32).reshape(16))
        vol_of.append(vi)
    return vols, np.array(worlds, np.float32), np.array(vol_of, np.int32)


@pytest.mark.parametrize("off,scale,flat,shear", [(1.3e5, 1.0, 0.0, False), (4.5e5, 1.0, 0.0, False), (1e6, 5.0, 0.0, False),
                                                  (1.7e4, 0.02, 0.0, False), (6e4, 0.03, 0.0, False), (1.0, 1.0, -5.0, False),
                                                  (10.0, 1.0, -1.0, True), (1e5, 1.0, -2.0, False)])
@pytest.mark.parametrize("seed", [0, 1])
def test_far_and_ill_conditioned(vxl, ctx, off, scale, flat, shear, seed):
    rng = np.random.default_rng(seed)
    at = np.array([1.0, 0.3, -0.7]) * off
    vols, worlds, vol_of = _scene(rng, at, scale, flat, shear)
    cam = (at + scale * np.array([2.5, 6.0, -4.0])).astype(np.float32)
    tgt = (at + scale * np.array([2.5, 2.0, 2.5])).astype(np.float32)
    W, H = 160, 100
    got = _run_primary(vxl, ctx, vols, worlds, vol_of, cam, tgt, W, H, 0)
    want = oracle.primary(vols, worlds, vol_of, cam, tgt, W, H, frame=0)
    assert (want["instance"] >= 0).mean() > 0.05
    _assert_same(got, want)
