"""Primary visibility where the entry depth of a box decides whether it is walked: boxes that overlap and contain one
another, scaled unevenly, mirrored, flattened, far from the camera, and around it. Bit for bit the oracle's."""
import numpy as np
import pytest

import oracle
from tests.test_gpu_primary import _assert_same, _run_primary, _volumes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["overlap", "uneven", "mirror", "flat", "far", "inside"])
def test_entry_depth(vxl, ctx, kind):
    from voxelengine_gb300 import scenes

    rng = np.random.default_rng(len(kind))
    vols = _volumes(8, 6, 8, 48)
    worlds, vol_of = [], []
    at = np.array([3000.0, 900.0, -2000.0]) if kind == "far" else np.zeros(3)
    for i in range(70):
        vi = int(rng.integers(0, len(vols)))
        R = scenes.rotation_matrix(rng)
        scale = np.ones(3)
        if kind == "uneven":
            scale = rng.uniform(0.2, 3.0, 3)
        elif kind == "mirror":
            scale = rng.choice([-1.0, 1.0], 3) * rng.uniform(0.5, 1.5)
        elif kind == "flat" and i % 3 == 0:
            scale[int(rng.integers(0, 3))] = rng.choice([1e-6, 1e-3])
        m = np.eye(4)
        m[:3, :3] = R * scale
        m[:3, 3] = at + rng.uniform(0.0, 4.0 if kind == "overlap" else 8.0, 3) - m[:3, :3] @ (0.05 * np.array(vols[vi].shape[::-1]))
        worlds.append(m.T.astype(np.float32).reshape(16))
        vol_of.append(vi)
    worlds, vol_of = np.array(worlds, np.float32), np.array(vol_of, np.int32)
    cam, tgt = at + np.array([4.0, 11.0, -5.0]), at + np.array([4.0, 3.0, 4.0])
    if kind == "far":
        cam = np.array([4.0, 11.0, -5.0])
    if kind == "inside":
        cam, tgt = np.array([4.0, 4.0, 4.0]), np.array([7.0, 3.0, 6.0])
    cam, tgt = cam.astype(np.float32), tgt.astype(np.float32)
    fov = dict(tan_half_fov=0.004) if kind == "far" else {}
    import torch

    if fov:  # a telescope's view
        n, W, H = 128 * 80, 128, 80
        vs = vxl.VolumeSet(ctx, vols)
        pos, nrm = (torch.empty(n * 3, dtype=torch.float32, device="cuda") for _ in range(2))
        depth = torch.empty(n, dtype=torch.float32, device="cuda")
        mat, inst = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
        vxl.trace_primary(ctx, vs, worlds, vol_of, cam, tgt, W, H, pos, nrm, depth, mat, inst, **fov)
        torch.cuda.synchronize()
        got = dict(pos=pos.cpu().numpy().reshape(n, 3), nrm=nrm.cpu().numpy().reshape(n, 3), depth=depth.cpu().numpy(),
                   material=mat.cpu().numpy(), instance=inst.cpu().numpy())
    else:
        W, H = 128, 80
        got = _run_primary(vxl, ctx, vols, worlds, vol_of, cam, tgt, W, H, 0)
    want = oracle.primary(vols, worlds, vol_of, cam, tgt, W, H, frame=0, **fov)
    _assert_same(got, want)
    assert (want["instance"] >= 0).mean() > 0.05
