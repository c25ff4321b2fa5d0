"""The pooled marchers where a step is longer than the grid: the positions a ray tests are then rounded to whole cells and
more, and every one of them that lands in the grid is tested as the one before it. Records against the oracle, bit for bit."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import assert_recs_equal, dev, empty, grid_from_r8, rec_buffer, recs_np

pytestmark = pytest.mark.gpu
DIMS = (510, 130, 66)
F = np.float32


def _grid():
    f = np.random.default_rng(1).random(DIMS[::-1]) < 0.05
    f[:, :, 500:] = True  # slabs that rays enter and leave by
    f[:, :, :10] = True
    return oracle.fine_to_r8(f)


def _rays(rng, n, mode, lo, hi):
    """Directions of length 2^lo to 2^hi, aimed so that test k of the batch (the last one mostly) lands at a face."""
    step0 = (0.5, 2.5)[mode - 1]
    o = rng.uniform(1, np.array(DIMS) - 1.0, (n, 3))
    d = np.zeros((n, 3))
    d[:, 0] = rng.choice([-1.0, 1.0], n) * 2.0 ** rng.uniform(lo, hi, n)
    d = d.astype(F)
    k = rng.choice([3, 3, 3, 1, 2, 7, 11], n)
    face = np.where(rng.random(n) < 0.5, DIMS[0], 0) + rng.integers(-12, 4, n)
    o[:, 0] = face - k * (step0 * d[:, 0].astype(np.float64))
    o = np.clip(o, 128.0 - 2.0 ** 30, 2.0 ** 30 - 128.0)
    return np.concatenate([o.astype(F), d, np.full((n, 1), 128.0, F)], 1)


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("lo,hi", [(17, 20), (20, 24), (24, 28)])
def test_long_steps(vxl, ctx, mode, lo, hi):
    import torch

    g = _grid()
    rays = _rays(np.random.default_rng(lo), 20000, mode, lo, hi)
    # three fused steps of 2^24 end two cells beyond where three rounded ones do
    rays[0] = [50331532.0, 100.5, 50.5, -33554014.0, 0.0, 0.0, 128.0]
    rec = rec_buffer(len(rays))
    vxl.trace_rays(ctx, grid_from_r8(vxl, ctx, g), dev(rays), len(rays), mode, rec)
    torch.cuda.synchronize()
    want = oracle.trace_rays(g, rays, mode=mode)
    if mode == 1:
        assert (want["vx"][0], want["t"][0], want["steps"][0]) == (508, 2.0, 4)
    assert 0.1 < (want["flags"] & 1).mean() < 1.0
    assert_recs_equal(recs_np(rec), want)


def test_long_reflections(vxl, ctx):
    """A reflected direction is as long as its noise makes it."""
    import torch

    g = _grid()
    n, rng = 20000, np.random.default_rng(2)
    nz = (2.0 ** rng.uniform(20, 27, n)).astype(F)
    noise = np.stack([np.zeros(n), np.zeros(n), np.full(n, 0.5), nz], 1).astype(F)
    vr = np.zeros((n, 3), F)
    vr[:, 0] = rng.choice([-1.0, 1.0], n)
    face = np.where(rng.random(n) < 0.5, DIMS[0], 0) + rng.integers(-12, 4, n)
    step = 0.5 * (1.0 + nz.astype(np.float64) * 0.5)
    wcp = np.stack([face - 3 * step * vr[:, 0], rng.uniform(1, 129, n), rng.uniform(1, 65, n)], 1).astype(F)
    nrm, rough = np.zeros((n, 3), F), np.zeros(n, F)
    want, _ = oracle.light_reflection(g, wcp, nrm, vr, rough, noise)
    out = empty(n, torch.float32)
    vxl.light_reflection(ctx, grid_from_r8(vxl, ctx, g), dev(wcp), dev(nrm), dev(vr), dev(rough), dev(noise), n, out)
    torch.cuda.synchronize()
    assert 0.1 < (want != 256.0).mean() < 1.0
    assert np.array_equal(out.cpu().numpy(), want)


@pytest.mark.parametrize("mode", [1, 2])
def test_along_the_faces(vxl, ctx, mode):
    """Rays within half a cell of the faces of a long grid, where positions are rounded most, along them and across."""
    import torch

    dims, rng, n = (32000, 34, 30), np.random.default_rng(9 + mode), 20000
    g = np.zeros((15, 17, 16000), np.uint8)
    for at in (slice(0, 200), slice(15800, 16000)):
        g[:, :, at] = rng.choice(np.array([0, 0, 0, 0, 0, 0, 0, 1, 64, 255], np.uint8), (15, 17, 200))
    off = rng.choice([0.0, 1.0 / 64, 1.0 / 32, 3.0 / 64, 0.2, 0.4999, 0.5, -1.0 / 64, -0.3], (n, 3))
    o = np.where(rng.random((n, 3)) < 0.5, off, np.array(dims) - off)
    inner = rng.random((n, 3)) < 0.5
    o[inner] = (rng.random((n, 3)) * dims)[inner]
    o[:, 0] = np.where(rng.random(n) < 0.5, np.minimum(o[:, 0], 390.0), np.maximum(o[:, 0], 31610.0))
    d = rng.normal(size=(n, 3)) * rng.choice([0.0, 1.0, 1.0, 1e-3], (n, 3))
    d[np.abs(d).max(1) == 0.0] = [1.0, 0.0, 0.0]
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d, rng.choice([128.0, 256.0, 40.0], (n, 1))], 1).astype(F)
    rec = rec_buffer(n)
    vxl.trace_rays(ctx, grid_from_r8(vxl, ctx, g), dev(rays), n, mode, rec)
    torch.cuda.synchronize()
    want = oracle.trace_rays(g, rays, mode=mode)
    assert 0.1 < (want["flags"] & 1).mean() < 1.0
    assert_recs_equal(recs_np(rec), want)


@pytest.mark.parametrize("dims", [(6, 10, 14), (40, 34, 52)])
@pytest.mark.parametrize("n", [1, 33, 129, 20000])
def test_records_of_rays_that_leave(vxl, ctx, dims, n):
    """Small grids, which rays leave in their fine part or their coarse one, before their first test or at their last:
    sparse rays of every length and the light passes' records, which name the last position all the same."""
    import torch

    rng = np.random.default_rng(n + dims[0])
    g = oracle.fine_to_r8(rng.random(dims[::-1]) < 0.01)
    G = grid_from_r8(vxl, ctx, g)
    o = rng.uniform(-8.0, np.array(dims) + 8.0, (n, 3))
    d = rng.normal(size=(n, 3)) * rng.choice([0.0, 1.0, 1.0, 4.0], (n, 3))
    dist = rng.choice([128.0, 256.0, 0.0, -1.0, 15.75, 16.0, 16.5, 17.0, 17.5, 18.0, 20.0, 22.5, 163.0, 164.0, np.inf], (n, 1))
    rays = np.concatenate([o, d, dist], 1).astype(F)
    rec = rec_buffer(n)
    vxl.trace_rays(ctx, G, dev(rays), n, 1, rec)
    torch.cuda.synchronize()
    assert_recs_equal(recs_np(rec), oracle.trace_rays(g, rays, mode=1))
    wcp, nrm = o.astype(F), np.eye(3, dtype=F)[rng.integers(0, 3, n)]
    depth, noise = rng.uniform(0, 0.3, n).astype(F), rng.random((n, 4)).astype(F)
    rough, vr = rng.uniform(0.05, 1, n).astype(F), rng.normal(size=(n, 3)).astype(F)
    rec2, rec1 = rec_buffer(2 * n), rec_buffer(n)
    a, b, c = (empty(n, torch.float32) for _ in range(3))
    vxl.light_ambient(ctx, G, dev(wcp), dev(nrm), dev(depth), dev(noise), n, a, b, rec2)
    vxl.light_reflection(ctx, G, dev(wcp), dev(nrm), dev(vr), dev(rough), dev(noise), n, c, rec1)
    torch.cuda.synchronize()
    assert_recs_equal(recs_np(rec2), oracle.light_ambient(g, wcp, nrm, depth, noise)[2].reshape(-1))
    assert_recs_equal(recs_np(rec1), oracle.light_reflection(g, wcp, nrm, vr, rough, noise)[1].reshape(-1))
