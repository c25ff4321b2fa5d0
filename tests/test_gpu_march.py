"""The pooled marchers (march_pool.cuh) and DDA rays against the oracle, bit for bit: pools of every fill, positions on the
quarter-cell boundaries of the fetch, outside the grid and on its way out, lengths around the parts' limits."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import assert_recs_equal, dev, empty, grid_from_r8, rec_buffer, recs_np, same_bits

pytestmark = pytest.mark.gpu


def _grid(dims, seed):
    f = np.random.default_rng(seed).random(dims[::-1]) < 0.02
    return oracle.fine_to_r8(f)


def _rays(dims, n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-6.0, np.array(dims) + 6.0, (n, 3))
    d = rng.normal(size=(n, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    kind = rng.integers(0, 8, n)
    q = kind < 3
    o[q] = np.round(o[q] * 4.0) / 4.0
    axis = (kind == 1) | (kind == 4)
    d[axis] = np.eye(3)[rng.integers(0, 3, axis.sum())] * rng.choice([-1.0, 1.0], (axis.sum(), 1))
    d[kind == 2] = np.round(d[kind == 2] * 4.0) / 4.0
    d[kind == 5] *= rng.choice([1e-3, 3.0, 1e30, 1e38], ((kind == 5).sum(), 1))
    o[kind == 6] = rng.choice([-2.0, -1.75, -0.25, -0.0, 0.0, 1e-30, 0.25], ((kind == 6).sum(), 3))
    dist = rng.choice([128.0, 256.0, 0.0, -1.0, 15.75, 16.0, 16.5, 17.5, 17.75, 100.3, 164.0, 1e30, np.inf, np.nan], n)
    rays = np.concatenate([o, d, dist[:, None]], 1).astype(np.float32)
    bad = rng.integers(0, n, max(1, n // 50))
    rays[bad, rng.integers(0, 6, len(bad))] = rng.choice([np.nan, np.inf, -np.inf, 2.0 ** 30], len(bad))
    return rays


# 700000 rays: the largest pools (below 622592 rays on this GPU they are smaller)
@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 4097, 700000])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("dims", [(6, 10, 14), (130, 66, 34)])
def test_ray_records(vxl, ctx, dims, mode, n):
    import torch

    if n == 700000 and dims[0] < 100:
        dims = (96, 96, 96)
    g = _grid(dims, 7)
    rays = _rays(dims, n, n + mode)
    rec = rec_buffer(n)
    vxl.trace_rays(ctx, grid_from_r8(vxl, ctx, g), dev(rays), n, mode, rec)
    torch.cuda.synchronize()
    assert_recs_equal(recs_np(rec), oracle.trace_rays(g, rays, mode=mode), "mode %d" % mode)


def test_dda_records_of_a_large_grid(vxl, ctx):
    """Beyond 64 MiB of words the kernel keeps the current brick in registers."""
    import torch

    rng = np.random.default_rng(3)
    g = np.zeros((65, 65, 16000), np.uint8)
    for at in (slice(0, 40), slice(15960, 16000)):
        g[:, :, at] = rng.choice(np.array([0, 0, 0, 0, 0, 1, 64, 130, 255], np.uint8), (65, 65, 40))
    rays = _rays((130, 130, 130), 4097, 9)
    rays[::2, 0] += np.float32(31870.0)
    G = grid_from_r8(vxl, ctx, g)
    assert G.describe().words_bytes > 64 << 20
    rec = rec_buffer(len(rays))
    vxl.trace_rays(ctx, G, dev(rays), len(rays), 0, rec)
    torch.cuda.synchronize()
    assert_recs_equal(recs_np(rec), oracle.trace_rays(g, rays, mode=0))


@pytest.mark.parametrize("n", [1, 33, 5000, 640000])
def test_light_passes_without_records(vxl, ctx, n):
    import torch

    dims = (96, 64, 80)
    g = _grid(dims, 5)
    G = grid_from_r8(vxl, ctx, g)
    rng = np.random.default_rng(n)
    axes = np.concatenate([np.eye(3), -np.eye(3), np.zeros((1, 3))]).astype(np.float32)
    wcp = rng.uniform(-4, 100, (n, 3)).astype(np.float32)
    wcp[rng.integers(0, n, n // 100)] = np.nan
    nrm = axes[rng.integers(0, 7, n)]
    depth = rng.uniform(0, 0.3, n).astype(np.float32)
    noise = rng.random((n, 4)).astype(np.float32)
    rough = rng.uniform(0.05, 1, n).astype(np.float32)
    vr = rng.normal(size=(n, 3)).astype(np.float32)
    sh, irr, _ = oracle.light_ambient(g, wcp, nrm, depth, noise)
    t, _ = oracle.light_reflection(g, wcp, nrm, vr, rough, noise)
    d_sh, d_irr, d_t = (empty(n, torch.float32) for _ in range(3))
    vxl.light_ambient(ctx, G, dev(wcp), dev(nrm), dev(depth), dev(noise), n, d_sh, d_irr)
    vxl.light_reflection(ctx, G, dev(wcp), dev(nrm), dev(vr), dev(rough), dev(noise), n, d_t)
    torch.cuda.synchronize()
    assert np.array_equal(d_sh.cpu().numpy(), sh)
    assert same_bits(d_irr.cpu().numpy(), irr).all()
    assert same_bits(d_t.cpu().numpy(), t).all()
    lights = [(rng.uniform(0.0, 9.0, 3).astype(np.float32), float(rng.uniform(0.5, 5.0)), bool(l % 2)) for l in range(5)]
    wpos = (wcp * np.float32(0.1)).astype(np.float32)
    lit = torch.full((n,), -1, dtype=torch.int64, device="cuda")
    vxl.light_points(ctx, G, dev(wpos), dev(nrm), dev(noise), n, lights, lit)
    torch.cuda.synchronize()
    want = np.zeros(n, np.uint64)
    for l, (lp, r, spot) in enumerate(lights):
        s, _ = oracle.light_point(g, wpos, nrm, noise, lp, r, spot=spot, init=np.full(n, -7.0, np.float32))
        want |= np.where(s == 1.0, np.uint64(1) << np.uint64(l), np.uint64(0))
    assert np.array_equal(lit.cpu().numpy().view(np.uint64), want)
