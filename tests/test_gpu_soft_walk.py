"""The batched walk of the soft pass against the FP64 model: grids smaller than a batch, walks to the 256-cell cap, rays
that enter from the padding cells beyond the data, directions with zero components, and values past an opaque stack
that the walk must not touch. Tolerances as in test_gpu_soft.py."""
import numpy as np
import pytest

import oracle
from tests.gpu_util import dev

pytestmark = pytest.mark.gpu


def _run(vxl, ctx, vox, pos, nrm, kw):
    import torch

    n = len(pos)
    P = vxl.make_soft_params(**kw)
    soft, dp, dn = dev(vox), dev(pos), dev(nrm)
    img, light = (torch.empty((n, 3), dtype=torch.float32, device="cuda") for _ in range(2))
    vxl.trace_soft_fwd(ctx, soft, dp, dn, n, P, img, light)
    gi = torch.linspace(-1.0, 1.0, 3 * n, device="cuda").view(n, 3).contiguous()
    grad = torch.zeros_like(soft)
    vxl.trace_soft_bwd(ctx, soft, dp, dn, n, P, gi, light, grad)
    torch.cuda.synchronize()
    want, wgrad = oracle.soft_render(vox, pos, nrm, oracle.make_soft_params(**kw), grad_image=gi.cpu().numpy())
    return img.cpu().numpy(), want, grad.cpu().numpy(), wgrad


def _surface(dims, n, rng):
    """Points on the faces of cells of the grid, the outermost cells among them."""
    axis, sign = rng.integers(0, 3, n), rng.choice([-1.0, 1.0], n)
    nrm = np.zeros((n, 3), np.float32)
    nrm[np.arange(n), axis] = sign
    cell = np.stack([rng.integers(0, d, n) for d in dims], 1)
    edge = rng.random(n) < 0.4
    cell[edge, axis[edge]] = np.where(sign[edge] > 0, np.array(dims)[axis[edge]] - 1, 0)
    pos = cell + rng.uniform(0.1, 0.9, (n, 3))
    pos[np.arange(n), axis] = cell[np.arange(n), axis] + (sign > 0)
    return pos.astype(np.float32), nrm


@pytest.mark.parametrize("dims", [(2, 2, 2), (4, 6, 10), (34, 18, 22), (300, 6, 300)])
@pytest.mark.parametrize("light,length,n_ao", [((0.3, 0.8, 0.5), 24.0, 5), ((0.0, 1.0, 0.0), 8.0, 1), ((0.6, -0.0, 0.8), 300.0, 31),
                                               ((0.70710677, 1e-3, 0.70710677), 400.0, 3)])
def test_walk_matches_fp64(vxl, ctx, dims, light, length, n_ao):
    rng = np.random.default_rng(dims[0] + n_ao)
    vox = rng.random(dims[::-1] + (4,)).astype(np.float32)
    vox[..., 0] = rng.uniform(0.0, 0.05, dims[::-1])  # thin: walks run to their length, the bounds or the cap
    pos, nrm = _surface(dims, 77, rng)
    img, want, grad, wgrad = _run(vxl, ctx, vox, pos, nrm, dict(light_dir=light, length=length, n_ao=n_ao, seed=5))
    assert np.abs(img - want).max() < 2e-5
    assert np.linalg.norm(grad - wgrad) <= 1e-3 * np.linalg.norm(wgrad)


@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_nothing_behind_an_opaque_stack_is_touched(vxl, ctx, value):
    import torch

    vox = np.full((32, 32, 32, 4), 0.5, np.float32)
    vox[..., 0] = 1.0
    vox[:, 10:, :, 0] = 0.0  # floor below y = 10, then air; a roof of 4 opaque layers from y = 13, wild values above
    vox[:, 13:17, :, 0] = 1.0
    vox[:, 17:, :, 1:] = value
    rng = np.random.default_rng(2)
    pos = np.stack([rng.uniform(14, 18, 40), np.full(40, 10.0), rng.uniform(14, 18, 40)], 1).astype(np.float32)
    nrm = np.tile(np.array([[0, 1, 0]], np.float32), (40, 1))
    P = vxl.make_soft_params(light_dir=(0.01, 1.0, 0.02), length=12.0, n_ao=0, seed=5)
    soft = dev(vox)
    img, light = (torch.empty((40, 3), dtype=torch.float32, device="cuda") for _ in range(2))
    vxl.trace_soft_fwd(ctx, soft, dev(pos), dev(nrm), 40, P, img, light)
    grad = torch.zeros_like(soft)
    vxl.trace_soft_bwd(ctx, soft, dev(pos), dev(nrm), 40, P, torch.ones_like(img), light, grad)
    torch.cuda.synchronize()
    assert torch.isfinite(img).all() and torch.isfinite(grad).all()
    assert float(light.abs().max()) < 1e-10
