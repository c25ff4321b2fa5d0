"""The structures derived from a grid's words (tile map, trace layout) against
a numpy restatement of their definition in include/vxl.h, at sizes around the
brick, row-pair and tile edges."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIMS = [(2, 2, 2), (4, 6, 8), (10, 2, 6), (62, 64, 66), (250, 30, 126), (256, 14, 18), (506, 12, 10)]


@pytest.fixture(scope="module")
def vxl():
    import voxelengine_gb300 as V

    V.build()
    return V


@pytest.fixture(scope="module")
def ctx(vxl):
    return vxl.Context(0)


def random_words(d, seed):
    """Brick words with voxels inside the grid only, as a dense bool volume and packed."""
    rng = np.random.default_rng(seed)
    occ = np.zeros((4 * d.bz, 4 * d.by, 4 * d.bx), bool)
    occ[: d.nz, : d.ny, : d.nx] = rng.random((d.nz, d.ny, d.nx)) < 0.02
    return occ, pack(occ)


def pack(occ):
    bz, by, bx = (s // 4 for s in occ.shape)
    b = occ.reshape(bz, 4, by, 4, bx, 4).transpose(0, 2, 4, 1, 3, 5).reshape(bz, by, bx, 64)
    return np.packbits(b, axis=-1, bitorder="little").view(np.uint64).reshape(bz, by, bx)


def want_tiles(words, d):
    t = np.zeros((2 * d.tz, 2 * d.ty, 2 * d.tx), bool)
    t[: d.bz, : d.by, : d.bx] = words != 0
    t = t.reshape(d.tz, 2, d.ty, 2, d.tx, 2).any(axis=(1, 3, 5)).reshape(-1)
    out = np.zeros(-(-t.size // 32) * 32, bool)
    out[: t.size] = t
    return np.packbits(out, bitorder="little").view(np.uint32)


def want_layout(occ, d):
    n = (d.nx, d.ny, d.nz)
    full = np.zeros((4 * d.trace_bz, 4 << d.trace_lby, 4 << d.trace_lbx), bool)
    full[4: 4 + d.nz, 4: 4 + d.ny, 4: 4 + d.nx] = occ[: d.nz, : d.ny, : d.nx]
    box = full[3: d.nz + 7, 3: d.ny + 7, 3: d.nx + 7]
    assert box.shape == tuple(v + 4 for v in reversed(n))
    box[[0, -1]] = True
    box[:, [0, -1]] = True
    box[:, :, [0, -1]] = True
    return pack(full)


def read(ptr, nbytes, dtype):
    import torch

    class Mem:
        __cuda_array_interface__ = dict(shape=(nbytes // 4,), typestr="<i4", data=(ptr, False), version=3)

    return torch.as_tensor(Mem(), device="cuda").cpu().numpy().view(dtype)


@pytest.mark.parametrize("dims", DIMS)
def test_grid(vxl, ctx, dims):
    import torch

    G = vxl.Grid(ctx, *dims)
    d = G.describe()
    occ, words = random_words(d, sum(dims))
    r8 = occ[: d.nz, : d.ny, : d.nx].reshape(d.nz // 2, 2, d.ny // 2, 2, d.nx // 2, 2).transpose(0, 2, 4, 1, 3, 5)
    r8 = np.packbits(r8.reshape(d.nz // 2, d.ny // 2, d.nx // 2, 8), axis=-1, bitorder="little")
    G.import_r8(torch.from_numpy(r8).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(read(d.words, d.words_bytes, np.uint64), words.reshape(-1))
    assert np.array_equal(read(d.tile_mask, d.tile_mask_bytes, np.uint32), want_tiles(words, d))
    assert np.array_equal(read(d.trace_words, d.trace_words_bytes, np.uint64), want_layout(occ, d).reshape(-1))


@pytest.mark.parametrize("dims,odd", [((10, 2, 6), 0), ((250, 30, 126), 1), ((62, 64, 66), 1)])
def test_caller_buffers(vxl, ctx, dims, odd):
    """vxl_voxelize_noalloc on buffers of the caller that hold anything, the
    layout 16- or only 8-byte aligned: every word is written, padding included."""
    import torch

    G = vxl.Grid(ctx, *dims)
    d = G.describe()
    occ, words = random_words(d, 1)
    t_words = torch.from_numpy(words.reshape(-1).view(np.int64)).cuda()
    t_mask = torch.full((d.tile_mask_bytes // 4,), -1, dtype=torch.int32, device="cuda")
    t_lay = torch.full((d.trace_words_bytes // 8 + 2,), -1, dtype=torch.int64, device="cuda")
    own = vxl.GridDesc()
    C.memmove(C.byref(own), C.byref(d), C.sizeof(d))
    own.words, own.tile_mask, own.trace_words = t_words.data_ptr(), t_mask.data_ptr(), t_lay.data_ptr() + 8 * odd
    model = torch.full((1, 1, 1), 20, dtype=torch.uint8, device="cuda")
    m = np.eye(4, dtype=np.float32)
    m[3, :3] = [0.05, 0.05, 0.05]  # the voxel at cell (0, 0, 0)
    vxl.voxelize_noalloc(own, [(model.data_ptr(), 1, 1, 1)], [(m.reshape(16), 0, vxl.OP_SET)])
    occ[0, 0, 0] = True
    words = pack(occ)
    assert np.array_equal(t_words.cpu().numpy().view(np.uint64), words.reshape(-1))
    assert np.array_equal(t_mask.cpu().numpy().view(np.uint32), want_tiles(words, d))
    lay = t_lay.cpu().numpy().view(np.uint64)
    n = d.trace_words_bytes // 8
    assert np.array_equal(lay[odd: odd + n], want_layout(occ, d).reshape(-1))
    rest = np.delete(lay, np.arange(odd, odd + n))
    assert (rest == np.uint64(0xFFFFFFFFFFFFFFFF)).all()
