"""A model of more than 2^24 voxels along z, whose z coordinates are no longer all floats: each is rounded as the
conversion of the whole number is, not as a count that goes up in floats."""
import numpy as np
import pytest

from tests.test_gpu_voxel_tiles import check

pytestmark = pytest.mark.gpu
F = np.float32


def _scale(z):
    """A z scale for which the cells of the coordinates z and z + 2 differ."""
    m = F(29.9999 / z)
    for _ in range(1 << 16):
        m = np.nextafter(m, F(1))
        a, b = (int((m * F(0.1)) * F(v) * F(10.0)) for v in (z, z + 2))
        if a != b:
            return m
    raise AssertionError("no such scale")


@pytest.mark.parametrize("noalloc", [False, True])
def test_coordinates_beyond_2_24(vxl, ctx, noalloc):
    n = (1 << 24) + 600
    model = np.zeros((n, 1, 1), np.uint8)
    model[(1 << 24) + 3] = 200  # as a float 2^24 + 4; counted up from 2^24 + 1 by twos 2^24 + 2
    model[5 :: 1 << 20] = 200
    m = np.eye(4, dtype=F)
    m[2, 2] = _scale((1 << 24) + 2)
    m[3, :3] = [0.25, 0.25, 0.0]
    check(vxl, ctx, 64, [model], [(m.reshape(16), 0, vxl.OP_SET)], noalloc)
