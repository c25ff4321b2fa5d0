"""The instance and entity tables of the binding hold what their fields assigned one by one hold, in every form of input
that the fields take; what the fields refuse stays refused."""
import ctypes as C

import numpy as np
import pytest
import torch

import voxelengine_gb300 as V


def _by_field(instances):
    arr = (V.Instance * max(1, len(instances)))()
    for i, (m, mi, op) in enumerate(instances):
        arr[i].matrix[:] = [float(x) for x in np.asarray(m, np.float32).reshape(16)]
        arr[i].model, arr[i].op = mi, op
    return arr


M = np.random.default_rng(3).normal(size=16) * 1e3
FORMS = {
    "float32": lambda k: M.astype(np.float32) + k,
    "float64": lambda k: M + k,
    "4x4": lambda k: (M + k).reshape(4, 4),
    "fortran": lambda k: np.asfortranarray((M + k).reshape(4, 4)),
    "strided": lambda k: np.repeat(M + k, 2)[::2],
    "list": lambda k: [float(x) + k for x in M],
    "ints": lambda k: list(range(k, k + 16)),
    "tensor": lambda k: torch.from_numpy(M + k),
    "odd one": lambda k: (M + k).reshape(4, 4) if k == 1 else M + k,
}


@pytest.mark.parametrize("form", sorted(FORMS))
@pytest.mark.parametrize("n", [0, 1, 3, 9])
def test_instance_table(form, n):
    ins = [(FORMS[form](k), k if k else np.int64(7), (1 << 32) + 1 if k == 2 else 1) for k in range(n)]
    assert bytes(V._instances(ins)) == bytes(_by_field(ins))


def test_entity_table():
    ents = [(M + k, FORMS["list"](k), (k, 0.1, -2), k) for k in range(7)]
    arr = (V.Entity * 7)()
    for i, (pw, w, pv, mi) in enumerate(ents):
        arr[i].prev_world[:], arr[i].world[:] = [[float(x) for x in np.asarray(q, np.float32)] for q in (pw, w)]
        arr[i].pivot[:], arr[i].model = [float(x) for x in np.asarray(pv, np.float32)], mi
    assert bytes(V._entities(ents)) == bytes(arr)
    assert C.sizeof(V.Entity) == V.ENTITY_DTYPE.itemsize and C.sizeof(V.Instance) == V.INSTANCE_DTYPE.itemsize


@pytest.mark.parametrize("bad", [(M[:15], 0, 1), (M, 1.0, 1), (M, 0), (M, 0, 1, 2), ("x", 0, 1), (M, "0", 1)])
def test_refused(bad):
    for table in (_by_field, V._instances):
        for ins in ([bad], [(M, 0, 1)] * 8 + [bad], [bad] + [(M, 0, 1)] * 8):
            with pytest.raises((TypeError, ValueError)):
                table(ins)
