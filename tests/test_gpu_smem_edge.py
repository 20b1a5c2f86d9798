"""Layer tensors whose lines take nearly the 48 KB of shared memory that need no
limit set, which hold the kernel's static arrays too: the field against the
oracle's layer-pair convolution (FP32 1e-5, FP64 1e-11 of its norm, as elsewhere)."""
import numpy as np
import pytest

import oracle as O
from helpers import random_spins, rel_err

pytestmark = pytest.mark.gpu

AB = ("XX", "XY", "XZ", "YX", "YY", "YZ", "ZX", "ZY", "ZZ")


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


# the first two take 47.7 KB of dynamic and 0.5 KB of static shared memory
@pytest.mark.parametrize("dims,precision", [((1, 62, 16), "f32"), ((6, 62, 16), "f32"), ((4, 75, 13), "f32"),
                                            ((5, 30, 16), "f64"), ((3, 62, 8), "f64"), ((2, 60, 16), "f32"),
                                            ((2, 124, 8), "f32"), ((2, 58, 17), "f32")])
def test_layer_tensors(M, dims, precision):
    nx, ny, nz = dims
    r = np.random.default_rng(92)
    T = r.normal(size=(nz, nz, 9, ny, nx)) / (nx * ny)
    s = random_spins(nx * ny * nz, 93)
    ss = M.SpinSystem(*dims, precision=precision)
    ss.setSpinArrays(*s)
    op = M.LongRange2D(ss)
    op.setNewDataRequired(False)
    for i in range(nz):
        for j in range(nz):
            for q, ab in enumerate(AB):
                op.setTensorArray(i + 1, j + 1, ab, T[i, j, q].reshape(-1))
    op.setCompileRequired(True)
    op.apply(ss)
    h = np.stack(ss.fieldArrays("LongRange2D"))
    ref = O.longrange2d_apply(s.reshape(3, nz, ny, nx), T, np.ones(nz), np.ones(nz))
    assert rel_err(h, np.asarray(ref).reshape(3, -1)) <= (1e-5 if precision == "f32" else 1e-11)
