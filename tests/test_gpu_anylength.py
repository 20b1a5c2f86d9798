"""Dipole field on lattices whose edges are not powers of two (and of FP64
state), against the oracle's lattice sum: every butterfly radix the transforms
use, single rows and columns, odd row counts, one layer to more than are
unrolled, and a unit cell without the tensor parities the layer sum needs.

Tolerances: a transform of N points loses about log2(N) rounding errors of
its precision, so fields agree to well within 1e-5 (FP32, unit roundoff
6e-8) and 1e-11 (FP64) of their norm."""
import numpy as np
import pytest

import oracle as O
from helpers import random_spins, rel_err

pytestmark = pytest.mark.gpu

TOL = {"f32": 1e-5, "f64": 1e-11}


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


def _compare(M, dims, precision, trunc=12, cell=None):
    n = int(np.prod(dims))
    s = random_spins(n, 91, lengths=True)
    ss = M.SpinSystem(*dims, precision=precision)
    ss.setSpinArrays(*s)
    dip = M.Dipole(ss)
    dip.setStrength(0.3)
    dip.setTruncation(trunc)
    kw = {}
    if cell is not None:
        dip.setUnitCell(cell[0:3], cell[3:6], cell[6:9])
        kw["ABC"] = cell
    dip.apply(ss)
    h = np.stack(ss.fieldArrays("Dipole"))
    o = O.SpinSystem(*dims)
    o.set_spins(*s)
    O.LongRange(*dims, O.dipole_tensor(*dims, gmax=(trunc,) * 4, **kw)).apply(o, 0.3)
    assert rel_err(h, o.field("Dipole")) <= TOL[precision]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("dims", [(9, 10, 1), (11, 13, 2), (17, 19, 3), (23, 29, 1), (31, 62, 2), (30, 25, 4),
                                  (84, 45, 5), (36, 14, 6), (49, 22, 7), (200, 26, 8), (12, 10, 9), (6, 15, 33),
                                  (2, 3, 2), (1, 6, 2), (6, 1, 1), (1, 1, 3), (5, 241 - 1, 1)])
def test_periodic_field(M, dims, precision):
    _compare(M, dims, precision)


@pytest.mark.parametrize("dims", [(32, 32, 1), (64, 128, 4), (256, 16, 8)])
def test_periodic_field_powers_of_two_fp64(M, dims):
    _compare(M, dims, "f64")


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("dims", [(20, 16, 8), (9, 16, 16), (33, 32, 1), (16, 32, 16), (40, 64, 3), (8, 64, 7),
                                  (64, 128, 5), (300, 128, 2), (12, 256, 6), (7, 512, 4), (2, 512, 8)])
def test_power_of_two_rows_of_y(M, dims, precision):
    """The (y,z) pass for power-of-two Py: every width, layer counts in turn,
    few and many CTAs (few: large CTAs of several items per thread)."""
    _compare(M, dims, precision)


@pytest.mark.parametrize("precision", ["f32", "f64"])
def test_sheared_cell_keeps_the_full_tensor(M, precision):
    _compare(M, (12, 10, 3), precision, cell=(1, 0, 0, 0.3, 1, 0, 0.2, 0.1, 1))


@pytest.mark.parametrize("dims,precision", [((9, 31, 5), "f32"), ((30, 13, 1), "f32"), ((16, 6, 9), "f32"),
                                            ((128, 58, 4), "f32"), ((12, 17, 3), "f64"), ((7, 64, 6), "f64")])
def test_layer_tensors(M, dims, precision):
    """LongRange2D over the same passes: prime rows, one layer, layer counts
    off the four that are loaded together; the field on its own and inside
    captured steps (whose inverse x pass runs in the step)."""
    nx, ny, nz = dims
    r = np.random.default_rng(92)
    T = r.normal(size=(nz, nz, 9, ny, nx)) / (nx * ny)
    src, dst = r.uniform(0.5, 1.5, nz), r.uniform(0.5, 1.5, nz)
    s = random_spins(nx * ny * nz, 93)
    res = []
    for captured in (False, True):
        ss = M.SpinSystem(*dims, precision=precision)
        ss.setSpinArrays(*s, np.ones(nx * ny * nz))
        ss.setAlpha(0.1)
        ss.setTimeStep(0.01)
        ex = M.Exchange(ss)
        ex.addPaths(*O.nn_paths(*dims, pbc=(1, 1, 0)))
        op = M.LongRange2D(ss)
        op.setNewDataRequired(False)
        for i in range(nz):
            for j in range(nz):
                for q, ab in enumerate(("XX", "XY", "XZ", "YX", "YY", "YZ", "ZX", "ZY", "ZZ")):
                    op.setTensorArray(i + 1, j + 1, ab, T[i, j, q].reshape(-1))
        for z in range(nz):
            op.setSourceMomentScale(z + 1, src[z])
            op.setDestinationFieldScale(z + 1, dst[z])
        op.setCompileRequired(True)
        op.apply(ss)
        h = np.stack(ss.fieldArrays("LongRange2D"))
        ref = O.longrange2d_apply(s.reshape(3, nz, ny, nx), T, src, dst)
        assert rel_err(h, np.asarray(ref).reshape(3, -1)) <= TOL[precision]
        llg = M.LLG.new("Quaternion")
        if captured:
            M.run(ss, [ex, op], llg, 5)
        else:
            for _ in range(5):
                ss.resetFields()
                ex.apply(ss)
                op.apply(ss)
                ss.sumFields()
                llg.apply(ss)
        res.append(np.stack(ss.spinArrays()[:3]))
    np.testing.assert_array_equal(res[0], res[1])
