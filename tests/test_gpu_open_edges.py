"""Open films in captured steps: lines half empty or more, where the padded ends
are left out of the transforms and of the site loop.  Edge lengths that fill
half a line, end just past its quarter and on single columns; every CTA share of
the fused x pass.  The captured steps equal the single calls bit for bit, and the
field of the last state is the direct sum (FP32, unit roundoff 6e-8, 15
butterfly levels: well within 1e-5 of its norm)."""
import numpy as np
import pytest

import oracle as O
from helpers import random_spins, rel_err

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


@pytest.mark.parametrize("llg", ["Cartesian", "Quaternion"])
@pytest.mark.parametrize("dims", [(16, 12, 2), (9, 8, 3), (32, 6, 1), (17, 10, 4), (64, 4, 2), (33, 160, 6), (128, 2, 3),
                                  (65, 64, 16), (127, 6, 1), (1, 8, 2), (40, 64, 24), (5, 128, 40)])
def test_open_steps(M, dims, llg):
    n = int(np.prod(dims))
    s = random_spins(n, 77)
    res = []
    for captured in (False, True):
        ss = M.SpinSystem(*dims)
        ss.setSpinArrays(*s)
        ss.setAlpha(0.1)
        ss.setTimeStep(0.01)
        ex = M.Exchange(ss)
        ex.addPaths(*O.nn_paths(*dims, pbc=(0, 0, 0)))
        ani = M.Anisotropy(ss)
        ani.addMany(np.arange(n), np.tile([0, 0, 1.0], (n, 1)), np.full(n, 0.2))
        dip = M.Dipole(ss)
        dip.setOpen(True, True, True)
        dip.setStrength(0.3)
        ops, l = [ex, ani, dip], M.LLG.new(llg)
        if captured:
            M.run(ss, ops, l, 4)
        else:
            for _ in range(4):
                ss.resetFields()
                for op in ops:
                    op.apply(ss)
                ss.sumFields()
                l.apply(ss)
        res.append(np.stack(ss.spinArrays()[:3]))
    np.testing.assert_array_equal(res[0], res[1])
    dip.apply(ss)
    if n <= 20000:
        o = O.SpinSystem(*dims)
        o.set_spins(*res[1])
        assert rel_err(np.stack(ss.fieldArrays("Dipole")), O.dipole_direct(o, 0.3)) <= 1e-5
