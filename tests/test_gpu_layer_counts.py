"""The (y,z) pass with the layer sum at 9 to 16 layers, one kernel for all of them: the
field against the oracle's lattice sum (tolerances as for the other sizes: the
rounding of a transform, 1e-5 in FP32 and 1e-11 in FP64 of the norm), and packed
ensembles, whose fused x pass every class has to take."""
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


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("dims", [(16, 16, 9), (10, 16, 15), (330, 16, 12), (32, 32, 10), (9, 32, 14), (24, 64, 11),
                                  (16, 64, 13), (300, 64, 15), (32, 64, 16)])
def test_field(M, dims, precision):
    n = int(np.prod(dims))
    s = random_spins(n, 91, lengths=True)
    ss = M.SpinSystem(*dims, precision=precision)
    ss.setSpinArrays(*s)
    dip = M.Dipole(ss)
    dip.setStrength(0.3)
    dip.setTruncation(6)
    dip.apply(ss)
    o = O.SpinSystem(*dims)
    o.set_spins(*s)
    O.LongRange(*dims, O.dipole_tensor(*dims, gmax=(6,) * 4)).apply(o, 0.3)
    assert rel_err(np.stack(ss.fieldArrays("Dipole")), o.field("Dipole")) <= TOL[precision]


@pytest.mark.parametrize("dims", [[(16, 16, 12), (32, 32, 4)], [(20, 10, 9), (17, 30, 15), (16, 16, 16)]])
def test_ensemble_takes_the_fused_pass(M, dims, monkeypatch):
    monkeypatch.setenv("MLB_TUNE_CACHE", "off")
    e = M.Ensemble(dims)
    e.configure(alpha=0.1, dt=0.01, J=1.0, pbc=(0, 0, 0), K=0.2, axis=(0, 0, 1.0), g=0.05, open_xy=True)
    starts = [random_spins(int(np.prod(d)), 600 + r) for r, d in enumerate(dims)]
    for r, s in enumerate(starts):
        e.setSpins(r, *s)
    e.run(4)
    assert "k_xens" in e.tuneLog()
    for r, d in enumerate(dims):
        n = int(np.prod(d))
        ss = M.SpinSystem(*d)
        ss.setSpinArrays(*starts[r])
        ss.setAlpha(0.1)
        ss.setTimeStep(0.01)
        ex = M.Exchange(ss)
        ex.addPaths(*O.nn_paths(*d, pbc=(0, 0, 0)))
        ani = M.Anisotropy(ss)
        ani.addMany(np.arange(n), np.tile([0, 0, 1.0], (n, 1)), np.full(n, 0.2))
        dip = M.Dipole(ss)
        dip.setOpen(True, True, True)
        dip.setStrength(0.05)
        M.run(ss, [ex, ani, dip], M.LLG.new("Cartesian"), 4)
        # four steps of dt 0.01 in fields below 10 that differ by 1e-6 of them
        assert np.abs(np.stack(e.spins(r)) - np.stack(ss.spinArrays()[:3])).max() <= 1e-5
