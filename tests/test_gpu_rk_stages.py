"""Runge-Kutta steps whose stages run as fused passes (inverse x pass, local
terms and every row a stage contributes to in one kernel) against the same
steps through llg:apply chains.  The second field operator of the "chains"
system (the applied field in two halves, in slots of their own) keeps its steps
off the fused passes; both compute the same field.

Tolerance: a step's spins differ by the rounding of its dozen updates, well
within 1e-6 (FP32) and 1e-13 (FP64)."""
import numpy as np
import pytest

import oracle as O
from helpers import rel_err, tilted_spins

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


def _steps(M, dims, precision, scheme, llg, fused, temp, n=3):
    N = int(np.prod(dims))
    ss = M.SpinSystem(*dims, precision=precision)
    ss.setSpinArrays(*tilted_spins(N, 51, deg=30.0), np.ones(N))
    ss.setAlpha(0.1)
    ss.setTimeStep(0.02)
    ex = M.Exchange(ss)
    ex.addPaths(*O.nn_paths(*dims, pbc=(1, 1, 0)))
    ani = M.Anisotropy(ss)
    ani.addMany(np.arange(N), np.tile([0, 0, 1.0], (N, 1)), np.full(N, 0.2))
    dip = M.Dipole(ss)
    dip.setStrength(0.05)
    dip.setTruncation(12)
    ops = [ex, ani, dip]
    for k, b in enumerate([0.3] if fused else [0.15, 0.15]):
        z = M.AppliedField(ss)
        z.set(b, 0, 0)
        z.setSlotName("Zeeman%d" % k)
        ops.insert(2, z)
    th = None
    if temp:
        th = M.Thermal(ss, M.Random.Philox(7))
        th.setTemperature(0.1)
    rk = M.RungeKutta(ss, scheme, ops, M.LLG.new(llg), temp=th)
    rk.step(n)
    fields = {name: np.stack(ss.fieldArrays(name)) for name in ("Exchange", "Anisotropy", "Dipole", "Total")}
    return np.stack(ss.spinArrays()[:3]), fields, ss.time()


@pytest.mark.parametrize("dims,precision,scheme,llg,temp", [
    ((64, 16, 2), "f32", "RK4", "Quaternion", False),
    ((32, 128, 3), "f32", "RK6", "Cartesian", True),
    ((512, 4, 1), "f32", "K3", "Quaternion", True),
    ((32, 9, 3), "f32", "BS3", "Quaternion", False),   # odd rows: the any-length x pass
    ((34, 10, 2), "f32", "RK2", "Cartesian", False),
    ((20, 14, 2), "f64", "RK4_38", "Quaternion", True),
    ((64, 8, 1), "f64", "RK1", "Quaternion", False),
])
def test_fused_stages_follow_the_chains(M, dims, precision, scheme, llg, temp):
    a, fa, ta = _steps(M, dims, precision, scheme, llg, True, temp)
    b, fb, tb = _steps(M, dims, precision, scheme, llg, False, temp)
    tol = 1e-6 if precision == "f32" else 1e-13
    assert np.abs(a - b).max() <= tol
    assert ta == tb
    # after a step the slots hold the fields of its start (zero after a kick)
    for name in fa:
        if np.abs(fb[name]).max() == 0:
            assert np.abs(fa[name]).max() == 0
        else:
            assert rel_err(fa[name], fb[name]) <= 10 * tol
