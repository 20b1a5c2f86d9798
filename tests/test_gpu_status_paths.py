"""The status word's non-finite bit (mlb_system_status) on the step kernels that
tests of small lattices do not reach: two sites at a time, any length, the
Runge-Kutta stages and packed ensembles.

One site's spin is large enough that its Cartesian torque M x (M x h) leaves the
number range, while every other site stays finite: with M of 1e20 (FP32) or 1e110
(FP64) that site's torque is about M^3, above 3.4e38 and 1.8e308, its
neighbours' about M."""
import numpy as np
import pytest

import oracle as O
from helpers import random_spins, tilted_spins

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


def _system(M, dims, precision, site):
    n = int(np.prod(dims))
    s = tilted_spins(n, 96, deg=20.0)
    if site is not None:
        s[0, site] = 1e20 if precision == "f32" else 1e110
    ss = M.SpinSystem(*dims, precision=precision)
    ss.setSpinArrays(*s, np.ones(n))
    ss.setAlpha(0.1)
    ss.setTimeStep(0.01)
    ex = M.Exchange(ss)
    ex.addPaths(*O.nn_paths(*dims, pbc=(1, 1, 0)))
    dip = M.Dipole(ss)
    dip.setStrength(0.05)
    dip.setTruncation(4)
    return ss, [ex, dip], M.LLG.new("Cartesian")


@pytest.mark.parametrize("dims,precision", [((64, 32, 2), "f32"), ((256, 64, 8), "f32"), ((128, 8, 1), "f32"),
                                            ((64, 9, 2), "f32"), ((30, 14, 3), "f32"), ((30, 14, 3), "f64"),
                                            ((64, 8, 2), "f64")])
@pytest.mark.parametrize("row", [4, 5])   # the two sites of a pair
def test_one_site(M, dims, precision, row):
    site = row * dims[0] + 7
    ss, ops, llg = _system(M, dims, precision, None)
    M.run(ss, ops, llg, 1)
    assert ss.status() == 0
    ss, ops, llg = _system(M, dims, precision, site)
    M.run(ss, ops, llg, 1)
    bad = ~np.isfinite(np.stack(ss.spinArrays()[:3])).all(0)
    assert list(np.flatnonzero(bad)) == [site]
    assert ss.status() & 1


@pytest.mark.parametrize("dims,precision", [((64, 32, 2), "f32"), ((64, 9, 2), "f32"), ((30, 14, 3), "f64")])
@pytest.mark.parametrize("path", ["run", "plan", "rk", "rk graph"])
def test_captured_steps_and_schemes(M, dims, precision, path):
    for site in (None, dims[0] + 3):
        ss, ops, llg = _system(M, dims, precision, site)
        if path == "run":
            M.run(ss, ops, llg, 6)
        elif path == "plan":
            M.Plan(ss, ops, llg).launch(6)
        else:
            M.RungeKutta(ss, "RK2", ops, llg).step(1 if path == "rk" else 4)
        assert (ss.status() & 1) == (site is not None)


@pytest.mark.parametrize("llg", ["Cartesian", "Quaternion"])
def test_packed_ensemble(M, llg):
    dims = [(20, 18, 2), (32, 6, 1), (20, 18, 2)]
    for broken in (False, True):
        e = M.Ensemble(dims)
        e.configure(dt=0.01, K=0.2, g=0.05, llg=llg)
        for r, d in enumerate(dims):
            s = random_spins(int(np.prod(d)), 700 + r)
            if broken and r == 2:
                s[1, 40] = np.nan
            e.setSpins(r, *s)
        e.run(2)
        assert (e.status() & 1) == broken
