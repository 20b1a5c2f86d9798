"""Packed ensembles whose size classes all take the fused x pass: edge lengths
at and off the transform lengths, a spectrum carried over steps, spins replaced
between runs, and noise drawn as in the unfused step.  Batching as in
SpinOperation::apply(SpinSystem**, n) (M/cpu/core/spinoperation.cpp:288-300)."""
import numpy as np
import pytest

import oracle as O
from helpers import random_spins

pytestmark = pytest.mark.gpu

# unit spins, a few steps of dt = 0.01 in FP32: rounding of the fields (1e-6
# of |H| < 10) times dt times the steps, and of the spins, stays below 5e-6
TOL = 1e-5


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


def _ensemble(M, dims, llg, open_xy, T=0.0):
    e = M.Ensemble(dims)
    e.configure(alpha=0.1, dt=0.01, J=1.0, pbc=(0, 0, 0), K=0.2, axis=(0, 0, 1.0), T=T, seed=7, B=(0, 0, 0),
                dB=(0, 0, 0), g=0.05, open_xy=open_xy, llg=llg)
    return e


def _single(M, dims, s, llg, open_xy, nsteps, B, dB):
    n = int(np.prod(dims))
    ss = M.SpinSystem(*dims)
    ss.setSpinArrays(*s)
    ss.setAlpha(0.1)
    ss.setTimeStep(0.01)
    ex = M.Exchange(ss)
    ex.addPaths(*O.nn_paths(*dims, pbc=(0, 0, 0)))
    ani = M.Anisotropy(ss)
    ani.addMany(np.arange(n), np.tile([0, 0, 1.0], (n, 1)), np.full(n, 0.2))
    z = M.AppliedField(ss)
    z.set(*B)
    z.setSweep(*dB)
    dip = M.Dipole(ss)
    dip.setOpen(open_xy, open_xy, True)
    dip.setStrength(0.05)
    M.run(ss, [ex, ani, z, dip], M.LLG.new(llg), nsteps)
    return np.stack(ss.spinArrays()[:3])


@pytest.mark.parametrize("open_xy,dims", [
    (True, [(16, 16, 4), (17, 10, 2), (16, 16, 4)]),
    (True, [(128, 6, 1), (100, 4, 3), (33, 64, 1)]),
    (False, [(32, 32, 2), (256, 2, 1), (32, 32, 2), (128, 16, 8)])])
@pytest.mark.parametrize("llg", ["Cartesian", "Quaternion"])
def test_carried_spectrum(M, llg, open_xy, dims):
    e = _ensemble(M, dims, llg, open_xy)
    fields = [((0.0, 0.1 * r, -0.2), (1e-3 * r, 0.0, -1e-3)) for r in range(len(dims))]
    for r, d in enumerate(dims):
        e.setSpins(r, *random_spins(int(np.prod(d)), 200 + r))
        e.setReplicaParams(r, 0.0, *fields[r])
    e.run(3)
    # replica 0 starts anew, the others go on from the carried spectrum
    starts = [random_spins(int(np.prod(dims[0])), 300)] + [np.stack(e.spins(r)) for r in range(1, len(dims))]
    e.setSpins(0, *starts[0])
    e.run(4)
    for r, d in enumerate(dims):
        B, dB = fields[r]
        B3 = tuple(np.float64(b) + 3 * np.float64(x) for b, x in zip(B, dB))
        ref = _single(M, d, starts[r], llg, open_xy, 4, B3, dB)
        got = np.stack(e.spins(r))
        assert np.abs(got - ref).max() <= TOL, (d, np.abs(got - ref).max())


@pytest.mark.parametrize("dims", [[(32, 16, 2), (24, 6, 3)], [(128, 4, 1), (16, 32, 1), (128, 4, 1)]])
def test_noise_as_unfused(M, dims):
    """A class outside the fused pass, packed last, sends the whole ensemble
    through the separate kernels: same packed sites, same noise."""
    outs = []
    for extra in ([], [(4, 6, 2)]):
        e = _ensemble(M, dims + extra, "Cartesian", True, T=0.3)
        for r, d in enumerate(dims + extra):
            e.setSpins(r, *random_spins(int(np.prod(d)), 400 + r))
            e.setReplicaParams(r, 0.2 + 0.1 * r, (0.0, 0.0, 0.1), (0.0, 0.0, 0.0))
        e.run(5)
        outs.append([np.stack(e.spins(r)) for r in range(len(dims))])
    for a, b in zip(*outs):
        assert np.abs(a - b).max() <= TOL
