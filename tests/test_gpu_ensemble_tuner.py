"""What the ensemble's tuner reports: the kernels that run.  An ensemble whose step
runs inside its classes' x passes has no choice to time; one class outside
them, and tile sizes, grids and (y,z) passes are timed for all."""
import numpy as np
import pytest

from helpers import random_spins

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


@pytest.mark.parametrize("extra", [[], [(4, 6, 2)]])
def test_log_names_what_runs(M, extra, tmp_path, monkeypatch):
    monkeypatch.setenv("MLB_TUNE_CACHE", str(tmp_path / "tune.txt"))
    dims = [(20, 18, 2), (32, 6, 1)] + extra
    e = M.Ensemble(dims)
    e.configure(dt=0.01, K=0.2, g=0.05)
    for r, d in enumerate(dims):
        e.setSpins(r, *random_spins(int(np.prod(d)), 500 + r))
    e.run(3)
    log = e.tuneLog()
    assert ("k_xens" in log) == (not extra)
    assert ("CTAs (one per tile)" in log) == bool(extra)
    assert (" us" in log) == bool(extra)
    assert e.info()["block_size"] in (128, 256, 512)
    # without exchange the step runs apart: the choices are made anew
    e.configure(dt=0.01, K=0.2, g=0.05, J=0.0)
    e.run(1)
    assert "CTAs (one per tile)" in e.tuneLog()
