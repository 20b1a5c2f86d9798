"""Systems on streams of their own that read each other's spins: a copy or an LLG
update that waits behind the reader's queue still sees the source's spins as they were
when it was called, whatever the source does next (as every call of the reference
is done when it returns)."""
import numpy as np
import pytest

import oracle as O
from helpers import random_spins

pytestmark = pytest.mark.gpu

DIMS = (256, 128, 4)


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


def _system(M, seed):
    n = int(np.prod(DIMS))
    ss = M.SpinSystem(*DIMS)
    ss.setSpinArrays(*random_spins(n, seed), np.ones(n))
    ss.setAlpha(0.1)
    ss.setTimeStep(0.01)
    ex = M.Exchange(ss)
    ex.addPaths(*O.nn_paths(*DIMS, pbc=(1, 1, 0)))
    dip = M.Dipole(ss)
    dip.setStrength(0.1)
    dip.setTruncation(4)
    return ss, [ex, dip], M.LLG.new("Quaternion")


@pytest.mark.parametrize("how", ["copy", "llg"])
def test_reader_behind_its_queue(M, how):
    res = []
    for wait in (True, False):
        src, ops, llg = _system(M, 1)
        dst, ops_d, _ = _system(M, 2)
        M.run(src, ops, llg, 4)
        src.resetFields()
        for op in ops:
            op.apply(src)
        src.sumFields()
        src.synchronize()
        M.run(dst, ops_d, llg, 8)
        dst.synchronize()
        M.run(dst, ops_d, llg, 1500)   # the reader's stream is busy for some 10 ms
        if how == "copy":
            src.copySpinsTo(dst)
        else:
            llg.apply(src, 1.0, src, dst)   # dst takes src's spins a step on
        if wait:
            dst.synchronize()
        M.run(src, ops, llg, 4)
        src.synchronize()
        res.append(np.stack(dst.spinArrays()[:3]))
    np.testing.assert_array_equal(res[0], res[1])


def test_short_runs_in_turn(M):
    """Two systems with one operator, a hundred runs of three steps each and none
    waited for: the graphs of a run outlive it until they have run."""
    res = []
    for wait in (True, False):
        a, ops, llg = _system(M, 1)
        b, _, _ = _system(M, 2)
        for k in range(100):
            for ss in (a, b):
                M.run(ss, ops, llg, 3)
                if wait:
                    ss.synchronize()
        res.append([np.stack(ss.spinArrays()[:3]) for ss in (a, b)])
    for x, y in zip(*res):
        np.testing.assert_array_equal(x, y)
