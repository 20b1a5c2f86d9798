"""Captured steps with more than one long-range operator, or with one operator
listed twice: the spectrum a step carries into the next is its last operator's
alone, so every captured step (single, carried, several to a launch) equals the
single calls bit for bit.  The field slots of the last step equal theirs too."""
import numpy as np
import pytest

import oracle as O
from helpers import random_spins

pytestmark = pytest.mark.gpu

STEPS = 11   # an uncarried step, single carried ones, two launches of several steps


@pytest.fixture(scope="module")
def M():
    import maglua_b200 as M
    M.init(0)
    return M


def _dipole(M, ss, g, slot=None, trunc=8):
    dip = M.Dipole(ss)
    dip.setStrength(g)
    dip.setTruncation(trunc)
    if slot:
        dip.setSlotName(slot)
    return dip


def _layers(M, ss):
    nx, ny, nz = ss.nx(), ss.ny(), ss.nz()
    r = np.random.default_rng(5)
    op = M.LongRange2D(ss)
    op.setNewDataRequired(False)
    for i in range(nz):
        for j in range(nz):
            for ab in ("XX", "XY", "XZ", "YX", "YY", "YZ", "ZX", "ZY", "ZZ"):
                op.setTensorArray(i + 1, j + 1, ab, 0.3 * r.normal(size=nx * ny) / np.sqrt(nx * ny))
    return op


def _magnetostatic(M, ss):
    op = M.Magnetostatic(ss)
    op.setStrength(0.05)
    op.setTruncation(4)
    return op


def _operators(M, ss, kind):
    if kind == "two dipoles":
        return [_dipole(M, ss, 0.1, "near", 3), _dipole(M, ss, 0.06, "far", 9)]
    if kind == "twice":
        return [_dipole(M, ss, 0.1)] * 2
    make = {"dipole": lambda: _dipole(M, ss, 0.1), "layers": lambda: _layers(M, ss),
            "magnetostatic": lambda: _magnetostatic(M, ss)}
    return [make[name]() for name in kind.split(",")]


def _build(M, dims, precision, kind, per_site=False, T=0.0, llg="Quaternion"):
    n = int(np.prod(dims))
    ss = M.SpinSystem(*dims, precision=precision)
    ss.setSpinArrays(*random_spins(n, 31), np.ones(n))
    ss.setAlpha(0.1)
    ss.setTimeStep(0.01)
    ex = M.Exchange(ss)
    ex.addPaths(*O.nn_paths(*dims, pbc=(1, 1, 0)))
    ani = M.Anisotropy(ss)
    r = np.random.default_rng(8)
    ani.addMany(np.arange(n), np.tile([0, 0, 1.0], (n, 1)), r.uniform(0.1, 0.3, n) if per_site else np.full(n, 0.2))
    z = M.AppliedField(ss)
    z.set(0.2, 0, 0)
    ops = [ex, ani, z]
    if T > 0:
        th = M.Thermal(ss, M.Random.Philox(3))
        th.setTemperature(T)
        ops.append(th)
    return ss, ops + _operators(M, ss, kind), M.LLG.new(llg)


def _calls(ss, ops, llg, n):
    for _ in range(n):
        ss.resetFields()
        for op in ops:
            op.apply(ss)
        ss.sumFields()
        llg.apply(ss)


def _compare(M, a, ops_a, b, ops_b, what):
    np.testing.assert_array_equal(np.stack(a.spinArrays()[:3]), np.stack(b.spinArrays()[:3]), err_msg=what)
    for name in {op.slotName() for op in ops_a}:
        np.testing.assert_array_equal(np.stack(a.fieldArrays(name)), np.stack(b.fieldArrays(name)),
                                      err_msg=what + " field " + name)


KINDS = ["dipole,layers", "layers,dipole", "dipole,magnetostatic", "magnetostatic,dipole", "two dipoles", "twice"]
# rows in pairs and lines of a power of two; any length; odd rows
DIMS = [(64, 32, 2), (30, 14, 3), (32, 9, 2)]


@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("dims", DIMS)
@pytest.mark.parametrize("kind", KINDS)
def test_captured_steps_equal_single_calls(M, kind, dims, precision):
    ref, ops_r, llg = _build(M, dims, precision, kind)
    _calls(ref, ops_r, llg, STEPS)
    ss, ops, llg = _build(M, dims, precision, kind)
    M.run(ss, ops, llg, STEPS)
    _compare(M, ref, ops_r, ss, ops, "run")
    ss, ops, llg = _build(M, dims, precision, kind)
    plan = M.Plan(ss, ops, llg)
    plan.launch(STEPS - 2)
    plan.launch(1)
    plan.launch(1)
    _compare(M, ref, ops_r, ss, ops, "plan")


# (plan, steps) in turn: a plan whose steps end in the fused x pass, then one without a
# convolution, with the same operator and another one that comes last, or with
# its operators in the other order (no fused x pass), then the first again
@pytest.mark.parametrize("precision", ["f32", "f64"])
@pytest.mark.parametrize("dims", DIMS[:2])
@pytest.mark.parametrize("between", ["none", "near,far", "far,near"])
def test_plans_in_turn(M, between, dims, precision):
    turns = [("near", 3), (between, 2), ("near", 5), (between, 1), ("near", 2)]
    res = []
    for captured in (False, True):
        ss, ops, llg = _build(M, dims, precision, "two dipoles")
        base, near, far = ops[:-2], ops[-2], ops[-1]
        lists = {"none": [], "near": [near], "near,far": [near, far], "far,near": [far, near]}
        near.apply(ss)   # its slot comes first in the sum
        ss.resetFields()
        plans = {name: M.Plan(ss, base + lists[name], llg) for name in ("near", between)}
        for name, n in turns:
            if captured:
                plans[name].launch(n)
            else:
                _calls(ss, base + lists[name], llg, n)
        # a short run takes up what the last plan left
        if captured:
            plans[between].launch(2)
            M.run(ss, base + [near], llg, 2)
        else:
            _calls(ss, base + lists[between], llg, 2)
            _calls(ss, base + [near], llg, 2)
        res.append(np.stack(ss.spinArrays()[:3]))
    np.testing.assert_array_equal(res[0], res[1])


@pytest.mark.parametrize("dims,precision", [((64, 32, 2), "f32"), ((30, 14, 3), "f64")])
def test_operator_shared_by_two_systems(M, dims, precision):
    """A plan of another system runs the shared operator in between."""
    res = []
    for captured in (False, True):
        ss, ops, llg = _build(M, dims, precision, "two dipoles")
        other, ops2, _ = _build(M, dims, precision, "two dipoles")
        base, near, far = ops[:-2], ops[-2], ops[-1]
        mine = M.Plan(ss, base + [near], llg)
        theirs = M.Plan(other, base + [near, far], llg)
        for k in range(3):
            if captured:
                mine.launch(3)
                ss.synchronize()
                theirs.launch(2)
            else:
                _calls(ss, base + [near], llg, 3)
                ss.synchronize()
                _calls(other, base + [near, far], llg, 2)
            other.synchronize()
        res.append((np.stack(ss.spinArrays()[:3]), np.stack(other.spinArrays()[:3])))
    np.testing.assert_array_equal(res[0][0], res[1][0])
    np.testing.assert_array_equal(res[0][1], res[1][1])


@pytest.mark.parametrize("precision,make", [("f32", "dipole"), ("f64", "dipole"), ("f32", "layers")])
@pytest.mark.parametrize("dims", [(256, 128, 4), (150, 100, 3)])
def test_operator_applied_to_many_systems(M, dims, precision, make):
    """The systems run on streams of their own; the operator's one spectrum serves
    them in turn (SpinOperation::apply(SpinSystem**, n))."""
    n = int(np.prod(dims))
    systems = []
    for k in range(6):
        ss = M.SpinSystem(*dims, precision=precision)
        ss.setSpinArrays(*random_spins(n, 70 + k), np.ones(n))
        ss.setAlpha(0.1)
        ss.setTimeStep(0.01)
        systems.append(ss)
    op = _dipole(M, systems[0], 0.1, trunc=5) if make == "dipole" else _layers(M, systems[0])
    name = op.slotName()
    want = []
    for ss in systems:
        ss.resetFields()
        op.apply(ss)
        ss.synchronize()
        want.append(np.stack(ss.fieldArrays(name)))
    for attempt in range(3):
        for ss in systems:
            ss.resetFields()
        op.apply(systems)
        for ss, w in zip(systems, want):
            np.testing.assert_array_equal(np.stack(ss.fieldArrays(name)), w)
    # and their captured steps, launched one after the other
    llg = M.LLG.new("Quaternion")
    start = [np.stack(ss.spinArrays()[:3]) for ss in systems]
    res = []
    for wait in (True, False):
        for ss, s in zip(systems, start):
            ss.setSpinArrays(*s, np.ones(n))
        plans = [M.Plan(ss, [op], llg) for ss in systems]
        for k in range(4):
            for ss, p in zip(systems, plans):
                p.launch(2)
                if wait:
                    ss.synchronize()
        res.append([np.stack(ss.spinArrays()[:3]) for ss in systems])
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("make", ["dipole", "layers"])
@pytest.mark.parametrize("dims", DIMS[:2])
def test_operator_shared_by_both_precisions(M, dims, make):
    """The operator's spectrum is rebuilt whenever the precision changes; plans
    captured on the one that went are captured again."""
    res = []
    for captured in (False, True):
        systems = {p: _build(M, dims, p, make) for p in ("f32", "f64")}
        op = systems["f32"][1][-1]
        llg = M.LLG.new("Quaternion")
        lists = {p: systems[p][1][:-1] + [op] for p in systems}
        if captured:
            plans = {p: M.Plan(systems[p][0], lists[p], llg) for p in systems}
        for k in range(2):
            for p in systems:
                if captured:
                    plans[p].launch(6)
                else:
                    _calls(systems[p][0], lists[p], llg, 6)
        res.append([np.stack(systems[p][0].spinArrays()[:3]) for p in systems])
    for a, b in zip(*res):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("dims,precision,kind", [((64, 32, 2), "f32", "dipole,layers"), ((32, 9, 2), "f32", "layers"),
                                                 ((30, 14, 3), "f32", "two dipoles"), ((30, 14, 3), "f64", "layers,dipole"),
                                                 ((64, 32, 2), "f64", "dipole")])
@pytest.mark.parametrize("llg,T", [("Quaternion", 0.0), ("Cartesian", 0.3)])
def test_per_site_terms_beside_convolutions(M, dims, precision, kind, llg, T):
    """The general step with its last convolution's x pass fused and other addends
    in slots: a constant per site and noise beside them."""
    ref, ops_r, l = _build(M, dims, precision, kind, per_site=True, T=T, llg=llg)
    _calls(ref, ops_r, l, STEPS)
    ss, ops, l = _build(M, dims, precision, kind, per_site=True, T=T, llg=llg)
    M.run(ss, ops, l, STEPS)
    _compare(M, ref, [o for o in ops_r if o.slotName() != "Thermal"], ss, ops, "run")
