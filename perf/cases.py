"""What the framework is timed on: stretches of spin dynamics as MagLua
scripts run them, each through the public classes of maglua_b200.

Every case advances a magnetic system by some steps and reads what a script
reads after such a stretch: the spins, and where a script records a curve its
net moments.  The kinds:

  film      a thin film or an open body with the canonical operator set
            (exchange, anisotropy, Langevin noise, applied field with its
            sweep, dipole) stepped by a captured Plan
  script    the same operators applied one call at a time, the loop of an
            ordinary script, with its moment read every few steps
  grains    a granular film: easy axes, moments and exchange differ from
            grain to grain
  rk        the film stepped by a Runge-Kutta scheme with a thermal kick
  layers    a stack of layers coupled by layer-pair tensors (LongRange2D)
  ensemble  independent replicas of uneven sizes stepped together

exact() integrates the same equations in torch float64: the same lattice sums
and FFT convolutions, and the same Philox4x32-10 noise (Salmon et al.,
SC'11).
"""
import math

import numpy as np
import torch

import maglua_b200 as M

GAMMA = 1.0


# ---------------------------------------------------------------- the cases
def _film(nx, ny, nz, steps, precision="f32", open_xy=False, llg="Quaternion", T=0.0, alpha=0.05, dt=0.005,
          K=0.05, cubic=False, g=0.02, field=0.1, sweep=0.0, start="tilted"):
    return {"kind": "film", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "precision": precision,
            "open": open_xy, "llg": llg, "T": T, "alpha": alpha, "dt": dt, "K": K, "cubic": cubic, "g": g,
            "field": field, "sweep": sweep, "start": start}


def listed():
    return [
        # a few steps of an ordinary script on a small sample, moments printed
        # every fifth step: launches and host calls count
        dict(_film(16, 12, 3, 10, T=0.3, alpha=0.1, dt=0.01, g=0.05), name="script_16x12x3", kind="script"),
        # a small relaxation in the reference's own precision
        dict(_film(32, 32, 1, 200, precision="f64", llg="Cartesian", alpha=0.1, dt=0.01, K=0.1, g=0.01, field=0.0,
                   start="random"), name="film_32x32x1_f64"),
        # the usual thin film at temperature
        dict(_film(256, 256, 8, 100, T=0.5), name="film_256x256x8"),
        # a wide film in the stripe-forming regime
        dict(_film(512, 512, 4, 50, T=0.1, alpha=0.02, K=0.02, g=0.05, field=0.0, start="random"),
             name="film_512x512x4"),
        # a film whose edges are what the sample has, not powers of two
        dict(_film(200, 150, 5, 50, T=0.3), name="film_200x150x5"),
        # a film in double precision
        dict(_film(128, 128, 4, 100, precision="f64", T=0.2), name="film_128x128x4_f64"),
        # a hysteresis branch of an open nanodot
        dict(_film(50, 40, 3, 200, open_xy=True, llg="Cartesian", alpha=0.5, dt=0.01, K=0.1, g=0.1,
                   field=0.5, sweep=-0.001), name="dot_50x40x3_open"),
        # the bulk sample: an open cube, split transforms
        dict(_film(128, 128, 128, 20, open_xy=True, T=0.3, cubic=True, g=0.03, field=0.0), name="cube_128_open"),
        # a granular recording layer at temperature
        {"name": "grains_128x128x4", "kind": "grains", "nx": 128, "ny": 128, "nz": 4, "steps": 50, "grain": 8.0,
         "T": 0.2, "alpha": 0.1, "dt": 0.005, "g": 0.05, "field": -0.1},
        # accurate trajectories: RK4 with the thermal kick
        dict(_film(256, 256, 8, 5, T=0.5), name="rk4_256x256x8", kind="rk", scheme="RK4"),
        # a coupled multilayer
        {"name": "layers_128x128x4", "kind": "layers", "nx": 128, "ny": 128, "nz": 4, "steps": 50, "T": 0.1,
         "alpha": 0.1, "dt": 0.01, "K": 0.1, "g": 0.05, "spacing": 1.5},
        # reversal statistics of many small particles of several sizes
        {"name": "ensemble_512", "kind": "ensemble", "replicas": 512, "mix": 3, "steps": 20, "T": 0.2, "alpha": 0.1,
         "dt": 0.01, "K": 0.2, "g": 0.02, "llg": "Cartesian", "sweep": -0.5 / 20000},
    ]


ENSEMBLE_SIZES = [(16, 16, 16), (32, 32, 4), (48, 48, 2), (64, 64, 4)]


def _ensemble_dims(case):
    r = np.random.default_rng(case["mix"])
    return [ENSEMBLE_SIZES[k] for k in r.integers(0, len(ENSEMBLE_SIZES), case["replicas"])]


def _length(rng, lo, hi):
    """A lattice edge: half of them powers of two, the others any length
    without a prime factor above 31 (what the transforms take)."""
    if rng.random() < 0.5:
        a, b = math.ceil(math.log2(lo)), math.floor(math.log2(hi))
        return 2 ** rng.randint(a, b)
    while True:
        n = round(math.exp(rng.uniform(math.log(lo), math.log(hi))))
        m = n
        for p in (2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31):
            while m % p == 0:
                m //= p
        if m == 1:
            return n


def _steps(rng, sites, budget):
    return max(5, min(200, int(budget / sites * rng.uniform(0.5, 1.0))))


def draw(rng):
    kind = rng.choice(["film", "film", "film", "film", "f64", "dot", "cube", "script", "grains", "rk", "layers",
                       "ensemble"])
    if kind in ("film", "f64"):
        hi = 512 if kind == "film" else 256
        while True:
            nx, ny, nz = _length(rng, 16, hi), _length(rng, 16, hi), rng.randint(1, 8)
            if nx * ny * nz <= (1 << 20 if kind == "film" else 1 << 18):
                break
        n = nx * ny * nz
        return dict(_film(nx, ny, nz, _steps(rng, n, 3e7 if kind == "film" else 6e6),
                          precision="f32" if kind == "film" else "f64", llg=rng.choice(["Quaternion", "Cartesian"]),
                          T=rng.choice([0.0, 0.1, 0.5]), g=rng.choice([0.01, 0.05])))
    if kind == "dot":
        nx, ny, nz = rng.randint(12, 128), rng.randint(12, 128), rng.randint(1, 4)
        return dict(_film(nx, ny, nz, _steps(rng, _padded(nx, True) * _padded(ny, True) * nz, 1.6e7), open_xy=True,
                          llg=rng.choice(["Quaternion", "Cartesian"]), T=rng.choice([0.0, 0.1]), alpha=0.5, dt=0.01,
                          K=0.1, g=0.1, field=0.5, sweep=-0.001))
    if kind == "cube":
        n = rng.randint(24, 128)
        return dict(_film(n, n, n, _steps(rng, _padded(n, True) ** 3 // 8, 4e7), open_xy=True, T=0.3, cubic=True, g=0.03, field=0.0))
    if kind == "script":
        nx, ny, nz = _length(rng, 8, 64), _length(rng, 8, 64), rng.randint(1, 4)
        return dict(_film(nx, ny, nz, 5 * rng.randint(1, 4), T=rng.choice([0.0, 0.3]), alpha=0.1, dt=0.01, g=0.05),
                    kind="script")
    if kind == "grains":
        nx, ny, nz = _length(rng, 32, 256), _length(rng, 32, 256), rng.randint(1, 4)
        return {"kind": "grains", "nx": nx, "ny": ny, "nz": nz, "steps": _steps(rng, nx * ny * nz, 4e6),
                "grain": rng.choice([6.0, 8.0, 12.0]), "T": rng.choice([0.0, 0.2]), "alpha": 0.1, "dt": 0.005,
                "g": 0.05, "field": rng.choice([-0.1, 0.2])}
    if kind == "rk":
        nx, ny, nz = _length(rng, 32, 256), _length(rng, 32, 256), rng.randint(1, 8)
        return dict(_film(nx, ny, nz, rng.randint(3, 8), T=rng.choice([0.0, 0.5])), kind="rk",
                    scheme=rng.choice(["RK2", "RK4"]))
    if kind == "layers":
        nx, ny, nz = _length(rng, 32, 160), _length(rng, 32, 160), rng.randint(2, 6)
        return {"kind": "layers", "nx": nx, "ny": ny, "nz": nz, "steps": _steps(rng, nx * ny * nz, 4e6),
                "T": rng.choice([0.0, 0.1]), "alpha": 0.1, "dt": 0.01, "K": 0.1, "g": 0.05,
                "spacing": rng.choice([1.0, 1.5])}
    return {"kind": "ensemble", "replicas": rng.randint(24, 400), "mix": rng.randint(4, 1000),
            "steps": rng.randint(5, 20), "T": rng.choice([0.0, 0.2]), "alpha": 0.1, "dt": 0.01, "K": 0.2, "g": 0.02,
            "llg": rng.choice(["Cartesian", "Quaternion"]), "sweep": -0.5 / 20000}


# ---------------------------------------------------------------- inputs
def _unit(v):
    return v / np.linalg.norm(v, axis=0)


def _start_spins(case, n, seed):
    """Saturated along z with a 5 degree tilt, or uniform on the sphere."""
    r = np.random.default_rng(seed)
    if case.get("start", "tilted") == "random":
        return _unit(r.normal(size=(3, n)))
    phi = r.uniform(0, 2 * np.pi, n)
    th = np.deg2rad(5.0)
    return _unit(np.stack([np.sin(th) * np.cos(phi), np.sin(th) * np.sin(phi), np.full(n, np.cos(th))]))


def _neighbours(nx, ny, nz, pbc):
    """(from, to) of every nearest-neighbour pathway, direction by direction."""
    idx = np.arange(nx * ny * nz, dtype=np.int32).reshape(nz, ny, nx)
    frm, to = [], []
    for ax, n in ((2, nx), (1, ny), (0, nz)):
        if n == 1:
            continue
        for sgn in (1, -1):
            src, dst = idx, np.roll(idx, -sgn, axis=ax)
            if not pbc[2 - ax]:
                cut = [slice(None)] * 3
                cut[ax] = slice(0, n - 1) if sgn == 1 else slice(1, n)
                src, dst = src[tuple(cut)], dst[tuple(cut)]
            frm.append(src.ravel())
            to.append(dst.ravel())
    return np.concatenate(frm), np.concatenate(to)


def _grains(case, seed):
    """Grain of every site (nearest of scattered centres, columnar), and each
    grain's easy axis, anisotropy constant and moment; exchange is weak
    across grain boundaries."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    r = np.random.default_rng(seed + 77)
    ng = max(4, int(nx * ny / case["grain"] ** 2))
    centres = r.uniform(0, 1, (ng, 2)) * [nx, ny]
    yy, xx = np.divmod(np.arange(nx * ny), nx)
    dx = torch.tensor(xx)[:, None] - torch.tensor(centres[:, 0])
    dy = torch.tensor(yy)[:, None] - torch.tensor(centres[:, 1])
    dx = dx - nx * torch.round(dx / nx)
    dy = dy - ny * torch.round(dy / ny)
    label = np.tile((dx * dx + dy * dy).argmin(1).numpy(), nz)
    axis = _unit(r.normal(0, 0.1, (3, ng)) + np.array([[0.0], [0.0], [1.0]])).T
    K = r.normal(0.3, 0.03, ng)
    ms = np.exp(r.normal(0.0, 0.1, ng))
    frm, to = _neighbours(nx, ny, nz, (1, 1, 0))
    J = np.where(label[frm] == label[to], 1.0, 0.15)
    return {"axis": axis[label], "K": K[label], "ms": ms[label], "from": frm, "to": to, "J": J}


def _layer_tensor(case):
    """Point-dipole coupling of every pair of layers, nearest image: array
    [dest][src][ab][y][x] at offset (x, y) and layer distance."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    x = np.arange(nx)
    y = np.arange(ny)
    x = (x + nx // 2) % nx - nx // 2
    y = (y + ny // 2) % ny - ny // 2
    out = np.zeros((nz, nz, 9, ny, nx))
    for d in range(nz):
        for s in range(nz):
            r = [np.broadcast_to(x[None, :], (ny, nx)).astype(float), np.broadcast_to(y[:, None], (ny, nx)).astype(float),
                 np.full((ny, nx), case["spacing"] * (d - s))]
            r2 = r[0] ** 2 + r[1] ** 2 + r[2] ** 2
            r2[r2 == 0] = np.inf
            for a in range(3):
                for b in range(3):
                    out[d, s, 3 * a + b] = case["g"] * (3 * r[a] * r[b] / r2 ** 2.5 - (a == b) / r2 ** 1.5)
    return out


def _reader(ss, n, precision):
    """The spins after a stretch: into pinned FP32 arrays, or the FP64 arrays
    of a double-precision system."""
    if precision == "f64":
        return lambda: list(ss.spinArrays()[:3])
    out = [torch.empty(n, dtype=torch.float32, pin_memory=True) for _ in range(3)]
    views = [o.numpy() for o in out]

    def read():
        ss.downloadF32(*views)
        return out
    return read


def _film_objects(case, seed):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    ss = M.SpinSystem(nx, ny, nz, precision=case["precision"])
    ss.setSpinArrays(*_start_spins(case, n, seed))
    ss.setAlpha(case["alpha"])
    ss.setTimeStep(case["dt"])
    pbc = (0, 0, 0) if case["open"] else (1, 1, 0)
    ex = M.Exchange(ss)
    frm, to = _neighbours(nx, ny, nz, pbc)
    ex.addPaths(frm, to, np.ones(len(frm)))
    sites = np.arange(n)
    if case["cubic"]:
        ani = M.AnisotropyCubic(ss)
        ani.addMany(sites, np.tile([1.0, 0, 0], (n, 1)), np.tile([0, 1.0, 0], (n, 1)),
                    np.tile([case["K"], 0, 0], (n, 1)))
    else:
        ani = M.Anisotropy(ss)
        ani.addMany(sites, np.tile([0, 0, 1.0], (n, 1)), np.full(n, case["K"]))
    ops = [ex, ani]
    th = None
    if case["T"] > 0:
        th = M.Thermal(ss, M.Random.Philox(1000 + seed))
        th.setTemperature(case["T"])
    z = M.AppliedField(ss)
    z.set(case["field"], 0, 0)
    if case["sweep"]:
        z.setSweep(case["sweep"], 0, 0)
    dip = M.Dipole(ss)
    dip.setStrength(case["g"])
    if case["open"]:
        dip.setOpen(True, True, True)
    ops += [z, dip]
    return ss, ops, th, M.LLG.new(case["llg"])


def prepare(case, seed):
    kind, steps = case["kind"], case["steps"]
    if kind == "ensemble":
        dims = _ensemble_dims(case)
        e = M.Ensemble(dims)
        e.configure(alpha=case["alpha"], dt=case["dt"], J=1.0, pbc=(0, 0, 0), K=case["K"], axis=(0, 0, 1), T=case["T"],
                    seed=seed, B=(0, 0, 0), dB=(0, 0, case["sweep"]), g=case["g"], open_xy=True, llg=case["llg"])
        for r, d in enumerate(dims):
            e.setSpins(r, *_start_spins(case, int(np.prod(d)), seed * 1000 + r))
        probes = [dims.index(d) for d in ENSEMBLE_SIZES if d in dims]
        return {"kind": kind, "ensemble": e, "steps": steps, "probes": probes}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    if kind == "grains":
        gr = _grains(case, seed)
        ss = M.SpinSystem(nx, ny, nz)
        ss.setSpinArrays(*(_start_spins(case, n, seed) * gr["ms"]))
        ss.setAlpha(case["alpha"])
        ss.setTimeStep(case["dt"])
        ex = M.Exchange(ss)
        ex.addPaths(gr["from"], gr["to"], gr["J"])
        ani = M.Anisotropy(ss)
        ani.addMany(np.arange(n), gr["axis"], gr["K"])
        ops = [ex, ani]
        if case["T"] > 0:
            th = M.Thermal(ss, M.Random.Philox(1000 + seed))
            th.setTemperature(case["T"])
            ops.append(th)
        z = M.AppliedField(ss)
        z.set(0, 0, case["field"])
        dip = M.Dipole(ss)
        dip.setStrength(case["g"])
        ops += [z, dip]
        return {"kind": "plan", "plan": M.Plan(ss, ops, M.LLG.new("Quaternion")), "steps": steps,
                "read": _reader(ss, n, "f32")}
    if kind == "layers":
        ss = M.SpinSystem(nx, ny, nz)
        ss.setSpinArrays(*_start_spins(case, n, seed))
        ss.setAlpha(case["alpha"])
        ss.setTimeStep(case["dt"])
        ex = M.Exchange(ss)
        # exchange within the layers only
        frm, to = _neighbours(nx, ny, nz, (1, 1, 0))
        same = frm // (nx * ny) == to // (nx * ny)
        ex.addPaths(frm[same], to[same], np.ones(int(same.sum())))
        ani = M.Anisotropy(ss)
        ani.addMany(np.arange(n), np.tile([0, 0, 1.0], (n, 1)), np.full(n, case["K"]))
        tensor = _layer_tensor(case)
        lr = M.LongRange2D(ss)

        def make(op):
            for d in range(nz):
                for s in range(nz):
                    for q, ab in enumerate(("XX", "XY", "XZ", "YX", "YY", "YZ", "ZX", "ZY", "ZZ")):
                        op.setTensorArray(d + 1, s + 1, ab, tensor[d, s, q].ravel())
        lr.setMakeDataFunction(make)
        lr.makeData()
        ops = [ex, ani]
        if case["T"] > 0:
            th = M.Thermal(ss, M.Random.Philox(1000 + seed))
            th.setTemperature(case["T"])
            ops.append(th)
        ops.append(lr)
        return {"kind": "plan", "plan": M.Plan(ss, ops, M.LLG.new("Quaternion")), "steps": steps,
                "read": _reader(ss, n, "f32")}
    ss, ops, th, llg = _film_objects(case, seed)
    read = _reader(ss, n, case["precision"])
    if kind == "rk":
        return {"kind": "rk", "rk": M.RungeKutta(ss, case["scheme"], ops, llg, temp=th), "steps": steps, "read": read}
    if th is not None:
        ops.insert(2, th)
    if kind == "script":
        return {"kind": "script", "ss": ss, "ops": ops, "llg": llg, "steps": steps, "read": read}
    return {"kind": "plan", "plan": M.Plan(ss, ops, llg), "steps": steps, "read": read}


# ---------------------------------------------------------------- one pass
def run(state):
    kind, steps = state["kind"], state["steps"]
    if kind == "plan":
        state["plan"].launch(steps)
        return state["read"]()
    if kind == "rk":
        state["rk"].step(steps)
        return state["read"]()
    if kind == "script":
        ss, ops, llg = state["ss"], state["ops"], state["llg"]
        curve = []
        for k in range(steps):
            ss.resetFields()
            for op in ops:
                op.apply(ss)
            ss.sumFields()
            llg.apply(ss)
            if k % 5 == 4:
                curve.append(ss.netMoment()[:3])
        # sums of FP32 spins: recorded as the FP32 numbers they stand for
        return state["read"]() + [np.asarray(curve, dtype=np.float32)]
    e = state["ensemble"]
    e.run(steps)
    # every replica's moment, and the spins of one particle of each size
    out = [np.asarray(e.netMoment()[:, :3], dtype=np.float32)]
    for r in state["probes"]:
        out.append(np.asarray(e.spins(r), dtype=np.float32))
    return out


# ---------------------------------------------------------------- necessary work
def _padded(n, is_open):
    if not is_open or n == 1:
        return n
    p = 1
    while p < 2 * n - 1:
        p *= 2
    return p


def _conv_work(nx, ny, nz, open_xy):
    """(k-points of the half spectrum, operations) of one dipole field: real
    transforms of three components there and back, the symmetric tensor."""
    P = [_padded(nx, open_xy), _padded(ny, open_xy), _padded(nz, True)]
    total = P[0] * P[1] * P[2]
    k = (P[0] // 2 + 1) * P[1] * P[2]
    return k, 6 * 2.5 * total * math.log2(max(2, total)) + 30 * k


def work(case):
    """Spins read and written once each step, the tensor spectrum (an eighth
    of it is distinct for a point-dipole tensor) read once a pass; the
    operations of the transforms and about 150 per site for the local terms
    and the rotation."""
    steps = case["steps"]
    if case["kind"] == "ensemble":
        b = f = 0.0
        for d in _ensemble_dims(case):
            n = d[0] * d[1] * d[2]
            b += steps * 24.0 * n
            f += steps * (_conv_work(*d, True)[1] + 150.0 * n)
        for d in ENSEMBLE_SIZES:
            b += _conv_work(*d, True)[0] * 24.0 / 4
        return {"bytes": b, "flops": f}
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    w = 8 if case.get("precision") == "f64" else 4
    evals = steps * {"RK2": 2, "RK4": 4}.get(case.get("scheme"), 1)
    if case["kind"] == "layers":
        k = (nx // 2 + 1) * ny
        return {"bytes": steps * 24.0 * n + 72.0 * nz * nz * k,
                "flops": steps * (6 * 2.5 * n * math.log2(nx * ny) + 72.0 * nz * nz * k + 150.0 * n)}
    k, f = _conv_work(nx, ny, nz, case.get("open", False))
    b = evals * 6.0 * n * w + k * 6.0 * w / 4
    if case["kind"] == "grains":
        b += steps * n * (4.0 + 16.0 + 6 * 8.0)   # moments, axes and constants, pathways
    return {"bytes": b, "flops": evals * (f + 150.0 * n)}


# ---------------------------------------------------------------- the same in 64 bits
def _philox_normals(sites, counter, seed):
    """Three standard normals per site: Philox4x32-10 words to uniforms (24
    high bits) to Box-Muller pairs."""
    m32 = 0xFFFFFFFF
    c = [sites.clone(), torch.full_like(sites, counter & m32), torch.full_like(sites, counter >> 32),
         torch.full_like(sites, 0x6D6C6232)]
    k0, k1 = seed & m32, (seed >> 32) & m32

    def mul(a, m):   # 32x32 -> (high, low) words within signed 64 bits
        lo = a * (m & 0xFFFF)
        hi = a * (m >> 16)
        t = lo + ((hi & 0xFFFF) << 16)
        return (hi >> 16) + (t >> 32), t & m32
    for r in range(10):
        if r:
            k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
    u = [((v >> 8).double() + 0.5) * 2.0 ** -24 for v in c]
    ra, rb = torch.sqrt(-2 * torch.log(u[0])), torch.sqrt(-2 * torch.log(u[2]))
    return torch.stack([ra * torch.cos(2 * math.pi * u[1]), ra * torch.sin(2 * math.pi * u[1]),
                        rb * torch.cos(2 * math.pi * u[3])])


def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _gamma6(x, y, z):
    r2 = x * x + y * y + z * z
    r2 = torch.where(r2 == 0, torch.full_like(r2, math.inf), r2)
    i3, i5 = r2 ** -1.5, r2 ** -2.5
    return [3 * x * x * i5 - i3, 3 * x * y * i5, 3 * x * z * i5, 3 * y * y * i5 - i3, 3 * y * z * i5,
            3 * z * z * i5 - i3]


class _DipoleField:
    """Field of [B, 3, nz, ny, nx] spins: the images within 1000 cells of a
    periodic film (each layer's element at source minus target height, as
    the reference defines it), or the open body."""

    def __init__(self, nx, ny, nz, g, open_xy):
        dev = _dev()
        self.n = (nz, ny, nx)
        P = [_padded(nz, True), _padded(ny, open_xy), _padded(nx, open_xy)]
        W = torch.zeros(6, *P, dtype=torch.float64, device=dev)
        for k in range(-(nz - 1), nz):
            if open_xy:
                xs, ys = torch.arange(-(nx - 1), nx, device=dev), torch.arange(-(ny - 1), ny, device=dev)
            else:
                xs = ys = torch.arange(-1000, 1001, device=dev)
            xx, yy = xs[None, :].double(), ys[:, None].double()
            # an empty z component at a distance k, everything within the sphere
            elems = _gamma6(xx + 0 * yy, yy + 0 * xx, torch.full((len(ys), len(xs)), float(k), device=dev,
                                                                 dtype=torch.float64))
            inside = (xx * xx + yy * yy + k * k <= 1000.0 ** 2) | torch.tensor(open_xy, device=dev)
            at = ((ys % P[1])[:, None] * P[2] + (xs % P[2])[None, :]).reshape(-1)
            z = (k if open_xy else -k) % P[0]
            for q in range(6):
                W[q, z].view(-1).index_add_(0, at, torch.where(inside, elems[q], torch.zeros_like(elems[q])).reshape(-1))
        self.P = P
        self.T = torch.fft.rfftn(W, dim=(1, 2, 3)) * g

    def __call__(self, s):
        S = torch.fft.rfftn(s, s=self.P, dim=(2, 3, 4))
        t = self.T
        x, y, z = S[:, 0], S[:, 1], S[:, 2]
        H = torch.stack([t[0] * x + t[1] * y + t[2] * z, t[1] * x + t[3] * y + t[4] * z,
                         t[2] * x + t[4] * y + t[5] * z], dim=1)
        nz, ny, nx = self.n
        return torch.fft.irfftn(H, s=self.P, dim=(2, 3, 4))[:, :, :nz, :ny, :nx]


class _LayerField:
    def __init__(self, case):
        t = torch.tensor(_layer_tensor(case), device=_dev())
        # the field of layer d takes the arrays set for (dest s, src d)
        self.T = torch.fft.rfftn(t.transpose(0, 1).reshape(case["nz"], case["nz"], 3, 3, case["ny"], case["nx"]),
                                 dim=(4, 5))
        self.s = (case["ny"], case["nx"])

    def __call__(self, s):
        S = torch.fft.rfftn(s[0], dim=(2, 3))
        return torch.fft.irfftn(torch.einsum("dsabyx,bsyx->adyx", self.T, S), s=self.s, dim=(2, 3))[None]


def _shift_sum(s, pbc, in_plane=False):
    """Sum of the nearest neighbours' spins."""
    h = torch.zeros_like(s)
    for ax, periodic in ((4, pbc[0]), (3, pbc[1]), (2, pbc[2])):
        n = s.shape[ax]
        if n == 1 or (in_plane and ax == 2):
            continue
        for d in (1, -1):
            r = torch.roll(s, d, dims=ax)
            if not periodic:
                r.narrow(ax, 0 if d == 1 else n - 1, 1).zero_()
            h += r
    return h


def _cross(a, b):
    return torch.stack([a[:, 1] * b[:, 2] - a[:, 2] * b[:, 1], a[:, 2] * b[:, 0] - a[:, 0] * b[:, 2],
                        a[:, 0] * b[:, 1] - a[:, 1] * b[:, 0]], dim=1)


def _advance(S, Mx, H, Hth, llg, alpha, dt, ms):
    """One LLG update of the spins S by the torque of spins Mx in field H;
    the noise enters the precession only.  Lengths restored."""
    h = H - Hth
    if llg == "Cartesian":
        gaa = GAMMA / (1 + alpha * alpha)
        S = S + dt * (-gaa * _cross(Mx, H) - alpha / ms * gaa * _cross(Mx, _cross(Mx, h)))
    else:
        w = H + alpha / ms * _cross(Mx, h)
        L = torch.sqrt((w * w).sum(1, keepdim=True))
        u = w / torch.where(L == 0, torch.ones_like(L), L)
        th = GAMMA * L * dt / (1 + alpha * alpha)
        S = S * torch.cos(th) + _cross(u, S) * torch.sin(th) + u * (u * S).sum(1, keepdim=True) * (1 - torch.cos(th))
    return S * (ms / torch.sqrt((S * S).sum(1, keepdim=True)))


def _noise(case, sites, counter, seed, shape, ms, dt):
    n = _philox_normals(sites, counter, seed)
    sd = torch.sqrt(torch.as_tensor(2 * case["alpha"] * case["T"] / (ms * dt * GAMMA)))
    return sd * n.reshape(3, *shape).transpose(0, 1)


def _cubic(s, K):
    """First-order cubic field with the reference's cubed third component in
    the first term."""
    x, y, z = s[:, 0], s[:, 1], s[:, 2]
    return torch.stack([2 * K * x * (y * y + z ** 3), 2 * K * y * (x * x + z * z), 2 * K * z * (x * x + y * y)], dim=1)


RK = {"RK2": [[0.5], [0.0, 1.0]],
      "RK4": [[0.5], [0.0, 0.5], [0.0, 0.0, 1.0], [1 / 6, 1 / 3, 1 / 3, 1 / 6]]}


def exact(case, seed):
    dev = _dev()
    if case["kind"] == "ensemble":
        return _exact_ensemble(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    n = nx * ny * nz
    shape = (1, nz, ny, nx)
    s = torch.tensor(_start_spins(case, n, seed), device=dev)
    ms = torch.ones(n, dtype=torch.float64, device=dev)
    if case["kind"] == "grains":
        gr = _grains(case, seed)
        ms = torch.tensor(gr["ms"], device=dev)
        s = s * ms
        frm, to = torch.tensor(gr["from"], device=dev).long(), torch.tensor(gr["to"], device=dev).long()
        J = torch.tensor(gr["J"], device=dev) / (ms[frm] * ms[to])
        axis = torch.tensor(gr["axis"].T.copy(), device=dev).reshape(1, 3, *shape[1:])
        K = torch.tensor(gr["K"], device=dev).reshape(1, 1, *shape[1:])
    S = s.reshape(1, 3, *shape[1:])
    ms = ms.reshape(1, 1, *shape[1:])
    sites = torch.arange(n, dtype=torch.int64, device=dev)
    long_range = _LayerField(case) if case["kind"] == "layers" else _DipoleField(nx, ny, nz, case["g"],
                                                                                 case.get("open", False))
    pbc = (0, 0, 0) if case.get("open") else (1, 1, 0)

    def local(S, B):
        if case["kind"] == "grains":
            flat = S.reshape(3, n)
            h = torch.zeros_like(flat).index_add_(1, to, flat[:, frm] * J).reshape(S.shape)
            h = h + 2 * K * (S * axis).sum(1, keepdim=True) / (ms * ms) * axis
            h[:, 2] += case["field"]
            return h
        h = _shift_sum(S, pbc, in_plane=case["kind"] == "layers")
        if case.get("cubic"):
            h = h + _cubic(S, case["K"])
        else:
            h[:, 2] += 2 * case["K"] * S[:, 2]
        h[:, 0] += B
        return h

    B, llg, dt, alpha = case.get("field", 0.0), case.get("llg", "Quaternion"), case["dt"], case["alpha"]
    curve = []
    for k in range(case["steps"]):
        noise = _noise(case, sites, k, 1000 + seed, shape, ms, dt) if case["T"] > 0 else torch.zeros_like(S)
        if case["kind"] == "rk":
            table = RK[case["scheme"]]
            stages = [(S, local(S, B) + long_range(S))]
            for i, row in enumerate(table):
                zero = torch.zeros_like(S)
                new = _advance(S, S, stages[0][1], zero, llg, alpha, row[0] * dt, ms)
                for j in range(1, len(row)):
                    if row[j] != 0:
                        new = _advance(new, stages[j][0], stages[j][1], zero, llg, alpha, row[j] * dt, ms)
                if i < len(table) - 1:
                    stages.append((new, local(new, B) + long_range(new)))
            S = new
            if case["T"] > 0:
                S = _advance(S, S, noise, noise, llg, alpha, dt, ms)
            continue
        H = (local(S, B) if case["kind"] != "layers" else local(S, 0.0)) + long_range(S) + noise
        S = _advance(S, S, H, noise, llg, alpha, dt, ms)
        B += case.get("sweep", 0.0)
        if case["kind"] == "script" and k % 5 == 4:
            curve.append(S.reshape(3, n).sum(1).tolist())
    out = [v.cpu().numpy() for v in S.reshape(3, n)]
    if case["kind"] == "script":
        out.append(np.asarray(curve))
    return out


def _exact_ensemble(case, seed):
    dev = _dev()
    dims = _ensemble_dims(case)
    order = []   # sizes in order of first appearance: replicas share one noise stream over this packing
    for d in dims:
        if d not in order:
            order.append(d)
    moments = np.zeros((len(dims), 3))
    probes = {}
    base = 0
    for d in order:
        nx, ny, nz = d
        n = nx * ny * nz
        reps = [r for r, e in enumerate(dims) if e == d]
        s = np.stack([_start_spins(case, n, seed * 1000 + r) for r in reps])
        S = torch.tensor(s, device=dev).reshape(len(reps), 3, nz, ny, nx)
        sites = base + torch.arange(n * len(reps), dtype=torch.int64, device=dev)
        base += n * len(reps)
        dip = _DipoleField(nx, ny, nz, case["g"], True)
        ms = torch.ones((), dtype=torch.float64, device=dev)
        B = 0.0
        for k in range(case["steps"]):
            H = _shift_sum(S, (0, 0, 0)) + dip(S)
            H[:, 2] += 2 * case["K"] * S[:, 2] + B
            noise = (_noise(case, sites, k, seed, (len(reps), nz, ny, nx), ms, case["dt"]) if case["T"] > 0
                     else torch.zeros_like(S))
            S = _advance(S, S, H + noise, noise, case["llg"], case["alpha"], case["dt"], ms)
            B += case["sweep"]
        flat = S.reshape(len(reps), 3, n).cpu().numpy()
        for i, r in enumerate(reps):
            moments[r] = flat[i].sum(1)
        probes[d] = flat[0]
    return [moments] + [probes[d] for d in ENSEMBLE_SIZES if d in probes]
