"""The workloads this framework is measured on: what a user's program asks of
its public entry points (`paraiso_gb300`), from one generation of the smallest
example mesh to the largest grids of the benchmark.

Families: `life` (examples/Life), `hydro` (examples/Hydro, periodic and open,
FP32 and FP64), `ensemble` (uneven Hydro grids advanced together), `adjoint`
(the gradient of a loss over many Hydro steps) and `graph` (a machine compiled
from its Orthotope Machine graph).
"""
import math

import numpy as np
import torch

import paraiso_gb300 as pg
from paraiso_gb300 import omgraph as og
from paraiso_gb300 import omgraph_examples as examples

FIELDS = ("density", "velocity0", "velocity1", "pressure")
JET_GAMMA = 5.0 / 3.0   # examples/Hydro
KH_GAMMA = 1.4          # the Kelvin-Helmholtz configurations
HYDRO_FLOPS = 549       # per cell and step, counted on the scheme
ADJOINT_FLOPS = 3 * HYDRO_FLOPS  # forward, and a reverse of about twice that
LIFE_OPS = 0.5          # per cell and generation: 16 word operations per 32 cells


# --------------------------------------------------------------------------
# cases
# --------------------------------------------------------------------------
def _life(n0, n1, gens, host=False, p=0.3):
    return {"family": "life", "n0": n0, "n1": n1, "gens": gens, "host": host, "p": p}


def _hydro(n0, n1, steps, precision=32, boundary="cyclic"):
    return {"family": "hydro", "n0": n0, "n1": n1, "steps": steps, "precision": precision,
            "boundary": boundary}


def _ensemble(count, lo, hi, step, size_seed, steps):
    return {"family": "ensemble", "count": count, "lo": lo, "hi": hi, "step": step,
            "size_seed": size_seed, "steps": steps}


def _adjoint(n0, n1, steps):
    return {"family": "adjoint", "n0": n0, "n1": n1, "steps": steps}


def _graph(machine, n0, n1, steps):
    return {"family": "graph", "machine": machine, "n0": n0, "n1": n1, "steps": steps}


def listed():
    return [
        # examples/Life/main.cpp: its 80 x 48 mesh, one proceed() per shown
        # generation, the cells read on the host each time
        dict(_life(80, 48, 1, host=True), name="life_example_step"),
        # the small benchmark grid: 1000 generations and their populations
        dict(_life(128, 128, 1000), name="life_128"),
        # a mesh whose rows are no whole number of packed words
        dict(_life(1000, 700, 100), name="life_ragged"),
        # an ordinary grid that fits in the L2
        dict(_life(2048, 2048, 100), name="life_2048"),
        # the large benchmark grid
        dict(_life(16384, 16384, 100), name="life_16384"),
        # examples/Hydro as generated: 1024^2, double, open, jet inflow
        dict(_hydro(1024, 1024, 4, 64, "open"), name="hydro_example_f64"),
        # a double-precision reference run on a small periodic grid
        dict(_hydro(384, 256, 10, 64), name="hydro_f64_small"),
        # the large Kelvin-Helmholtz benchmark grid, single precision
        dict(_hydro(4096, 4096, 20), name="hydro_4096"),
        # a grid whose sides suit no tile
        dict(_hydro(500, 300, 20), name="hydro_ragged"),
        # 64 uneven grids advanced together
        dict(_ensemble(64, 256, 2048, 32, 1, 10), name="ensemble_64"),
        # the gradient of a loss over 200 steps
        dict(_adjoint(1024, 1024, 200), name="adjoint_1024"),
        # examples/Hydro compiled from its graph, single precision
        dict(_graph("hydro", 1024, 1024, 10), name="graph_hydro"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _sides(rng, lo, hi, most):
    """Two sides in [lo, hi] with a product of at most `most`; half of the
    draws are whole multiples of 32, as tuned grids are."""
    while True:
        n0, n1 = _log(rng, lo, hi), _log(rng, lo, hi)
        if rng.random() < 0.5:
            n0, n1 = max(64, n0 // 32 * 32), max(64, n1 // 32 * 32)
        if n0 * n1 <= most:
            return n0, n1


def draw(rng):
    family = rng.choice(("life", "life", "life", "hydro", "hydro", "hydro", "hydro", "ensemble",
                         "adjoint", "graph"))
    if family == "life":
        n0, n1 = _sides(rng, 48, 16384, 16384 * 16384)
        gens = _log(rng, 1, 1000)
        return _life(n0, n1, min(gens, max(1, 27_000_000_000 // (n0 * n1))),
                     host=n0 * n1 <= 1 << 16 and gens < 10, p=round(rng.uniform(0.1, 0.6), 3))
    if family == "hydro":
        precision = rng.choice((32, 32, 64))
        boundary = rng.choice(("cyclic", "cyclic", "open"))
        n0, n1 = _sides(rng, 40, 4096, 1 << (24 if precision == 32 else 20))
        most = (330_000_000 if precision == 32 else 4_200_000) // (n0 * n1)
        return _hydro(n0, n1, max(1, min(_log(rng, 1, 40), most)), precision, boundary)
    if family == "ensemble":
        lo = _log(rng, 64, 400)
        return _ensemble(_log(rng, 2, 40), lo, lo + 32 * _log(rng, 1, 32), rng.choice((32, 32, 4)),
                         rng.randrange(1, 1 << 30), _log(rng, 1, 10))
    if family == "adjoint":
        n0, n1 = _sides(rng, 96, 1536, 1 << 20)
        return _adjoint(n0, n1, _log(rng, 4, 100))
    n0, n1 = _sides(rng, 96, 2048, 1 << 20)
    return _graph(rng.choice(("hydro", "life")), n0, n1, _log(rng, 1, 20))


# --------------------------------------------------------------------------
# inputs
# --------------------------------------------------------------------------
def _rng(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _life_start(case, seed):
    """i.i.d. cells, alive with probability p, as [y, x] int32."""
    u = torch.rand(case["n1"], case["n0"], generator=_rng(seed), device="cuda")
    return (u < case.get("p", 0.3)).to(torch.int32)


def _kh_start(n0, n1, seed, dtype, bump=False):
    """Kelvin-Helmholtz shear layers on the unit square with seeded noise in
    the transverse velocity; `bump` adds a pressure peak, so that one cell
    alone sets the time step."""
    x = ((torch.arange(n0, device="cuda", dtype=torch.float64) + 0.5) / n0)[None, :]
    y = ((torch.arange(n1, device="cuda", dtype=torch.float64) + 0.5) / n1)[:, None]
    band = ((y - 0.5).abs() < 0.25).expand(n1, n0)
    noise = torch.rand(n1, n0, generator=_rng(seed), device="cuda", dtype=torch.float64)
    rho = torch.where(band, 2.0, 1.0).double()
    v0 = torch.where(band, 0.5, -0.5).double()
    v1 = 0.01 * torch.sin(4 * math.pi * x) + 0.01 * (2 * noise - 1)
    p = torch.full((n1, n0), 2.5, device="cuda", dtype=torch.float64)
    if bump:
        p = p + 1.5 * torch.exp(-((x - 0.37) ** 2 + (y - 0.46) ** 2) / 0.01)
    return [t.contiguous().to(dtype) for t in (rho, v0, v1, p)]


def _jet_start(n0, n1, seed, dtype):
    """The quiescent ambient gas of examples/Hydro's `init` with a seeded
    perturbation, on the memory array of an open mesh (margins of 3)."""
    x = ((torch.arange(n0 + 6, device="cuda", dtype=torch.float64) - 3) / n0)[None, :]
    factor = 1 + 1e-3 * torch.sin(6 * math.pi * x)
    noise = torch.rand(n1 + 6, n0 + 6, generator=_rng(seed), device="cuda", dtype=torch.float64)
    rho = factor * JET_GAMMA ** 2 * 10 * (1 + 0.02 * (noise - 0.5))
    p = 0.6 * factor * (1 + 0.02 * (noise.flip(0) - 0.5))
    zero = torch.zeros_like(rho)
    return [t.contiguous().to(dtype) for t in (rho, zero, zero, p)]


def _hydro_start(case, seed, dtype):
    start = _jet_start if case["boundary"] == "open" else _kh_start
    return start(case["n0"], case["n1"], seed, dtype)


def _instances(case):
    return pg.ensemble_sizes(case["count"], case["size_seed"], case["lo"], case["hi"], case["step"])


def _target(n0, n1, seed, dtype):
    """A smooth field around the mean density: eight random Fourier modes."""
    r = np.random.RandomState(int(seed) % (1 << 31))
    x = ((np.arange(n0) + 0.5) / n0)[None, :]
    y = ((np.arange(n1) + 0.5) / n1)[:, None]
    f = np.full((n1, n0), 1.5)
    for _ in range(8):
        kx, ky, a, ph = r.randint(-3, 4), r.randint(-3, 4), r.uniform(0.02, 0.1), r.uniform(0, 6.28)
        f += a * np.cos(2 * np.pi * (kx * x + ky * y) + ph)
    return f.astype(dtype)


def _set_scalars(m, case):
    real = np.float32 if case.get("precision", 32) == 32 else np.float64
    for name, v in (("time", 0.0), ("cfl", 0.4), ("extent0", 1.0), ("extent1", 1.0),
                    ("dR0", float(real(1) / real(case["n0"]))),
                    ("dR1", float(real(1) / real(case["n1"])))):
        m.set_scalar(name, v)


def _write(m, name, t):
    m.write_from_pointer(name, t.data_ptr(), t.numel() * t.element_size())


class _View:
    """Device memory of a machine, which lives as long as the tensor on it."""

    def __init__(self, machine, ptr, shape, typestr):
        self.machine = machine
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr,
                                         "version": 2}


def _on_device(m, name):
    """A static of the machine where it lies on the GPU."""
    typestr = np.dtype(m.array_dtypes[name]).str
    return torch.as_tensor(_View(m, m.device_pointer(name), m.memory_shape, typestr), device="cuda")


def prepare(case, seed):
    family = case["family"]
    state = {"case": case}
    if family == "life":
        m = pg.Life((case["n0"], case["n1"]))
        start = _life_start(case, seed)
        torch.cuda.synchronize()
        _write(m, "cell", start)
    elif family == "hydro":
        m = pg.Hydro((case["n0"], case["n1"]), precision=case["precision"],
                     gamma=JET_GAMMA if case["boundary"] == "open" else KH_GAMMA,
                     boundary=pg.OPEN if case["boundary"] == "open" else pg.CYCLIC)
        _set_scalars(m, case)
        dtype = torch.float64 if case["precision"] == 64 else torch.float32
        start = _hydro_start(case, seed, dtype)
        torch.cuda.synchronize()
        for name, t in zip(FIELDS, start):
            _write(m, name, t)
    elif family == "ensemble":
        sizes = _instances(case)
        m = pg.Ensemble(sizes, precision=32, gamma=KH_GAMMA)
        for k, (n0, n1) in enumerate(sizes):
            start = _kh_start(n0, n1, seed + 7919 * k, torch.float32)
            torch.cuda.synchronize()
            for name, t in zip(FIELDS, start):
                m.write_from_pointer(k, name, t.data_ptr(), t.numel() * 4)
        cells = sum(a * b for a, b in sizes)
        state["out"] = {f: torch.empty(cells, device="cuda") for f in FIELDS}
    elif family == "adjoint":
        m = pg.Hydro((case["n0"], case["n1"]), precision=32, gamma=KH_GAMMA)
        _set_scalars(m, case)
        state["start"] = _kh_start(case["n0"], case["n1"], seed, torch.float32, bump=True)
        state["target"] = _target(case["n0"], case["n1"], seed, np.float32)
        torch.cuda.synchronize()
    else:
        n = (case["n0"], case["n1"])
        if case["machine"] == "life":
            m = pg.GraphMachine(examples.life(n))
            start = _life_start(case, seed)
            torch.cuda.synchronize()
            _write(m, "cell", start)
        else:
            m = pg.GraphMachine(examples.hydro(n, KH_GAMMA, "cyclic", og.Float))
            _set_scalars(m, case)
            start = _kh_start(*n, seed, torch.float32)
            torch.cuda.synchronize()
            for name, t in zip(FIELDS, start):
                _write(m, name, t)
    state["machine"] = m
    return state


# --------------------------------------------------------------------------
# one pass
# --------------------------------------------------------------------------
def run(state):
    case, m = state["case"], state["machine"]
    family = case["family"]
    if family == "life":
        m.proceed(case["gens"])
        cells = m.read("cell") if case["host"] else _on_device(m, "cell")
        return {"cell": cells, "population": m.population_history(case["gens"])}
    if family == "hydro":
        m.proceed(case["steps"])
        out = {f: _on_device(m, f) for f in FIELDS}
        return dict(out, dt=m.dt_history(case["steps"]))
    if family == "ensemble":
        m.step(case["steps"])
        at = 0
        for k, (n0, n1) in enumerate(m.sizes):
            for f in FIELDS:
                m.read_to_pointer(k, f, state["out"][f].data_ptr() + 4 * at, 4 * n0 * n1)
            at += n0 * n1
        return state["out"]
    if family == "adjoint":
        # an iteration of a fit: back to the current guess, then its gradient
        for name, t in zip(FIELDS, state["start"]):
            _write(m, name, t)
        loss, grads = m.adjoint_run(case["steps"], state["target"])
        return dict(zip(FIELDS, grads), loss=loss)
    if case["machine"] == "life":
        m.run("proceed", case["steps"])
        return {"cell": _on_device(m, "cell"), "population": int(m.get_scalar("population"))}
    m.run("proceed", case["steps"])
    return {f: _on_device(m, f) for f in FIELDS}


def work(case):
    family = case["family"]
    if family == "ensemble":
        cells = sum(a * b for a, b in _instances(case))
        return {"bytes": 32 * cells, "flops": HYDRO_FLOPS * cells * case["steps"]}
    cells = case["n0"] * case["n1"]
    if family == "life" or (family == "graph" and case["machine"] == "life"):
        gens = case["gens"] if family == "life" else case["steps"]
        return {"bytes": 8 * cells + 4 * gens, "flops": LIFE_OPS * cells * gens}
    if family == "adjoint":
        return {"bytes": 4 * (4 + 1 + 4) * cells, "flops": ADJOINT_FLOPS * cells * case["steps"]}
    size = case.get("precision", 32) // 8
    return {"bytes": 8 * size * cells, "flops": HYDRO_FLOPS * cells * case["steps"]}


# --------------------------------------------------------------------------
# the same results in 64 bits, by plain torch
# --------------------------------------------------------------------------
def _life_exact(cells, gens):
    c = cells.to(torch.uint8)
    pops = []
    for _ in range(gens):
        rows = c + c.roll(1, 0) + c.roll(-1, 0)
        near = rows + rows.roll(1, 1) + rows.roll(-1, 1)  # the cell itself included
        c = ((near == 3) | ((near == 4) & (c == 1))).to(torch.uint8)
        pops.append(c.sum(dtype=torch.int64))
    return c.to(torch.int32), torch.stack(pops).to(torch.int32).cpu()


def _conserved(g, q):
    rho, v0, v1, p = q
    return rho, rho * v0, rho * v1, 0.5 * rho * (v0 * v0 + v1 * v1) + p / (g - 1)


def _primitive(g, u):
    rho, m0, m1, e = u
    v0, v1 = m0 / rho, m1 / rho
    p = (g - 1) * (e - 0.5 * (v0 * m0 + v1 * m1))
    return rho.clamp_min(1e-2), v0, v1, p.clamp_min(1e-2)


def _flux(u, un, p, ax):
    rho, m0, m1, e = u
    f = [rho * un, m0 * un, m1 * un, (e + p) * un]
    f[1 + ax] = f[1 + ax] + p
    return f


def _sound(g, q):
    return torch.sqrt(g * q[3] / q[0])


def _hllc(g, L, R, ax):
    """Fluxes between the states left (L) and right (R) of a wall."""
    cL, cR = _sound(g, L), _sound(g, R)
    uL, uR = L[1 + ax], R[1 + ax]
    star = (L[3] + R[3]) / 2 - (L[0] + R[0]) / 2 * (cL + cR) / 2 * (uR - uL)
    star = star.clamp_min(0.0)

    def q(p):
        return torch.where(p <= star, torch.ones_like(p),
                           torch.sqrt((1 + (g + 1) / (2 * g) * (star / p - 1)).clamp_min(1e-300)))

    sL, sR = uL - cL * q(L[3]), uR + cR * q(R[3])
    aL, aR = L[0] * (sL - uL), R[0] * (sR - uR)
    s = (R[3] - L[3] + aL * uL - aR * uR) / (aL - aR)

    def side(W, S):
        u = _conserved(g, W)
        un = W[1 + ax]
        plain = _flux(u, un, W[3], ax)
        rho = W[0] * (S - un) / (S - s)
        v = [W[1], W[2]]
        v[ax] = s
        e = rho * (u[3] / W[0] + (s - un) * (s + W[3] / W[0] / (S - un)))
        p = (g - 1) * (e - 0.5 * rho * (v[0] * v[0] + v[1] * v[1]))
        return plain, _flux((rho, rho * v[0], rho * v[1], e), s, p, ax)

    (fL, fLs), (fR, fRs) = side(L, sL), side(R, sR)
    return [torch.where(sL > 0, a, torch.where(s > 0, b, torch.where(sR > 0, c, d)))
            for a, b, c, d in zip(fL, fLs, fRs, fR)]


def _minmod(a, b):
    return torch.where(a * b <= 0, torch.zeros_like(a), torch.where(a.abs() < b.abs(), a, b))


def _advance(g, base, from_, dt, dR, order):
    """base advanced by dt with the walls reconstructed from `from_`."""
    u = _conserved(g, base)
    for ax in (0, 1):
        d = 1 - ax  # axis 0 is the fast one
        if order == 1:
            L, R = [q.roll(1, d) for q in from_], from_
        else:
            L, R = [], []
            for q in from_:
                step = q - q.roll(1, d)
                slope = _minmod(step, step.roll(-1, d))
                L.append((q + slope / 2).roll(1, d))
                R.append(q - slope / 2)
        f = _hllc(g, L, R, ax)
        u = [a + dt / dR[ax] * (b - b.roll(-1, d)) for a, b in zip(u, f)]
    return _primitive(g, u)


def _hydro_step(g, q, dR, cfl):
    c = _sound(g, q)
    ts = torch.minimum(dR[0] / (c + q[1].abs()), dR[1] / (c + q[2].abs()))
    dt = cfl * ts.min()
    half = _advance(g, q, q, dt / 2, dR, 1)
    return _advance(g, q, half, dt, dR, 2), dt


def _jet_margins(n0, n1, dR):
    """The margin cells of an open mesh and the state they hold."""
    ix = torch.arange(-3, n0 + 3, device="cuda")[None, :].expand(n1 + 6, n0 + 6)
    iy = torch.arange(-3, n1 + 3, device="cuda")[:, None].expand(n1 + 6, n0 + 6)
    out = (ix < 0) | (iy < 0) | (ix >= n0) | (iy >= n1)
    jet = (dR[1] * iy > 0.47) & (dR[1] * iy < 0.53) & (ix < 0)
    one = torch.ones(n1 + 6, n0 + 6, device="cuda", dtype=torch.float64)
    rho = JET_GAMMA ** 2 * torch.where(jet, one, 10 * one)
    return out, (rho, torch.where(jet, 6 * one, 0 * one), 0 * one, 0.6 * one)


def _hydro_exact(case, start, steps):
    real = np.float32 if case.get("precision", 32) == 32 else np.float64
    dR = [float(real(1) / real(case["n0"])), float(real(1) / real(case["n1"]))]
    q, dts = [t.double() for t in start], []
    if case.get("boundary", "cyclic") == "cyclic":
        for _ in range(steps):
            q, dt = _hydro_step(KH_GAMMA, q, dR, 0.4)
            dts.append(float(dt))
        return q, dts
    out, jet = _jet_margins(case["n0"], case["n1"], dR)
    for _ in range(steps):
        q = [torch.where(out, j, a) for a, j in zip(q, jet)]
        q, dt = _hydro_step(JET_GAMMA, q, dR, 0.4)
        dts.append(float(dt))
    return [torch.where(out, torch.zeros_like(a), a) for a in q], dts


def _adjoint_exact(case, start, target, steps):
    """Loss and gradient by reverse accumulation, one step's graph at a time."""
    real = np.float32
    dR = [float(real(1) / real(case["n0"])), float(real(1) / real(case["n1"]))]
    kept = [[t.double() for t in start]]
    with torch.no_grad():
        for _ in range(steps):
            kept.append(_hydro_step(KH_GAMMA, kept[-1], dR, 0.4)[0])
    d = kept[-1][0] - torch.as_tensor(target, device="cuda").double()
    cot = [2 * d / d.numel()] + [torch.zeros_like(d) for _ in range(3)]
    for k in range(steps - 1, -1, -1):
        with torch.enable_grad():
            q = [t.clone().requires_grad_() for t in kept[k]]
            new, _ = _hydro_step(KH_GAMMA, q, dR, 0.4)
            cot = torch.autograd.grad(new, q, cot)
    return float((d * d).mean()), [c.cpu().numpy() for c in cot]


def exact(case, seed):
    family = case["family"]
    if family == "life" or (family == "graph" and case["machine"] == "life"):
        gens = case["gens"] if family == "life" else case["steps"]
        cells, pops = _life_exact(_life_start(case, seed), gens)
        return {"cell": cells, "population": pops.numpy() if family == "life" else int(pops[-1])}
    if family == "hydro":
        dtype = torch.float64 if case["precision"] == 64 else torch.float32
        q, dts = _hydro_exact(case, _hydro_start(case, seed, dtype), case["steps"])
        return dict(zip(FIELDS, q), dt=np.array(dts))
    if family == "ensemble":
        parts = {f: [] for f in FIELDS}
        for k, (n0, n1) in enumerate(_instances(case)):
            one = {"n0": n0, "n1": n1, "precision": 64}  # an ensemble keeps dR in 64 bits
            q, _ = _hydro_exact(one, _kh_start(n0, n1, seed + 7919 * k, torch.float32),
                                case["steps"])
            for f, t in zip(FIELDS, q):
                parts[f].append(t.reshape(-1).float())
        return {f: torch.cat(v) for f, v in parts.items()}
    if family == "adjoint":
        if case["steps"] * case["n0"] * case["n1"] > 220_000_000:
            return None
        loss, grads = _adjoint_exact(
            case, _kh_start(case["n0"], case["n1"], seed, torch.float32, bump=True),
            _target(case["n0"], case["n1"], seed, np.float32), case["steps"])
        return dict(zip(FIELDS, grads), loss=loss)
    q, _ = _hydro_exact(case, _kh_start(case["n0"], case["n1"], seed, torch.float32),
                        case["steps"])
    return dict(zip(FIELDS, q))
