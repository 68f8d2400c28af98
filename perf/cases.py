"""The workloads this package's speed is measured on, each through the calls a user's program
makes: molecular-dynamics runs of one cell and of batches of cells (``MDDriver``,
``BatchedMDDriver``), the drop-in run loop, a whole session from host arrays to results, g(r),
and the warm-start network's training.

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges, ``prepare(case, seed)``
what a program holds before the call, ``run(state)`` one pass, ``work(case)`` the bytes and
operations a pass cannot do without, ``exact(case, seed)`` the same results in 64-bit torch.

The potentials are generic many-body tables (inverse-power pair terms and densities, a
square-root embedding, a smooth cutoff) on the grids of the files the package is used with:
2,000 nodes to 6.8 A for the two-element alloy, 10,000 to 5.5065 A for the single element,
10,001 to 6.5 A for the ternary. Cells start with every atom displaced by its thermal amplitude
and Maxwell-Boltzmann velocities, so a pass meets the distances of a thermalised crystal.

Results of FP64 runs are float64. The mixed-precision path evaluates its pair terms in FP32;
its results are kept in float32, the precision they carry.
"""

import math
import os
import sys

import numpy as np
import torch

import mdelast_b200
from mdelast_b200.lattice import initial_state
from mdelast_b200.mlp import MLP
from mdelast_b200.potentials import SetflTables, make_objects
from mdelast_b200.systems import Cell, make_batch, make_driver
from mdelast_b200.units import Units as U

_LIB = os.path.join(os.path.dirname(os.path.abspath(mdelast_b200.__file__)), "lib")
if _LIB not in sys.path:
    sys.path.insert(0, _LIB)

# per element: symbol, Z, atomic weight, length scale of the pair and density terms [A], set
# for a zero-temperature lattice constant near the real one's
_ELEMENTS = {"cu": [("Cu", 29, 63.546, 3.70)],
             "cuzn": [("Zn", 30, 65.38, 3.83), ("Cu", 29, 63.546, 3.685)],
             "nialco": [("Ni", 28, 58.6934, 3.52), ("Al", 13, 26.9815, 4.02),
                        ("Co", 27, 58.9332, 3.54)]}
# nodes in r and rho, cutoff [A]
_GRID = {"cu": (10000, 10000, 5.5065), "cuzn": (2000, 2000, 6.8), "nialco": (10001, 10001, 6.5)}
_EPS, _C, _RHO_UNIT, _RHO_MAX = 0.012382, 39.432, 120.0, 8.0  # eV, -, -, A^-3
_TAU_T, _TAU_P, _SKIN, _REBUILD = 5e-14, 5e-13, 1.2, 20
_FIELDS = ("epot_atom", "epot_eam_atom", "ekin_atom", "etot_cons", "virial", "total_laplacian",
           "total_force2", "temperature_kin", "temperature_conf_inverse", "pressure", "volume",
           "born_stress_tensor", "stress_tensor", "born_elasticity_tensor")
_LOOP_FIELDS = tuple(f for f in _FIELDS if f not in ("virial", "volume"))


def listed():
    return [
        # the smallest call: the reference's run loop on the 500-atom single-element cell, one
        # integrate() and its reads per step
        dict(name="loop_500_fp64", kind="loop", pot="cu", side=5, ensemble=1, T=300.0, dt=1.0,
             precision="fp64", steps=20),
        # the same example as its script sets it up: no neighbour list (an all-pairs search
        # in every step), NPT, g(r) of the production steps
        dict(name="allpairs_500_npt_fp64", kind="loop", pot="cu", side=5, ensemble=2, T=300.0,
             dt=1.0, precision="fp64", steps=20, neighbors=False, gr=True),
        # the 500-atom alloy sample case, NPT stage: 100 steps of its 50,000, every one sampled
        dict(name="run_500_npt_fp64", kind="run", pot="cuzn", side=5, x=0.06, ensemble=2, T=300.0,
             precision="fp64", steps=100),
        # the plain FP64 path on the 13,500-atom cell
        dict(name="run_13500_nvt_fp64", kind="run", pot="cuzn", side=15, x=0.06, ensemble=1,
             T=300.0, precision="fp64", steps=100),
        # warm-start training set: 64 cells of 2,048 atoms in NPT, every fifth step sampled
        dict(name="batch_64x2048_npt_mixed", kind="run", pot="cuzn", side=8, x=0.15, ensemble=2,
             T=450.0, precision="mixed", steps=40, replicas=64, stride=5),
        # the throughput workload: 16 cells of 13,500 atoms, mixed precision
        dict(name="batch_16x13500_nvt_mixed", kind="run", pot="cuzn", side=15, x=0.06, ensemble=1,
             T=300.0, precision="mixed", steps=40, replicas=16),
        # the 32,000-atom ordered cell at 5 K
        dict(name="run_32000_ordered_mixed", kind="run", pot="cuzn", side=20, x=0.75, ordered=True,
             ensemble=1, T=5.0, precision="mixed", steps=40),
        # 64 uneven cells: 256 to 32,000 atoms, their own compositions and temperatures
        dict(name="batch_64_uneven_mixed", kind="run", pot="cuzn", side=4, side_max=20, x=0.3,
             ensemble=1, T=900.0, precision="mixed", steps=20, replicas=64),
        # the largest single cell: ternary, 108,000 atoms, every fifth step sampled
        dict(name="run_108000_ternary_mixed", kind="run", pot="nialco", side=30, ensemble=1,
             T=300.0, precision="mixed", steps=20, stride=5),
        # a whole session: batch built from host arrays, every step's observables read, final
        # positions and velocities
        dict(name="session_4x13500_mixed", kind="session", pot="cuzn", side=15, x=0.06, ensemble=1,
             T=300.0, precision="mixed", steps=20, replicas=4),
        # g(r) and its partials of the 13,500-atom cell
        dict(name="gr_13500", kind="gr", pot="cuzn", side=15, x=0.06, ensemble=1, T=300.0,
             precision="fp64"),
        # the network's training on 2,048 runs, 200 steps, and its proposals
        dict(name="mlp_train_2048", kind="mlp", rows=2048, inputs=2, steps=200),
    ]


def draw(rng):
    """A case of the listed ranges: sizes over their logarithm, odd atom counts (vacancies)
    and uneven edges among them, every option."""
    kind = rng.choice(["run", "run", "run", "run", "loop", "session", "gr", "mlp"])
    if kind == "mlp":
        return dict(kind="mlp", rows=int(round(math.exp(rng.uniform(math.log(97), math.log(2048))))),
                    inputs=rng.choice([2, 3]), steps=rng.randrange(50, 201))
    side_hi = {"run": 22, "loop": 12, "session": 15, "gr": 16}[kind]
    side = int(round(math.exp(rng.uniform(math.log(4.6), math.log(side_hi)))))
    pot = rng.choice(["cuzn", "cuzn", "cuzn", "cu", "nialco"])
    case = dict(kind=kind, pot=pot, side=side, side_z=side + rng.choice([0, 0, 1, 2]),
                x=round(rng.uniform(0.0, 0.3), 3), vacancies=rng.choice([0, 0, 1, 2, 3, 5, 7]),
                ensemble=rng.choice([0, 1, 1, 2]), T=round(math.exp(rng.uniform(math.log(5.0), math.log(900.0))), 1),
                precision=rng.choice(["fp64", "mixed"]), dt=rng.choice([1.0, 2.0]))
    atoms = 4 * side * side * case["side_z"]
    if kind in ("run", "session"):
        most = max(1, min(64, 200_000 // atoms))
        case["replicas"] = int(round(math.exp(rng.uniform(0.0, math.log(most + 0.4)))))
    if kind != "gr":
        case["steps"] = rng.randrange(10, 41) if kind == "run" else rng.randrange(5, 21)
    if kind == "run":
        case["stride"] = rng.choice([1, 1, 5])
    if kind == "loop":
        case["neighbors"] = rng.random() < 0.8
    if pot == "cuzn" and kind != "gr" and rng.random() < 0.15:
        case["interpolation"] = "bspline"
    return case


# ------------------------------------------------------------------------------ inputs
def _derivs(f, x):
    """Values, first and second derivatives of f at the nodes x, by automatic differentiation."""
    x = torch.tensor(x, dtype=torch.float64, requires_grad=True)
    y = f(x)
    d1, = torch.autograd.grad(y.sum(), x, create_graph=True)
    d2, = torch.autograd.grad(d1.sum(), x)
    return y.detach().numpy(), d1.detach().numpy(), d2.numpy()


_TABLES = {}


def _tables(pot):
    """Node arrays (cgs) of one potential."""
    if pot in _TABLES:
        return _TABLES[pot]
    els, (n_r, n_rho, rc) = _ELEMENTS[pot], _GRID[pot]
    r, rho = np.linspace(0.0, rc, n_r), np.linspace(0.0, _RHO_MAX, n_rho)

    def cut(x):  # 1 up to 1.5 A below the cutoff, then a quintic step to 0
        u = ((x - (rc - 1.5)) / 1.5).clamp(0.0, 1.0)
        return 1.0 - u ** 3 * (10.0 - 15.0 * u + 6.0 * u * u)

    def power(a, n):
        return lambda x: (a * a / (x * x + 0.36)) ** (0.5 * n) * cut(x)

    phi, den, emb = [], [], []
    for j in range(len(els)):
        for i in range(j + 1):
            pair = power(0.5 * (els[i][3] + els[j][3]), 9)
            phi.append(_derivs(lambda x: _EPS * pair(x), r))
        dens = power(els[j][3], 6)
        den.append(_derivs(lambda x: dens(x) / _RHO_UNIT, r))
        emb.append(_derivs(lambda y: -_EPS * _C * (torch.sqrt(_RHO_UNIT * y + 0.01) - 0.1), rho))
    A, A3 = U.angstrom, U.angstrom ** 3
    t = SetflTables(
        elements=[list(e) for e in els], n_r=n_r, dr=rc * A / (n_r - 1), n_rho=n_rho,
        drho=_RHO_MAX / A3 / (n_rho - 1), rcut=rc * A, rhomax=_RHO_MAX / A3, rmin_fatal=1e-2 * A,
        phi=np.array([p[0] for p in phi]) * U.ev, dphi=np.array([p[1] for p in phi]) * U.ev / A,
        d2phi=np.array([p[2] for p in phi]) * U.ev / A ** 2,
        rho=np.array([p[0] for p in den]) / A3, drho_dr=np.array([p[1] for p in den]) / A3 / A,
        d2rho_dr2=np.array([p[2] for p in den]) / A3 / A ** 2,
        F=np.array([p[0] for p in emb]) * U.ev, dF=np.array([p[1] for p in emb]) * U.ev * A3,
        d2F=np.array([p[2] for p in emb]) * U.ev * A3 ** 2, source="generic")
    _TABLES[pot] = t
    return t


_BASIS = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])


def _cell(case, rs, side, x, T):
    """One FCC cell, thermally displaced, with its velocities and thermostat state."""
    t = _tables(case["pot"])
    edge = np.array([side, side, side + case.get("side_z", case["side"]) - case["side"]])
    grid = np.stack(np.meshgrid(*[np.arange(n) for n in edge], indexing="ij"), -1).reshape(-1, 1, 3)
    sites = (grid + _BASIS + 0.25).reshape(-1, 3)
    n = len(sites)
    if case["pot"] == "cu":
        types, a = np.zeros(n, np.uint32), 3.615
    elif case["pot"] == "nialco":
        types, a = rs.choice(3, size=n, p=rs.dirichlet([2.0, 2.0, 2.0])).astype(np.uint32), None
        a = sum(np.mean(types == k) * e[3] for k, e in enumerate(t.elements)) * 0.983
    else:
        if case.get("ordered"):  # one minority corner site and three majority face sites
            types = np.tile([1, 0, 0, 0], n // 4).astype(np.uint32)
        else:
            types = np.ones(n, np.uint32)
            types[rs.permutation(n)[: int(round(x * n))]] = 0
        a = 3.62 + 0.14 * np.mean(types == 0)
    keep = np.sort(rs.permutation(n)[case.get("vacancies", 0):])
    sites, types = sites[keep], types[keep]
    a *= (1.0 + 1.7e-5 * T) * U.angstrom
    L = edge * a
    pos = sites * a + rs.normal(size=sites.shape) * 0.08e-8 * math.sqrt(T / 300.0) - L / 2
    pos = (pos / L - np.floor(pos / L + 0.5)) * L
    mass = np.array(t.masses)[types]
    st = initial_state(mass, T, T, _TAU_T, _TAU_P, random_seed=int(rs.randint(1 << 31)))
    return Cell(positions=pos, velocities=st.velocities, types=types, box=L, T=T,
                ensemble=case["ensemble"], thermo_q=st.thermo_q, thermo_p_eta=st.thermo_p_eta,
                baro_q=st.baro_q, baro_p_eta=st.baro_p_eta, baro_w=st.baro_w,
                baro_p_eps=st.baro_p_eps, Nf=st.Nf)


def _cells(case, seed):
    rs = np.random.RandomState(seed % (1 << 32))
    cells = []
    # the sizes, compositions and temperatures of uneven replicas belong to the case
    own = np.random.RandomState(2026)
    for _ in range(case.get("replicas", 1)):
        side, x, T = case["side"], case.get("x", 0.0), case["T"]
        if "side_max" in case:
            side = int(own.randint(side, case["side_max"] + 1))
            x, T = float(own.uniform(0.0, x)), float(own.uniform(5.0, T))
        cells.append(_cell(case, rs, side, x, T))
    return cells


def _mlp_inputs(case, seed):
    """Standardised (composition, temperature) rows, their smooth targets with the noise of
    short runs, and starting weights."""
    rs = np.random.RandomState(seed % (1 << 32))
    widths = [case["inputs"], 64, 64, 64, 4]
    x = rs.uniform(-1.7, 1.7, (case["rows"], case["inputs"])).astype(np.float32)
    mix = rs.normal(size=(case["inputs"], 4))
    y = (np.tanh(x @ mix) + 0.2 * (x ** 2) @ mix + 0.05 * rs.normal(size=(case["rows"], 4))).astype(np.float32)
    params = np.concatenate([np.concatenate([rs.normal(size=a * b) * math.sqrt(2.0 / (a + b)), np.zeros(b)])
                             for a, b in zip(widths, widths[1:])]).astype(np.float32)
    return widths, x, y, params


def prepare(case, seed):
    if case["kind"] == "mlp":
        widths, x, y, params = _mlp_inputs(case, seed)
        return dict(case=case, net=MLP(widths), x=x, y=y, params=params)
    import md_driver_module as m
    t, cells = _tables(case["pot"]), _cells(case, seed)
    state = dict(case=case, m=m, t=t, cells=cells)
    dt = case.get("dt", 2.0) * U.fs
    if case["kind"] == "loop":
        state["driver"] = _one_driver(m, t, case, cells[0], dt)
    elif case["kind"] != "session":
        state["batch"] = _batch(m, t, case, cells, dt)
        state["batch"].set_sample_ring(0)  # long runs read the last step and the running sums
    return state


def _with_interpolation(m, t, case):
    _, pots, eams = make_objects(m, t, case["interpolation"])
    return m.PotentialVector(pots), m.EAMVector(eams)


def _thermostats(m, c):
    th = m.Thermostat(c.T, list(c.thermo_q), list(c.thermo_p_eta), c.Nf)
    return th, m.Barostat(c.pressure, c.baro_w, c.baro_p_eps,
                          m.Thermostat(c.T, list(c.baro_q), list(c.baro_p_eta), 1.0))


def _rg(cells):
    drg = 3.6345 * U.angstrom / 500.0
    return [(k + 0.5) * drg for k in range(int(min(min(c.box) for c in cells) / 2.0 / drg))]


def _one_driver(m, t, case, c, dt):
    if "interpolation" not in case:
        return make_driver(m, t, c, dt=dt, neighbors=case.get("neighbors", True), r_skin=_SKIN,
                           precision=case["precision"])
    pots, eams = _with_interpolation(m, t, case)
    th, baro = _thermostats(m, c)
    return m.MDDriver([m.Vector3d(*p) for p in c.positions], [m.Vector3d(*v) for v in c.velocities],
                      pots, eams, m.MDDriver.Ensamble(c.ensemble), m.MDDriver.ThermostatCoupling(0),
                      th, baro, m.Box(np.diag(c.box)), _rg([c]), c.Nf, list(t.masses),
                      [int(k) for k in c.types], dt, case.get("neighbors", True), _SKIN, 1e3,
                      precision=case["precision"])


def _batch(m, t, case, cells, dt):
    if "interpolation" not in case:
        return make_batch(m, t, cells, dt=dt, r_skin=_SKIN, precision=case["precision"])
    pots, eams = _with_interpolation(m, t, case)
    ths, baros = zip(*[_thermostats(m, c) for c in cells])
    return m.BatchedMDDriver([c.positions for c in cells], [c.velocities for c in cells],
                             [c.types for c in cells], pots, eams,
                             [m.MDDriver.Ensamble(c.ensemble) for c in cells], list(ths), list(baros),
                             [m.Box(np.diag(c.box)) for c in cells], [c.Nf for c in cells],
                             list(t.masses), dt, neighbors=True, r_skin=_SKIN,
                             fatal_conservation=1e3, precision=case["precision"], device=0,
                             rg=_rg(cells))


# -------------------------------------------------------------------------------- passes
def _kept(case, out):
    if case["precision"] != "mixed":
        return out
    return {k: np.asarray(v, dtype=np.float32) for k, v in out.items()}


def _frame(m, batch):
    """Every replica's positions and velocities, one array each."""
    n = range(batch.n_replicas)
    return {"positions": np.concatenate([batch.atoms(r, m.ATOM_POSITIONS) for r in n]),
            "velocities": np.concatenate([batch.atoms(r, m.ATOM_VELOCITIES) for r in n])}


def run(state):
    return {"loop": _run_loop, "run": _run_batch, "session": _run_session, "gr": _run_gr,
            "mlp": _run_mlp}[state["case"]["kind"]](state)


def _run_loop(state):
    """The reference's run loop: the list rebuild, one step, the reads of a sample."""
    case, d, m = state["case"], state["driver"], state["m"]
    series = {f: [] for f in _LOOP_FIELDS}
    volume = []
    for _ in range(case["steps"]):
        if case.get("neighbors", True) and d.cycle % _REBUILD == 0:
            d.calculate_neighbors()
        d.sample_observables = True
        d.integrate()
        for f in _LOOP_FIELDS:
            series[f].append(np.copy(getattr(d, f)))
        volume.append(d.box.volume())
    out = {f: np.array(v) for f, v in series.items()}
    out["volume"] = np.array(volume)
    out["positions"], out["velocities"] = d.atoms_array(m.ATOM_POSITIONS), d.atoms_array(m.ATOM_VELOCITIES)
    if case.get("gr"):
        d.calculate_pair_correlation()
        out["gr"] = np.array(d.gr)
    return _kept(case, out)


def _run_batch(state):
    """A stretch of a run on the device, then the observables and a frame."""
    case, b = state["case"], state["batch"]
    b.run(case["steps"], _REBUILD, case.get("stride", 1), False)
    o = b.observables_all()
    return _kept(case, {**{f: o[f] for f in _FIELDS}, **_frame(state["m"], b)})


def _run_session(state):
    """Batch from host arrays, every step's observables, the final frame."""
    case, m = state["case"], state["m"]
    b = _batch(m, state["t"], case, state["cells"], case.get("dt", 2.0) * U.fs)
    steps = []
    for _ in range(case["steps"]):
        b.run(1, _REBUILD, 1, False)
        steps.append(b.observables_all())
    return _kept(case, {**{f: np.array([o[f] for o in steps]) for f in _FIELDS}, **_frame(m, b)})


def _run_gr(state):
    g, partial = state["batch"].pair_correlation(0, 1)
    return {"gr": g, "gr_partial": partial}


def _run_mlp(state):
    net = state["net"]
    net.params = state["params"]  # starting weights: the optimiser starts anew
    loss = net.train(state["x"], state["y"], state["case"]["steps"], 1e-3)
    return {"params": net.params, "loss": loss, "proposed": net(state["x"])}


def work(case):
    """Bytes: per step each atom's coordinates, velocity, force and type read or written once.
    Operations: about 250 for each pair within the cutoff on a sampled step (three functions
    with two derivatives, forces, stress and elasticity terms) and 120 on the others; g(r) tests
    every pair; a network step takes 6 per weight and row."""
    if case["kind"] == "mlp":
        w = [case["inputs"], 64, 64, 64, 4]
        weights = sum(a * b for a, b in zip(w, w[1:]))
        return {"bytes": 4.0 * (case["rows"] * (w[0] + 4) * 2 + 2 * weights),
                "flops": 6.0 * weights * case["rows"] * case["steps"]}
    own = np.random.RandomState(2026)
    atoms = 0
    for _ in range(case.get("replicas", 1)):
        side = case["side"]
        if "side_max" in case:
            side = int(own.randint(side, case["side_max"] + 1))
            own.uniform(size=2)
        atoms += 4 * side * side * (side + case.get("side_z", case["side"]) - case["side"])
    if case["kind"] == "gr":
        return {"bytes": 32.0 * atoms, "flops": 10.0 * atoms * atoms}
    rc = _GRID[case["pot"]][2]
    pairs = atoms * 0.5 * 4.0 / 3.0 * math.pi * rc ** 3 * 4.0 / 3.65 ** 3
    sampled = case["steps"] / case.get("stride", 1)
    return {"bytes": case["steps"] * atoms * 128.0,
            "flops": pairs * (250.0 * sampled + 120.0 * (case["steps"] - sampled))}


# ----------------------------------------------------------------- the same in 64-bit torch
def exact(case, seed):
    if case["kind"] == "mlp":
        return _exact_mlp(case, seed)
    cells = _cells(case, seed)
    if case["kind"] == "gr":
        return _exact_gr(case, cells[0], cells[0].positions / cells[0].box, cells[0].box, partial=True)
    every = case["kind"] != "run"
    runs = [_exact_run(case, c, every) for c in cells]
    fields = _LOOP_FIELDS + ("volume",) if case["kind"] == "loop" else _FIELDS
    out = {f: np.array([r[0][f] for r in runs]) for f in fields}
    if case["kind"] == "loop":
        out = {f: v[0] for f, v in out.items()}
    elif case["kind"] == "session":
        out = {f: np.swapaxes(v, 0, 1) for f, v in out.items()}
    out["positions"] = np.concatenate([r[1] for r in runs])
    out["velocities"] = np.concatenate([r[2] for r in runs])
    if case.get("gr"):
        out["gr"] = _exact_gr(case, cells[0], runs[0][3], runs[0][4])["gr"]
    return out


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _spline(f, h):
    """Cubics in t (4 coefficients per interval) of the clamped cubic spline through the
    nodes, end slopes from the second-order one-sided differences."""
    m = len(f)
    d0 = (-3 * f[0] + 4 * f[1] - f[2]) / (2 * h)
    d1 = (3 * f[-1] - 4 * f[-2] + f[-3]) / (2 * h)
    i = torch.arange(m, device=f.device)
    A = torch.zeros(m, m, dtype=f.dtype, device=f.device)
    A[i, i] = 4.0
    A[i[1:], i[:-1]] = A[i[:-1], i[1:]] = 1.0
    A[0, 1] = A[-1, -2] = 2.0
    rhs = 6 * f
    rhs[0] += 2 * h * d0
    rhs[-1] -= 2 * h * d1
    b = torch.linalg.solve(A, rhs)
    b = torch.cat([(b[1] - 2 * h * d0)[None], b, (b[-2] + 2 * h * d1)[None]])
    p, q, r, s = b[:-3], b[1:-2], b[2:-1], b[3:]
    return torch.stack([(p + 4 * q + r) / 6, (r - p) / 2, (p - 2 * q + r) / 2, (s - 3 * r + 3 * q - p) / 6], -1)


class _Functions:
    """A set of tabulated functions on one grid: value and two derivatives at x of function k."""

    def __init__(self, f, f1, f2, h, spline):
        f, f1, f2 = (torch.tensor(v, dtype=torch.float64, device=_dev()) for v in (f, f1, f2))
        self.h, self.spline, self.n = h, spline, f.shape[1] - 1
        if spline:
            self.c = torch.stack([torch.cat([_spline(u, h) for u in v], -1) for v in zip(f, f1, f2)])
        else:  # the quintic Hermite polynomial of each interval
            y0, y1, d0, d1 = f[:, :-1], f[:, 1:], h * f1[:, :-1], h * f1[:, 1:]
            s0, s1, dy = h * h * f2[:, :-1], h * h * f2[:, 1:], y1 - y0
            self.c = torch.stack([y0, d0, s0 / 2, 10 * dy - 6 * d0 - 4 * d1 - 1.5 * s0 + 0.5 * s1,
                                  -15 * dy + 8 * d0 + 7 * d1 + 1.5 * s0 - s1,
                                  6 * dy - 3 * (d0 + d1) - 0.5 * (s0 - s1)], -1)

    def __call__(self, k, x):
        u = x / self.h
        i = u.long().clamp(0, self.n - 1)
        t = u - i
        c = self.c[k, i].unbind(-1)
        if self.spline:
            return tuple(c[q] + t * (c[q + 1] + t * (c[q + 2] + t * c[q + 3])) for q in (0, 4, 8))
        return (c[0] + t * (c[1] + t * (c[2] + t * (c[3] + t * (c[4] + t * c[5])))),
                (c[1] + t * (2 * c[2] + t * (3 * c[3] + t * (4 * c[4] + t * 5 * c[5])))) / self.h,
                (2 * c[2] + t * (6 * c[3] + t * (12 * c[4] + t * 20 * c[5]))) / self.h ** 2)


_FUNCTIONS = {}


def _functions(case):
    key = (case["pot"], case.get("interpolation"))
    if key not in _FUNCTIONS:
        t, sp = _tables(case["pot"]), case.get("interpolation") == "bspline"
        _FUNCTIONS[key] = (_Functions(t.phi, t.dphi, t.d2phi, t.dr, sp),
                           _Functions(t.rho, t.drho_dr, t.d2rho_dr2, t.dr, sp),
                           _Functions(t.F, t.dF, t.d2F, t.drho, sp))
    return _FUNCTIONS[key]


def _pairs(s, L, radius):
    """Index pairs (each once) within the radius, minimum image; s scaled coordinates."""
    n = len(s)
    cells = [int(v // radius) for v in L.tolist()]
    if n <= 3000 or min(cells) < 3:
        out = []
        for b in range(0, n, 1024):
            d = s[b:b + 1024, None] - s[None]
            r2 = (((d - torch.round(d)) * L) ** 2).sum(-1)
            i, j = torch.nonzero(r2 <= radius ** 2, as_tuple=True)
            k = i + b < j
            out.append(torch.stack([i[k] + b, j[k]]))
        return torch.cat(out, 1)
    nc = torch.tensor(cells, device=s.device)
    at = ((s - torch.floor(s)) * nc).long().minimum(nc - 1)
    cid = (at[:, 0] * nc[1] + at[:, 1]) * nc[2] + at[:, 2]
    order = torch.argsort(cid)
    count = torch.bincount(cid, minlength=int(nc.prod()))
    start = torch.cumsum(count, 0) - count
    slot = torch.arange(n, device=s.device) - start[cid[order]]
    table = torch.full((len(count), int(count.max())), -1, device=s.device)
    table[cid[order], slot] = order
    grid = torch.stack(torch.meshgrid(*[torch.arange(v, device=s.device) for v in cells], indexing="ij"), -1).reshape(-1, 3)
    out = []
    for off in [(x, y, z) for x in (-1, 0, 1) for y in (-1, 0, 1) for z in (-1, 0, 1)]:
        if off < (0, 0, 0):
            continue
        nb = (grid + torch.tensor(off, device=s.device)) % nc
        other = table[(nb[:, 0] * nc[1] + nb[:, 1]) * nc[2] + nb[:, 2]]
        i, j = torch.broadcast_tensors(table[:, :, None], other[:, None, :])
        k = (i >= 0) & (j >= 0) & ((i < j) if off == (0, 0, 0) else True)
        i, j = i[k], j[k]
        d = s[i] - s[j]
        k = (((d - torch.round(d)) * L) ** 2).sum(-1) <= radius ** 2
        out.append(torch.stack([i[k], j[k]]))
    return torch.cat(out, 1)


_VOIGT = ((0, 0), (1, 1), (2, 2), (1, 2), (0, 2), (0, 1))


def _forces(case, s, L, types, pairs):
    """Forces and the sums of one configuration, cgs."""
    phi, den, emb = _functions(case)
    i, j = pairs
    d = s[i] - s[j]
    p = (d - torch.round(d)) * L
    r = p.square().sum(-1).sqrt()
    k = r <= _tables(case["pot"]).rcut
    i, j, p, r = i[k], j[k], p[k], r[k]
    ti, tj = types[i], types[j]
    hi, lo = torch.maximum(ti, tj), torch.minimum(ti, tj)
    V, V1, V2 = phi(hi * (hi + 1) // 2 + lo, r)
    ri, ri1, ri2 = den(ti, r)
    rj, rj1, rj2 = den(tj, r)
    n = len(s)

    def gather(at_i, at_j):
        z = torch.zeros((n,) + at_i.shape[1:], dtype=s.dtype, device=s.device)
        return z.index_add(0, i, at_i).index_add(0, j, at_j)

    F, F1, F2 = emb(types, gather(rj, ri))
    pp = torch.stack([p[:, a] * p[:, b] for a, b in _VOIGT], -1)
    g = gather((rj1 / r)[:, None] * pp, (ri1 / r)[:, None] * pp)
    hv = gather((rj1 / r)[:, None] * p, -(ri1 / r)[:, None] * p)
    de = V1 + F1[i] * rj1 + F1[j] * ri1
    f = gather(-(de / r)[:, None] * p, (de / r)[:, None] * p)
    X = (V2 - V1 / r + F1[i] * (rj2 - rj1 / r) + F1[j] * (ri2 - ri1 / r)) / (r * r)
    lap = (2 * (V2 + 2 * V1 / r) + 2 * (F1[j] * (ri2 + 2 * ri1 / r) + F1[i] * (rj2 + 2 * rj1 / r)) +
           F2[i] * rj1 ** 2 + F2[j] * ri1 ** 2)
    born = (X[:, None] * pp).T @ pp + (F2[:, None] * g).T @ g
    return dict(f=f, epot=float(V.sum() + F.sum()), emb=float(F.sum()), virial=float((r * de).sum()) / -3.0,
                sigma=((de / r)[:, None] * pp).sum(0).cpu().numpy(), born=torch.triu(born).cpu().numpy(),
                lap=float(lap.sum() + (F2 * hv.square().sum(-1)).sum()), f2=float(f.square().sum()))


_W7 = [0.784513610477560, 0.235573213359357, -1.17767998417887]
_W7 = _W7 + [1.0 - 2.0 * sum(_W7)] + _W7[::-1]


def _phi1(x):
    """(1 - exp(-x)) / x"""
    return -math.expm1(-x) / x if x else 1.0


class _Chain:
    """A Nose-Hoover chain and its half step (seven Suzuki-Yoshida weights)."""

    def __init__(self, T, q, p, nf):
        self.kT, self.q, self.p, self.nf = U.k_boltz * T, list(map(float, q)), list(map(float, p)), nf
        self.eta = [0.0] * len(self.q)

    def _link(self, k, dt, ec):
        G = self.p[k - 1] ** 2 / self.q[k - 1] - self.kT if k else 2.0 * ec - self.nf * self.kT
        if k == len(self.q) - 1:
            self.p[k] += dt * G
        else:
            x = dt * self.p[k + 1] / self.q[k + 1]
            self.p[k] = self.p[k] * math.exp(-x) + dt * G * _phi1(x)

    def half(self, dt, energy):
        """energy(scale) of the coupled momenta scaled by `scale`; returns the scale."""
        S, m = 1.0, len(self.q)
        for w in _W7:
            for k in reversed(range(m)):
                self._link(k, 0.5 * w * dt, energy(S))
            S *= math.exp(-w * dt * self.p[0] / self.q[0])
            self.eta = [e + w * dt * p / q for e, p, q in zip(self.eta, self.p, self.q)]
            for k in range(m):
                self._link(k, 0.5 * w * dt, energy(S))
        return S

    def energy(self):
        return self.kT * (self.nf * self.eta[0] + sum(self.eta[1:])) + sum(0.5 * p * p / q for p, q in zip(self.p, self.q))


def _exact_run(case, c, every):
    """The run's observables (of every step, or of the last), final positions, velocities,
    scaled coordinates and box."""
    t, dev = _tables(case["pot"]), _dev()
    dt, N = case.get("dt", 2.0) * U.fs, c.n_atoms
    npt, nvt = c.ensemble == 2, c.ensemble >= 1
    h0 = torch.tensor(c.box, dtype=torch.float64, device=dev)
    s = torch.tensor(c.positions, dtype=torch.float64, device=dev) / h0
    v = torch.tensor(c.velocities, dtype=torch.float64, device=dev)
    types = torch.tensor(c.types.astype(np.int64), device=dev)
    m = torch.tensor(np.array(t.masses), device=dev)[types][:, None]
    h, h_pos, eps, p_eps, w = h0, h0, 0.0, c.baro_p_eps, c.baro_w
    th = _Chain(c.T, c.thermo_q, c.thermo_p_eta, c.Nf)
    bth = _Chain(c.T, c.baro_q, c.baro_p_eta, 1.0)
    alpha = 1.0 + 3.0 / c.Nf

    def chains(ekin):
        nonlocal p_eps
        S = th.half(0.5 * dt, lambda z: ekin * z * z) if nvt else 1.0
        if npt:
            p_eps *= bth.half(0.5 * dt, lambda z: 0.5 * (p_eps * z) ** 2 / w)
        return S

    def push(ekin, virial):
        nonlocal p_eps
        p_eps += (2.0 * alpha * ekin + 3.0 * virial - 3.0 * c.pressure * float(h.prod())) * 0.5 * dt

    margin = 0.6 * U.angstrom
    pairs, s_ref = _pairs(s, h, t.rcut + margin), s
    q = _forces(case, s, h, types, pairs)
    ekin = float((0.5 * m * v * v).sum())
    out = {f: [] for f in _FIELDS}
    lap = q["lap"]
    born, tci = None, None
    for k in range(case["steps"]):
        S = chains(ekin)
        ekin *= S * S
        v = v * S
        e, cc = 1.0, 1.0
        if npt:
            push(ekin, q["virial"])
            x = alpha * 0.5 * dt * p_eps / w
            e, cc = math.exp(-x), _phi1(x)
        v = v * e + cc * 0.5 * dt * q["f"] / m
        x = dt * p_eps / w if npt else 0.0
        eps += x
        s = s + _phi1(x) * dt * v / h
        h_pos, h = h, h0 * math.exp(eps) if npt else h
        if float(((s - s_ref) * h).square().sum(-1).max()) > (0.48 * margin) ** 2:
            pairs, s_ref = _pairs(s, h, t.rcut + margin), s
        q = _forces(case, s, h, types, pairs)
        v = v * e + cc * 0.5 * dt * q["f"] / m
        ekin = float((0.5 * m * v * v).sum())
        mvv = np.array([float((m[:, 0] * v[:, a] * v[:, b]).sum()) for a, b in _VOIGT])
        if npt:
            push(ekin, q["virial"])
        S = chains(ekin)
        ekin *= S * S
        v = v * S
        V = float(h.prod())
        if (k + 1) % case.get("stride", 1) == 0:  # a sampled step
            lap, f2 = q["lap"], q["f2"]
            born, tci = q["born"] / V, U.k_boltz * lap / f2
        if every or k == case["steps"] - 1:
            cons = ekin + q["epot"] + (th.energy() if nvt else 0.0)
            if npt:
                cons += V * c.pressure + 0.5 * p_eps ** 2 / w + bth.energy()
            now = dict(epot_atom=q["epot"] / N, epot_eam_atom=q["emb"] / N, ekin_atom=ekin / N,
                       etot_cons=cons, virial=q["virial"], total_laplacian=lap,
                       total_force2=f2, temperature_kin=2.0 * ekin / (U.k_boltz * c.Nf),
                       temperature_conf_inverse=tci, pressure=(2.0 * ekin / 3.0 + q["virial"]) / V,
                       volume=V, born_stress_tensor=q["sigma"] / V,
                       stress_tensor=(-q["sigma"] + S * S * mvv) / V, born_elasticity_tensor=born)
            for f in _FIELDS:
                out[f].append(now[f])
    if not every:
        out = {f: x[-1] for f, x in out.items()}
    pos = (s - torch.round(s)) * h_pos
    return out, pos.cpu().numpy(), v.cpu().numpy(), s.cpu().numpy(), h.cpu().numpy()


def _exact_gr(case, c, scaled, box, partial=False):
    drg = 3.6345 * U.angstrom / 500.0
    n_rg = int(min(c.box) / 2.0 / drg)
    rmax = (n_rg - 0.5) * drg + 0.5 * drg
    dev = _dev()
    L = torch.tensor(box, dtype=torch.float64, device=dev)
    s = torch.tensor(scaled, dtype=torch.float64, device=dev)
    types = torch.tensor(c.types.astype(np.int64), device=dev)
    nt, N = len(_ELEMENTS[case["pot"]]), len(s)
    total = torch.zeros(n_rg, dtype=torch.int64, device=dev)
    parts = torch.zeros(nt * (nt + 1) // 2, n_rg, dtype=torch.int64, device=dev)
    for b in range(0, N, 512):
        d = s[b:b + 512, None] - s[None]
        r = ((d - torch.round(d)) * L).square().sum(-1).sqrt()
        i, j = torch.nonzero(r < rmax, as_tuple=True)
        k = i + b < j
        i, j = i[k], j[k]
        at = torch.floor(r[i, j] / drg).long().clamp(max=n_rg - 1)
        total += torch.bincount(at, minlength=n_rg)
        ta, tb = types[i + b], types[j]
        slot = torch.maximum(ta, tb) * (torch.maximum(ta, tb) + 1) // 2 + torch.minimum(ta, tb)
        parts += torch.bincount(slot * n_rg + at, minlength=parts.numel()).reshape(parts.shape)
    rg, V = (np.arange(n_rg) + 0.5) * drg, float(np.prod(box))
    out = {"gr": total.cpu().numpy() * V / (2.0 * math.pi * N * N * rg * rg * drg)}
    if partial:
        counts = np.bincount(c.types, minlength=nt)
        rows = []
        for b in range(nt):
            for a in range(b + 1):
                n = counts[a] * (counts[a] - 1) / 2 if a == b else counts[a] * counts[b]
                row = parts[len(rows)].cpu().numpy() * V / (4.0 * math.pi * max(n, 1) * drg * rg * rg)
                rows.append(row if n > 0 else row * 0.0)
        out["gr_partial"] = np.array(rows)
    return out


def _exact_mlp(case, seed):
    widths, x, y, params = _mlp_inputs(case, seed)
    dev = _dev()
    x, y = (torch.tensor(v, dtype=torch.float64, device=dev) for v in (x, y))
    p = torch.tensor(params, dtype=torch.float64, device=dev, requires_grad=True)

    def net():
        a, at = x, 0
        for k, (i, o) in enumerate(zip(widths, widths[1:])):
            a = a @ p[at:at + i * o].reshape(i, o) + p[at + i * o:at + i * o + o]
            at += i * o + o
            if k < len(widths) - 2:
                a = torch.nn.functional.gelu(a)
        return a

    m1, m2 = torch.zeros_like(p), torch.zeros_like(p)
    for step in range(1, case["steps"] + 1):
        loss = (net() - y).square().mean()
        g, = torch.autograd.grad(loss, p)
        with torch.no_grad():
            m1 = 0.9 * m1 + 0.1 * g
            m2 = 0.999 * m2 + 0.001 * g * g
            p -= 1e-3 * (m1 / (1 - 0.9 ** step)) / ((m2 / (1 - 0.999 ** step)).sqrt() + 1e-8)
    with torch.no_grad():
        proposed = net()
        return {"params": p.detach(), "loss": float((proposed - y).square().mean()), "proposed": proposed}
