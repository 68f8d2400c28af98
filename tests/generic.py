"""Generic many-body tables (no potential file needed) and cells of odd sizes, for tests of
kernel variants against the oracle: inverse-power pair terms and densities with a smooth
cutoff, a square-root embedding, node derivatives from the readers' quintic spline."""

import numpy as np

from helpers import Case
from mdelast_b200.lattice import initial_state
from mdelast_b200.potentials import SetflTables, get_derivatives
from mdelast_b200.units import Units as U

_SIZES = (3.85, 3.70, 3.60)  # length scale of each type [A]
_MASS = (65.38, 63.546, 58.693)


def generic_tables(n_types=2, n_r=800, rcut=6.0, n_rho=800):
    A, A3 = U.angstrom, U.angstrom ** 3
    r, rho = np.linspace(0.0, rcut, n_r) * A, np.linspace(0.0, 8.0, n_rho) / A3

    def radial(a, n):
        x = r / A
        u = np.clip((x - (rcut - 1.5)) / 1.5, 0.0, 1.0)
        return (a * a / (x * x + 0.36)) ** (0.5 * n) * (1.0 - u ** 3 * (10.0 - 15.0 * u + 6.0 * u * u))

    phi = [0.0124 * U.ev * radial(0.5 * (_SIZES[i] + _SIZES[j]), 9)
           for j in range(n_types) for i in range(j + 1)]
    den = [radial(_SIZES[t], 6) / 120.0 / A3 for t in range(n_types)]
    emb = [-0.488 * U.ev * (np.sqrt(120.0 * rho * A3 + 0.01) - 0.1) for _ in range(n_types)]
    d = {k: [get_derivatives(x, y) for y in v] for k, x, v in (("phi", r, phi), ("rho", r, den), ("F", rho, emb))}
    return SetflTables(elements=[["X", 1, _MASS[t], 0.0] for t in range(n_types)], n_r=n_r,
                       dr=r[1], n_rho=n_rho, drho=rho[1], rcut=float(r[-1]), rhomax=float(rho[-1]),
                       rmin_fatal=1e-2 * A, phi=np.array(phi), dphi=np.array([x[0] for x in d["phi"]]),
                       d2phi=np.array([x[1] for x in d["phi"]]), rho=np.array(den),
                       drho_dr=np.array([x[0] for x in d["rho"]]),
                       d2rho_dr2=np.array([x[1] for x in d["rho"]]), F=np.array(emb),
                       dF=np.array([x[0] for x in d["F"]]), d2F=np.array([x[1] for x in d["F"]]))


def generic_case(tables, edges=(5, 5, 5), vacancies=0, ensemble=1, T=300.0, seed=1, dt=2e-15,
                 a_ang=3.64, neighbors=True, sigma_ang=0.08, coupling=0):
    """An FCC cell of edges[0] x edges[1] x edges[2] unit cells with random types, `vacancies`
    atoms missing, every atom displaced."""
    rs = np.random.RandomState(seed)
    basis = np.array([[0, 0, 0], [0.5, 0.5, 0], [0.5, 0, 0.5], [0, 0.5, 0.5]])
    grid = np.stack(np.meshgrid(*[np.arange(n) for n in edges], indexing="ij"), -1).reshape(-1, 1, 3)
    sites = (grid + basis + 0.25).reshape(-1, 3)
    sites = sites[np.sort(rs.permutation(len(sites))[vacancies:])]
    a = a_ang * U.angstrom
    L = np.array(edges) * a
    pos = sites * a + rs.normal(size=sites.shape) * sigma_ang * U.angstrom - L / 2
    pos = (pos / L - np.floor(pos / L + 0.5)) * L
    types = rs.randint(0, tables.n_types, len(sites))
    st = initial_state(np.array(tables.masses)[types], T, T, 5e-14, 5e-13, random_seed=seed)
    return Case(tables, pos, st.velocities, types, np.diag(L), ensemble=ensemble, coupling=coupling,
                thermo=(T, st.thermo_q, st.thermo_p_eta, st.Nf),
                baro=(1e-10 * U.GPa, st.baro_w, st.baro_p_eps),
                baro_thermo=(T, st.baro_q, st.baro_p_eta, 1.0), Nf=st.Nf, dt=dt,
                neighbors=neighbors, r_skin=1.2 if neighbors else 1.0)
