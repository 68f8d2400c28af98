"""The table forms that no setfl file gives and every pair pass has its own code for: "bspline" tables,
density functions cut below the pair cutoff, and pair potentials without EAM, in FP64 and mixed
precision, for every lanes-per-atom variant and with the force tables staged, against the oracle.
Tolerances are those of test_gpu_pair_sums.py on the same cells: FP64 1e-10 static and 1e-9 after
steps, mixed forces 2e-5, energies 1e-6, tensors 1e-4."""

import copy

import pytest

from generic import generic_case, generic_tables
from oracle.ref import OracleDriver
from test_gpu_pair_sums import _check as check_sums

pytestmark = pytest.mark.gpu


def _pair(c, precision, eam):
    """The driver and the oracle of case c; eam: "same", "cut" (at 0.75 of the pair cutoff), "none"."""
    import md_driver_module as m
    t = copy.copy(c.tables)
    cut = 0.75 * t.rcut if eam == "cut" else t.rcut
    t.eam_rcut = cut
    kw = c.kw()
    o = OracleDriver(t, c.positions, c.velocities, c.types, interpolation=c.interpolation,
                     has_eam=eam != "none", **kw)
    eams = [m.EAM(cut, t.rhomax, t.dr, t.drho, t.rho[k], t.drho_dr[k], t.d2rho_dr2[k], t.F[k], t.dF[k],
                  t.d2F[k], c.interpolation) for k in range(t.n_types)] if eam != "none" else []
    pots = [m.TablePotential(t.rcut, t.rmin_fatal, t.dr, t.phi[k], t.dphi[k], t.d2phi[k], c.interpolation)
            for k in range(t.phi.shape[0])]
    th = m.Thermostat(c.thermo[0], list(c.thermo[1]), list(c.thermo[2]), c.Nf)
    ba = m.Barostat(c.baro[0], c.baro[1], c.baro[2],
                    m.Thermostat(c.baro_thermo[0], list(c.baro_thermo[1]), list(c.baro_thermo[2]), 1.0))
    g = m.MDDriver([m.Vector3d(*p) for p in c.positions], [m.Vector3d(*v) for v in c.velocities],
                   m.PotentialVector(pots), m.EAMVector(eams), m.MDDriver.Ensamble(c.ensemble),
                   m.MDDriver.ThermostatCoupling(c.coupling), th, ba, m.Box(c.box), list(c.rg), c.Nf,
                   list(t.masses), [int(x) for x in c.types], c.dt, c.neighbors, c.r_skin,
                   c.fatal_conservation, precision=precision)
    return g, o


def _check(g, o, precision, tol):
    check_sums(g, o, *((tol,) * 3 if precision == "fp64" else (2e-5, 1e-6, 1e-4)))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("interpolation,eam", [("bspline", "same"), ("bspline", "cut"), ("quintic", "cut"),
                                               ("quintic", "none"), ("bspline", "none")])
@pytest.mark.parametrize("types,edges,vacancies", [(1, (5, 4, 6), 3), (3, (7, 7, 8), 1)])
def test_table_forms(types, edges, vacancies, interpolation, eam, precision):
    c = generic_case(generic_tables(types), edges, vacancies)
    c.interpolation = interpolation
    g, o = _pair(c, precision, eam)
    _check(g, o, precision, 1e-10)
    for tpa in (1, 4, 8, 16):
        g.set_launch(tpa, tpa, 148 * 8, 148 * 8)
        _check(g, o, precision, 1e-10)
    if precision == "mixed" and interpolation == "quintic" and eam != "none":
        g.force_staging = True
        _check(g, o, precision, 1e-10)
    for k in range(4):
        if k == 2:
            g.calculate_neighbors()
            o.calculate_neighbors()
        g.integrate()
        o.integrate()
    _check(g, o, precision, 1e-9)
