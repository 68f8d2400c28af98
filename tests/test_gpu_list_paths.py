"""Which search builds a replica's list (all pairs for small replicas and for idle SMs, cells else)
and which replicas' pair lists a step refreshes leave the results unchanged: the same list as the
oracle's entry for entry by either search, trajectories at 1e-9, and batches of more replicas
than a block has threads, due at different steps."""

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, gpu_atoms, oracle, rel_err

pytestmark = pytest.mark.gpu


def _batch(cases, precision="fp64"):
    import md_driver_module as m
    from mdelast_b200.potentials import make_objects
    c = cases[0]
    _, pots, eams = make_objects(m, c.tables)
    th = [m.Thermostat(x.thermo[0], list(x.thermo[1]), list(x.thermo[2]), x.Nf) for x in cases]
    ba = [m.Barostat(x.baro[0], x.baro[1], x.baro[2],
                     m.Thermostat(x.baro_thermo[0], list(x.baro_thermo[1]), list(x.baro_thermo[2]), 1.0))
          for x in cases]
    return m.BatchedMDDriver([x.positions for x in cases], [x.velocities for x in cases],
                             [np.asarray(x.types, np.uint32) for x in cases], m.PotentialVector(pots),
                             m.EAMVector(eams), [m.MDDriver.Ensamble(x.ensemble) for x in cases], th, ba,
                             [m.Box(x.box) for x in cases], [x.Nf for x in cases],
                             list(c.tables.masses), c.dt, neighbors=c.neighbors, r_skin=c.r_skin,
                             fatal_conservation=1e3, precision=precision, device=0, rg=list(c.rg))


def _run(o, steps):
    for s in range(steps):
        if s % 20 == 0:
            o.calculate_neighbors()
        o.integrate()


# rcut, edges, copies: all pairs by size (500 atoms), all pairs on idle SMs, cells (enough
# copies), each with atom counts off the warp and block sizes
@pytest.mark.parametrize("rcut,edges,vacancies,copies", [
    (4.5, (5, 5, 5), 3, 1), (4.5, (5, 5, 5), 0, 8), (6.0, (8, 8, 8), 1, 1), (6.0, (8, 7, 9), 5, 6),
    (4.5, (8, 8, 8), 2, 3), (6.0, (10, 9, 9), 7, 1), (4.5, (11, 10, 10), 1, 1)])
def test_lists_and_trajectories(rcut, edges, vacancies, copies):
    t = generic_tables(2, rcut=rcut)
    cases = [generic_case(t, edges, vacancies, ensemble=2, T=600.0, seed=10 + k) for k in range(copies)]
    b = _batch(cases)
    last = copies - 1
    o = oracle(cases[last])
    po, no = o.neighbors()
    pg, ng = b.neighbor_list(last)
    assert np.array_equal(np.asarray(pg), po) and np.array_equal(np.asarray(ng), no)
    b.run(45, 20, 1, False)
    _run(o, 45)
    import md_driver_module as m
    for code, name in ((m.ATOM_POSITIONS, "positions"), (m.ATOM_FORCES, "forces")):
        assert rel_err(b.atoms(last, code), o.atoms(name)) <= 1e-9, name
    pg, ng = b.neighbor_list(last)
    po, no = o.neighbors()
    assert np.array_equal(np.asarray(pg), po) and np.array_equal(np.asarray(ng), no)


def test_shrinking_box_on_cells():
    """A batch large enough for cells whose boxes shrink below the grid of their run's start: the
    widened search of k_nbr_build, for every replica."""
    t = generic_tables(1, rcut=6.0)
    cases = [generic_case(t, (8, 8, 8), 0, ensemble=2, a_ang=3.64 * 1.08, seed=3 + k) for k in range(3)]
    for c in cases:
        c.r_skin = 1.1
    r_list = 6.0e-8 * 1.1
    nc = int(cases[0].box[0, 0] // (r_list * 1.05))
    assert 3 * nc ** 3 >= 148
    b = _batch(cases)
    b.run(60, 20, 1, False)
    for k in (0, 2):
        o = oracle(cases[k])
        _run(o, 60)
        import md_driver_module as m
        assert rel_err(b.atoms(k, m.ATOM_FORCES), o.atoms("forces")) <= 1e-9
        pg, ng = b.neighbor_list(k)
        po, no = o.neighbors()
        assert np.array_equal(np.asarray(pg), po) and np.array_equal(np.asarray(ng), no)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_many_replicas_due_at_different_steps(precision):
    t = generic_tables(1, rcut=4.5)
    Ts = [5.0, 300.0, 900.0]
    cases = [generic_case(t, (3, 3, 3 + k % 2), k % 3, T=Ts[k % 3], seed=100 + k,
                          sigma_ang=0.08 * (Ts[k % 3] / 300.0) ** 0.5) for k in range(300)]
    b = _batch(cases, precision)
    b.run(33, 20, 1, False)
    import md_driver_module as m
    for k in (0, 1, 2, 128, 255, 256, 299):
        o = oracle(cases[k])
        _run(o, 33)
        tol = 1e-9 if precision == "fp64" else 2e-5
        assert rel_err(b.atoms(k, m.ATOM_POSITIONS), o.atoms("positions")) <= tol
        assert rel_err(b.observables(k)["epot_atom"], o.scalar_dict()["epot_atom"]) <= tol
