"""A launch shape that a caller names is the one that runs: 16 lanes per atom, set by set_launch or
MDELAST_TPA, sum an atom's row in the same order on a small driver (whose default is a warp per atom)
as on a large one, so every atom's density, energy and force has the same bits on both. The tuners
report shapes that set_launch takes, and 32 is not among them."""

import os

import numpy as np
import pytest

from generic import generic_case, generic_tables

pytestmark = pytest.mark.gpu


def _batch(c, copies, precision):
    import md_driver_module as m
    from mdelast_b200.potentials import make_objects
    _, pots, eams = make_objects(m, c.tables)
    th = m.Thermostat(c.thermo[0], list(c.thermo[1]), list(c.thermo[2]), c.Nf)
    ba = m.Barostat(c.baro[0], c.baro[1], c.baro[2],
                    m.Thermostat(c.baro_thermo[0], list(c.baro_thermo[1]), list(c.baro_thermo[2]), 1.0))
    n = copies
    return m.BatchedMDDriver([c.positions] * n, [c.velocities] * n, [np.asarray(c.types, np.uint32)] * n,
                             m.PotentialVector(pots), m.EAMVector(eams),
                             [m.MDDriver.Ensamble(c.ensemble)] * n, [th] * n, [ba] * n, [m.Box(c.box)] * n,
                             [c.Nf] * n, list(c.tables.masses), c.dt, neighbors=c.neighbors,
                             r_skin=c.r_skin, fatal_conservation=1e3, precision=precision, device=0,
                             rg=list(c.rg))


def _fields(b):
    import md_driver_module as m
    return [np.array(b.atoms(0, f)) for f in (m.ATOM_RHO, m.ATOM_EPOT, m.ATOM_FORCES)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("how", ["set_launch", "environment"])
def test_named_lanes_run(precision, how):
    c = generic_case(generic_tables(2), (5, 5, 5), 0)
    old = os.environ.get("MDELAST_TPA")
    try:
        if how == "environment":
            os.environ["MDELAST_TPA"] = "16"
        small, large = _batch(c, 1, precision), _batch(c, 8, precision)
    finally:
        os.environ.pop("MDELAST_TPA", None) if old is None else os.environ.update(MDELAST_TPA=old)
    if how == "set_launch":
        small.set_launch(16, 16, 148 * 32, 148 * 32)
        large.set_launch(16, 16, 148 * 32, 148 * 32)
    for steps in (0, 3):
        if steps:
            small.run(steps, 20, 1, False)
            large.run(steps, 20, 1, False)
        for a, b in zip(_fields(small), _fields(large)):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_tuners_report_what_set_launch_takes(precision):
    c = generic_case(generic_tables(2), (5, 5, 5), 0)
    b = _batch(c, 1, precision)
    with pytest.raises(RuntimeError):
        b.set_launch(32, 32, 148 * 32, 148 * 32)
    for choice in (b.autotune(2), b.autotune_steps(2, 20)):
        assert choice["tpa_density"] in (1, 4, 8, 16) and choice["tpa_force"] in (1, 4, 8, 16)
    b.set_launch(choice["tpa_density"], choice["tpa_force"], 148 * 32, 148 * 32)
    b.run(2, 20, 1, False)
