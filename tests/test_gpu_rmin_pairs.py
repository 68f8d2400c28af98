"""r_min of its own for every pair type (potential.hpp:92-104 warns of a pair below its potential's
r_min): the warning goes by each pair's own value, for values just off the smallest distance of each
pair type, shared ones, negative ones and ones beyond the cutoff, and costs the mixed pass no second
look at the rows whose distances lie between one type's r_min and another's."""

import itertools

import numpy as np
import pytest

from generic import generic_case, generic_tables
from mdelast_b200.potentials import make_objects

pytestmark = pytest.mark.gpu

WARN_RMIN = 0x200
A = 1e-8


def _driver(c, rmins, precision, copies=1):
    """A batch of `copies` of case c with the given r_min [A] of the pair types aa, ab, bb, ..."""
    import md_driver_module as m
    t = c.tables
    _, _, eams = make_objects(m, t)
    pots = [m.TablePotential(t.rcut, r * A, t.dr, t.phi[k], t.dphi[k], t.d2phi[k], "quintic")
            for k, r in enumerate(rmins)]
    th = m.Thermostat(c.thermo[0], list(c.thermo[1]), list(c.thermo[2]), c.Nf)
    ba = m.Barostat(c.baro[0], c.baro[1], c.baro[2],
                    m.Thermostat(c.baro_thermo[0], list(c.baro_thermo[1]), list(c.baro_thermo[2]), 1.0))
    n = copies
    return m.BatchedMDDriver([c.positions] * n, [c.velocities] * n, [np.asarray(c.types, np.uint32)] * n,
                             m.PotentialVector(pots), m.EAMVector(eams),
                             [m.MDDriver.Ensamble(c.ensemble)] * n, [th] * n, [ba] * n, [m.Box(c.box)] * n,
                             [c.Nf] * n, list(t.masses), c.dt, neighbors=c.neighbors, r_skin=c.r_skin,
                             fatal_conservation=1e3, precision=precision, device=0, rg=list(c.rg))


def _smallest(c):
    """Smallest distance [A] of each pair type."""
    d = c.positions[:, None] - c.positions[None]
    L = c.box.diagonal()
    d -= np.rint(d / L) * L
    r = np.sqrt((d * d).sum(-1)) / A
    np.fill_diagonal(r, np.inf)
    ty = np.asarray(c.types)
    return [r[np.ix_(ty == a, ty == b)].min() for b in range(c.tables.n_types) for a in range(b + 1)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("types", [1, 2, 3])
def test_each_pair_types_own_value(types, precision):
    c = generic_case(generic_tables(types), (5, 4, 6), 3)
    low = _smallest(c)
    for off in itertools.product((-0.002, 0.002), repeat=len(low)) if types < 3 else \
            [tuple(0.002 if k == q else -0.002 for k in range(6)) for q in range(-1, 6)]:
        want = any(o > 0 for o in off)
        b = _driver(c, [d + o for d, o in zip(low, off)], precision)
        assert bool(int(b.status()[0]) & WARN_RMIN) == want, off
    for shared, want in ((min(low) - 0.002, False), (min(low) + 0.002, True), (-1.0, False),
                         (0.0, False), (c.tables.rcut / A + 1.0, True)):
        b = _driver(c, [shared] * len(low), precision)
        assert bool(int(b.status()[0]) & WARN_RMIN) == want, shared


def test_no_second_look():
    """Force pass of 30,784 atoms with every nearest neighbour but the bb ones below bb's r_min,
    against one shared r_min: a look at the rows again took 1.45 times as long; a test per pair is
    two instructions of some 150."""
    c = generic_case(generic_tables(2), (13, 16, 37), 0, T=300.0)
    types = np.zeros(len(c.types), int)  # b atoms no nearest neighbours of each other: one in each cube
    types[::4] = 1
    c.types = types
    mass = np.array(c.tables.masses)[types][:, None]
    c.velocities = np.asarray(c.velocities) - (mass * c.velocities).sum(0) / mass.sum()
    low = 1.9
    best = {}
    for name, rmins in (("shared", [low] * 3), ("own", [low, low, 2.9])):
        b = _driver(c, rmins, "mixed")
        assert not int(b.status()[0]) & WARN_RMIN
        b.kernel_times(5)
        best[name] = min(b.kernel_times(10)[3] for _ in range(5))
    assert best["own"] <= 1.25 * best["shared"], best
