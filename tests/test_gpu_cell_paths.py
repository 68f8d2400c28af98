"""The cell search where only it can serve, on cells above every limit of the all-pairs rule: a run whose
boxes shrink below the grid it started with (the widened reach, for some replicas of a batch and
not for others), and a run that outgrows its list capacity at an in-step rebuild."""

import os
import re

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, oracle, rel_err
from test_gpu_list_paths import _batch, _run
from test_gpu_parity import compare_state

pytestmark = pytest.mark.gpu

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mdelast_b200", "csrc", "driver.cu")


def _on_cells(n_atoms, box, r_list):
    """Whether a replica is searched by cells whatever its batch: more atoms than any limit of the rule
    beside configure_cells, and three cells per edge; the cells per edge."""
    limits = [int(x) for x in re.findall(r"kBrute(?:Atoms|Few|Idle) = (\d+)", open(SRC).read())]
    assert len(limits) == 3
    nc = np.floor(box / (r_list * 1.05)).astype(int)
    assert n_atoms > max(limits) and nc.min() >= 3
    return nc


def test_some_boxes_shrink_below_their_grid():
    t = generic_tables(1, rcut=6.0)
    wide = [generic_case(t, (8, 10, 10), k, ensemble=2, a_ang=3.64 * 1.12, seed=3 + k) for k in range(3)]
    near = [generic_case(t, (9, 9, 10), k, ensemble=2, a_ang=3.64, seed=13 + k) for k in range(2)]
    cases = [wide[0], near[0], wide[1], near[1], wide[2]]
    r_list = wide[0].box[0, 0] / (4 * 1.05 * 1.003)
    for c in cases:
        c.r_skin = r_list / t.rcut
    nc = [_on_cells(len(c.positions), c.box.diagonal(), r_list) for c in cases]
    b = _batch(cases)
    b.run(60, 20, 1, False)
    import md_driver_module as m
    for k, c in enumerate(cases):
        o = oracle(c)
        for s in range(60):
            if s % 20 == 0:
                o.calculate_neighbors()
                # the boxes at the last in-run build: wide ones below their grid, the others not
                widths = np.array(o.scalar_dict()["box"]).reshape(3, 3).diagonal() / nc[k]
                narrow = bool((widths < r_list).any())
            o.integrate()
        assert narrow == any(c is w for w in wide), k
        po, no = o.neighbors()
        pg, ng = b.neighbor_list(k)
        assert np.array_equal(np.asarray(pg), po) and np.array_equal(np.asarray(ng), no), k
        assert rel_err(b.atoms(k, m.ATOM_FORCES), o.atoms("forces")) <= 1e-9
        assert rel_err(b.atoms(k, m.ATOM_POSITIONS), o.atoms("positions")) <= 1e-9


def test_regrow_on_cells():
    c = generic_case(generic_tables(2, rcut=5.0), (9, 9, 10), 5, ensemble=2, a_ang=3.64 * 1.08)
    _on_cells(len(c.positions), c.box.diagonal(), 5.0e-8 * c.r_skin)
    old = os.environ.get("MDELAST_LIST_HEADROOM")
    os.environ["MDELAST_LIST_HEADROOM"] = "0"
    try:
        g = gpu(c)
        maxn0, _ = g.list_capacity
        for _ in range(3):
            g.run(40, 20, 1, False)
        maxn1, regrowths = g.list_capacity
    finally:
        if old is None:
            os.environ.pop("MDELAST_LIST_HEADROOM", None)
        else:
            os.environ["MDELAST_LIST_HEADROOM"] = old
    o = oracle(c)
    _run(o, 120)
    assert regrowths > 0 and maxn1 > maxn0, (maxn0, maxn1, regrowths)
    compare_state(g, o, 1e-9)
