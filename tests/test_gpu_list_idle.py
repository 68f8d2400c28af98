"""The all-pairs search of replicas of 1,000 to 3,000 atoms while their cells leave SMs idle: the
oracle's list entry for entry and its forces on both sides of the rule, and two replicas whose
cells are the faster search do not build their lists by all pairs."""

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import oracle, rel_err
from test_gpu_list_paths import _batch, _run

pytestmark = pytest.mark.gpu


# all pairs: 1,372 atoms at 51 atoms a group, 2,916 at 46; cells: 2,916 at 23, two of 2,916 at 46, five
# of 2,916 at 108; one of the first beside a larger replica on cells
@pytest.mark.parametrize("rcut,cells", [
    (5.5, [((7, 7, 7), 0)]), (5.5, [((9, 9, 9), 0)]), (5.0, [((9, 9, 9), 3)]), (5.5, [((9, 9, 9), 1)] * 2),
    (6.8, [((9, 9, 9), 0)] * 5), (5.5, [((7, 7, 7), 2), ((9, 9, 10), 1)])])
def test_both_sides(rcut, cells):
    t = generic_tables(2, rcut=rcut)
    cases = [generic_case(t, e, v, T=600.0, seed=k) for k, (e, v) in enumerate(cells)]
    b = _batch(cases)
    b.run(25, 20, 1, False)
    import md_driver_module as m
    for k in {0, len(cases) - 1}:
        o = oracle(cases[k])
        _run(o, 25)
        pg, ng = b.neighbor_list(k)
        po, no = o.neighbors()
        assert np.array_equal(np.asarray(pg), po) and np.array_equal(np.asarray(ng), no)
        assert rel_err(b.atoms(k, m.ATOM_FORCES), o.atoms("forces")) <= 1e-9


def test_two_replicas_take_the_faster_search():
    """2,916 atoms at a list radius of 6.6 A: one replica by all pairs 0.064 ms, two by all pairs 0.107 (1.67
    times), by cells 0.073 (1.14 times)."""
    t = generic_tables(2, rcut=5.5)
    cases = [generic_case(t, (9, 9, 9), 0, seed=k) for k in range(2)]
    ms = []
    for n in (1, 2):
        b = _batch(cases[:n])
        ms.append(min(b.kernel_times(20)[-1] for _ in range(5)))
    assert ms[1] <= 1.4 * ms[0], ms
