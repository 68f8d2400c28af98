"""16 lanes per atom run as 32 on drivers of at most 1,536 atom slots in all: around that limit,
and in the force pass reading shared-memory tables, against 8 lanes per atom and the oracle.
FP64 tolerances are those of the parity tests (1e-10 static), mixed ones those of the mixed tests
(forces 2e-5, tensors 1e-4); the two table variants give the same bits per atom."""

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, gpu_atoms, gpu_scalars, oracle, rel_err

pytestmark = pytest.mark.gpu

SUMS = ("epot_atom", "born_stress_tensor", "born_elasticity_tensor", "total_laplacian", "pressure")


@pytest.mark.parametrize("precision,tol_f,tol_s", [("fp64", 1e-10, 1e-10), ("mixed", 2e-5, 1e-4)])
@pytest.mark.parametrize("neighbors", [True, False])
@pytest.mark.parametrize("edges,vacancies", [((4, 4, 4), 1), ((6, 8, 8), 0), ((6, 8, 8), 1), ((8, 7, 7), 31)])
def test_limit(edges, vacancies, neighbors, precision, tol_f, tol_s):
    c = generic_case(generic_tables(2), edges, vacancies, neighbors=neighbors)
    g, h, o = gpu(c, precision=precision), gpu(c, precision=precision), oracle(c)
    g.set_launch(16, 16, 148 * 32, 148 * 32)
    h.set_launch(8, 8, 148 * 32, 148 * 32)
    for _ in range(2):
        so = o.scalar_dict()
        for d in (g, h):
            s = gpu_scalars(d)
            assert rel_err(gpu_atoms(d, "forces"), o.atoms("forces")) <= tol_f
            for k in SUMS:
                assert rel_err(s[k], so[k]) <= tol_s, k
        for d in (g, h, o):
            d.integrate()


def test_staged_same_bits():
    c = generic_case(generic_tables(2), (5, 5, 5), 7)
    a, b = gpu(c, precision="mixed"), gpu(c, precision="mixed")
    for d in (a, b):
        d.set_launch(16, 16, 148 * 32, 148 * 32)
    b.force_staging = True
    for _ in range(3):
        a.integrate()
        b.integrate()
    assert b.force_staging and not a.force_staging
    assert np.array_equal(gpu_atoms(a, "forces"), gpu_atoms(b, "forces"))
