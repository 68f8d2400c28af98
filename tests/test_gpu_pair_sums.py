"""The pair passes' sums over warps, lanes per atom and block remainders, against the oracle,
for every lanes-per-atom variant, with and without sampling, on cells whose atom counts leave
partial warps and blocks. FP64 tolerances are those of the parity tests (1e-10 static, 1e-9
after steps), mixed ones those of the mixed tests (forces 2e-5, energies 1e-6, tensors 1e-4)."""

import numpy as np
import pytest

from generic import generic_case, generic_tables
from helpers import gpu, gpu_atoms, gpu_scalars, oracle, rel_err

pytestmark = pytest.mark.gpu

SUMS = ("born_stress_tensor", "stress_tensor", "born_elasticity_tensor", "total_laplacian",
        "total_force2", "pressure")


def _check(g, o, tol_f, tol_e, tol_s):
    so, sg = o.scalar_dict(), gpu_scalars(g)
    assert rel_err(gpu_atoms(g, "forces"), o.atoms("forces")) <= tol_f
    for k in ("epot_atom", "epot_eam_atom", "ekin_atom", "etot_cons"):
        assert rel_err(sg[k], so[k]) <= tol_e, k
    for k in SUMS:
        assert rel_err(sg[k], so[k]) <= tol_s, k


@pytest.mark.parametrize("tpa", [1, 4, 8, 16])
@pytest.mark.parametrize("types,edges,vacancies", [(1, (5, 4, 6), 3), (2, (5, 5, 5), 7), (3, (7, 7, 8), 1)])
def test_fp64(types, edges, vacancies, tpa):
    c = generic_case(generic_tables(types), edges, vacancies)
    g, o = gpu(c), oracle(c)
    g.set_launch(tpa, tpa, 148 * 8, 148 * 8)
    _check(g, o, 1e-10, 1e-10, 1e-10)
    for sample in (True, False, False, True):  # a sampled step after unsampled ones
        g.sample_observables = sample
        g.integrate()
        o.integrate()
    _check(g, o, 1e-9, 1e-9, 1e-9)


@pytest.mark.parametrize("tpa", [1, 4, 8, 16])
@pytest.mark.parametrize("types,edges,vacancies", [(1, (5, 4, 6), 3), (2, (5, 5, 5), 7), (3, (7, 7, 8), 1)])
def test_mixed(types, edges, vacancies, tpa):
    c = generic_case(generic_tables(types), edges, vacancies)
    g, o = gpu(c, precision="mixed"), oracle(c)
    g.set_launch(tpa, tpa, 148 * 8, 148 * 8)
    _check(g, o, 2e-5, 1e-6, 1e-4)
    f = gpu_atoms(g, "forces")
    assert np.abs(f.sum(axis=0)).max() <= 1e-12 * np.abs(f).sum()
    for sample in (True, False, False, True):
        g.sample_observables = sample
        g.integrate()
        o.integrate()
    _check(g, o, 2e-5, 1e-6, 1e-4)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("rmin_ang,warns", [(1.0, False), (2.45, True)])
def test_rmin_warning(precision, rmin_ang, warns):
    """The r_min warning, which the mixed pass decides from each row's smallest distance."""
    t = generic_tables(2)
    t.rmin_fatal = rmin_ang * 1e-8
    c = generic_case(t, (5, 5, 5), 7)
    g, o = gpu(c, precision=precision), oracle(c)
    assert g.status == o.status() and (g.status != 0) == warns
