"""The K apply from the reduced element matrices (written by assemble(1)) against the
one from the packed matrices (assemble(0)), in FP64, on random vectors with
non-zero values in the constrained DOFs; in place of the atomic scatter also the
deterministic one.

Tolerance: both forms sum <= 12 products per element and <= 6 elements per node;
the reduced one adds the rounding of two subtractions and a rotation per DOF.
With |K_e| |u| / |K u| <= 100 for random u: 100 * (12 + 6 + 4) eps = 5e-13."""
import numpy as np
import pytest

from conftest import rel
from dimspers_b200 import StokesContext, inputs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("pin", [False, True])
@pytest.mark.parametrize("nr,nt", [(1, 3), (2, 3), (3, 5), (16, 17), (31, 20), (32, 256)])
def test_reduced_apply_matches_packed(nr, nt, pin, deterministic):
    rng = np.random.default_rng(11)
    with StokesContext(nr, nt, "discontinuous", pin_rotation=pin) as c:
        m = inputs.make_material(c.mesh, "aniso", seed=4)
        c.set_material_ti(m.eta_ip, m.rho, m.g, m.delta, m.dir_x, m.dir_y)
        if deterministic:
            c.set_deterministic(True)
        u = rng.standard_normal(2 * c.nnod)
        c.assemble(0)
        packed = c.apply_K(u)
        c.assemble(1)
        reduced = c.apply_K(u)
        assert rel(reduced, packed) < 5e-13
        assert np.all(reduced[c.mesh.omega] == 0.0)
        # an FP64 assembly of other data does not leave the old reduced matrices in use
        c.set_material_ti(2.0 * m.eta_ip, m.rho, m.g, m.delta, m.dir_x, m.dir_y)
        c.assemble(0)
        assert rel(c.apply_K(u), 2.0 * packed) < 5e-13


def test_solve_after_fp64_assembly_uses_the_current_material():
    """assemble(0) of new data, then a refined solve: the refined path's matrices are
    those of the new data."""
    with StokesContext(8, 64, "discontinuous") as c:
        m = inputs.make_material(c.mesh, "aniso", seed=5)
        opts = dict(precision=1, schur_pc=1, itmax=3000, rtol=1e-9)
        c.set_material_ti(m.eta_ip, m.rho, m.g, m.delta, m.dir_x, m.dir_y)
        c.assemble(1)
        U1, P1, _, _ = c.solve(**opts)
        c.set_material_ti(4.0 * m.eta_ip, m.rho, m.g, m.delta, m.dir_x, m.dir_y)
        c.assemble(0)
        U4, P4, _, rep = c.solve(**opts)
        # Stokes flow of a stiffer material: the same pressure, velocities in inverse proportion
        # (both solves to 1e-9 of a problem whose answer varies by kappa(S) * rtol: 1e-5)
        assert rep["mom_residual"] < 1e-8
        assert rel(U4, U1 / 4.0) < 1e-5 and rel(P4, P1) < 1e-5
