"""The dense inverse of the coarsest level (block Gauss-Jordan, one launch per
32 pivots) on meshes whose finest level is the coarsest: one V-cycle is then
K^-1, so a single inner PCG iteration has to solve the momentum equation.

Sizes n = 4 (2 nr + 1) nt with odd and even panel counts, a last panel of 32, 28
and 16 pivots, and n that are and are not multiples of the 64-row tile.  Tolerance:
the residual of an explicit inverse is bounded by n eps cond(K); uniform
viscosity on these meshes keeps cond(K) below 1e5, n <= 1536: 1536 * 1.1e-16 *
1e5 = 1.7e-8."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("deterministic", [False, True])
@pytest.mark.parametrize("nr,nt", [(1, 37), (2, 24), (3, 20), (5, 16), (4, 32), (3, 53), (4, 42)])
def test_single_level_vcycle_is_the_inverse(nr, nt, deterministic):
    from dimspers_b200 import StokesContext
    n = 4 * (2 * nr + 1) * nt
    assert n <= 1536
    with StokesContext(nr, nt, "discontinuous") as ctx:
        if deterministic:
            ctx.set_deterministic(True)
        rho = np.cos(3 * ctx.mesh.theta) * (ctx.mesh.r - 1.22)
        ctx.set_material(np.ones((ctx.nel, 7)), rho, 1e3)
        ctx.assemble(0)
        _, _, _, rep = ctx.solve(precision=0, itmax=2, itmin=1, inner_itmax=1, raise_on_status=False)
    assert rep["mg_levels"] == 1
    assert rep["status"] in (0, 1)
    assert rep["mom_residual"] < 1.7e-8
