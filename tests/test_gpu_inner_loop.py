"""The inner solve's first iteration stands before its loop: a zero right-hand
side must still come back as zero (nothing iterates, nothing is counted), and
leave no trace in the context's vectors for the solves after it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,nr,nt", [(0, 8, 64), (1, 8, 64), (2, 8, 64), (1, 36, 288)])
def test_zero_right_hand_side_leaves_no_trace(precision, nr, nt):
    from dimspers_b200 import StokesContext, inputs

    def solve(ctx, m, scale):
        ctx.set_material_ti(m.eta_ip, scale * m.rho, m.g, m.delta, m.dir_x, m.dir_y)
        ctx.assemble(precision)
        return ctx.solve(precision=precision, schur_pc=1, itmax=3, itmin=1, rtol=1e-30, want_cart=False,
                         raise_on_status=False, remove_rotation=0)

    with StokesContext(nr, nt, "discontinuous") as ctx, StokesContext(nr, nt, "discontinuous") as fresh:
        m = inputs.make_material(ctx.mesh, "aniso", seed=3)
        for c in (ctx, fresh):
            c.set_deterministic(True)
        U0, P0, _, rep0 = solve(ctx, m, 0.0)
        assert not U0.any() and not P0.any() and rep0["inner_iterations"] == 0
        U, P, _, rep = solve(ctx, m, 1.0)
        Uf, Pf, _, repf = solve(fresh, m, 1.0)
    assert np.array_equal(U, Uf) and np.array_equal(P, Pf)
    assert rep["inner_iterations"] == repf["inner_iterations"] > 0
