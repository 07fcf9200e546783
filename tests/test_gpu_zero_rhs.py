"""A solve with a zero right-hand side, then a real one on the same context, with the sums of
p.Ap and r.z taken by atomics inside other kernels (the default mode).  With b = 0 the
first inner iteration runs on 0/0 and adds NaN to both accumulators; the next solve must
not see it.  Sizes: whole smoothing passes on the fine level (8x64), single stencil
steps (32x256), element applies (64x512).

What the two solves may differ by: their inner solves stop at 1e-10 of their right-hand
side (so the last momentum residual lies below 1e-8 of F, |F + G P| being a few |F|), and
the order of the atomics may move an inner solve's stop by an iteration or two.  A trace
of the zero solve is NaN, or an alpha or beta off by O(1)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nr,nt", [(8, 64), (32, 256), (64, 512)])
@pytest.mark.parametrize("precision", [0, 1, 2])
def test_zero_right_hand_side_leaves_no_trace_in_the_default_mode(precision, nr, nt):
    from conftest import rel
    from dimspers_b200 import StokesContext, inputs

    def solve(ctx, m, scale):
        ctx.set_material_ti(m.eta_ip, m.rho, scale * m.g, m.delta, m.dir_x, m.dir_y)   # no gravity: F = 0
        ctx.assemble(precision)
        return ctx.solve(precision=precision, schur_pc=1, itmax=3, itmin=1, rtol=1e-30, inner_rtol=1e-10,
                         want_cart=False, raise_on_status=False)

    with StokesContext(nr, nt, "discontinuous") as ctx, StokesContext(nr, nt, "discontinuous") as fresh:
        m = inputs.make_material(ctx.mesh, "aniso", seed=3)
        U0, P0, _, rep0 = solve(ctx, m, 0.0)
        assert not U0.any() and not P0.any() and rep0["inner_iterations"] == 0
        U, P, _, rep = solve(ctx, m, 1.0)
        Uf, Pf, _, repf = solve(fresh, m, 1.0)
    assert np.isfinite(U).all() and np.isfinite(P).all()
    assert rep["mom_residual"] < 1e-8 and repf["mom_residual"] < 1e-8
    n, nf = rep["inner_iterations"], repf["inner_iterations"]
    assert nf > 0 and abs(n - nf) <= 4 + 0.05 * nf
    assert rel(P, Pf) < 1e-3
