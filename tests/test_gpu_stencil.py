"""The node-stencil smoother of the small multigrid levels against the forms it
replaces: the element-by-element levels of the cluster tail (coarse levels) and
the matrix-free fine level, which never uses stencils.

One inner PCG iteration per K-solve makes U a fixed number of V-cycles of the
data, so the comparison sees the V-cycle itself and not a converged solution.
Tolerances: the two forms sum the same products in another order.  A V-cycle is
~50 operator applications with O(1) amplification, each with a rounding error
of ~20 eps, and the Schur step's differences cancel at most two digits:
50 * 20 * 100 * eps = 1e5 eps, i.e. 2.2e-11 in FP64; the FP32 hierarchy enters
through a preconditioner only, 50 * 20 * eps32 = 6e-5 before the same factor,
taken once per V-cycle (there are three): 2e-4."""
import numpy as np
import pytest

from conftest import rel

pytestmark = pytest.mark.gpu

# (radial, angular) cells: whole hierarchies whose levels have odd radial counts,
# counts that leave partly filled warps, and the largest level with stencils
SIZES = [(6, 40), (10, 72), (12, 96), (16, 128), (28, 208), (32, 256)]


def _solve(nr, nt, precision, **opts):
    from dimspers_b200 import StokesContext, inputs
    with StokesContext(nr, nt, "discontinuous") as ctx:
        m = inputs.make_material(ctx.mesh, "aniso", seed=3)
        ctx.set_material_ti(m.eta_ip, m.rho, m.g, m.delta, m.dir_x, m.dir_y)
        ctx.assemble(precision)
        U, P, _, rep = ctx.solve(precision=precision, schur_pc=1, itmax=1, itmin=1, inner_itmax=1, want_cart=False,
                                 raise_on_status=False, remove_rotation=0, **opts)
    assert rep["status"] == 1 and np.isfinite(U).all()
    return U, P


@pytest.mark.parametrize("precision,tol", [(0, 2.2e-11), (1, 2e-4)])
@pytest.mark.parametrize("nr,nt", SIZES)
def test_stencil_vcycle_matches_element_forms(nr, nt, precision, tol):
    U, P = _solve(nr, nt, precision)
    Um, Pm = _solve(nr, nt, precision, matrix_free=1)                    # fine level without stencils
    Ut, Pt = _solve(nr, nt, precision, matrix_free=1, mg_tail=1 << 20)   # no level with stencils
    for a, b in ((U, Um), (Um, Ut)):
        assert rel(a, b) < tol
    for a, b in ((P, Pm), (Pm, Pt)):
        assert rel(a, b) < tol


@pytest.mark.parametrize("degree", [1, 2, 4])
def test_stencil_smoother_degrees(degree):
    """Degree 1 keeps the element form; even and odd step counts end in either d buffer."""
    U, P = _solve(16, 128, 0, cheb_degree=degree)
    Ut, Pt = _solve(16, 128, 0, cheb_degree=degree, matrix_free=1, mg_tail=1 << 20)
    assert rel(U, Ut) < 2.2e-11 and rel(P, Pt) < 2.2e-11


@pytest.mark.parametrize("degree", [2, 3])
@pytest.mark.parametrize("nr,nt", [(140, 292), (128, 640)])
def test_late_x_smoother(nr, nt, degree):
    """Levels too large for stencils put x together after the smoothing (degrees 2 and 3): two such
    levels, reached by either form of the restriction, against the cluster tail's step-by-step x.
    (140, 292) halves once only, so that its coarsest level is smoothed too."""
    U, P = _solve(nr, nt, 0, cheb_degree=degree)
    Ut, Pt = _solve(nr, nt, 0, cheb_degree=degree, matrix_free=1, mg_tail=1 << 20)
    assert rel(U, Ut) < 2.2e-11 and rel(P, Pt) < 2.2e-11


@pytest.mark.parametrize("precision,tol", [(0, 2.2e-11), (1, 2e-4)])
@pytest.mark.parametrize("nr,nt", [(2, 8), (2, 148), (16, 148), (18, 148), (20, 148), (20, 152), (22, 40)])
def test_whole_pass_smoother_edges(nr, nt, precision, tol):
    """The edges of the levels smoothed by whole passes: the fewest cells either way, the radial counts
    that fill a block in FP64 (16) and FP32 (20) and the next ones, one wave of blocks and more."""
    U, P = _solve(nr, nt, precision)
    Ut, Pt = _solve(nr, nt, precision, matrix_free=1, mg_tail=1 << 20)
    assert rel(U, Ut) < tol and rel(P, Pt) < tol
