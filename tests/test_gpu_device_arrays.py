"""Calls on device arrays (read and written in place) against the same calls on host
arrays (staged): bit for bit the same results, also with leading dimensions above
nel, arrays that are only 8-byte aligned, and outputs that overlap an input (which
fall back to staging).  The host forms are checked against the oracle elsewhere."""
import ctypes as C

import numpy as np
import pytest

from dimspers_b200 import StokesContext, inputs
from dimspers_b200 import kernel_times as KT
from dimspers_b200._lib import Arrhenius, DP_MEM_DEVICE, lib
from dimspers_b200.fabric import DEM

pytestmark = pytest.mark.gpu
SIZES = [(1, 3), (7, 9), (13, 21), (16, 128)]


def dev(a, pad=0, shift=0):
    """Device copy of a (columns, nel) array with `pad` extra rows per column, its first
    entry `shift` doubles into an allocation."""
    import torch
    a = np.atleast_2d(a)
    full = np.zeros((a.shape[0], a.shape[1] + pad))
    full[:, :a.shape[1]] = a
    t = torch.zeros(full.size + shift, dtype=torch.float64, device="cuda")
    t[shift:] = torch.from_numpy(full.ravel()).cuda()
    return t[shift:]


def ptrs(ts):
    return C.cast((C.c_void_p * len(ts))(*[t.data_ptr() for t in ts]), C.POINTER(C.c_void_p))


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("nr,nt", SIZES)
def test_stress(nr, nt, shift):
    import torch
    with StokesContext(nr, nt) as c:
        m = inputs.make_material(c.mesh, "aniso", seed=1)
        U = np.random.default_rng(0).standard_normal(2 * c.nnod)
        for C6 in (None, m.C6):
            ref = np.stack(list(c.stress(U, m.eta_ip, C6).values())).transpose(0, 2, 1)
            eta, Ud = dev(m.eta_ip.T, pad=5), dev(U, shift=shift)
            Cd = [dev(f.T, pad=3) for f in C6] if C6 else None
            out = torch.empty(56 * c.nel + shift, dtype=torch.float64, device="cuda")[shift:]
            c._chk(lib().dp_stress(c.h, Ud.data_ptr(), eta.data_ptr(), c.nel + 5, ptrs(Cd) if Cd else None,
                                   c.nel + 3 if Cd else 0, out.data_ptr(), DP_MEM_DEVICE))
            assert np.array_equal(out.cpu().numpy().reshape(8, 7, c.nel), ref)
        # the result over the viscosity columns
        both = torch.cat([dev(m.eta_ip.T), torch.zeros(49 * c.nel, dtype=torch.float64, device="cuda")])
        Cd = [dev(f.T) for f in m.C6]
        c._chk(lib().dp_stress(c.h, Ud.data_ptr(), both.data_ptr(), c.nel, ptrs(Cd), c.nel, both.data_ptr(),
                               DP_MEM_DEVICE))
        assert np.array_equal(both.cpu().numpy().reshape(8, 7, c.nel), ref)
        assert c.profile_kernel(3, 1) > 0


@pytest.mark.parametrize("nr,nt", SIZES)
def test_viscosity(nr, nt):
    with StokesContext(nr, nt) as c:
        T, P, r, eps, tau, coh = KT.inputs_viscosity(c.mesh, nr, nt, np.random.default_rng(1))
        eta0 = np.full((c.nel, 7), 3.3e21)
        ref = c.viscosity_arrhenius(eta0, T, P, r, eps, tau, coh, phi=30.0)
        law = Arrhenius(5e20, 8.314, 100e3, 1e-6, 1600.0, 30.0)
        d = [dev(a) for a in (T, P, r, eps.T, tau.T, coh.T, eta0.T)]
        call = lambda eta: c._chk(lib().dp_viscosity_arrhenius(     # noqa: E731
            c.h, C.byref(law), d[0].data_ptr(), d[1].data_ptr(), d[1].numel(), d[2].data_ptr(), d[3].data_ptr(),
            d[4].data_ptr(), d[5].data_ptr(), eta.data_ptr(), DP_MEM_DEVICE))
        call(d[6])
        assert np.array_equal(d[6].cpu().numpy().reshape(7, c.nel).T, ref)
        d[4].fill_(0.0)        # eta written over the strain rate: nothing yields, etaTP elsewhere
        ref0 = c.viscosity_arrhenius(eps, T, P, r, eps, 0 * tau, coh, phi=30.0)
        call(d[3])
        assert np.array_equal(d[3].cpu().numpy().reshape(7, c.nel).T, ref0)


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("nr,nt", SIZES)
def test_fse_and_dem_tensor(nr, nt, shift):
    import os

    from conftest import ROOT
    t = np.load(os.path.join(ROOT, "tests", "golden", "dem_1e-3_vol30.npz"))
    dem = DEM(t["C"], t["ax"], 0.02)
    rng = np.random.default_rng(2)
    with StokesContext(nr, nt) as c:
        n, ld = c.nel, c.nel + 7
        F = np.eye(2) + 0.4 * rng.standard_normal((n, 6, 2, 2))
        ref = c.fse(F)
        Fd = dev(F.transpose(1, 0, 3, 2).ravel(), shift=shift)
        out = [dev(np.zeros((6, ld))) for _ in range(6)]
        c._chk(lib().dp_fse(c.h, Fd.data_ptr(), ptrs(out), ld, DP_MEM_DEVICE))
        for o, k in zip(out, ("vx1", "vx2", "vy1", "vy2", "a1", "a2")):
            assert np.array_equal(o.cpu().numpy().reshape(6, ld)[:, :n].T, ref[k])
        x, y, r1, r2 = KT.inputs_dem(n, rng)
        ref = c.anisotropic_tensor(dem, x, y, r1, r2)
        d = [dev(a.T, pad=7) for a in (x, y, r1, r2)]
        out = [dev(np.zeros((7, n))) for _ in range(6)]
        s = dem.struct()
        c._chk(lib().dp_anisotropic_tensor(c.h, C.byref(s), *[a.data_ptr() for a in d], ld, ptrs(out), n,
                                           DP_MEM_DEVICE))
        for o, k in zip(out, ref):
            assert np.array_equal(o.cpu().numpy().reshape(7, n).T, k)
        # the first output over the inputs x and y
        xy, r1d, r2d = dev(np.concatenate([x.T, y.T])), dev(r1.T), dev(r2.T)
        out[0] = xy
        c._chk(lib().dp_anisotropic_tensor(c.h, C.byref(s), xy.data_ptr(), xy[6 * n:].data_ptr(), r1d.data_ptr(),
                                           r2d.data_ptr(), n, ptrs(out), n, DP_MEM_DEVICE))
        assert np.array_equal(xy.cpu().numpy()[:7 * n].reshape(7, n).T, ref[0])


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("nr,nt", SIZES)
def test_operators(nr, nt, shift):
    import torch
    rng = np.random.default_rng(3)
    with StokesContext(nr, nt) as c:
        m = inputs.make_material(c.mesh, "aniso", seed=2)
        eta, rho = dev(m.eta_ip.T, pad=2), dev(m.rho, shift=shift)
        Cd = [dev(f.T, pad=4) for f in m.C6]
        c.set_material(m.eta_ip, m.rho, m.g, m.C6)
        c.set_deterministic(True)          # sums in a fixed order, so that the two forms can be compared bit for bit
        c.assemble(0)
        u, p = rng.standard_normal(2 * c.nnod), rng.standard_normal(c.npres)
        ref = (c.apply_K(u), c.apply_G(p), c.apply_GT(u), c.rhs()[0])
        c.set_material_device(eta.data_ptr(), c.nel + 2, rho.data_ptr(), m.g, [f.data_ptr() for f in Cd], c.nel + 4)
        c.assemble(0)
        for fn, x, want in ((lib().dp_apply_K, u, ref[0]), (lib().dp_apply_G, p, ref[1]), (lib().dp_apply_GT, u, ref[2])):
            xd = dev(x, shift=shift)
            yd = torch.empty(want.size + shift, dtype=torch.float64, device="cuda")[shift:]
            c._chk(fn(c.h, xd.data_ptr(), yd.data_ptr(), DP_MEM_DEVICE))
            assert np.array_equal(yd.cpu().numpy(), want)
        xd = dev(u, shift=shift)
        c._chk(lib().dp_apply_K(c.h, xd.data_ptr(), xd.data_ptr(), DP_MEM_DEVICE))    # in place
        assert np.array_equal(xd.cpu().numpy(), ref[0])
        assert np.array_equal(c.rhs()[0], ref[3])
