"""Where a caller's device arrays may lie.  Kernels work on arrays of the context's GPU in
place; arrays that only a copy can reach (here: at an address that is no multiple of 8)
give the same results through staging, and a host address handed over as device memory
is refused with a status, as the copies refuse it, before any kernel could fault on it."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import ROOT
from dimspers_b200 import StokesContext, _lib, default_opts, inputs
from dimspers_b200 import kernel_times as KT
from dimspers_b200._lib import Arrhenius, DP_MEM_DEVICE, SolveReport, ThermalOpts, lib
from dimspers_b200.fabric import DEM

pytestmark = pytest.mark.gpu
NR, NT = 8, 36


class Array:
    """A float64 array as the entry points get it: on the GPU, 4 bytes behind an 8-byte boundary
    ("odd"), or in host memory."""

    def __init__(self, a, where):
        import torch
        self.n = a.size
        raw = np.ascontiguousarray(a, np.float64).ravel().view(np.uint8)
        self.raw = torch.zeros(raw.size + 16, dtype=torch.uint8, device="cpu" if where == "host" else "cuda")
        shift = 4 if where == "odd" else 0
        self.ptr = self.raw.data_ptr() + shift
        self.bytes = self.raw[shift:shift + raw.size]
        self.bytes.copy_(torch.from_numpy(raw))

    def get(self):
        return self.bytes.cpu().numpy().view(np.float64)


def ptrs(arrays):
    return C.cast((C.c_void_p * len(arrays))(*[a.ptr for a in arrays]), C.POINTER(C.c_void_p))


def calls(c, where):
    """name -> (status of the call, output arrays, the same results through host arrays)."""
    rng = np.random.default_rng(5)
    mk = lambda a: Array(np.asarray(a), where)                       # noqa: E731
    new = lambda n: Array(np.zeros(n), where)                        # noqa: E731
    n, nn = c.nel, c.nnod
    m = inputs.make_material(c.mesh, "aniso", seed=4)
    out = {}

    U = rng.standard_normal(2 * nn)
    ref = np.stack(list(c.stress(U, m.eta_ip, m.C6).values())).transpose(0, 2, 1)
    a, o = [mk(U), mk(m.eta_ip.T)] + [mk(f.T) for f in m.C6], new(56 * n)
    st = lib().dp_stress(c.h, a[0].ptr, a[1].ptr, n, ptrs(a[2:]), n, o.ptr, DP_MEM_DEVICE)
    out["stress"] = (st, [o], [ref])

    T, P, r, eps, tau, coh = KT.inputs_viscosity(c.mesh, NR, NT, rng)
    eta0 = np.full((n, 7), 3.3e21)
    ref = c.viscosity_arrhenius(eta0, T, P, r, eps, tau, coh, phi=30.0)
    law = Arrhenius(5e20, 8.314, 100e3, 1e-6, 1600.0, 30.0)
    a = [mk(v) for v in (T, P, r, eps.T, tau.T, coh.T, eta0.T)]
    st = lib().dp_viscosity_arrhenius(c.h, C.byref(law), a[0].ptr, a[1].ptr, P.size, a[2].ptr, a[3].ptr, a[4].ptr,
                                      a[5].ptr, a[6].ptr, DP_MEM_DEVICE)
    out["viscosity"] = (st, [a[6]], [ref.T])

    F = np.eye(2) + 0.4 * rng.standard_normal((n, 6, 2, 2))
    ref = c.fse(F)
    a, o = mk(F.transpose(1, 0, 3, 2)), [new(6 * n) for _ in range(6)]
    st = lib().dp_fse(c.h, a.ptr, ptrs(o), n, DP_MEM_DEVICE)
    out["fse"] = (st, o, [ref[k].T for k in ("vx1", "vx2", "vy1", "vy2", "a1", "a2")])

    t = np.load(os.path.join(ROOT, "tests", "golden", "dem_1e-3_vol30.npz"))
    dem = DEM(t["C"], t["ax"], 0.02)
    s = dem.struct()
    x = KT.inputs_dem(n, rng)
    ref = c.anisotropic_tensor(dem, *x)
    a, o = [mk(v.T) for v in x], [new(7 * n) for _ in range(6)]
    st = lib().dp_anisotropic_tensor(c.h, C.byref(s), *[v.ptr for v in a], n, ptrs(o), n, DP_MEM_DEVICE)
    out["dem"] = (st, o, [v.T for v in ref])

    c.set_deterministic(True)     # sums in a fixed order: the two forms are the same bit for bit
    c.set_material(m.eta_ip, m.rho, m.g, m.C6)
    c.assemble(0)
    u, p = rng.standard_normal(2 * nn), rng.standard_normal(c.npres)
    for name, fn, ref, v in (("K", lib().dp_apply_K, c.apply_K(u), u), ("G", lib().dp_apply_G, c.apply_G(p), p),
                             ("GT", lib().dp_apply_GT, c.apply_GT(u), u)):
        a, o = mk(v), new(ref.size)
        out[name] = (fn(c.h, a.ptr, o.ptr, DP_MEM_DEVICE), [o], [ref])

    if where != "host":           # the viscosity and the tensor are copied either way, only rho is read in place
        rhs = c.rhs()[0]
        a = [mk(v) for v in [m.eta_ip.T, m.rho] + [f.T for f in m.C6]]
        c.set_material(m.eta_ip, 2.0 * m.rho, m.g, m.C6)
        st = lib().dp_set_material(c.h, a[0].ptr, n, ptrs(a[2:]), n, a[1].ptr, float(m.g), DP_MEM_DEVICE)
        c.assemble(0)
        out["material"] = (st, [Array(c.rhs()[0], "host")], [rhs])

    opts = default_opts(schur_pc=1, itmax=3, itmin=1, rtol=1e-30)
    ref = c.solve(schur_pc=1, itmax=3, itmin=1, rtol=1e-30, raise_on_status=False)[:3]
    o, rep = [new(v.size) for v in ref], SolveReport()
    st = lib().dp_solve(c.h, *[v.ptr for v in o], C.byref(opts), C.byref(rep), DP_MEM_DEVICE)
    out["solve"] = (0 if st == 1 else st, o, list(ref))      # 1: the cap of three iterations
    c.set_deterministic(False)
    return out


@pytest.fixture
def ctx():
    with StokesContext(NR, NT, "discontinuous") as c:
        yield c


@pytest.mark.parametrize("where", ["gpu", "odd"])
def test_results_do_not_depend_on_where_the_arrays_lie(ctx, where):
    for name, (st, outs, refs) in calls(ctx, where).items():
        assert st == 0, (name, lib().dp_last_error(ctx.h))
        for o, r in zip(outs, refs):
            assert np.array_equal(o.get(), np.ascontiguousarray(r).ravel()), name


def test_host_addresses_as_device_memory_are_refused(ctx):
    for name, (st, _, _) in calls(ctx, "host").items():
        assert st in (_lib.DP_BAD_ARG, _lib.DP_CUDA_ERROR), name


def thermal(c, where):
    rng = np.random.default_rng(6)
    T, rho, dt = KT.inputs_thermal(c.mesh, NR, rng)
    ref = c.thermal_step(T, rho, dt, rtol=1e-13)[0]
    o = ThermalOpts()
    lib().dp_default_thermal_opts(C.byref(o))
    o.dt, o.rtol = dt, 1e-13
    Td, rd, it, rel = Array(T, where), Array(rho, where), C.c_int32(), C.c_double()
    st = lib().dp_thermal_step(c.h, C.byref(o), rd.ptr, Td.ptr, C.byref(it), C.byref(rel), DP_MEM_DEVICE)
    return st, Td.get(), ref


def test_thermal_step(ctx):
    for where in ("gpu", "odd"):
        st, T, ref = thermal(ctx, where)
        assert st == 0 and np.allclose(T, ref, rtol=1e-10, atol=0)   # both stop at 1e-13 of the right-hand side
    assert thermal(ctx, "host")[0] == _lib.DP_BAD_ARG


def test_network_output_and_guess():
    import torch

    from dimspers_b200.learned import GuessNet, grid_shape
    nrg, ntg = grid_shape(NR, NT)
    net = GuessNet(nrg, ntg, 8, 2, (1, 1), 1)
    net.init_params(1)
    x = torch.randn((1, 4, nrg, ntg), device="cuda")
    y = torch.empty((1, 1, nrg, ntg), device="cuda")
    torch.cuda.synchronize()
    net.forward(x, y)
    host = torch.zeros(nrg * ntg)
    assert lib().dp_cnn_forward(net.h, x.data_ptr(), host.data_ptr(), 1) in (_lib.DP_BAD_ARG, _lib.DP_CUDA_ERROR)
    with StokesContext(NR, NT, "discontinuous") as c:
        ref = np.zeros(c.npres)
        args = (c.h, y.data_ptr(), nrg, ntg, 2.5)
        assert lib().dp_guess_from_grid(*args, ref.ctypes.data, 0) == 0
        for where in ("gpu", "odd"):
            P = Array(np.zeros(c.npres), where)
            assert lib().dp_guess_from_grid(*args, P.ptr, DP_MEM_DEVICE) == 0
            assert np.array_equal(P.get(), ref)
        assert lib().dp_guess_from_grid(*args, Array(ref, "host").ptr, DP_MEM_DEVICE) == _lib.DP_BAD_ARG
    net.close()
