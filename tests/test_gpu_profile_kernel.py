"""dp_profile_kernel times kernels on a call's own inputs or not at all."""
import ctypes as C
import os

import numpy as np
import pytest

from conftest import ROOT
from dimspers_b200 import StokesContext, inputs
from dimspers_b200 import kernel_times as KT
from dimspers_b200._lib import Arrhenius, DP_MEM_DEVICE, lib
from dimspers_b200.fabric import DEM

pytestmark = pytest.mark.gpu


def test_staged_kernels_are_timed_on_a_calls_inputs_or_refused():
    import torch
    nr, nt = 8, 36
    cuda = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()      # noqa: E731
    new = lambda n: torch.zeros(n, dtype=torch.float64, device="cuda")     # noqa: E731
    ptrs = lambda ts: C.cast((C.c_void_p * len(ts))(*[t.data_ptr() for t in ts]), C.POINTER(C.c_void_p))  # noqa: E731
    with StokesContext(nr, nt, "discontinuous") as c:
        m = inputs.make_material(c.mesh, "aniso", seed=4)
        rng = np.random.default_rng(5)
        n = c.nel
        U = rng.standard_normal(2 * c.nnod)
        vis = KT.inputs_viscosity(c.mesh, nr, nt, rng)
        eta0 = np.full((n, 7), 3.3e21)
        law = Arrhenius(5e20, 8.314, 100e3, 1e-6, 1600.0, 30.0)
        t = np.load(os.path.join(ROOT, "tests", "golden", "dem_1e-3_vol30.npz"))
        dem = DEM(t["C"], t["ax"], 0.02)
        s = dem.struct()
        x = KT.inputs_dem(n, rng)
        F = np.eye(2) + 0.4 * rng.standard_normal((n, 6, 2, 2))

        def device_calls():
            a = [cuda(U), cuda(m.eta_ip.T)] + [cuda(f.T) for f in m.C6] + [new(56 * n)]
            c._chk(lib().dp_stress(c.h, a[0].data_ptr(), a[1].data_ptr(), n, ptrs(a[2:8]), n, a[8].data_ptr(),
                                   DP_MEM_DEVICE))
            b = [cuda(v) for v in (*vis[:3], vis[3].T, vis[4].T, vis[5].T, eta0.T)]
            c._chk(lib().dp_viscosity_arrhenius(c.h, C.byref(law), b[0].data_ptr(), b[1].data_ptr(), b[1].numel(),
                                                *[v.data_ptr() for v in b[2:]], DP_MEM_DEVICE))
            d, o = [cuda(v.T) for v in x], [new(7 * n) for _ in range(6)]
            c._chk(lib().dp_anisotropic_tensor(c.h, C.byref(s), *[v.data_ptr() for v in d], n, ptrs(o), n,
                                               DP_MEM_DEVICE))
            Fd = cuda(F.transpose(1, 0, 3, 2))
            c._chk(lib().dp_fse(c.h, Fd.data_ptr(), ptrs(o), n, DP_MEM_DEVICE))

        device_calls()                    # in place: nothing is staged
        for which in (3, 4, 5):
            with pytest.raises(Exception, match="host arrays"):
                c.profile_kernel(which, 1)
        c.stress(U, m.eta_ip)             # without the tensor, whose columns stay unset
        c.viscosity_arrhenius(eta0, *vis, phi=30.0)
        c.anisotropic_tensor(dem, *x)
        device_calls()                    # these leave the staged inputs alone
        for which in (3, 4, 5):
            assert c.profile_kernel(which, 1) > 0
        c.fse(F)                          # staged over the tensor lookup's inputs
        with pytest.raises(Exception, match="host arrays"):
            c.profile_kernel(5, 1)


def test_timed_region_holds_the_kernel_alone():
    """What the GPU runs in a call with 3 + 1 launches of the thermal apply: as many kernels, and no
    more copies or memsets than the call's set-up has whatever the launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile
    with StokesContext(16, 128, "continuous") as c:
        T, rho, dt = KT.inputs_thermal(c.mesh, 16, np.random.default_rng(0))
        c.thermal_step(T, rho, dt)
        c.profile_kernel(6, 1)
        seen = {}
        for reps in (1, 3):
            torch.cuda.synchronize()
            with profile(activities=[ProfilerActivity.CUDA]) as prof:
                c.profile_kernel(6, reps)
                torch.cuda.synchronize()
            names = [e.name for e in prof.events()]
            seen[reps] = (sum("k_th_apply" in k for k in names), sum("emset" in k for k in names))
    assert seen[1][0] == 2 and seen[3][0] == 4
    assert seen[1][1] == seen[3][1] > 0


def test_fp64_apply_of_the_benchmark_is_the_kernel_it_names():
    import sys

    import torch
    from torch.profiler import ProfilerActivity, profile
    sys.path.insert(0, ROOT)
    import bench
    with StokesContext(16, 128, "discontinuous") as c:
        m = inputs.make_material(c.mesh, "aniso", seed=4)
        c.set_material(m.eta_ip, m.rho, m.g, m.C6)
        c.assemble(1)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            rec = bench.fp64_apply_roofline(c, c.nel, c.nnod, 6546.2)
            torch.cuda.synchronize()
    named = rec["kernel"].split(" ")[0].rstrip(">")          # k_apply_R<double
    applies = [e.name for e in prof.events() if "k_apply_" in e.name]
    assert len(applies) == 21 and all(named in k for k in applies), (named, set(applies))
