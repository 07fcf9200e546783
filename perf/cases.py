"""Workloads that the library's speed is measured on: the calls of one time step
of an annulus convection program (Stokes solve, operator update, stress,
viscosity, fabric, thermal diffusion) and the learned guess (prediction,
training), each through the public entry points with device-resident arrays.

A program keeps one context per mesh and gives it new fields every step, so a
context (and the mesh arrays) is kept per mesh here too; every pass hands all of
its inputs over again.  Sizes: 32x256, 128x1024, 256x2048 and 512x4096 are the
configurations of this repository's benchmark and tests; the others are generic.
"""
import ctypes as C
import math

import numpy as np
import torch

from dimspers_b200 import StokesContext, learned
from dimspers_b200._lib import Arrhenius, DP_MEM_DEVICE, ThermalOpts, lib
from dimspers_b200.fabric import DEM

R_IN, R_OUT = 1.22, 2.22
F64 = torch.float64
# the fast path of the benchmark: FP32 element data and multigrid under an FP64 Krylov
FAST = dict(precision=1, cheb_degree=3, cheb_lo=0.05, inner_rtol=1e-10, inner_relax=1e-2, relax_base=1e-8, schur_pc=1)
# the reference's algorithm (lumped-mass Schur preconditioner, tight inner solves), all FP64
PLAIN = dict(precision=0, cheb_degree=3, cheb_lo=0.05, inner_rtol=1e-10, inner_relax=0.0, schur_pc=0)
ARRHENIUS = dict(eta0=5e20, R=8.314, Ea=100e3, Va=1e-6, T0=1600.0, phi_deg=30.0)
THERMAL = dict(K=3.3, Cp=1.2e3, Ttop=300.0, Tbot=4000.0)
ARCH = dict(channels=32, layers=6, dilations=(1, 2, 4, 8, 16, 1))  # the committed network


def listed():
    return [
        # a small exploratory model in the reference's own setting: vertex (continuous)
        # pressure, FP64, the reference's preconditioner
        dict(name="solve_16x128_fp64", kind="solve", nr=16, nt=128, pressure="continuous", material="aniso",
             precision=0, outer=0, deterministic=False),
        # the fast path on a small mesh (66k velocity DOF, discontinuous pressure), with the
        # options' default cap of 200 outer iterations, where the solve of a time step stops
        dict(name="solve_32x256_200", kind="solve", nr=32, nt=256, pressure="discontinuous", material="aniso",
             precision=1, outer=200, deterministic=False),
        # the ordinary production mesh (1.05M velocity DOF), with the same cap
        dict(name="solve_128x1024_200", kind="solve", nr=128, nt=1024, pressure="discontinuous", material="aniso",
             precision=1, outer=200, deterministic=False),
        # the headline mesh (16.8M velocity DOF): the fixed-length solve that the
        # autotuner scores settings with (material, assembly, set-up, 30 outer iterations)
        dict(name="solve_512x4096_30", kind="solve", nr=512, nt=4096, pressure="discontinuous",
             material="fabric", precision=1, outer=30, deterministic=False),
        # one nonlinear (Picard) residual: new tensors, assembly, K u, G p, G^T u
        dict(name="operator_256x2048", kind="operator", nr=256, nt=2048, pressure="discontinuous", material="aniso",
             precision=0),
        # strain rate and stress after a solve: a small ragged mesh (latency), a large one
        dict(name="stress_31x200", kind="stress", nr=31, nt=200, tensor=False),
        dict(name="stress_256x2048", kind="stress", nr=256, nt=2048, tensor=True),
        # the material update of a time step: Arrhenius viscosity with plasticity ...
        dict(name="viscosity_128x1024", kind="viscosity", nr=128, nt=1024),
        # ... and finite-strain ellipsoids with the DEM tensor lookup, on an odd mesh
        dict(name="fabric_121x901", kind="fabric", nr=121, nt=901),
        # backward-Euler diffusion step of the temperature
        dict(name="thermal_128x1024", kind="thermal", nr=128, nt=1024, heated=True),
        # learned initial guess: network inputs, prediction, prolongation to the pressure
        dict(name="guess_128x1024", kind="guess", nr=128, nt=1024),
        # training of that network: one Adam step on a batch of 8
        dict(name="train_128x1024_b8", kind="train", nr=128, nt=1024, batch=8),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("solve", "solve", "solve", "operator", "stress", "viscosity", "fabric", "thermal", "guess",
                       "train"))
    if kind == "solve":
        # meshes that halve down to the dense coarsest level, as users choose them
        halvings = rng.randint(2, 5)
        nr, nt = rng.randint(2, 4) << halvings, rng.randint(24, 36) << halvings
        precision = rng.choice((1, 1, 0))
        cont = rng.random() < 0.3
        outer = 0 if cont and halvings <= 4 else rng.randint(8, 24)
        return dict(kind=kind, nr=nr, nt=nt, pressure="continuous" if cont else "discontinuous",
                    material=rng.choice(("iso", "aniso", "fabric")), precision=precision, outer=outer,
                    deterministic=not cont and rng.random() < 0.2)
    if kind == "operator":
        nr = _log_int(rng, 12, 256)
        return dict(kind=kind, nr=nr, nt=_log_int(rng, 4 * nr, 9 * nr),
                    pressure=rng.choice(("discontinuous", "continuous")), material=rng.choice(("iso", "aniso")),
                    precision=rng.choice((0, 1)))
    if kind in ("stress", "viscosity", "fabric", "thermal"):
        nr = _log_int(rng, 20, 256)
        d = dict(kind=kind, nr=nr, nt=_log_int(rng, 4 * nr, 9 * nr))
        if kind == "stress":
            d["tensor"] = rng.random() < 0.6
        if kind == "thermal":
            d["heated"] = rng.random() < 0.7
        return d
    nr = 2 * _log_int(rng, 17, 96)
    nt = 32 * _log_int(rng, max(4, nr // 8), max(5, nr // 4))
    d = dict(kind=kind, nr=nr, nt=nt)
    if kind == "train":
        d["batch"] = rng.randint(1, 8) if nr * nt < 100000 else rng.randint(1, 4)
    return d


# ---- meshes and fields ---------------------------------------------------------------
_kept = {}


def _mesh(nr, nt, pressure="discontinuous", deterministic=False):
    """(context, theta, r, e2n) of a mesh, node arrays on the GPU; the last one is kept."""
    key = (nr, nt, pressure, deterministic)
    if key not in _kept:
        for old in list(_kept.values()):
            old[0].close()
        _kept.clear()
        ctx = StokesContext(nr, nt, pressure)
        if deterministic:
            ctx.set_deterministic(True)
        _kept[key] = (ctx, torch.from_numpy(ctx.mesh.theta).cuda(), torch.from_numpy(ctx.mesh.r).cuda(),
                      torch.from_numpy(np.ascontiguousarray(ctx.mesh.e2n)).cuda())
    return _kept[key]


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _rand(g, *shape):
    return torch.rand(*shape, generator=g, device="cuda", dtype=F64)


def _ips6():
    """The 6-point rule of the Stokes assembly: points and weights."""
    b = math.sqrt(38.0 - 44.0 * math.sqrt(0.4))
    g1, g2 = (8.0 - math.sqrt(10.0) + b) / 18.0, (8.0 - math.sqrt(10.0) - b) / 18.0
    c = math.sqrt(213125.0 - 53320.0 * math.sqrt(10.0))
    w1, w2 = (620.0 + c) / 3720.0, (620.0 - c) / 3720.0
    pts = [(1 - 2 * g1, g1), (g1, 1 - 2 * g1), (g1, g1), (1 - 2 * g2, g2), (g2, 1 - 2 * g2), (g2, g2)]
    return pts, [0.5 * w1] * 3 + [0.5 * w2] * 3


def _ips7():
    """The 7-point rule of the stress, viscosity and thermal kernels."""
    q = math.sqrt(15.0)
    g1, g2 = (6.0 - q) / 21.0, (6.0 + q) / 21.0
    w1, w2 = (155.0 - q) / 1200.0, (155.0 + q) / 1200.0
    pts = [(1 / 3, 1 / 3), (1 - 2 * g1, g1), (g1, 1 - 2 * g1), (g1, g1), (1 - 2 * g2, g2), (g2, 1 - 2 * g2), (g2, g2)]
    return pts, [0.5 * 0.225] + [0.5 * w1] * 3 + [0.5 * w2] * 3


def _n3(p):
    return torch.tensor([1 - p[0] - p[1], p[0], p[1]], dtype=F64, device="cuda")


def _n6(p):
    r, s = p
    t = 1 - r - s
    return torch.tensor([t * (2 * t - 1), r * (2 * r - 1), s * (2 * s - 1), 4 * r * t, 4 * r * s, 4 * s * t], dtype=F64,
                        device="cuda")


def _dn6(p):
    r, s = p
    t = 1 - r - s
    return torch.tensor([[1 - 4 * t, 4 * r - 1, 0, 4 * (t - r), 4 * s, -4 * s],
                         [1 - 4 * t, 0, 4 * s - 1, -4 * r, 4 * r, 4 * (t - s)]], dtype=F64, device="cuda")


def _fourier(th, r, phases):
    rho = (r - R_IN) / (R_OUT - R_IN)
    return sum(torch.cos(m * th + (1 + m % 3) * math.pi * rho + 2 * math.pi * phases[m - 1]) / m
               for m in range(1, 1 + len(phases)))


def _material(case, seed):
    """Viscosity at the IPs (7, nel), nodal density, gravity factor and, if anisotropic,
    delta and director per element: a conductive profile with plumes (radius 0.05-0.2,
    amplitude up to 0.3), temperature-dependent viscosity of contrast 1e3 (iso), 1e5
    (aniso) or 1e6 (fabric), weak-plane factor delta in [1, 10]."""
    _, th, r, e2n = _mesh(case["nr"], case["nt"], case.get("pressure", "discontinuous"),
                          case.get("deterministic", False))
    g = _gen(seed)
    T = torch.log(r / R_OUT) / math.log(R_IN / R_OUT)
    for a, b, w, amp in _rand(g, 8, 4).tolist():
        x, z = r * torch.sin(th) - (R_IN + 0.1 + 0.8 * b) * math.sin(2 * math.pi * a), \
            r * torch.cos(th) - (R_IN + 0.1 + 0.8 * b) * math.cos(2 * math.pi * a)
        T = T + 0.3 * (2 * amp - 1) * torch.exp(-(x * x + z * z) / (0.05 + 0.15 * w) ** 2)
    contrast = {"iso": 1e3, "aniso": 1e5, "fabric": 1e6}[case["material"]]
    N7 = torch.stack([_n6(p) for p in _ips6()[0]] + [_n6((1 / 3, 1 / 3))])
    eta = torch.stack([torch.exp(-math.log(contrast) * sum(n[k] * T[e2n[k]] for k in range(6))) for n in N7])
    m = dict(eta=eta.contiguous(), rho=T.contiguous(), g=1e5)
    if case["material"] != "iso":
        nel = e2n.shape[1]
        thc = th[e2n[0]] + (math.pi / case["nt"])     # an element's angle, without the seam
        rc = r[e2n[:3]].mean(0)
        m["delta"] = (1 + 9 * _rand(g, nel)).contiguous()
        ph = _rand(g, 4, 8).tolist()
        if case["material"] == "aniso":
            phi = _fourier(thc, rc, ph[0])
            vx, vy = torch.cos(phi), torch.sin(phi)
        else:                                          # major axis of F F^T, F = I + 0.5 G
            f = [0.5 * _fourier(thc, rc, q) for q in ph]
            vx, vy, _, _ = _axes(1 + f[0], f[1], f[2], 1 + f[3])
        m["dx"], m["dy"] = vx.contiguous(), vy.contiguous()
    return m


def _axes(f11, f21, f12, f22):
    """Major unit eigenvector and the semi-axes of F F^T."""
    l11, l12, l22 = f11 * f11 + f12 * f12, f11 * f21 + f12 * f22, f21 * f21 + f22 * f22
    lmax = 0.5 * (l11 + l22) + torch.sqrt(0.25 * (l11 - l22) ** 2 + l12 * l12)
    a, b = (l12, lmax - l11), (lmax - l22, l12)
    use = a[0] ** 2 + a[1] ** 2 >= b[0] ** 2 + b[1] ** 2
    vx, vy = torch.where(use, a[0], b[0]), torch.where(use, a[1], b[1])
    n = torch.sqrt(vx * vx + vy * vy)
    none = n == 0
    vx, vy = torch.where(none, 1.0, vx / n.clamp_min(1e-300)), torch.where(none, 0.0, vy / n.clamp_min(1e-300))
    a1 = torch.sqrt(lmax)
    return vx, vy, a1, (f11 * f22 - f12 * f21).abs() / a1


def _rotated(delta, dx, dy):
    """The transversely isotropic tensor (C11, C33, C55, C13, C15, C35) about the director."""
    return _rotate(dx, dy, 4 / 3, 4 / 3, 1 / delta, -2 / 3)


def _rotate(dx, dy, a, c, e, h):
    n = 1 / torch.sqrt(dx * dx + dy * dy)
    cs, sn = dx * n, dy * n
    x1, y2, x2, y1 = cs, cs, sn, -sn
    m = x1 * y2 + x2 * y1
    p, q = a * x1 * x1 + h * x2 * x2, c * x2 * x2 + h * x1 * x1
    return (p * x1 * x1 + (q + 4 * e * x1 * x1) * x2 * x2,
            (a * y1 * y1 + h * y2 * y2) * y1 * y1 + (c * y2 * y2 + h * y1 * y1 + 4 * e * y1 * y1) * y2 * y2,
            (c * x2 * y2 + h * x1 * y1) * x2 * y2 + m * m * e + (a * x1 * y1 + h * x2 * y2) * x1 * y1,
            (q * y2 + 4 * e * x1 * x2 * y1) * y2 + p * y1 * y1,
            (q * y2 + 2 * m * e * x1) * x2 + p * x1 * y1,
            ((c * y2 * y2 + h * y1 * y1) * x2 + 2 * m * e * y1) * y2 + (a * y1 * y1 + h * y2 * y2) * x1 * y1)


def _tensor7(m):
    """Six tensor fields, (7, nel) each (the same at every IP of an element)."""
    return [c.expand(7, -1).contiguous() for c in _rotated(m["delta"], m["dx"], m["dy"])]


def _ptrs(tensors):
    return (C.c_void_p * len(tensors))(*[t.data_ptr() for t in tensors])


def _dem():
    """A DEM table of the reference's shape: 10 x 10 inclusion shapes, the weak-plane
    viscosity falling with the aspect ratio."""
    s = np.linspace(0.0, 1.8, 10)
    a1, a3 = np.meshgrid(10.0 ** s, 10.0 ** (-1.1 * s), indexing="ij")
    a1, a3 = a1.ravel(), a3.ravel()
    t = np.zeros((100, 9))
    aspect = np.log10(a1 / a3)
    for k, (c0, c1) in enumerate(((1.3, 0.1), (1.3, 0.05), (1.25, 0.12), (1, -0.1), (1, -0.24), (1, -0.05), (-0.6, 0.02),
                                  (-0.65, 0.04), (-0.6, 0.01))):
        t[:, k] = c0 + c1 * aspect
    return DEM(t, np.stack([a1, np.ones(100), a3], 1), 0.02)


# ---- prepare -----------------------------------------------------------------------------
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return globals()["_run_" + state["case"]["kind"]](state)


def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    with torch.no_grad() if case["kind"] != "train" else torch.enable_grad():
        return f(case, seed) if f else None


def _set_material(ctx, m, C6=None):
    nel = ctx.nel
    if C6 is not None:
        ctx.set_material_device(m["eta"].data_ptr(), nel, m["rho"].data_ptr(), m["g"], [c.data_ptr() for c in C6], nel)
    elif "delta" in m:
        ctx.set_material_ti_device(m["eta"].data_ptr(), nel, m["rho"].data_ptr(), m["g"], m["delta"].data_ptr(),
                                   m["dx"].data_ptr(), m["dy"].data_ptr())
    else:
        ctx.set_material_device(m["eta"].data_ptr(), nel, m["rho"].data_ptr(), m["g"])


def _prepare_solve(case, seed):
    ctx = _mesh(case["nr"], case["nt"], case["pressure"], case["deterministic"])[0]
    o = dict(FAST if case["precision"] == 1 else PLAIN)
    if case["pressure"] == "continuous":
        o["schur_pc"] = 0
    o.update(rtol=1e-8, itmax=case["outer"] or 20000)
    return dict(case=case, ctx=ctx, m=_material(case, seed), o=o,
                U=torch.zeros(2 * ctx.nnod, dtype=F64, device="cuda"),
                P=torch.zeros(ctx.npres, dtype=F64, device="cuda"))


def _run_solve(s):
    ctx = s["ctx"]
    _set_material(ctx, s["m"])
    ctx.assemble(s["o"]["precision"])
    ctx.solve_device(s["U"].data_ptr(), s["P"].data_ptr(), **s["o"])
    return s["U"], s["P"]


def _prepare_operator(case, seed):
    ctx = _mesh(case["nr"], case["nt"], case["pressure"])[0]
    m = _material(case, seed)
    g = _gen(seed + 1000003)
    return dict(case=case, ctx=ctx, m=m, C6=_tensor7(m) if "delta" in m else None,
                u=2 * _rand(g, 2 * ctx.nnod) - 1, p=2 * _rand(g, ctx.npres) - 1,
                Ku=torch.empty(2 * ctx.nnod, dtype=F64, device="cuda"),
                Gp=torch.empty(2 * ctx.nnod, dtype=F64, device="cuda"),
                Gu=torch.empty(ctx.npres, dtype=F64, device="cuda"))


def _run_operator(s):
    ctx, L = s["ctx"], lib()
    _set_material(ctx, s["m"], s["C6"])
    ctx.assemble(s["case"]["precision"])
    ctx._chk(L.dp_apply_K(ctx.h, s["u"].data_ptr(), s["Ku"].data_ptr(), DP_MEM_DEVICE))
    ctx._chk(L.dp_apply_G(ctx.h, s["p"].data_ptr(), s["Gp"].data_ptr(), DP_MEM_DEVICE))
    ctx._chk(L.dp_apply_GT(ctx.h, s["u"].data_ptr(), s["Gu"].data_ptr(), DP_MEM_DEVICE))
    return s["Ku"], s["Gp"], s["Gu"]


def _prepare_stress(case, seed):
    ctx, th, r, _ = _mesh(case["nr"], case["nt"])
    m = _material(dict(case, material="aniso"), seed)
    g = _gen(seed + 1000003)
    u = torch.stack([_fourier(th, r, _rand(g, 8).tolist()) for _ in range(2)], 1) + 1e-3 * _rand(g, ctx.nnod, 2)
    return dict(case=case, ctx=ctx, eta=m["eta"], C6=_tensor7(m) if case["tensor"] else None,
                U=u.reshape(-1).contiguous(), out=torch.empty(8, 7, ctx.nel, dtype=F64, device="cuda"))


def _run_stress(s):
    ctx = s["ctx"]
    C6 = C.cast(_ptrs(s["C6"]), C.POINTER(C.c_void_p)) if s["C6"] else None
    ctx._chk(lib().dp_stress(ctx.h, s["U"].data_ptr(), s["eta"].data_ptr(), ctx.nel, C6, ctx.nel if C6 else 0,
                             s["out"].data_ptr(), DP_MEM_DEVICE))
    return s["out"]


def _prepare_viscosity(case, seed):
    ctx, _, r, _ = _mesh(case["nr"], case["nt"])
    g = _gen(seed)
    nv = (case["nr"] + 1) * case["nt"]
    return dict(case=case, ctx=ctx, T=1300 + 1200 * _rand(g, ctx.nnod), r=3.48e6 + (r - R_IN) * 2.87e6,
                P=2e9 * torch.randn(nv, generator=g, device="cuda", dtype=F64),
                eps=1e-15 * _rand(g, 7, ctx.nel), tau=4e9 * _rand(g, 7, ctx.nel),
                coh=30e6 * (_rand(g, 7, ctx.nel) >= 0.3).to(F64),
                eta=torch.full((7, ctx.nel), 3.3e21, dtype=F64, device="cuda"))


def _run_viscosity(s):
    ctx, law = s["ctx"], Arrhenius(*[ARRHENIUS[k] for k in ("eta0", "R", "Ea", "Va", "T0", "phi_deg")])
    ctx._chk(lib().dp_viscosity_arrhenius(ctx.h, C.byref(law), s["T"].data_ptr(), s["P"].data_ptr(), s["P"].numel(),
                                          s["r"].data_ptr(), s["eps"].data_ptr(), s["tau"].data_ptr(),
                                          s["coh"].data_ptr(), s["eta"].data_ptr(), DP_MEM_DEVICE))
    return s["eta"]


def _prepare_fabric(case, seed):
    ctx = _mesh(case["nr"], case["nt"])[0]
    g, n = _gen(seed), ctx.nel
    ang = math.pi * (2 * _rand(g, 6, n) - 1)
    s1, s2 = torch.exp(4 * _rand(g, 6, n)), torch.exp(-2 * _rand(g, 6, n))
    c, s = torch.cos(ang), torch.sin(ang)
    F = torch.stack([c * s1, s * s1, -s * s2, c * s2], 2).contiguous()   # F11, F21, F12, F22 of R diag(s1, s2)
    new = lambda k: torch.empty(k, n, dtype=F64, device="cuda")          # noqa: E731
    return dict(case=case, ctx=ctx, dem=_dem(), F=F, r1=-0.3 + 2.3 * _rand(g, 6, n), r2=-0.3 + 2.6 * _rand(g, 6, n),
                fse=[new(6) for _ in range(6)], C6=[new(7) for _ in range(6)])


def _run_fabric(s):
    ctx, n, L = s["ctx"], s["ctx"].nel, lib()
    ctx._chk(L.dp_fse(ctx.h, s["F"].data_ptr(), _ptrs(s["fse"]), n, DP_MEM_DEVICE))
    d = s["dem"].struct()
    ctx._chk(L.dp_anisotropic_tensor(ctx.h, C.byref(d), s["fse"][0].data_ptr(), s["fse"][2].data_ptr(),
                                     s["r1"].data_ptr(), s["r2"].data_ptr(), n, _ptrs(s["C6"]), n, DP_MEM_DEVICE))
    return s["fse"], s["C6"]


def _prepare_thermal(case, seed):
    ctx, th, r, _ = _mesh(case["nr"], case["nt"])
    g = _gen(seed)
    T = (4000 + (300 - 4000) * torch.log(r / R_IN) / math.log(R_OUT / R_IN)
         + 200 * torch.sin(3 * th + 2 * math.pi * float(_rand(g, 1))) * torch.sin(math.pi * (r - R_IN)))
    rho = 3300 * (1 + 0.05 * torch.randn(ctx.nnod, generator=g, device="cuda", dtype=F64))
    o = ThermalOpts()
    lib().dp_default_thermal_opts(C.byref(o))
    for k, v in dict(THERMAL, dt=3300 * 1.2e3 / 3.3 / case["nr"] ** 2, heated=int(case["heated"])).items():
        setattr(o, k, v)
    return dict(case=case, ctx=ctx, T=T.contiguous(), rho=rho, o=o)


def _run_thermal(s):
    ctx = s["ctx"]                                      # the next step starts from this one's T
    ctx._chk(lib().dp_thermal_step(ctx.h, C.byref(s["o"]), s["rho"].data_ptr(), s["T"].data_ptr(), None, None,
                                   DP_MEM_DEVICE))
    return s["T"]


def _net(nr, nt, batch):
    """The committed network (trained at 128x1024) on the mesh's own grid."""
    grid = learned.grid_shape(nr, nt)
    net = learned.GuessNet.load(learned.weights_path(128, 1024), max_batch=batch)
    return net if grid == (net.nrg, net.ntg) else net.for_grid(*grid, max_batch=batch)


def _prepare_guess(case, seed):
    ctx = _mesh(case["nr"], case["nt"])[0]
    return dict(case=case, ctx=ctx, m=_material(dict(case, material="aniso"), seed),
                guess=learned.LearnedGuess(_net(case["nr"], case["nt"], 1), ctx),
                P=torch.zeros(ctx.npres, dtype=F64, device="cuda"))


def _run_guess(s):
    _set_material(s["ctx"], s["m"])
    s["guess"].predict(s["m"]["g"], s["P"].data_ptr())
    return s["guess"].y, s["P"]


def _train_batch(case, seed):
    """Smooth normalised network inputs and targets, and initial weights."""
    nrg, ntg = learned.grid_shape(case["nr"], case["nt"])
    g, b = _gen(seed), case["batch"]
    r = torch.linspace(R_IN, R_OUT, nrg, dtype=F64, device="cuda")[:, None]
    th = torch.arange(ntg, dtype=F64, device="cuda")[None] * (2 * math.pi / ntg)
    field = lambda: _fourier(th.expand(nrg, -1), r.expand(-1, ntg), _rand(g, 8).tolist())   # noqa: E731
    x = torch.stack([torch.stack([field() for _ in range(4)]) for _ in range(b)]).float()
    t = torch.stack([field()[None] for _ in range(b)]).float()
    chans = [4] + [ARCH["channels"]] * (ARCH["layers"] - 1) + [1]
    parts = []
    for ci, co in zip(chans, chans[1:]):
        lim = math.sqrt(6.0 / (ci * 9)) * (0.1 if co == 1 else 1.0)
        parts += [lim * (2 * _rand(g, co * ci * 9) - 1), 0.01 * _rand(g, co)]
    return (x + 0.05 * torch.randn(x.shape, generator=g, device="cuda")).contiguous(), t.contiguous(), \
        torch.cat(parts).float()


def _prepare_train(case, seed):
    x, t, p = _train_batch(case, seed)
    net = learned.GuessNet(*learned.grid_shape(case["nr"], case["nt"]), max_batch=case["batch"], **ARCH)
    net.set_params(p.cpu().numpy())
    return dict(case=case, net=net, x=x, t=t)


def _run_train(s):
    loss = s["net"].train_step(s["x"], s["t"], 2e-3)
    return (loss,) + s["net"].get_params(grads=True)


# ---- least work -------------------------------------------------------------------------
def work(case):
    """Inputs read once and outputs written once; for a solve also the vectors of the
    outer iterations (5 pressure and 2 velocity vectors each) and the element blocks'
    multiply-adds, for the network its convolutions."""
    nr, nt, kind = case["nr"], case["nt"], case["kind"]
    nel, nn = 2 * nr * nt, (2 * nr + 1) * 2 * nt
    nv = (nr + 1) * nt
    npres = 3 * nel if case.get("pressure", "discontinuous") == "discontinuous" else nv
    if kind == "solve":
        its = case["outer"] or (60 if case["pressure"] == "continuous" else 900)
        return dict(bytes=8.0 * (9 * nel + nn + its * (5 * npres + 2 * 2 * nn)), flops=its * 2.0 * 144 * nel)
    if kind == "operator":
        return dict(bytes=8.0 * ((6 + 36) * nel + nn + 3 * 2 * nn + 2 * npres), flops=6.0 * 700 * nel)
    if kind == "stress":
        return dict(bytes=8.0 * (nel * (7 + 56 + (42 if case["tensor"] else 0)) + 2 * nn), flops=7.0 * 110 * nel)
    if kind == "viscosity":
        return dict(bytes=8.0 * (nel * 35 + 2 * nn + nv), flops=7.0 * 80 * nel)
    if kind == "fabric":
        return dict(bytes=8.0 * nel * (24 + 36 + 12 + 42), flops=6.0 * 200 * nel)
    if kind == "thermal":
        return dict(bytes=8.0 * 3 * nn, flops=7.0 * 300 * nel + 50 * 2.0 * 36 * nel)
    grid = (nr // 2 + 1) * (nt // 2)
    macs = 9.0 * grid * (4 * 32 + 4 * 32 * 32 + 32)
    if kind == "guess":
        return dict(bytes=8.0 * (9 * nel + nn + npres), flops=2 * macs)
    return dict(bytes=4.0 * case["batch"] * 5 * grid, flops=2 * macs * 3 * case["batch"])


# ---- 64-bit values -------------------------------------------------------------------------
def _geometry(nr, nt):
    """Lattice nodes of the elements (6, nel), reference number of each lattice node,
    seam-free vertex angles and radii (3, nel), node angles."""
    dev = "cuda"
    A, B = 2 * nr + 1, 2 * nt
    q = torch.arange(nr * nt, device=dev)
    a0, b0 = 2 * (q % nr), 2 * torch.div(q, nr, rounding_mode="floor")
    off = (((0, 0), (0, 2), (2, 0), (0, 1), (1, 1), (1, 0)), ((0, 2), (2, 2), (2, 0), (1, 2), (2, 1), (1, 1)))
    la = torch.stack([torch.stack([a0 + off[t][k][0] for t in (0, 1)], 1).reshape(-1) for k in range(6)])
    lb = torch.stack([torch.stack([b0 + off[t][k][1] for t in (0, 1)], 1).reshape(-1) for k in range(6)])
    lat = la + A * (lb % B)
    ref = torch.empty(A * B, dtype=torch.int64, device=dev)
    ref[lat[:3]] = torch.div(la[:3], 2, rounding_mode="floor") + (nr + 1) * torch.div(lb[:3] % B, 2, rounding_mode="floor")
    mid = lat[3:].T.reshape(-1)                        # midpoints in first-seen order
    uniq, inv = torch.unique(mid, return_inverse=True)
    first = torch.full((uniq.numel(),), mid.numel(), device=dev).scatter_reduce(
        0, inv, torch.arange(mid.numel(), device=dev), "amin")
    ref[uniq[torch.argsort(first)]] = (nr + 1) * nt + torch.arange(uniq.numel(), device=dev)
    th = lb[:3].to(F64) * (math.pi / nt)
    rr = R_IN + (R_OUT - R_IN) * la[:3].to(F64) / (2 * nr)
    n = torch.arange(A * B, device=dev)
    return lat, ref, th, rr, torch.div(n, A, rounding_mode="floor").to(F64) * (math.pi / nt), n % A


def _derivatives(th, rr, p):
    """dN/dx, dN/dz (6, nel) and r det J at the point p of every element."""
    n3, dn = _n3(p), _dn6(p)
    t_ip, r_ip = n3 @ th, n3 @ rr
    T21, T31, R21, R31 = th[1] - th[0], th[2] - th[0], rr[1] - rr[0], rr[2] - rr[0]
    det = T21 * R31 - T31 * R21
    s, c = torch.sin(t_ip), torch.cos(t_ip)
    dx = (dn[0][:, None] * (R31 * c / r_ip - T31 * s) + dn[1][:, None] * (-R21 * c / r_ip + T21 * s)) / det
    dz = (dn[0][:, None] * (-R31 * s / r_ip - T31 * c) + dn[1][:, None] * (R21 * s / r_ip + T21 * c)) / det
    return dx, dz, r_ip * det, t_ip


class _Stokes:
    """The Stokes operators of a mesh and a material, polar DOFs in the reference
    numbering (u_theta, u_r per node), free slip and one tangential pin."""

    def __init__(self, case, m, C6):
        nr, nt = case["nr"], case["nt"]
        self.lat, ref, self.th, self.rr, ang, a = _geometry(nr, nt)
        self.e = ref[self.lat]
        self.nn, self.nel = ref.numel(), self.lat.shape[1]
        self.ang = torch.empty_like(ang)
        self.ang[ref] = ang
        rad = torch.empty_like(a)
        rad[ref] = a
        self.r = R_IN + (R_OUT - R_IN) * rad.to(F64) / (2 * nr)
        free = torch.ones(self.nn, 2, dtype=F64, device="cuda")
        free[:, 1] = ((rad != 0) & (rad != 2 * nr)).to(F64)
        free[ref[2 * nr], 0] = 0.0
        self.free = free
        self.cont = case["pressure"] == "continuous"
        self.pd = self.e[:3] if self.cont else torch.arange(3 * self.nel, device="cuda").reshape(-1, 3).T
        self.np_ = int(self.pd.max()) + 1
        self.m, self.C6 = m, C6

    def _d(self, ip):
        v = self.m["eta"][ip]
        c = [4 / 3, 4 / 3, 1.0, -2 / 3, 0.0, 0.0] if self.C6 is None else [f[ip] for f in self.C6]
        return [x * v for x in c]                       # D11, D22, D33, D12, D13, D23

    def to_cart(self, u):
        u = u.reshape(-1, 2)
        c, s = torch.cos(self.ang), torch.sin(self.ang)
        return torch.stack([c * u[:, 0] + s * u[:, 1], c * u[:, 1] - s * u[:, 0]], 1)

    def from_elements(self, fx, fz):
        f = torch.zeros(self.nn, 2, dtype=F64, device="cuda")
        f.index_add_(0, self.e.reshape(-1), torch.stack([fx.reshape(-1), fz.reshape(-1)], 1))
        c, s = torch.cos(self.ang), torch.sin(self.ang)
        return (torch.stack([c * f[:, 0] - s * f[:, 1], s * f[:, 0] + c * f[:, 1]], 1) * self.free).reshape(-1)

    def K(self, u):
        uc = self.to_cart((u.reshape(-1, 2) * self.free).reshape(-1))
        ux, uz = uc[:, 0][self.e], uc[:, 1][self.e]
        fx, fz = torch.zeros_like(ux), torch.zeros_like(uz)
        for ip, (p, w) in enumerate(zip(*_ips6())):
            dx, dz, om, _ = _derivatives(self.th, self.rr, p)
            exx, ezz, gxz = (dx * ux).sum(0), (dz * uz).sum(0), (dz * ux + dx * uz).sum(0)
            d11, d22, d33, d12, d13, d23 = self._d(ip)
            sxx = (d11 * exx + d12 * ezz + d13 * gxz) * om * w
            szz = (d12 * exx + d22 * ezz + d23 * gxz) * om * w
            sxz = (d13 * exx + d23 * ezz + d33 * gxz) * om * w
            fx += dx * sxx + dz * sxz
            fz += dz * szz + dx * sxz
        return self.from_elements(fx, fz)

    def G(self, p):
        pe = p[self.pd]
        fx = torch.zeros(6, self.nel, dtype=F64, device="cuda")
        fz = torch.zeros_like(fx)
        for q, w in zip(*_ips6()):
            dx, dz, om, _ = _derivatives(self.th, self.rr, q)
            t = (_n3(q) @ pe) * om * w
            fx += dx * t
            fz += dz * t
        return self.from_elements(fx, fz)

    def GT(self, u):
        uc = self.to_cart((u.reshape(-1, 2) * self.free).reshape(-1))
        out = torch.zeros(self.np_, dtype=F64, device="cuda")
        for q, w in zip(*_ips6()):
            dx, dz, om, _ = _derivatives(self.th, self.rr, q)
            div = (dx * uc[:, 0][self.e] + dz * uc[:, 1][self.e]).sum(0) * om * w
            out.index_add_(0, self.pd.reshape(-1), (_n3(q)[:, None] * div).reshape(-1))
        return out

    def F(self):
        fx = torch.zeros(6, self.nel, dtype=F64, device="cuda")
        fz = torch.zeros_like(fx)
        for q, w in zip(*_ips6()):
            _, _, om, t = _derivatives(self.th, self.rr, q)
            b = _n6(q)[:, None] * ((_n3(q) @ self.m["rho"][self.e[:3]]) * self.m["g"] * om * w)
            fx += torch.sin(t) * b
            fz += torch.cos(t) * b
        return self.from_elements(fx, fz)

    def rotation(self, u):
        """The rigid angular velocity: int rho u_theta / int rho r."""
        num = den = 0.0
        ut, rho = u.reshape(-1, 2)[:, 0], self.m["rho"]
        for q, w in zip(*_ips6()):
            _, _, om, _ = _derivatives(self.th, self.rr, q)
            num = num + ((_n6(q) @ (ut * rho)[self.e]) * om * w).sum()
            den = den + ((_n6(q) @ (self.r * rho)[self.e]) * om * w).sum()
        return num / den


def _exact_operator(case, seed):
    s = _prepare_operator(case, seed)
    o = _Stokes(case, s["m"], s["C6"])
    return o.K(s["u"]), o.G(s["p"]), o.GT(s["u"])


def _exact_solve(case, seed):
    """Dense elimination of the velocity and of the Schur complement (small meshes,
    solves to convergence)."""
    nel, nn = 2 * case["nr"] * case["nt"], (2 * case["nr"] + 1) * 2 * case["nt"]
    if case["outer"] or nn > 9000 or (case["pressure"] == "discontinuous" and nel > 4200):
        return None
    m = _material(case, seed)
    o = _Stokes(case, m, [c.expand(7, -1) for c in _rotated(m["delta"], m["dx"], m["dy"])] if "delta" in m else None)
    idx = torch.nonzero(o.free.reshape(-1)).reshape(-1)
    place = torch.full((2 * o.nn,), -1, device="cuda")
    place[idx] = torch.arange(idx.numel(), device="cuda")
    # element matrices by applying the element operator to unit vectors
    c, s = torch.cos(o.ang)[o.e], torch.sin(o.ang)[o.e]                            # (6, nel)
    Ke = torch.zeros(o.nel, 12, 12, dtype=F64, device="cuda")
    Ge = torch.zeros(o.nel, 12, 3, dtype=F64, device="cuda")
    for ip, (p, w) in enumerate(zip(*_ips6())):
        dx, dz, om, _ = _derivatives(o.th, o.rr, p)
        Bt = torch.zeros(o.nel, 12, 3, dtype=F64, device="cuda")                    # polar B^T
        bx = torch.stack([dx, 0 * dx, dz], -1)                                      # (6, nel, 3)
        bz = torch.stack([0 * dx, dz, dx], -1)
        Bt[:, 0::2] = (c[..., None] * bx - s[..., None] * bz).transpose(0, 1)
        Bt[:, 1::2] = (s[..., None] * bx + c[..., None] * bz).transpose(0, 1)
        d11, d22, d33, d12, d13, d23 = [torch.as_tensor(v, device="cuda") * om * w for v in o._d(ip)]
        D = torch.stack([torch.stack([d11, d12, d13], -1), torch.stack([d12, d22, d23], -1),
                         torch.stack([d13, d23, d33], -1)], -2)
        Ke += Bt @ D @ Bt.transpose(1, 2)
        div = Bt[:, :, 0] + Bt[:, :, 1]
        Ge += div[:, :, None] * (_n3(p)[None, :] * (om * w)[:, None])[:, None, :]
    dof = torch.stack([2 * o.e, 2 * o.e + 1], 1).reshape(12, -1).T                  # (nel, 12)
    row = place[dof]
    n = idx.numel()
    K = torch.zeros(n * n, dtype=F64, device="cuda")
    ok = (row[:, :, None] >= 0) & (row[:, None, :] >= 0)
    K.index_add_(0, (row[:, :, None] * n + row[:, None, :])[ok], Ke[ok])
    G = torch.zeros(n * o.np_, dtype=F64, device="cuda")
    pd = o.pd.T
    okg = (row[:, :, None] >= 0).expand(-1, -1, 3)
    G.index_add_(0, (row[:, :, None] * o.np_ + pd[:, None, :])[okg], Ge[okg])
    K, G, F = K.view(n, n), G.view(n, o.np_), o.F()[idx]
    chol = torch.linalg.cholesky(K)
    KiG = torch.cholesky_solve(G, chol)
    KiF = torch.cholesky_solve(F[:, None], chol)[:, 0]
    S = G.T @ KiG
    S += S.diagonal().mean() / o.np_                       # the constant pressure
    P = torch.linalg.solve(S, -(G.T @ KiF))
    P = P - P.mean()
    U = torch.zeros(2 * o.nn, dtype=F64, device="cuda")
    U[idx] = KiF + KiG @ P
    om = o.rotation(U)
    U.view(-1, 2)[:, 0] -= om * o.r
    return U, P


def _exact_stress(case, seed):
    s = _prepare_stress(case, seed)
    lat, ref, th, rr, _, _ = _geometry(case["nr"], case["nt"])
    u = s["U"].reshape(-1, 2)[ref[lat]]
    out = torch.empty_like(s["out"])
    for ip, p in enumerate(_ips7()[0]):
        dx, dz, _, _ = _derivatives(th, rr, p)
        exx, ezz = (dx * u[..., 0]).sum(0), (dz * u[..., 1]).sum(0)
        exz = 0.5 * (dz * u[..., 0] + dx * u[..., 1]).sum(0)
        et = s["eta"][ip]
        if s["C6"]:
            c11, c33, c55, c13, c15, c35 = [f[ip] * et for f in s["C6"]]
            a, b = -exx / 3 + 2 * ezz / 3, 2 * exx / 3 - ezz / 3
            t = (c13 * a + c11 * b + c15 * exz, c33 * a + c13 * b + 2 * c35 * exz, c35 * a + c15 * b + c55 * exz)
        else:
            t = (et * (4 * exx - 2 * ezz) / 3, et * (4 * ezz - 2 * exx) / 3, 2 * et * exz)
        second = lambda x, z, y: torch.sqrt(0.5 * (x * x + z * z) + y * y)   # noqa: E731
        for k, v in enumerate((exx, ezz, exz, second(exx, ezz, exz), *t, second(*t))):
            out[k, ip] = v
    return out


def _exact_viscosity(case, seed):
    s, law = _prepare_viscosity(case, seed), ARRHENIUS
    lat, ref, _, _, _, _ = _geometry(case["nr"], case["nt"])
    e = ref[lat]
    out = s["eta"].clone()
    phi = math.radians(law["phi_deg"])
    for ip, p in enumerate(_ips7()[0]):
        T, z = _n6(p) @ s["T"][e], _n6(p) @ s["r"][e]
        P = _n3(p) @ s["P"][e[:3]] + s["P"].min().abs()
        depth = s["r"].max() - z
        lam = torch.full_like(z, 10.0)
        lam[depth > 2780e3], lam[depth < 660e3] = 1e-3, 1.0
        eta = (lam * law["eta0"] * torch.exp((law["Ea"] + P * law["Va"]) / law["R"] / T
                                             - law["Ea"] / law["R"] / law["T0"])).clamp(1e18, 1e25)
        plastic = (s["coh"][ip] > 0) & (s["eps"][ip] != 0)
        ty = math.cos(phi) * s["coh"][ip] + math.sin(phi) * P
        weak = (0.5 * ty / s["eps"][ip]).clamp(1e18, 1e25)
        out[ip] = torch.where(plastic, torch.where(ty < s["tau"][ip], weak, out[ip]), eta)
    return out


def _exact_fabric(case, seed):
    s = _prepare_fabric(case, seed)
    F, d = s["F"], s["dem"]
    vx, vy, a1, a2 = _axes(F[..., 0], F[..., 1], F[..., 2], F[..., 3])

    def nearest(v, b):                                   # the first i with |v - b_i| < |v - b_i+1|
        dist = (v[..., None] - torch.from_numpy(b).cuda()).abs()
        up = torch.cat([dist[..., :-1] < dist[..., 1:], torch.ones_like(dist[..., :1], dtype=torch.bool)], -1)
        return up.to(torch.int8).argmax(-1)

    perm = torch.from_numpy(d.permutation_blk).cuda()
    row = d.sblk * nearest(s["r1"], d.a1a2_blk) + perm[nearest(s["r2"], d.a2a3_blk)] - 1
    tab = torch.from_numpy(np.ascontiguousarray(d.C)).cuda()
    n = list(_rotate(vx, vy, tab[row, 0], tab[row, 2], tab[row, 4].clamp_min(d.w), tab[row, 7]))
    n[2] = n[2].clamp_min(d.w)
    return [vx, -vy, vy, vx, a1, a2], [torch.cat([c, c.mean(0, keepdim=True)]) for c in n]


def _exact_thermal(case, seed):
    s = _prepare_thermal(case, seed)
    lat, ref, th, rr, _, a = _geometry(case["nr"], case["nt"])
    e, nn, dt = ref[lat], ref.numel(), s["o"].dt
    Ke = torch.zeros(lat.shape[1], 6, 6, dtype=F64, device="cuda")
    Me = torch.zeros_like(Ke)
    for p, w in zip(*_ips7()):
        dx, dz, om, _ = _derivatives(th, rr, p)
        Ke += torch.einsum("ie,je,e->eij", dx, dx, om * w * THERMAL["K"])
        Ke += torch.einsum("ie,je,e->eij", dz, dz, om * w * THERMAL["K"])
        N = _n6(p)
        Me += torch.outer(N, N)[None] * ((_n3(p) @ s["rho"][e[:3]]) * om * w * THERMAL["Cp"])[:, None, None]
    Ae = Me + dt * Ke
    rad = torch.empty_like(a)
    rad[ref] = a
    fixed = rad == 2 * case["nr"]
    Tbc = torch.where(fixed, THERMAL["Ttop"], 0.0).to(F64)
    if case["heated"]:
        fixed, Tbc = fixed | (rad == 0), torch.where(rad == 0, THERMAL["Tbot"], Tbc)
    free = (~fixed).to(F64)

    def mul(M, x):
        out = torch.zeros(nn, dtype=F64, device="cuda")
        return out.index_add_(0, e.reshape(-1), (M @ x[e].T[:, :, None])[:, :, 0].T.reshape(-1))

    b = (mul(Me, s["T"]) - mul(Ae, Tbc)) * free
    dg = torch.zeros(nn, dtype=F64, device="cuda")
    dg.index_add_(0, e.reshape(-1), torch.diagonal(Ae, dim1=1, dim2=2).T.reshape(-1))
    x = torch.zeros_like(b)
    r = b.clone()
    z = r / dg
    p, rz, stop = z.clone(), r @ z, 1e-14 * float(b.norm())
    for _ in range(2000):
        q = mul(Ae, p) * free
        al = rz / (p @ q)
        x += al * p
        r -= al * q
        if float(r.norm()) < stop:
            break
        z = r / dg
        new = r @ z
        p, rz = z + (new / rz) * p, new
    return x + Tbc


def _network(x, params, grid):
    """The network in 64 bits on (batch, 4, nrg, ntg); params a flat tensor."""
    chans = [4] + [ARCH["channels"]] * (ARCH["layers"] - 1) + [1]
    off = 0
    for layer, (ci, co) in enumerate(zip(chans, chans[1:])):
        w = params[off:off + co * ci * 9].view(co, ci, 3, 3)
        bias = params[off + co * ci * 9:off + co * ci * 9 + co]
        off += co * ci * 9 + co
        d = ARCH["dilations"][layer]
        xp = torch.nn.functional.pad(x[..., torch.arange(-d, grid[1] + d, device="cuda") % grid[1]], (0, 0, d, d))
        # nine shifted products (no 64-bit convolution library needed)
        y = bias.view(1, -1, 1, 1)
        for i in range(3):
            for j in range(3):
                y = y + torch.einsum("oc,bcij->boij", w[:, :, i, j],
                                     xp[:, :, i * d:i * d + grid[0], j * d:j * d + grid[1]])
        x = torch.relu(y) if layer < ARCH["layers"] - 1 else y
    return x


def _exact_guess(case, seed):
    s = _prepare_guess(case, seed)
    net, m, nr, nt = s["guess"].net, s["m"], case["nr"], case["nt"]
    nrg, ntg = learned.grid_shape(nr, nt)
    i, j = torch.arange(nrg, device="cuda")[:, None], torch.arange(ntg, device="cuda")[None]
    e = 2 * ((2 * i).clamp_max(nr - 1) + nr * 2 * j)
    x = torch.stack([m["rho"][2 * i + (nr + 1) * 2 * j], torch.log10(m["eta"][:6])[:, e].mean(0),
                     m["dx"][e] ** 2 - m["dy"][e] ** 2, 2 * m["dx"][e] * m["dy"][e]])[None]
    mean, std = (torch.from_numpy(np.asarray(v, dtype=np.float64)).cuda().view(1, 4, 1, 1) for v in (net.x_mean, net.x_std))
    y = _network((x - mean) / std, torch.from_numpy(net.get_params()).cuda().double(), (nrg, ntg))
    y = y * net.y_std + net.y_mean
    # bilinear prolongation to the vertices, then to the elements' three pressure DOFs
    g = y[0, 0]
    v = torch.empty(nr + 1, nt, dtype=F64, device="cuda")
    v[::2, ::2] = g
    v[1::2, ::2] = 0.5 * (g[:-1] + g[1:])
    v[:, 1::2] = 0.5 * (v[:, ::2] + v[:, ::2].roll(-1, 1))
    ref_vertex = v.T.reshape(-1) * m["g"]
    lat, ref, _, _, _, _ = _geometry(nr, nt)
    return y, ref_vertex[ref[lat[:3]]].T.reshape(-1)


def _exact_train(case, seed):
    x, t, p = _train_batch(case, seed)
    p = p.double().requires_grad_()
    y = _network(x.double(), p, learned.grid_shape(case["nr"], case["nt"]))
    loss = ((y - t.double()) ** 2).mean()
    loss.backward()
    g = p.grad
    step = 2e-3 * g / (g.abs() + 1e-8)                    # Adam's first step
    return float(loss), (p.detach() - step).float().cpu().numpy().astype(np.float64), g.cpu().numpy()
