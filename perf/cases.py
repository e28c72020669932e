"""What this framework is used for, as cases that can be timed and compared.

Kinds of case (`kind`), each through a public entry point:

  step       one time step of a flow: `compute` and `timestep` from `simulation.setup`
             (wall-bounded cavity, channel with inflow and outlet, periodic vortex; quad4, quad9,
             hex8; FP64 or mixed precision; every pressure preconditioner)
  transport  the same with a passive scalar carried along (SUPG or plain)
  poisson    one pressure-Poisson solve (`fem_pressure_solve`, `fem_pressure_solve_mixed`)
  operator   one element-by-element product (`core.element_mult`)
  inverse    loss and adjoint gradient of a short flow-and-scalar rollout
  serve      a batch of independent requests through `serving.PackedServer` / `serving.Server`

`exact` restates all of it in plain torch in 64 bits: unassembled element products by gather and
index_add, Krylov solves to rounding level, cosine transforms for the Poisson solves.
"""
import ctypes
import math

import numpy as np
import torch

F64 = torch.float64
PI = math.pi


def listed():
    return [
        # the lid-driven cavity everyone starts with; the smallest step, bound by latency
        dict(name="cavity_64_q1", kind="step", flow="cavity", order=1, nx=64, ny=64, base=4, precond="multigrid",
             precision="fp64", nu=0.01, dt=0.01, tol=1e-8),
        # the Taylor-Green validation run, 256 x 256 quad9, periodic: the headline workload
        dict(name="vortex_256_q2", kind="step", flow="vortex", order=2, nx=256, ny=256, base=4, precond="multigrid",
             precision="fp64", nu=0.01, dt=1e-3, tol=1e-8),
        # the same in mixed precision, as a user who wants speed runs it
        dict(name="vortex_256_q2_mixed", kind="step", flow="vortex", order=2, nx=256, ny=256, base=4,
             precond="multigrid", precision="mixed", nu=0.01, dt=1e-3, tol=1e-8),
        # 2D channel with inflow and outlet, a ragged oblong mesh, the series preconditioner
        dict(name="channel_90x33_q2_series", kind="step", flow="channel", order=2, nx=90, ny=33, base=0,
             precond="approx_inv", precision="fp64", nu=0.005, dt=2e-3, tol=1e-8),
        # the 3D channel production run, 1.09 million nodes
        dict(name="channel3d_256x64x64", kind="step", flow="channel3d", order=1, nx=256, ny=64, nz=64, base=8,
             precond="multigrid", precision="fp64", nu=0.005, dt=2e-3, tol=1e-8),
        # a small odd-sized 3D box with the Jacobi preconditioner
        dict(name="channel3d_50x21x19_jacobi", kind="step", flow="channel3d", order=1, nx=50, ny=21, nz=19, base=0,
             precond="jacobi", precision="fp64", nu=0.01, dt=5e-3, tol=1e-8),
        # a scalar in a recirculating flow
        dict(name="scalar_128_q1", kind="transport", order=1, n=128, base=4, supg=True, nu=1e-3, D=1e-4, dt=0.01,
             tol=1e-8),
        # Poisson solves of an ordinary and of the largest size
        dict(name="poisson_1024", kind="poisson", n=1024, base=4, tol=1e-8, precision="fp64"),
        dict(name="poisson_4096", kind="poisson", n=4096, base=4, tol=1e-8, precision="fp64"),
        # one matrix-free Laplacian product beyond the caches, the building block of users' own solvers
        dict(name="laplacian_4096_q1", kind="operator", op="laplacian", order=1, nx=4096, ny=4096),
        # gradient of an inverse problem with respect to the initial velocity
        dict(name="inverse_128", kind="inverse", n=128, steps=2, nu=1e-3, D=1e-4, dt=0.01, supg=True),
        # twelve users' small problems at once
        dict(name="serve_12", kind="serve", server="packed", count=12, steps=10, most=128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _tol(rng):
    return float("%.2g" % 10.0 ** rng.uniform(-9, -7))


def _mg_size(rng, lo, hi):
    """(n, base): n = base * 2^k near a size drawn over the logarithm of the range."""
    n = _log_int(rng, lo, hi)
    base = rng.choice([4, 5, 6, 7, 9])
    k = max(0, int(round(math.log2(max(1.0, n / base)))))
    while base << k > hi:
        k -= 1
    return base << max(k, 1), base


def draw(rng):
    kind = rng.choice(["step", "step", "step", "transport", "poisson", "poisson", "operator", "inverse", "serve"])
    if kind == "step":
        flow = rng.choice(["cavity", "vortex", "channel", "channel3d"])
        nu, dt = 10.0 ** rng.uniform(-3, -1), 10.0 ** rng.uniform(-3, -2)
        if flow == "channel3d":
            if rng.random() < 0.5:
                base, k = rng.randint(4, 8), rng.randint(1, 3)
                while (4 * (base << k) + 1) * ((base << k) + 1) ** 2 > 1.1e6:
                    base -= 1
                m = base << k
                return dict(kind=kind, flow=flow, order=1, nx=4 * m, ny=m, nz=m, base=base, precond="multigrid",
                            precision=rng.choice(["fp64", "fp64", "mixed"]), nu=nu, dt=dt, tol=_tol(rng))
            return dict(kind=kind, flow=flow, order=1, nx=rng.randint(20, 70), ny=rng.randint(9, 30),
                        nz=rng.randint(9, 30), base=0, precond=rng.choice(["jacobi", "approx_inv"]),
                        precision="fp64", nu=nu, dt=dt, tol=_tol(rng))
        order = rng.choice([1, 2])
        if rng.random() < 0.75:
            n, base = _mg_size(rng, 16, 512 if order == 1 else 256)
            aspect = rng.choice([1, 1, 2]) if flow == "channel" and n <= 256 // order else 1
            return dict(kind=kind, flow=flow, order=order, nx=aspect * n, ny=n, base=base, precond="multigrid",
                        precision=rng.choice(["fp64", "fp64", "fp64", "mixed"]), nu=nu, dt=dt, tol=_tol(rng))
        return dict(kind=kind, flow=flow, order=order, nx=_log_int(rng, 12, 100), ny=_log_int(rng, 12, 100), base=0,
                    precond=rng.choice(["jacobi", "approx_inv"]), precision="fp64", nu=nu, dt=dt, tol=_tol(rng))
    if kind == "transport":
        n, base = _mg_size(rng, 24, 256)
        return dict(kind=kind, order=rng.choice([1, 1, 2]) if n <= 128 else 1, n=n, base=base,
                    supg=rng.random() < 0.6, nu=10.0 ** rng.uniform(-3, -1), D=10.0 ** rng.uniform(-4, -2),
                    dt=10.0 ** rng.uniform(-3, -2), tol=_tol(rng))
    if kind == "poisson":
        n, base = _mg_size(rng, 16, 4096)
        return dict(kind=kind, n=n, base=base, tol=_tol(rng),
                    precision="mixed" if 512 <= n <= 2048 and rng.random() < 0.3 else "fp64")
    if kind == "operator":
        op, order = rng.choice(["laplacian", "mass", "visc_conv"]), rng.choice([1, 2])
        hi = (512 if op == "visc_conv" else 4096) // order
        return dict(kind=kind, op=op, order=order, nx=_log_int(rng, 15, hi), ny=_log_int(rng, 15, hi))
    if kind == "inverse":
        return dict(kind=kind, n=rng.choice([16, 32, 64, 128]), steps=rng.randint(1, 3), nu=10.0 ** rng.uniform(-3, -2),
                    D=10.0 ** rng.uniform(-4, -3), dt=10.0 ** rng.uniform(-2.5, -2), supg=rng.random() < 0.7)
    return dict(kind=kind, server=rng.choice(["packed", "stream"]), count=rng.randint(4, 12),
                steps=2 * rng.randint(3, 5), most=rng.choice([64, 128]))


# ---------------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------------
def _axis(n_elem, order, length, periodic):
    n = order * n_elem + (0 if periodic else 1)
    return torch.arange(n, dtype=F64, device="cuda") * (length / (order * n_elem))


def _coeffs(seed, count, salt=0):
    g = torch.Generator().manual_seed(1000 * int(seed) + salt)
    return torch.randn(count, generator=g, dtype=F64).tolist()


def _wall(k, x):
    """sin(k pi x) sin(pi x) and its derivative: both vanish at 0 and 1."""
    s, c = torch.sin(k * PI * x), torch.cos(k * PI * x)
    return s * torch.sin(PI * x), PI * (k * c * torch.sin(PI * x) + s * torch.cos(PI * x))


def _eddies(seed, X, Y, modes=4):
    """Divergence-free (u, v), zero on the walls of the unit square, |u| of about 1."""
    u, v = torch.zeros_like(X), torch.zeros_like(X)
    a = iter(_coeffs(seed, modes * modes))
    for k in range(1, modes + 1):
        sx, dx = _wall(k, X)
        for m in range(1, modes + 1):
            sy, dy = _wall(m, Y)
            w = next(a) / (k * k + m * m) / PI
            u, v = u + w * sx * dy, v - w * dx * sy
    s = torch.sqrt(u * u + v * v).max()
    return u / s, v / s


def _bumps(seed, X, Y, modes=3):
    p = torch.zeros_like(X)
    a = iter(_coeffs(seed, modes * modes, 7))
    for k in range(1, modes + 1):
        for m in range(1, modes + 1):
            p = p + next(a) / (k * k + m * m) * torch.cos(k * PI * X) * torch.cos(m * PI * Y)
    return p


def _box(c):
    if c["flow"] == "vortex":
        return (2 * PI, 2 * PI)
    if c["flow"] == "channel3d":
        return (4.0, 1.0, 1.0)
    return (c["nx"] / c["ny"], 1.0)


def _flow_inputs(c, seed):
    """(U, P, rule) at the nodes (x fastest); rule(face axis values) is the inflow or lid."""
    L = _box(c)
    per = c["flow"] == "vortex"
    x, y = _axis(c["nx"], c["order"], L[0], per), _axis(c["ny"], c["order"], L[1], per)
    if c["flow"] == "channel3d":
        z = _axis(c["nz"], 1, L[2], False)
        Z, Y, X = torch.meshgrid(z, y, x, indexing="ij")
        u, v = _eddies(seed, X / L[0], Y)
        q = torch.sin(PI * Z) ** 2
        u = 16 * Y * (1 - Y) * Z * (1 - Z) + 0.3 * L[0] * u * q
        v = 0.3 * v * q
        P = (1 - X / L[0]) * (0.1 + 0.05 * _bumps(seed, X / L[0], Y) * torch.cos(PI * Z))
        return torch.cat([u.reshape(-1), v.reshape(-1), torch.zeros_like(u).reshape(-1)]), P.reshape(-1)
    Y, X = torch.meshgrid(y, x, indexing="ij")
    if per:  # the Taylor-Green vortex, of any strength and place
        a = _coeffs(seed, 3)
        s, X, Y = 1.0 + 0.2 * math.tanh(a[0]), X + a[1], Y + a[2]
        u, v = s * torch.sin(X) * torch.cos(Y), -s * torch.cos(X) * torch.sin(Y)
        P = 0.25 * s * s * (torch.cos(2 * X) + torch.cos(2 * Y))
        P = P - P.mean()
    elif c["flow"] == "cavity":
        u, v = _eddies(seed, X / L[0], Y / L[1])
        v = v * (L[1] / L[0])
        P = 0.1 * _bumps(seed, X / L[0], Y / L[1])
        P = P - P[0, 0]
        u = u.clone()
        u[-1, :] = 1.0
    else:
        u, v = _eddies(seed, X / L[0], Y / L[1])
        u, v = 4 * Y * (1 - Y) + 0.3 * L[0] * u, 0.3 * v
        P = (1 - X / L[0]) * (0.1 + 0.05 * _bumps(seed, X / L[0], Y))
    return torch.cat([u.reshape(-1), v.reshape(-1)]), P.reshape(-1)


def _faces(c):
    """(Dirichlet faces, outlet faces)."""
    return {"vortex": ([], []), "cavity": ([0, 1, 2, 3], []), "channel": ([0, 2, 3], [1]),
            "channel3d": ([0, 2, 3, 4, 5], [1])}[c["flow"]]


def _ns_config(sim, c):
    d, o = _faces(c)
    f = None
    if c["precond"] == "multigrid":
        k = c["ny"] // c["base"]
        f = [n // k for n in ([c["nx"], c["ny"], c["nz"]] if c["flow"] == "channel3d" else [c["nx"], c["ny"]])]
    return sim.StandardSolverConfig(dirichlet_faces=d, symmetry_faces=[], outlet_faces=o, streamline_diff=False,
                                    solver_tol=c["tol"], set_zeroP=c["flow"] != "vortex", pressure_precond=c["precond"],
                                    final_multigrid_mesh=f, precision=c["precision"])


def _mesh_config(sim, c):
    n = [c["nx"], c["ny"], c["nz"]] if c["flow"] == "channel3d" else [c["nx"], c["ny"]]
    return sim.SimpleMeshConfig(num_elem=n, domain_size=list(_box(c)), shape_func_ord=c["order"],
                                periodic=c["flow"] == "vortex")


def _drive(sim, c, coords, sn, gd, nn, Ud):
    """The moving lid or the inflow profile on the Dirichlet values."""
    if c["flow"] == "cavity":
        return sim.set_face_velocity(Ud, sn[2], gd, 1.0, nn, var=1)
    if c["flow"] == "channel":
        y = coords[sn[3], 1]
        return sim.set_face_velocity(Ud, sn[3], gd, 4 * y * (1 - y), nn, var=1)
    if c["flow"] == "channel3d":
        y, z = coords[sn[3], 1], coords[sn[3], 2]
        return sim.set_face_velocity(Ud, sn[3], gd, 16 * y * (1 - y) * z * (1 - z), nn, var=1)
    return Ud


def _scalar_flow(c):
    return dict(kind="step", flow="cavity", order=c.get("order", 1), nx=c["n"], ny=c["n"], base=c.get("base", 4),
                precond="multigrid", precision="fp64", nu=c["nu"], dt=c["dt"], tol=c.get("tol", 1e-8))


def _scalar_start(c, seed):
    x = _axis(c["n"], c.get("order", 1), 1.0, False)
    Y, X = torch.meshgrid(x, x, indexing="ij")
    a = _coeffs(seed, 4, 11)
    cx, cy = 0.5 + 0.15 * math.tanh(a[0]), 0.4 + 0.15 * math.tanh(a[1])
    phi = torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / (2 * 0.1 ** 2))
    return phi.reshape(-1)


def _requests(c, seed):
    """Requests of every size in turn, as the serving benchmark's stream makes them."""
    import dataclasses

    from jax_fem_cfd_b200.serving import make_requests
    sizes = [n for n in (32, 64, 128) if n <= c["most"]]
    out = []
    for i in range(c["count"]):
        r, = make_requests(1, seed=1000 * int(seed) + i, sizes=[sizes[i % len(sizes)]], steps=c["steps"])
        out.append(dataclasses.replace(r, rid=i))
    return out


def _operator_inputs(c, seed):
    s = c["order"]
    n = (s * c["nx"] + 1) * (s * c["ny"] + 1)
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    L = (c["nx"] / c["ny"], 1.0)
    if c["op"] != "visc_conv":
        return torch.randn(n, generator=g, dtype=F64, device="cuda"), None, L
    Y, X = torch.meshgrid(_axis(c["ny"], s, L[1], False), _axis(c["nx"], s, L[0], False), indexing="ij")
    u, v = _eddies(seed, X / L[0], Y)
    return (torch.randn(2 * n, generator=g, dtype=F64, device="cuda"),
            torch.cat([u.reshape(-1), v.reshape(-1)]), L)


def prepare(case, seed):
    import jax_fem_cfd_b200.setup.simulation as sim
    c, s = case, dict(case=case)
    if c["kind"] == "step":
        cfg = sim.Config(mesh="simple", solver="standard", mesh_config=_mesh_config(sim, c),
                         solver_config=_ns_config(sim, c))
        s["compute"], s["timestep"], coords, sn, _, nn, gd, Ud = sim.setup(cfg)
        s["Ud"] = _drive(sim, c, coords, sn, gd, nn, Ud)
        s["U"], s["P"] = _flow_inputs(c, seed)
    elif c["kind"] == "transport":
        f = _scalar_flow(c)
        cfg = sim.Config(mesh="simple", solver="passive_transport", mesh_config=_mesh_config(sim, f),
                         solver_config=sim.PassiveTransportConfig(
                             NS_config=_ns_config(sim, f),
                             ADE_config=sim.ADEConfig(phi_dirichlet_faces=[0], phi_SUPG=c["supg"])))
        s["compute"], s["timestep"], coords, sn, _, nn, _, _, gd, Ud, gphi = sim.setup(cfg)
        s["Ud"] = _drive(sim, f, coords, sn, gd, nn, Ud)
        s["U"], s["P"] = _flow_inputs(f, seed)
        s["phi"] = _scalar_start(c, seed)
        s["phi_d"] = torch.zeros(gphi.numel(), dtype=F64, device="cuda")
    elif c["kind"] == "poisson":
        from jax_fem_cfd_b200.context import Context, Mesh, make_mask
        from jax_fem_cfd_b200.core import multigrid as mg
        n = c["n"]
        s["ctx"] = ctx = Context(Mesh(0, False, n, n, 1, 1.0, 1.0))
        s["pin"] = make_mask(np.array([0]), ctx.nn)
        ctx.set_bc(None, s["pin"], True)
        nlev = int(math.log2(n // c["base"])) + 1
        s["hier"] = mg.Hierarchy(ctx, nlev, [np.array([0])] * nlev, c["tol"])
        s["b"] = _poisson_rhs(c, seed)
    elif c["kind"] == "operator":
        from jax_fem_cfd_b200.core import element_calc as ec
        from jax_fem_cfd_b200.core import shape_functions as sf
        from jax_fem_cfd_b200.setup import regular_mesh as rm
        x, vel, L = _operator_inputs(c, seed)
        make = rm.create_mesh_2d if c["order"] == 1 else rm.create_mesh_2d_quad9
        coords, s["nconn"], *_ = make(c["nx"], c["ny"], *L)
        s["nn"] = coords.shape[0]
        shape = sf.quad4_shape_functions if c["order"] == 1 else sf.quad9_shape_functions
        s["wq"], s["N"], s["dN"] = shape(coords[s["nconn"][0]])
        s["Le"] = ec.laplacian_element_calc(s["wq"], s["dN"])
        s["Me"] = ec.lumped_mass_matrix(s["nconn"], s["wq"], s["N"], s["nn"], 1)[1]
        s["x"], s["vel"] = x, vel
    elif c["kind"] == "inverse":
        from jax_fem_cfd_b200.solvers.inverse_transport import InverseTransport
        s["prob"] = InverseTransport(n=c["n"], steps=c["steps"], nu=c["nu"], D=c["D"], dt=c["dt"], ckpt=2,
                                     supg=c["supg"], seed=int(seed))
        s["U"] = s["prob"].initial_velocity().to(F64)
    else:
        from jax_fem_cfd_b200 import serving
        s["reqs"] = _requests(c, seed)
        s["server"] = (serving.PackedServer(ctas_by_size={32: 1, 64: 2, 128: 4}) if c["server"] == "packed"
                       else serving.Server(share=16))
        s["server"].prewarm(s["reqs"])
    return s


def _poisson_rhs(c, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    b = torch.randn((c["n"] + 1) ** 2, generator=g, dtype=F64, device="cuda")
    b[0] = 0.0
    return b


def run(s):
    c = s["case"]
    if c["kind"] == "step":
        Fp, F = s["compute"](s["Ud"], None, 0.0, c["dt"])
        U, P, ui, pi = s["timestep"](s["U"], s["P"], c["dt"], 1.0, c["nu"], s["Ud"], Fp, F)
        return {"U": U, "P": P, "U_iters": ui, "P_iters": pi}
    if c["kind"] == "transport":
        Fp, F = s["compute"](s["Ud"], None, 0.0, c["dt"])
        U, P, phi, ui, pi, fi = s["timestep"](s["U"], s["P"], s["phi"], c["dt"], 1.0, c["nu"], c["D"], s["Ud"],
                                              s["phi_d"], Fp, F, None)
        return {"U": U, "P": P, "phi": phi, "U_iters": ui, "P_iters": pi, "phi_iters": fi}
    if c["kind"] == "poisson":
        from jax_fem_cfd_b200 import _lib
        from jax_fem_cfd_b200.context import ptr, stream
        b, h = s["b"], s["ctx"].handle
        x = torch.zeros_like(b)
        if c["precision"] == "mixed":
            cyc, res = ctypes.c_int(0), ctypes.c_double(0.0)
            _lib.call("fem_pressure_solve_mixed", h, ptr(b), ptr(x), c["tol"], 8, 50, ctypes.byref(cyc),
                      ctypes.byref(res), stream())
            return {"x": x, "cycles": cyc.value}
        it = torch.zeros(2, dtype=torch.int32, device="cuda")
        _lib.call("fem_pressure_solve", h, ptr(b), ptr(x), c["tol"], 0.0, 1000, 4, 0, 1, ptr(it), ptr(it[1:]), stream())
        return {"x": x, "iters": it[0], "status": it[1]}
    if c["kind"] == "operator":
        from jax_fem_cfd_b200.core import element_calc as ec
        from jax_fem_cfd_b200.core import element_mult as em
        if c["op"] == "laplacian":
            return em.laplacian_element_mult(s["x"], s["Le"], s["nconn"], s["nn"])
        if c["op"] == "mass":
            return em.consistent_mass_mult(s["x"], s["Me"], s["nconn"], s["nn"], 1)
        Ce = ec.conservative_convec_elem_calc(s["nconn"], s["vel"], s["wq"], s["N"], s["dN"], s["nn"], 2, 0.5)
        return em.visc_conv_mult(s["x"], Ce, s["Le"], 0.01, 1.0, s["nconn"], s["nn"], 2)
    if c["kind"] == "inverse":
        L, g = s["prob"].value_and_grad(s["U"])
        return {"loss": L, "gradient": g}
    done, _ = s["server"].run(s["reqs"], realtime=False)
    return {"%03d" % d["rid"]: {"U": d["U"], "P": d["P"], "status": d["status"]} for d in done}


# ---------------------------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------------------------
def work(case):
    """Bytes: every input read once, every output written once. Operations: the Krylov
    iterations that the stop rule asks for (typical counts), each at one product with the
    operator and its vector updates, a multigrid cycle counted as four finest-level products."""
    c = case
    if c["kind"] == "step" or c["kind"] == "transport":
        f = _scalar_flow(c) if c["kind"] == "transport" else c
        nd = 3 if f["flow"] == "channel3d" else 2
        s = f["order"]
        nn = (s * f["nx"] + 1) * (s * f["ny"] + 1) * ((f["nz"] + 1) if nd == 3 else 1)
        row = 27 if nd == 3 else (9 if s == 1 else 20)  # entries of an assembled row, on average
        if f["precond"] == "multigrid":
            pressure = 8 * (5 * 2 * row + 12)
        else:
            pressure = 1.5 * max(f["nx"], f["ny"]) * (2 * row + 12) * s
        momentum = 4 * nd * 2 * (2 * row + 10)
        scalar = 6 * 2 * (2 * row + 10) if c["kind"] == "transport" else 0
        vectors = 2 * (nd + 1) + (2 if scalar else 0)
        return {"bytes": 8.0 * vectors * nn, "flops": float(nn * (pressure + momentum + scalar))}
    if c["kind"] == "poisson":
        nn = (c["n"] + 1) ** 2
        return {"bytes": 16.0 * nn, "flops": 10.0 * nn * (5 * 18 + 12)}
    if c["kind"] == "operator":
        s = c["order"]
        nn, ne = (s * c["nx"] + 1) * (s * c["ny"] + 1), c["nx"] * c["ny"]
        if c["op"] == "visc_conv":
            nen = 4 if s == 1 else 9
            return {"bytes": 8.0 * 6 * nn, "flops": float(ne * nen * nen * (4 + 4 * nen))}
        return {"bytes": 16.0 * nn, "flops": float(nn * 2 * (9 if s == 1 else 20))}
    if c["kind"] == "inverse":
        nn = (c["n"] + 1) ** 2
        return {"bytes": 8.0 * 4 * nn, "flops": float(3 * c["steps"] * nn * (10 * 102 + 8 * 4 * 28))}
    nn = 0
    for n in [n for n in (32, 64, 128) if n <= c["most"]]:
        nn += (n + 1) ** 2 * c["count"] / (3 if c["most"] == 128 else 2)
    return {"bytes": 8.0 * 5 * nn, "flops": float(c["steps"] * nn * (8 * 102 + 4 * 4 * 28))}


# ---------------------------------------------------------------------------------------------
# the same in plain torch, 64 bits
# ---------------------------------------------------------------------------------------------
class _Fem:
    """Element data of a uniform box mesh: local nodes in lexicographic order (x fastest)."""

    def __init__(self, order, n, L, periodic=False):
        nd, dev = len(n), "cuda"
        q, w = np.polynomial.legendre.leggauss(order + 1)
        if order == 1:
            B = np.stack([(1 - q) / 2, (1 + q) / 2], 1)
            dB = np.stack([-0.5 + 0 * q, 0.5 + 0 * q], 1)
        else:
            B = np.stack([q * (q - 1) / 2, 1 - q * q, q * (q + 1) / 2], 1)
            dB = np.stack([q - 0.5, -2 * q, q + 0.5], 1)
        h = [L[d] / n[d] for d in range(nd)]
        N, dN, W = None, None, None
        for d in range(nd):  # later axes vary slowest
            Dd = dB * (2 / h[d])
            if N is None:
                N, dN, W = B, [Dd], w * h[d] / 2
            else:
                dN = [np.kron(B, x) for x in dN] + [np.kron(Dd, N)]
                N, W = np.kron(B, N), np.kron(w * h[d] / 2, W)
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev)
        self.w, self.N, self.dN = t(W), t(N), t(np.stack(dN, 1))
        self.Me = torch.einsum("q,qa,qb->ab", self.w, self.N, self.N)
        self.Le = torch.einsum("q,qda,qdb->ab", self.w, self.dN, self.dN)
        self.Ge = torch.einsum("q,qa,qdb->dab", self.w, self.N, self.dN)
        self.nd, self.nen = nd, self.N.shape[1]
        ext = [order * n[d] + (0 if periodic else 1) for d in range(nd)]
        self.ext, self.nn = ext, int(np.prod(ext))
        conn = torch.zeros([1] * (2 * nd), dtype=torch.int64, device=dev)
        stride = 1
        for d in range(nd):
            e = torch.arange(n[d], device=dev)[:, None] * order + torch.arange(order + 1, device=dev)[None]
            e = (e % ext[d]) * stride
            shape = [1] * (2 * nd)
            shape[nd - 1 - d], shape[2 * nd - 1 - d] = n[d], order + 1
            conn = conn + e.reshape(shape)
            stride *= ext[d]
        self.conn = conn.reshape(-1, self.nen)
        self.flat = self.conn.reshape(-1)
        self.M = self.scatter(self.Me.sum(1).expand(self.conn.shape))  # lumped mass

    def scatter(self, Y):
        return torch.zeros(self.nn, dtype=F64, device="cuda").index_add(0, self.flat, Y.reshape(-1))

    def shared(self, K, x):
        return self.scatter(x[self.conn] @ K.T)

    def each(self, Ke, x):
        return self.scatter(torch.einsum("eab,eb->ea", Ke, x[self.conn]))

    def vec(self, f, U):
        return torch.cat([f(U[d * self.nn:(d + 1) * self.nn]) for d in range(self.nd)])

    def grad(self, p):
        return torch.cat([self.shared(self.Ge[d], p) for d in range(self.nd)])

    def div(self, U):
        out = 0
        for d in range(self.nd):
            out = out + self.shared(self.Ge[d].T, U[d * self.nn:(d + 1) * self.nn])
        return out

    def conv(self, U, beta):
        Ue = torch.stack([U[d * self.nn:(d + 1) * self.nn][self.conn] for d in range(self.nd)], 1)
        Uq = torch.einsum("qa,eda->eqd", self.N, Ue)
        dv = torch.einsum("qda,eda->eq", self.dN, Ue)
        T = torch.einsum("eqd,qdb->eqb", Uq, self.dN) + beta * dv[:, :, None] * self.N[None]
        return torch.einsum("qa,eqb->eab", self.w[:, None] * self.N, T)

    def at(self, U):
        return torch.stack([U[d * self.nn:(d + 1) * self.nn][self.conn] @ self.N.T for d in range(self.nd)], 2)


def _cg(A, b, D, its=20000, tol=1e-14):
    x, r = torch.zeros_like(b), b.clone()
    z = r / D
    p, g = z.clone(), torch.dot(r, z)
    stop = tol * float(b.norm())
    best, since = math.inf, 0
    for k in range(its):
        if k % 20 == 0:
            rn = float(r.norm())
            since = since + 1 if rn > 0.5 * best else 0
            best = min(best, rn)
            if rn <= stop or since > 60:
                break
        Ap = A(p)
        a = g / torch.dot(p, Ap)
        x, r = x + a * p, r - a * Ap
        z = r / D
        g, g0 = torch.dot(r, z), g
        p = z + (g / g0) * p
    return x


def _bicgstab(A, b, x, its=400, tol=1e-15):
    stop = tol * float(b.norm())
    for _ in range(3):  # restarted on the true residual
        r = b - A(x)
        if float(r.norm()) <= stop:
            break
        r0, p = r.clone(), r.clone()
        rho = torch.dot(r0, r)
        for k in range(its):
            q = A(p)
            a = rho / torch.dot(r0, q)
            s = r - a * q
            t = A(s)
            w = torch.dot(t, s) / torch.dot(t, t)
            if not math.isfinite(float(w)):
                break
            x, r = x + a * p + w * s, s - w * t
            if float(r.norm()) <= stop:
                break
            rho, old = torch.dot(r0, r), rho
            p = r + (rho / old) * (a / w) * (p - w * q)
    return x


class _Momentum(torch.autograd.Function):
    """x with sum_e K_e x = rhs on the free rows and x = rhs on the others, per component."""

    @staticmethod
    def forward(ctx, Ke, rhs, m, fixed, comps):
        def A(x, K=Ke):
            y = torch.cat([m.each(K, xc) for xc in x.view(comps, m.nn)])
            return torch.where(fixed, x, y)
        x = _bicgstab(A, rhs, rhs.clone())
        ctx.saved = (Ke, x, m, fixed, comps)
        return x

    @staticmethod
    def backward(ctx, g):
        Ke, x, m, fixed, comps = ctx.saved
        KT = Ke.transpose(1, 2).contiguous()

        def A(y):
            z = torch.cat([m.each(KT, yc) for yc in y.view(comps, m.nn)])
            return torch.where(fixed, y, z)
        lam = _bicgstab(A, torch.where(fixed, torch.zeros_like(g), g), torch.zeros_like(g))
        back = torch.cat([m.each(KT, yc) for yc in lam.view(comps, m.nn)])
        gK = 0
        for c in range(comps):
            gK = gK - lam.view(comps, m.nn)[c][m.conn][:, :, None] * x.view(comps, m.nn)[c][m.conn][:, None, :]
        return gK, torch.where(fixed, g - back, lam), None, None, None


class _Pressure(torch.autograd.Function):
    """The pinned or mean-zero pressure solve: symmetric in its right-hand side."""

    @staticmethod
    def solve(rhs, m, pin):
        D = m.scatter(torch.diagonal(m.Le).expand(m.conn.shape))
        if pin is None:
            b = rhs - rhs.mean()
            x = _cg(lambda p: m.shared(m.Le, p), b, D)
            return x - x.mean()
        zero = torch.zeros_like(rhs)
        return _cg(lambda p: torch.where(pin, zero, m.shared(m.Le, p)), torch.where(pin, zero, rhs), D)

    @staticmethod
    def forward(ctx, rhs, m, pin):
        ctx.saved = (m, pin)
        return _Pressure.solve(rhs, m, pin)

    @staticmethod
    def backward(ctx, g):
        return _Pressure.solve(g, *ctx.saved), None, None


def _boundary(c, m):
    """(fixed, Ud, pin, F_p): Dirichlet mask and values on all components, pinned pressure
    nodes, and the boundary integral of u_d . n over the Dirichlet faces."""
    nd, nn, ext = m.nd, m.nn, m.ext
    fixed = torch.zeros(nd, nn, dtype=torch.bool, device="cuda")
    Ud = torch.zeros(nd, nn, dtype=F64, device="cuda")
    Fp = torch.zeros(nn, dtype=F64, device="cuda")
    if c["flow"] == "vortex":
        return fixed.reshape(-1), Ud.reshape(-1), None, Fp
    ids = torch.arange(nn, device="cuda").reshape(list(reversed(ext)))
    L = _box(c)
    lex = lambda f: {0: (1, 0), 1: (0, 1), 2: (1, 1), 3: (0, 0), 4: (2, 0), 5: (2, 1)}[f]  # (axis, side)
    face = lambda f: ids.select(nd - 1 - lex(f)[0], -1 if lex(f)[1] else 0)
    dfaces, ofaces = _faces(c)
    for f in dfaces:
        fixed[:, face(f).reshape(-1)] = True
    if c["flow"] == "cavity":
        Ud[0, face(2)] = 1.0
    else:
        y = _axis(c["ny"], c["order"], L[1], False)
        if nd == 2:
            Ud[0, face(3)] = 4 * y * (1 - y)
        else:
            z = _axis(c["nz"], 1, L[2], False)
            Ud[0, face(3)] = 16 * (y * (1 - y))[None, :] * (z * (1 - z))[:, None]
    pin = torch.zeros(nn, dtype=torch.bool, device="cuda")
    if ofaces:
        for f in ofaces:
            pin[face(f).reshape(-1)] = True
    else:
        pin[0] = True
    n = [c["nx"], c["ny"], c.get("nz", 1)][:nd]
    for f in dfaces:
        ax, side = lex(f)
        un = Ud[ax] * (1.0 if side else -1.0)
        rest = [d for d in range(nd) if d != ax]
        e = _Fem(c["order"], [n[d] for d in rest], [L[d] for d in rest])
        Fp[face(f).reshape(-1)] += e.shared(e.Me, un[face(f).reshape(-1)])
    return fixed.reshape(-1), Ud.reshape(-1), pin, Fp


def _step(m, U, P, dt, nu, fixed, Ud, pin, Fp):
    Ce = m.conv(U, 0.5)
    rhs = (m.vec(lambda x: m.shared(m.Me, x), U) / dt
           - 0.5 * m.vec(lambda x: m.each(Ce, x) + nu * m.shared(m.Le, x), U) - m.grad(P))
    rhs = torch.where(fixed, Ud, rhs)
    K = m.Me / dt + 0.5 * (Ce + nu * m.Le)
    Uh = _Momentum.apply(K, rhs, m, fixed, m.nd)
    M = m.M.repeat(m.nd)
    Us = Uh + dt * m.grad(P) / M
    P1 = _Pressure.apply((m.div(Us) - Fp) / dt, m, pin)
    U1 = Us - dt * m.grad(P1) / M
    return torch.where(fixed, Ud, U1), P1


def _scalar(m, Un, U, phi, dt, D, supg, fixed, phid):
    Cn, C = m.conv(Un, 1.0), m.conv(U, 1.0)
    E, B = 0.5 * C, -0.5 * Cn
    if supg:
        Uq = m.at(Un)
        a = torch.einsum("eqd,qdb->eqb", Uq, m.dN)
        Ct = torch.einsum("q,eqa,eqb->eab", m.w, a, a)
        ce, kt = (C ** 2).sum((1, 2)).sqrt(), (Ct ** 2).sum((1, 2)).sqrt()
        t1 = ce / kt
        t3 = t1 * ((Uq ** 2).sum(2).mean(1) * ce) / ((D + 1e-6) * kt)
        tau = ((t1 ** -2 + (dt / 2) ** -2 + t3 ** -2) ** -0.5)[:, None, None]
        E = E + tau * (Cn.transpose(1, 2) / dt + 0.5 * Ct)
        B = B + tau * (Cn.transpose(1, 2) / dt - 0.5 * Ct)
    rhs = m.each(m.Me / dt - 0.5 * D * m.Le + B, phi)
    rhs = torch.where(fixed, phid, rhs)
    return _Momentum.apply(m.Me / dt + 0.5 * D * m.Le + E, rhs, m, fixed, 1)


def exact(case, seed):
    c = case
    if c["kind"] in ("step", "transport"):
        f = _scalar_flow(c) if c["kind"] == "transport" else c
        n = [f["nx"], f["ny"]] + ([f["nz"]] if f["flow"] == "channel3d" else [])
        m = _Fem(f["order"], n, _box(f), f["flow"] == "vortex")
        U, P = _flow_inputs(f, seed)
        with torch.no_grad():
            U1, P1 = _step(m, U, P, f["dt"], f["nu"], *_boundary(f, m))
            out = {"U": U1, "P": P1, "U_iters": None, "P_iters": None}
            if c["kind"] == "transport":
                fixed = torch.zeros(m.nn, dtype=torch.bool, device="cuda")
                fixed[:m.ext[0]] = True
                out["phi"] = _scalar(m, U, U1, _scalar_start(c, seed), c["dt"], c["D"], c["supg"], fixed,
                                     torch.zeros(m.nn, dtype=F64, device="cuda"))
                out["phi_iters"] = None
        return out
    if c["kind"] == "poisson":
        x = _poisson_exact(c["n"], _poisson_rhs(c, seed))
        return {"x": x, "cycles": None} if c["precision"] == "mixed" else {"x": x, "iters": None, "status": None}
    if c["kind"] == "operator":
        x, vel, L = _operator_inputs(c, seed)
        m = _Fem(c["order"], [c["nx"], c["ny"]], L)
        if c["op"] == "laplacian":
            return m.shared(m.Le, x)
        if c["op"] == "mass":
            return m.shared(m.Me, x)
        Ce = m.conv(vel, 0.5)
        return m.vec(lambda v: m.each(Ce, v) + 0.01 * m.shared(m.Le, v), x)
    if c["kind"] == "inverse":
        return _inverse_exact(c, seed)
    # a request is its own initial velocity on a cavity at rest, over its steps
    out = {}
    for r in _requests(c, seed):
        f = dict(kind="step", flow="cavity", order=1, nx=r.n, ny=r.n)
        m = _Fem(1, [r.n, r.n], (1.0, 1.0))
        fixed, Ud, pin, _ = _boundary(f, m)
        Ud = torch.zeros_like(Ud)
        U, P = torch.as_tensor(r.U0, device="cuda"), torch.zeros(m.nn, dtype=F64, device="cuda")
        with torch.no_grad():
            for _ in range(r.steps):
                U, P = _step(m, U, P, r.dt, r.nu, fixed, Ud, pin, 0.0)
        out["%03d" % r.rid] = {"U": U.cpu().numpy(), "P": P.cpu().numpy(), "status": None}
    return out


def _poisson_exact(n, b):
    """Cosines diagonalise the quad4 stiffness and mass of a uniform line: x of the pinned system."""
    k = torch.arange(n + 1, dtype=torch.int64, device="cuda")
    V = torch.cos((k[:, None] * k[None, :] % (2 * n)).to(F64) * (PI / n))
    th = k.to(F64) * (PI / n)
    lk, lm = 4 * torch.sin(th / 2) ** 2 * n * n, (2 + torch.cos(th)) / 3
    norm = torch.full((n + 1,), 0.5, dtype=F64, device="cuda")
    norm[0] = norm[-1] = 1.0
    B = b.clone()
    B[0] = 0.0
    B[0] = -B.sum()
    lam = lk[None, :] * lm[:, None] + lm[None, :] * lk[:, None]
    lam[0, 0] = 1.0
    T = (V.T @ B.view(n + 1, n + 1) @ V) / (lam * norm[:, None] * norm[None, :])
    T[0, 0] = 0.0
    x = (V @ T @ V.T).reshape(-1)
    return x - x[0]


def _inverse_exact(c, seed):
    """The loss and its gradient by torch.autograd through the restated steps."""
    n = c["n"]
    f = dict(kind="step", flow="cavity", order=1, nx=n, ny=n)
    m = _Fem(1, [n, n], (1.0, 1.0))
    fixed, Ud, pin, _ = _boundary(f, m)
    Ud = torch.zeros_like(Ud)
    none = torch.zeros(m.nn, dtype=torch.bool, device="cuda")
    x = _axis(n, 1, 1.0, False)
    Y, X = (t.reshape(-1) for t in torch.meshgrid(x, x, indexing="ij"))
    eps = 1e-12
    phi = ((X >= 0.4 - eps) & (X <= 0.6 + eps) & (Y >= 0.2 - eps) & (Y <= 0.4 + eps)).to(F64)
    target = torch.zeros(m.nn, dtype=F64, device="cuda")
    for cx, cy in np.random.default_rng(int(seed)).uniform(0.2, 0.8, size=(3, 2)):
        target += torch.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / (2 * 0.05 ** 2))
    g = torch.Generator(device="cpu").manual_seed(int(seed))
    U0 = (0.1 * torch.randn(2 * m.nn, generator=g, dtype=torch.float32)).to("cuda").to(F64).requires_grad_(True)
    U, P = U0, torch.zeros(m.nn, dtype=F64, device="cuda")
    for _ in range(c["steps"]):
        U1, P = _step(m, U, P, c["dt"], c["nu"], fixed, Ud, pin, 0.0)
        phi = _scalar(m, U, U1, phi, c["dt"], c["D"], c["supg"], none, torch.zeros_like(phi))
        U = U1
    L = (m.M * (phi - target) ** 2).sum()
    L.backward()
    return {"loss": float(L.detach()), "gradient": U0.grad}
