"""The dense operators of the coarse multigrid levels: on periodic lattices and with whole
faces pinned against the oracle's CG; shared by contexts; under captured solves and packs
when the boundary sets change."""
import ctypes
import gc

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# level 0 has a matrix of its own on the first two (289 quad9 nodes; 169 quad4 nodes)
SMALL = [(2, 8, 8, 2), (1, 12, 12, 2)]


def _context(order, nex, ney, nlev, pinned, periodic=False, pins=None, faces=()):
    from jax_fem_cfd_b200.context import Context, Mesh, make_mask
    from jax_fem_cfd_b200.core import multigrid as mg
    mesh = Mesh(order - 1, periodic, nex, ney, 1, 1.5, 1.0)
    ctx = Context(mesh)
    sets = mg.level_pin_sets(mesh, nlev, list(faces), None, order)
    ctx.set_bc(None, make_mask(sets[0], ctx.nn), pinned)
    ctx.hier = mg.Hierarchy(ctx, nlev, sets, 1e-8)
    if pins is not None:
        ctx.set_bc(None, pins, pinned)
    return ctx


def _solver(ctx, b, center=0, its=2):
    """(x, call): call() runs `its` CG iterations from zero into x."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import ptr, stream
    x, it = torch.zeros_like(b), torch.zeros(2, dtype=torch.int32, device="cuda")

    def call():
        x.zero_()
        _lib.call("fem_pressure_solve", ctx.handle, ptr(b), ptr(x), 1e-30, 0.0, its, _lib.PREC["multigrid"], center, 1,
                  ptr(it), ptr(it[1:]), stream())
        return x
    return x, call


def _rhs(nn):
    return torch.as_tensor(np.random.default_rng(nn).standard_normal(nn), device="cuda")


def _pins(nn):
    """Node 0 and every 7th node."""
    p = torch.zeros(nn, dtype=torch.uint8, device="cuda")
    p[::7] = 1
    return p


@pytest.mark.parametrize("periodic,faces", [(False, (1,)), (False, (0, 3)), (True, ())])
@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("order,nex,ney,nlev", SMALL + [(1, 24, 40, 4), (2, 16, 28, 3)])
def test_two_iterations(order, nex, ney, nlev, pinned, periodic, faces):
    """Two CG iterations against the oracle's with its coarsest CG to 1e-14: 1e-10, as for
    the CG's phases elsewhere."""
    from oracle import element as oel, emult as oem, mesh as om, multigrid as omg, shape as osh, solvers as osv
    from jax_fem_cfd_b200.core import multigrid as mg
    mf = {(1, False): om.create_mesh_2d, (1, True): om.create_periodic_mesh_2d,
          (2, False): om.create_mesh_2d_quad9, (2, True): om.create_periodic_mesh_2d_quad9}[order, periodic]
    sf = osh.quad4_shape_functions if order == 1 else osh.quad9_shape_functions
    nc, nconn, *_ = mf(nex, ney, 1.5, 1.0)
    data = omg.multigrid_setup([nex, ney], [nex >> (nlev - 1), ney >> (nlev - 1)], [1.5, 1.0], list(faces), mf, sf,
                               order, None)
    wq, _, dN = sf(nc[nconn[0]])
    Le = oel.laplacian_element_calc(wq, dN)
    ctx = _context(order, nex, ney, nlev, pinned, periodic, faces=faces)
    pins = mg.level_pin_sets(ctx.mesh, 1, list(faces), None, order)[0]
    b = np.random.default_rng(ctx.nn).standard_normal(ctx.nn)
    if pinned:
        b[pins] = 0.0
    else:
        b -= b.mean()

    def lhs(v):
        y = oem.laplacian_element_mult(v, Le, nconn, nc.shape[0])
        if pinned:
            y[pins] = 0.0
        return y

    xo, _ = osv.cg(lhs, b, x0=np.zeros_like(b), tol=1e-30, maxiter=2,
                   M=lambda r: omg.v_cycle(r, *data, 1e-14, periodic, pinned))
    if pinned:
        xo[pins] = 0.0
    else:
        xo = xo - xo.mean()
    x = _solver(ctx, torch.as_tensor(b, device="cuda"), 0 if pinned else 1)[1]()
    assert float(np.linalg.norm(x.cpu().numpy() - xo)) <= 1e-10 * float(np.linalg.norm(xo))


@pytest.mark.parametrize("order,nex,ney,nlev", SMALL + [(1, 64, 64, 4), (2, 40, 24, 3)])
def test_captured_solve_follows_set_bc(order, nex, ney, nlev):
    """A captured pinned solve, replayed after the pins changed and after the context went to
    mean-zero pressure: the bits of a direct pinned solve with the pins of that moment (the
    larger lattices read them in their sweeps, not in a matrix)."""
    ctx = _context(order, nex, ney, nlev, True)
    x, call = _solver(ctx, _rhs(ctx.nn))
    call()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        call()
    first, pins = None, _pins(ctx.nn)
    for p in (None, pins):
        if p is not None:
            ctx.set_bc(None, p, True)
        want = call().clone()
        g.replay()
        assert torch.equal(x, want) and (first is None or not torch.equal(first, want))
        first = want
    ctx.set_bc(None, pins, False)
    g.replay()
    assert torch.equal(x, first)


@pytest.mark.parametrize("order,nex,ney,nlev", SMALL + [(1, 64, 64, 4)])
def test_set_bc_is_captured(order, nex, ney, nlev):
    """fem_ctx_set_bc on a capturing stream; its replay takes the masks of that moment."""
    a, b = _context(order, nex, ney, nlev, True), _context(order, nex, ney, nlev, True)
    pins = a._pmask.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        a.set_bc(None, pins, True)
    new = _pins(a.nn)
    pins.copy_(new)
    g.replay()
    b.set_bc(None, new, True)
    rhs = _rhs(a.nn)
    assert torch.equal(_solver(a, rhs)[1](), _solver(b, rhs)[1]())


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("order,nex,ney,nlev", SMALL + [(1, 64, 64, 4)])
def test_shared_set_outlives_a_context(order, nex, ney, nlev, pinned):
    a, b = (_context(order, nex, ney, nlev, pinned) for _ in range(2))
    _, call = _solver(b, _rhs(b.nn))
    want = call().clone()
    del a
    gc.collect()
    assert torch.equal(call(), want)


def test_pack_follows_set_bc():
    """A pack of 12 x 12 members (level 0 dense) after new pins: fem_step4's bits."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import ptr, stream
    ctx = _context(1, 12, 12, 2, True)
    nn = ctx.nn
    rng = np.random.default_rng(5)
    U, P = (torch.as_tensor(0.1 * rng.standard_normal(n), device="cuda") for n in (2 * nn, nn))
    U1, P1, Uo, Po = (torch.zeros_like(t) for t in (U, P, U, P))
    stat, it = torch.zeros(5, dtype=torch.int32, device="cuda"), torch.zeros(4, dtype=torch.int32, device="cuda")
    vp = lambda v: (ctypes.c_void_p * 1)(v)
    h = ctypes.c_void_p()
    # a loose tolerance: pins that the hierarchy does not have make a poor preconditioner
    _lib.call("fem_pack_create", vp(ctx.handle.value), 1, vp(U.data_ptr()), vp(P.data_ptr()), vp(U1.data_ptr()),
              vp(P1.data_ptr()), None, ptr(stat), 0.5, _lib.PREC["multigrid"], ctypes.byref(h))
    ctx.set_bc(None, _pins(nn), True)
    _lib.call("fem_step4", ctx.handle, ptr(U), ptr(P), 1e-2, 1.0, 1e-2, None, None, None, 0.5, _lib.PREC["multigrid"],
              ptr(Uo), ptr(Po), ptr(it), ptr(it[2:]), stream())
    _lib.call("fem_pack_step", h, (ctypes.c_double * 1)(1e-2), (ctypes.c_double * 1)(1e-2), (ctypes.c_int * 1)(1),
              (ctypes.c_int * 1)(0), stream())
    torch.cuda.synchronize()
    _lib.load().fem_pack_destroy(h)
    assert torch.equal(U1, Uo) and torch.equal(P1, Po)
