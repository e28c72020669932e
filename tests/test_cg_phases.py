"""The 2D phases of the persistent CG at the sizes where their work splits: a
strip of 60 (quad4) or 28 (quad9) columns and one more, a coarse strip of 30 or
13, lattices narrower than a strip (periodic wraps inside it), odd and oblong
ones; with the dense coarse operator at several levels and without it. Against
the oracle's V-cycle and CG in numpy."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# (order, nex, ney, levels): columns of the finest lattice 61 / 60 / 59, 29 / 28, ...
CASES = [(1, 2, 2, 2), (1, 4, 6, 2), (1, 58, 6, 2), (1, 60, 62, 2), (1, 62, 58, 2), (1, 30, 120, 2), (1, 24, 40, 4),
         (2, 2, 2, 2), (2, 12, 14, 2), (2, 14, 12, 2), (2, 16, 28, 3), (2, 26, 10, 2)]


def _oracle(order, periodic, nex, ney, nlev):
    from oracle import element as oel, emult as oem, mesh as om, multigrid as omg, shape as osh
    mf = {(1, False): om.create_mesh_2d, (1, True): om.create_periodic_mesh_2d,
          (2, False): om.create_mesh_2d_quad9, (2, True): om.create_periodic_mesh_2d_quad9}[order, periodic]
    sf = osh.quad4_shape_functions if order == 1 else osh.quad9_shape_functions
    L = [1.5, 1.0]
    nc, nconn, *_ = mf(nex, ney, *L)
    data = omg.multigrid_setup([nex, ney], [nex >> (nlev - 1), ney >> (nlev - 1)], L, [], mf, sf, order, None)
    # the mesh generators of periodic meshes keep element 0's coordinates unwrapped
    wq, _, dN = sf(nc[nconn[0]])
    Le = oel.laplacian_element_calc(wq, dN)
    return data, lambda v: oem.laplacian_element_mult(v, Le, nconn, nc.shape[0])


def _context(order, periodic, nex, ney, nlev, pinned, coarse_tol):
    from jax_fem_cfd_b200.context import Context, Mesh, make_mask
    from jax_fem_cfd_b200.core import multigrid as mg
    ctx = Context(Mesh(order - 1, periodic, nex, ney, 1, 1.5, 1.0))
    ctx.set_bc(None, make_mask(np.array([0]), ctx.nn), pinned)
    return ctx, mg.Hierarchy(ctx, nlev, [np.array([0])] * nlev, coarse_tol)


def _rhs(nn, pinned):
    b = np.random.default_rng(nn).standard_normal(nn)
    if pinned:
        b[0] = 0.0
    return b if pinned else b - b.mean()


def _rel(a, b):
    return float(np.linalg.norm(a.cpu().numpy() - b) / np.linalg.norm(b))


@pytest.mark.parametrize("periodic", [False, True])
@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("order,nex,ney,nlev", CASES)
def test_vcycle(order, nex, ney, nlev, pinned, periodic):
    """One V-cycle. Every sum has at most 25 terms of like size and a level adds
    four of them: 1e-12 (1e-9 pinned, where the coarsest CG's last digits differ)."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import ptr, stream
    from oracle import multigrid as omg
    if periodic and min(nex, ney) >> (nlev - 1) < 2 * order:
        pytest.skip("coarsest periodic lattice narrower than its stencil")
    ctx, _ = _context(order, periodic, nex, ney, nlev, pinned, 1e-8)
    data, _ = _oracle(order, periodic, nex, ney, nlev)
    b = _rhs(ctx.nn, pinned)
    r = torch.as_tensor(b, device="cuda")
    z = torch.empty_like(r)
    _lib.call("fem_mg_vcycle", ctx.handle, ptr(r), ptr(z), stream())
    assert _rel(z, omg.v_cycle(b, *data, 1e-8, periodic, pinned)) < (1e-9 if pinned else 1e-12)


@pytest.mark.parametrize("pinned", [True, False])
@pytest.mark.parametrize("precond", ["multigrid", "jacobi", "approx_inv", None])
@pytest.mark.parametrize("order,nex,ney,nlev", [CASES[1], CASES[3], CASES[6], CASES[7], CASES[9], CASES[10]])
def test_two_iterations(order, nex, ney, nlev, precond, pinned):
    """Two CG iterations, so that a wrong preconditioner or sum shows in x. The
    dense operator holds the exact coarsest inverse, so the oracle's coarsest CG
    runs to 1e-14; 1e-10 for the two."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import ptr, stream
    from oracle import multigrid as omg, solvers as osv
    ctx, _ = _context(order, False, nex, ney, nlev, pinned, 1e-8)
    data, lap = _oracle(order, False, nex, ney, nlev)
    b = _rhs(ctx.nn, pinned)
    D = data[3][:ctx.nn]

    def lhs(v):
        y = lap(v)
        if pinned:
            y[0] = 0.0
        return y

    def approx(r):  # solvers/standard.py:225-234; the scalar pin of a mean-zero problem is node 0 too
        t = lap(r / D) / D
        t[0] = 0.0
        u = lap(t)
        u[0] = 0.0
        return 3 * (r / D) - 3 * t + u / D

    M = {"multigrid": lambda r: omg.v_cycle(r, *data, 1e-14, False, pinned), "jacobi": lambda r: r / D,
         "approx_inv": approx, None: None}[precond]
    xo, _ = osv.cg(lhs, b, x0=np.zeros_like(b), tol=1e-30, maxiter=2, M=M)
    if pinned:
        xo[0] = 0.0
    else:
        xo = xo - xo.mean()
    r = torch.as_tensor(b, device="cuda")
    x = torch.zeros_like(r)
    it = torch.zeros(2, dtype=torch.int32, device="cuda")
    _lib.call("fem_pressure_solve", ctx.handle, ptr(r), ptr(x), 1e-30, 0.0, 2, _lib.PREC[precond], 0 if pinned else 1,
              1, ptr(it), ptr(it[1:]), stream())
    assert int(it[0]) == 2 and _rel(x, xo) < 1e-10


def test_bits_do_not_depend_on_spare_ctas():
    """A wall-bounded quad4 solve has the same bits on its share of nodes / 512
    CTAs and on the whole device."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import ptr, stream
    ctx, _ = _context(1, False, 72, 48, 4, True, 1e-8)
    r = torch.as_tensor(_rhs(ctx.nn, True), device="cuda")
    out = []
    for ctas in (0, -(-ctx.nn // 512)):
        _lib.call("fem_ctx_set_max_ctas", ctx.handle, ctas, None)
        x = torch.zeros_like(r)
        it = torch.zeros(2, dtype=torch.int32, device="cuda")
        _lib.call("fem_pressure_solve", ctx.handle, ptr(r), ptr(x), 1e-10, 0.0, 100, 4, 0, 1, ptr(it), ptr(it[1:]),
                  stream())
        assert int(it[1]) == 0
        out.append(x)
    assert torch.equal(*out)
