"""The hex8 momentum operator applied from nodal velocities, where its columns of
30 x 11 nodes and runs of planes end, against the explicit element matrices."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [0, 1, 7])
@pytest.mark.parametrize("nex,ney,nez", [(1, 1, 1), (2, 3, 1), (29, 10, 2), (30, 11, 3), (28, 9, 5), (61, 22, 7)])
def test_step_from_nodal_velocities(nex, ney, nez, ctas, monkeypatch):
    """One fem_step4 on a random velocity (div u != 0) with random Dirichlet rows.
    Both forms solve to 1e-12; the pressure matrix's condition is below 1e4 here:
    1e-8 for either field."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import Context, Mesh, ptr, stream
    out = []
    for otf in ("1", "0"):
        monkeypatch.setenv("FEM_CONV_OTF", otf)
        ctx = Context(Mesh(2, False, nex, ney, nez, 2.0, 1.5, 0.7))
        nn = ctx.nn
        rng = np.random.default_rng(nn)
        dm = torch.as_tensor((rng.random(3 * nn) < 0.2).astype(np.uint8), device="cuda")
        pm = torch.zeros(nn, dtype=torch.uint8, device="cuda")
        pm[0] = 1
        ctx.set_bc(dm, pm, True)
        _lib.call("fem_ctx_set_max_ctas", ctx.handle, ctas, None)
        U, Ud, P = (torch.as_tensor(rng.standard_normal(n), device="cuda") for n in (3 * nn, 3 * nn, nn))
        Uo, Po = torch.empty_like(U), torch.empty_like(P)
        it = torch.zeros(4, dtype=torch.int32, device="cuda")
        _lib.call("fem_step4", ctx.handle, ptr(U), ptr(P), 2e-2, 1.0, 5e-2, ptr(Ud), None, None, 1e-12,
                  _lib.PREC["jacobi"], ptr(Uo), ptr(Po), ptr(it), ptr(it[2:]), stream())
        assert it[2:].tolist() == [0, 0], it.tolist()
        out.append((Uo.cpu().numpy(), Po.cpu().numpy()))
    for a, b in zip(*out):
        assert np.linalg.norm(a - b) <= 1e-8 * np.linalg.norm(b)


@pytest.mark.parametrize("ctas", [0, 1, 5])
@pytest.mark.parametrize("precond", ["jacobi", "approx_inv", None])
@pytest.mark.parametrize("nex,ney,nez", [(1, 1, 1), (29, 2, 1), (30, 3, 2), (59, 4, 3), (60, 5, 7)])
def test_cg_two_iterations(nex, ney, nez, precond, ctas):
    """Two CG iterations where the warps' columns of 30 x 2 nodes and runs of planes
    end, against the oracle's CG. Sums of at most 27 terms, two iterations: 1e-11."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import Context, Mesh, make_mask, ptr, stream
    from oracle import element as oel, emult as oem, mesh as om, shape as osh, solvers as osv
    box = (2.0, 1.5, 0.7)
    ctx = Context(Mesh(2, False, nex, ney, nez, *box))
    ctx.set_bc(None, make_mask(np.array([0]), ctx.nn), True)
    _lib.call("fem_ctx_set_max_ctas", ctx.handle, ctas, None)
    nc, nconn, *_ = om.create_mesh_3d(nex, ney, nez, *box)
    wq, _, dN = osh.hex8_shape_functions(nc[nconn[0]])
    Le = oel.laplacian_element_calc(wq, dN)
    D = oel.laplacian_diag(Le, nconn, ctx.nn)
    b = np.random.default_rng(ctx.nn).standard_normal(ctx.nn)
    b[0] = 0.0

    def lhs(v):
        y = oem.laplacian_element_mult(v, Le, nconn, ctx.nn)
        y[0] = 0.0
        return y

    def approx(r):  # solvers/standard.py:225-234
        t = lhs(r / D) / D
        return 3 * (r / D) - 3 * t + lhs(t) / D

    M = {"jacobi": lambda r: r / D, "approx_inv": approx, None: None}[precond]
    xo, _ = osv.cg(lhs, b, x0=np.zeros_like(b), tol=1e-30, maxiter=2, M=M)
    xo[0] = 0.0
    r = torch.as_tensor(b, device="cuda")
    x = torch.zeros_like(r)
    it = torch.zeros(2, dtype=torch.int32, device="cuda")
    _lib.call("fem_pressure_solve", ctx.handle, ptr(r), ptr(x), 1e-30, 0.0, 2, _lib.PREC[precond], 0, 1, ptr(it),
              ptr(it[1:]), stream())
    assert int(it[0]) == 2
    assert np.linalg.norm(x.cpu().numpy() - xo) <= 1e-11 * np.linalg.norm(xo)
