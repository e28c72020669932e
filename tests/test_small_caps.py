"""Quad4 solves on few CTAs and wide lattices: a plan has at least as many work items as
strips across the lattice (60 columns; 30 in the momentum solve and the restriction), which
is more than 16 per CTA from 481 elements across on one CTA and from 961 on two."""
import ctypes

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(480, 16, 1), (512, 16, 1), (1024, 8, 1), (1024, 8, 2)]  # elements, CTA cap


class _Problem:
    """A strip of square elements with random fields and Dirichlet rows, three levels."""

    def __init__(self, nex, ney, ctas, seed=0):
        from jax_fem_cfd_b200 import _lib
        from jax_fem_cfd_b200.context import Context, Mesh, make_mask
        from jax_fem_cfd_b200.core import multigrid as mg
        self.ctx = ctx = Context(Mesh(0, False, nex, ney, 1, nex / ney, 1.0))
        nn = ctx.nn
        rng = np.random.default_rng(nn + seed)
        dm = torch.as_tensor((rng.random(2 * nn) < 0.2).astype(np.uint8), device="cuda")
        ctx.set_bc(dm, make_mask(np.array([0]), nn), True)
        self.hier = mg.Hierarchy(ctx, 3, [np.array([0])] * 3, 1e-8)
        self.U, self.Ud, self.P, self.b = (torch.as_tensor(rng.standard_normal(n), device="cuda")
                                           for n in (2 * nn, 2 * nn, nn, nn))
        self.b[0] = 0.0
        _lib.call("fem_ctx_set_max_ctas", ctx.handle, ctas, None)

    def step(self, tol=1e-12):
        from jax_fem_cfd_b200 import _lib
        from jax_fem_cfd_b200.context import ptr, stream
        Uo, Po = torch.empty_like(self.U), torch.empty_like(self.P)
        it = torch.zeros(4, dtype=torch.int32, device="cuda")
        _lib.call("fem_step4", self.ctx.handle, ptr(self.U), ptr(self.P), 2e-2, 1.0, 5e-2, ptr(self.Ud), None, None,
                  tol, _lib.PREC["multigrid"], ptr(Uo), ptr(Po), ptr(it), ptr(it[2:]), stream())
        assert it[2:].tolist() == [0, 0], it.tolist()
        return Uo, Po, it[:2].tolist()


@pytest.mark.parametrize("precond", ["multigrid", "jacobi", "approx_inv", None])
@pytest.mark.parametrize("nex,ney,ctas", SIZES)
def test_two_cg_iterations(nex, ney, ctas, precond):
    """Two iterations, so that a wrong sum shows in x, against those of the whole device:
    the same sums in another order, 1e-10 as for the CG's phases elsewhere."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import ptr, stream
    out = []
    for cap in (ctas, 0):
        p = _Problem(nex, ney, cap)
        x = torch.zeros_like(p.b)
        it = torch.zeros(2, dtype=torch.int32, device="cuda")
        _lib.call("fem_pressure_solve", p.ctx.handle, ptr(p.b), ptr(x), 1e-30, 0.0, 2, _lib.PREC[precond], 0, 1,
                  ptr(it), ptr(it[1:]), stream())
        assert int(it[0]) == 2
        out.append(x)
    assert float(torch.linalg.norm(out[0] - out[1])) <= 1e-10 * float(torch.linalg.norm(out[1]))


@pytest.mark.parametrize("nex,ney,ctas", SIZES)
def test_step(nex, ney, ctas):
    """One step: the whole device's iteration counts to within one, and its fields to 1e-5
    (both solve to 1e-12; the pressure matrix of the longest strip has a condition of a few 1e6)."""
    a, b = _Problem(nex, ney, ctas).step(), _Problem(nex, ney, 0).step()
    for x, y in zip(a[:2], b[:2]):
        assert float(torch.linalg.norm(x - y)) <= 1e-5 * float(torch.linalg.norm(y))
    assert all(abs(i - j) <= 1 for i, j in zip(a[2], b[2])), (a[2], b[2])


@pytest.mark.parametrize("nex,ney,ctas", SIZES)
def test_packed_step(nex, ney, ctas):
    """Two packed members and their own steps on as many CTAs: the same bits."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import ptr, stream
    ps = [_Problem(nex, ney, ctas, seed) for seed in (0, 1)]
    solo = [p.step() for p in ps]
    U1, P1 = [torch.zeros_like(p.U) for p in ps], [torch.zeros_like(p.P) for p in ps]
    stat = torch.zeros(10, dtype=torch.int32, device="cuda")
    vp = lambda ts: (ctypes.c_void_p * 2)(*[t.data_ptr() for t in ts])
    h = ctypes.c_void_p()
    _lib.call("fem_pack_create", (ctypes.c_void_p * 2)(*[p.ctx.handle.value for p in ps]), 2, vp([p.U for p in ps]),
              vp([p.P for p in ps]), vp(U1), vp(P1), vp([p.Ud for p in ps]), ptr(stat), 1e-12,
              _lib.PREC["multigrid"], ctypes.byref(h))
    _lib.call("fem_pack_step", h, (ctypes.c_double * 2)(2e-2, 2e-2), (ctypes.c_double * 2)(5e-2, 5e-2),
              (ctypes.c_int * 2)(1, 1), (ctypes.c_int * 2)(0, 0), stream())
    torch.cuda.synchronize()
    _lib.load().fem_pack_destroy(h)
    st = stat.view(2, 5).tolist()
    for m in range(2):
        assert st[m][:2] == solo[m][2] and st[m][4] == 0, st[m]
        assert torch.equal(U1[m], solo[m][0]) and torch.equal(P1[m], solo[m][1]), m
