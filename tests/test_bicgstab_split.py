"""BiCGSTAB on explicit 2D element matrices on both sides of its split: 8-row tiles of
its small form (rows and columns at a tile's edge and one more), 16-row tiles."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ncomp", [1, 2])
@pytest.mark.parametrize("order,nex,ney", [(1, 1, 1), (1, 31, 7), (1, 32, 8), (1, 63, 40), (1, 400, 200),
                                           (2, 1, 1), (2, 15, 3), (2, 16, 4), (2, 220, 100)])
def test_residual(order, nex, ney, ncomp):
    """Element matrices near the identity: the solve to 1e-11 leaves a true residual
    within 1e-10 of the right-hand side."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import Context, Mesh, ptr, stream
    from oracle import mesh as om
    ctx = Context(Mesh(order - 1, False, nex, ney, 1, 1.5, 1.0))
    mf = om.create_mesh_2d if order == 1 else om.create_mesh_2d_quad9
    _, nconn, *_ = mf(nex, ney, 1.5, 1.0)
    nn, (ne, nen) = ctx.nn, nconn.shape
    rng = np.random.default_rng(nn)
    A = np.eye(nen) + 0.02 * rng.standard_normal((nen, nen))
    B = 0.02 * rng.standard_normal((ne, nen, nen))
    b = rng.standard_normal(ncomp * nn)
    d = [torch.as_tensor(np.ascontiguousarray(v), device="cuda") for v in (A, B, b)]
    x = torch.zeros(ncomp * nn, dtype=torch.float64, device="cuda")
    it = torch.zeros(2, dtype=torch.int32, device="cuda")
    _lib.call("fem_bicgstab_solve", ctx.handle, ncomp, 1.0, ptr(d[0]), 0.5, ptr(d[1]), 0.0, None, None, ptr(d[2]),
              ptr(x), 1e-11, 0.0, 0, ptr(it), ptr(it[1:]), stream())
    assert int(it[1]) == 0
    xs, bs = x.cpu().numpy().reshape(ncomp, nn), b.reshape(ncomp, nn)
    for c in range(ncomp):
        y = np.zeros(nn)
        np.add.at(y, nconn, np.einsum("eab,eb->ea", A + 0.5 * B, xs[c][nconn]))
        assert np.linalg.norm(y - bs[c]) <= 1e-10 * np.linalg.norm(bs)
