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
