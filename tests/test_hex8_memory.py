"""What a hex8 context holds: no element matrices until a scalar step needs them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def test_context_without_element_matrices(monkeypatch):
    """64^3 elements: smaller by the matrices' size than a context whose step uses them."""
    from jax_fem_cfd_b200.context import Context, Mesh
    held = []
    Context(Mesh(2, False, 2, 2, 2))  # the library's own memory
    for otf in ("1", "0"):
        monkeypatch.setenv("FEM_CONV_OTF", otf)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        ctx = Context(Mesh(2, False, 64, 64, 64))
        held.append(free - torch.cuda.mem_get_info()[0])
        del ctx
    assert held[1] - held[0] >= 64 ** 3 * 64 * 8


def test_scalar_step_makes_them(monkeypatch):
    """fem_transport_phi on a context without them: the bits of one that has them."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import Context, Mesh, ptr, stream
    out = []
    for otf in ("1", "0"):
        monkeypatch.setenv("FEM_CONV_OTF", otf)
        ctx = Context(Mesh(2, False, 7, 5, 6))
        rng = np.random.default_rng(2)
        Un, U, phi = (torch.as_tensor(rng.standard_normal(n), device="cuda") for n in (3 * ctx.nn, 3 * ctx.nn, ctx.nn))
        po, it = torch.zeros_like(phi), torch.zeros(2, dtype=torch.int32, device="cuda")
        _lib.call("fem_transport_phi", ctx.handle, ptr(Un), ptr(U), ptr(phi), 1e-2, 1e-2, 0, None, None, 1e-10, ptr(po),
                  ptr(it), ptr(it[1:]), stream())
        assert int(it[1]) == 0
        out.append(po)
    assert torch.equal(*out)
