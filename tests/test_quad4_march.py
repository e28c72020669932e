"""The quad4 momentum operator applied from nodal velocities, where its strips of 30
columns and runs of rows end, against the explicit element matrices."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

SIZES = [(False, 1, 1), (False, 2, 3), (False, 29, 5), (False, 30, 4), (False, 59, 40), (False, 60, 7),
         (True, 3, 3), (True, 4, 5), (True, 29, 30), (True, 30, 31), (True, 31, 64), (True, 60, 7)]


def _step(monkeypatch, otf, periodic, nex, ney, ctas):
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import Context, Mesh, ptr, stream
    monkeypatch.setenv("FEM_CONV_OTF", otf)
    ctx = Context(Mesh(0, periodic, nex, ney, 1, 2.0, 1.5))
    nn = ctx.nn
    rng = np.random.default_rng(nn)
    dm = torch.as_tensor((rng.random(2 * nn) < 0.2).astype(np.uint8), device="cuda")
    pm = torch.zeros(nn, dtype=torch.uint8, device="cuda")
    pm[0] = 1
    ctx.set_bc(dm, pm, True)
    _lib.call("fem_ctx_set_max_ctas", ctx.handle, ctas, None)
    U, Ud, P = (torch.as_tensor(rng.standard_normal(n), device="cuda") for n in (2 * nn, 2 * nn, nn))
    Uo, Po = torch.empty_like(U), torch.empty_like(P)
    it = torch.zeros(4, dtype=torch.int32, device="cuda")
    _lib.call("fem_step4", ctx.handle, ptr(U), ptr(P), 2e-2, 1.0, 5e-2, ptr(Ud), None, None, 1e-12,
              _lib.PREC["jacobi"], ptr(Uo), ptr(Po), ptr(it), ptr(it[2:]), stream())
    assert it[2:].tolist() == [0, 0], it.tolist()
    return Uo, Po


@pytest.mark.parametrize("periodic,nex,ney", SIZES)
def test_step_from_nodal_velocities(periodic, nex, ney, monkeypatch):
    """One fem_step4 on a random velocity (div u != 0) with random Dirichlet rows.
    Both forms solve to 1e-12; the pressure matrix's condition is below 1e6 here:
    1e-6 for either field."""
    a = _step(monkeypatch, "1", periodic, nex, ney, 0)
    b = _step(monkeypatch, "0", periodic, nex, ney, 0)
    for x, y in zip(a, b):
        assert float(torch.linalg.norm(x - y)) <= 1e-6 * float(torch.linalg.norm(y))


def test_bits_do_not_depend_on_spare_ctas(monkeypatch):
    """The same bits on nodes / 512 CTAs and on the whole device."""
    a = _step(monkeypatch, "1", False, 59, 40, 0)
    b = _step(monkeypatch, "1", False, 59, 40, -(-60 * 41 // 512))
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
