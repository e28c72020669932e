"""Small solves of two contexts on two streams run at the same time: a lone one leaves room
for another on the device."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# (kind, periodic, nex, ney, nez, levels): quad4 pinned and mean-zero, quad9, hex8
@pytest.mark.parametrize("kind,periodic,nex,ney,nez,nlev", [(0, False, 64, 64, 1, 5), (0, True, 64, 64, 1, 5),
                                                            (1, True, 32, 32, 1, 4), (1, False, 90, 33, 1, 1),
                                                            (2, False, 50, 21, 19, 1), (2, False, 9, 9, 9, 1)])
def test_two_streams_overlap(kind, periodic, nex, ney, nez, nlev):
    """Barrier times of two pressure solves of 200 iterations (milliseconds each; the second
    is launched some tens of microseconds after the first, in one of three tries): they
    overlap."""
    from jax_fem_cfd_b200 import _lib
    from jax_fem_cfd_b200.context import Context, Mesh, make_mask, ptr
    from jax_fem_cfd_b200.core import multigrid as mg
    cap = 1 << 15
    solves = []
    for _ in range(2):
        ctx = Context(Mesh(kind, periodic, nex, ney, nez))
        ctx.set_bc(None, make_mask(np.array([0]), ctx.nn), not periodic)
        if nlev > 1:
            ctx.hier = mg.Hierarchy(ctx, nlev, [np.array([0])] * nlev, 1e-8)
        b = torch.as_tensor(np.random.default_rng(0).standard_normal(ctx.nn), device="cuda")
        b -= b.mean()
        solves.append((ctx, b, torch.zeros_like(b), torch.zeros(2, dtype=torch.int32, device="cuda"),
                       torch.zeros(cap, dtype=torch.int64, device="cuda"), torch.cuda.Stream()))

    def run():
        for ctx, b, x, it, tr, s in solves:
            x.zero_()
        torch.cuda.synchronize()
        for ctx, b, x, it, tr, s in solves:
            _lib.call("fem_pressure_solve", ctx.handle, ptr(b), ptr(x), 0.0, 0.0, 200,
                      _lib.PREC["multigrid" if nlev > 1 else "jacobi"], 0, 1, ptr(it), ptr(it[1:]), s.cuda_stream)
        torch.cuda.synchronize()

    run()
    for s in solves:
        _lib.call("fem_ctx_set_trace", s[0].handle, ptr(s[4]), cap)
    spans = []
    for _ in range(3):
        for s in solves:
            s[4].zero_()
        run()
        t = [s[4].cpu().numpy() for s in solves]
        t = [v[1:int(v[0]) + 1] & ((1 << 56) - 1) for v in t]
        spans.append([(int(v.min()), int(v.max())) for v in t])
    for s in solves:
        _lib.call("fem_ctx_set_trace", s[0].handle, None, 0)
    assert all(a1 - a0 > 200_000 for (a0, a1), _ in spans), spans  # ns: long beside the launches
    assert any(max(a0, b0) < min(a1, b1) for (a0, a1), (b0, b1) in spans), spans
