"""Refined and exactly inverted plans of many small grids, which go in pieces of many functions (GPU).

Batches on both sides of a piece's and of a contraction chunk's end (32 functions): N = 8 in pieces of 4096 and 2048 functions,
N = 22 of 192 and 96, N = 50 of 16 and 8.  Against FP64 plans, relative 2-norm 1e-7; the host-buffer calls give the device
calls' bits.
"""
import numpy as np
import pytest

from conftest import so3_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,b", [(3, 4097), (10, 193), (10, 33), (24, 35), (24, 17)])
def test_pieces(gblib, L, b, real):
    import torch
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    t64, t32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    s = torch.cuda.current_stream().cuda_stream
    p = gblib.Plan(kind, L, b, "tc_bf16x3", "stable", gblib.FLAG_REFINE | gblib.FLAG_EXACT_INVERSE)
    q = gblib.Plan(kind, L, b, "fp64", "stable")
    c = torch.from_numpy(np.concatenate([so3_coeffs(L, seed=i % 97, complex_=not real) for i in range(b)])).to(t32)
    out = []
    for plan, dt in ((q, t64), (p, t32)):
        x = c.cuda().to(dt)
        g = torch.empty(b * p.grid_elems, dtype=dt, device="cuda")
        plan.inverse(x.data_ptr(), g.data_ptr(), s)
        f = (out[0][0] if out else g).to(t32).to(dt)
        y = torch.empty_like(x)
        plan.forward(f.data_ptr(), y.data_ptr(), s)
        plan.check()
        out.append((g, y))
    for ref, got in zip(*out):
        d = (got.to(t64) - ref).reshape(b, -1)
        assert float((torch.linalg.vector_norm(d, dim=1) / torch.linalg.vector_norm(ref.reshape(b, -1), dim=1)).max()) <= 1e-7
    f = out[0][0].to(t32).cpu()
    g, y = torch.empty_like(f), torch.empty_like(c)
    p.inverse_host(c.data_ptr(), g.data_ptr(), s)
    p.forward_host(f.data_ptr(), y.data_ptr(), s)
    assert torch.equal(g, out[1][0].cpu()) and torch.equal(y, out[1][1].cpu())
