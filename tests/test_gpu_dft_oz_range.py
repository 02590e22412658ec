"""The digit DFT on lines of wide dynamic range (GPU): refined forward and exact inverse against FP64 plans.

A line is held to 2^-33 of its largest folded value, so errors are relative to that, not to each value (nor is the exact
contraction, which keeps 2^-30 of a sum's largest term).  Samples of 1e-5 with spikes
up to 1, and a function of one large coefficient among ones of 1e-6: relative 2-norm 1e-7, the refined plans' contract.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L", [10, 40, 79, 110])
def test_range(gblib, L, real):
    import torch
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    t64, t32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    s = torch.cuda.current_stream().cuda_stream
    g = torch.Generator("cuda").manual_seed(L)
    p = gblib.Plan(kind, L, 1, "tc_bf16x3", "stable", gblib.FLAG_REFINE | gblib.FLAG_EXACT_INVERSE)
    q = gblib.Plan(kind, L, 1, "fp64", "stable")

    def both(x, n, call):
        out = []
        for plan, dt in ((p, t32), (q, t64)):
            i, o = x.to(dt).contiguous(), torch.empty(n, dtype=dt, device="cuda")
            getattr(plan, call)(i.data_ptr(), o.data_ptr(), s)
            plan.check()
            out.append(o.to(t64))
        d = out[0] - out[1]
        assert float(torch.linalg.vector_norm(d) / torch.linalg.vector_norm(out[1])) <= 1e-7
        return out[1]

    f = torch.randn(p.grid_elems, dtype=t32, device="cuda", generator=g) * 1e-5
    f[::1997] *= 1e3
    f[p.grid_elems // 2 + 7] = 1.0
    both(f, p.coeff_elems, "forward")
    c = torch.randn(p.coeff_elems, dtype=t32, device="cuda", generator=g) * 1e-6
    c[5] = 1.0
    both(both(c, p.grid_elems, "inverse").to(t32), p.coeff_elems, "forward")
