"""Tensor-core batches whose buckets may share table rows between the groups (m0, +-n0), mixed with ones that do not (GPU).

A bucket of at most 8 complex or 16 real functions can; the launch over all buckets does where that pays, by direction: neither,
the inverse alone, both.  Against FP64 plans of one function, relative 2-norm 1e-6, the path's contract.
"""
import numpy as np
import pytest

from conftest import so3_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real,lmax", [(False, [20] * 17 + [9]), (False, [20] * 9 + [19] * 8 + [18] * 8),
                                       (False, [9] * 9 + [20] * 8 + [33]), (True, [20] * 33 + [9] * 2),
                                       (True, [12] * 17 + [20] * 16 + [33] * 5)])
def test_mixed_buckets(gblib, real, lmax):
    import torch
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    t64, t32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    s = torch.cuda.current_stream().cuda_stream
    b = gblib.Batch(kind, lmax, "tc_bf16x3", "reference", gblib.FLAG_GRAPH)
    c = torch.empty(b.coeff_elems, dtype=t32, device="cuda")
    f = torch.empty(b.grid_elems, dtype=t32, device="cuda")
    want = []
    plans = {L: gblib.Plan(kind, L, 1, "fp64", "reference") for L in set(lmax)}
    for i, L in enumerate(lmax):
        p = plans[L]
        x = torch.from_numpy(so3_coeffs(L, seed=i, complex_=not real)).cuda().to(t32)
        g, y = torch.empty(p.grid_elems, dtype=t64, device="cuda"), torch.empty(p.coeff_elems, dtype=t64, device="cuda")
        p.inverse(x.to(t64).data_ptr(), g.data_ptr(), s)
        p.forward(g.to(t32).to(t64).data_ptr(), y.data_ptr(), s)
        co, go = slice(b.coeff_offset(i), b.coeff_offset(i) + x.numel()), slice(b.grid_offset(i), b.grid_offset(i) + g.numel())
        c[co], f[go] = x, g.to(t32)
        want.append((co, y, go, g))
    c2, f2 = torch.full_like(c, float("nan")), torch.full_like(f, float("nan"))
    b.forward(f.data_ptr(), c2.data_ptr(), s)
    b.inverse(c.data_ptr(), f2.data_ptr(), s)
    b.check()
    for co, y, go, g in want:
        for got, ref in ((c2[co], y), (f2[go], g)):
            assert float(torch.linalg.vector_norm(got.to(t64) - ref) / torch.linalg.vector_norm(ref)) <= 1e-6
