"""Tensor-core plans of the reference recursion keep its table, whatever the batch size (GPU).

From l_max 69 on that recursion's seeds underflow near beta = pi and d(m0, -n0) is no mirror image of d(m0, n0), so the groups
(m0, +-n0) must not share table rows.  At l_max 96 (the recursion's forward and inverse differ from the mathematical ones by
more than 1e-4) against FP64 plans of the same recursion, batches on both sides of the pairing's limits (8 complex and 16 real
functions in the beta-sum, 4 in the exact contraction; 9 and 17 in chunks of 8 leave a chunk of one function).  Bounds, relative
in the 2-norm: 1e-6, the FP32-data plans'; 1e-7 refined and exact.  l_max 68 is the last at which small batches pair.
"""
import numpy as np
import pytest

from conftest import so3_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,b,refined", [(96, 1, False), (96, 8, False), (96, 9, False), (96, 17, False), (68, 2, False),
                                         (69, 2, False), (96, 5, True), (96, 9, True), (96, 17, True), (68, 2, True)])
def test_reference_recursion(gblib, monkeypatch, L, b, refined, real):
    import torch
    if refined:
        monkeypatch.setenv("FFTSO3_REFINE_CHUNK", "8")
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    t64, t32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    s = torch.cuda.current_stream().cuda_stream
    ref = gblib.Plan(kind, L, 1, "fp64", "reference")
    tc = gblib.Plan(kind, L, b, "tc_bf16x3", "reference",
                    gblib.FLAG_REFINE | gblib.FLAG_EXACT_INVERSE if refined else 0)

    def inverse(c):
        g = torch.empty(ref.grid_elems, dtype=t64, device="cuda")
        ref.inverse(c.data_ptr(), g.data_ptr(), s)
        return g

    def forward(g):
        c = torch.empty(ref.coeff_elems, dtype=t64, device="cuda")
        ref.forward(g.data_ptr(), c.data_ptr(), s)
        return c

    c32 = torch.stack([torch.from_numpy(so3_coeffs(L, seed=900 + i, complex_=not real)).cuda().to(t32) for i in range(b)])
    grids = torch.empty((b, ref.grid_elems), dtype=t32, device="cuda")
    tc.inverse(c32.data_ptr(), grids.data_ptr(), s)
    smp = torch.stack([inverse(c.to(t64)).to(t32) for c in c32])
    got = torch.empty_like(c32)
    tc.forward(smp.data_ptr(), got.data_ptr(), s)
    tc.check()
    bound = 1e-7 if refined else 1e-6
    for i in sorted({0, b // 2, b - 1}):
        g, c = inverse(c32[i].to(t64)), forward(smp[i].to(t64))
        if refined:  # F0 + forward(f - inverse(F0)): the recursion's inverse is not the forward's
            c = 2 * c - forward(inverse(c))
        for x, y in ((grids[i], g), (got[i], c)):
            e = torch.linalg.vector_norm(x.to(t64) - y) / torch.linalg.vector_norm(y)
            assert float(e) <= bound, (i, float(e))
