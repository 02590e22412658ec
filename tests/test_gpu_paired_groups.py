"""Small batches: the groups (m0, n0) and (m0, -n0) share the contraction's column tiles (GPU).

A batch of at most half a column tile against the FP64 plans, at the edges of that rule: 8 and 9 complex functions, 16 and 17
real ones; refined plans 4 and 5.  Row tiles (128 degrees), K steps (64) and 16-byte runs with remainders: l_max 0 to 66, 130.
Bounds, relative in the 2-norm: 1e-6, the FP32-data plans'; 1e-7 refined and exact.
"""
import numpy as np
import pytest

from conftest import so3_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,b,refined", [(0, 8, False), (1, 1, False), (12, 8, False), (12, 9, False), (12, 16, False),
                                         (12, 17, False), (31, 2, False), (63, 1, False), (66, 3, False), (130, 1, False),
                                         (0, 1, True), (12, 4, True), (12, 5, True), (31, 4, True), (66, 1, True)])
def test_paired_groups(gblib, L, b, refined, real):
    import torch
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    t64, t32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    F = np.concatenate([so3_coeffs(L, seed=600 + L + i, complex_=not real) for i in range(b)])
    c32 = torch.from_numpy(F).cuda().to(t32)
    s = torch.cuda.current_stream().cuda_stream
    g32, out = None, []
    for precision, dt in (("fp64", t64), ("tc_bf16x3", t32)):
        flags = gblib.FLAG_REFINE | gblib.FLAG_EXACT_INVERSE if refined and precision != "fp64" else 0
        p = gblib.Plan(kind, L, b, precision, "stable", flags)
        c = c32.to(dt)
        g = torch.full((b * p.grid_elems,), float("nan"), dtype=dt, device="cuda")
        p.inverse(c.data_ptr(), g.data_ptr(), s)
        if g32 is None:
            g32 = g.to(t32)
        x, c2 = g32.to(dt), torch.full_like(c, float("nan"))
        p.forward(x.data_ptr(), c2.data_ptr(), s)
        p.check()
        out.append((g.reshape(b, -1), c2.reshape(b, -1)))
        del p
    for ref, got in zip(*out):
        d = torch.linalg.vector_norm(got.to(ref.dtype) - ref, dim=1) / torch.linalg.vector_norm(ref, dim=1)
        assert float(d.max()) <= (1e-7 if refined else 1e-6), d
