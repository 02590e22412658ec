"""FP64 S^2 sums over beta, folded by parity, eight lanes a degree (GPU), against the oracle.

l_max from 0 over the edges of eight samples a lane group (N / 2 = 8, 9), of a warp's four degrees of one parity and of a CTA's
(32 degrees a parity), and of the inverse's 128 samples a sweep (N / 2 = 128, 129).  Bound: 1e-12 of the result's norm (sums of
at most 260 terms in FP64).
"""
import numpy as np
import pytest

from conftest import s2_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,b", [(0, 2), (1, 1), (2, 1), (7, 3), (8, 1), (15, 2), (31, 1), (32, 1), (63, 1), (64, 1), (127, 1),
                                 (128, 1)])
def test_s2_fp64(gblib, oracle, L, b, real):
    import torch
    kind = gblib.S2_REAL if real else gblib.S2_COMPLEX
    dt = torch.float64 if real else torch.complex128
    F = np.stack([s2_coeffs(L, seed=800 + L + i, complex_=not real) for i in range(b)])
    ref = np.stack([(oracle.s2_inverse_real_grid if real else oracle.s2_inverse_complex_grid)(L, x).ravel() for x in F])
    p = gblib.Plan(kind, L, b, "fp64", "reference")
    s = torch.cuda.current_stream().cuda_stream
    c = torch.from_numpy(F.ravel()).to("cuda", dt)
    g = torch.full((b * p.grid_elems,), float("nan"), dtype=dt, device="cuda")
    p.inverse(c.data_ptr(), g.data_ptr(), s)
    c2 = torch.full_like(c, float("nan"))
    x = torch.from_numpy(ref.ravel()).to("cuda", dt)
    p.forward(x.data_ptr(), c2.data_ptr(), s)
    p.check()
    assert np.linalg.norm(g.cpu().numpy() - ref.ravel()) <= 1e-12 * np.linalg.norm(ref)
    assert np.linalg.norm(c2.cpu().numpy() - F.ravel()) <= 1e-12 * np.linalg.norm(F)
