"""Transforms over the power-of-two FFT passes, both launch forms, against the FP64 plans (GPU).

One launch per direction from 10 M samples, two below; S^2 one pass.  N = 64 to 1024 covers each split of the line FFT (8 x 8,
8 x 16 and 16 x 8, 16 x 16, 16 x 32, 32 x 32).  Bound, relative in the 2-norm of every function: twice the largest error of
the FP32-data plans, 5e-7 up to N = 256 and 1.6e-6 above (their sums over beta at N = 1024).
"""
import numpy as np
import pytest

from conftest import s2_coeffs, so3_coeffs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("family,L,b", [("so3", 31, 1), ("so3", 31, 39), ("so3", 63, 1), ("so3", 63, 5), ("so3", 127, 1),
                                        ("s2", 31, 3), ("s2", 63, 3), ("s2", 127, 2), ("s2", 255, 2), ("s2", 511, 2)])
def test_pow2_passes(gblib, family, L, b, real):
    import torch
    so3 = family == "so3"
    kind = {(True, True): gblib.SO3_REAL, (True, False): gblib.SO3_COMPLEX, (False, True): gblib.S2_REAL,
            (False, False): gblib.S2_COMPLEX}[so3, real]
    make = so3_coeffs if so3 else s2_coeffs
    F = np.concatenate([make(L, seed=4000 + L + i, complex_=not real) for i in range(b)])
    s = torch.cuda.current_stream().cuda_stream
    out = {}
    g32 = None
    for precision in ("fp64", "tc_bf16x3"):
        p = gblib.Plan(kind, L, b, precision, "stable" if so3 else "reference")
        dt = {("fp64", True): torch.float64, ("fp64", False): torch.complex128, ("tc_bf16x3", True): torch.float32,
              ("tc_bf16x3", False): torch.complex64}[precision, real]
        c32 = torch.from_numpy(F.astype(np.float32 if real else np.complex64)).cuda()
        c = c32.to(dt)
        g = torch.full((b * p.grid_elems,), float("nan"), dtype=dt, device="cuda")
        p.inverse(c.data_ptr(), g.data_ptr(), s)
        if g32 is None:
            g32 = g.to(torch.float32 if real else torch.complex64)
        x = g32.to(dt)
        c2 = torch.full_like(c, float("nan"))
        p.forward(x.data_ptr(), c2.data_ptr(), s)
        p.check()
        out[precision] = (g.reshape(b, -1), c2.reshape(b, -1))
        del p
    for got, ref in zip(out["tc_bf16x3"], out["fp64"]):
        d = torch.linalg.vector_norm(got.to(ref.dtype) - ref, dim=1) / torch.linalg.vector_norm(ref, dim=1)
        assert float(d.max()) <= (1e-6 if L <= 127 else 3.2e-6), d
