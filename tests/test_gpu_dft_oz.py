"""The digit DFT (exact digit sums on the tensor cores) of the refined and the exactly inverted SO(3) plans (GPU).

It serves every even N up to 222 but the powers of two from 64.  Against the FP64 plans on the same FP32 data:

* exact inverse: |g - g64| <= 2^-24 |g64| + 1.5e-8 rms(g64) per component: the output rounding, and six standard deviations
  (up to 10^7 values) of the contraction's dropped digit products, 2.2e-9 of the rms, and of the passes', 0.4e-9;
* refined forward: rel_rms <= 1e-7, rel_max (per degree, against its rms) <= 1e-6, the bounds of the other refined plans.

The sizes are the smallest, both sides of each step of the operand's rows (16 folded terms: N = 60, 62, 64; 32: 124, 126,
130; 48: 188, 190, 192), the smallest that the inverse takes to it (20, at 25 functions or more), odd and even N / 2, and
both sides of the largest (222, 224).
"""
import numpy as np
import pytest

from conftest import so3_coeffs
from test_gpu_exact_inverse import _exact_inverse
from test_gpu_refine import _refined, per_l_errors

pytestmark = pytest.mark.gpu


def _double(gblib, kind, L, x, forward):
    import torch
    b = x.shape[0]
    p = gblib.Plan(kind, L, b, "fp64", "stable")
    dt = torch.complex128 if kind == gblib.SO3_COMPLEX else torch.float64
    i = torch.from_numpy(np.ascontiguousarray(x).ravel()).to("cuda", dt)
    o = torch.empty(b * (p.coeff_elems if forward else p.grid_elems), dtype=dt, device="cuda")
    (p.forward if forward else p.inverse)(i.data_ptr(), o.data_ptr(), torch.cuda.current_stream().cuda_stream)
    p.check()
    out = o.cpu().numpy().reshape(b, -1)
    del p
    return out


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,scale", [(0, 1.0), (1, 1.0), (2, 1.0), (7, 1e-12), (8, 1e12), (9, 1.0), (28, 1.0), (29, 1.0), (30, 1.0),
                                     (32, 1.0), (61, 1.0), (62, 1.0), (64, 1.0), (93, 1.0), (94, 1.0), (95, 1.0), (110, 1.0),
                                     (111, 1.0)])
def test_digit_dft(gblib, L, scale, real):
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    b = 27 if L == 9 else 3 if L < 90 else 2
    F = np.stack([so3_coeffs(L, seed=9000 + 17 * L + i, complex_=not real, decay="pow") for i in range(b)]) * scale
    F32 = F.astype(np.float32 if real else np.complex64)
    env = {"FFTSO3_REFINE_CHUNK": "2"} if b == 3 else None
    got = _exact_inverse(gblib, kind, L, F32, env)
    ref = _double(gblib, kind, L, F32, False)
    for i in range(b):
        rms = np.sqrt(np.mean(np.abs(ref[i]) ** 2))
        for g, r in [(got[i], ref[i])] if real else [(got[i].real, ref[i].real), (got[i].imag, ref[i].imag)]:
            over = float((np.abs(g - r) - 2.0 ** -24 * np.abs(r)).max() / rms)
            assert over <= 1.5e-8, (i, over)
    out = _refined(gblib, kind, L, got, chunk=2 if b == 3 else None)
    ref = _double(gblib, kind, L, got, True)
    for i in range(b):
        rms, mx = per_l_errors(out[i], ref[i], L)
        assert rms <= 1e-7 and mx <= 1e-6, (i, rms, mx)
