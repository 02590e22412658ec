"""The direct DFT passes of the FP32-data plans (grid sizes the register FFT does not serve), against FP64 plans.

The sizes are the edges of the folding (N = 2, 4, 6: one folded term, N / 2 even and odd), of the four-output blocks
and the tiles, the smallest and largest N of each tile shape, primes, the last size before the fallback, and the first
and last of the tensor-core form (N = 80 and 222; N = 126 and 124: the folded terms fill whole chunks, or all but one).
Batches make half a million samples (a million on the sphere), from which the direct passes are used; a few are smaller.
Tolerance: relative L2 error 1e-6, the path's contract.  Each pass sums at most 101 folded products in FP32, a random
walk of 2^-25 sqrt(101) = 3e-7 of the line's norm; the beta-sum adds about the same.
"""
import numpy as np
import pytest

from conftest import s2_coeffs, so3_coeffs

pytestmark = pytest.mark.gpu

TOL = 1e-6


def _round_trip(gblib, kind, real, L, batch, precision, F):
    import torch

    dt = {True: torch.float64, False: torch.complex128}[real]
    dt32 = {True: torch.float32, False: torch.complex64}[real]
    p64 = gblib.Plan(kind, L, 1, "fp64", "stable")
    p32 = gblib.Plan(kind, L, batch, precision, "stable")
    s = torch.cuda.current_stream().cuda_stream
    F32 = torch.from_numpy(F).to(dt32).cuda()
    F64 = F32.to(dt)
    g32 = torch.empty(batch * p32.grid_elems, dtype=dt32, device="cuda")
    c32 = torch.empty_like(F32)
    p32.inverse(F32.data_ptr(), g32.data_ptr(), s)
    # samples that are not band-limited, so that every bin of the forward matters
    f32 = g32 + 0.1 * g32.abs().mean() * torch.randn(g32.shape, dtype=dt32, device="cuda",
                                                     generator=torch.Generator("cuda").manual_seed(L))
    p32.forward(f32.data_ptr(), c32.data_ptr(), s)
    p32.check()
    C, G = p32.coeff_elems, p32.grid_elems
    for i in sorted({0, batch // 2, batch - 1}):
        g = torch.empty(G, dtype=dt, device="cuda")
        c = torch.empty(C, dtype=dt, device="cuda")
        f = f32[i * G:(i + 1) * G].to(dt)
        p64.inverse(F64[i * C:].data_ptr(), g.data_ptr(), s)
        p64.forward(f.data_ptr(), c.data_ptr(), s)
        torch.cuda.synchronize()
        for got, ref in ((g32[i * G:(i + 1) * G], g), (c32[i * C:(i + 1) * C], c)):
            assert torch.linalg.vector_norm(got.to(dt) - ref) <= TOL * torch.linalg.vector_norm(ref), (i, got.numel())


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,batch", [(0, 1), (1, 8192), (2, 2500), (3, 1025), (6, 200), (14, 21), (16, 14), (16, 2), (30, 3),
                                     (32, 2), (38, 2), (39, 2), (46, 3), (61, 1), (62, 2), (64, 1), (78, 1), (110, 1),
                                     (111, 1)])
def test_so3(gblib, L, batch, real):
    F = np.concatenate([so3_coeffs(L, 7 + i % 5, not real) for i in range(batch)])
    _round_trip(gblib, 1 if real else 0, real, L, batch, "tc_bf16x3", F)


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,batch", [(0, 1), (2, 30000), (5, 7300), (12, 1601), (12, 33), (30, 300), (62, 67), (96, 29),
                                     (124, 17), (125, 18), (126, 17), (128, 16), (159, 11), (190, 8), (198, 7), (199, 8),
                                     (200, 7), (230, 2)])
def test_s2(gblib, L, batch, real):
    F = np.concatenate([s2_coeffs(L, 7 + i % 5, not real) for i in range(batch)])
    _round_trip(gblib, 3 if real else 2, real, L, batch, "tc_bf16x3", F)


@pytest.mark.parametrize("real", [False, True])
def test_fp32_precision(gblib, real):
    _round_trip(gblib, 1 if real else 0, real, 21, 7, "fp32", np.tile(so3_coeffs(21, 3, not real), 7))
