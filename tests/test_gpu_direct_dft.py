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


@pytest.mark.parametrize("real", [False, True])
def test_uneven_batch(gblib, real):
    """Both passes of every bucket in one launch (two million samples or more): the smallest N, powers of two (whose plans
    keep no work grid), primes and the largest N of the one-launch form; two calls on different buffers, from graphs."""
    import torch

    ls = [1, 2, 7, 15, 16, 31, 31, 36, 39, 47, 52, 63] + ([70, 105] if real else [77])
    kind = 1 if real else 0
    dt, dt32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    b = gblib.Batch(kind, ls, "tc_bf16x3", "stable", gblib.FLAG_GRAPH)
    assert b.grid_elems >= 2000000
    s = torch.cuda.current_stream().cuda_stream
    for call in range(2):
        F = torch.empty(b.coeff_elems, dtype=dt32, device="cuda")
        for i, L in enumerate(ls):
            c = torch.from_numpy(so3_coeffs(L, 11 + i + 50 * call, not real)).to(dt32).cuda()
            F[b.coeff_offset(i):b.coeff_offset(i) + c.numel()] = c
        g, F2 = torch.empty(b.grid_elems, dtype=dt32, device="cuda"), torch.empty_like(F)
        b.inverse(F.data_ptr(), g.data_ptr(), s)
        f = g + 0.1 * g.abs().mean() * torch.randn(g.shape, dtype=dt32, device="cuda")
        b.forward(f.data_ptr(), F2.data_ptr(), s)
        b.check()
        assert b.graph_kernels(0) == 3 and b.graph_kernels(1) == 3
        for i, L in enumerate(ls):
            p = gblib.Plan(kind, L, 1, "fp64", "stable")
            cs, gs = slice(b.coeff_offset(i), b.coeff_offset(i) + p.coeff_elems), slice(b.grid_offset(i), b.grid_offset(i) + p.grid_elems)
            g64, c64 = torch.empty(p.grid_elems, dtype=dt, device="cuda"), torch.empty(p.coeff_elems, dtype=dt, device="cuda")
            F64, f64 = F[cs].to(dt), f[gs].to(dt)
            p.inverse(F64.data_ptr(), g64.data_ptr(), s)
            p.forward(f64.data_ptr(), c64.data_ptr(), s)
            torch.cuda.synchronize()
            for got, ref in ((g[gs], g64), (F2[cs], c64)):
                assert torch.linalg.vector_norm(got.to(dt) - ref) <= TOL * torch.linalg.vector_norm(ref), (call, L)
