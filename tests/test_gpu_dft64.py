"""The FP64 plans' passes at the sizes where their form changes, against the oracle: the direct FP64 DFT (N <= 64, and N with
a prime factor too large for the mixed radices), the mixed-radix lines otherwise, and the halves of the real kinds.

Tolerance 1e-12 relative (L2), the FP64 path's contract: sums of at most 512 terms in FP64 are within 512 * 2^-53 = 6e-14."""
import numpy as np
import pytest

from conftest import rel_err, s2_coeffs, so3_coeffs

pytestmark = pytest.mark.gpu

TOL = 1e-12


def _run(gblib, kind, L, batch, F, grids, real):
    import torch

    dt = torch.float64 if real else torch.complex128
    p = gblib.Plan(kind, L, batch, "fp64", "stable")
    s = torch.cuda.current_stream().cuda_stream
    c = torch.from_numpy(F).to(dt).cuda()
    f = torch.from_numpy(grids).to(dt).cuda()
    g, out = torch.empty(batch * p.grid_elems, dtype=dt, device="cuda"), torch.empty_like(c)
    p.inverse(c.data_ptr(), g.data_ptr(), s)
    p.forward(f.data_ptr(), out.data_ptr(), s)
    torch.cuda.synchronize()
    return out.cpu().numpy(), g.cpu().numpy()


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,batch", [(0, 3), (1, 1), (2, 2), (3, 1), (10, 2), (15, 1), (16, 1), (22, 1), (30, 1), (31, 1), (32, 1),
                                     (36, 1)])
def test_so3(gblib, oracle, L, batch, real):
    N, C = 2 * (L + 1), gblib.lib().fftso3_coeff_elems(0, L)
    F = np.concatenate([so3_coeffs(L, 3 + i, not real) for i in range(batch)])
    rng = np.random.default_rng(L)
    f = rng.standard_normal((batch, N, N, N)) + (0 if real else 1j * rng.standard_normal((batch, N, N, N)))
    out, g = _run(gblib, 1 if real else 0, L, batch, F, f.reshape(-1), real)
    for i in range(batch):
        Fi = F[i * C:(i + 1) * C]
        ref = oracle.so3_forward_real(L, f[i]) if real else oracle.so3_forward_complex(L, f[i])
        grid = oracle.so3_inverse_real_grid(L, Fi) if real else oracle.so3_inverse_complex_grid(L, Fi)
        assert rel_err(out[i * C:(i + 1) * C], ref) < TOL
        assert rel_err(g[i * N ** 3:(i + 1) * N ** 3], grid.ravel()) < TOL


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("L,batch", [(0, 2), (2, 5), (31, 3), (32, 1), (46, 2), (47, 1), (96, 1), (100, 1), (250, 1)])
def test_s2(gblib, oracle, L, batch, real):
    N, C = 2 * (L + 1), (L + 1) ** 2
    F = np.concatenate([s2_coeffs(L, 3 + i, not real) for i in range(batch)])
    rng = np.random.default_rng(L)
    f = rng.standard_normal((batch, N, N)) + (0 if real else 1j * rng.standard_normal((batch, N, N)))
    out, g = _run(gblib, 3 if real else 2, L, batch, F, f.reshape(-1), real)
    for i in range(batch):
        Fi = F[i * C:(i + 1) * C]
        ref = oracle.s2_forward_real(L, f[i]) if real else oracle.s2_forward_complex(L, f[i])
        grid = oracle.s2_inverse_real_grid(L, Fi) if real else oracle.s2_inverse_complex_grid(L, Fi)
        assert rel_err(out[i * C:(i + 1) * C], ref) < TOL
        assert rel_err(g[i * N * N:(i + 1) * N * N], grid.ravel()) < TOL
