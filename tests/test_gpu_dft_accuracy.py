"""Accuracy of the generic-N DFT passes on smooth samples with noise (GPU).

Smooth samples put most of a line into a few bins.  A systematic error of those bins, unlike rounding, is not averaged by the
sum over beta, so it shows in the forward.  Bounds: 1.15 times (one function scatters by a tenth) the relative 2-norm errors that the mixed-radix FP32 FFT of these
plans had on these samples and coefficients (given beside each), which the DFT forms are not to exceed.
"""
import numpy as np
import pytest

from conftest import so3_coeffs

pytestmark = pytest.mark.gpu


def samples(N, b, real, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    x = np.arange(N) * (2 * np.pi / N)
    n = np.arange(6)

    def waves():
        c = rng.standard_normal((2, b, 6)) / (n + 1)
        return c[0] @ np.cos(n[:, None] * x) + c[1] @ np.sin(n[:, None] * x)

    def field():
        return 0.5 * rng.standard_normal((b, N, N, N)) * 0.1 + sum(
            waves()[:, :, None, None] * waves()[:, None, :, None] * waves()[:, None, None, :] for _ in range(2))

    return field().astype(np.float32) if real else (field() + 1j * field()).astype(np.complex64)


# (l_max, batch, real, forward, inverse)
TENSOR_CORES = [(96, 1, False, 4.836e-8, 2.387e-7), (96, 1, True, 4.699e-8, 2.691e-7), (59, 1, False, 1.579e-7, 1.495e-7)]

PACKED_FP32 = [(38, 2, False, 9.860e-8, 1.432e-7), (38, 2, True, 1.053e-7, 1.747e-7), (119, 1, False, 2.052e-7, 2.033e-7),
               (119, 1, True, 2.128e-7, 2.532e-7), (159, 1, False, 2.600e-7, 2.222e-7), (159, 1, True, 3.710e-7, 2.747e-7)]


def errors(gblib, L, real, smp, F):
    import torch
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    t64, t32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    s, b = torch.cuda.current_stream().cuda_stream, len(smp)
    out = []
    for precision, dt in (("fp64", t64), ("tc_bf16x3", t32)):
        p = gblib.Plan(kind, L, b, precision, "stable")
        f = torch.from_numpy(smp).cuda().to(dt)
        c = torch.from_numpy(F).cuda().to(t32).to(dt)
        c2, g = torch.empty_like(c), torch.empty_like(f)
        p.forward(f.data_ptr(), c2.data_ptr(), s)
        p.inverse(c.data_ptr(), g.data_ptr(), s)
        p.check()
        out.append((c2.reshape(-1), g.reshape(-1)))
        del p
    return [float(torch.linalg.vector_norm(y.to(x.dtype) - x) / torch.linalg.vector_norm(x)) for x, y in zip(*out)]


@pytest.mark.parametrize("L,b,real,fwd,inv", TENSOR_CORES + PACKED_FP32)
def test_errors(gblib, L, b, real, fwd, inv):
    F = np.concatenate([so3_coeffs(L, seed=L + i, complex_=not real, decay="pow") for i in range(b)])
    e = errors(gblib, L, real, samples(2 * L + 2, b, real, L), F)
    assert e[0] <= 1.15 * fwd and e[1] <= 1.15 * inv, e


@pytest.mark.parametrize("real", [False, True])
def test_scaling_by_powers_of_two(gblib, real):
    """Samples times 2^k give coefficients times 2^k, bit for bit: the leading terms' fixed point follows the line."""
    import torch
    L, b = 59, 1
    s = torch.cuda.current_stream().cuda_stream
    f = torch.from_numpy(samples(2 * L + 2, b, real, 5)).cuda()
    f.view(b, 2 * L + 2, -1)[:, 7] = 0  # lines of zeros
    f.view(-1)[12345] *= 1e4            # and a spike
    p = gblib.Plan(gblib.SO3_REAL if real else gblib.SO3_COMPLEX, L, b, "tc_bf16x3", "stable")
    out = []
    for k in (0, 50, -50):
        c = torch.empty(b * p.coeff_elems, dtype=f.dtype, device="cuda")
        g = (f * 2.0 ** k).contiguous()
        p.forward(g.data_ptr(), c.data_ptr(), s)
        p.check()
        out.append(c * 2.0 ** -k)
    assert bool(torch.isfinite(torch.view_as_real(out[0]) if not real else out[0]).all())
    assert torch.equal(out[0], out[1]) and torch.equal(out[0], out[2])
