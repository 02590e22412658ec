"""Real functions on the tensor cores: one of each two conjugate (m, n) pairs is summed (GPU).

Both directions of the real kinds against the FP64 plans, over each FFT form, whose half of the pencils differs (powers of two
and the CUDA-core DFT: q, tensor-core DFT: p, line FFTs and S^2 likewise), and over the edges of the 32-function (SO(3)) and
64-function (S^2) column tiles.  Bound: 1e-6 relative in the 2-norm, the FP32-data plans' own (3e-7 in the mean).
"""
import numpy as np
import pytest

from conftest import s2_coeffs, so3_coeffs

pytestmark = pytest.mark.gpu


def _run(gblib, kind, L, b, precision, x, forward):
    import torch
    dt = torch.float64 if precision == "fp64" else torch.float32
    p = gblib.Plan(kind, L, b, precision, "stable" if kind == gblib.SO3_REAL else "reference")
    i = torch.from_numpy(np.ascontiguousarray(x).ravel()).to("cuda", dt)
    o = torch.full((b * (p.coeff_elems if forward else p.grid_elems),), float("nan"), dtype=dt, device="cuda")
    (p.forward if forward else p.inverse)(i.data_ptr(), o.data_ptr(), torch.cuda.current_stream().cuda_stream)
    p.check()
    out = o.cpu().numpy().astype(np.float64)
    del p
    return out


@pytest.mark.parametrize("family,L,b", [
    ("so3", 0, 33), ("so3", 1, 1), ("so3", 7, 31), ("so3", 7, 32), ("so3", 7, 33), ("so3", 31, 1), ("so3", 31, 33),
    ("so3", 21, 8), ("so3", 39, 2), ("so3", 40, 1), ("so3", 63, 2), ("so3", 112, 1), ("s2", 0, 65), ("s2", 1, 3), ("s2", 24, 63),
    ("s2", 24, 64), ("s2", 31, 65), ("s2", 49, 101), ("s2", 63, 2), ("s2", 130, 20)])
def test_real_pairs(gblib, family, L, b):
    kind = gblib.SO3_REAL if family == "so3" else gblib.S2_REAL
    make = so3_coeffs if family == "so3" else s2_coeffs
    F = np.stack([make(L, seed=7000 + 31 * L + i, complex_=False) for i in range(b)]).astype(np.float32)
    grid = _run(gblib, kind, L, b, "fp64", F, False).astype(np.float32)
    for x, forward in [(F, False), (grid, True)]:
        got = _run(gblib, kind, L, b, "tc_bf16x3", x, forward)
        ref = _run(gblib, kind, L, b, "fp64", x, forward)
        assert np.linalg.norm(got - ref) <= 1e-6 * np.linalg.norm(ref)
        d = np.linalg.norm((got - ref).reshape(b, -1), axis=1) / np.linalg.norm(ref.reshape(b, -1), axis=1)
        assert d.max() <= 1e-6, d
