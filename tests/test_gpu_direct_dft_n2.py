"""The packed FP32 direct DFT of N = 2 (one folded term): l_max 0 in batches of half a million samples (GPU).

Tolerance: relative 2-norm 1e-6, the path's contract, against FP64 plans.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
@pytest.mark.parametrize("precision", ["tc_bf16x3", "fp32"])
def test_n2(gblib, precision, real):
    import torch
    b = 62500
    kind = gblib.SO3_REAL if real else gblib.SO3_COMPLEX
    t64, t32 = (torch.float64, torch.float32) if real else (torch.complex128, torch.complex64)
    s = torch.cuda.current_stream().cuda_stream
    g = torch.Generator("cuda").manual_seed(3)
    c = torch.randn(b, dtype=t32, device="cuda", generator=g)
    f = torch.randn(8 * b, dtype=t32, device="cuda", generator=g)
    out = []
    for prec, dt in (("fp64", t64), (precision, t32)):
        p = gblib.Plan(kind, 0, b, prec, "stable")
        p.set_timing(True)
        x, y = c.to(dt), f.to(dt)
        c2, f2 = torch.full_like(x, float("nan")), torch.full_like(y, float("nan"))
        p.inverse(x.data_ptr(), f2.data_ptr(), s)
        p.forward(y.data_ptr(), c2.data_ptr(), s)
        p.check()
        stages = p.stage_times()
        out.append((c2, f2))
        del p
    # the direct form: no pass that zeroes the Nyquist bins, none that transposes
    assert not [k for k in stages if "nyquist" in k or "pack" in k], stages
    for ref, got in zip(*out):
        assert float(torch.linalg.vector_norm(got.to(t64) - ref) / torch.linalg.vector_norm(ref)) <= 1e-6
