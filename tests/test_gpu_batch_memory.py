"""Device memory of the tensor-core DFT of uneven batches (GPU): work grids of the pencils that it moves, no more."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("real", [False, True])
def test_work_grids(gblib, monkeypatch, real):
    """Complex 8 bytes a sample; real functions half of that and one row of bins."""
    lmax = [63] * 8 + [127]
    size = {}
    for phases in ("0", "1"):
        monkeypatch.setenv("FFTSO3_BATCH_PHASES", phases)
        b = gblib.Batch(gblib.SO3_REAL if real else gblib.SO3_COMPLEX, lmax, "tc_bf16x3", "stable", 0)
        size[phases] = b.device_bytes
        del b
    # (the bucket of l_max 127 has no tensor-core DFT: N > 222)
    assert size["1"] == size["0"]
    lmax = [63] * 16
    for phases in ("0", "1"):
        monkeypatch.setenv("FFTSO3_BATCH_PHASES", phases)
        b = gblib.Batch(gblib.SO3_REAL if real else gblib.SO3_COMPLEX, lmax, "tc_bf16x3", "stable", 0)
        size[phases], samples = b.device_bytes, b.grid_elems
        del b
    bins = samples * (65 / 128 if real else 1)
    assert 8 * bins <= size["1"] - size["0"] <= 8 * bins + (1 << 20)
