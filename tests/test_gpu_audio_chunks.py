"""vs_audio's block scan at the edges of its runs (16 samples), warps and chunks (8192 samples): the
serial recursion's samples to the float32 rounding of values in [-1, 1] (one ulp, 2^-23, either way)."""
import numpy as np
import pytest

import audio_oracle as OA
import vocalsim_b200.audio as VA

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mul", [2, 15])
@pytest.mark.parametrize("n", [1, 15, 17, 512, 8191, 8192, 8193, 24600])
def test_lengths_at_run_and_chunk_edges(n, mul, cuda_ok):
    rng = np.random.default_rng(n + mul)
    x = rng.standard_normal((2, n)).astype(np.float32)
    got = VA.audio(x, mul).cpu().numpy()
    for i in range(2):
        assert np.max(np.abs(got[i] - OA.audio(x[i], mul))) <= 2.0 ** -22


def test_nan_reaches_every_later_sample_and_no_earlier_one(cuda_ok):
    x = np.random.default_rng(3).standard_normal(20000).astype(np.float32)
    x[9000] = np.nan
    got = VA.audio(x, 2).cpu().numpy().ravel()
    assert np.all(np.isfinite(got[:4500])) and np.all(np.isnan(got[4500:]))


@pytest.mark.parametrize("mul", [30, 64])
@pytest.mark.parametrize("n", [17, 8193, 24600])
def test_large_decimations(n, mul, cuda_ok):
    """The scan's own error grows with srate_mul, to 4e-12 at 64: still the float32 rounding's tolerance."""
    rng = np.random.default_rng(n + mul)
    x = rng.standard_normal((2, n)).astype(np.float32)
    got = VA.audio(x, mul).cpu().numpy()
    for i in range(2):
        assert np.max(np.abs(got[i] - OA.audio(x[i], mul))) <= 2.0 ** -22
