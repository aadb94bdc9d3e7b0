"""Batches with more 256-sample tiles than a launch has rows of blocks (65535)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("C,tiles", [(1, 65536), (2, 65535 + 300)])
def test_centring_of_a_long_batch(cuda_device, C, tiles):
    """Exact: one rounding of the double mean, one of the difference."""
    from kilosort_b200.preprocess import Preprocessor
    L = 256 * tiles - 100
    raw = np.random.default_rng(C).integers(-2000, 3000, (L, C), dtype=np.int16)
    p = Preprocessor(C, L, whiten=None, hp_filter=None, do_CAR=False,
                     artifact_threshold=float("inf"), device=cuda_device)
    got = p(torch.from_numpy(raw).to(cuda_device)).cpu().numpy()
    x = raw.T.astype(np.float32)
    mean = (raw.astype(np.int64).sum(0) / L).astype(np.float32)
    assert np.array_equal(got, x - mean[:, None])
