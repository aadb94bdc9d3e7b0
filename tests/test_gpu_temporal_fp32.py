"""The FP32 temporal projection at the edges of its tiles (128 samples x 16 channels,
taps in groups of 8, components in pairs): scores of single-entry templates, which
pick one (channel, component), against an FP64 correlation.  A score is nt fused
multiply-adds and sums with exact zeros: within nt * 2^-24 of the sum of the terms'
magnitudes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("C,L,P,nt", [(1, 300, 1, 1), (15, 127, 3, 7), (16, 128, 6, 61),
                                      (17, 129, 5, 15), (33, 1000, 8, 121), (40, 1153, 7, 9),
                                      (70, 63, 2, 61), (20, 5000, 8, 1023)])
def test_edges_of_the_tiles(cuda_device, C, L, P, nt):
    from kilosort_b200.template_matching import project_scores
    rng = np.random.default_rng(C + L)
    X = rng.standard_normal((C, L)).astype(np.float32)
    W = rng.standard_normal((P, nt)).astype(np.float32)
    picks = [(c, p) for c in {0, C // 2, min(15, C - 1), C - 1} for p in range(P)]
    U = np.zeros((len(picks), P, C), np.float32)
    for k, (c, p) in enumerate(picks):
        U[k, p, c] = 1.0
    B = project_scores(*(torch.from_numpy(a).to(DEV) for a in (X, U, W)), nt,
                       projection="fp32").cpu().numpy()
    pad = np.zeros((C, L + nt - 1))
    pad[:, nt // 2:nt // 2 + L] = X
    for k, (c, p) in enumerate(picks):
        ref = np.correlate(pad[c], W[p].astype(np.float64), "valid")
        mag = np.correlate(np.abs(pad[c]), np.abs(W[p]).astype(np.float64), "valid")
        assert (np.abs(B[k] - ref) <= nt * 2.0 ** -24 * mag + 1e-30).all()
