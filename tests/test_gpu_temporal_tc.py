"""The tensor-core temporal projection at the edges of its tiles (256 samples x 16
channels, 64 samples per MMA row set): the split form's scores with single-entry
templates, which pick one (channel, component) of the projection, against an
FP64 correlation.  Both operands are split in two bf16 parts each time, so a
product is off by at most 3 * 2^-16 of the sum of its terms' magnitudes plus the
FP32 accumulation (K+7 terms: 2^-24 * 128)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("C,L,P,nt", [(1, 300, 6, 61), (15, 255, 2, 1), (16, 256, 4, 41),
                                      (17, 257, 6, 61), (33, 3000, 8, 121), (40, 1153, 2, 61),
                                      (385, 63, 6, 61), (70, 40000, 6, 9)])
def test_edges_of_the_tiles(C, L, P, nt):
    from kilosort_b200.template_matching import project_scores
    rng = np.random.default_rng(C + L)
    X = rng.standard_normal((C, L)).astype(np.float32)
    W = rng.standard_normal((P, nt)).astype(np.float32)
    picks = [(c, p) for c in {0, C // 2, min(15, C - 1), C - 1} for p in (0, P - 1)]
    U = np.zeros((len(picks), P, C), np.float32)
    for k, (c, p) in enumerate(picks):
        U[k, p, c] = 1.0
    B = project_scores(*(torch.from_numpy(a).to(DEV) for a in (X, U, W)), nt,
                       projection="bf16x3").cpu().numpy()
    pad = np.zeros((C, L + nt - 1))
    pad[:, nt // 2:nt // 2 + L] = X
    eps = 3 * 2.0 ** -16 + 128 * 2.0 ** -24
    for k, (c, p) in enumerate(picks):
        ref = np.correlate(pad[c], W[p].astype(np.float64), "valid")
        mag = np.correlate(np.abs(pad[c]), np.abs(W[p]).astype(np.float64), "valid")
        # the projection, then its own split in the contraction
        assert (np.abs(B[k] - ref) <= 2 * eps * mag + 1e-30).all()
