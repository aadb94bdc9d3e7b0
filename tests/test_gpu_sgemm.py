"""The FP32 score contraction at the edges of its tiles (64, 96 and 128 template
rows, 128 and 256 samples) against float64: every score is one chain of Q fused
operations, so its error is at most Q 2^-24 times the sum of its terms'
magnitudes (the temporal projection's own chain added)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("K,L", [(1, 130), (63, 300), (64, 1000), (65, 257), (80, 129), (96, 511),
                                 (97, 256), (128, 128), (129, 3000), (193, 255), (600, 20001),
                                 (533, 33333), (1000, 1025)])
@pytest.mark.parametrize("tiled", [False, True])
def test_scores_within_the_chain_bound(K, L, tiled):
    from kilosort_b200.template_matching import project_scores
    C, P, nt = 20, 6, 21
    g = torch.Generator(device=DEV).manual_seed(K * 7 + L)
    X = torch.randn((C, L), generator=g, device=DEV)
    U = torch.randn((K, P, C), generator=g, device=DEV)
    W = torch.randn((P, nt), generator=g, device=DEV)
    B = project_scores(X, U, W, nt, projection="fp32", tiled=tiled)
    if tiled:
        pad = B[-1, :, L - (B.shape[0] - 1) * 32:]
        assert (pad == 0).all()
        B = B.permute(1, 0, 2).reshape(K, -1)[:, :L]

    def scores(X, U, W):
        Y = torch.stack([torch.nn.functional.conv1d(X.double()[:, None], W.double()[p:p + 1, None],
                                                    padding=nt // 2)[:, 0] for p in range(P)], 1)
        return U.double().permute(0, 2, 1).reshape(K, -1) @ Y.reshape(C * P, L)

    want, size = scores(X, U, W), scores(X.abs(), U.abs(), W.abs())
    assert ((B.double() - want).abs() <= (C * P + nt + 2) * 2.0 ** -24 * size).all()


@pytest.mark.parametrize("K,L", [(130, 60122), (160, 40000), (192, 47500), (385, 60122), (400, 25000)])
def test_tile_shape_does_not_change_a_score(K, L):
    """96-row heights and 256-column tiles on both sides of the line between them:
    a template's scores are those of the call with 64 templates, bit for bit."""
    from kilosort_b200.template_matching import project_scores
    g = torch.Generator(device=DEV).manual_seed(K)
    X = torch.randn((5, L), generator=g, device=DEV)
    U = torch.randn((K, 6, 5), generator=g, device=DEV)
    W = torch.randn((6, 21), generator=g, device=DEV)
    B = project_scores(X, U, W, 21, projection="fp32")
    for k in range(0, K, 64):
        part = project_scores(X, U[k:k + 64].contiguous(), W, 21, projection="fp32")
        assert torch.equal(part, B[k:k + 64])
