"""Template cross-correlations at the edges of their tiles (16 templates per
group, 128 lags per thread group, the Gram's 128 x 256 tiles and its diagonal)
against float64: a value is a chain of P^2 fused operations on Gram entries that
are chains of C, so its error is at most (C + nt + P^2) 2^-24 times the sum of
its terms' magnitudes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ctc64(U, W):
    K, P, C = U.shape
    nt = W.shape[1]
    WtW = torch.nn.functional.conv1d(W[:, None], W[:, None], padding=nt).flip(2)
    G = torch.einsum("ikc,jmc->ijkm", U, U)
    return torch.einsum("ijkm,kml->ijl", G, WtW)


@pytest.mark.parametrize("K,P,C,nt", [(1, 1, 3, 1), (15, 3, 20, 21), (16, 6, 33, 61), (17, 6, 40, 61),
                                      (33, 6, 12, 63), (45, 2, 20, 129), (100, 6, 24, 41),
                                      (43, 16, 8, 5), (200, 6, 50, 9)])
def test_ctc_within_the_chain_bound(K, P, C, nt):
    import kilosort_b200 as kb
    g = torch.Generator(device=DEV).manual_seed(K + 100 * P)
    U = torch.randn((K, P, C), generator=g, device=DEV)
    W = torch.randn((P, nt), generator=g, device=DEV)
    got = kb.prepare_matching(dict(nt=nt, wPCA=W), U).double()
    size = _ctc64(U.double().abs(), W.double().abs())
    err = (got - _ctc64(U.double(), W.double())).abs()
    assert (err <= (C + nt + P * P + 2) * 2.0 ** -24 * size + 1e-30).all()
