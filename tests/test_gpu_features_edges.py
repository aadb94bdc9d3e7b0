"""Spike features at the edges of the kernel's groups (4 channels, 8 components, 32
taps per step) against FP64.  A feature is a sum of nt products in FP32 (at most
ceil(nt/32) + 5 roundings deep) plus one rounded product: the error is within
(nt/32 + 8) * 2^-24 of the sum of the magnitudes."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("P,nt,nC,N", [(6, 61, 10, 500), (1, 1, 1, 1), (8, 64, 4, 9), (3, 65, 5, 33),
                                       (8, 151, 7, 100), (5, 33, 12, 8)])
def test_against_double(cuda_device, P, nt, nC, N):
    import kilosort_b200 as kb
    rng = np.random.default_rng(P * 100 + nt)
    C, L, K = 20, 2000, 11
    X = rng.standard_normal((C, L)).astype(np.float32)
    W = rng.standard_normal((P, nt)).astype(np.float32)
    st = np.stack([rng.integers(nt // 2, L - nt, N), rng.integers(0, K, N)], 1)
    amps = rng.uniform(5, 20, N).astype(np.float32)
    iCC = np.stack([rng.permutation(C)[:nC] for _ in range(C)], 1).astype(np.int64)   # [nC, C]
    iU = rng.integers(0, C, K)
    Ucc = rng.standard_normal((nC, K, P)).astype(np.float32)
    got = kb.spike_features(*(torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
                              for a in (X, st, amps, W, iCC, iU, Ucc))).cpu().numpy()
    Wd, Xd = W.astype(np.float64), X.astype(np.float64)
    for s, (t, k) in enumerate(st):
        win = Xd[iCC[:, iU[k]], t - nt // 2:t - nt // 2 + nt]            # [nC, nt]
        u = Ucc[:, k].astype(np.float64) * float(amps[s])
        ref, mag = win @ Wd.T + u, np.abs(win) @ np.abs(Wd).T + np.abs(u)
        assert (np.abs(got[s] - ref) <= (nt / 32 + 8) * 2.0 ** -24 * mag).all()


@pytest.mark.parametrize("P,nt,N", [(1, 31, 5), (6, 61, 300), (5, 95, 20), (8, 129, 9)])
def test_one_channel_alone(cuda_device, P, nt, N):
    """A single channel has its own form: the same bits as beside others."""
    import kilosort_b200 as kb
    g = torch.Generator(device=DEV).manual_seed(P)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    C, L, K, nC = 9, 1500, 5, 6
    st = torch.stack([torch.randint(nt, L - nt, (N,), generator=g, device=DEV),
                      torch.randint(0, K, (N,), generator=g, device=DEV)], 1)
    iCC = torch.randint(0, C, (nC, C), generator=g, device=DEV)
    args = rnd(C, L), st, rnd(N), rnd(P, nt)
    iU, Ucc = torch.randint(0, C, (K,), generator=g, device=DEV), rnd(nC, K, P)
    want = kb.spike_features(*args, iCC, iU, Ucc)
    for i in range(nC):
        got = kb.spike_features(*args, iCC[i:i + 1].contiguous(), iU, Ucc[i:i + 1].contiguous())
        assert torch.equal(got, want[:, i:i + 1])
