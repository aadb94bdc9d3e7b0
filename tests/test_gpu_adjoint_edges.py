"""Reconstruction loss and adjoint at the edges of their splits: taps around the
32-tap pieces of the adjoint's lanes (and past its 128-tap form), channel
counts around its chunks and the forward's 16-channel tiles, spikes at both
ends of the batch, many at one sample and with one template, templates without
support and without spikes."""
import numpy as np
import pytest
import torch

from oracle import adjoint as oa

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _case(C, K, P, nt, L, N, seed):
    g = torch.Generator().manual_seed(seed)
    X = torch.randn((C, L), generator=g)
    U = torch.randn((K, P, C), generator=g)
    U[:, :, torch.arange(C) % 48 >= 20] = 0           # tiles without support
    U[K - 1] = 0
    W = torch.randn((P, nt), generator=g) / nt ** 0.5
    tau = torch.randint(0, L, (N,), generator=g)
    k = torch.randint(0, max(K - 1, 1), (N,), generator=g)
    tau[:4] = torch.tensor([0, L - 1, min(3, L - 1), max(L - 4, 0)])
    tau[4:4 + N // 3] = L // 2                         # one crowded sample
    k[N // 2:N // 2 + N // 4] = 0                      # one crowded template
    st = torch.stack((tau, k), 1)
    return X, U, W, st, 1 + 0.3 * torch.randn(N, generator=g)


@pytest.mark.parametrize("C,K,P,nt,L,N", [
    (1, 1, 1, 1, 40, 9), (15, 3, 2, 31, 500, 40), (17, 5, 3, 33, 700, 130), (32, 4, 6, 61, 1000, 90),
    (33, 7, 6, 61, 2049, 400), (65, 6, 8, 65, 900, 100), (64, 3, 5, 97, 800, 70),
    (31, 4, 6, 127, 1200, 66), (20, 3, 4, 129, 1200, 50), (1100, 5, 2, 41, 300, 60)])
def test_loss_and_gradients(C, K, P, nt, L, N):
    from kilosort_b200.adjoint import reconstruct, reconstruction_loss
    X, U, W, st, amps = _case(C, K, P, nt, L, N, C + nt)
    Xd, std = X.to(DEV), st.to(DEV)
    q = [t.to(DEV).requires_grad_(True) for t in (amps, U, W)]
    reconstruction_loss(Xd, std, *q).backward()
    r = [t.double().requires_grad_(True) for t in (amps, U, W)]
    want = oa.recon_loss(X.double(), st, *r)
    want.backward()
    for got, ref in zip(q, r):
        # FP32 sums of up to a few thousand terms against 64 bits: the bar of
        # the other gradient checks
        err = (got.grad.cpu().double() - ref.grad).abs().max()
        assert err <= 1e-4 * ref.grad.abs().max() + 1e-6
    Xres, loss = reconstruct(Xd, std, amps.to(DEV), U.to(DEV), W.to(DEV))
    assert abs(float(loss) - float(want)) <= 1e-5 * float(want)
    # the same values again, bit for bit
    again = [t.detach().clone().requires_grad_(True) for t in q]
    reconstruction_loss(Xd, std, *again).backward()
    assert all(torch.equal(a.grad, b.grad) for a, b in zip(q, again))


def test_non_finite_amplitude_reaches_the_loss():
    """An infinite amplitude makes its whole window NaN or infinite, also on the
    channels where its template is zero."""
    from kilosort_b200.adjoint import reconstruct
    X, U, W, st, amps = _case(40, 3, 2, 31, 300, 20, 5)
    amps[0] = float("inf")
    Xres, loss = reconstruct(*(t.to(DEV) for t in (X, st, amps, U, W)))
    assert not np.isfinite(float(loss))
    lo, hi = max(0, int(st[0, 0]) - 15), min(300, int(st[0, 0]) + 16)
    assert not torch.isfinite(Xres[:, lo:hi]).any()


def test_more_channel_chunks_than_grid_rows():
    """65 to 128 taps go in chunks of 16 channels: 65537 of them here."""
    from kilosort_b200.adjoint import reconstruction_loss
    C, K, P, nt, L = 16 * 65536 + 5, 1, 1, 65, 6
    g = torch.Generator().manual_seed(11)
    X, U = torch.randn((C, L), generator=g), torch.randn((K, P, C), generator=g)
    W = torch.randn((P, nt), generator=g) / nt ** 0.5
    st, amps = torch.tensor([[1, 0], [4, 0]]), torch.tensor([1.5, -0.5])
    q = [t.to(DEV).requires_grad_(True) for t in (amps, U, W)]
    reconstruction_loss(X.to(DEV), st.to(DEV), *q).backward()
    r = [t.double().requires_grad_(True) for t in (amps, U, W)]
    oa.recon_loss(X.double(), st, *r).backward()
    for got, ref in zip(q, r):
        err = (got.grad.cpu().double() - ref.grad).abs().max()
        assert err <= 1e-4 * ref.grad.abs().max() + 1e-6


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_non_finite_basis_reaches_every_channel(bad):
    """A tap that is not finite gives NaN also on channels where the template is
    zero (0 times it), at that tap of every spike's window and nowhere else."""
    from kilosort_b200.adjoint import reconstruct
    X, U, W, st, amps = _case(70, 3, 2, 31, 300, 20, 6)
    W[1, 7] = bad
    Xres, _ = reconstruct(*(t.to(DEV) for t in (X, st, amps, U, W)))
    hit = torch.zeros(300, dtype=torch.bool)
    at = st[:, 0] - 15 + 7
    hit[at[(at >= 0) & (at < 300)]] = True
    finite = torch.isfinite(Xres.cpu())
    assert not finite[:, hit].any() and finite[:, ~hit].all()
