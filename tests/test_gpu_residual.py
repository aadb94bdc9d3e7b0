"""The residual pass: Xres from X, the spikes and their templates, at the edges
of its channel tiles (16), support mask (64 bits) and spike lists (32 and 64
per 32-column block), out of place, in place and through the batched launch."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
NT = 61


def _crowd(seed, C, K, P, L, n_at):
    """Templates on disjoint channel ranges and a batch with every one of them
    firing within 20 samples of one column (about K spikes meet one block),
    plus one spike at each end of the batch."""
    rng = np.random.default_rng(seed)
    t = np.arange(NT)
    W = np.linalg.qr(np.stack([np.exp(-0.5 * ((t - 20 - 3 * i) / 4.0) ** 2)
                               for i in range(P)], 1))[0].T.astype(np.float32)
    U = np.zeros((K, P, C), np.float32)
    per = C // K
    for k in range(K):
        U[k, :, k * per:(k + 1) * per] = rng.uniform(8, 14, (P, per)) * rng.choice([-1, 1], (P, 1))
    X = rng.standard_normal((C, L)).astype(np.float32)
    spikes = [(NT, 0), (L - NT - 1, 1)] + [(n_at + int(rng.integers(0, 20)), k) for k in range(K)]
    for tau, k in spikes:
        X[:, tau - NT // 2:tau + NT // 2 + 1] += (U[k].T @ W).astype(np.float32)
    return torch.from_numpy(X), torch.from_numpy(U), torch.from_numpy(W)


def _reference(X, U, W, st, amps):
    """(Xres, bound) in float64: every update's rounding (P fused sums, the
    product, the difference) is at most half an ulp of what it rounds."""
    X, U, W = (a.double().numpy() for a in (X, U, W))
    P = W.shape[0]
    err = np.zeros_like(X)
    u = 2.0 ** -24
    for (tau, k), a in zip(st.tolist(), amps.double().reshape(-1).tolist()):
        cols = slice(tau - NT // 2, tau + NT // 2 + 1)
        wave, mag = U[k].T @ W, np.abs(U[k]).T @ np.abs(W)
        X[:, cols] -= a * wave
        err[:, cols] += u * ((P + 1) * abs(a) * mag + np.abs(X[:, cols]))
    return X, 1.01 * err + 1e-12


@pytest.mark.parametrize("C,K,P", [(15, 3, 6), (17, 2, 3), (33, 4, 8), (48, 40, 6), (90, 70, 5),
                                   (1040, 80, 6), (1056, 33, 2)])
def test_residual_of_crowded_blocks(C, K, P):
    import kilosort_b200 as kb
    from kilosort_b200 import batched
    from kilosort_b200.template_matching import peel, project_scores, template_energy
    L, Th = 1500, 9.0
    X, U, W = _crowd(C * 100 + K, C, K, P, L, 700)
    Xd, Ud, Wd = (a.to(DEV) for a in (X, U, W))
    ops = dict(Th_learned=Th, nt=NT, max_peels=200, wPCA=Wd)
    ctc = kb.prepare_matching(ops, Ud)
    st, amps, _, Xres = kb.run_matching(ops, Xd, Ud, ctc, device=Xd.device)
    assert len(st) >= K and torch.equal(Xd.cpu(), X)
    want, bound = _reference(X, U, W, st.cpu(), amps.cpu())
    assert (np.abs(Xres.cpu().double().numpy() - want) <= bound).all()
    # in place (the peel's own entry point)
    B = project_scores(Xd, Ud, Wd, NT, tiled=True)
    Xi = Xd.clone()
    st2, amps2, _, _ = peel(B, Xi, Ud, Wd, ctc, template_energy(Ud), Th, NT, 200)
    assert torch.equal(st2, st) and torch.equal(Xi, Xres)
    # the batched launch, beside a batch without a spike
    rec = batched.Recording(U=Ud, wPCA=Wd, ctc=ctc, Th=Th, nt=NT, max_peels=200)
    quiet = torch.zeros((C, L - 33), device=DEV)
    got = batched.match_batches([rec], [(Xd, 0), (quiet, 0)], "fp32")
    assert torch.equal(got[0][0], st) and torch.equal(got[0][3], Xres)
    assert len(got[1][0]) == 0 and torch.equal(got[1][3], quiet)


def test_failed_batch_keeps_its_samples():
    """An overflowing batch: no result, Xres = X, and the other batches stand."""
    import kilosort_b200 as kb
    from kilosort_b200 import _lib, batched
    X, U, W = _crowd(5, 48, 40, 6, 1500, 700)
    Xd, Ud, Wd = (a.to(DEV) for a in (X, U, W))
    ops = dict(Th_learned=9.0, nt=NT, max_peels=200, wPCA=Wd)
    ctc = kb.prepare_matching(ops, Ud)
    rec = batched.Recording(U=Ud, wPCA=Wd, ctc=ctc, Th=9.0, nt=NT, max_peels=200, capacity=10)
    quiet = torch.zeros((48, 900), device=DEV)
    m = batched.BatchedMatcher([rec], [(1500, 0), (900, 0)], "fp32", teams=1, graph=False)
    m.X[0].copy_(Xd)
    m.X[1].copy_(quiet)
    m.launch()
    info = m.info.cpu()
    assert int(info[0, 1]) == _lib.KS_ERR_OVERFLOW and int(info[1, 1]) == _lib.KS_OK
    assert torch.equal(m.outs[0].Xres, Xd) and torch.equal(m.outs[1].Xres, quiet)


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_non_finite_basis_reaches_every_channel(bad):
    """The peel on given scores with a basis that is not finite at one tap: NaN at
    that tap of every spike's window, also where the template is zero."""
    import kilosort_b200 as kb
    from kilosort_b200.template_matching import peel, project_scores, template_energy
    X, U, W = (a.to(DEV) for a in _crowd(9, 48, 4, 6, 1500, 700))
    ctc = kb.prepare_matching(dict(nt=NT, wPCA=W), U)
    B = project_scores(X, U, W, NT, tiled=True)
    W = W.clone()
    W[2, 11] = bad
    st = peel(B, X, U, W, ctc, template_energy(U), 9.0, NT, 200)[0].cpu()
    assert len(st) >= 4
    hit = torch.zeros(1500, dtype=torch.bool)
    hit[st[:, 0] - NT // 2 + 11] = True
    finite = torch.isfinite(X.cpu())
    assert not finite[:, hit].any() and finite[:, ~hit].all()
