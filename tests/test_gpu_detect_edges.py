"""Detection at the edges of its kernels' splits, against float64: channel counts
with and without their own instantiation, sizes and waveforms below the general
bounds, odd batch lengths, windows from none to wider than the staged halo,
positions that are not among their own neighbours, more channels than a tile
stages."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("C,F,nC,nC2,ns,nk,L,nt0,own", [
    (24, 40, 10, 12, 5, 6, 777, 20, True), (24, 33, 10, 7, 5, 6, 1025, 20, False),
    (30, 31, 7, 9, 5, 6, 640, 0, True), (12, 5, 3, 5, 2, 3, 513, 31, True),
    (12, 9, 4, 6, 8, 8, 500, 40, True), (12, 6, 10, 4, 5, 6, 3000, 700, True),
    (90, 64, 10, 20, 5, 6, 2049, 20, True), (70, 40, 6, 8, 3, 5, 1023, 33, False)])
def test_peaks_and_amplitudes(C, F, nC, nC2, ns, nk, L, nt0, own):
    from kilosort_b200 import spikedetect
    rng = np.random.default_rng(C * 31 + F)
    nt, P, th = 21, 3, 3.0
    X = rng.standard_normal((C, L)).astype(np.float32)
    iC = np.stack([rng.permutation(C)[:nC] for _ in range(F)], 1)
    if own:
        iC2 = np.stack([np.concatenate([[f], rng.integers(0, F, nC2 - 1)]) for f in range(F)], 1)
    else:
        iC2 = np.stack([(f + 1 + rng.integers(0, F - 1, nC2)) % F for f in range(F)], 1)
    weigh = rng.uniform(0.1, 1, (ns, nC, F)).astype(np.float32)
    weigh /= np.sqrt((weigh ** 2).sum(1, keepdims=True))
    wT = rng.standard_normal((nk, nt)).astype(np.float32)
    wT /= np.linalg.norm(wT, axis=1, keepdims=True)
    ops = dict(wTEMP=torch.from_numpy(wT), wPCA=torch.from_numpy(wT[:1].repeat(P, 0).copy()),
               yc=rng.uniform(0, 100, C).astype(np.float32), nt=nt, settings=dict(nt0min=nt0),
               Th_universal=th)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    det = spikedetect.Detector(ops, t(iC), t(iC2), t(weigh), torch.device(DEV))
    xy, imax, amp, _, _, _ = (a.cpu().numpy() for a in det(t(X)))
    # float64: sums, largest magnitude, pooled neighbour maximum
    B = torch.nn.functional.conv1d(torch.from_numpy(X).double()[:, None],
                                   torch.from_numpy(wT).double()[:, None], padding=nt // 2).numpy()
    A = np.einsum("sjf,jfkt->skft", weigh.astype(np.float64), B[iC]).reshape(ns * nk, F, L)
    As = np.abs(A).max(0)
    nb = As[iC2].max(0)
    nb[:, :nt] = 0
    nb[:, L - nt:] = 0
    pool = torch.nn.functional.max_pool1d(torch.from_numpy(nb)[None], 2 * nt0 + 1, stride=1,
                                          padding=nt0)[0].numpy() if nt0 <= L else None
    # the sums are chains of at most 21 + 10 fused operations on values below 10
    tol = 1e-4
    f, s = xy[:, 0], xy[:, 1]
    assert (np.diff(f * L + s) > 0).all()
    assert (np.abs(amp - As[f, s]) <= tol).all()
    assert (As[f, s] > th - tol).all() and (np.abs(As[f, s] - pool[f, s]) <= tol).all()
    top2 = np.sort(np.abs(A), 0)[-2:][:, f, s] if ns * nk > 1 else None
    clear = top2[1] - top2[0] > tol
    assert (imax[clear] == np.abs(A).argmax(0)[f, s][clear]).all()
    # every clear peak is found: the pooled maximum is its own value and nothing
    # else in the window comes near (a value near its own one elsewhere may tie)
    found = set(zip(f.tolist(), s.tolist()))
    missed = 0
    for a, b in zip(*np.nonzero((pool == As) & (As > th + tol))):
        lo, hi = max(b - nt0, nt), min(b + nt0, L - nt - 1)
        w = As[iC2[:, a], lo:hi + 1].copy()
        near = (np.abs(w - As[a, b]) <= tol).sum()
        same = (iC2[:, a] == a).sum() if lo <= b <= hi else 0
        if near <= same and (a, b) not in found:
            missed += 1
    assert missed == 0 and (len(found) > 0 or not own)


@pytest.mark.parametrize("C,F,nC,nC2,ns,nk,L,nt0", [
    (24, 34, 10, 7, 5, 6, 1025, 20), (30, 64, 7, 1, 5, 6, 2100, 0), (12, 6, 4, 9, 8, 8, 700, 40),
    (90, 66, 10, 20, 5, 6, 2049, 600)])
def test_peaks_of_positions_without_their_own_row(C, F, nC, nC2, ns, nk, L, nt0):
    """A position that is not its own neighbour peaks where a neighbour ties with
    it: every position has a twin (same channels and weights, in another tile of
    positions where there are several) as its first neighbour."""
    from kilosort_b200 import spikedetect
    rng = np.random.default_rng(C + 7 * F)
    nt, th, half = 21, 3.0, F // 2
    X = rng.standard_normal((C, L)).astype(np.float32)
    iC = np.tile(np.stack([rng.permutation(C)[:nC] for _ in range(half)], 1), 2)
    weigh = rng.uniform(0.1, 1, (ns, nC, half)).astype(np.float32)
    weigh = np.tile(weigh / np.sqrt((weigh ** 2).sum(1, keepdims=True)), 2)
    twin = (np.arange(F) + half) % F
    others = [np.setdiff1d(np.arange(F), [f, twin[f]]) for f in range(F)]
    iC2 = np.stack([np.concatenate([[twin[f]], rng.choice(others[f], nC2 - 1)]) for f in range(F)], 1)
    wT = rng.standard_normal((nk, nt)).astype(np.float32)
    wT /= np.linalg.norm(wT, axis=1, keepdims=True)
    ops = dict(wTEMP=torch.from_numpy(wT), wPCA=torch.from_numpy(wT[:1].copy()),
               yc=np.arange(C, dtype=np.float32), nt=nt, settings=dict(nt0min=nt0), Th_universal=th)
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    xy, _, amp, _ = (a.cpu().numpy() for a in spikedetect.template_match(
        t(X), ops, t(iC), t(iC2), t(weigh), torch.device(DEV)))
    B = torch.nn.functional.conv1d(torch.from_numpy(X).double()[:, None],
                                   torch.from_numpy(wT).double()[:, None], padding=nt // 2).numpy()
    As = np.abs(np.einsum("sjf,jfkt->skft", weigh.astype(np.float64), B[iC])).reshape(-1, F, L).max(0)
    As[half:] = As[:half]                # twins are the same numbers, not only close ones
    tol = 1e-4                           # as above
    f, s = xy[:, 0], xy[:, 1]
    assert (np.abs(amp - As[f, s]) <= tol).all()
    found, clear = set(zip(f.tolist(), s.tolist())), 0
    for a, b in zip(*np.nonzero(As > th + tol)):
        lo, hi = max(b - nt0, nt), min(b + nt0, L - nt - 1)
        if not lo <= b <= hi:
            continue
        w = As[iC2[:, a], lo:hi + 1]
        rest = w > As[a, b] - tol        # in the twin's column the twin alone
        rest[iC2[:, a] == twin[a], b - lo] = False
        if w.max() > As[a, b] + tol:
            assert (a, b) not in found
        elif not rest.any():
            assert (a, b) in found
            clear += 1
    assert clear > 0
