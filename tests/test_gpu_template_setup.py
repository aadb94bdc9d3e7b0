"""The template set-up of a matching call (energies, group order, bounds, in
one kernel per step) and the transpose of the cross-correlations, at odd sizes:
both move or compute the values of the separate entry points bit for bit."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("K,nt", [(1, 1), (3, 61), (8, 63), (9, 65), (37, 61), (65, 151)])
def test_transpose_moves_every_row(K, nt):
    from kilosort_b200.template_matching import transpose_ctc
    g = torch.Generator().manual_seed(K * 1000 + nt)
    a = torch.randn(K, K, 2 * nt + 1, generator=g).to(DEV)
    assert torch.equal(transpose_ctc(a, nt), a.transpose(0, 1))


@pytest.mark.parametrize("K,C,P,scale", [(1, 1, 1, 1.0), (31, 15, 8, 1.0), (33, 257, 6, 1e-4),
                                         (70, 385, 3, 1e3)])
def test_set_up_of_a_call_equals_the_separate_steps(K, C, P, scale):
    """A whole call against projection, energies and peel called in turn (the peel
    reads the energies there)."""
    import kilosort_b200 as kb
    from kilosort_b200.template_matching import peel, project_scores, run_matching, template_energy
    nt = 61
    rng = np.random.default_rng(K + C)
    W = np.ascontiguousarray(np.linalg.qr(rng.standard_normal((nt, P)))[0].T, np.float32)
    W = torch.from_numpy(W).to(DEV)
    U = torch.from_numpy(rng.standard_normal((K, P, C)).astype(np.float32) * scale).to(DEV)
    U[K // 2, :, C // 2 + 1:] = 0
    X = torch.from_numpy(rng.standard_normal((C, 3000)).astype(np.float32)).to(DEV)
    for k in range(0, K, 3):                    # planted: a few spikes of every third template
        w = torch.einsum("pc,pt->ct", U[k], W)
        for t in rng.integers(100, 2800, 4):
            X[:, t:t + nt] += w * (20.0 / float(U[k].norm()))
    ops = dict(nt=nt, wPCA=W, max_peels=40, Th_learned=6.0)
    ctc = kb.prepare_matching(ops, U)
    nm = template_energy(U)
    B = project_scores(X, U, W, nt, tiled=True)
    Xres = X.clone()
    st, amps, th, _ = peel(B, Xres, U, W, ctc, nm, 6.0, nt, 40)
    got = run_matching(ops, X, U, ctc)
    assert len(st) > 0
    assert torch.equal(got[0], st) and torch.equal(got[1], amps)
    assert torch.equal(got[2], th) and torch.equal(got[3], Xres)
