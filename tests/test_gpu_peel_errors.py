"""Errors that the peel's blocks find on the device: the call reports the first
one, every block leaves, and the next call is not affected."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _templates(K, C, nt):
    import kilosort_b200 as kb
    W = torch.full((1, nt), nt ** -0.5, device=DEV)
    U = torch.zeros((K, 1, C), device=DEV)
    for k in range(K):
        U[k, 0, k % C] = 1.0
    return U, W, kb.prepare_matching(dict(nt=nt, wPCA=W), U)


def _spikes(L, C, nt, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    X = torch.randn((C, L), generator=g, device=DEV)
    for i, t in enumerate(range(2 * nt, L - 2 * nt, 5 * nt)):
        X[i % C, t - nt // 2:t + nt // 2 + 1] += 6.0
    return X


@pytest.mark.parametrize("L,K", [(400, 1), (5000, 3), (60122, 40)])
def test_plateau_is_reported_and_forgotten(L, K):
    """A constant batch scores the same at every sample: more peaks touch a block
    than its list holds (KS_ERR_DEGENERATE, recorded by many threads at once)."""
    import kilosort_b200 as kb
    from kilosort_b200 import _lib
    nt, C = 61, 4
    U, W, ctc = _templates(K, C, nt)
    ops = dict(Th_learned=8.0, nt=nt, max_peels=100, wPCA=W)
    good = _spikes(L, C, nt, L)
    want = kb.run_matching(ops, good, U, ctc)
    assert want[0].shape[0] > 0
    for _ in range(3):
        with pytest.raises(_lib.KilosortB200Error) as e:
            kb.run_matching(ops, torch.full((C, L), 10.0, device=DEV), U, ctc)
        assert e.value.status == _lib.KS_ERR_DEGENERATE
        got = kb.run_matching(ops, good, U, ctc)
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("teams", [1, 2, 5])
def test_plateau_in_one_batch_of_several(teams):
    import kilosort_b200 as kb
    from kilosort_b200 import _lib, batched
    nt, C, K = 61, 4, 40
    U, W, ctc = _templates(K, C, nt)
    rec = batched.Recording(U=U, wPCA=W, ctc=ctc, Th=8.0, nt=nt)
    good = [_spikes(L, C, nt, L) for L in (9000, 4000, 700, 3000)]
    with pytest.raises(_lib.KilosortB200Error) as e:
        batched.match_batches([rec], [(x, 0) for x in [torch.full((C, 20000), 10.0, device=DEV)] + good],
                              "fp32", teams=teams)
    assert e.value.status == _lib.KS_ERR_DEGENERATE
    ops = dict(Th_learned=8.0, nt=nt, max_peels=100, wPCA=W)
    for x, got in zip(good, batched.match_batches([rec], [(x, 0) for x in good], "fp32",
                                                  teams=teams)):
        want = kb.run_matching(ops, x, U, ctc)
        assert all(torch.equal(a, b) for a, b in zip(got, want))
