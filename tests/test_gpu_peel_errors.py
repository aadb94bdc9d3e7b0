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


@pytest.mark.parametrize("teams", [1, 2, 8])
def test_quiet_and_overflowing_batches_in_place(teams):
    """In place (Xres = X) a batch without spikes, or with more than fit, has no
    residual pass, and its team goes straight on to the next batch in the same
    scratch, laid out for another length."""
    import kilosort_b200 as kb
    from kilosort_b200 import _lib, batched
    nt, C, K, cap = 61, 4, 70, 60
    U, W, ctc = _templates(K, C, nt)
    rec = batched.Recording(U=U, wPCA=W, ctc=ctc, Th=8.0, nt=nt, capacity=cap)
    ops = dict(Th_learned=8.0, nt=nt, max_peels=100, wPCA=W)
    lengths = [9000, 40000, 500, 62, 8191, 40000, 700, 20001, 300, 9000, 33, 12345] * 4
    X = [torch.zeros((C, L), device=DEV) if i % 3 == 0 or L < 300 else _spikes(L, C, nt, i)
         for i, L in enumerate(lengths)]
    want = [kb.run_matching(ops, x, U, ctc) for x in X]
    counts = [w[0].shape[0] for w in want]
    assert 0 in counts and max(counts) > cap and any(0 < n <= cap for n in counts)
    for _ in range(3):
        items = [(x.clone(), 0) for x in X]
        outs = [batched._Outputs(rec, C, x.shape[1], DEV, Xres=x) for x, _ in items]
        info = torch.full((len(items), 4), -9, dtype=torch.int64, device=DEV)
        ws = torch.empty(batched.workspace_size([rec], items, "fp32", teams), dtype=torch.uint8,
                         device=DEV)
        batched._launch([rec], items, outs, info, ws, "fp32", teams)
        for o, (n, status, _it, need), w, x in zip(outs, info.cpu().tolist(), want, X):
            assert need == w[0].shape[0]
            if need > cap:
                assert status == _lib.KS_ERR_OVERFLOW and torch.equal(o.Xres, x)
                continue
            assert status == _lib.KS_OK and n == need
            assert torch.equal(o.st[:n], w[0]) and torch.equal(o.amps[:n], w[1])
            assert torch.equal(o.th_amps[:n], w[2]) and torch.equal(o.Xres, w[3])
