"""The grouped update against the ungrouped one (ks_peel_static, every row of a
touched column rewritten): spikes, amplitudes, scores and residual identical at
the edges of the groups (32 templates), blocks (32 columns), detection chunks
(256 columns, by warps or by blocks) and of the score comparison's range."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _inputs(K, NT, nt, P, scale, seed):
    import kilosort_b200 as kb
    from kilosort_b200 import synth
    from kilosort_b200.template_matching import project_scores, template_energy
    rec = synth.make_recording(seed, n_chan=24, probe="np1", n_templates=K, nt=nt, n_pcs=P,
                               t_trough=nt // 3, batch_lengths=[NT], rate_hz=(20.0, 60.0))
    U = rec.U.copy()
    if scale:                       # energies outside [2^-30, 2^30], a template without energy
        U[::3] *= 1e-7
        U[1::5] *= 1e6
        U[K // 2] = 0
    X, Ud, W = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
                for a in (rec.batch(0), U, rec.wPCA))
    ctc = kb.prepare_matching(dict(nt=nt, wPCA=W), Ud)
    return X, Ud, W, ctc, template_energy(Ud), project_scores(X, Ud, W, nt, tiled=True)


@pytest.mark.parametrize("K,NT,nt,P,scale", [
    (1, 700, 61, 6, False), (5, 512, 61, 6, True), (31, 3000, 61, 6, False),
    (32, 2977, 41, 4, False), (33, 3001, 61, 6, True), (65, 6000, 63, 5, False),
    (70, 70000, 61, 6, False), (480, 2500, 61, 6, False), (40, 2000, 129, 6, False),
    (40, 2000, 401, 3, True)])
def test_grouped_update_equals_ungrouped(K, NT, nt, P, scale):
    from kilosort_b200 import _lib
    from kilosort_b200.template_matching import peel, transpose_ctc
    X, U, W, ctc, nm, B = _inputs(K, NT, nt, P, scale, 1000 + K + nt)
    C, L = X.shape
    Bs, Xs = B.clone(), X.clone()
    cap = 20000
    st = torch.zeros((cap, 2), dtype=torch.int64, device=DEV)
    amps, th = torch.zeros((cap, 1), device=DEV), torch.zeros((cap, 1), device=DEV)
    info = torch.zeros(4, dtype=torch.int64, device=DEV)
    lib = _lib.load()
    _lib.check(lib.ks_peel_static(Bs.data_ptr(), Xs.data_ptr(), U.data_ptr(), W.data_ptr(),
                                  transpose_ctc(ctc, nt).data_ptr(), nm.data_ptr(), C, L, K, P, nt,
                                  49.0, 100, cap, st.data_ptr(), amps.data_ptr(), th.data_ptr(),
                                  info.data_ptr(), torch.cuda.current_stream().cuda_stream),
               "ks_peel_static")
    n, status = int(info[0]), int(info[1])
    assert status == 0 and n > 0
    got = peel(B, X, U, W, ctc, nm, 7.0, nt, 100, capacity=cap)
    assert torch.equal(got[0], st[:n]) and torch.equal(got[1], amps[:n])
    assert torch.equal(got[2], th[:n]) and torch.equal(B, Bs) and torch.equal(X, Xs)


@pytest.mark.parametrize("teams", [1, 3, 12])
def test_teams_equal_single_batches(teams):
    """Large and small teams (detection by blocks and by warps, units dealt and
    claimed) against one run_matching per batch."""
    import kilosort_b200 as kb
    from kilosort_b200 import batched
    X, U, W, ctc, _, _ = _inputs(96, 40000, 61, 6, False, 77)
    ops = dict(Th_learned=7.0, nt=61, max_peels=100, wPCA=W)
    Xs = [X[:, :n].contiguous() for n in (40122, 1000, 31, 20001, 256, 257, 40122, 5000, 40000,
                                          39999, 12345, 122)]
    rec = batched.Recording(U=U, wPCA=W, ctc=ctc, Th=7.0, nt=61)
    out = batched.match_batches([rec], [(x, 0) for x in Xs], "fp32", teams=teams)
    for x, got in zip(Xs, out):
        want = kb.run_matching(ops, x, U, ctc, device=x.device)
        assert all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("e", [30, 44, 47, 50, 53, 56, 58, 60, 62, 64])
@pytest.mark.parametrize("spread", [False, True])
def test_scores_at_the_end_of_the_range(e, spread):
    """Scores whose squares pass through the end of FP32's range (some rows' are
    infinite, others' are not, whatever their order by b/sqrt(nm)), with template
    energies close together and spread over most of 2^-30 .. 2^30."""
    from kilosort_b200 import _lib
    from kilosort_b200.template_matching import peel, project_scores, template_energy, transpose_ctc
    import kilosort_b200 as kb
    K, NT, nt, P = 70, 1500, 61, 6
    X, U, W, _, _, _ = _inputs(K, NT, nt, P, False, 4000 + e)
    if spread:
        g = torch.Generator(device=DEV).manual_seed(e + 100)
        U = U * torch.exp2(19 * torch.rand((K, 1, 1), generator=g, device=DEV) - 11)
    X = torch.ldexp(X, torch.tensor(e, device=DEV)).contiguous()
    ctc, nm = kb.prepare_matching(dict(nt=nt, wPCA=W), U), template_energy(U)
    assert 2.0 ** -30 <= nm.min() and nm.max() <= 2.0 ** 30
    B = project_scores(X, U, W, nt, tiled=True)
    (C, L), cap, th = X.shape, 60000, 2.0 ** e
    Bs, Xs = B.clone(), X.clone()
    st = torch.zeros((cap, 2), dtype=torch.int64, device=DEV)
    amps, tha = torch.zeros((cap, 1), device=DEV), torch.zeros((cap, 1), device=DEV)
    info = torch.zeros(4, dtype=torch.int64, device=DEV)
    th2 = min(th * th, 1e38)
    lib = _lib.load()
    _lib.check(lib.ks_peel_static(Bs.data_ptr(), Xs.data_ptr(), U.data_ptr(), W.data_ptr(),
                                  transpose_ctc(ctc, nt).data_ptr(), nm.data_ptr(), C, L, K, P, nt,
                                  th2, 6, cap, st.data_ptr(), amps.data_ptr(), tha.data_ptr(),
                                  info.data_ptr(), torch.cuda.current_stream().cuda_stream),
               "ks_peel_static")
    n, status = int(info[0]), int(info[1])
    assert status == 0
    got = peel(B, X, U, W, ctc, nm, th2 ** 0.5, nt, 6, capacity=cap)
    same = lambda a, b: torch.equal(torch.nan_to_num(a), torch.nan_to_num(b))
    assert torch.equal(got[0], st[:n]) and same(got[1], amps[:n]) and same(got[2], tha[:n])
    assert same(B, Bs) and same(X, Xs)
