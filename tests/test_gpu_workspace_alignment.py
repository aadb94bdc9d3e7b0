"""Entry points that align their workspace themselves: with one that starts 8 bytes
off a 16-byte boundary they give what they give with an aligned one."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _workspace(nbytes, off):
    """(tensor, address) of exactly nbytes from `off` past a 256-byte boundary,
    behind and before bytes that no call may change."""
    buf = torch.full((nbytes + 512,), 0xA5, dtype=torch.uint8, device=DEV)
    at = 256 + off
    assert buf.data_ptr() % 256 == 0
    return buf, buf.data_ptr() + at, lambda: bool((buf[:at] == 0xA5).all() and
                                                  (buf[at + nbytes:] == 0xA5).all())


@pytest.mark.parametrize("K,NT", [(5, 512), (40, 9000), (70, 30000)])
def test_peel(K, NT):
    import kilosort_b200 as kb
    from kilosort_b200 import _lib, synth
    from kilosort_b200.template_matching import project_scores, template_energy, transpose_ctc
    nt, P = 61, 6
    rec = synth.make_recording(K, n_chan=24, probe="np1", n_templates=K, nt=nt, n_pcs=P,
                               t_trough=20, batch_lengths=[NT], rate_hz=(20.0, 60.0))
    X, U, W = (torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
               for a in (rec.batch(0), rec.U, rec.wPCA))
    ctcT = transpose_ctc(kb.prepare_matching(dict(nt=nt, wPCA=W), U), nt)
    B, nm, cap = project_scores(X, U, W, nt, tiled=True), template_energy(U), 20000
    (C, L), lib, res = X.shape, _lib.load(), []
    for off in (0, 8):
        Bo, Xo = B.clone(), X.clone()
        st = torch.zeros((cap, 2), dtype=torch.int64, device=DEV)
        amps, th = torch.zeros(cap, device=DEV), torch.zeros(cap, device=DEV)
        info = torch.zeros(4, dtype=torch.int64, device=DEV)
        n = lib.ks_peel_workspace_size(L, K, nt, _lib.KS_B_TILED, _lib.KS_CTC_KJL)
        buf, ws, intact = _workspace(n, off)
        _lib.check(lib.ks_peel(Bo.data_ptr(), 0, _lib.KS_B_TILED, Xo.data_ptr(), U.data_ptr(),
                               W.data_ptr(), ctcT.data_ptr(), _lib.KS_CTC_KJL, nm.data_ptr(), C, L,
                               K, P, nt, 49.0, 100, cap, st.data_ptr(), amps.data_ptr(),
                               th.data_ptr(), info.data_ptr(), ws, n,
                               torch.cuda.current_stream().cuda_stream), "ks_peel")
        assert info[1] == 0 and info[0] > 0 and intact()
        res.append((Bo, Xo, st, amps, th, info))
    assert all(torch.equal(a, b) for a, b in zip(*res))


@pytest.mark.parametrize("C,K,P,nt,L,N", [(5, 3, 2, 31, 300, 7), (40, 33, 6, 61, 3000, 501)])
def test_reconstruction(C, K, P, nt, L, N):
    from kilosort_b200 import _lib
    g = torch.Generator(device=DEV).manual_seed(N)
    rnd = lambda *s: torch.randn(s, generator=g, device=DEV)
    X, U, W, amps, one = rnd(C, L), rnd(K, P, C), rnd(P, nt), rnd(N), torch.ones(1, device=DEV)
    st = torch.stack([torch.randint(0, n, (N,), generator=g, device=DEV) for n in (L, K)], 1)
    lib, res, s = _lib.load(), [], torch.cuda.current_stream().cuda_stream
    for off in (0, 8):
        n = lib.ks_recon_workspace_size(C, L, K, P, nt, N)
        buf, ws, intact = _workspace(n, off)
        Xres, dU, dW, da = (torch.zeros_like(t) for t in (X, U, W, amps))
        loss = torch.zeros(1, dtype=torch.float64, device=DEV)
        status = torch.full((2,), -1, dtype=torch.int32, device=DEV)
        args = (st.data_ptr(), amps.data_ptr(), N, U.data_ptr(), W.data_ptr(), C, L, K, P, nt)
        _lib.check(lib.ks_recon_loss(X.data_ptr(), *args, Xres.data_ptr(), loss.data_ptr(),
                                     status.data_ptr(), ws, n, s), "ks_recon_loss")
        _lib.check(lib.ks_recon_adjoint(Xres.data_ptr(), *args, one.data_ptr(), dU.data_ptr(),
                                        dW.data_ptr(), da.data_ptr(), status[1:].data_ptr(), ws, n,
                                        s), "ks_recon_adjoint")
        assert status.tolist() == [0, 0] and intact()
        res.append((Xres, loss, dU, dW, da))
    assert all(torch.equal(a, b) for a, b in zip(*res))
