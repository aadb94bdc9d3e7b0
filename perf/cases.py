"""Performance cases of the template-matching framework.

Each case is one pass through a public entry point of ``kilosort_b200`` as a
spike-sorting program calls it, on synthetic recordings drawn on the device
from the generative model of ``kilosort_b200.synth`` (probe geometries,
biphasic waveforms on Gaussian footprints, the SVD basis, N(0, 1) noise,
Poisson trains with a refractory period; every spike's amplitude varies by a
few per cent, as in real units).  The kinds:

* ``match``     ``run_matching`` on one padded batch (the drop-in call)
* ``batches``   a ``BatchedMatcher`` over resident batches of one recording
* ``uneven``    ``match_batches`` over batches of several recordings
* ``extract``   the drop-in ``extract`` from an int16 file to host arrays
* ``detect``    universal-template detection of one batch (``Detector``)
* ``filter``    the batch filter of one raw int16 batch (``Preprocessor``)
* ``prepare``   ``prepare_matching`` (template cross-correlations)
* ``adjoint``   ``reconstruction_loss`` forward and backward
* ``features``  per-spike PC features of one matched batch

Spikes are collected in arrays that the program allocates once, with room for
more than the recording holds, as the reference's own loop does (rows past the
count stay zero).

``listed()`` gives the cases, ``draw(rng)`` one more of the same ranges;
``prepare(case, seed)`` builds what a program holds before the call,
``run(state)`` makes one pass, ``work(case)`` says what a pass cannot do
without and ``exact(case, seed)`` gives the outputs in 64 bits by plain torch.
"""
import math

import numpy as np
import torch

from kilosort_b200 import synth

DEV = "cuda"
FS = 30000.0
TROUGH = 20          # sample of the waveform trough (nt0min)
TH = 8.0             # Th_learned
MAX_PEELS = 100


def listed():
    return [
        # the smallest calls: a tetrode-sized group or a short snippet of a
        # small probe, where launches and latency are what a caller waits for
        dict(name="match_small", kind="match", probe="np1", C=32, K=24, NT=4000, nt=61, P=6,
             projection="fp32", rate_lo=10.0, rate_hi=30.0),
        # a linear probe's ordinary two-second batch, default projection
        dict(name="match_linear", kind="match", probe="linear", C=96, K=80, NT=60000, nt=61, P=6,
             projection="fp32", rate_lo=5.0, rate_hi=5.0),
        # the headline batch: Neuropixels 1.0, 600 templates, default projection
        dict(name="match_np1", kind="match", probe="np1", C=384, K=600, NT=60000, nt=61, P=6,
             projection="fp32", rate_lo=2.0, rate_hi=15.0),
        # the tensor-core projection on a ragged batch (a recording's tail) of
        # a probe with some channels dropped
        dict(name="match_ragged_split", kind="match", probe="np1", C=371, K=533, NT=43217, nt=61,
             P=6, projection="bf16x3", rate_lo=2.0, rate_hi=15.0),
        # the largest: a long recording's batches matched a group at a time,
        # one team of blocks per batch, captured once and replayed
        dict(name="batches_np1", kind="batches", probe="np1", C=384, K=600, NT=60000, nt=61, P=6,
             n=16, projection="bf16x3", rate_lo=2.0, rate_hi=15.0),
        # several recordings with batches of uneven length in one call
        dict(name="uneven_three", kind="uneven", n=15, NT_lo=8000, NT_hi=60000, nt=61, P=6,
             projection="bf16x3", rate_lo=2.0, rate_hi=15.0, recordings=3),
        # the whole drop-in call: int16 file in host memory -> sorted spikes
        # and features on the host
        dict(name="extract_np1", kind="extract", probe="np1", C=384, K=600, NT=60000, nt=61, P=6,
             n=4, projection="bf16x3", rate_lo=2.0, rate_hi=15.0),
        # universal-template detection of one Neuropixels batch
        dict(name="detect_np1", kind="detect", probe="np1", C=384, K=600, NT=60000, nt=61, P=6,
             rate_lo=2.0, rate_hi=15.0),
        # the batch filter of one 385-channel int16 batch
        dict(name="filter_np1", kind="filter", probe="np1", C=384, NT=60000, nt=61),
        # cross-correlations of a session's templates, once per recording and
        # after every template refinement
        dict(name="prepare_k600", kind="prepare", probe="np1", C=384, K=600, nt=61, P=6),
        # one gradient step of template refinement: loss, dU, dwPCA, damps
        dict(name="adjoint_np1", kind="adjoint", probe="np1", C=384, K=600, NT=60000, nt=61, P=6,
             rate_lo=5.0, rate_hi=37.0),
        # the PC features of one matched batch's spikes
        dict(name="features_np1", kind="features", probe="np1", C=384, K=600, NT=60000, nt=61, P=6,
             rate_lo=2.0, rate_hi=15.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["match", "match", "match", "match", "batches", "uneven", "extract",
                       "detect", "filter", "prepare", "adjoint", "features"])
    probe = rng.choice(["np1", "np1", "linear"])
    C = _log(rng, 32, 384) if probe == "np1" else _log(rng, 16, 128)
    K = max(12, min(1000, int(C * rng.uniform(0.7, 2.6))))
    nt, P = rng.choice([(61, 6), (61, 6), (61, 6), (41, 4)])
    NT = _log(rng, 4000, 60000)
    rates = dict(rate_lo=2.0, rate_hi=rng.choice([8.0, 15.0, 25.0]))
    if kind == "match":
        return dict(kind=kind, probe=probe, C=C, K=K, NT=NT, nt=nt, P=P,
                    projection=rng.choice(["fp32", "fp32", "bf16x3"]), **rates)
    if kind == "batches":
        return dict(kind=kind, probe=probe, C=C, K=min(K, 600), NT=NT, nt=nt, P=P,
                    n=rng.randint(2, 12), projection=rng.choice(["bf16x3", "bf16x3", "fp32"]),
                    **dict(rates, rate_hi=min(rates["rate_hi"], 15.0)))
    if kind == "uneven":
        return dict(kind=kind, n=rng.randint(4, 14), NT_lo=8000, NT_hi=rng.randint(16000, 60000),
                    nt=61, P=6, projection="bf16x3", recordings=rng.randint(2, 3),
                    **dict(rates, rate_hi=min(rates["rate_hi"], 15.0)))
    if kind == "extract":
        return dict(kind=kind, probe=probe, C=C, K=min(K, 600), NT=max(NT, 8000), nt=61, P=6,
                    n=rng.randint(2, 4), projection=rng.choice(["bf16x3", "fp32"]),
                    **dict(rates, rate_hi=min(rates["rate_hi"], 15.0)))
    if kind == "filter":
        return dict(kind=kind, probe=probe, C=C, NT=NT, nt=61)
    if kind == "prepare":
        return dict(kind=kind, probe=probe, C=C, K=K, nt=nt, P=P)
    if kind == "detect":
        nt, P = 61, 6
    return dict(kind=kind, probe=probe, C=C, K=min(K, 600), NT=NT, nt=nt, P=P, **rates)


# ------------------------------------------------------------------ inputs
def _rngs(seed):
    """A host generator for the small arrays, a device one for the signals."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(1 + 7919 * int(seed))
    return np.random.default_rng(int(seed)), gen


def _templates(rng, probe, C, K, nt, P):
    """xc, yc, wPCA [P, nt] and U [K, P, C] (numpy float32): biphasic waveforms
    on Gaussian footprints (sigma 30 um), amplitudes of 6 to 30 noise sd,
    near-proportional templates redrawn as a pipeline merges them."""
    xc, yc = synth.probe_geometry(probe, C)
    trough = TROUGH if nt == 61 else nt // 3
    W = synth._basis(rng, nt, P, trough, n_wave=2000)

    def units(n):
        sx, sy = rng.uniform(xc.min(), xc.max(), n), rng.uniform(yc.min(), yc.max(), n)
        d2 = (xc[None] - sx[:, None]) ** 2 + (yc[None] - sy[:, None]) ** 2
        sp = np.exp(-d2 / (2 * 30.0 ** 2)) * rng.uniform(6.0, 30.0, (n, 1))
        return sp, synth._waveforms(rng, n, nt, trough) @ W.T.astype(np.float64)

    sp, cf = units(K)
    for _ in range(50):
        a = sp / np.linalg.norm(sp, axis=1, keepdims=True)
        b = cf / np.linalg.norm(cf, axis=1, keepdims=True)
        bad = np.unique(np.nonzero(np.triu((a @ a.T) * (b @ b.T) > 0.99, 1))[1])
        if len(bad) == 0:
            break
        sp[bad], cf[bad] = units(len(bad))
    U = (cf.astype(np.float32)[:, :, None] * sp.astype(np.float32)[:, None, :])
    return xc, yc, W, np.ascontiguousarray(U)


def _trains(gen, case, K, L, nt):
    """[K, L] amplitude factor of the spike whose window is centred on each
    sample, 0 where there is none: Poisson trains, refractory over nt samples."""
    lo, hi = case["rate_lo"], case["rate_hi"]
    rate = lo + (hi - lo) * torch.rand((K, 1), generator=gen, device=DEV)
    mean = (FS / rate - nt).clamp(min=1.0)
    n = int((L / FS) * hi * 1.5) + 16
    isi = nt + torch.empty((K, n), device=DEV).exponential_(generator=gen) * mean
    t = nt + torch.cumsum(isi.double(), 1).floor().long()
    amp = 1.0 + 0.05 * torch.randn((K, n), generator=gen, device=DEV)
    keep = t < L - nt
    k = torch.arange(K, device=DEV)[:, None].expand(K, n)
    S = torch.zeros((K, L), device=DEV)
    S[k[keep], t[keep]] = amp[keep]
    return S


def _project_out(U, S, W):
    """[C, L]: sum over spikes of S[k, tau] * U_k x W centred on tau."""
    nt = W.shape[1]
    A = torch.einsum("kpc,kl->cpl", U, S)
    with torch.backends.cudnn.flags(enabled=True, benchmark=False, deterministic=True,
                                    allow_tf32=False):
        return torch.nn.functional.conv1d(A, W.flip(1)[None], padding=nt // 2)[:, 0]


def _conv(X, W):
    """[C, P, L]: every channel correlated with every basis row."""
    with torch.backends.cudnn.flags(enabled=True, benchmark=False, deterministic=True,
                                    allow_tf32=False):
        return torch.nn.functional.conv1d(X[:, None], W[:, None], padding=W.shape[1] // 2)


def _signal(gen, case, U, W, L):
    """One whitened padded batch [C, L]."""
    S = _trains(gen, case, U.shape[0], L, W.shape[1])
    return torch.randn((U.shape[2], L), generator=gen, device=DEV) + _project_out(U, S, W)


def _ctc(U, W):
    """Template cross-correlations [K, K, 2nt+1], in the dtype of U."""
    K, P, C = U.shape
    nt = W.shape[1]
    WtW = torch.zeros((P, P, 2 * nt + 1), dtype=U.dtype, device=U.device)
    for l in range(1, 2 * nt):
        # WtW[k, m, l] = sum_t W[m, t] W[k, t + nt - l]
        d = nt - l
        a, b = W[:, max(0, -d):nt - max(0, d)], W[:, max(0, d):nt - max(0, -d)]
        WtW[:, :, l] = b @ a.T
    G = (U.reshape(K * P, C) @ U.reshape(K * P, C).T).reshape(K, P, K, P)
    out = torch.empty((K, K, 2 * nt + 1), dtype=U.dtype, device=U.device)
    for i in range(0, K, 64):
        out[i:i + 64] = G[i:i + 64].permute(0, 2, 1, 3).reshape(-1, K, P * P) \
            @ WtW.reshape(P * P, -1)
    return out


def _recording(case, seed):
    """Geometry, basis and templates of a case, on the device."""
    rng, gen = _rngs(seed)
    xc, yc, W, U = _templates(rng, case["probe"], case["C"], case["K"], case["nt"], case["P"])
    return rng, gen, xc, yc, torch.from_numpy(W).to(DEV), torch.from_numpy(U).to(DEV)


def _match_inputs(case, seed, n=1):
    _, gen, _, _, W, U = _recording(case, seed)
    L = case["NT"] + 2 * case["nt"]
    return W, U, [_signal(gen, case, U, W, L) for _ in range(n)]


# three recordings with uneven batches: a small probe, an ordinary and a dense sort
_UNEVEN = [dict(probe="linear", C=96, K=150), dict(probe="np1", C=384, K=600),
           dict(probe="np1", C=384, K=1000)]


def _uneven_inputs(case, seed):
    rng, gen = _rngs(seed)
    recs = []
    for spec in _UNEVEN[:case["recordings"]]:
        _, _, W, U = _templates(rng, spec["probe"], spec["C"], spec["K"], case["nt"], case["P"])
        recs.append((torch.from_numpy(W).to(DEV), torch.from_numpy(U).to(DEV)))
    # lengths and their recordings are the case's, signals are the seed's
    lens = np.random.default_rng(case["n"] * 100003 + case["NT_hi"])
    NTs = lens.integers(case["NT_lo"], case["NT_hi"] + 1, case["n"])
    NTs[-1] = max(case["NT_lo"] // 2, int(NTs[-1]) // 4)          # a short tail
    items = []
    for i, NT in enumerate(NTs):
        r = i % len(recs)
        W, U = recs[r]
        items.append((_signal(gen, case, U, W, int(NT) + 2 * case["nt"]), r))
    return recs, items


def _raw(rng, gen, signal, n_bin, gain):
    """int16 [T, n_bin] file samples: the signal at ``gain`` on the first
    channels, plus what the filter removes (offsets, slow drifts, a 50 Hz
    common mode) and noise."""
    C, T = signal.shape
    f = lambda a: torch.from_numpy(np.asarray(a, np.float32)).to(DEV)
    off, amp = f(rng.uniform(-500, 500, n_bin)), f(rng.uniform(20, 120, n_bin))
    frq, ph = f(rng.uniform(1, 8, n_bin)), f(rng.uniform(0, 2 * np.pi, n_bin))
    out = torch.empty((T, n_bin), dtype=torch.int16, device=DEV)
    for s in range(0, T, 1 << 16):
        e = min(T, s + (1 << 16))
        t = torch.arange(s, e, device=DEV, dtype=torch.float64)[:, None] / FS
        x = torch.sin((2 * np.pi * t * frq).remainder(2 * np.pi) + ph).float() * amp + off
        x += (60 * torch.sin(2 * np.pi * 50 * t)).float()
        x += 15 * torch.randn((e - s, 1), generator=gen, device=DEV)
        x += 20 * torch.randn((e - s, n_bin), generator=gen, device=DEV)
        x[:, :C] += gain * signal[:, s:e].T
        out[s:e] = x.round().clamp(-32768, 32767).to(torch.int16)
    return out


GAIN = 200.0


def _hp_filter():
    from kilosort_b200.preprocess import highpass_filter
    return highpass_filter()


def _filter_inputs(case, seed):
    rng, gen = _rngs(seed)
    C, L = case["C"], case["NT"] + 2 * case["nt"]
    raw = _raw(rng, gen, torch.randn((C, L), generator=gen, device=DEV) * 1.5, C + 1, GAIN)
    # a whitening matrix: the inverse gain, mixing a few neighbouring channels
    ch = torch.arange(C, device=DEV, dtype=torch.float32)
    M = torch.exp(-(ch[:, None] - ch[None]).abs())
    Wrot = (torch.eye(C, device=DEV) - 0.25 * (M - torch.eye(C, device=DEV))) / GAIN
    return raw, Wrot


def _extract_inputs(case, seed):
    rng, gen, xc, yc, W, U = _recording(case, seed)
    C, T = case["C"], case["n"] * case["NT"]
    raw = _raw(rng, gen, _signal(gen, case, U, W, T), C + 1, GAIN).cpu().numpy()
    xc, yc = xc.astype(np.float32), yc.astype(np.float32)
    pos = np.vstack((xc, yc)).T
    d2 = ((pos[:, None, :] - pos[None, :, :]) ** 2).sum(-1)
    Kxx = torch.from_numpy(np.exp(-d2 / (2 * 20.0 ** 2)))
    iKxx = torch.linalg.inv(Kxx + 0.01 * torch.eye(C)).to(DEV)
    ops = dict(Th_learned=TH, nt=case["nt"], max_peels=MAX_PEELS, wPCA=W,
               projection=case["projection"], nt0min=TROUGH, batch_size=case["NT"], xc=xc, yc=yc,
               nblocks=1, yblk=np.array([yc.mean()]), probe=dict(xc=xc, yc=yc), iKxx=iKxx,
               settings=dict(nearest_chans=10, position_limit=100, n_pcs=case["P"],
                             sig_interp=20.0))
    return raw, torch.eye(C) / GAIN, rng.uniform(-5.0, 5.0, (case["n"], 1)), ops, U


def _detect_inputs(case, seed):
    rng, gen, xc, yc, W, U = _recording(case, seed)
    wave = synth._waveforms(rng, 6, case["nt"], TROUGH)
    wTEMP = torch.from_numpy((wave / np.linalg.norm(wave, axis=1, keepdims=True))
                             .astype(np.float32)).to(DEV)
    settings = dict(nearest_chans=10, nearest_templates=100, min_template_size=10,
                    template_sizes=5, dmin=None, dminx=32, n_templates=6, n_pcs=6,
                    nt0min=TROUGH)
    C = case["C"]
    ops = dict(settings=settings, xc=xc.astype(np.float32), yc=yc.astype(np.float32),
               kcoords=np.zeros(C, np.float32), nt=case["nt"], batch_size=case["NT"], fs=FS,
               Th_universal=9.0, max_channel_distance=32.0, wTEMP=wTEMP, wPCA=W)
    return ops, _signal(gen, case, U, W, case["NT"] + 2 * case["nt"])


def _spikes(gen, case, K, L, nt):
    """st [N, 2], amps [N] and their [K, L] map S, N the expected spike count
    of the case's rates: at most two spikes per sample, templates by their
    rates, in the order the matcher emits them (in time within each of about
    forty rounds)."""
    lo, hi = case["rate_lo"], case["rate_hi"]
    N = max(1, int(K * (lo + hi) / 2 * (L - 2 * nt) / FS))
    rate = lo + (hi - lo) * torch.rand(K, generator=gen, device=DEV)
    tau = nt + torch.randperm(2 * (L - 2 * nt), generator=gen, device=DEV)[:N] // 2
    tau = tau.sort().values
    cum = torch.cumsum(rate.double(), 0)
    k = torch.searchsorted(cum, torch.rand(N, generator=gen, device=DEV).double() * cum[-1])
    st = torch.stack((tau, k.clamp(max=K - 1)), 1)
    st = st[torch.argsort(torch.arange(N, device=DEV) % 40, stable=True)].contiguous()
    amps = 1.0 + 0.05 * torch.randn(N, generator=gen, device=DEV)
    S = torch.zeros((K, L), device=DEV)
    S.index_put_((st[:, 1], st[:, 0]), amps, accumulate=True)
    return st, amps, S


def _adjoint_inputs(case, seed):
    _, gen, _, _, W, U = _recording(case, seed)
    L = case["NT"] + 2 * case["nt"]
    st, amps, S = _spikes(gen, case, case["K"], L, case["nt"])
    X = torch.randn((case["C"], L), generator=gen, device=DEV) + _project_out(U, S, W)
    # the amplitudes and templates of an iteration on the way to the optimum
    amps = amps * (1 + 0.05 * torch.randn(len(st), generator=gen, device=DEV))
    U = U * (1 + 0.02 * torch.randn(U.shape, generator=gen, device=DEV))
    return X, st, amps, U, W


def _features_inputs(case, seed):
    _, gen, xc, yc, W, U = _recording(case, seed)
    L = case["NT"] + 2 * case["nt"]
    st, amps, _ = _spikes(gen, case, case["K"], L, case["nt"])
    return (torch.randn((case["C"], L), generator=gen, device=DEV), st, amps[:, None].contiguous(),
            W, U, xc, yc)


# ---------------------------------------------------------------- the calls
def _room(case, NT=None, K=None):
    """Spike rows a program allocates for one batch: twice the highest rate."""
    return int(2 * (K or case["K"]) * case["rate_hi"] * (NT or case["NT"]) / FS) + 1000


def _zeros(*shape, dtype=torch.float32, device=DEV):
    return torch.zeros(shape, dtype=dtype, device=device)


def _spike_rows(*lead):
    return dict(st=_zeros(*lead, 2, dtype=torch.int64), amps=_zeros(*lead, 1),
                th_amps=_zeros(*lead, 1))


def _collect(rows, st, amps, th_amps, i=None):
    """One batch's spikes into the program's arrays (row i of them)."""
    for name, v in (("st", st), ("amps", amps), ("th_amps", th_amps)):
        dst = rows[name] if i is None else rows[name][i]
        dst[:len(v)] = v


def prepare(case, seed):
    import kilosort_b200 as kb
    from kilosort_b200 import batched, preprocess, spikedetect
    kind = case["kind"]
    if kind == "match":
        W, U, (X,) = _match_inputs(case, seed)
        ops = dict(Th_learned=TH, nt=case["nt"], max_peels=MAX_PEELS, wPCA=W,
                   projection=case["projection"])
        return dict(kind=kind, ops=ops, X=X, U=U, ctc=_ctc(U, W), rows=_spike_rows(_room(case)))
    if kind == "batches":
        W, U, Xs = _match_inputs(case, seed, case["n"])
        rec = batched.Recording(U=U, wPCA=W, ctc=_ctc(U, W), Th=TH, nt=case["nt"],
                                max_peels=MAX_PEELS)
        m = batched.BatchedMatcher([rec], [(X.shape[1], 0) for X in Xs], case["projection"],
                                   teams=case["n"])
        return dict(kind=kind, matcher=m, Xs=Xs, rows=_spike_rows(case["n"], _room(case)))
    if kind == "uneven":
        recs, items = _uneven_inputs(case, seed)
        recs = [batched.Recording(U=U, wPCA=W, ctc=_ctc(U, W), Th=TH, nt=case["nt"],
                                  max_peels=MAX_PEELS, capacity=50000) for W, U in recs]
        return dict(kind=kind, recs=recs, items=items, projection=case["projection"],
                    rows=_spike_rows(case["n"], _room(case, case["NT_hi"], 1000)))
    if kind == "extract":
        raw, whiten, dshift, ops, U = _extract_inputs(case, seed)
        src = synth.FilteredBinary(raw, NT=case["NT"], nt=case["nt"],
                                   chan_map=np.arange(case["C"]), hp_filter=_hp_filter(),
                                   whiten_mat=whiten, dshift=dshift, device=DEV)
        room = case["n"] * _room(case)
        return dict(kind=kind, ops=ops, src=src, U=U, st=np.zeros((room, 3)),
                    tF=_zeros(room, min(10, case["C"]), case["P"], device="cpu"))
    if kind == "detect":
        ops, X = _detect_inputs(case, seed)
        iC, iC2, weigh = spikedetect.geometry(ops, device=torch.device(DEV))
        room, nC = _room(case), iC.shape[0]
        i64 = torch.int64
        return dict(kind=kind, X=X, out=(_zeros(room, 2, dtype=i64), _zeros(room, dtype=i64),
                                         _zeros(room), _zeros(nC, room), _zeros(room),
                                         _zeros(room, nC, case["P"])),
                    detector=spikedetect.Detector(ops, iC, iC2, weigh, torch.device(DEV)))
    if kind == "filter":
        raw, Wrot = _filter_inputs(case, seed)
        p = preprocess.Preprocessor(case["C"] + 1, raw.shape[0], whiten=Wrot,
                                    chan_map=np.arange(case["C"]), hp_filter=_hp_filter(),
                                    device=torch.device(DEV))
        return dict(kind=kind, filter=p, raw=raw)
    if kind == "prepare":
        _, _, _, _, W, U = _recording(case, seed)
        return dict(kind=kind, ops=dict(nt=case["nt"], wPCA=W), U=U)
    if kind == "adjoint":
        X, st, amps, U, W = _adjoint_inputs(case, seed)
        amps, U, W = (t.clone().requires_grad_(True) for t in (amps, U, W))
        return dict(kind=kind, X=X, st=st, amps=amps, U=U, W=W)
    if kind == "features":
        Xres, st, amps, W, U, xc, yc = _features_inputs(case, seed)
        iCC, _, iU, Ucc = kb.prepare_extract(xc, yc, U, min(10, case["C"]), 100,
                                             device=torch.device(DEV))
        return dict(kind=kind, args=(Xres, st, amps, W, iCC.contiguous(), iU, Ucc))
    raise ValueError(kind)


def run(state):
    import kilosort_b200 as kb
    from kilosort_b200 import batched
    from kilosort_b200.adjoint import reconstruction_loss
    from kilosort_b200.template_matching import spike_features
    s, kind = state, state["kind"]
    if kind == "match":
        st, amps, th, Xres = kb.run_matching(s["ops"], s["X"], s["U"], s["ctc"],
                                             device=s["X"].device)
        _collect(s["rows"], st, amps, th)
        return dict(s["rows"], Xres=Xres)
    if kind in ("batches", "uneven"):
        got = s["matcher"].run(s["Xs"]) if kind == "batches" else \
            batched.match_batches(s["recs"], s["items"], s["projection"])
        for i, (st, amps, th, _) in enumerate(got):
            _collect(s["rows"], st, amps, th, i)
        return dict(s["rows"], Xres=[g[3] for g in got])
    if kind == "extract":
        st, tF, _ = kb.extract(dict(s["ops"]), s["src"], s["U"], device=torch.device(DEV))
        s["st"][:len(st)] = st
        s["tF"][:len(tF)] = tF
        return s["st"], s["tF"]
    if kind == "detect":
        for dst, v in zip(s["out"], s["detector"](s["X"])):
            if dst.dim() == 2 and dst.dtype == torch.float32:         # adist [nC, n]
                dst[:, :v.shape[1]] = v
            else:
                dst[:len(v)] = v
        return s["out"]
    if kind == "filter":
        return s["filter"](s["raw"])
    if kind == "prepare":
        return kb.prepare_matching(s["ops"], s["U"])
    if kind == "adjoint":
        for t in (s["amps"], s["U"], s["W"]):
            t.grad = None
        loss = reconstruction_loss(s["X"], s["st"], s["amps"], s["U"], s["W"])
        loss.backward()
        return loss.detach(), s["U"].grad, s["W"].grad, s["amps"].grad
    if kind == "features":
        return spike_features(*s["args"])
    raise ValueError(kind)


# --------------------------------------------------------------------- work
def _match_work(C, K, P, nt, L, rate):
    """One batch: projection and contraction, then per spike the scores of
    every template around it and its waveform out of the residual."""
    n = K * rate * L / FS
    flops = 2 * C * P * nt * L + 2 * K * C * P * L + n * (2 * K * (2 * nt + 1)
                                                          + 2 * C * nt * (P + 1))
    return 8 * C * L + 24 * n, flops


def work(case):
    kind, nt, P = case["kind"], case["nt"], case.get("P", 6)
    C, K = case.get("C", 0), case.get("K", 0)
    L = case.get("NT", 0) + 2 * nt
    rate = (case.get("rate_lo", 0) + case.get("rate_hi", 0)) / 2
    templates = 4 * K * P * C + 4 * K * K * (2 * nt + 1)
    if kind in ("match", "batches"):
        b, f = _match_work(C, K, P, nt, L, rate)
        n = case.get("n", 1)
        return dict(bytes=n * b + templates, flops=n * f)
    if kind == "uneven":
        mean = (case["NT_lo"] + case["NT_hi"]) / 2 + 2 * nt
        specs = _UNEVEN[:case["recordings"]]
        per = [_match_work(r["C"], r["K"], P, nt, mean, rate) for r in specs]
        n = case["n"] / len(specs)
        t = sum(4 * r["K"] * P * r["C"] + 4 * r["K"] ** 2 * (2 * nt + 1) for r in specs)
        return dict(bytes=t + n * sum(p[0] for p in per), flops=n * sum(p[1] for p in per))
    if kind == "extract":
        n = case["n"]
        b, f = _match_work(C, K, P, nt, L, rate)
        ns = n * K * rate * L / FS
        # the samples in, spikes and 10 channels of features out; filter
        # (1023 taps, whitening) and matching in between
        return dict(bytes=2 * n * (C + 1) * L + templates + ns * (24 + 40 * P),
                    flops=n * (f + 2 * C * L * 1023 + 2 * C * C * L) + ns * 20 * nt * P)
    if kind == "detect":
        xc, yc = synth.probe_geometry(case["probe"], C)
        rows = len(np.unique(yc))
        # positions: half the row spacing down the probe, 16 um across
        nf = (2 * rows - 1) * (int(round((xc.max() - xc.min()) / 16)) + 1)
        return dict(bytes=4 * C * L, flops=2 * C * 6 * nt * L + 2 * nf * L * 30 * min(10, C))
    if kind == "filter":
        return dict(bytes=2 * L * (C + 1) + 4 * C * L + 4 * C * C,
                    flops=2 * C * L * 1023 + 2 * C * C * L)
    if kind == "prepare":
        return dict(bytes=4 * K * P * C + 4 * K * K * (2 * nt + 1),
                    flops=2 * (K * P) ** 2 * C + 2 * K * K * P * P * (2 * nt + 1))
    n = K * rate * L / FS
    if kind == "adjoint":
        return dict(bytes=8 * C * L + 8 * K * P * C + 24 * n, flops=n * C * nt * (2 * P + 6))
    if kind == "features":
        return dict(bytes=n * 10 * (4 * nt + 4 * P) + 20 * n, flops=2 * n * 10 * nt * P)
    raise ValueError(kind)


# -------------------------------------------------------------------- exact
def _peel64(X, U, W, ctc, nt):
    """(amps, th_amps, Xres, st) of the greedy matching of one batch, 64 bits."""
    X, U, W, ctc = (t.double() for t in (X, U, W, ctc))
    K, P, C = U.shape
    L = X.shape[1]
    nm = (U ** 2).sum((1, 2))
    B = torch.zeros((K, L), dtype=torch.float64, device=X.device)
    for p in range(P):
        B += U[:, p] @ _conv(X, W[p:p + 1])[:, 0]
    res = X.clone()
    lags = torch.arange(-nt, nt + 1, device=X.device)
    taps = torch.arange(-(nt // 2), nt // 2 + 1, device=X.device)
    sts, amps, ths = [], [], []
    for _ in range(MAX_PEELS):
        score = B.clamp(min=0) ** 2 / nm[:, None]
        best, arg = score.max(0)
        best[:nt] = 0
        best[L - nt:] = 0
        pool = torch.nn.functional.max_pool1d(best[None, None], 2 * nt + 1, stride=1,
                                              padding=nt)[0, 0]
        tau = torch.nonzero((pool > TH ** 2) & (pool == best))[:, 0]
        if len(tau) == 0:
            break
        k = arg[tau]
        a = B[k, tau] / nm[k]
        sts.append(torch.stack((tau, k), 1))
        amps.append(a[:, None])
        ths.append(pool[tau].sqrt()[:, None])
        # peaks lie more than nt apart, so every other one's lag windows and
        # all residual windows are disjoint
        for g in (0, 1):
            t, kk, aa = tau[g::2], k[g::2], a[g::2]
            wave = torch.einsum("kpc,pt->ckt", U[kk], W)
            res[:, t[:, None] + taps] -= aa[:, None] * wave
            for c in range(0, len(t), 64):
                B[:, t[c:c + 64, None] + lags] -= aa[c:c + 64, None] * ctc[:, kk[c:c + 64], :]
    if not sts:
        z = torch.zeros((0, 1), dtype=torch.float64, device=X.device)
        return z, z, res, torch.zeros((0, 2), dtype=torch.int64, device=X.device)
    return torch.cat(amps), torch.cat(ths), res, torch.cat(sts)


def _padded(v, room, dim=0):
    """``v`` with zeros up to ``room`` along ``dim``."""
    shape = list(v.shape)
    shape[dim] = max(0, room - shape[dim])
    return torch.cat((v, v.new_zeros(shape)), dim)


def _match64(items, room, nt, one=False):
    """The outputs of the batches ``items`` of (X, U, W, ctc)."""
    got = [_peel64(X, U, W, ctc, nt) for X, U, W, ctc in items]
    amps = [_padded(g[0], room) for g in got]
    ths = [_padded(g[1], room) for g in got]
    if one:
        return dict(st=None, amps=amps[0], th_amps=ths[0], Xres=got[0][2])
    return dict(st=None, amps=torch.stack(amps), th_amps=torch.stack(ths),
                Xres=[g[2] for g in got])


def _filter64(raw, C, hp, Wrot):
    """[C, L]: mean, common median, Fourier-domain high-pass, whitening."""
    X = raw[:, :C].T.double()
    X = X - X.mean(1, keepdim=True)
    X = X - X.median(0).values
    L, n = X.shape[1], len(hp)
    h = hp.double().to(X.device)
    if n < L:
        h = torch.nn.functional.pad(h, ((L - n) // 2, L - n - (L - n) // 2))
    elif n > L:
        h = h[(n - L) // 2:(n - L) // 2 + L]
    X = torch.fft.ifft(torch.fft.fft(X) * torch.fft.fft(h).conj()).real
    return Wrot.double().to(X.device) @ torch.fft.fftshift(X, dim=-1)


def _features64(res, st, amps, U, W, xc, yc, nC):
    d2 = (xc[None] - xc[:, None]) ** 2 + (yc[None] - yc[:, None]) ** 2
    near = torch.from_numpy(np.argsort(d2, 0)[:nC]).to(res.device)
    ch = near[:, (U ** 2).sum(1).argmax(1)[st[:, 1]]]                  # [nC, N]
    nt = W.shape[1]
    taps = torch.arange(-(nt // 2), nt // 2 + 1, device=res.device)
    win = res.double()[ch[:, :, None], st[:, 0][None, :, None] + taps]
    f = win @ W.double().T
    f += amps.double().reshape(1, -1, 1) * U.double()[st[:, 1][None], :, ch]
    return f.transpose(0, 1).contiguous()


def _extract64(case, seed):
    raw, whiten, dshift, ops, U = _extract_inputs(case, seed)
    C, NT, nt, W = case["C"], case["NT"], case["nt"], ops["wPCA"]
    ctc = _ctc(U.double(), W.double())
    pos = torch.from_numpy(np.vstack((ops["xc"], ops["yc"])).T).double().to(DEV)
    rows, feats = [], []
    for b in range(case["n"]):
        part = torch.from_numpy(raw[max(0, b * NT - nt):(b + 1) * NT + nt]).to(DEV)
        if b == 0:
            part = torch.cat((part[:1].expand(nt, -1), part))
        if len(part) < NT + 2 * nt:
            part = torch.cat((part, part[-1:].expand(NT + 2 * nt - len(part), -1)))
        moved = pos.clone()
        moved[:, 1] -= float(dshift[b, 0])
        d2 = ((moved[:, None] - pos[None]) ** 2).sum(-1)
        drift = torch.exp(-d2 / (2 * 20.0 ** 2)) @ ops["iKxx"].double()
        X = _filter64(part, C, _hp_filter(), drift @ whiten.to(DEV).double())
        amps, ths, res, st = _peel64(X, U, W, ctc, nt)
        tF = _features64(res, st, amps, U, W, ops["xc"].astype(np.float64),
                         ops["yc"].astype(np.float64), min(10, C))
        t = st[:, 0].double() - nt - nt // 2 + TROUGH
        keep = (t >= 0) if b == 0 else torch.ones_like(t, dtype=torch.bool)
        rows.append(torch.stack((t + b * NT, st[:, 1].double(), ths[:, 0]), 1)[keep])
        feats.append(tF[keep])
    rows, feats = torch.cat(rows).cpu().numpy(), torch.cat(feats).cpu()
    order = np.argsort(rows[:, 0])
    room = case["n"] * _room(case)
    return (_padded(torch.from_numpy(rows[order]), room), _padded(feats[order], room))


def _detect64(case, seed):
    from kilosort_b200 import spikedetect
    ops, X = _detect_inputs(case, seed)
    s, nt = ops["settings"], case["nt"]
    iC, iC2, weigh = spikedetect.geometry(ops, device=torch.device(DEV))
    X, weigh = X.double(), weigh.double()
    nC, F = iC.shape
    L = X.shape[1]
    B = _conv(X, ops["wTEMP"].double())                               # [C, 6, L]
    As, im = torch.zeros((F, L), dtype=torch.float64, device=DEV), \
        torch.zeros((F, L), dtype=torch.int64, device=DEV)
    for f in range(0, F, 16):
        A = torch.einsum("sjf,jfkl->skfl", weigh[:, :, f:f + 16], B[iC[:, f:f + 16]])
        A = A.flatten(0, 1)
        m, i = A.abs().max(0)
        As[f:f + 16] = m
        im[f:f + 16] = (1 + i) * torch.gather(A, 0, i[None])[0].sign().long()
    nb = torch.zeros_like(As)
    for j in range(iC2.shape[0]):
        nb = torch.maximum(nb, As[iC2[j]])
    nb[:, :nt] = 0
    nb[:, L - nt:] = 0
    pool = torch.nn.functional.max_pool1d(nb[None], 2 * s["nt0min"] + 1, stride=1,
                                          padding=s["nt0min"])[0]
    xy = torch.nonzero((pool == As) & (As > ops["Th_universal"]))
    f, t = xy[:, 0], xy[:, 1]
    sg, k = im[f, t].sign(), im[f, t].abs() - 1
    adist = B[iC[:, f], (k % 6)[None], t[None]] * sg
    r = adist.clamp(min=0)
    y = (r / r.sum(0) * torch.from_numpy(ops["yc"]).double().to(DEV)[iC[:, f]]).sum(0)
    taps = torch.arange(-(nt // 2), nt // 2 + 1, device=DEV)
    tF = X[iC[:, f][:, :, None], t[None, :, None] + taps] @ ops["wPCA"].double().T
    room = _room(case)
    return (None, None, _padded(As[f, t], room), _padded(adist, room, 1), _padded(y, room),
            _padded(tF.transpose(0, 1), room))


def _adjoint64(case, seed):
    X, st, amps, U, W = (t if t.dtype == torch.int64 else t.double()
                         for t in _adjoint_inputs(case, seed))
    K, P, C = U.shape
    L, nt = X.shape[1], W.shape[1]
    S = torch.zeros((K, L), dtype=torch.float64, device=DEV)
    S.index_put_((st[:, 1], st[:, 0]), amps, accumulate=True)
    R = torch.zeros_like(X)
    A = [U[:, p].T @ S for p in range(P)]
    for p in range(P):
        R += torch.nn.functional.conv1d(A[p][:, None], W[p:p + 1].flip(1)[None],
                                        padding=nt // 2)[:, 0]
    res = X - R
    G = -2 * res
    dU, dW, da = torch.empty_like(U), torch.empty_like(W), torch.zeros(len(st), device=DEV,
                                                                     dtype=torch.float64)
    pad = torch.nn.functional.pad(G, (nt // 2, nt // 2))
    for p in range(P):
        Y = _conv(G, W[p:p + 1])[:, 0]                                # [C, L]
        dU[:, p] = S @ Y.T
        for i in range(0, len(st), 4096):
            da[i:i + 4096] += (U[st[i:i + 4096, 1], p] * Y[:, st[i:i + 4096, 0]].T).sum(1)
        for t in range(nt):
            dW[p, t] = (A[p] * pad[:, t:t + L]).sum()
    return (res ** 2).sum(), dU, dW, da


def exact(case, seed):
    kind = case["kind"]
    if kind == "match":
        W, U, (X,) = _match_inputs(case, seed)
        return _match64([(X, U, W, _ctc(U, W))], _room(case), case["nt"], one=True)
    if kind == "batches":
        W, U, Xs = _match_inputs(case, seed, case["n"])
        ctc = _ctc(U, W)
        return _match64([(X, U, W, ctc) for X in Xs], _room(case), case["nt"])
    if kind == "uneven":
        recs, items = _uneven_inputs(case, seed)
        ctcs = [_ctc(U, W) for W, U in recs]
        return _match64([(X, recs[r][1], recs[r][0], ctcs[r]) for X, r in items],
                        _room(case, case["NT_hi"], 1000), case["nt"])
    if kind == "extract":
        return _extract64(case, seed)
    if kind == "detect":
        return _detect64(case, seed)
    if kind == "filter":
        raw, Wrot = _filter_inputs(case, seed)
        return _filter64(raw, case["C"], _hp_filter(), Wrot)
    if kind == "prepare":
        _, _, _, _, W, U = _recording(case, seed)
        return _ctc(U.double(), W.double())
    if kind == "adjoint":
        return _adjoint64(case, seed)
    if kind == "features":
        Xres, st, amps, W, U, xc, yc = _features_inputs(case, seed)
        return _features64(Xres, st, amps, U, W, xc, yc, min(10, case["C"]))
    raise ValueError(kind)
