"""Centring and common average reference at the edges of their tiles (32 samples,
256 for the sums; 32 channels a register, registers in fours): without filter and
whitening the result is a chain of single FP32 roundings, so it is compared exactly.
The inputs put few, all or one of two values into the buckets of the median."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = torch.device("cuda:0")


def _raw(kind, rng, L, n_bin):
    if kind == "constant":
        return np.full((L, n_bin), 7, np.int16)
    if kind == "two":
        return rng.choice([-300, 300], (L, n_bin)).astype(np.int16)
    raw = rng.normal(0, 90, (L, n_bin))
    if kind == "outliers":
        raw[rng.random((L, n_bin)) < 0.02] = 32767
        raw[:, 0] = -32768
    return np.clip(raw, -32768, 32767).astype(np.int16)


@pytest.mark.parametrize("n_bin,C,L,car,inv,kind", [
    (1, 1, 1, True, False, "normal"), (2, 2, 31, True, True, "two"),
    (40, 31, 257, True, False, "normal"), (33, 33, 1000, True, True, "constant"),
    (129, 128, 255, True, False, "outliers"), (129, 129, 513, True, False, "two"),
    (385, 384, 4099, True, False, "normal"), (385, 385, 256, True, True, "outliers"),
    (512, 500, 777, True, False, "normal"), (700, 641, 300, True, False, "outliers"),
    (900, 897, 65, True, True, "two"), (1024, 1024, 100, True, False, "normal"),
    (385, 200, 1500, False, True, "normal"), (1024, 1000, 33, False, False, "outliers")])
def test_exact_values(cuda_device, n_bin, C, L, car, inv, kind):
    from kilosort_b200.preprocess import Preprocessor
    rng = np.random.default_rng(n_bin + 7 * L)
    raw = _raw(kind, rng, L, n_bin)
    cmap = rng.permutation(n_bin)[:C]
    p = Preprocessor(n_bin, L, whiten=None, chan_map=cmap, hp_filter=None, do_CAR=car,
                     invert_sign=inv, artifact_threshold=float("inf"), device=DEV)
    got = p(torch.from_numpy(raw).to(DEV)).cpu().numpy()
    x = raw[:, cmap].astype(np.float32).T * np.float32(-1.0 if inv else 1.0)
    mean = (x.astype(np.float64).sum(1) / L).astype(np.float32)
    ref = x - mean[:, None]
    if car:
        ref = ref - np.sort(ref, axis=0)[(C - 1) // 2]
    assert got.dtype == np.float32 and np.array_equal(got, ref)


@pytest.mark.parametrize("C,L,hp", [(129, 700, True), (300, 1057, False), (300, 3000, True)])
def test_channel_groups_without_the_median(cuda_device, C, L, hp):
    """Without the common average channels do not meet: any split of them gives the
    same values as all together (blocks take 128)."""
    from kilosort_b200.preprocess import Preprocessor
    rng = np.random.default_rng(C + L)
    raw = torch.from_numpy(_raw("normal", rng, L, C + 5)).to(DEV)
    cmap = rng.permutation(C + 5)[:C]
    filt = torch.from_numpy(rng.standard_normal(401).astype(np.float32)) / 20 if hp else None
    run = lambda m: Preprocessor(C + 5, L, whiten=None, chan_map=m, hp_filter=filt, do_CAR=False,
                                 artifact_threshold=float("inf"), device=DEV)(raw)
    assert torch.equal(run(cmap), torch.cat([run(cmap[i:i + 77]) for i in range(0, C, 77)]))
