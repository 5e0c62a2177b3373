"""The early-out of the overlapped FP64 search (csrc/cs_search_f64.cuh,
slot_bound): its FP32 bound may never be below the FP64 metric it stands for.
On the CPU the bound is restated in FP32 and compared with the FP64 metric of
profiles whose bins are far larger than their folds; on the GPU the records
above thresholds just below single metrics are those of search_f64, which has no
bound, for spectra with strong tones, values past FP32's range and no numbers."""
import numpy as np
import pytest

from coherentsearch_c_b200.search import Options, Session

f32 = np.float32


def metric(rows, K, widths, scale):
    """The FP64 metric of K-fold profiles, rows [n][K * nk]."""
    n, nb = rows.shape
    nk = nb // K
    x = rows.reshape(n, K, nk).sum(1) / K
    p = np.concatenate([np.zeros((n, 1)), np.cumsum(np.concatenate([x, x], 1), 1)], 1)
    best = np.full(n, -np.inf)
    for w, s in zip(widths, scale):
        mx = (p[:, w:w + nk] - p[:, :nk]).max(1)
        best = np.maximum(best, (mx - w / nk * p[:, nk]) * s)
    return best


def bound(rows, K, widths, scale):
    """slot_bound, in FP32 in its order."""
    r = rows.astype(f32)
    n, nb = r.shape
    nk = nb // K
    x = r[:, :nk].copy()
    for q in range(1, K):
        x += r[:, q * nk:(q + 1) * nk]
    m1 = x.max(1)
    m2 = (x + np.roll(x, 1, 1)).max(1)
    tot = np.zeros(n, f32)
    for j in range(0, nk, 2):
        tot += x[:, j] + x[:, j + 1]
    size = np.abs(r).max(1)
    margin = (np.abs(tot) + f32(nk) * np.abs(m1)) * f32(nk + 16) * f32(2.4e-7)
    margin += f32(2 * K * (K + 1) * max(widths)) * f32(6.0e-8) * size + f32(1e-30)
    best = np.full(n, f32(-np.inf))
    for w, s in zip(widths, scale):
        m = m1 if w == 1 else f32(w >> 1) * m2 + (m1 if w & 1 else f32(0))
        best = np.maximum(best, (m - f32(w) / f32(nk) * tot + margin) * f32(s))
    return best / f32(K)


@pytest.mark.parametrize("K,nk,widths", [(1, 32, (1, 2, 3, 4, 6)), (2, 16, (2, 3)), (3, 40, (2, 3, 4, 6)),
                                         (4, 8, (2,)), (5, 24, (2, 3, 4, 6)), (6, 20, (6,))])
@pytest.mark.parametrize("tone", [0.0, 1e3, 3e4, 1e6, 1e8])
def test_bound_is_not_below_the_metric(K, nk, widths, tone):
    rng = np.random.default_rng(K * 100 + nk)
    nb = K * nk
    t = 2 * np.pi * np.arange(nb) / nb
    rows = rng.standard_normal((4000, nb))
    rows += tone * np.cos(t[None, :] + 6.28 * rng.random((4000, 1)))     # cancels in a fold
    scale = 1.0 / np.sqrt(np.array(widths, float) * (1 - np.array(widths) / nk))
    assert (bound(rows, K, widths, scale) >= metric(rows, K, widths, scale)).all()


def _noise(N, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(f32), rng


def _search(opts, N, amps, monkeypatch, generic, thresholds):
    if generic:
        monkeypatch.setenv("CS_B200_GENERIC_KERNEL", "1")
    ses = Session(N, 64e-6, opts)
    if generic:
        monkeypatch.delenv("CS_B200_GENERIC_KERNEL")
    out = [ses.run_raw(amps, threshold=t) for t in thresholds]
    ses.close()
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("nharms,fold", [(16, 4), (32, 4), (60, 6), (13, 1), (7, 1)])
@pytest.mark.parametrize("tone", [30.0, 1e5, 1e6, 1e7])
def test_thresholds_below_single_metrics(gpu_ready, monkeypatch, nharms, fold, tone):
    N = 120000                                      # trials up to bin 960
    amps, rng = _noise(N, nharms)
    amps *= 3                                       # metrics past 6: the wide kernel's
    tones = np.arange(301, 900, 31)                 # first harmonic on a tone, the others not
    for b in tones:
        z = 3 * tone * np.exp(6.28j * rng.random())
        amps[2 * b:2 * b + 2] = z.real, z.imag
    opts = Options(nharms=nharms, blocksize=1000, precision=1)
    every = _search(opts, N, amps, monkeypatch, True, [-1e30])[0]
    sel = every[every["nharm"] == nharms // fold]
    sel = sel[np.argsort(sel["r"])]
    near = np.abs(sel["r"][:, None] / fold - tones).min(1) < 4.0
    tops = []                                       # what a sub-tile of 32 trials has most
    for a in range(0, sel.size - 64, 64):
        if near[a:a + 64].all():
            tops.append(sel["metric"][a:a + 64].max())
    tops = np.sort(tops)                            # the least: the tone cancelled in the fold
    thr = tops[tops > 6.1][:60] * (1 - 1e-6)
    assert thr.size >= 12
    new = _search(opts, N, amps, monkeypatch, False, thr)
    old = _search(opts, N, amps, monkeypatch, True, thr)
    for t, a, b in zip(thr, new, old):
        assert b.size > 0
        a, b = (x[np.abs(x["metric"] - t) > 1e-8 * t] for x in (a, b))
        assert a.size == b.size, (t, a.size, b.size)
        np.testing.assert_array_equal(a["r"], b["r"])
        np.testing.assert_array_equal(a["nharm"], b["nharm"])
        np.testing.assert_allclose(a["metric"], b["metric"], rtol=1e-9,
                                   atol=1e-9 * every["metric"].max())


@pytest.mark.gpu
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 1e38, 1e-42])
def test_values_fp32_sums_do_not_hold(gpu_ready, monkeypatch, value):
    N = 30000
    amps, _ = _noise(N, 3)
    thr = [4.0, 1e3]
    if abs(value) < 1.0:                        # a spectrum below FP32's normal range
        amps *= f32(value)
        thr = [4.0 * value, 1e-60, 1e-45]
    else:
        for b in (97, 1201, 5003, 5004, 9001):
            amps[2 * b] = value
    opts = Options(nharms=60, blocksize=1000, precision=1)
    new = _search(opts, N, amps, monkeypatch, False, thr)
    old = _search(opts, N, amps, monkeypatch, True, thr)
    assert old[0].size > 0
    for a, b in zip(new, old):
        assert a.size == b.size
        np.testing.assert_array_equal(a["r"], b["r"])
        np.testing.assert_array_equal(a["nharm"], b["nharm"])
        top = b["metric"].max() if b.size else 0.0
        np.testing.assert_allclose(a["metric"], b["metric"], rtol=1e-9, atol=1e-9 * top)


@pytest.mark.gpu
@pytest.mark.parametrize("threshold", [4.0, 8.0])
def test_few_harmonics_are_not_slower_than_search_f64(gpu_ready, monkeypatch, threshold):
    """Where noise reaches the threshold the bound is of no use."""
    N = 1 << 18
    amps, _ = _noise(N, 1)
    opts = Options(nharms=7, precision=1, threshold=threshold)
    took = []
    for generic in (True, False):
        if generic:
            monkeypatch.setenv("CS_B200_GENERIC_KERNEL", "1")
        ses = Session(N, 64e-6, opts)
        monkeypatch.delenv("CS_B200_GENERIC_KERNEL", raising=False)
        ses.run_raw(amps)
        ms = []
        for _ in range(15):
            ses.enqueue(None)
            ms.append(ses.collect()[1])
        ses.close()
        took.append(float(np.median(ms)))
    assert took[1] < 1.15 * took[0]
