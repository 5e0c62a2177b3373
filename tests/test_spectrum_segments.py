"""SpectrumMaker's normalisation at lengths and widths that move the rednoise
blocks' edges (a single block, no block of the final width, a last block of one
bin), against the running block medians in FP64: 2e-5 of a bin's size, the
tolerance of the spectrum tests."""
import math

import numpy as np
import pytest

from coherentsearch_c_b200.spectrum import SpectrumMaker


def restated(x, dt, startwidth, endwidth, endfreq):
    N = x.size
    S = np.fft.rfft(x.astype(np.float64))[:N // 2]
    n2, T = N // 2, np.float32(N * dt)
    starts, lens, pos = [1], [startwidth], 1 + startwidth
    width = int(startwidth * math.log(pos))
    while pos < n2:
        n = min(width, n2 - pos)
        starts.append(pos)
        lens.append(n)
        pos += n
        width = int(startwidth * math.log(pos)) if np.float32(pos) / T < endfreq else endwidth
    p = np.abs(S) ** 2
    lv = np.array([np.sort(p[a:a + n])[(n - 1) // 2] for a, n in zip(starts, lens)]) / math.log(2)
    mid = [a + n // 2 for a, n in zip(starts, lens)]
    out = np.empty(n2, np.complex128)
    out[0] = 1.0
    for k in range(1, n2):
        b = int(np.searchsorted(mid, k, side="right")) - 1
        if b < 0:
            level = lv[0]
        else:
            nb = min(b + 1, len(lv) - 1)
            slope = 1.0 if len(lv) == 1 else \
                (lv[nb] - lv[nb - 1]) / (0.5 * (lens[nb - 1] + lens[nb]))
            level = lv[b] + slope * (k - mid[b])
        y = np.float64(np.array(0x5f3759df - (np.float32(level).view(np.int32) >> 1),
                                np.int32).view(np.float32))
        out[k] = S[k] * y * (1.5 - 0.5 * level * y * y)
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("N,dt,start,end,freq", [(16, 64e-6, 6, 100, 6.0), (40, 64e-6, 6, 100, 6.0),
                                                 (2000, 64e-6, 6, 100, 6.0),
                                                 (20002, 64e-6, 6, 100, 6.0),
                                                 (40000, 64e-6, 6, 100, 1e9),
                                                 (2 * (1 + 6 + 11 + 100 * 9 + 1), 64e-6, 6, 100, 0.1),
                                                 (9000, 2e-3, 3, 64, 6.0), (5000, 64e-6, 2, 128, 0.1)])
def test_normalisation_against_restatement(gpu_ready, N, dt, start, end, freq):
    x = np.random.default_rng(N).standard_normal(N).astype(np.float32)
    try:
        maker = SpectrumMaker(N, dt, start, end, freq)
    except RuntimeError:
        assert freq == 1e9 and start * math.log(N / 2) > end    # the reference stops here too
        return
    with maker:
        got = maker.run(x).view(np.complex64)
    want = restated(x, dt, start, end, freq)
    assert np.abs(got - want).max() <= 2e-5 * max(1.0, np.abs(want).max())
