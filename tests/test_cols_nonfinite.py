"""A spectrum bin that is not finite reaches the trials whose own taps have it and
no others: a session of the register-block search kernel, whose windows are wider
than a trial's taps, against search_ws bit for bit (also with bins that are finite but
flagged as too large), with such bins at both ends, beside each other and under a
pulsar, by each way its records are collected, and finite spectra after it."""
import numpy as np
import pytest

from coherentsearch_c_b200.search import Options, Session


@pytest.mark.gpu
@pytest.mark.parametrize("nharms,hidr", [(60, 0.5), (60, 1.0), (32, 0.5), (16, 0.25)])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan, 3.2e38])
def test_same_bits_as_search_ws(gpu_ready, monkeypatch, nharms, hidr, value):
    N = 131072
    rng = np.random.default_rng(nharms)
    amps = (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)
    for h in range(1, 61):                          # a pulsar, one harmonic spoiled
        amps[2 * 411 * h:2 * 411 * h + 2] = 6.0
    for at in (0, 1, 2 * 411 * 7 - 18, 2 * 411 * 7 + 17, 40001, 40002, 90007, amps.size - 1):
        amps[at] = value
    out = []
    for ws in (False, True):
        if ws:
            monkeypatch.setenv("CS_B200_WS_KERNEL", "1")
        ses = Session(N, 64e-6, Options(nharms=nharms, hidr=hidr, threshold=3.0))
        got = [ses.run_raw(amps)]                   # uploads it
        ses.enqueue(None)
        got.append(ses.collect()[0])
        ses.enqueue(None, threshold=8.0)            # a short list, and a long one
        got.append(ses.collect_collapsed(threshold=8.0)[0])
        ses.enqueue(None)
        got.append(ses.collect_collapsed()[0])
        ses.enqueue(None, threshold=6.0)
        assert ses.collapse_enqueue(threshold=6.0) == 0
        got.append(ses.collapse_wait()[0])
        got.append(ses.run_raw(np.nan_to_num(amps, nan=0.5, posinf=1.0, neginf=1.0) % 8.0))
        ses.close()
        out.append(got)
    assert all(a.size > 10 for a in out[1][:2]) and out[1][2].size > 0
    for new, old in zip(*out):
        for f in ("r", "metric", "nharm"):
            np.testing.assert_array_equal(new[f], old[f])


@pytest.mark.gpu
@pytest.mark.parametrize("at", [0, 1, 199, 30006])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_one_component_alone(gpu_ready, monkeypatch, at, value):
    """Beside a finite other component, which a maximum of the two would show."""
    N = 65536
    rng = np.random.default_rng(at)
    amps = (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)
    amps[at] = value
    out = []
    for ws in (False, True):
        if ws:
            monkeypatch.setenv("CS_B200_WS_KERNEL", "1")
        ses = Session(N, 64e-6, Options(threshold=3.0))
        out.append(np.sort(ses.run_raw(amps), order=["r", "nharm"]))
        ses.close()
    assert out[1].size > 100
    for f in ("r", "metric", "nharm"):
        np.testing.assert_array_equal(out[0][f], out[1][f])
