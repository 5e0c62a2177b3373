"""The register-block search kernel against search_ws, bit for bit, over ladder
configurations, trial spacings (which set the number of window stages: fewer than
interpolation warps at hidr 1, the most at 0.5) and sizes from less than a tile
a CTA to several phase blocks a CTA."""
import numpy as np
import pytest

from coherentsearch_c_b200.search import Options, Session


@pytest.mark.gpu
@pytest.mark.parametrize("nharms", [60, 32, 16])
@pytest.mark.parametrize("hidr", [0.25, 0.5, 1.0])
@pytest.mark.parametrize("N", [9000, 131072, 700001])
def test_same_bits_as_search_ws(gpu_ready, monkeypatch, nharms, hidr, N):
    rng = np.random.default_rng(N)
    amps = (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)
    amps[2 * 411:2 * 411 + 2] = 30.0
    out = []
    for ws in (False, True):
        if ws:
            monkeypatch.setenv("CS_B200_WS_KERNEL", "1")
        ses = Session(N, 64e-6, Options(nharms=nharms, hidr=hidr, threshold=4.0))
        raw = ses.run_raw(amps)
        ses.close()
        out.append(np.sort(raw, order=["r", "nharm"]))
    assert out[0].size > 0
    for f in ("r", "metric", "nharm"):
        np.testing.assert_array_equal(out[0][f], out[1][f])
