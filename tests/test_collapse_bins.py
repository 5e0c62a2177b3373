"""remove_duplicates by bins along r (in memory for long record lists, hashed for
short ones), and by the sort where the bins or the runs are too many: tolerances on both sides of that rule, runs of many
bins, equal metrics, against the host's post-processing of the same raw list."""
import numpy as np
import pytest

from coherentsearch_c_b200.search import Options, Session


@pytest.mark.gpu
@pytest.mark.parametrize("drtol", [1e-3, 0.037, 0.5, 1.0, 7.3, 1e9])
@pytest.mark.parametrize("kind", ["noise", "repeated"])
@pytest.mark.parametrize("want", [40, 1500, 4000, 4500, 30000])
def test_bins_equal_host_collapse(gpu_ready, drtol, kind, want):
    N, dt = 60000, 64e-6
    rng = np.random.default_rng(want)
    if kind == "noise":
        amps = rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)
    else:                                           # the same metric at many places
        amps = np.tile(rng.standard_normal(200), N // 2 // 100 + 1)[:2 * (N // 2)]
    amps = amps.astype(np.float32)
    every = Session(N, dt, Options(threshold=1.0, blocksize=5000))
    met = np.sort(every.run_raw(amps)["metric"])[::-1]
    every.close()
    assert met.size > want + 1
    thr = float(0.5 * (met[want - 1] + met[want]))
    harm = want < 10000                             # a long list walks serially
    ses = Session(N, dt, Options(threshold=thr, blocksize=5000, drtol=drtol, harm_remove=harm))
    raw = ses.run_raw(amps)
    host = ses.collapse(raw)
    assert (raw.size > 4096) == (want > 4096)
    for _ in range(2):                              # first use of the buffers, and again
        ses.enqueue(None)
        got, _, rc = ses.collect_collapsed()
        assert rc == 0
        for f in ("freq", "metric", "r", "nharm"):
            np.testing.assert_array_equal(got[f], host[f])
    ses.close()
