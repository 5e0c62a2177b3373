"""The one-launch collapse of short record lists and its hand-over to the
long-list path: lists around the block sizes and the 4096-record limit, every
switch combination, against the host's post-processing of the same raw list."""
import itertools

import numpy as np
import pytest

from coherentsearch_c_b200.search import Options, Session


@pytest.mark.gpu
@pytest.mark.parametrize("want", [1, 31, 513, 1025, 4096, 4097, 9000])
def test_short_lists_equal_host_collapse(gpu_ready, want):
    N, dt = 60000, 64e-6
    rng = np.random.default_rng(want)
    amps = (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)
    amps[2 * 400:2 * 400 + 2] = 40.0                # a strong line among noise
    every = Session(N, dt, Options(threshold=1.0, blocksize=5000))
    met = np.sort(every.run_raw(amps)["metric"])[::-1]
    every.close()
    assert met.size > want + 1
    thr = float(0.5 * (met[want - 1] + met[want]))
    for remove, harm in itertools.product((True, False), repeat=2):
        ses = Session(N, dt, Options(threshold=thr, blocksize=5000, remove=remove,
                                     harm_remove=harm))
        raw = ses.run_raw(amps)
        host = ses.collapse(raw)
        assert abs(raw.size - want) <= 2            # equal metrics at the cut
        ses.enqueue(None)
        one, _, rc = ses.collect_collapsed()
        ses.enqueue(None)
        assert ses.collapse_enqueue() == 0          # the two halves
        two, _ = ses.collapse_wait()
        ses.close()
        assert rc == 0
        for f in ("freq", "metric", "r", "nharm"):
            np.testing.assert_array_equal(one[f], host[f])
            np.testing.assert_array_equal(two[f], host[f])
