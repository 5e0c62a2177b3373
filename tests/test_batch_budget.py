"""The batch engine's device memory against its budget: a slot holds no more than was
admitted, whatever the search kernels keep beside the spectrum, and a request that
the budget just takes is taken."""
import threading

import numpy as np
import pytest

from coherentsearch_c_b200 import native as nt
from coherentsearch_c_b200.batch import Batch
from coherentsearch_c_b200.search import Options, Session

DT = 64e-6
OPTS = Options(nharms=60, blocksize=65536, threshold=6.0)


def _spectrum(N, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)


def _needs(N):
    """What admission asks for: spectrum, records, tiles, chunks and 4 MB."""
    total = OPTS.geometry(N, DT)[2]
    nchunks = total // OPTS.blocksize + 2 * OPTS.nharms + 2
    recs = total * 7 // 16 + 4096
    return 8 * (N // 2) + 16 * recs + 12 * (total // 128 + nchunks + 1) + 512 * nchunks + (4 << 20)


@pytest.mark.gpu
@pytest.mark.parametrize("slots,spare", [(1, 1.001), (1, 1.2), (1, 3.0), (2, 2.05), (3, 4.0)])
def test_slots_hold_what_was_admitted(gpu_ready, slots, spare):
    N = 1 << 20
    data = [_spectrum(N, s) for s in range(3)]
    ses = Session(N, DT, OPTS)
    want = [ses.run_raw(a) for a in data]
    ses.close()
    nt.gpu_lib().cs_b200_session_park_drain()
    budget, seen, stop = int(spare * _needs(N)), [], threading.Event()
    with Batch(nslots=slots, mem_budget=budget) as b:
        def look():
            while not stop.is_set():
                seen.append(b.device_bytes())
                stop.wait(2e-4)

        watch = threading.Thread(target=look, daemon=True)
        watch.start()
        try:
            ids = [b.submit(data[i % 3], N, DT, OPTS) for i in range(9)]
            got = [b.wait(i)[0] for i in ids]
        finally:                                    # also where a request failed
            stop.set()
            watch.join()
        seen.append(b.device_bytes())
    for i, g in enumerate(got):
        for f in ("r", "metric", "nharm"):
            np.testing.assert_array_equal(g[f], want[i % 3][f])
    assert 0 < max(seen) <= budget
