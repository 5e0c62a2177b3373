"""remove_harmonics on the device for lists past what one CTA orders in shared
memory (csrc/cs_collapse.cu, order_and_walk): lists of every record, and runs that
stay more than that after remove_duplicates, around the walk's own limit, against
the host's post-processing; and the time of the ordering, which may not grow with
the square of the list."""
import ctypes as C
import time

import numpy as np
import pytest

from coherentsearch_c_b200 import native as nt
from coherentsearch_c_b200.search import Options, Session


def _spectrum(N, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)


def _thresholds(N, amps, wants, **kw):
    every = Session(N, 64e-6, Options(threshold=1.0, blocksize=5000, **kw))
    met = np.sort(every.run_raw(amps)["metric"])[::-1]
    every.close()
    assert met.size > max(wants) + 1
    return [float(0.5 * (met[w - 1] + met[w])) for w in wants]


@pytest.mark.gpu
@pytest.mark.parametrize("remove,drtol", [(False, 1.0), (True, 1e-3), (True, 0.02)])
@pytest.mark.parametrize("want", [4097, 8192, 8193, 20000, 60000])
def test_long_lists_equal_host_collapse(gpu_ready, remove, drtol, want):
    N = 60000
    amps = _spectrum(N, want)
    thr, = _thresholds(N, amps, [want])
    ses = Session(N, 64e-6, Options(threshold=thr, blocksize=5000, remove=remove, drtol=drtol))
    raw = ses.run_raw(amps)
    host = ses.collapse(raw)
    ses.enqueue(None)
    one, _, rc = ses.collect_collapsed()
    ses.enqueue(None)
    assert ses.collapse_enqueue() == 0
    two, _ = ses.collapse_wait()
    ses.close()
    assert rc == 0 and raw.size > 4096
    for f in ("freq", "metric", "r", "nharm"):
        np.testing.assert_array_equal(one[f], host[f])
        np.testing.assert_array_equal(two[f], host[f])


def _time(N, amps, thr, opts, remove, harm_tol):
    """Best wall time of a collapse, and the number of its candidates."""
    ses = Session(N, 64e-6, opts)
    ses.run_raw(amps)
    best, n = 1e9, 0
    for _ in range(5):
        cl, ms = nt.CandidateList(), C.c_float(0)
        ses.enqueue(None)
        ses.gpu.cs_b200_session_sync(ses.sess)
        t0 = time.perf_counter()
        rc = ses.gpu.cs_b200_session_collect_collapsed(ses.sess, thr, int(remove), 1e-3, 1, 16,
                                                       harm_tol, C.byref(cl), C.byref(ms))
        best = min(best, time.perf_counter() - t0)
        assert rc == 0
        n = cl.n
        ses.host.candlist_free(C.byref(cl))
    ses.close()
    return best, n


@pytest.mark.gpu
@pytest.mark.parametrize("remove", [False, True])
def test_ordering_does_not_grow_with_the_square(gpu_ready, remove):
    """Every candidate is related to the first (a tolerance as wide as the band), so
    the walk is one step and the ordering is what is timed."""
    N, wants = 200000, (8000, 64000)
    amps = _spectrum(N, 5)
    took = []
    for thr, want in zip(_thresholds(N, amps, wants, lofreq=12.0), wants):
        opts = Options(threshold=thr, blocksize=5000, lofreq=12.0)
        t, n = _time(N, amps, thr, opts, remove, 1e12)
        assert 0 < n < want // 8
        took.append(t)
    assert took[1] < 22.0 * took[0]                 # between linear, 8, and the square, 64


@pytest.mark.gpu
def test_one_launch_is_not_the_slower_one(gpu_ready):
    """Noise, some hundred candidates kept: a list just short enough for one launch
    against one just past it, whose walk is the plain one."""
    N, wants = 400000, (4090, 4110)
    amps = _spectrum(N, 6)
    short, long = (_time(N, amps, thr, Options(threshold=thr), False, 1.0)[0]
                   for thr in _thresholds(N, amps, wants))
    assert short < 1.05 * long


@pytest.mark.gpu
@pytest.mark.parametrize("numharm", [1 << 19, 1 << 21, (1 << 21) + 1, 1 << 24])
@pytest.mark.parametrize("want", [300, 1500, 4500])
def test_many_harmonics(gpu_ready, want, numharm):
    """Numbers of (candidate, harmonic) pairs around 2^31 and past 2^32."""
    N = 60000
    amps = _spectrum(N, want)
    thr, = _thresholds(N, amps, [want])
    ses = Session(N, 64e-6, Options(threshold=thr, blocksize=5000, numharm=numharm, remove=False))
    host = ses.collapse(ses.run_raw(amps))
    ses.enqueue(None)
    got, _, rc = ses.collect_collapsed()
    ses.close()
    assert rc == 0 and 0 < host.size < want // 4
    for f in ("freq", "metric", "r", "nharm"):
        np.testing.assert_array_equal(got[f], host[f])
