"""The overlapped FP64 search (csrc/cs_search_f64.cuh, search_f64_wide) against
the oracle's FP64 metric of every trial and slot, at harmonic counts off the
matrix instruction's multiples, other tap counts and last sub-tiles of every
size; and against search_f64, which geometries without room for it take."""
import ctypes as C

import numpy as np
import pytest

from coherentsearch_c_b200.search import Options, Session

F64_RTOL = 1e-9          # the FP64 tests' tolerance


@pytest.mark.gpu
@pytest.mark.parametrize("nharms,hidr,m,N", [(60, 0.5, 16, 9000), (60, 0.5, 16, 4099),
                                             (32, 0.5, 16, 9001), (16, 0.25, 16, 9002),
                                             (7, 0.5, 16, 20000), (13, 0.5, 12, 12000),
                                             (45, 0.5, 16, 8000), (3, 0.5, 16, 5000)])
def test_all_trial_metrics_against_oracle(gpu_ready, monkeypatch, nharms, hidr, m, N):
    import refbind as rb
    dt = 64e-6
    rng = np.random.default_rng(N)
    amps = (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)
    opts = Options(nharms=nharms, hidr=hidr, m=m, blocksize=1000, threshold=-1e30, remove=False,
                   harm_remove=False, precision=1)
    ses = Session(N, dt, opts)
    assert ses.info().kernel == 2
    raw = ses.run_raw(amps)
    decims = np.array(list(ses.params.decimations)[:ses.params.ndecim], dtype=np.int32)
    nslot = 1 + int((decims > 1).sum())
    met = np.zeros((nslot, ses.total))
    assert rb.oracle_lib().cso_trial_metrics(
        amps.ctypes.data_as(C.POINTER(C.c_float)), amps.size // 2, N, nharms, m, hidr, decims.size,
        decims.ctypes.data_as(C.POINTER(C.c_int)), opts.boxcar_fsp, opts.boxcar_maxfrac, ses.r_lo,
        ses.cstarts.ctypes.data_as(C.POINTER(C.c_longlong)), ses.cstarts.size, ses.total, 0,
        ses.total, 1, met.ctypes.data_as(C.POINTER(C.c_double))) == nslot
    ora = rb.oracle_candidates(met, (ses.r_lo, ses.lodr, ses.total, ses.cstarts, decims), N, dt,
                               opts)
    ses.close()
    monkeypatch.setenv("CS_B200_GENERIC_KERNEL", "1")
    old = Session(N, dt, opts)
    was = old.run_raw(amps)
    old.close()
    for got in (raw, was):
        assert got.size == ora.size
        np.testing.assert_array_equal(got["r"], ora["r"])
        np.testing.assert_array_equal(got["nharm"], ora["nharm"])
        d = np.abs(got["metric"] - ora["metric"]).max()
        assert d <= F64_RTOL * max(1.0, np.abs(ora["metric"]).max())
