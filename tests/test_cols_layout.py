"""The register-block search kernel's geometry (csrc/cs_search_cols.cuh,
cols_geometry and table_kernel), restated and checked on the CPU against the
per-trial window start of the reference plan (src/interp.c:219-281): every
trial's window lies where its group's zero-padded weight row expects it, inside
its TMA box, and columns are a fixed even number of bins apart.  On the GPU the
kernel's metrics are compared with the oracle's at the edges of its tiles."""
import math

import numpy as np
import pytest

TI, TC, M, FRONT = 16, 8, 16, 16


def geometry(nh, q, p):
    D = 2 * q
    while D % TI:
        D += 2 * q
    if D > 4096:
        return None
    nts, bws = [], []
    for hb in range(nh // 4):
        nt = bw = 0
        for h in range(4 * hb + 1, 4 * hb + 5):
            nt = max(nt, (16 + 1 + -(-3 * h * p // q) + 1) // 2 * 2)
            bw = max(bw, (-(-12 * h * p // q) + 1) // 2 * 2)
        if nt > 20:
            return None
        bw += nt
        bw += 2 if bw % 4 != 2 else 0
        nts.append(nt)
        bws.append(bw)
    return D, nts, bws


def starts(h, r_lo, q, p, t):
    """First bin of the 16-tap window of harmonic h at trials t."""
    hr = h * r_lo
    rf0 = math.floor(hr)
    dr0 = hr - rf0
    prod = t * (h * p)
    carry = (dr0 + (prod % q) / q >= 1.0).astype(np.int64)
    return rf0 + prod // q + carry + 1 - M // 2


@pytest.mark.parametrize("nh,q,p", [(60, 120, 1), (60, 240, 1), (60, 200, 1), (60, 60, 1),
                                    (32, 64, 1), (32, 128, 1), (32, 96, 1), (16, 32, 1),
                                    (16, 64, 1), (16, 80, 3), (60, 1200, 7), (60, 150, 1)])
@pytest.mark.parametrize("r_lo", [0.83886, 100.0, 53.687091, 12.5, 0.0008, 6710.8864])
def test_windows_fit_their_boxes(nh, q, p, r_lo):
    geo = geometry(nh, q, p)
    if geo is None:
        assert q > 1024 or 3 * nh * p > 3 * q     # refused: falls back
        return
    D, nts, bws = geo
    t = np.arange(D, dtype=np.int64)
    for h in range(1, nh + 1):
        nt, bw = nts[(h - 1) // 4], bws[(h - 1) // 4]
        shift = h * p * (D // q)
        assert shift % 2 == 0 and D % q == 0
        b = starts(h, r_lo, q, p, t)
        np.testing.assert_array_equal(starts(h, r_lo, q, p, t + 5 * D), b + 5 * shift)
        b = b.reshape(-1, TI) + FRONT
        assert b.min() >= 0
        x0 = b[:, :1] & ~1
        lead = b[:, ::4] & ~1                     # group starts
        goff = lead - x0
        assert (goff >= 0).all() and (goff // 2 < 256).all()
        assert (goff + nt <= bw).all()
        sh = b.reshape(-1, 4, 4) - lead[:, :, None]
        assert sh.min() >= 0 and sh.max() + M <= nt


@pytest.mark.gpu
@pytest.mark.parametrize("nharms,hidr,N,dt", [
    (60, 0.5, 4096, 64e-6),        # fewer trials than one tile's columns
    (60, 0.5, 40002, 64e-6),
    (60, 0.25, 30000, 64e-6),      # a grid the search_ws kernel does not take
    (60, 1.0, 60001, 64e-6),
    (60, 0.5, 60000, 1.3e-4),      # harmonics run off the top of the spectrum
    (32, 0.5, 50000, 64e-6), (32, 0.3, 33333, 1.3e-4),
    (16, 0.5, 70001, 64e-6), (16, 0.25, 5000, 1.3e-4)])
def test_trial_metrics_against_oracle(gpu_ready, nharms, hidr, N, dt):
    """Every trial's metric of every slot, bound as the other kernels' tests
    bind it: 2e-4 of the largest."""
    import ctypes as C
    import refbind as rb
    from coherentsearch_c_b200.search import Options, Session
    rng = np.random.default_rng(N)
    amps = (rng.standard_normal(2 * (N // 2)) * math.sqrt(0.5)).astype(np.float32)
    opts = Options(nharms=nharms, hidr=hidr, blocksize=1000, threshold=-1e30, remove=False,
                   harm_remove=False)
    ses = Session(N, dt, opts)
    assert ses.info().kernel == 1
    raw = ses.run_raw(amps)
    decims = np.array(list(ses.params.decimations)[:ses.params.ndecim], dtype=np.int32)
    nslot = 1 + int((decims > 1).sum())
    met = np.zeros((nslot, ses.total))
    fp, dp = C.POINTER(C.c_float), C.POINTER(C.c_double)
    assert rb.oracle_lib().cso_trial_metrics(
        amps.ctypes.data_as(fp), amps.size // 2, N, nharms, opts.m, hidr, decims.size,
        decims.ctypes.data_as(C.POINTER(C.c_int)), opts.boxcar_fsp, opts.boxcar_maxfrac, ses.r_lo,
        ses.cstarts.ctypes.data_as(C.POINTER(C.c_longlong)), ses.cstarts.size, ses.total, 0,
        ses.total, 0, met.ctypes.data_as(dp)) == nslot
    geo = (ses.r_lo, ses.lodr, ses.total, ses.cstarts, decims)
    ora = rb.oracle_candidates(met, geo, N, dt, opts)
    ses.close()
    assert raw.size == ora.size
    np.testing.assert_array_equal(raw["r"], ora["r"])
    np.testing.assert_array_equal(raw["nharm"], ora["nharm"])
    err = np.abs(raw["metric"] - ora["metric"]).max()
    assert err <= 2e-4 * max(1.0, np.abs(ora["metric"]).max())
