"""A session says which kernel it launches, the fast ones apart from those that take over
where they do not fit."""
import pytest

from coherentsearch_c_b200.search import Options, Session


@pytest.mark.gpu
@pytest.mark.parametrize("env,kw,multi,name", [
    (None, {}, False, "search_cols"), (None, {"nharms": 32}, False, "search_cols"),
    (None, {"nharms": 16, "hidr": 0.25}, False, "search_cols"),
    ("CS_B200_WS_KERNEL", {}, False, "search_ws"), (None, {"hidr": 2.0}, False, "search_ws"),
    ("CS_B200_TMA_KERNEL", {}, False, "search_tma"), (None, {"nharms": 7}, False, "cs_search_kernel"),
    ("CS_B200_GENERIC_KERNEL", {}, False, "cs_search_kernel"), (None, {}, True, "search_ws"),
    (None, {"precision": 1}, False, "search_f64_wide"),
    ("CS_B200_GENERIC_KERNEL", {"precision": 1}, False, "search_f64")])
def test_kernel_name(gpu_ready, monkeypatch, env, kw, multi, name):
    from coherentsearch_c_b200 import native as nt
    nt.gpu_lib().cs_b200_session_park_drain()
    if env:
        monkeypatch.setenv(env, "1")
    ses = Session(131072, 64e-6, Options(**kw), multi=multi)
    assert ses.kernel_name() == name
    ses.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nharms,waves,sizes", [(60, 0, (4096, 12288)), (32, 1, (16384, 29000, 33000)),
                                                (16, 2, (65536, 131072, 160000))])
def test_small_searches_take_the_shorter_way(gpu_ready, monkeypatch, nharms, waves, sizes):
    """search_ws for less than a wave or two of tiles, with the same candidates."""
    import numpy as np
    import torch
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    names = set()
    for N in sizes:
        rng = np.random.default_rng(N)
        amps = (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)
        got = []
        for env in (None, "CS_B200_GENERIC_KERNEL"):
            if env:
                monkeypatch.setenv(env, "1")
            ses = Session(N, 64e-6, Options(nharms=nharms, threshold=4.0))
            if env:
                monkeypatch.delenv(env)
            else:
                few = ses.info().ntiles <= waves * sms
                assert ses.kernel_name() == ("search_ws" if few else "search_cols")
                names.add(ses.kernel_name())
            got.append(np.sort(ses.run_raw(amps), order=["r", "nharm"]))
            ses.close()
        assert got[0].size > 0
        for f in ("r", "metric", "nharm"):
            np.testing.assert_array_equal(got[0][f], got[1][f])
    assert len(names) == (2 if waves else 1)
