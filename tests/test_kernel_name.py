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
    ses = Session(65536, 64e-6, Options(**kw), multi=multi)
    assert ses.kernel_name() == name
    ses.close()
