"""Sessions for multi-spectrum launches: without the second spectrum copy and the tables
of the kernel that they never launch, and with the same candidates."""
import numpy as np
import pytest

from coherentsearch_c_b200 import native as nt
from coherentsearch_c_b200.search import Options, Session, multi_search
from coherentsearch_c_b200.sweep import search_list

DT = 64e-6


def _spectrum(N, seed):
    rng = np.random.default_rng(seed)
    return (rng.standard_normal(2 * (N // 2)) * np.sqrt(0.5)).astype(np.float32)


def _taken(make):
    """Device bytes that `make`'s session takes; the first one loads the kernels."""
    import torch
    for _ in range(2):
        nt.gpu_lib().cs_b200_session_park_drain()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        ses = make()
        after = torch.cuda.mem_get_info()[0]
        ses.close()
    nt.gpu_lib().cs_b200_session_park_drain()
    return before - after


@pytest.mark.gpu
@pytest.mark.parametrize("nharms", [60, 32, 16])
def test_multi_sessions_hold_one_spectrum(gpu_ready, nharms):
    N = 1 << 23
    opts = Options(nharms=nharms)
    one = _taken(lambda: Session(N, DT, opts))
    many = _taken(lambda: Session(N, DT, opts, multi=True))
    assert one - many >= 8 * (N // 2)


@pytest.mark.gpu
def test_same_candidates(gpu_ready):
    import torch
    opts = Options(threshold=4.5)
    data = [(N, _spectrum(N, N)) for N in (65536, 90002, 131072)]
    plain, multi = [], []
    for N, amps in data:
        for sessions, kw in ((plain, {}), (multi, {"multi": True})):
            ses = Session(N, DT, opts, **kw)
            sessions.append((ses, ses.run_raw(amps)))
    got, _ = multi_search([s for s, _ in multi])
    dev = [torch.from_numpy(a).cuda() for _, a in data]
    torch.cuda.synchronize()
    listed = search_list([(N, d.data_ptr()) for (N, _), d in zip(data, dev)], DT, opts, 2)
    for (_, want), (_, alone), a, b in zip(plain, multi, got, listed):
        assert want.size > 0
        for x in (alone, a, b):
            for f in ("r", "metric", "nharm"):
                np.testing.assert_array_equal(x[f], want[f])
    for s, _ in plain + multi:
        s.close()
