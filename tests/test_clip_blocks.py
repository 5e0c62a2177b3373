"""The clip decisions for long blocks, around the length where the statistics
kernel's shared memory needs the device's opt-in (its arrays of fixed size
included) and at the longest, bit for bit against the restatement of clip_times;
and two threads whose blocks differ, whose limits must not meet."""
import ctypes as C
import threading

import numpy as np
import pytest

from test_clip_kernels import clip_times


def _run(raw, L, sigma, stream=None):
    import torch
    from coherentsearch_c_b200 import native as nt
    d = torch.from_numpy(raw).cuda()
    nblk, nchan = raw.shape[0] // L, raw.shape[1]
    flags = torch.full((nblk * L,), 9, dtype=torch.uint8, device="cuda")
    levels = torch.full((nblk, nchan), -1.0, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    n = C.c_longlong(0)
    rc = nt.gpu_lib().cs_clip_levels(d.data_ptr(), raw.shape[0], nchan, L, sigma, C.byref(n),
                                     flags.data_ptr(), levels.data_ptr(), None, 0, stream, 0)
    return rc, flags.cpu().numpy(), levels.cpu().numpy()


def _raw(nblk, L, nchan):
    rng = np.random.default_rng(L)
    raw = np.clip(np.rint(128 + 12 * rng.standard_normal((nblk * L, nchan))), 0, 255).astype(np.uint8)
    raw[L // 3] = 255
    return raw


@pytest.mark.gpu
@pytest.mark.parametrize("L", [2047, 2048, 3061, 3062, 3071, 3072, 8191, 8192])
def test_long_blocks_against_restatement(gpu_ready, L):
    raw = _raw(2, L, 16)
    want_f, want_l = clip_times(raw, L, 4.0)
    rc, flags, levels = _run(raw, L, 4.0)
    assert rc == 0
    np.testing.assert_array_equal(flags, want_f)
    np.testing.assert_array_equal(levels.view(np.uint32), want_l.view(np.uint32))


@pytest.mark.gpu
def test_threads_with_different_blocks(gpu_ready):
    lengths = (3100, 5000, 8192)
    data = {L: _raw(1, L, 16) for L in lengths}
    ref = {L: _run(data[L], L, 4.0) for L in lengths}
    bad = []

    def work(L):
        for _ in range(60):
            got = _run(data[L], L, 4.0)
            if got[0] != 0 or any((a != b).any() for a, b in zip(got[1:], ref[L][1:])):
                bad.append(L)

    threads = [threading.Thread(target=work, args=(L,)) for L in lengths]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert all(r[0] == 0 for r in ref.values()) and not bad
