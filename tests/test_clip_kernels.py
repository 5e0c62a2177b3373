"""The clip decisions and channel levels on the device against a plain
restatement of clip_times (PRESTO clipping.c:47-230, avg_var of
misc_utils.c:641-676), bit for bit, at the edges of the kernels' shapes: channel
counts around a warp's columns and off the 16-byte path, blocks around the CTA
sizes, a block without good spectra, cut-offs that move with interference."""
import numpy as np
import pytest


def _avg_var(x):
    """The sequential mean and variance of avg_var in FP64."""
    if len(x) == 0:
        return 0.0, 0.0
    mean, acc = np.float64(x[0]), np.float64(0.0)
    for n in range(1, len(x)):
        an, an1 = np.float64(n + 1), np.float64(n)
        dx = (np.float64(x[n]) - mean) / an
        acc = acc + an * an1 * dx * dx
        mean = mean + dx
    return mean, acc / np.float64(len(x) - 1) if len(x) > 1 else acc


def clip_times(raw, L, clip_sigma):
    nblk, nchan = raw.shape[0] // L, raw.shape[1]
    flags = np.zeros(nblk * L, np.uint8)
    levels = np.zeros((nblk, nchan), np.float32)
    f32, f64 = np.float32, np.float64
    ravg = rstd = f32(0)
    lev = np.zeros(nchan, np.float32)
    for b in range(nblk):
        rows = raw[b * L:(b + 1) * L].astype(np.int64)
        z = rows.sum(1).astype(np.float32)
        med = f64(np.sort(z)[(L - 1) // 2])
        sd = np.sqrt(_avg_var(z)[1])
        lo, hi = f32(med - 3.0 * sd), f32(med + 3.0 * sd)
        good = (z > lo) & (z < hi)
        ng = int(good.sum())
        mean, var = _avg_var(z[good])
        cur = (mean, np.sqrt(var)) if ng else (f64(ravg), f64(rstd))
        cl = rows[good].sum(0).astype(np.float32).astype(f64) / f64(max(ng, 1))
        cl = cl if ng else lev.astype(f64)
        if b:
            ravg = f32(0.9 * f64(ravg) + 0.1 * cur[0])
            rstd = f32(0.9 * f64(rstd) + 0.1 * cur[1])
            lev = (0.9 * lev.astype(f64) + 0.1 * cl).astype(np.float32)
        else:
            ravg, rstd, lev = f32(cur[0]), f32(cur[1]), cl.astype(np.float32)
        trig = f32(clip_sigma) * rstd
        flags[b * L:(b + 1) * L] = np.abs((z - ravg).astype(f64)) > f64(trig)
        levels[b] = lev
    return flags, levels


@pytest.mark.gpu
@pytest.mark.parametrize("nchan,L,nblk", [(16, 1, 3), (16, 2, 40), (48, 239, 17), (512, 240, 5),
                                          (528, 241, 4), (1024, 300, 33), (1040, 257, 3),
                                          (2064, 64, 3), (4096, 31, 2), (4112, 31, 2),
                                          (33, 256, 5), (64, 2400, 3)])
def test_levels_against_restatement(gpu_ready, nchan, L, nblk):
    import ctypes as C
    import torch
    from coherentsearch_c_b200 import native as nt
    rng = np.random.default_rng(nchan * 1000 + L)
    raw = np.clip(np.rint(128 + 12 * rng.standard_normal((nblk * L + L // 2, nchan))), 0,
                  255).astype(np.uint8)
    raw[L // 3] = 255                               # a burst, a dropout, a flat block
    raw[(nblk - 1) * L + L // 2] = 0
    raw[(nblk // 2) * L:(nblk // 2 + 1) * L] = 7
    want_f, want_l = clip_times(raw, L, 4.0)
    d = torch.from_numpy(raw).cuda()
    flags = torch.full((nblk * L,), 9, dtype=torch.uint8, device="cuda")
    levels = torch.full((nblk, nchan), -1.0, dtype=torch.float32, device="cuda")
    n = C.c_longlong(0)
    gpu = nt.gpu_lib()
    for lev in (levels, None):
        fn = gpu.cs_clip_levels if lev is not None else gpu.cs_clip_count
        args = (d.data_ptr(), raw.shape[0], nchan, L, 4.0, C.byref(n), flags.data_ptr())
        args += ((lev.data_ptr(),) if lev is not None else ()) + (None, 0, None, 0)
        assert fn(*args) == 0
        torch.cuda.synchronize()
        assert n.value == int(want_f.sum())
        np.testing.assert_array_equal(flags.cpu().numpy(), want_f)
    np.testing.assert_array_equal(levels.cpu().numpy().view(np.uint32), want_l.view(np.uint32))
