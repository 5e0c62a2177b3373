"""Clipped dedispersion split into integer and FP32 items, and the register form
of the subband stage, against a plain FP32 restatement of PRESTO's sums
(dispersion.c:245-264, 346-362: channels from 0, then subbands from -0, in
ascending order), bit for bit: no spectrum flagged, one at either end, runs that
touch single tiles, and every spectrum."""
import numpy as np
import pytest

from coherentsearch_c_b200.dedisp import Dedisperser, dedisp_tables

L = 600


def restated(raw, t, flags, levels, nout):
    nspec, nchan = raw.shape
    x = raw[:, ::-1].astype(np.float32)                    # ascending frequency
    on = np.flatnonzero(flags)
    x[on] = levels[on // L][:, ::-1]
    cps = nchan // t.nsub
    n = nout + int(t.offsets.max())
    S = np.zeros((t.nsub, n), np.float32)
    for c in range(nchan):
        S[c // cps] += x[t.idispdt[c]:t.idispdt[c] + n, c]
    out = np.full((t.ndm, nout), -0.0, np.float32)
    for d in range(t.ndm):
        for s in range(t.nsub):
            out[d] += S[s, t.offsets[d, s]:t.offsets[d, s] + nout]
    return out


@pytest.mark.gpu
@pytest.mark.parametrize("nchan,nsub,ndm", [(256, 16, 40), (256, 32, 33), (1024, 64, 70),
                                            (96, 8, 5), (512, 16, 17)])
@pytest.mark.parametrize("pattern", ["none", "first", "last", "runs", "all"])
def test_split_equals_fp32_sums(gpu_ready, nchan, nsub, ndm, pattern):
    import torch
    t = dedisp_tables(nchan, nsub, ndm, 0.0, 2.0, 1250.0, 300.0 / nchan, 64e-6, L)
    nspec = 11 * L * t.blocks_per_read + 77
    rng = np.random.default_rng(nchan + nsub + ndm)
    raw = rng.integers(0, 256, (nspec, nchan), dtype=np.uint8)
    nblk = nspec // L
    flags = np.zeros(nblk * L, np.uint8)
    levels = rng.uniform(90, 160, (nblk, nchan)).astype(np.float32)
    with Dedisperser(t, max_spectra=nspec) as dd:
        nout = dd.output_length(nspec)
        assert nout > 0
        flags[{"none": [], "first": [0], "last": [flags.size - 1], "all": slice(None),
               "runs": [nout // 3, nout // 3 + 1, nout // 2 + 255, nout // 2 + 256]}[pattern]] = 1
        d = [torch.from_numpy(a).cuda() for a in (raw, flags, levels)]
        stride = (nout + 3) // 4 * 4
        for _ in range(2):                                 # nothing carries over
            out = torch.full((ndm, stride), -1.0, dtype=torch.float32, device="cuda")
            dd.run_device_clipped(d[0].data_ptr(), nspec, d[1].data_ptr(), d[2].data_ptr(),
                                  out.data_ptr(), stride)
            torch.cuda.synchronize()
            want = restated(raw, t, flags, levels, nout)
            np.testing.assert_array_equal(out.cpu().numpy()[:, :nout].view(np.uint32),
                                          want.view(np.uint32))
        if pattern == "none":
            plain = torch.full((ndm, stride), -1.0, dtype=torch.float32, device="cuda")
            dd.run_device(d[0].data_ptr(), nspec, plain.data_ptr(), stride)
            torch.cuda.synchronize()
            np.testing.assert_array_equal(plain.cpu().numpy()[:, :nout].view(np.uint32),
                                          want.view(np.uint32))
