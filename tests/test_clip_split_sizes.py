"""Which clipped runs are split into integer and FP32 items: large ones, bit for bit what
the FP32 rounds kernel gives for the same plan, and small ones not, whose launches
would cost more than they save."""
import time

import numpy as np
import pytest

from coherentsearch_c_b200.dedisp import Dedisperser, dedisp_tables

L = 2400


def _plan(nspec, nchan, nsub, ndm, step):
    lofreq = 1400.0 + 0.5 * 300.0 / nchan - 150.0
    t = dedisp_tables(nchan, nsub, ndm, 0.0, step, lofreq, 300.0 / nchan, 64e-6, L)
    dd = Dedisperser(t, max_spectra=nspec)
    return dd, dd.output_length(nspec)


def _raw(nspec, nchan):
    import torch
    g = torch.Generator(device="cuda").manual_seed(nspec)
    return torch.randint(0, 256, (nspec, nchan), generator=g, device="cuda", dtype=torch.uint8)


@pytest.mark.gpu
@pytest.mark.parametrize("nspec,nchan,nsub,ndm,step", [(100001, 1024, 64, 9, 0.4),
                                                       (300000, 256, 16, 33, 1.0),
                                                       (130000, 256, 32, 200, 0.5),
                                                       (60000, 1024, 64, 65, 3.0)])
def test_large_runs_equal_fp32_rounds(gpu_ready, monkeypatch, nspec, nchan, nsub, ndm, step):
    import torch
    dd, nout = _plan(nspec, nchan, nsub, ndm, step)
    raw = _raw(nspec, nchan)
    nblk = nspec // L
    levels = 100.0 + 50.0 * torch.rand(nblk, nchan, device="cuda")
    stride = (nout + 3) // 4 * 4
    for at in ([], [0], [nblk * L - 1], [nout // 3, nout // 3 + 255, nout // 2 + 256, nout - 1],
               slice(None)):
        flags = torch.zeros(nblk * L, dtype=torch.uint8, device="cuda")
        flags[at] = 1
        out = []
        for rounds in (False, True):
            if rounds:
                monkeypatch.setenv("CS_B200_DEDISP_ROUNDS", "1")
            o = torch.full((ndm, stride), -1.0, device="cuda")
            torch.cuda.synchronize()
            dd.run_device_clipped(raw.data_ptr(), nspec, flags.data_ptr(), levels.data_ptr(),
                                  o.data_ptr(), stride)
            torch.cuda.synchronize()
            monkeypatch.delenv("CS_B200_DEDISP_ROUNDS", raising=False)
            out.append(o[:, :nout].view(torch.int32))
        assert torch.equal(out[0], out[1])
    dd.close()


@pytest.mark.gpu
@pytest.mark.parametrize("nspec,nchan,nsub,ndm,step", [(12000, 256, 16, 20, 1.0),
                                                       (60000, 64, 16, 20, 1.0)])
def test_small_runs_are_not_split(gpu_ready, nspec, nchan, nsub, ndm, step):
    """With a burst such a run takes up to twice the plain one's two kernels in FP32; the
    split's launches made it 2.6 and 1.9 times, against 1.8 and 1.25."""
    import torch
    dd, nout = _plan(nspec, nchan, nsub, ndm, step)
    raw, stride = _raw(nspec, nchan), (nout + 3) // 4 * 4
    flags = torch.zeros(nspec // L * L, dtype=torch.uint8, device="cuda")
    flags[5000:5004] = 1
    levels = torch.full((nspec // L, nchan), 128.0, device="cuda")
    out = torch.empty(ndm, stride, device="cuda")

    def took(run):
        ts = []
        for _ in range(40):
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            run()
            torch.cuda.synchronize()
            ts.append(time.perf_counter() - t0)
        return float(np.median(ts[8:]))

    st = torch.cuda.current_stream().cuda_stream
    plain = took(lambda: dd.run_device(raw.data_ptr(), nspec, out.data_ptr(), stride, -1, st))
    clipped = took(lambda: dd.run_device_clipped(raw.data_ptr(), nspec, flags.data_ptr(),
                                                 levels.data_ptr(), out.data_ptr(), stride, -1, st))
    dd.close()
    assert clipped < (2.2 if nchan == 256 else 1.6) * plain
