"""Dedispersion plans of different geometry side by side: each runs after the other was
made, whichever needs more shared memory, and gives what it gives alone."""
import numpy as np
import pytest

from coherentsearch_c_b200.dedisp import Dedisperser, dedisp_tables

L = 2400
GEOMETRIES = [(50000, 1024, 64, 130, 0.4), (30000, 64, 16, 8, 1.0)]


def _make(nspec, nchan, nsub, ndm, step):
    lofreq = 1400.0 + 0.5 * 300.0 / nchan - 150.0
    t = dedisp_tables(nchan, nsub, ndm, 0.0, step, lofreq, 300.0 / nchan, 64e-6, L)
    return Dedisperser(t, max_spectra=nspec)


def _run(dd, geometry):
    import torch
    nspec, nchan, _, ndm, _ = geometry
    g = torch.Generator(device="cuda").manual_seed(nchan)
    raw = torch.randint(0, 256, (nspec, nchan), generator=g, device="cuda", dtype=torch.uint8)
    flags = torch.zeros(nspec // L * L, dtype=torch.uint8, device="cuda")
    flags[9000:9004] = 1
    levels = torch.full((nspec // L, nchan), 100.25, device="cuda")
    nout = dd.output_length(nspec)
    out = [torch.full((ndm, (nout + 3) // 4 * 4), -1.0, device="cuda") for _ in range(2)]
    torch.cuda.synchronize()
    dd.run_device(raw.data_ptr(), nspec, out[0].data_ptr(), out[0].shape[1])
    dd.run_device_clipped(raw.data_ptr(), nspec, flags.data_ptr(), levels.data_ptr(),
                          out[1].data_ptr(), out[1].shape[1])
    torch.cuda.synchronize()
    return [o[:, :nout].cpu().numpy() for o in out]


@pytest.mark.gpu
@pytest.mark.parametrize("order", [(0, 1), (1, 0)])
def test_plans_side_by_side(gpu_ready, order):
    alone = []
    for g in GEOMETRIES:
        with _make(*g) as dd:
            alone.append(_run(dd, g))
    plans = {i: _make(*GEOMETRIES[i]) for i in order}
    for i in order:
        for got, want in zip(_run(plans[i], GEOMETRIES[i]), alone[i]):
            np.testing.assert_array_equal(got, want)
    for dd in plans.values():
        dd.close()
