"""The work a user of this package has it do, as measurable cases.

Kinds of case, each through the entry point a program calls for it:

  search    Session.enqueue + Session.collect_collapsed on a spectrum that is
            already on the device: one spectrum of a survey pointing or DM
            series, tables kept by the program, the candidate list out.
  file      search_spectrum on a host spectrum: the whole per-file call
            (planning, session, upload, search, collapse), as the list driver
            makes it.
  dedisp    Dedisperser.run_device on an 8-bit filterbank on the device; with
            `clipped`, the run prepsubband makes by default: clip_levels, then
            run_device_clipped.
  spectrum  SpectrumMaker.run_device: time series to normalised spectrum.
  prep      PrepSearch.run: filterbank to the candidates of every DM.

A search case's dict holds the series length N, the harmonic count, the trial
spacing hidr and the precision; a dedispersion case the filterbank's shape and
the DM grid.
"""
import math
from fractions import Fraction

import numpy as np
import torch

from coherentsearch_c_b200.dedisp import Dedisperser, dedisp_tables
from coherentsearch_c_b200.prep import PrepSearch
from coherentsearch_c_b200.search import Options, Session, search_spectrum
from coherentsearch_c_b200.spectrum import SpectrumMaker

DT = 64e-6
TAPS = 16
THRESHOLD = 8.0
MAXDECIM = 6
LOFREQ, HIFREQ = 0.1, 125.0
BLOCKSIZE = 65536
FCTR, BW = 1400.0, 300.0        # MHz
SPECTRA_PER_SUBINT = 2400
CLIP_SIGMA = 6.0


def search_case(name, N, nharms=60, hidr=0.5, precision=0, kind="search"):
    return {"name": name, "kind": kind, "N": N, "nharms": nharms, "hidr": hidr,
            "precision": precision}


def dedisp_case(name, nspec, nchan, nsub, ndm, dmstep, clipped=False, kind="dedisp"):
    return {"name": name, "kind": kind, "nspec": nspec, "nchan": nchan, "nsub": nsub, "ndm": ndm,
            "dmstep": dmstep, "clipped": clipped}


def listed():
    return [
        # a short pointing: one call's latency counts
        search_case("search_128k", 1 << 17),
        # an ordinary pointing of about a minute
        search_case("search_1m", 1 << 20),
        # a nine-minute pointing, the longest the sweeps search
        search_case("search_8m", 1 << 23),
        # fewer harmonics, a ragged length
        search_case("search_3m_nh32", 3141590, nharms=32),
        # few harmonics at half the usual trial spacing
        search_case("search_2m_nh16", 2200002, nharms=16, hidr=0.25),
        # the FP64 precision mode
        search_case("search_512k_f64", 1 << 19, precision=1),
        # the per-file call of a list driver, spectrum in host memory
        search_case("file_1500k", 1500000, kind="file"),
        # a survey beam's front end: 1024 channels, 500 DMs
        dedisp_case("dedisp_500dm", 500000, 1024, 64, 500, 0.4),
        # the same with prepsubband's clipping, a few bursts of interference
        dedisp_case("dedisp_clip_500dm", 300000, 1024, 64, 500, 0.4, clipped=True),
        # a narrow grid over a small filterbank
        dedisp_case("dedisp_40dm", 100001, 256, 16, 40, 1.0),
        # one series to its normalised spectrum, a ragged length
        {"name": "spectrum_4m", "kind": "spectrum", "N": 4100000},
        # a small filterbank all the way to candidates
        dedisp_case("prep_32dm", 150000, 256, 32, 32, 1.0, kind="prep"),
    ]


def draw(rng):
    def log_size(lo, hi):
        return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))

    u = rng.random()
    if u < 0.45:
        nharms = rng.choice([60, 60, 60, 32, 16])
        hidr = rng.choice([0.5, 0.5, 0.5, 0.25])
        c = search_case("", log_size(1 << 17, 1 << 23 if hidr == 0.5 else 1 << 22), nharms, hidr)
    elif u < 0.55:
        c = search_case("", log_size(1 << 16, 1 << 19), rng.choice([60, 32, 16]), precision=1)
    elif u < 0.62:
        c = search_case("", log_size(1 << 17, 1 << 22), rng.choice([60, 60, 32, 16]), kind="file")
    elif u < 0.85:
        if rng.random() < 0.6:
            c = dedisp_case("", log_size(60000, 500000), 1024, 64, rng.randint(100, 500), 0.4)
        else:
            c = dedisp_case("", log_size(40000, 300000), 256, rng.choice([16, 32]),
                            rng.randint(20, 120), rng.choice([0.5, 1.0]))
        c["clipped"] = rng.random() < 0.4
        if c["clipped"]:
            c["nspec"] = min(c["nspec"], 300000)
    elif u < 0.95:
        c = {"name": "", "kind": "spectrum", "N": 2 * log_size(1 << 16, 1 << 22)}
    else:
        c = dedisp_case("", log_size(60000, 150000), 256, 32, rng.randint(8, 32), 1.0, kind="prep")
    del c["name"]
    return c


# ---------------------------------------------------------------- inputs


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _pulse(phase, duty):
    """A von Mises pulse of FWHM `duty` turns at `phase` turns."""
    kappa = math.log(2.0) / (1.0 - math.cos(math.pi * duty))
    return torch.exp(kappa * (torch.cos(2.0 * math.pi * phase) - 1.0))


def _series(N, seed):
    """White noise with three pulsars (1.7, 29.4 and 311 Hz)."""
    g = _generator(seed)
    x = torch.randn(N, generator=g, device="cuda", dtype=torch.float64)
    t = torch.arange(N, device="cuda", dtype=torch.float64) * DT
    shift = torch.rand(6, generator=g, device="cuda", dtype=torch.float64).tolist()
    for i, (f0, duty, snr) in enumerate([(1.7, 0.10, 40.0), (29.4, 0.05, 20.0),
                                         (311.0, 0.02, 10.0)]):
        s = _pulse(t * (f0 * (1.0 + 0.01 * shift[i])) + shift[3 + i], duty)
        s -= s.mean()
        x += s * (snr / s.norm())
    return x


def _spectrum(N, seed):
    """complex64[N/2], unit mean noise power, bin 0 as rednoise leaves it."""
    S = torch.fft.rfft(_series(N, seed))[:N // 2] / math.sqrt(N)
    S[0] = 1.0
    return S.to(torch.complex64).contiguous()


def _filterbank(case, seed):
    """[nspec][nchan] uint8, highest frequency first, a pulsar at DM 30."""
    nspec, nchan = case["nspec"], case["nchan"]
    g = _generator(seed)
    freqs = _lofreq(nchan) + (BW / nchan) * torch.arange(nchan, device="cuda", dtype=torch.float64)
    delay = 30.0 / (0.000241 * freqs * freqs)
    raw = torch.empty((nspec, nchan), dtype=torch.uint8, device="cuda")
    for t0 in range(0, nspec, 1 << 15):
        n = min(1 << 15, nspec - t0)
        t = (t0 + torch.arange(n, device="cuda", dtype=torch.float64))[:, None] * DT
        pulse = _pulse((4.1 * (t - delay[None, :])).float(), 0.04)
        x = 128.0 + 12.0 * (torch.randn((n, nchan), generator=g, device="cuda") + 0.4 * pulse)
        raw[t0:t0 + n] = x.round_().clamp_(0, 255).flip(1).to(torch.uint8)
    if case["clipped"]:             # broadband bursts of four spectra
        at = torch.randint(0, nspec - 4, (12,), generator=g, device="cuda").tolist()
        for a in at:
            raw[a:a + 4] = 255
    return raw


def _lofreq(nchan):
    return FCTR + 0.5 * BW / nchan - 0.5 * BW


def _tables(case):
    return dedisp_tables(case["nchan"], case["nsub"], case["ndm"], 0.0, case["dmstep"],
                         _lofreq(case["nchan"]), BW / case["nchan"], DT)


def _options(case):
    return Options(nharms=case["nharms"], hidr=case["hidr"], threshold=THRESHOLD,
                   maxdecim=MAXDECIM, precision=case["precision"])


# ---------------------------------------------------------------- the calls


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "search":
        s["amps"] = _spectrum(case["N"], seed)
        s["session"] = Session(case["N"], DT, _options(case))
    elif kind == "file":
        s["amps"] = _spectrum(case["N"], seed).cpu().numpy()
    elif kind == "spectrum":
        s["series"] = _series(case["N"], seed).float()
        s["out"] = torch.empty(case["N"], dtype=torch.float32, device="cuda")
        s["maker"] = SpectrumMaker(case["N"], DT)
    else:
        t = _tables(case)
        s["raw"] = _filterbank(case, seed)
        if kind == "prep":
            opts = Options(nharms=60, threshold=THRESHOLD, maxdecim=MAXDECIM)
            s["prep"] = PrepSearch(t, case["nspec"], case["nspec"] & ~1, DT, opts,
                                   clip_sigma=CLIP_SIGMA)
        else:
            d = Dedisperser(t, max_spectra=case["nspec"])
            s["dedisp"], s["nout"] = d, d.output_length(case["nspec"])
            s["out"] = torch.empty((case["ndm"], (s["nout"] + 3) // 4 * 4), dtype=torch.float32,
                                   device="cuda")
            if case["clipped"]:
                nblk = case["nspec"] // SPECTRA_PER_SUBINT
                s["flags"] = torch.empty(nblk * SPECTRA_PER_SUBINT, dtype=torch.uint8,
                                         device="cuda")
                s["levels"] = torch.empty((nblk, case["nchan"]), dtype=torch.float32,
                                          device="cuda")
                s["scratch"] = torch.empty(d.clip_scratch_bytes(case["nspec"]),
                                           dtype=torch.uint8, device="cuda")
    return s


def _columns(cands):
    """A candidate list as columns, with zeros after its last candidate."""
    n = len(cands["r"])
    room = max(1, -(-n // 1024)) * 1024
    out = {"count": n}
    for f in ("freq", "metric", "r", "nharm"):
        out[f] = np.zeros(room, cands[f].dtype)
        out[f][:n] = cands[f]
    return out


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "search":
        ses, stream = state["session"], torch.cuda.current_stream().cuda_stream
        f64 = case["precision"] == 1            # collapsed on the host
        again = 1
        while again == 1:           # 1: the record buffer was grown, search again
            ses.enqueue(state["amps"].data_ptr(), after_stream=stream)
            cands, _, again = ses.collect() if f64 else ses.collect_collapsed()
        return _columns(ses.collapse(cands) if f64 else cands)
    if kind == "file":
        return _columns(search_spectrum(state["amps"], case["N"], DT, _options(case)))
    if kind == "spectrum":
        state["maker"].run_device(state["series"].data_ptr(), state["out"].data_ptr())
        return state["out"]
    if kind == "prep":
        lists = state["prep"].run(state["raw"].data_ptr(), case["nspec"])
        out = _columns(np.concatenate(lists))
        out["counts"] = np.array([c.size for c in lists])
        return out
    d, raw, out, nspec = state["dedisp"], state["raw"], state["out"], case["nspec"]
    if not case["clipped"]:
        d.run_device(raw.data_ptr(), nspec, out.data_ptr(), out.shape[1])
        return out[:, :state["nout"]]
    flags, levels, scratch = state["flags"], state["levels"], state["scratch"]
    stream = torch.cuda.current_stream().cuda_stream
    d.clip_levels(raw.data_ptr(), nspec, flags.data_ptr(), levels.data_ptr(), CLIP_SIGMA, stream,
                  scratch.data_ptr(), scratch.numel())
    d.run_device_clipped(raw.data_ptr(), nspec, flags.data_ptr(), levels.data_ptr(),
                         out.data_ptr(), out.shape[1], -1, stream)
    return {"flags": flags, "levels": levels, "series": out[:, :state["nout"]]}


# ---------------------------------------------------------------- least work


def _trials(case):
    T = case["N"] * DT
    lodr = case["hidr"] / case["nharms"]
    return int(math.floor((HIFREQ * T - LOFREQ * T) / lodr)) + 1


def _search_work(case):
    """Bytes and flops of one search: the spectrum once; per trial the
    windowed sums and rotations, an FFT's flops for the profile, and one add
    and one maximum per profile bin and width."""
    nh = case["nharms"]
    per = nh * (4 * TAPS + 6) + 5 * nh * math.log2(2 * nh)
    for k in range(1, MAXDECIM + 1):
        nb = 2 * (nh // k)
        per += nb + 2 * nb * len(_widths(nb, k))
    return {"bytes": 8 * (case["N"] // 2), "flops": per * _trials(case)}


def _out_length(case):
    T = _tables_np(case)[2]
    nb = case["nspec"] // SPECTRA_PER_SUBINT
    return max((nb - 1) // T - 1, 0) * SPECTRA_PER_SUBINT * T if nb >= 1 else 0


def _dedisp_work(case):
    nout = _out_length(case)
    return {"bytes": case["nspec"] * case["nchan"] + 4 * case["ndm"] * nout,
            "flops": case["nspec"] * case["nchan"] + case["ndm"] * case["nsub"] * nout}


def _spectrum_work(N):
    return {"bytes": 8 * N, "flops": 2.5 * N * math.log2(N) + 6 * N}


def work(case):
    kind = case["kind"]
    if kind in ("search", "file"):
        return _search_work(case)
    if kind == "spectrum":
        return _spectrum_work(case["N"])
    if kind == "dedisp":
        return _dedisp_work(case)
    w, N = _dedisp_work(case), case["nspec"] & ~1
    one = _search_work({"N": N, "nharms": 60, "hidr": 0.5})
    s = _spectrum_work(N)
    return {"bytes": w["bytes"], "flops": w["flops"] + case["ndm"] * (one["flops"] + s["flops"])}


# ---------------------------------------------------------------- 64-bit results


def _widths(nb, k):
    """The ladder's boxcar widths of an nb-bin profile at decimation k."""
    wmax = min(max(int(math.floor(0.3 * nb)), 1), nb - 1)
    full, w = [], 1
    while w <= wmax:
        full.append(w)
        w = max(int(math.floor(1.5 * w)), w + 1)
    kept = [w for w in full if (w >= 2 or k == 1) and (w <= 6 or k == MAXDECIM)]
    return kept or full


def _noise_scales(filled, k, nh):
    """shape[w] / sigma of decimation k for one set of active harmonics."""
    H = nh // k
    nb = 2 * H
    j = np.arange(1, H)
    low = filled[j * k - 1]
    nyq = filled[H * k - 1]
    sigma = math.sqrt(2.0 * low.sum() + 0.5 * nyq)
    out = []
    for w in _widths(nb, k):
        d = np.sin(np.pi * ((j * w / nb) % 2.0)) / np.sin(np.pi * (j / nb))
        v = float((2.0 * d * d)[low].sum())
        if nyq:
            v += 0.5 * math.sin(math.pi * ((0.5 * w) % 2.0)) ** 2
        out.append(1.0 / math.sqrt(v) if sigma > 0 and v > 1e-12 else 0.0)
    return out


def _exact_search(amps, N, nh, hidr):
    """Every trial's metrics in FP64, thresholded and collapsed."""
    T = N * DT
    r_lo, lodr = LOFREQ * T, hidr / nh
    case = {"N": N, "nharms": nh, "hidr": hidr}
    total = _trials(case)
    grid = Fraction(lodr).limit_denominator(1 << 16)
    pnum, q = grid.numerator, grid.denominator
    a = amps.to(torch.complex128)
    namps, m2 = a.numel(), TAPS // 2
    h = torch.arange(1, nh + 1, device="cuda")
    hr = h.double() * r_lo
    rf0 = torch.floor(hr)
    dr0, rf0 = hr - rf0, rf0.long()
    tap = torch.arange(TAPS, device="cuda")
    found = []
    for i0 in range(0, total, 32768):
        t = torch.arange(i0, min(total, i0 + 32768), device="cuda")
        prod = t[:, None] * (h * pnum)[None, :]
        whole, res = prod // q, prod % q
        u = dr0 + res.double() / q
        carry = (u >= 1.0)
        dr = torch.where(carry, u - 1.0, u)
        base = rf0 + whole + carry.long()
        fits = (base + 2 - m2 >= 1) & (base + 1 + m2 <= namps) & (rf0 + whole < N // 2)
        v = a[(base[:, :, None] + (1 - m2) + tap).clamp_(0, namps - 1)]
        off = dr[:, :, None] - (tap + 1 - m2).double()
        w = torch.where(dr[:, :, None] == 0.0, (tap == m2 - 1).double(), 1.0 / off)
        s, c = torch.sin(math.pi * dr), torch.cos(math.pi * dr)
        gain = torch.complex(s * c, -s * s) / math.pi
        gain = torch.where(dr == 0.0, torch.ones_like(gain), gain)
        X = torch.where(fits, gain * (v * w).sum(2), torch.zeros_like(gain))
        pats, which = torch.unique(fits, dim=0, return_inverse=True)
        pats = pats.cpu().numpy()
        for slot, k in enumerate(range(1, MAXDECIM + 1)):
            H = nh // k
            nb = 2 * H
            stack = torch.zeros((t.numel(), H + 1), dtype=torch.complex128, device="cuda")
            stack[:, 1:] = X[:, k - 1:H * k:k]
            stack[:, H].imag.zero_()
            y = torch.fft.irfft(stack, n=nb, norm="forward")
            scale = torch.tensor([_noise_scales(p, k, nh) for p in pats], device="cuda",
                                 dtype=torch.float64)[which]
            ps = torch.nn.functional.pad(torch.cumsum(torch.cat([y, y], 1), 1), (1, 0))
            total_sum = ps[:, nb]
            best = torch.full((t.numel(),), -math.inf, dtype=torch.float64, device="cuda")
            for i, wd in enumerate(_widths(nb, k)):
                mx = (ps[:, wd:wd + nb] - ps[:, :nb]).amax(1)
                best = torch.maximum(best, (mx - wd / nb * total_sum) * scale[:, i])
            r = k * (r_lo + t.double() * lodr)
            ok = best > THRESHOLD
            if k > 1:
                ok &= r < N / 2.0
            at = torch.nonzero(ok).flatten()
            for tt, rr, mm in zip(t[at].tolist(), r[at].tolist(), best[at].tolist()):
                found.append((tt // BLOCKSIZE, slot, tt, rr, mm, H))
    found.sort(key=lambda c: c[:3])
    return _collapse([c[3:] for c in found], T)


def _collapse(cands, T):
    """Candidates (r, metric, nharm) with runs and harmonics removed."""
    cands = sorted(cands, key=lambda c: c[0])
    kept, last = [], None
    for c in cands:
        if last is not None and c[0] - last <= 1.0:
            if c[1] > kept[-1][1]:
                kept[-1] = c
        else:
            kept.append(c)
        last = c[0]
    out = []
    m = np.arange(1, 17)
    for c in sorted(kept, key=lambda c: -c[1]):
        if out:
            r = np.array([o[0] for o in out])
            lo, hi = np.minimum(r, c[0])[:, None], np.maximum(r, c[0])[:, None]
            n = np.rint(m * hi / lo)
            if ((n >= 1) & (n <= 16) & (np.abs(m * hi - n * lo) <= m)).any():
                continue
        out.append(c)
    out.sort(key=lambda c: c[0])
    r = np.array([c[0] for c in out], dtype=np.float64)
    return _columns({"freq": r / T, "metric": np.array([c[1] for c in out], dtype=np.float64),
                     "r": r, "nharm": np.array([c[2] for c in out], dtype=np.int32)})


def _exact_spectrum(x, startwidth=6, endwidth=100, endfreq=6.0):
    """rfft and running block-median normalisation in FP64 (the inverse
    square root is the one the normalisation is defined with: an estimate
    from the level's bits and one Newton step)."""
    N = x.numel()
    S = torch.fft.rfft(x.double())[:N // 2]
    n2, T = N // 2, N * DT
    starts, lens, pos = [1], [startwidth], 1 + startwidth
    width = int(startwidth * math.log(pos))
    while pos < n2:
        n = min(width, n2 - pos)
        starts.append(pos)
        lens.append(n)
        pos += n
        width = int(startwidth * math.log(pos)) if np.float32(pos) / np.float32(T) < endfreq \
            else endwidth
    power = (S.real ** 2 + S.imag ** 2).cpu().numpy()
    level = np.array([np.partition(power[a:a + n], (n - 1) // 2)[(n - 1) // 2]
                      for a, n in zip(starts, lens)]) / math.log(2.0)
    mid = np.array([a + n // 2 for a, n in zip(starts, lens)])
    span = 0.5 * (np.array(lens[:-1]) + np.array(lens[1:]))
    slope = np.diff(level) / span
    slope = np.append(slope, slope[-1] if slope.size else 1.0)
    k = np.arange(1, n2)
    seg = np.searchsorted(mid, k, side="right") - 1
    at = np.maximum(seg, 0)
    lv = np.where(seg < 0, level[0], level[at] + slope[at] * (k - mid[at]))
    bits = lv.astype(np.float32).view(np.int32)
    y = (np.int32(0x5f3759df) - (bits >> 1)).view(np.float32).astype(np.float64)
    norm = y * (1.5 - 0.5 * lv * y * y)
    S[1:] *= torch.from_numpy(norm).cuda()
    S[0] = 1.0
    return torch.view_as_real(S).reshape(-1)


def _tables_np(case):
    """Channel delays, subband offsets and blocks per read of the DM grid."""
    nchan, nsub, ndm = case["nchan"], case["nsub"], case["ndm"]
    chanwid, lofreq = BW / nchan, _lofreq(nchan)
    cps = nchan // nsub
    dms = case["dmstep"] * np.arange(ndm)
    avg = dms.sum() / ndm
    fch = lofreq + chanwid * np.arange(nchan)
    fsub = lofreq + chanwid * cps - chanwid + chanwid * cps * np.arange(nsub)
    near = lambda v: np.floor(v + 0.5).astype(np.int64)     # noqa: E731
    chan = near((avg / (0.000241 * fch * fch) - np.repeat(avg / (0.000241 * fsub * fsub), cps)) / DT)
    sub = dms[:, None] / (0.000241 * fsub * fsub)
    offs = near((sub - sub[:, -1:]) / DT)
    sweep = dms[-1] / 0.000241 * (lofreq ** -2 - fch[-1] ** -2)
    return chan, offs, int(sweep / DT) // SPECTRA_PER_SUBINT + 1


def _exact_dedisp(case, raw):
    chan, offs, _ = _tables_np(case)
    nout, nsub = _out_length(case), case["nsub"]
    cps = case["nchan"] // nsub
    n = nout + int(offs.max())
    X = raw.flip(1)
    S = torch.zeros((nsub, n), dtype=torch.float64, device="cuda")
    for c in range(case["nchan"]):
        S[c // cps] += X[chan[c]:chan[c] + n, c]
    out = torch.zeros((case["ndm"], nout), dtype=torch.float64, device="cuda")
    for d in range(case["ndm"]):
        for s in range(nsub):
            out[d] += S[s, offs[d, s]:offs[d, s] + nout]
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind in ("search", "file"):
        return _exact_search(_spectrum(case["N"], seed), case["N"], case["nharms"], case["hidr"])
    if kind == "spectrum":
        return _exact_spectrum(_series(case["N"], seed).float())
    if kind == "dedisp" and not case["clipped"]:
        return _exact_dedisp(case, _filterbank(case, seed))
    # the clipped runs' levels and flags follow from float running statistics
    # that have no 64-bit counterpart
    return None
