/*
 * The FP64 search (--precision f64, the reference's CS_PREC_F64): the same
 * trials, chunks and records as the FP32 kernels, with the profile stage in
 * double precision as the reference computes it (src/cuda.cu:579-584, 621,
 * 726, 1004-1014 on its GPU; src/search.c:288-292, 333-400, 641-656 and
 * src/boxcar.c:203-252, 715-731 on its CPU):
 *
 *   1. interpolation in FP32, bit-identical to the FP32 kernels, the
 *      amplitude then widened to double (src/interp.c:555-573: "the products
 *      are formed in f32 and widened per element");
 *   2. the unnormalised c2r of each profile-producing slot (the base profile
 *      and every decimation that does not fold) in FP64.  The reference runs
 *      FFTW / cuFFT Z2D; here it is a dense half-spectrum DFT: for bin
 *      n = 0..Hk the cosine part C_n = sum_h Re X_h c_hn and the sine part
 *      S_n = sum_h Im X_h s_hn, so x[n] = C_n - S_n and x[2Hk-n] = C_n + S_n
 *      (cs_tables_dft_f64).  Each thread accumulates 4 trials x 2 bins of
 *      both parts with DFMA from shared memory;
 *   3. the k-fold averages (fold_row_f64: left-to-right sum, times 1/k), the
 *      cyclic prefix sums and the exact boxcar scan (profile_boxcar_f64) in
 *      double with the reference's expression order, one warp per slot and
 *      one lane per trial; the scan is the exact one the reference's f64 gate
 *      falls back to for every trial that can reach the threshold;
 *   4. threshold in double and warp-ballot compaction into CsRec64 records.
 *
 * Work unit: 32 trials (a quarter of a 128-trial tile).  One CTA of 256
 * threads per SM, persistent over the sub-tiles.
 *
 * Shared memory: the DFT tables (cos then sin, nh x ucols doubles each), the
 * profile rows (32 x prs doubles, prs odd so lanes on consecutive trials hit
 * different banks) and the prefix-sum arrays of every slot (pos-major, 32
 * trials a row).  The FP32 amplitudes of step 1 live in the prefix-sum
 * region, which is free until step 3.
 */
#pragma once

namespace f64k {

constexpr int TT = 32;              /* trials per sub-tile */
constexpr int NT = 256;             /* threads per CTA */

struct Extra {
    const double *bcs;              /* cos table [nh][ucols], then sin table */
    int nunit, ucols;
    int unit0[CS_MAX_SLOT];         /* first DFT unit of a profile slot, or -1 */
    int prs;                        /* profile row stride (doubles, odd) */
    int ps_off[CS_MAX_SLOT];        /* prefix-sum array of each slot (doubles) */
    int ps_total;                   /* doubles in all prefix-sum arrays */
    const double *scales;           /* per chunk CS_F64_SCALES */
    /* search_f64_wide, 16 taps: weights by (harmonic, tap quad, phase), so that
     * lanes on consecutive phases read consecutive 16-byte words */
    const float4 *wt;
    int wt_off[CS_MAX_NH];
    CsRec64 *recs;
};

/* Shared-memory bytes of the kernel for a table layout. */
static __host__ __device__ inline int smem_bytes(int nh, int ucols, int prs, int ps_total)
{
    return 2 * nh * ucols * 8 + TT * prs * 8 + ps_total * 8;
}

/* x[j] of a slot's profile for one trial: its own DFT columns, or the k-fold
 * average of the base profile (src/search.c:333-365: a = s[j], a += s[j +
 * q*nk] for q = 1..k-1, times 1/k). */
static __device__ __forceinline__ double slot_value(const double *row, const CsSlot &sl,
                                                    double invk, int j)
{
    if (!sl.fold) return row[sl.col0 + j];
    double a = row[j];
    for (int q = 1; q < sl.k; q++) a = __dadd_rn(a, row[j + q * sl.nk]);
    return __dmul_rn(a, invk);
}

template <int MT>
__global__ void __launch_bounds__(NT, 1)
search_f64(const SearchArgs args, const Extra ex)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CsHarm harm_s[CS_MAX_NH];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nh = args.nh, ucols = ex.ucols, prs = ex.prs;
    const int m = MT ? MT : args.m;
    double *bc = reinterpret_cast<double *>(smem);
    double *bs = bc + (size_t)nh * ucols;
    double *pr = bs + (size_t)nh * ucols;
    double *ps = pr + (size_t)TT * prs;
    float *xr = reinterpret_cast<float *>(ps);       /* [nh][TT], then xi */
    float *xi = xr + (size_t)nh * TT;

    for (int h = tid; h < nh; h += NT) harm_s[h] = args.harm[h];
    for (int i = tid; i < 2 * nh * ucols; i += NT) bc[i] = ex.bcs[i];
    __syncthreads();

    const int nsub = args.ntiles * (CS_TILE_M / TT);
    for (int item = blockIdx.x; item < nsub; item += gridDim.x) {
        const int tile = item / (CS_TILE_M / TT), sub = item % (CS_TILE_M / TT);
        const int ci = args.tiles[3 * tile + 0];
        const int j0 = args.tiles[3 * tile + 1] + sub * TT;
        const int cnt = args.tiles[3 * tile + 2] - sub * TT;
        if (cnt <= 0) continue;                     /* uniform over the CTA */
        const CsChunk &ch = args.chunks[ci];

        /* ---- 1. FP32 interpolation: lane = trial, warp = harmonic phase ---- */
        {
            const int r = lane;
            const bool valid = r < cnt;
            const long long t = ch.i0 + j0 + r;
            const long long tp = t * (long long)args.pnum;
            const long long Q = tp / args.q;
            const uint32_t R = (uint32_t)(tp - Q * args.q);
            for (int h = warp + 1; h <= nh; h += NT / 32) {
                float2 x = make_float2(0.0f, 0.0f);
                if (valid && ((ch.filled >> (h - 1)) & 1ULL))
                    x = interp_amp<MT>(args, harm_s[h - 1], h, m, Q, R);
                xr[(h - 1) * TT + r] = x.x;
                xi[(h - 1) * TT + r] = x.y;
            }
        }
        __syncthreads();

        /* ---- 2. FP64 half-spectrum DFT: 4 trials x 2 units per item ---- */
        for (int w = tid; w < (TT / 4) * (ucols / 2); w += NT) {
            const int tg = w & (TT / 4 - 1), ug = w / (TT / 4);
            double c[4][2], s[4][2];
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) c[i][j] = s[i][j] = 0.0;
            const float4 *xr4 = reinterpret_cast<const float4 *>(xr) + tg;
            const float4 *xi4 = reinterpret_cast<const float4 *>(xi) + tg;
            const double2 *bc2 = reinterpret_cast<const double2 *>(bc) + ug;
            const double2 *bs2 = reinterpret_cast<const double2 *>(bs) + ug;
            for (int h = 0; h < nh; h++) {
                const float4 a = xr4[h * (TT / 4)], b = xi4[h * (TT / 4)];
                const double2 cw = bc2[h * (ucols / 2)], sw = bs2[h * (ucols / 2)];
                const double ar[4] = {a.x, a.y, a.z, a.w}, ai[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    c[i][0] = __fma_rn(ar[i], cw.x, c[i][0]);
                    c[i][1] = __fma_rn(ar[i], cw.y, c[i][1]);
                    s[i][0] = __fma_rn(ai[i], sw.x, s[i][0]);
                    s[i][1] = __fma_rn(ai[i], sw.y, s[i][1]);
                }
            }
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int u = 2 * ug + j;
                if (u >= ex.nunit) continue;
                int sl = 0;
                for (int q = 0; q < args.nslot; q++)
                    if (ex.unit0[q] >= 0 && u >= ex.unit0[q]) sl = q;
                const int n = u - ex.unit0[sl], Hk = args.slot[sl].Hk;
                const int col0 = args.slot[sl].col0;
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    double *row = pr + (size_t)(4 * tg + i) * prs + col0;
                    row[n] = __dsub_rn(c[i][j], s[i][j]);
                    if (n > 0 && n < Hk) row[2 * Hk - n] = __dadd_rn(c[i][j], s[i][j]);
                }
            }
        }
        __syncthreads();

        /* ---- 3. folds, prefix sums, boxcar scan: warp = slot, lane = trial ---- */
        if (warp < args.nslot) {
            const CsSlot &sl = args.slot[warp];
            const int r = lane, nk = sl.nk;
            const double *row = pr + (size_t)r * prs;
            double *P = ps + ex.ps_off[warp];
            const double invk = 1.0 / (double)sl.k;
            /* psum[i] = psum[i-1] + x[(i-1) mod nk], i = 1..nk+wmax
             * (src/boxcar.c:203-211 with b = 0) */
            double acc = 0.0;
            P[r] = 0.0;
            for (int i = 1; i <= nk + sl.wmax; i++) {
                const int idx = i > nk ? i - nk : i;
                acc = __dadd_rn(acc, slot_value(row, sl, invk, idx - 1));
                P[i * TT + r] = acc;
            }
            const double *sc = ex.scales + (size_t)ci * CS_F64_SCALES + warp * (CS_NWMAX + 1);
            double best = -INFINITY;
            if (!(sc[0] > 0.0)) {
                best = 0.0;                     /* profile_boxcar_f64: no noise scale */
            } else {
                const double stot = __dsub_rn(P[nk * TT + r], P[r]);
                for (int a = 0; a < sl.nw; a++) {
                    const int w = sl.widths[a];
                    const double duty = __ddiv_rn((double)w, (double)nk);
                    double mx = __dsub_rn(P[w * TT + r], P[r]);
                    for (int p = 2; p <= nk; p++) {
                        const double d = __dsub_rn(P[(p + w - 1) * TT + r], P[(p - 1) * TT + r]);
                        if (d > mx) mx = d;
                    }
                    const double cand = __dmul_rn(__dsub_rn(mx, __dmul_rn(duty, stot)), sc[1 + a]);
                    if (cand > best) best = cand;
                }
            }
            /* ---- 4. threshold + warp-aggregated compaction ---- */
            const int j = j0 + r;
            const bool hit = r < cnt && j < ch.nvalid[warp] && best > args.thresh;
            const unsigned mask = __ballot_sync(0xffffffffu, hit);
            if (mask) {
                unsigned basei = 0;
                if (lane == 0) basei = atomicAdd(args.count, (unsigned)__popc(mask));
                basei = __shfl_sync(0xffffffffu, basei, 0);
                if (hit) {
                    const unsigned pos = basei + (unsigned)__popc(mask & ((1u << lane) - 1u));
                    if (pos < args.cap) {
                        CsRec64 rec;
                        rec.chunk = ci;
                        rec.slot = warp;
                        rec.j = j;
                        rec.pad = 0;
                        rec.metric = best;
                        ex.recs[pos] = rec;
                    }
                }
            }
        }
        __syncthreads();
    }
}

/* ---------------------------------------------------------------------------
 * The same search with its stages overlapped and spread over the warps.
 *
 * search_f64 above keeps one warp a slot busy with the prefix sums and the scan
 * while the others wait: 59 k cycles a sub-tile, of which the DFT is 8 k (its
 * operands' shared-memory reads).  Here, with 16 warps:
 *   DFT      on the FP64 matrix instruction (mma.sync m8n8k4): a warp owns 16
 *            trials x 8 columns of both parts, and each operand read serves 8
 *            products of a row or column instead of 2 or 4;
 *   bound    warps 0 .. nslot - 1, a slot each: whether any of the 32 trials can
 *            reach the threshold (slot_bound); almost none can, and then the
 *            rest is not needed.  The other warps interpolate the next
 *            sub-tile's harmonics meanwhile (its operand, X, is not read again);
 *   prefix   the same warps, 8 bins read ahead of the chain of additions;
 *   scan     split over all warps by bins (Task): partial maxima in shared
 *            memory, where the profile rows were; a warp a slot takes their
 *            maximum, which does not depend on the split.
 * The additions of a chain, the differences and the final expression are
 * search_f64's; only the DFT's summation is grouped by the matrix instruction
 * (1e-16 of a profile bin).  Bound by the latency of the serial stages and the
 * barriers between them: some 16 k cycles a sub-tile, 3.7 k of them the DFT's
 * arithmetic.  N = 2^19, nharms 60: 0.86 ms against 3.30.  It needs room for X beside the
 * prefix sums; geometries that only fit without it take search_f64, as do few
 * harmonics at low thresholds. */
constexpr int WNT = 512, NW = WNT / 32;
constexpr int XS = TT + 4;          /* X row stride (doubles): fragment rows hit all banks */

struct Task {
    int slot, p0, p1;               /* bins p0 + 1 .. p1 of a slot's profile */
};

struct Wide {
    int bstr;                       /* DFT table row stride (doubles) */
    int kp;                         /* harmonics rounded up to 4 */
    int nwmax;                      /* most widths of a slot */
    int ntask;
    Task task[NW];
    int reg_pr;                     /* doubles of the profile rows / partial maxima */
};

static __host__ inline int table_stride(int ucols)
{
    int b = (ucols + 7) / 8 * 8;
    while (b % 16 != 4 && b % 16 != 12) b++;
    return b;
}

static __host__ inline int wide_smem(const Wide &w, int ps_total)
{
    return 8 * (2 * w.kp * w.bstr + 2 * w.kp * XS + w.reg_pr + ps_total);
}

/* Deal the scan out: every slot with bins a task, then the next one to the slot
 * with most bins a task. */
static __host__ inline void deal(Wide &w, int nslot, const CsSlot *slot)
{
    int parts[CS_MAX_SLOT], n = nslot;
    for (int s = 0; s < nslot; s++) parts[s] = 1;
    for (; n < NW; n++) {
        int best = 0;
        for (int s = 1; s < nslot; s++)
            if (slot[s].nk * parts[best] > slot[best].nk * parts[s]) best = s;
        if (parts[best] >= slot[best].nk) break;
        parts[best]++;
    }
    w.ntask = 0;
    for (int s = 0; s < nslot; s++)
        for (int i = 0; i < parts[s]; i++) {
            Task &t = w.task[w.ntask++];
            t.slot = s;
            t.p0 = slot[s].nk * i / parts[s];
            t.p1 = slot[s].nk * (i + 1) / parts[s];
        }
}

static __device__ __forceinline__ void dmma(double (&c)[2], double a, double b)
{
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

/* Largest window difference of N widths over bins p0 + 1 .. p1. */
template <int N>
static __device__ __forceinline__ void scan_bins(const double *P, const CsSlot &sl, int p0, int p1,
                                                 double *part)
{
    double mx[N];
    int w[N];
#pragma unroll
    for (int a = 0; a < N; a++) {
        mx[a] = -INFINITY;
        w[a] = (sl.widths[a] - 1) * TT;
    }
#pragma unroll 2
    for (int p = p0 + 1; p <= p1; p++) {
        const double base = P[(p - 1) * TT];
#pragma unroll
        for (int a = 0; a < N; a++) {
            const double d = __dsub_rn(P[p * TT + w[a]], base);
            if (d > mx[a]) mx[a] = d;
        }
    }
#pragma unroll
    for (int a = 0; a < N; a++) part[a * TT] = mx[a];
}

/* Largest bin, largest pair of neighbours (cyclic) and total of the KC-fold
 * sums (KC 0: k-fold) of an FP32 row, and the largest size of its own bins. */
template <int KC>
static __device__ __forceinline__ void row_sums(const float *row, int nk, int k, float &m1,
                                                float &m2, float &tot, float &size)
{
    const int K = KC ? KC : k;
    float last = -INFINITY, first = 0.0f;
    m1 = m2 = -INFINITY;
    tot = size = 0.0f;
#pragma unroll 4
    for (int j = 0; j < nk; j += 2) {           /* nk = 2 Hk is even */
        float a = row[j], b = row[j + 1];
        size = wsk::fmax3(size, fabsf(a), fabsf(b));
#pragma unroll
        for (int q = 1; q < K; q++) {
            const float x = row[j + q * nk], y = row[j + 1 + q * nk];
            size = wsk::fmax3(size, fabsf(x), fabsf(y));
            a += x;
            b += y;
        }
        if (j == 0) first = a;
        tot += a + b;
        m1 = wsk::fmax3(m1, a, b);
        m2 = wsk::fmax3(m2, a + last, b + a);
        last = b;
    }
    m2 = fmaxf(m2, first + last);
}

/* A bound of the FP64 metric of one profile, from its bins in FP32 (row: this
 * trial's).  As in the FP32 kernels, the largest bin and the largest pair of
 * neighbours bound every wider window.  The margin has two parts, u = 2^-24:
 *   - a sum over the profile is at most |tot| + nk * m1 in size, and wrong by nk * u
 *     of that;
 *   - a folded bin is wrong by u of the K bins it was made of, each up to `size`
 *     and rounded to FP32 before they cancel: K + K (K - 1) of u * size, or K^2.
 *     The pairs' additions add 2 K, a window of w bins and its share of the total
 *     have w of both: w * 2 K (K + 1) * u * size.  A tone at a harmonic that is no
 *     multiple of K leaves a fold that small beside its bins.
 * Where FP32 does not hold the bins (or one is no number) the answer is infinity,
 * and what lies below its range is covered by an absolute 1e-30. */
static __device__ __forceinline__ float slot_bound(const float *row, const CsSlot &sl,
                                                   const double *sc)
{
    const double s0 = sc[0];
    float scale[CS_NWMAX];                      /* ahead of the sums */
#pragma unroll
    for (int a = 0; a < CS_NWMAX; a++) scale[a] = a < sl.nw ? (float)sc[1 + a] : 0.0f;
    const int nk = sl.nk, K = sl.fold ? sl.k : 1;
    row += sl.fold ? 0 : sl.col0;
    float m1, m2, tot, size;
    switch (K) {
    case 1: row_sums<1>(row, nk, 1, m1, m2, tot, size); break;
    case 2: row_sums<2>(row, nk, 2, m1, m2, tot, size); break;
    case 3: row_sums<3>(row, nk, 3, m1, m2, tot, size); break;
    case 4: row_sums<4>(row, nk, 4, m1, m2, tot, size); break;
    case 5: row_sums<5>(row, nk, 5, m1, m2, tot, size); break;
    case 6: row_sums<6>(row, nk, 6, m1, m2, tot, size); break;
    default: row_sums<0>(row, nk, K, m1, m2, tot, size);
    }
    if (!(size < 1e30f) || tot != tot) return INFINITY;
    const float margin = (fabsf(tot) + nk * fabsf(m1)) * (nk + 16) * 2.4e-7f +
                         (float)(2 * K * (K + 1) * sl.wmax) * 6.0e-8f * size + 1e-30f;
    float bound = -INFINITY;
#pragma unroll
    for (int a = 0; a < CS_NWMAX; a++) {
        if (a >= sl.nw) break;
        const int w = sl.widths[a];
        const float m = w == 1 ? m1 : (w & 1) ? (w >> 1) * m2 + m1 : (w >> 1) * m2;
        bound = fmaxf(bound, (m - (float)w / (float)nk * tot + margin) * scale[a]);
    }
    if (!(s0 > 0.0)) return 0.0f;               /* profile_boxcar_f64: no noise scale */
    return K > 1 ? bound / (float)K : bound;
}

template <int MT>
__global__ void __launch_bounds__(WNT, 1)
search_f64_wide(const __grid_constant__ SearchArgs args, const __grid_constant__ Extra ex,
                const __grid_constant__ Wide wd)
{
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ CsHarm harm_s[CS_MAX_NH];
    __shared__ int want[CS_MAX_SLOT];                /* slots that need the exact scan */
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int nh = args.nh, kp = wd.kp, bstr = wd.bstr, prs = ex.prs;
    const int m = MT ? MT : args.m;
    double *bc = reinterpret_cast<double *>(smem);
    double *bs = bc + kp * bstr;
    double *xr = bs + kp * bstr;                     /* [kp][XS], then xi */
    double *xi = xr + kp * XS;
    double *pr = xi + kp * XS;                       /* profile rows, then partial maxima */
    double *ps = pr + wd.reg_pr;

    float *pf = reinterpret_cast<float *>(ps);       /* the rows in FP32, until the prefix sums */

    for (int h = tid; h < nh; h += WNT) harm_s[h] = args.harm[h];
    for (int i = tid; i < kp * bstr; i += WNT) {
        const int h = i / bstr, u = i - h * bstr;
        const bool in = h < nh && u < ex.ucols;
        bc[i] = in ? ex.bcs[h * ex.ucols + u] : 0.0;
        bs[i] = in ? ex.bcs[(nh + h) * ex.ucols + u] : 0.0;
    }
    for (int i = tid; i < 2 * kp * XS; i += WNT) xr[i] = 0.0;
    __syncthreads();

    /* a little below the threshold: FP32 scales and sums */
    const float need = __double2float_rd(args.thresh) * (args.thresh > 0.0 ? 0.9999f : 1.0001f);
    const int nsub = args.ntiles * (CS_TILE_M / TT);
    /* A sub-tile with trials, from number `item` on: where it is, found by one
     * thread an item ahead (dependent reads of global memory). */
    struct Item {
        unsigned long long filled;
        long long t0;                           /* first trial */
        int item, ci, j0, cnt;
    };
    __shared__ Item ahead;
    auto find = [&](int item) {
        Item r;
        r.filled = 0;
        r.t0 = 0;
        r.ci = r.j0 = r.cnt = 0;
        for (; item < nsub; item += gridDim.x) {
            const int tile = item / (CS_TILE_M / TT), sub = item % (CS_TILE_M / TT);
            r.cnt = args.tiles[3 * tile + 2] - sub * TT;
            if (r.cnt <= 0) continue;
            r.ci = args.tiles[3 * tile + 0];
            r.j0 = args.tiles[3 * tile + 1] + sub * TT;
            r.t0 = args.chunks[r.ci].i0 + r.j0;
            r.filled = args.chunks[r.ci].filled;
            break;
        }
        r.item = item;
        return r;
    };
    /* FP32 amplitudes of an item, widened: lane = trial, harmonics first, first +
     * step, ... */
    auto interpolate = [&](const Item &it, int first, int step) {
        const bool valid = lane < it.cnt;
        const long long tp = (it.t0 + lane) * (long long)args.pnum;
        const long long Q = tp / args.q;
        const uint32_t R = (uint32_t)(tp - Q * args.q);
        const unsigned long long filled = it.filled;
        int h = first + 1;
        if (MT == 16) {
            /* U harmonics together: their table rows, then their windows, are in
             * flight at once.  An active harmonic's window is inside the spectrum
             * by construction; clamped for safety. */
            constexpr int U = 3;
            for (; h + (U - 1) * step <= nh; h += U * step) {
                int row[U], ph[U];
                long long b0[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const int hu = h + u * step;
                    uint32_t qd, res;
                    divmod_q((uint32_t)hu * R, (uint32_t)args.q, args.qmagic, qd, res);
                    ph[u] = args.rowtab[(size_t)(hu - 1) * args.q + res];
                    row[u] = harm_s[hu - 1].woff + ph[u];
                    b0[u] = harm_s[hu - 1].rfloor0 + (long long)hu * Q + qd + 1 - 8;
                }
                float2 g[U], acc[U];
                const float4 *wr[U];
                const float2 *ap[U];
                bool on[U];
#pragma unroll
                for (int u = 0; u < U; u++) {
                    on[u] = valid && ((filled >> (h + u * step - 1)) & 1ULL);
                    if (!on[u]) row[u] = harm_s[h + u * step - 1].woff + (ph[u] = 0);
                    const long long b = b0[u] + args.carry[row[u]];
                    const long long c = min(max(b, 0ll), args.namps - 16);
                    on[u] = on[u] && b == c;
                    ap[u] = args.amps + max(c, 0ll);
                    wr[u] = ex.wt + ex.wt_off[h + u * step - 1] + ph[u];
                    g[u] = __ldg(args.A + row[u]);
                    acc[u] = make_float2(0.0f, 0.0f);
                }
                if (args.namps >= 16) {
#pragma unroll
                    for (int i = 0; i < 4; i++)
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const float4 w = __ldg(wr[u] + i * harm_s[h + u * step - 1].P);
                            const float2 a0 = __ldg(ap[u] + 4 * i), a1 = __ldg(ap[u] + 4 * i + 1);
                            const float2 a2 = __ldg(ap[u] + 4 * i + 2), a3 = __ldg(ap[u] + 4 * i + 3);
                            acc[u].x = __fmaf_rn(w.x, a0.x, acc[u].x);
                            acc[u].y = __fmaf_rn(w.x, a0.y, acc[u].y);
                            acc[u].x = __fmaf_rn(w.y, a1.x, acc[u].x);
                            acc[u].y = __fmaf_rn(w.y, a1.y, acc[u].y);
                            acc[u].x = __fmaf_rn(w.z, a2.x, acc[u].x);
                            acc[u].y = __fmaf_rn(w.z, a2.y, acc[u].y);
                            acc[u].x = __fmaf_rn(w.w, a3.x, acc[u].x);
                            acc[u].y = __fmaf_rn(w.w, a3.y, acc[u].y);
                        }
                }
#pragma unroll
                for (int u = 0; u < U; u++) {
                    const float re = __fsub_rn(__fmul_rn(g[u].x, acc[u].x), __fmul_rn(g[u].y, acc[u].y));
                    const float im = __fadd_rn(__fmul_rn(g[u].x, acc[u].y), __fmul_rn(g[u].y, acc[u].x));
                    const int at = (h + u * step - 1) * XS + lane;
                    xr[at] = on[u] ? (double)re : 0.0;
                    xi[at] = on[u] ? (double)im : 0.0;
                }
            }
        }
        for (; h <= nh; h += step) {
            float2 x = make_float2(0.0f, 0.0f);
            if (valid && ((filled >> (h - 1)) & 1ULL))
                x = interp_amp<MT>(args, harm_s[h - 1], h, m, Q, R);
            xr[(h - 1) * XS + lane] = (double)x.x;
            xi[(h - 1) * XS + lane] = (double)x.y;
        }
    };

    Item cur = find(blockIdx.x);
    if (cur.item < nsub) interpolate(cur, warp, NW);
    if (tid == WNT - 1) ahead = find(cur.item + gridDim.x);
    __syncthreads();
    while (cur.item < nsub) {
        const int ci = cur.ci, j0 = cur.j0, cnt = cur.cnt;
        const CsChunk &ch = args.chunks[ci];
        const Item nxt = ahead;

        /* ---- DFT: warp = 16 trials x every (NW / 2)-th 8 columns ---- */
        {
            const int t0 = (warp & 1) * 16, fr = lane >> 2, fc = lane & 3;
            for (int u0 = (warp >> 1) * 8; u0 < ex.nunit; u0 += NW / 2 * 8) {
                double c[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, s[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
                const double *ar = xr + fc * XS + t0 + fr, *ai = xi + fc * XS + t0 + fr;
                const double *cb = bc + fc * bstr + u0 + fr, *sb = bs + fc * bstr + u0 + fr;
#pragma unroll 3
                for (int k = 0; k < kp; k += 4) {
                    const double b0 = cb[k * bstr], b1 = sb[k * bstr];
                    dmma(c[0], ar[k * XS], b0);
                    dmma(c[1], ar[k * XS + 8], b0);
                    dmma(s[0], ai[k * XS], b1);
                    dmma(s[1], ai[k * XS + 8], b1);
                }
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    const int u = u0 + 2 * fc + j;
                    if (u >= ex.nunit) continue;
                    int sl = 0;
                    for (int q = 0; q < args.nslot; q++)
                        if (ex.unit0[q] >= 0 && u >= ex.unit0[q]) sl = q;
                    const int n = u - ex.unit0[sl], Hk = args.slot[sl].Hk;
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const int at = (t0 + 8 * i + fr) * prs + args.slot[sl].col0;
                        const double x0 = __dsub_rn(c[i][j], s[i][j]);
                        pr[at + n] = x0;
                        pf[at + n] = (float)x0;
                        if (n > 0 && n < Hk) {
                            const double x1 = __dadd_rn(c[i][j], s[i][j]);
                            pr[at + 2 * Hk - n] = x1;
                            pf[at + 2 * Hk - n] = (float)x1;
                        }
                    }
                }
            }
        }
        __syncthreads();

        /* ---- can any trial reach the threshold? (the other warps interpolate
         * the next item's harmonics meanwhile) ---- */
        if (warp < args.nslot) {
            const float bound = slot_bound(pf + lane * prs, args.slot[warp],
                                           ex.scales + (size_t)ci * CS_F64_SCALES + warp * (CS_NWMAX + 1));
            const bool w = lane < cnt && !(bound <= need);
            const unsigned any = __ballot_sync(0xffffffffu, w);
            if (lane == 0) want[warp] = any != 0;
        } else if (nxt.item < nsub) {
            if (tid == WNT - 1) ahead = find(nxt.item + gridDim.x);
            interpolate(nxt, warp - args.nslot, NW - args.nslot);
        }
        __syncthreads();
        int exact = 0;
        for (int q = 0; q < args.nslot; q++) exact |= want[q];
        if (!exact) {                           /* the same in every thread */
            cur = nxt;
            continue;
        }

        /* ---- prefix sums ---- */
        if (warp < args.nslot && want[warp]) {
            const CsSlot &sl = args.slot[warp];
            const int nk = sl.nk, n = nk + sl.wmax, K = sl.fold ? sl.k : 1;
            const double *row = pr + (size_t)lane * prs + (sl.fold ? 0 : sl.col0);
            double *P = ps + ex.ps_off[warp] + lane;
            const double invk = sl.fold ? 1.0 / (double)sl.k : 1.0;
            double acc = 0.0;
            P[0] = 0.0;
            for (int i0 = 0; i0 < n; i0 += 8) {
                double v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const int i = min(i0 + u, n - 1);
                    v[u] = row[i >= nk ? i - nk : i];
                }
                for (int q = 1; q < K; q++)
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        const int i = min(i0 + u, n - 1);
                        v[u] = __dadd_rn(v[u], row[(i >= nk ? i - nk : i) + q * nk]);
                    }
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    acc = __dadd_rn(acc, K > 1 ? __dmul_rn(v[u], invk) : v[u]);
                    if (i0 + u < n) P[(i0 + u + 1) * TT] = acc;
                }
            }
        }
        __syncthreads();

        /* ---- scan: a run of bins a warp; the profile rows are read, their room
         * takes the partial maxima ---- */
        if (warp < wd.ntask && want[wd.task[warp].slot]) {
            const Task &t = wd.task[warp];
            const CsSlot &sl = args.slot[t.slot];
            const double *P = ps + ex.ps_off[t.slot] + lane;
            double *part = pr + warp * wd.nwmax * TT + lane;
            switch (sl.nw) {
            case 1: scan_bins<1>(P, sl, t.p0, t.p1, part); break;
            case 2: scan_bins<2>(P, sl, t.p0, t.p1, part); break;
            case 3: scan_bins<3>(P, sl, t.p0, t.p1, part); break;
            case 4: scan_bins<4>(P, sl, t.p0, t.p1, part); break;
            case 5: scan_bins<5>(P, sl, t.p0, t.p1, part); break;
            default:
                for (int a = 0; a < sl.nw; a++) {
                    const int w = sl.widths[a];
                    double mx = -INFINITY;
                    for (int p = t.p0 + 1; p <= t.p1; p++) {
                        const double d = __dsub_rn(P[(p + w - 1) * TT], P[(p - 1) * TT]);
                        if (d > mx) mx = d;
                    }
                    part[a * TT] = mx;
                }
            }
        }
        __syncthreads();

        /* ---- the best width, threshold, compaction: warp = slot ---- */
        if (warp < args.nslot && want[warp]) {
            const CsSlot &sl = args.slot[warp];
            const int nk = sl.nk;
            const double *P = ps + ex.ps_off[warp] + lane;
            const double *sc = ex.scales + (size_t)ci * CS_F64_SCALES + warp * (CS_NWMAX + 1);
            double best = -INFINITY;
            if (!(sc[0] > 0.0)) {
                best = 0.0;                     /* profile_boxcar_f64: no noise scale */
            } else {
                const double stot = __dsub_rn(P[nk * TT], P[0]);
                for (int a = 0; a < sl.nw; a++) {
                    double mx = -INFINITY;
                    for (int k = 0; k < wd.ntask; k++)
                        if (wd.task[k].slot == warp) {
                            const double d = pr[(k * wd.nwmax + a) * TT + lane];
                            if (d > mx) mx = d;
                        }
                    const double duty = __ddiv_rn((double)sl.widths[a], (double)nk);
                    const double cand = __dmul_rn(__dsub_rn(mx, __dmul_rn(duty, stot)), sc[1 + a]);
                    if (cand > best) best = cand;
                }
            }
            const int j = j0 + lane;
            const bool hit = lane < cnt && j < ch.nvalid[warp] && best > args.thresh;
            const unsigned mask = __ballot_sync(0xffffffffu, hit);
            if (mask) {
                unsigned basei = 0;
                if (lane == 0) basei = atomicAdd(args.count, (unsigned)__popc(mask));
                basei = __shfl_sync(0xffffffffu, basei, 0);
                if (hit) {
                    const unsigned pos = basei + (unsigned)__popc(mask & ((1u << lane) - 1u));
                    if (pos < args.cap) {
                        CsRec64 rec;
                        rec.chunk = ci;
                        rec.slot = warp;
                        rec.j = j;
                        rec.pad = 0;
                        rec.metric = best;
                        ex.recs[pos] = rec;
                    }
                }
            }
        }
        __syncthreads();                        /* the partial maxima are read */
        cur = nxt;
    }
}

}  // namespace f64k
