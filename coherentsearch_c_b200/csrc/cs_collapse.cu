/*
 * Candidate harvest and collapse on the GPU: the post-processing of the
 * reference's search_file (src/search.c:1467-1478) applied to a session's
 * raw candidate records without sending them to the host.
 *
 *   harvest          record (chunk, slot, j, metric) -> (r, freq, nharm)
 *                    exactly as the host harvest (src/cuda.cu:837-881):
 *                    metric > threshold, r = k * (r_lo + i0*lodr + j*lodr),
 *                    decimated slots only below the Nyquist bin;
 *   base order       records sorted by (chunk, slot, j): the order
 *                    cs_gpu_session_run returns;
 *   remove           remove_duplicates (src/candidate.c:98-128): a stable
 *                    sort by r, runs whose consecutive r differ by at most
 *                    dr_tol, the first member of largest metric of each run
 *                    (a segmented argmax by 64-bit atomicMax);
 *                    the result is in r order, which is also its frequency
 *                    order (freq = r / T, and two members of one list never
 *                    tie in freq without falling into one run);
 *   no remove        a stable sort by frequency (src/search.c:1472);
 *   harm_remove      remove_harmonics (src/candidate.c:130-161): a stable
 *                    sort by descending metric, then greedily each candidate
 *                    not harmonically related to one already kept is kept;
 *                    the kept ones come out in the input (frequency) order,
 *                    which is what the reference's final stable frequency
 *                    sort gives (kept candidates never tie in frequency:
 *                    equal frequencies are related with m = n = 1).
 *
 * remove without a sort at all: bins along r (bin_kernel).  What follows is
 * the way without remove and where the bins would be too many.
 *
 * Ordering without a sort on r: within one decimation slot, r (and freq)
 * rises strictly with the trial index, so a CUB radix sort on (slot, chunk,
 * j) lines every slot up in r order, and a merge places each candidate at
 * its own position in its slot plus, for every other slot, the number of
 * candidates there that come before it in (r, chunk, slot, j) order (a
 * binary search): the stable r order of the (chunk, slot, j) base order.
 * The
 * metrics are FP32 values, so the metric sort uses 32-bit float keys (in shared
 * memory up to CAP candidates, a device radix sort past that).  The greedy
 * pass runs in one CTA: for each kept candidate, in metric order, the threads mark every later
 * candidate it is related to; a candidate is kept when no earlier kept one
 * marked it, as in the host loop.  The FP64 expressions are the host's.
 */
#include <cuda_runtime.h>

#include <atomic>
#include <cub/cub.cuh>

#include <algorithm>
#include <cmath>
#include <cstddef>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "cs_internal.h"
#include "cs_collapse.h"

namespace cl {

constexpr int NT = 256;

struct SlotInfo {
    int k[CS_MAX_SLOT];
    int Hk[CS_MAX_SLOT];
};

__global__ void harvest_kernel(const CsRec *recs, unsigned n, const CsChunk *chunks,
                               long long nchunks, SlotInfo si, int nslot, int nprof,
                               double r_lo, double lodr, double nyq, double T, double thr,
                               uint64_t *key, uint64_t *bkey, int *slot_of, unsigned *idx,
                               double *r, double *freq, double *metric, int *nharm,
                               unsigned *nvalid, unsigned *slot_cnt)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const CsRec rc = recs[i];
    const double m = (double)rc.metric;
    bool ok = m > thr && rc.slot >= 0 && rc.slot < nslot;
    double rsel = INFINITY;
    if (ok) {
        const double rstart = r_lo + (double)chunks[rc.chunk].i0 * lodr;
        const double rfreq = rstart + (double)rc.j * lodr;
        const double kmul = (double)si.k[rc.slot];
        rsel = kmul != 1.0 ? kmul * rfreq : rfreq;
        if (rc.slot != 0 && !(rsel < nyq)) ok = false;
    }
    idx[i] = i;
    if (ok) {
        /* sort key (slot, chunk, j); tie-break key (chunk, slot, j), the base order */
        key[i] = ((uint64_t)rc.slot * (uint64_t)nchunks + (uint64_t)rc.chunk) * (uint64_t)nprof +
                 (uint64_t)rc.j;
        bkey[i] = ((uint64_t)rc.chunk * (uint64_t)nslot + (uint64_t)rc.slot) * (uint64_t)nprof +
                  (uint64_t)rc.j;
        slot_of[i] = rc.slot;
        atomicAdd(&slot_cnt[rc.slot], 1u);
        r[i] = rsel;
        freq[i] = rsel / T;
        metric[i] = m;
        nharm[i] = si.Hk[rc.slot];
        atomicAdd(nvalid, 1u);
    } else {
        key[i] = ~0ull;                 /* after every valid record */
        bkey[i] = ~0ull;
        slot_of[i] = 0;
        r[i] = INFINITY;
        freq[i] = INFINITY;
        metric[i] = -INFINITY;
        nharm[i] = 0;
    }
}

__global__ void slot_starts_kernel(const unsigned *cnt, int nslot, unsigned *start)
{
    unsigned acc = 0;
    for (int s = 0; s < nslot; s++) { start[s] = acc; acc += cnt[s]; }
}

/* order1 holds the valid records grouped by slot, each group in trial order
 * (so in strictly rising v); out receives them in (v, base key) order */
__global__ void merge_kernel(const unsigned *order1, const unsigned *nv, const int *slot_of,
                             const uint64_t *bkey, const double *v, const unsigned *start,
                             const unsigned *cnt, int nslot, unsigned *out)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nv) return;
    const unsigned x = order1[i];
    const int s = slot_of[x];
    const double vx = v[x];
    const uint64_t bx = bkey[x];
    unsigned rank = i - start[s];
    for (int t = 0; t < nslot; t++) {
        if (t == s || cnt[t] == 0) continue;
        unsigned lo = start[t], hi = start[t] + cnt[t], a = lo, b = hi;
        while (a < b) {
            const unsigned mid = (a + b) >> 1;
            if (v[order1[mid]] < vx) a = mid + 1; else b = mid;
        }
        unsigned c = a - lo;
        if (a < hi && v[order1[a]] == vx && bkey[order1[a]] < bx) c++;
        rank += c;
    }
    out[rank] = x;
}

/* run starts of remove_duplicates over the first nv of the r-sorted list
 * (zero past nv, so that a scan over all n entries counts only real runs) */
__global__ void run_flags_kernel(const unsigned *order, const double *r, unsigned n,
                                 const unsigned *nv, double drtol, unsigned *flag)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    flag[i] = i < *nv && (i == 0 || r[order[i]] - r[order[i - 1]] > drtol) ? 1u : 0u;
}

/* the first member of largest metric of each run, as a segmented argmax:
 * every candidate offers (metric, earliest position) to its run with one
 * 64-bit atomicMax.  The metrics are FP32 values, so their float bits (made
 * order-preserving) compare like the doubles the host compares. */
static __device__ __forceinline__ uint32_t ordered_bits(float f)
{
    const uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__global__ void run_offer_kernel(const unsigned *order, const double *metric,
                                 const unsigned *flag, const unsigned *runid,
                                 const unsigned *nv, unsigned long long *best)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= *nv) return;
    const unsigned run = runid[i] + flag[i] - 1u;
    const unsigned long long key =
        ((unsigned long long)ordered_bits((float)metric[order[i]]) << 32) |
        (unsigned long long)(0xFFFFFFFFu - i);
    atomicMax(&best[run], key);
}

__global__ void run_take_kernel(const unsigned *order, const unsigned long long *best,
                                unsigned n, const unsigned *m, unsigned *out)
{
    const unsigned r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n || r >= *m) return;
    out[r] = order[0xFFFFFFFFu - (unsigned)(best[r] & 0xFFFFFFFFull)];
}

__global__ void count_runs_kernel(const unsigned *flag, const unsigned *runid, unsigned n,
                                  unsigned *m)
{
    *m = runid[n - 1] + flag[n - 1];
}

__global__ void copy_count_kernel(const unsigned *src, unsigned *dst)
{
    *dst = *src;
}

/* whether the mm-th harmonic of the one is some harmonic of the other */
static __device__ __forceinline__ bool related_at(double r1, double r2, int mm, int numharm, double tol)
{
    const double lo = r1 < r2 ? r1 : r2;
    const double hi = r1 < r2 ? r2 : r1;
    if (!(lo > 0.0)) return false;
    const int nn = (int)rint((double)mm * hi / lo);
    if (nn < 1 || nn > numharm) return false;
    return fabs((double)mm * hi - (double)nn * lo) <= tol * (double)mm;
}

static __device__ bool related(double r1, double r2, int numharm, double tol)
{
    const double lo = r1 < r2 ? r1 : r2;
    const double hi = r1 < r2 ? r2 : r1;
    if (!(lo > 0.0)) return false;
    for (int mm = 1; mm <= numharm; mm++) {
        const int nn = (int)rint((double)mm * hi / lo);
        if (nn < 1 || nn > numharm) continue;
        if (fabs((double)mm * hi - (double)nn * lo) <= tol * (double)mm) return true;
    }
    return false;
}

/* ---- the last steps, in one CTA of FT threads ----
 * remove_harmonics over a list of m candidates in frequency order: the
 * stable descending metric order, the greedy walk over it, and the kept ones out
 * in list order.  With up to CAP candidates everything is in shared memory; a
 * step of the walk, which is serial in the list, then costs a shared read. */
constexpr int FT = 1024;
constexpr unsigned CAP = 4096;
using MetricSort = cub::BlockRadixSort<uint32_t, FT, CAP / FT, uint16_t>;

struct FinishShared {
    double rs[CAP];                 /* r in metric order */
    uint16_t pos[CAP];              /* list position of each */
    unsigned char rm[CAP];          /* removed, in metric order */
    unsigned char keep[CAP];        /* by list position */
    unsigned warp_tot[32];
    unsigned base;
};

/* keep[] for the m <= CAP candidates whose metric and r get(p) gives; stmp is
 * the radix sort's storage.  Short lists are ranked by counting. */
template <class Get>
static __device__ void harmonics_keep(FinishShared &f, MetricSort::TempStorage &stmp, unsigned m,
                                      int numharm, double tol, Get get)
{
    const unsigned tid = threadIdx.x;
    if (m <= FT / 2) {
        uint32_t *key = reinterpret_cast<uint32_t *>(&stmp);
        double r = 0.0;
        uint32_t k = 0;
        if (tid < m) {
            float mt;
            get(tid, mt, r);
            k = ordered_bits(mt + 0.0f);        /* -0 and 0 compare equal */
            key[tid] = k;
        }
        __syncthreads();
        if (tid < m) {
            unsigned rank = 0;
            for (unsigned i = 0; i < m; i++) {
                const uint32_t o = key[i];
                rank += o > k || (o == k && i < tid) ? 1u : 0u;
            }
            f.rs[rank] = r;
            f.pos[rank] = (uint16_t)tid;
            f.rm[rank] = 0;
        }
    } else {
        uint32_t k[CAP / FT];
        uint16_t v[CAP / FT];
#pragma unroll
        for (unsigned u = 0; u < CAP / FT; u++) {
            const unsigned p = tid * (CAP / FT) + u;
            float mt = 0.0f;
            double r;
            if (p < m) get(p, mt, r);
            k[u] = p < m ? ~ordered_bits(mt + 0.0f) : 0xFFFFFFFFu;
            v[u] = (uint16_t)p;
        }
        __syncthreads();
        MetricSort(stmp).Sort(k, v);        /* stable: equal metrics stay in list order */
        __syncthreads();
#pragma unroll
        for (unsigned u = 0; u < CAP / FT; u++) {
            const unsigned q = tid * (CAP / FT) + u;
            if (q < m) {
                float mt;
                double r;
                get(v[u], mt, r);
                f.rs[q] = r;
                f.pos[q] = v[u];
                f.rm[q] = 0;
            }
        }
    }
    __syncthreads();
    /* the next one not removed: the same in every thread, since a step writes no
     * mark before its own */
    auto next = [&](unsigned i) {
        while (i < m && f.rm[i]) i++;
        return i;
    };
    /* While more follow than half the threads, a thread has a candidate and stops at
     * its first related harmonic; then a thread for each (candidate, harmonic), a
     * step being one FP64 division deep and not numharm of them (40 candidates, 4
     * kept: 20 k cycles -> 8 k).  (What 53 k records of noise
     * leave after remove_duplicates: 3.14 ms with pairs all the way, 2.33 so; 4 k
     * trials of one pulsar 344 us and 305.)  Harmonics past 2^31 / FT never pair:
     * the number of pairs stays in 32 bits. */
    const unsigned nh = numharm > 0 ? (unsigned)numharm : 0u;
    unsigned i = next(0);
    for (; i < m && (m - i - 1 > FT / 2 || nh > (1u << 31) / FT); i = next(i + 1)) {
        const double ri = f.rs[i];
        for (unsigned j = i + 1 + tid; j < m; j += FT)
            if (!f.rm[j] && related(f.rs[j], ri, numharm, tol)) f.rm[j] = 1;
        __syncthreads();
    }
    for (; i < m; i = next(i + 1)) {
        const double ri = f.rs[i];
        const unsigned pairs = (m - i - 1) * nh;
        for (unsigned q = tid; q < pairs; q += FT) {
            const unsigned d = q / nh, j = i + 1 + d;
            if (!f.rm[j] && related_at(f.rs[j], ri, (int)(q - d * nh) + 1, numharm, tol)) f.rm[j] = 1;
        }
        __syncthreads();
    }
    for (unsigned q = tid; q < m; q += FT) f.keep[f.pos[q]] = !f.rm[q];
    __syncthreads();
}

/* The candidates p < m with keep(p), in order, to out; their number. */
template <class Keep, class Put>
static __device__ unsigned emit_kept(FinishShared &f, unsigned m, Keep keep, Put put)
{
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (threadIdx.x == 0) f.base = 0;
    __syncthreads();
    for (unsigned s = 0; s < m; s += FT) {
        const unsigned i = s + threadIdx.x;
        const bool k = i < m && keep(i);
        const unsigned bal = __ballot_sync(0xffffffffu, k);
        if (lane == 0) f.warp_tot[w] = __popc(bal);
        __syncthreads();
        unsigned off = f.base, all = 0;
        for (unsigned q = 0; q < FT / 32; q++) {
            if (q < w) off += f.warp_tot[q];
            all += f.warp_tot[q];
        }
        if (k) put(i, off + __popc(bal & ((1u << lane) - 1u)));
        __syncthreads();
        if (threadIdx.x == 0) f.base += all;
        __syncthreads();
    }
    return f.base;
}

static __device__ __forceinline__ Candidate make_cand(double r, double freq, double metric, int nharm)
{
    Candidate c;
    c.freq = freq;
    c.metric = metric;
    c.r = r;
    c.nharm = nharm;
    c.ducy = NAN;
    return c;
}

/* ---- remove_duplicates without a sort ----
 * Bins of just under dr_tol along r: two records of one bin always belong to
 * one run, two with two empty bins between them never do, and neighbours are
 * decided by the largest r of the one and the smallest of the other, which are
 * the two values the sorted list would compare.  So a run is a stretch of bins,
 * and its first member of largest metric is the first of its bins' bests.  Four
 * kernels and one memset on the list take the place of the radix sort on
 * (slot, chunk, j), the merge of the slots and the scan: launches are what a list
 * of some ten thousand records costs.  (A list of 10 k records from 150 k points:
 * 100 -> 33 us of kernels; 32 of them with their searches 6.4 -> 4.5 ms.) */
constexpr int BT = 1024;                /* bins in a block */
constexpr unsigned NONE = 0xFFFFFFFFu;
constexpr unsigned long long BINS_PER_REC = 1024, BINS_MOST = 1u << 24;

struct Bins {                           /* all ones before a list */
    unsigned long long *best;           /* [n] by run: inverted (metric, earliest bin) */
    unsigned long long *lo, *nhi;       /* [nb] bits of the smallest r; inverted, of the largest */
    unsigned *idx;                      /* [nb] the first record of largest metric */
    unsigned *starts;                   /* bit per bin: a run starts there */
    unsigned *cnt;                      /* per block of BT bins: run starts */
    unsigned nb;
    double inv;                         /* bins per unit of r */
};

struct RecGeo {                         /* what gives a record its r */
    const CsRec *recs;
    const CsChunk *chunks;
    SlotInfo si;
    int nslot, nprof;
    double r_lo, lodr, nyq, T, thr;
};

static __device__ __forceinline__ double rec_r(const RecGeo &g, const CsRec &rc)
{
    const double rstart = g.r_lo + (double)g.chunks[rc.chunk].i0 * g.lodr;
    const double rfreq = rstart + (double)rc.j * g.lodr;
    const double kmul = (double)g.si.k[rc.slot];
    return kmul != 1.0 ? kmul * rfreq : rfreq;
}

/* Records to their bins.  The lists are short and in the L2: the chains of
 * dependent reads bound it, so no value is written that is already beaten. */
__global__ void __launch_bounds__(NT) bin_kernel(const __grid_constant__ RecGeo g, unsigned n,
                                                 const __grid_constant__ Bins bn, double *r,
                                                 double *freq, double *metric, int *nharm)
{
    const unsigned i = blockIdx.x * NT + threadIdx.x;
    if (i >= n) return;
    const CsRec rc = g.recs[i];
    if (!((double)rc.metric > g.thr) || rc.slot < 0 || rc.slot >= g.nslot) return;
    const double x = rec_r(g, rc);
    if (rc.slot != 0 && !(x < g.nyq)) return;
    r[i] = x;
    freq[i] = x / g.T;
    metric[i] = (double)rc.metric;
    nharm[i] = g.si.Hk[rc.slot];
    const unsigned b = min((unsigned)(x * bn.inv), bn.nb - 1u);
    const unsigned long long xb = (unsigned long long)__double_as_longlong(x);
    volatile const unsigned long long *lo = bn.lo, *nhi = bn.nhi;
    if (xb < lo[b]) atomicMin(&bn.lo[b], xb);
    if (~xb < nhi[b]) atomicMin(&bn.nhi[b], ~xb);
    unsigned old = *(volatile unsigned *)&bn.idx[b];
    for (;;) {
        if (old != NONE) {
            const CsRec ro = g.recs[old];
            if (ro.metric > rc.metric) break;
            if (ro.metric == rc.metric) {       /* the earlier in (r, chunk, slot, j) order */
                const double xo = rec_r(g, ro);
                if (xo < x) break;
                if (xo == x && (ro.chunk < rc.chunk ||
                                (ro.chunk == rc.chunk &&
                                 (ro.slot < rc.slot || (ro.slot == rc.slot && ro.j <= rc.j)))))
                    break;
            }
        }
        const unsigned was = atomicCAS(&bn.idx[b], old, i);
        if (was == old) break;
        old = was;
    }
}

/* The bins where a run starts: a word for every 32, their number for every BT. */
__global__ void __launch_bounds__(BT) bin_starts_kernel(const __grid_constant__ Bins bn, double drtol)
{
    const unsigned b = blockIdx.x * BT + threadIdx.x;
    bool start = false;
    if (b < bn.nb && bn.idx[b] != NONE) {
        start = true;
        unsigned p = NONE;
        if (b >= 1 && bn.idx[b - 1] != NONE) p = b - 1;
        else if (b >= 2 && bn.idx[b - 2] != NONE) p = b - 2;
        if (p != NONE)
            start = __longlong_as_double((long long)bn.lo[b]) -
                        __longlong_as_double((long long)~bn.nhi[p]) > drtol;
    }
    const unsigned w = __ballot_sync(0xffffffffu, start);
    if ((threadIdx.x & 31) == 0) bn.starts[b >> 5] = w;
    const int c = __syncthreads_count(start);
    if (threadIdx.x == 0) bn.cnt[blockIdx.x] = (unsigned)c;
}

/* Every bin's best to its run; the number of runs to *m. */
__global__ void __launch_bounds__(BT) bin_offer_kernel(const __grid_constant__ Bins bn,
                                                       const CsRec *recs, unsigned *m)
{
    __shared__ unsigned wsum[BT / 32], wpre[BT / 32];
    __shared__ unsigned base;
    const unsigned lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned b = blockIdx.x * BT + threadIdx.x;
    const unsigned word = bn.starts[b >> 5];
    unsigned s = 0;                             /* the runs of the blocks before */
    for (unsigned q = threadIdx.x; q < blockIdx.x; q += BT) s += bn.cnt[q];
    s = __reduce_add_sync(0xffffffffu, s);
    if (lane == 0) {
        wsum[w] = s;
        wpre[w] = __popc(word);
    }
    __syncthreads();
    if (w == 0) {
        const unsigned all = __reduce_add_sync(0xffffffffu, wsum[lane]);
        const unsigned own = wpre[lane];
        unsigned inc = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned o = __shfl_up_sync(0xffffffffu, inc, d);
            if (lane >= (unsigned)d) inc += o;
        }
        wpre[lane] = inc - own;
        if (lane == 0) base = all;
        if (lane == 31 && blockIdx.x == gridDim.x - 1) *m = all + inc;
    }
    __syncthreads();
    if (b >= bn.nb) return;
    const unsigned x = bn.idx[b];
    if (x == NONE) return;
    const unsigned run = base + wpre[w] + __popc(word & (0xffffffffu >> (31 - lane))) - 1u;
    const unsigned long long inv =
        ~(((unsigned long long)ordered_bits(recs[x].metric + 0.0f) << 32) |
          (unsigned long long)(0xFFFFFFFFu - b));
    if (inv < *(volatile unsigned long long *)&bn.best[run]) atomicMin(&bn.best[run], inv);
}

struct FinishSmem {
    FinishShared f;
    union {
        MetricSort::TempStorage sort;
        uint32_t keys[FT];
    } t;
};

/* The last steps for a list in global memory, which the runs' bests give first
 * when there are any.  `keep` says which candidates stay; null: found here for up to
 * CAP of them, and a longer list is left for order_and_walk, with its length in
 * nout[1].  The first CAP of the result also go to pinned memory, with the number: no
 * copy, and one wait less. */
__global__ void __launch_bounds__(FT) finish_kernel(unsigned *list, const unsigned long long *best,
                                                    const unsigned *bidx, const unsigned *mp,
                                                    int harm_remove, int numharm, double tol,
                                                    const double *r, const double *freq,
                                                    const double *metric, const int *nharm,
                                                    const unsigned char *keep, Candidate *out,
                                                    Candidate *pinned, unsigned *nout)
{
    extern __shared__ __align__(16) unsigned char fsm[];
    FinishSmem &sm = *reinterpret_cast<FinishSmem *>(fsm);
    const unsigned m = *mp;
    if (best) {
        for (unsigned p = threadIdx.x; p < m; p += FT) list[p] = bidx[(unsigned)best[p]];
        __syncthreads();
    }
    if (harm_remove && !keep) {
        if (m > CAP) {
            if (threadIdx.x == 0) {
                nout[0] = 0;
                nout[1] = m;
            }
            return;
        }
        harmonics_keep(sm.f, sm.t.sort, m, numharm, tol, [&](unsigned p, float &mt, double &rr) {
            const unsigned c = list[p];
            mt = (float)metric[c];              /* FP32 values: exact */
            rr = r[c];
        });
    }
    const unsigned n = emit_kept(
        sm.f, m, [&](unsigned i) { return !harm_remove || (keep ? keep[i] : sm.f.keep[i]); },
        [&](unsigned i, unsigned o) {
            const unsigned c = list[i];
            const Candidate x = make_cand(r[c], freq[c], metric[c], nharm[c]);
            out[o] = x;
            if (o < CAP) pinned[o] = x;
        });
    if (threadIdx.x == 0) {
        nout[0] = n;
        nout[1] = 0;
    }
}

/* ---- remove_harmonics of more than CAP candidates ---- */
/* metric keys of the list, for the stable descending sort */
__global__ void metric_keys_kernel(const unsigned *list, const double *metric, unsigned n,
                                   const unsigned *m, float *key, unsigned *pos)
{
    const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    key[i] = i < *m ? (float)metric[list[i]] : -INFINITY;     /* FP32 values: exact */
    pos[i] = i;
}

/* The greedy walk over the metric order (one CTA), serial in the list: up to
 * WALK_SMEM candidates' r and marks are in shared memory, so that a step costs a
 * shared read and not two dependent global ones. */
constexpr unsigned WALK_SMEM = 8192;
constexpr size_t WALK_BYTES = WALK_SMEM * (sizeof(double) + 1);
__global__ void __launch_bounds__(FT) walk_kernel(const unsigned *list, const unsigned *pos,
                                                  const double *r, const unsigned *mp, int numharm,
                                                  double tol, unsigned char *removed,
                                                  unsigned char *keep)
{
    extern __shared__ double wsm[];
    const unsigned m = *mp;
    auto walk = [&](unsigned char *rm, auto at) {
        for (unsigned i = 0; i < m; i++) {
            if (rm[i]) continue;                /* the same value in every thread */
            const double ri = at(i);
            for (unsigned j = i + 1 + threadIdx.x; j < m; j += FT)
                if (!rm[j] && related(at(j), ri, numharm, tol)) rm[j] = 1;
            __syncthreads();
        }
        for (unsigned q = threadIdx.x; q < m; q += FT) keep[pos[q]] = !rm[q];
    };
    unsigned char *rs = reinterpret_cast<unsigned char *>(wsm + WALK_SMEM);
    for (unsigned j = threadIdx.x; j < m; j += FT) {
        if (m <= WALK_SMEM) {
            wsm[j] = r[list[pos[j]]];
            rs[j] = 0;
        } else {
            removed[j] = 0;
        }
    }
    __syncthreads();
    if (m <= WALK_SMEM) walk(rs, [&](unsigned i) { return wsm[i]; });
    else walk(removed, [&](unsigned i) { return r[list[pos[i]]]; });
}

/* ---- the whole collapse of up to CAP records in one CTA ----
 * The same steps on shared memory: one launch where the long-list path has
 * about twenty, none of which has work for more than a CTA then.  It reads the
 * record count on the device, so it can be queued behind a search whose count
 * the host does not know yet, and writes the list to pinned host memory: one
 * wait in all.  (1 M points, 2000 records: 14 us of kernel, 33 with the records
 * sorted, against 75 us of kernels, two waits and a copy; a whole pass 523 -> 428
 * -> 410 us.) */
template <unsigned IT>
using SlotSort = cub::BlockRadixSort<uint32_t, FT, IT, uint16_t>;

struct SmallArgs {
    const CsRec *recs;
    const unsigned *count;
    const int *err;
    unsigned cap;                   /* of the record buffer */
    const CsChunk *chunks;
    SlotInfo si;
    int nslot;
    uint32_t total;                 /* trials; nslot * total < 2^32 - 1 */
    int end_bit;
    double r_lo, lodr, nyq, T, thr;
    int remove, harm_remove, numharm;
    double drtol, tol;
    double inv;                     /* bins per unit of r; negative: order the records instead */
    Candidate *out;                 /* pinned, CAP */
    unsigned *status;               /* pinned: records, error flag, list length, done */
};

/* The bins of a short list, in a hash table: a bin takes a place when its first
 * record comes.  All ones before. */
constexpr unsigned HS = 5120;           /* places; at most CAP are taken */
constexpr unsigned RUNS = FT;           /* runs that are ranked by counting */
struct Hashed {
    uint32_t key[HS];               /* bin */
    uint32_t nmet[HS];              /* inverted order of the largest metric */
    uint32_t qlo[HS], nqhi[HS];     /* smallest place in the bin, inverted largest */
    uint16_t bi[HS];                /* first record of largest metric */
    uint16_t li[HS], hi[HS];        /* records of smallest (later the run) and largest r */
    uint16_t occ[CAP];              /* taken places */
    uint32_t sbin[RUNS], order[RUNS];   /* bins where a run starts, as found and in order */
    unsigned long long best[RUNS];
    unsigned nocc, nstart;
};

struct SmallSmem {
    double rr[CAP];                 /* r of each record */
    float met[CAP];
    int chunk[CAP];
    unsigned char slot[CAP];
    uint16_t list[CAP];             /* the best of each run */
    unsigned cnt[CS_MAX_SLOT + 1], start[CS_MAX_SLOT + 1];
    unsigned m;
    union {
        struct {
            double v[CAP];          /* sort value (r or freq), slots in turn, rising in each */
            uint16_t idx[CAP];      /* its record */
            uint16_t ord[CAP];      /* records in (value, base) order */
            union {
                unsigned long long best[CAP];
                SlotSort<1>::TempStorage sort1;
                SlotSort<2>::TempStorage sort2;
                SlotSort<4>::TempStorage sort4;
            } u;
            typename cub::BlockScan<unsigned, FT>::TempStorage scan;
        } o;
        Hashed h;
        FinishSmem fin;             /* once the list is made */
    };
};
static_assert(offsetof(Hashed, occ) % 16 == 0, "cleared in 16-byte stores");
static_assert(sizeof(SmallSmem) <= 220 * 1024 && CAP == 4 * FT, "one CTA's shared memory");

static __device__ __forceinline__ unsigned hash_place(uint32_t b)
{
    return __umulhi(b * 2654435761u, HS);
}

static __device__ __forceinline__ unsigned hash_find(const Hashed &h, uint32_t b)
{
    for (unsigned s = hash_place(b);; s = s + 1 == HS ? 0 : s + 1) {
        const uint32_t k = h.key[s];
        if (k == b) return s;
        if (k == NONE) return NONE;
    }
}

/* slot = i where wins(i, the record there) */
template <class Wins>
static __device__ __forceinline__ void offer16(uint16_t *slot, unsigned i, Wins wins)
{
    unsigned short old = *(volatile uint16_t *)slot;
    while (old == 0xFFFF || wins(i, (unsigned)old)) {
        const unsigned short was = atomicCAS((unsigned short *)slot, old, (unsigned short)i);
        if (was == old) break;
        old = was;
    }
}

/* Harvest and remove_duplicates of n <= CAP records by bins (above): sm.list and
 * sm.m, or false when there are more than RUNS runs.  A run is often hundreds of
 * records (a strong line at every trial and decimation around it), so few bins are
 * ordered where the sort orders all records: 2000 records in 19 runs, 40 k cycles
 * by sort and merge, 15 k so.  What the bins need exactly (the earliest of equal metrics, the
 * r at a bin's ends) is found in two steps, 32-bit atomics first and comparisons
 * between the few that tie. */
static __device__ bool hash_list(SmallSmem &sm, const SmallArgs &a, unsigned n)
{
    Hashed &h = sm.h;
    const unsigned tid = threadIdx.x;
    for (unsigned i = tid; i < offsetof(Hashed, occ) / 16; i += FT)
        reinterpret_cast<uint4 *>(&h)[i] = make_uint4(NONE, NONE, NONE, NONE);
    h.best[tid] = 0;
    if (tid == 0) h.nocc = h.nstart = 0;
    __syncthreads();
    unsigned place[CAP / FT];
    uint32_t nm[CAP / FT], q[CAP / FT];
#pragma unroll
    for (unsigned u = 0; u < CAP / FT; u++) {
        place[u] = NONE;
        nm[u] = q[u] = 0;
        if (u * FT >= n) continue;
        const unsigned i = u * FT + tid;
        if (i < n) {
            const CsRec rc = a.recs[i];
            bool ok = (double)rc.metric > a.thr && rc.slot >= 0 && rc.slot < a.nslot;
            double x = 0.0;
            if (ok) {
                const double rstart = a.r_lo + (double)a.chunks[rc.chunk].i0 * a.lodr;
                const double rfreq = rstart + (double)rc.j * a.lodr;
                const double kmul = (double)a.si.k[rc.slot];
                x = kmul != 1.0 ? kmul * rfreq : rfreq;
                ok = rc.slot == 0 || x < a.nyq;
            }
            if (ok) {
                sm.rr[i] = x;
                sm.met[i] = rc.metric;
                sm.chunk[i] = rc.chunk;
                sm.slot[i] = (unsigned char)rc.slot;
                const double p = x * a.inv;
                const uint32_t b = (uint32_t)p;
                nm[u] = ~ordered_bits(rc.metric + 0.0f);
                q[u] = (uint32_t)((p - (double)b) * 4294967296.0);
                for (unsigned s = hash_place(b);; s = s + 1 == HS ? 0 : s + 1) {
                    uint32_t k = *(volatile uint32_t *)&h.key[s];
                    if (k == NONE) {
                        k = atomicCAS(&h.key[s], NONE, b);
                        if (k == NONE) {
                            h.occ[atomicAdd(&h.nocc, 1u)] = (uint16_t)s;
                            k = b;
                        }
                    }
                    if (k == b) {
                        place[u] = s;
                        break;
                    }
                }
            }
        }
        __syncwarp();
        int same;
        __match_all_sync(0xffffffffu, place[u], &same);
        if (same) {                         /* neighbours in the list often share a bin */
            const uint32_t m0 = __reduce_min_sync(0xffffffffu, nm[u]);
            const uint32_t l0 = __reduce_min_sync(0xffffffffu, q[u]);
            const uint32_t h0 = __reduce_min_sync(0xffffffffu, ~q[u]);
            if (place[u] != NONE && (tid & 31) == 0) {
                atomicMin(&h.nmet[place[u]], m0);
                atomicMin(&h.qlo[place[u]], l0);
                atomicMin(&h.nqhi[place[u]], h0);
            }
        } else if (place[u] != NONE) {
            atomicMin(&h.nmet[place[u]], nm[u]);
            atomicMin(&h.qlo[place[u]], q[u]);
            atomicMin(&h.nqhi[place[u]], ~q[u]);
        }
    }
    __syncthreads();
#pragma unroll
    for (unsigned u = 0; u < CAP / FT; u++) {
        const unsigned s = place[u], i = u * FT + tid;
        if (s == NONE) continue;
        if (h.nmet[s] == nm[u])
            offer16(&h.bi[s], i, [&](unsigned y, unsigned o) {
                if (sm.rr[y] != sm.rr[o]) return sm.rr[y] < sm.rr[o];
                return sm.chunk[y] < sm.chunk[o] ||
                       (sm.chunk[y] == sm.chunk[o] && sm.slot[y] < sm.slot[o]);
            });
        if (h.qlo[s] == q[u])
            offer16(&h.li[s], i, [&](unsigned y, unsigned o) { return sm.rr[y] < sm.rr[o]; });
        if (h.nqhi[s] == ~q[u])
            offer16(&h.hi[s], i, [&](unsigned y, unsigned o) { return sm.rr[y] > sm.rr[o]; });
    }
    __syncthreads();
    const unsigned nocc = h.nocc;
    for (unsigned o = tid; o < nocc; o += FT) {
        const unsigned s = h.occ[o];
        const uint32_t b = h.key[s];
        unsigned p = b >= 1 ? hash_find(h, b - 1) : NONE;
        if (p == NONE && b >= 2) p = hash_find(h, b - 2);
        if (p == NONE || sm.rr[h.li[s]] - sm.rr[h.hi[p]] > a.drtol) {
            const unsigned at = atomicAdd(&h.nstart, 1u);
            if (at < RUNS) h.sbin[at] = b;
        }
    }
    __syncthreads();
    const unsigned m = h.nstart;
    if (m > RUNS) return false;
    if (tid < m) {
        const uint32_t b = h.sbin[tid];
        unsigned rank = 0;
#pragma unroll 4
        for (unsigned i = 0; i < m; i++) rank += h.sbin[i] < b ? 1u : 0u;
        h.order[rank] = b;
    }
    __syncthreads();
    for (unsigned o = tid; o < nocc; o += FT) {
        const unsigned s = h.occ[o];
        const uint32_t b = h.key[s];
        unsigned lo = 0, e = m;             /* the last start at or before b */
        while (e - lo > 1) {
            const unsigned mid = (lo + e) >> 1;
            if (h.order[mid] <= b) lo = mid;
            else e = mid;
        }
        h.li[s] = (uint16_t)lo;
        atomicMax(&h.best[lo], ((unsigned long long)~h.nmet[s] << 32) |
                                   (unsigned long long)(0xFFFFFFFFu - b));
    }
    __syncthreads();
    for (unsigned o = tid; o < nocc; o += FT) {
        const unsigned s = h.occ[o];
        const unsigned long long key = ((unsigned long long)~h.nmet[s] << 32) |
                                       (unsigned long long)(0xFFFFFFFFu - h.key[s]);
        if (h.best[h.li[s]] == key) sm.list[h.li[s]] = h.bi[s];
    }
    if (tid == 0) sm.m = m;
    __syncthreads();
    return true;
}

/* Harvest, order and remove_duplicates of n <= IT * FT records: sm.list, sm.m. */
template <unsigned IT>
static __device__ void small_list(SmallSmem &sm, const SmallArgs &a, unsigned n,
                                  typename SlotSort<IT>::TempStorage &tmp)
{
    const unsigned tid = threadIdx.x;
    if (tid <= CS_MAX_SLOT) sm.cnt[tid] = 0;
    __syncthreads();
    /* harvest */
    uint32_t key[IT];
    uint16_t val[IT];
#pragma unroll
    for (unsigned u = 0; u < IT; u++) {
        const unsigned i = tid * IT + u;
        key[u] = a.total * (uint32_t)a.nslot;       /* after every valid record */
        val[u] = (uint16_t)i;
        if (i >= n) continue;
        const CsRec rc = a.recs[i];
        if (!((double)rc.metric > a.thr) || rc.slot < 0 || rc.slot >= a.nslot) continue;
        const long long i0 = a.chunks[rc.chunk].i0;
        const double rstart = a.r_lo + (double)i0 * a.lodr;
        const double rfreq = rstart + (double)rc.j * a.lodr;
        const double kmul = (double)a.si.k[rc.slot];
        const double rsel = kmul != 1.0 ? kmul * rfreq : rfreq;
        if (rc.slot != 0 && !(rsel < a.nyq)) continue;
        key[u] = (uint32_t)rc.slot * a.total + (uint32_t)(i0 + rc.j);
        sm.rr[i] = rsel;
        sm.met[i] = rc.metric;
        sm.chunk[i] = rc.chunk;
        sm.slot[i] = (unsigned char)rc.slot;
        atomicAdd(&sm.cnt[rc.slot], 1u);
    }
    __syncthreads();
    SlotSort<IT>(tmp).Sort(key, val, 0, a.end_bit);
    if (tid == 0) {
        unsigned acc = 0;
        for (int s = 0; s < a.nslot; s++) {
            sm.start[s] = acc;
            acc += sm.cnt[s];
        }
        sm.start[a.nslot] = acc;
    }
    __syncthreads();
    const unsigned nv = sm.start[a.nslot];
#pragma unroll
    for (unsigned u = 0; u < IT; u++) {
        const unsigned p = tid * IT + u;
        if (p < nv) {
            sm.o.idx[p] = val[u];
            sm.o.v[p] = a.remove ? sm.rr[val[u]] : sm.rr[val[u]] / a.T;
        }
    }
    __syncthreads();
    /* merge the slots: a record's place in its own plus, for every other, the
     * records there before it in (value, chunk, slot) order */
    for (unsigned p = tid; p < nv; p += FT) {
        const unsigned x = sm.o.idx[p];
        const int s = sm.slot[x];
        const double vx = sm.o.v[p];
        unsigned rank = p - sm.start[s];
        for (int t = 0; t < a.nslot; t++) {
            if (t == s) continue;
            const unsigned lo = sm.start[t], hi = sm.start[t + 1];
            unsigned b = lo, e = hi;
            while (b < e) {
                const unsigned mid = (b + e) >> 1;
                if (sm.o.v[mid] < vx) b = mid + 1;
                else e = mid;
            }
            rank += b - lo;
            if (b < hi && sm.o.v[b] == vx) {
                const int cy = sm.chunk[sm.o.idx[b]], cx = sm.chunk[x];
                if (cy < cx || (cy == cx && t < s)) rank++;
            }
        }
        sm.o.ord[rank] = (uint16_t)x;
    }
    __syncthreads();
    if (a.remove) {
        for (unsigned i = tid; i < nv; i += FT) sm.o.u.best[i] = 0;
        unsigned flag[IT], run[IT];
#pragma unroll
        for (unsigned u = 0; u < IT; u++) {
            const unsigned i = tid * IT + u;
            flag[u] = i < nv && (i == 0 || sm.rr[sm.o.ord[i]] - sm.rr[sm.o.ord[i - 1]] > a.drtol) ? 1u : 0u;
        }
        unsigned runs;
        cub::BlockScan<unsigned, FT>(sm.o.scan).InclusiveSum(flag, run, runs);
        __syncthreads();
#pragma unroll
        for (unsigned u = 0; u < IT; u++) {
            const unsigned i = tid * IT + u;
            if (i < nv)
                atomicMax(&sm.o.u.best[run[u] - 1],
                          ((unsigned long long)ordered_bits(sm.met[sm.o.ord[i]]) << 32) |
                              (unsigned long long)(0xFFFFFFFFu - i));
        }
        __syncthreads();
        for (unsigned q = tid; q < runs; q += FT)
            sm.list[q] = sm.o.ord[0xFFFFFFFFu - (unsigned)(sm.o.u.best[q] & 0xFFFFFFFFull)];
        if (tid == 0) sm.m = runs;
    } else {
        for (unsigned q = tid; q < nv; q += FT) sm.list[q] = sm.o.ord[q];
        if (tid == 0) sm.m = nv;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(FT) collapse_small(const __grid_constant__ SmallArgs a)
{
    extern __shared__ __align__(16) unsigned char ssm[];
    SmallSmem &sm = *reinterpret_cast<SmallSmem *>(ssm);
    const unsigned tid = threadIdx.x;
    const unsigned n = *a.count;
    const int err = *a.err;
    if (tid == 0) {
        a.status[0] = n;
        a.status[1] = (unsigned)err;
        a.status[2] = 0;
        a.status[3] = err == 0 && n <= a.cap && n <= CAP ? 1u : 0u;
    }
    if (err != 0 || n > a.cap || n > CAP || n == 0) return;
    if (a.inv < 0.0 || !hash_list(sm, a, n)) {
        if (n <= FT) small_list<1>(sm, a, n, sm.o.u.sort1);
        else if (n <= 2 * FT) small_list<2>(sm, a, n, sm.o.u.sort2);
        else small_list<4>(sm, a, n, sm.o.u.sort4);
    }
    const unsigned m = sm.m;
    if (a.harm_remove)
        harmonics_keep(sm.fin.f, sm.fin.t.sort, m, a.numharm, a.tol,
                       [&](unsigned p, float &mt, double &r) {
                           mt = sm.met[sm.list[p]];
                           r = sm.rr[sm.list[p]];
                       });
    const unsigned kept = emit_kept(
        sm.fin.f, m, [&](unsigned i) { return !a.harm_remove || sm.fin.f.keep[i]; },
        [&](unsigned i, unsigned o) {
            const unsigned c = sm.list[i];
            a.out[o] = make_cand(sm.rr[c], sm.rr[c] / a.T, (double)sm.met[c], a.si.Hk[sm.slot[c]]);
        });
    if (tid == 0) a.status[2] = kept;
}

}  // namespace cl

/* The one-CTA kernels' shared-memory limits, raised once per device (the
 * attribute belongs to the device that is current when it is set). */
static cudaError_t finish_prepare()
{
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess || dev < 0 || dev >= 64) return e;
    const unsigned long long bit = 1ULL << dev;
    if (done.load(std::memory_order_acquire) & bit) return cudaSuccess;
    e = cudaFuncSetAttribute((const void *)cl::finish_kernel,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(cl::FinishSmem));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void *)cl::walk_kernel,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cl::WALK_BYTES);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute((const void *)cl::collapse_small,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)sizeof(cl::SmallSmem));
    if (e == cudaSuccess) done.fetch_or(bit, std::memory_order_acq_rel);
    return e;
}

struct CsCollapse {
    size_t cap;                     /* records */
    uint64_t *key[2];
    unsigned *idx[2];
    uint64_t *bkey;
    int *slot_of;
    unsigned *merged;
    double *r, *freq, *metric;
    int *nharm;
    unsigned *flag, *runid, *list;
    float *mkey[2];
    unsigned *mpos[2];
    unsigned char *removed, *keep;
    Candidate *out;
    unsigned *counters;             /* device: valid, runs; then per-slot counts and
                                       starts (CS_MAX_SLOT each) */
    unsigned *h_counters;           /* pinned: the length of the list; of one that
                                       order_and_walk has yet to do, or 0 */
    void *bins;                     /* Bins, for the longest list so far */
    size_t bins_bytes;
    Candidate *h_out;               /* pinned */
    size_t h_out_cap;
    void *temp;
    size_t temp_bytes;
    unsigned pending_n;             /* records of the enqueued collapse */
    unsigned *pending_list;         /* its list, and the harmonics' settings */
    int numharm, device;
    double harm_tol;
    /* collapse_small's list and status (pinned), and whether it is queued */
    Candidate *s_out;
    unsigned *s_status;
    bool small;
};

static void collapse_release_buffers(CsCollapse *w)
{
    for (int b = 0; b < 2; b++) {
        cudaFree(w->key[b]); cudaFree(w->idx[b]); cudaFree(w->mkey[b]); cudaFree(w->mpos[b]);
        w->key[b] = nullptr; w->idx[b] = nullptr; w->mkey[b] = nullptr; w->mpos[b] = nullptr;
    }
    cudaFree(w->bkey); cudaFree(w->slot_of); cudaFree(w->merged);
    w->bkey = nullptr; w->slot_of = nullptr; w->merged = nullptr;
    cudaFree(w->r); cudaFree(w->freq); cudaFree(w->metric); cudaFree(w->nharm);
    cudaFree(w->flag); cudaFree(w->runid); cudaFree(w->list);
    cudaFree(w->removed); cudaFree(w->keep); cudaFree(w->out); cudaFree(w->temp);
    w->r = w->freq = w->metric = nullptr;
    w->nharm = nullptr;
    w->flag = w->runid = w->list = nullptr;
    w->removed = w->keep = nullptr;
    w->out = nullptr;
    w->temp = nullptr;
    w->temp_bytes = 0;
    w->cap = 0;
}

static cudaError_t collapse_reserve(CsCollapse *w, size_t n)
{
    if (n <= w->cap) return cudaSuccess;
    collapse_release_buffers(w);
    const size_t c = n + n / 4 + 1024;
    cudaError_t e = cudaSuccess;
#define AL(p, bytes) if (e == cudaSuccess) e = cudaMalloc((void **)&(p), (bytes))
    for (int b = 0; b < 2; b++) {
        AL(w->key[b], c * sizeof(uint64_t));
        AL(w->idx[b], c * sizeof(unsigned));
        AL(w->mkey[b], c * sizeof(float));
        AL(w->mpos[b], c * sizeof(unsigned));
    }
    AL(w->bkey, c * sizeof(uint64_t));
    AL(w->slot_of, c * sizeof(int));
    AL(w->merged, c * sizeof(unsigned));
    AL(w->r, c * sizeof(double));
    AL(w->freq, c * sizeof(double));
    AL(w->metric, c * sizeof(double));
    AL(w->nharm, c * sizeof(int));
    AL(w->flag, c * sizeof(unsigned));
    AL(w->runid, c * sizeof(unsigned));
    AL(w->list, c * sizeof(unsigned));
    AL(w->removed, c);
    AL(w->keep, c);
    AL(w->out, c * sizeof(Candidate));
    if (!w->counters) AL(w->counters, (4 + 2 * CS_MAX_SLOT) * sizeof(unsigned));
#undef AL
    if (e != cudaSuccess) return e;
    /* the largest CUB scratch any step needs at this capacity */
    size_t t1 = 0, t2 = 0, t3 = 0;
    cub::DoubleBuffer<uint64_t> kb(w->key[0], w->key[1]);
    cub::DoubleBuffer<unsigned> ib(w->idx[0], w->idx[1]);
    cub::DoubleBuffer<float> mb(w->mkey[0], w->mkey[1]);
    cub::DoubleBuffer<unsigned> pb(w->mpos[0], w->mpos[1]);
    e = cub::DeviceRadixSort::SortPairs(nullptr, t1, kb, ib, (int)c);
    if (e == cudaSuccess) e = cub::DeviceRadixSort::SortPairsDescending(nullptr, t2, mb, pb, (int)c);
    if (e == cudaSuccess) e = cub::DeviceScan::ExclusiveSum(nullptr, t3, w->flag, w->runid, (int)c);
    if (e != cudaSuccess) return e;
    w->temp_bytes = std::max(t1, std::max(t2, t3));
    e = cudaMalloc(&w->temp, w->temp_bytes);
    if (e == cudaSuccess) w->cap = c;
    return e;
}

CsCollapse *cs_collapse_new(void)
{
    CsCollapse *w = (CsCollapse *)calloc(1, sizeof(CsCollapse));
    if (!w) return nullptr;
    /* one pinned block: a short result, then its status and the length */
    if (cudaMallocHost((void **)&w->s_out, cl::CAP * sizeof(Candidate) + 8 * sizeof(unsigned)) !=
        cudaSuccess) {
        free(w);
        return nullptr;
    }
    w->s_status = (unsigned *)(w->s_out + cl::CAP);
    w->h_counters = w->s_status + 4;
    return w;
}

void cs_collapse_free(CsCollapse *w)
{
    if (!w) return;
    collapse_release_buffers(w);
    cudaFree(w->counters);
    cudaFree(w->bins);
    if (w->h_out) cudaFreeHost(w->h_out);
    if (w->s_out) cudaFreeHost(w->s_out);
    free(w);
}

static int bit_length_u64(uint64_t v)
{
    int b = 0;
    while (v) { b++; v >>= 1; }
    return b;
}

/* Bins along r for a search's trials; inv is negative where they do not hold.
 * They are a millionth narrower than dr_tol; rounding of r and of its product
 * with inv stays below that for up to 2^27 of them.  r >= 0 keeps the order of
 * the bits. */
struct BinScale {
    double inv, bins;
};

static BinScale bin_scale(double r_lo, double lodr, double trials, int k0, double N, double dr_tol)
{
    BinScale s = {-1.0, 0.0};
    if (!(dr_tol > 0.0) || !(r_lo >= 0.0) || !(lodr > 0.0)) return s;
    const double width = dr_tol * (1.0 - 1e-6);
    s.bins = std::max(N / 2.0, (r_lo + trials * lodr) * (double)k0) / width + 2.0;
    if (s.bins < (double)(1 << 27)) s.inv = 1.0 / width;
    return s;
}

int cs_collapse_small_enqueue(CsCollapse *w, const CsRec *recs, const unsigned *count,
                              const int *err, unsigned cap, const CsChunk *chunks,
                              const int *slot_k, const int *slot_Hk, int nslot, long long total,
                              double r_lo, double lodr, double N, double T, double threshold,
                              int remove, double dr_tol, int harm_remove, int numharm,
                              double harm_tol, cudaStream_t st)
{
    if (!w || nslot < 1 || nslot > CS_MAX_SLOT || total < 1) return -1;
    if ((unsigned long long)total * (unsigned long long)nslot >= 0xFFFFFFFFull) return 1;
    cl::SmallArgs a;
    memset(&a, 0, sizeof(a));
    a.recs = recs;
    a.count = count;
    a.err = err;
    a.cap = cap;
    a.chunks = chunks;
    for (int s = 0; s < nslot; s++) { a.si.k[s] = slot_k[s]; a.si.Hk[s] = slot_Hk[s]; }
    a.nslot = nslot;
    a.total = (uint32_t)total;
    a.end_bit = bit_length_u64((uint64_t)total * (uint64_t)nslot);
    a.r_lo = r_lo;
    a.lodr = lodr;
    a.nyq = N / 2.0;
    a.T = T;
    a.thr = threshold;
    a.remove = remove;
    a.harm_remove = harm_remove;
    a.numharm = numharm;
    a.drtol = dr_tol;
    a.tol = harm_tol;
    a.inv = remove ? bin_scale(r_lo, lodr, (double)total, slot_k[0], N, dr_tol).inv : -1.0;
    a.out = w->s_out;
    a.status = w->s_status;
    w->s_status[3] = 0;
    cudaError_t e = finish_prepare();
    if (e == cudaSuccess) {
        cl::collapse_small<<<1, cl::FT, sizeof(cl::SmallSmem), st>>>(a);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        fprintf(stderr, "Error: candidate collapse on the GPU: %s\n", cudaGetErrorString(e));
        return -1;
    }
    w->small = true;
    return 0;
}

unsigned cs_collapse_small_cap(void)
{
    return cl::CAP;
}

int cs_collapse_small_status(const CsCollapse *w, unsigned *n, int *err)
{
    *n = w->s_status[0];
    *err = (int)w->s_status[1];
    return w->s_status[3] ? 1 : 0;
}

/* The bins of a list, all ones, on the stream; false when the sort is the way.
 * A bin is 20 bytes to clear and to read, a record about 100 in the sort's passes
 * and its list some 20 launches.  Sort against bins, with both waits: 5 k records
 * in 0.1, 0.5 and 4.2 M bins 156:78, 166:96 and 194:147 us, 80 k records in the
 * same 267:105, 345:222 and 662:564.  The ends would meet near 2 k bins a record;
 * BINS_MOST bounds the memory (336 MB). */
static bool bins_for(CsCollapse *w, unsigned n, long long nchunks, const cl::SlotInfo &si,
                     int nprof, double r_lo, double lodr, double N, double dr_tol, cudaStream_t st,
                     cl::Bins &bn)
{
    const BinScale sc = bin_scale(r_lo, lodr, (double)nchunks * (double)nprof, si.k[0], N, dr_tol);
    const unsigned long long most =
        std::min((unsigned long long)n * cl::BINS_PER_REC, cl::BINS_MOST);
    if (!(sc.inv >= 0.0) || !(sc.bins < (double)most)) return false;
    bn.nb = (unsigned)sc.bins;
    bn.inv = sc.inv;
    const size_t pad = ((size_t)bn.nb + cl::BT - 1) / cl::BT * cl::BT, blocks = pad / cl::BT;
    const size_t ones = ((size_t)n + 2 * (size_t)bn.nb) * sizeof(uint64_t) + (size_t)bn.nb * 4;
    const size_t bytes = ones + pad / 8 + blocks * 4;
    if (bytes > w->bins_bytes) {
        cudaFree(w->bins);
        w->bins = nullptr;
        w->bins_bytes = 0;
        const size_t c = bytes + (size_t)n * 2;     /* room for a quarter more records */
        if (cudaMalloc(&w->bins, c) != cudaSuccess) {
            cudaGetLastError();
            w->bins = nullptr;
            return false;
        }
        w->bins_bytes = c;
    }
    bn.best = (unsigned long long *)w->bins;
    bn.lo = bn.best + n;
    bn.nhi = bn.lo + bn.nb;
    bn.idx = (unsigned *)(bn.nhi + bn.nb);
    bn.starts = bn.idx + bn.nb;
    bn.cnt = bn.starts + pad / 32;
    return cudaMemsetAsync(w->bins, 0xFF, ones, st) == cudaSuccess;
}

/* keep[] of a list of up to n candidates, any length: the radix sort by metric,
 * then the walk.  (Ranked by counting in one CTA, a list of
 * 53 k records took 243 ms in all and one of 200 k 3.0 s; so 41 and 179 ms.) */
static cudaError_t order_and_walk(CsCollapse *w, const unsigned *list, unsigned n, int numharm,
                                  double tol, cudaStream_t st)
{
    const unsigned *m = w->counters + 1;
    cub::DoubleBuffer<float> mb(w->mkey[0], w->mkey[1]);
    cub::DoubleBuffer<unsigned> pb(w->mpos[0], w->mpos[1]);
    size_t tb = w->temp_bytes;
    cl::metric_keys_kernel<<<(n + cl::NT - 1) / cl::NT, cl::NT, 0, st>>>(list, w->metric, n, m,
                                                                        w->mkey[0], w->mpos[0]);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess)
        e = cub::DeviceRadixSort::SortPairsDescending(w->temp, tb, mb, pb, (int)n, 0, 32, st);
    if (e == cudaSuccess) {
        cl::walk_kernel<<<1, cl::FT, cl::WALK_BYTES, st>>>(list, pb.Current(), w->r, m, numharm, tol,
                                                           w->removed, w->keep);
        e = cudaGetLastError();
    }
    return e;
}

int cs_collapse_enqueue(CsCollapse *w, const CsRec *recs, unsigned n, const CsChunk *chunks,
                        long long nchunks, const int *slot_k, const int *slot_Hk, int nslot,
                        int nprof, double r_lo, double lodr, double N, double T,
                        double threshold, int remove, double dr_tol, int harm_remove,
                        int numharm, double harm_tol, cudaStream_t st)
{
    if (!w || nslot < 1 || nslot > CS_MAX_SLOT || nprof < 1 || nchunks < 1) return -1;
    w->pending_n = n;
    w->small = false;
    if (n == 0) return 0;
    cl::SlotInfo si;
    memset(&si, 0, sizeof(si));
    for (int s = 0; s < nslot; s++) { si.k[s] = slot_k[s]; si.Hk[s] = slot_Hk[s]; }
    const unsigned g = (n + cl::NT - 1) / cl::NT;
    cudaError_t e = collapse_reserve(w, n);       /* allocates the counters on first use */
    if (e == cudaSuccess && !w->counters) e = cudaErrorMemoryAllocation;
    if (e == cudaSuccess) e = finish_prepare();
    if (e != cudaSuccess) {
        fprintf(stderr, "Error: candidate collapse on the GPU: %s\n", cudaGetErrorString(e));
        return -1;
    }
    unsigned *nv = w->counters, *m = w->counters + 1;
    cl::Bins bn;
    unsigned *list = w->list;
    const bool binned = remove && bins_for(w, n, nchunks, si, nprof, r_lo, lodr, N, dr_tol, st, bn);
    if (binned) {
        const cl::RecGeo geo = {recs, chunks, si, nslot, nprof, r_lo, lodr, N / 2.0, T, threshold};
        const unsigned gb = (bn.nb + cl::BT - 1) / cl::BT;
        cl::bin_kernel<<<g, cl::NT, 0, st>>>(geo, n, bn, w->r, w->freq, w->metric, w->nharm);
        cl::bin_starts_kernel<<<gb, cl::BT, 0, st>>>(bn, dr_tol);
        cl::bin_offer_kernel<<<gb, cl::BT, 0, st>>>(bn, recs, m);
        e = cudaGetLastError();
    } else {
        const int end_bit =
            bit_length_u64((uint64_t)nchunks * (uint64_t)nslot * (uint64_t)nprof);
        e = cudaMemsetAsync(w->counters, 0, (4 + 2 * CS_MAX_SLOT) * sizeof(unsigned), st);
        unsigned *slot_cnt = w->counters + 4, *slot_start = w->counters + 4 + CS_MAX_SLOT;
        if (e == cudaSuccess) {
            cl::harvest_kernel<<<g, cl::NT, 0, st>>>(recs, n, chunks, nchunks, si, nslot, nprof,
                                                     r_lo, lodr, N / 2.0, T, threshold, w->key[0],
                                                     w->bkey, w->slot_of, w->idx[0], w->r, w->freq,
                                                     w->metric, w->nharm, nv, slot_cnt);
            e = cudaGetLastError();
        }
        /* every slot's records in trial order; invalid records (all-ones key) last */
        cub::DoubleBuffer<uint64_t> kb(w->key[0], w->key[1]);
        cub::DoubleBuffer<unsigned> ib(w->idx[0], w->idx[1]);
        size_t tb = w->temp_bytes;
        if (e == cudaSuccess)
            e = cub::DeviceRadixSort::SortPairs(w->temp, tb, kb, ib, (int)n, 0, end_bit, st);
        /* merged into stable r order (remove) or stable frequency order */
        if (e == cudaSuccess) {
            cl::slot_starts_kernel<<<1, 1, 0, st>>>(slot_cnt, nslot, slot_start);
            cl::merge_kernel<<<g, cl::NT, 0, st>>>(ib.Current(), nv, w->slot_of, w->bkey,
                                                   remove ? w->r : w->freq, slot_start, slot_cnt,
                                                   nslot, w->merged);
            e = cudaGetLastError();
        }
        if (remove) {
            if (e == cudaSuccess) {
                cl::run_flags_kernel<<<g, cl::NT, 0, st>>>(w->merged, w->r, n, nv, dr_tol, w->flag);
                e = cudaGetLastError();
            }
            if (e == cudaSuccess) {
                tb = w->temp_bytes;
                e = cub::DeviceScan::ExclusiveSum(w->temp, tb, w->flag, w->runid, (int)n, st);
            }
            /* the key buffers are free once the merge has run: best-of-run slots */
            unsigned long long *best = reinterpret_cast<unsigned long long *>(w->key[0]);
            if (e == cudaSuccess) e = cudaMemsetAsync(best, 0, (size_t)n * sizeof(uint64_t), st);
            if (e == cudaSuccess) {
                cl::count_runs_kernel<<<1, 1, 0, st>>>(w->flag, w->runid, n, m);
                cl::run_offer_kernel<<<g, cl::NT, 0, st>>>(w->merged, w->metric, w->flag, w->runid,
                                                           nv, best);
                cl::run_take_kernel<<<g, cl::NT, 0, st>>>(w->merged, best, n, m, w->list);
                e = cudaGetLastError();
            }
        } else {
            if (e == cudaSuccess) {
                cl::copy_count_kernel<<<1, 1, 0, st>>>(nv, m);
                e = cudaGetLastError();
            }
            list = w->merged;
        }
    }
    w->pending_list = list;
    w->numharm = numharm;
    w->harm_tol = harm_tol;
    if (e == cudaSuccess) e = cudaGetDevice(&w->device);
    /* with every record in the list it is too long for finish_kernel; after
     * remove_duplicates it seldom is, and cs_collapse_finish sees to that */
    const bool all = harm_remove && !remove && n > cl::CAP;
    if (e == cudaSuccess && all) e = order_and_walk(w, list, n, numharm, harm_tol, st);
    if (e == cudaSuccess) {
        cl::finish_kernel<<<1, cl::FT, sizeof(cl::FinishSmem), st>>>(
            list, binned ? bn.best : nullptr, binned ? bn.idx : nullptr, m, harm_remove, numharm,
            harm_tol, w->r, w->freq, w->metric, w->nharm, all ? w->keep : nullptr, w->out, w->s_out,
            w->h_counters);
        e = cudaGetLastError();
    }
    if (e != cudaSuccess) {
        fprintf(stderr, "Error: candidate collapse on the GPU: %s\n", cudaGetErrorString(e));
        return -1;
    }
    return 0;
}

int cs_collapse_finish(CsCollapse *w, cudaStream_t st, CandidateList *out)
{
    candlist_init(out);
    if (!w) return -1;
    if (!w->small && w->pending_n == 0) return 0;
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) goto fail;
    if (w->small) {
        const unsigned nout = w->s_status[2];
        w->small = false;
        if (nout) {
            out->v = (Candidate *)malloc((size_t)nout * sizeof(Candidate));
            if (!out->v) return -1;
            memcpy(out->v, w->s_out, (size_t)nout * sizeof(Candidate));
            out->n = nout;
            out->cap = nout;
        }
        return 0;
    }
    if (w->h_counters[1]) {
        int here = w->device;                   /* the waiting thread may be on another */
        e = cudaGetDevice(&here);
        if (e == cudaSuccess) e = cudaSetDevice(w->device);
        if (e == cudaSuccess)
            e = order_and_walk(w, w->pending_list, w->h_counters[1], w->numharm, w->harm_tol, st);
        if (e == cudaSuccess) {
            cl::finish_kernel<<<1, cl::FT, sizeof(cl::FinishSmem), st>>>(
                w->pending_list, nullptr, nullptr, w->counters + 1, 1, w->numharm, w->harm_tol, w->r,
                w->freq, w->metric, w->nharm, w->keep, w->out, w->s_out, w->h_counters);
            e = cudaGetLastError();
        }
        if (e == cudaSuccess) e = cudaStreamSynchronize(st);
        if (here != w->device) cudaSetDevice(here);
        if (e != cudaSuccess) goto fail;
    }
    {
        const unsigned nout = w->h_counters[0];
        const bool pinned = nout <= cl::CAP;
        if (!pinned && nout > w->h_out_cap) {
            if (w->h_out) cudaFreeHost(w->h_out);
            w->h_out = nullptr;
            w->h_out_cap = 0;
            e = cudaMallocHost((void **)&w->h_out,
                               (size_t)(nout + nout / 4 + 256) * sizeof(Candidate));
            if (e != cudaSuccess) goto fail;
            w->h_out_cap = nout + nout / 4 + 256;
        }
        if (!pinned) {
            e = cudaMemcpyAsync(w->h_out, w->out, (size_t)nout * sizeof(Candidate),
                                cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            if (e != cudaSuccess) goto fail;
        }
        if (nout) {
            out->v = (Candidate *)malloc((size_t)nout * sizeof(Candidate));
            if (!out->v) return -1;
            memcpy(out->v, pinned ? w->s_out : w->h_out, (size_t)nout * sizeof(Candidate));
            out->n = nout;
            out->cap = nout;
        }
    }
    w->pending_n = 0;
    return 0;
fail:
    fprintf(stderr, "Error: candidate collapse on the GPU: %s\n", cudaGetErrorString(e));
    return -1;
}
