/*
 * The decisions of prepsubband's time-domain clipping on the GPU: which
 * spectra PRESTO's clip_times (third_party/presto/src/clipping.c:47-230)
 * replaces when the reference runs its front end with -clip clip_sigma (its
 * default is 6).  clip_times runs on every raw block of L spectra in read
 * order (backend_common.c:976-986), with running statistics carried from
 * block to block:
 *
 *   zero-DM series   the sum of each spectrum over all channels (exact for
 *                    8-bit data: an integer below 2^24 as a float);
 *   block stats      avg_var (misc_utils.c:641-676, AS 52 recurrence in
 *                    double) and the lower median (median.c, element
 *                    (L-1)/2 of the sorted block); the "good" samples lie
 *                    strictly inside median -+ 3 sigma (float cut-offs), and
 *                    their avg_var gives the block's mean and sigma (the
 *                    running values stand in when no sample is good);
 *   running values   floats: mean and sigma of the first block, then
 *                    0.9 * old + 0.1 * new, evaluated in double;
 *   decision         spectrum t is replaced when
 *                    |zdm[t] - running_mean| > clip_sigma * running_sigma
 *                    (the difference in float, the test in double).
 *
 *   replacement      a replaced spectrum takes the block's channel levels:
 *                    per channel the sum over the block's good spectra (an
 *                    integer, exact) over their number, in double, then the
 *                    running level, a float: the first block's value, then
 *                    0.9 * old + 0.1 * new in double (clipping.c:118-160);
 *                    a block without good spectra keeps the old level.
 *
 * cs_clip_count gives the number of replaced spectra (and optionally the
 * flags); cs_clip_levels adds the levels, which the clipped dedispersion
 * (cs_dedisp_run_device_clipped) substitutes.  The arithmetic is the
 * reference's as its build compiles it (-ffp-contract=off, src/Makefile:43):
 * this file is built with -fmad=false.  Its -Ofast may still rewrite a
 * division by the good count as a reciprocal product; that changes the
 * double value by an ulp at most, below what the float level keeps.
 */
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>

#include "cs_b200.h"

#define CS_EXPORT extern "C" __attribute__((visibility("default")))

namespace ck {

constexpr int MAX_L = 8192;
constexpr int NT = 256;
constexpr int AV = 8;        /* samples read ahead of an avg_var chain */

/* zero-DM sum of each spectrum: one warp per spectrum */
__global__ void zdm_kernel(const uint8_t *raw, long long nspec, int nchan, int vec16, int *zdm)
{
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (t >= nspec) return;
    const uint8_t *row = raw + t * (long long)nchan;
    unsigned s = 0;
    if (vec16) {
        const uint4 *r4 = reinterpret_cast<const uint4 *>(row);
        for (int i = lane; i < nchan / 16; i += 32) {
            const uint4 w = __ldg(r4 + i);
            s = __dp4a(w.x, 0x01010101u, s);
            s = __dp4a(w.y, 0x01010101u, s);
            s = __dp4a(w.z, 0x01010101u, s);
            s = __dp4a(w.w, 0x01010101u, s);
        }
    } else {
        for (int c = lane; c < nchan; c += 32) s += row[c];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) zdm[t] = (int)s;
}

/* One pass over the raw data (nchan a multiple of 16 up to 512 * K, 16-byte
 * aligned): the zero-DM sum of each spectrum and, per block, the sum of every
 * channel column over ALL its spectra (fix_cols_kernel takes the spectra that
 * are not good out again; integers, so the order does not matter).  CTA =
 * CR consecutive spectra of one block, a warp per spectrum at a time; a lane
 * keeps its columns' byte sums in 16-bit halves (at most CR / 8 spectra a
 * warp, so they cannot carry).  Bound by the read of raw, once: reading it a
 * second time for the columns cost 400 us beside the 47 us the bytes take (300 k
 * spectra of 1024 channels).  Measured there: 83 us for both sums, and 24 us
 * for fix_cols_kernel. */
constexpr int CR = 240;
template <int K>
__global__ void __launch_bounds__(NT) zdm_cols_kernel(const uint8_t *raw, int L, int nchan,
                                                      int *zdm, unsigned *cols)
{
    extern __shared__ unsigned csum[];                 /* [nchan] */
    const long long b = blockIdx.x;
    const int r0 = blockIdx.y * CR, r1 = min(L, r0 + CR);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = nchan >> 4;                          /* 16-byte groups a row */
    for (int c = threadIdx.x; c < nchan; c += NT) csum[c] = 0;
    __syncthreads();
    unsigned ev[K][4], od[K][4];                       /* even and odd bytes' sums */
#pragma unroll
    for (int k = 0; k < K; k++)
#pragma unroll
        for (int q = 0; q < 4; q++) ev[k][q] = od[k][q] = 0;
    const uint4 *rows = reinterpret_cast<const uint4 *>(raw + b * L * (long long)nchan);
    constexpr int U = K <= 2 ? 4 : 1;                  /* spectra in flight a warp */
    for (int r = r0 + warp * U; r < r1; r += (NT / 32) * U) {
        uint4 v[U][K];
#pragma unroll
        for (int u = 0; u < U; u++)
#pragma unroll
            for (int k = 0; k < K; k++)
                v[u][k] = r + u < r1 && lane + 32 * k < G
                              ? __ldg(rows + (long long)(r + u) * G + lane + 32 * k)
                              : make_uint4(0, 0, 0, 0);
#pragma unroll
        for (int u = 0; u < U; u++) {
            unsigned s = 0;
#pragma unroll
            for (int k = 0; k < K; k++) {
                const unsigned w[4] = {v[u][k].x, v[u][k].y, v[u][k].z, v[u][k].w};
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    s = __dp4a(w[q], 0x01010101u, s);
                    ev[k][q] += w[q] & 0x00ff00ffu;
                    od[k][q] += (w[q] >> 8) & 0x00ff00ffu;
                }
            }
            s = __reduce_add_sync(0xffffffffu, s);
            if (lane == 0 && r + u < r1) zdm[b * L + r + u] = (int)s;
        }
    }
#pragma unroll
    for (int k = 0; k < K; k++)
        if (lane + 32 * k < G) {
            unsigned *c = csum + 16 * (lane + 32 * k);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                atomicAdd(c + 4 * q, ev[k][q] & 0xffffu);
                atomicAdd(c + 4 * q + 1, od[k][q] & 0xffffu);
                atomicAdd(c + 4 * q + 2, ev[k][q] >> 16);
                atomicAdd(c + 4 * q + 3, od[k][q] >> 16);
            }
        }
    __syncthreads();
    for (int c = threadIdx.x; c < nchan; c += NT) atomicAdd(cols + b * nchan + c, csum[c]);
}

/* stats_kernel's dynamic shared memory: reciprocals, samples, good samples */
static size_t stats_smem(int L)
{
    return (size_t)(L + 2) * sizeof(double) + 2 * (size_t)L * sizeof(int);
}

struct BlockStats {
    int ngood;
    float lo, hi;            /* good samples lie strictly between */
    double mean, sigma;      /* of the good samples */
};

/* avg_var (misc_utils.c:641-676) over n floats, in order: mean and variance.
 * Its update is one chain of dependent FP64 operations a sample,
 *     dx = (x - mean) / an;  var += an * (an - 1) * dx * dx;  mean += dx,
 * and the division is most of it.  Here dx comes from the correctly rounded
 * reciprocal rcp[an] by one residual correction (P. Markstein, IBM J. Res.
 * Dev. 34, 1990): q = d * r, dx = q + (d - q * an) * r with fused operations.
 * That is the correctly rounded quotient: the residual is exact, the
 * corrected value is within 2^-50 ulp of d / an before its rounding, and d /
 * an cannot be that near a rounding boundary without lying on a float, since
 * an has at most 14 bits (a 54-bit midpoint times an differs from d by at
 * least half a unit, so by 2^-15 ulp in the quotient).  Five dependent
 * operations a sample instead of a division's dozen and more. */
static __device__ void avg_var(const int *x, int n, const double *rcp, double &mean_out,
                               double &var_out)
{
    double mean = 0.0, acc = 0.0;
    if (n > 0) mean = (double)(float)x[0];
    double an = 1.0;
    auto push = [&](float xf, double r) {
        const double an1 = an;
        an += 1.0;
        const double d = (double)xf - mean;
        const double q = d * r;
        const double dx = __fma_rn(__fma_rn(-q, an, d), r, q);
        acc += an * an1 * dx * dx;
        mean += dx;
    };
    int i = 1;
    for (; i + AV <= n; i += AV) {
        float v[AV];
        double r[AV];
#pragma unroll
        for (int k = 0; k < AV; k++) {
            v[k] = (float)x[i + k];
            r[k] = rcp[i + k + 1];
        }
#pragma unroll
        for (int k = 0; k < AV; k++) push(v[k], r[k]);
    }
    for (; i < n; i++) push((float)x[i], rcp[i + 1]);
    mean_out = mean;
    var_out = n > 1 ? acc / (double)(n - 1) : acc;
}

/* One CTA per block of L spectra: the lower median, then avg_var over all
 * samples and over the good ones.
 *
 * The two avg_var chains bound it (L dependent steps each), and the second
 * needs the first one's sigma only through the float cut-offs lo and hi.  So
 * sigma is first taken from a parallel two-pass sum, whose cut-offs are the
 * chain's unless they straddle a rounding of the last bit; warps 0 and 1 then
 * run the two chains side by side, and where the exact cut-offs turn out
 * different the second chain is run again from them.
 *
 * The median is the (L-1)/2-th smallest of integers: found bit by bit from
 * the top over the shared samples (count the values below a trial prefix),
 * nbits passes of L / NT comparisons a thread.
 *
 * Measured for 125 blocks of 2400: 110 us, against 262 us for a bitonic
 * sort and 1201 us for the two chains with divisions, one thread a block. */
__global__ void __launch_bounds__(NT) stats_kernel(const int *zdm, int L, int nbits,
                                                   BlockStats *out)
{
    extern __shared__ double dsm[];
    double *rcp = dsm;                                  /* [L + 2] */
    int *x = reinterpret_cast<int *>(rcp + L + 2);      /* [L] all samples */
    int *good = x + L;                                  /* [L] good ones, in order */
    __shared__ double red[NT / 32];
    __shared__ int cnt[2][NT / 32];
    __shared__ double s_var, s_gmean, s_gvar;
    const long long b = blockIdx.x;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    for (int i = tid; i < L + 2; i += NT) rcp[i] = i ? 1.0 / (double)i : 0.0;
    double s = 0.0;
    for (int i = tid; i < L; i += NT) {
        const int v = zdm[b * L + i];
        x[i] = v;
        s += (double)(float)v;
    }
    auto block_sum = [&](double v) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        __syncthreads();
        if (lane == 0) red[warp] = v;
        __syncthreads();
        double t = 0.0;
        for (int w = 0; w < NT / 32; w++) t += red[w];
        return t;
    };
    const double mean0 = block_sum(s) / (double)L;
    s = 0.0;
    for (int i = tid; i < L; i += NT) {
        const double d = (double)(float)x[i] - mean0;
        s += d * d;
    }
    const double var0 = block_sum(s) / (double)max(1, L - 1);

    int med = 0;
    const int rank = (L - 1) / 2;
    for (int bit = nbits - 1; bit >= 0; bit--) {
        const int trial = med | (1 << bit);
        int c = 0;
        for (int i = tid; i < L; i += NT) c += x[i] < trial ? 1 : 0;
        c = __reduce_add_sync(0xffffffffu, c);
        int *cb = cnt[bit & 1];
        if (lane == 0) cb[warp] = c;
        __syncthreads();
        int below = 0;
        for (int w = 0; w < NT / 32; w++) below += cb[w];
        if (below <= rank) med |= 1 << bit;
    }

    /* the good samples for cut-offs from variance v, in order; their number */
    auto select = [&](double v, float &lo, float &hi) {
        const double sd = sqrt(v);
        lo = (float)((double)(float)med - 3.0 * sd);
        hi = (float)((double)(float)med + 3.0 * sd);
        int base = 0;
        for (int i0 = 0; i0 < L; i0 += NT) {
            const int i = i0 + tid;
            const bool g = i < L && (float)x[i] > lo && (float)x[i] < hi;
            const unsigned m = __ballot_sync(0xffffffffu, g);
            __syncthreads();
            if (lane == 0) cnt[0][warp] = __popc(m);
            __syncthreads();
            int before = base;
            for (int w = 0; w < NT / 32; w++) {
                const int c = cnt[0][w];
                if (w < warp) before += c;
                base += c;
            }
            if (g) good[before + __popc(m & ((1u << lane) - 1u))] = x[i];
        }
        __syncthreads();
        return base;
    };
    float lo, hi, elo, ehi;
    int ng = select(var0, lo, hi);
    if (tid == 0) {
        double m;
        avg_var(x, L, rcp, m, s_var);
    } else if (tid == 32) {
        avg_var(good, ng, rcp, s_gmean, s_gvar);
    }
    __syncthreads();
    const double sd = sqrt(s_var);
    elo = (float)((double)(float)med - 3.0 * sd);
    ehi = (float)((double)(float)med + 3.0 * sd);
    if (elo != lo || ehi != hi) {                       /* uniform over the CTA */
        ng = select(s_var, lo, hi);
        if (tid == 0) avg_var(good, ng, rcp, s_gmean, s_gvar);
        __syncthreads();
    }
    if (tid == 0) {
        BlockStats o;
        o.ngood = ng;
        o.lo = lo;
        o.hi = hi;
        o.mean = ng ? s_gmean : 0.0;
        o.sigma = ng ? sqrt(s_gvar) : 0.0;
        out[b] = o;
    }
}

__global__ void decide_kernel(const int *zdm, long long n, int L, const float *ravg,
                              const float *trig, unsigned long long *count, uint8_t *flags)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const long long b = t / L;
    const float d = (float)zdm[t] - ravg[b];
    const bool clip = fabs((double)d) > (double)trig[b];
    if (flags) flags[t] = clip ? 1 : 0;
    if (clip) atomicAdd(count, 1ull);
}

/* per (block, channel column): the sum of the column over the block's good
 * spectra (any channel count and alignment) */
__global__ void chan_sum_kernel(const uint8_t *raw, int L, int nchan, const int *zdm,
                                const BlockStats *st, unsigned *sums)
{
    const long long b = blockIdx.x;
    const int c = blockIdx.y * blockDim.x + threadIdx.x;
    if (c >= nchan) return;
    const float lo = st[b].lo, hi = st[b].hi;
    const uint8_t *col = raw + b * L * (long long)nchan + c;
    unsigned s = 0;
    for (int i = 0; i < L; i++) {
        const float v = (float)zdm[b * L + i];
        if (v > lo && v < hi) s += __ldg(col + (long long)i * nchan);
    }
    sums[b * nchan + c] = s;
}

/* zdm_cols_kernel's column sums without the spectra that are not good: they
 * are few (the tails past 3 sigma), so only their rows are read again.  A CTA
 * looks through NT spectra of one block and adds up the rows it found. */
__global__ void __launch_bounds__(NT) fix_cols_kernel(const uint8_t *raw, int L, int nchan,
                                                      const int *zdm, const BlockStats *st,
                                                      unsigned *sums)
{
    __shared__ int bad[NT];
    __shared__ int nbad;
    const long long b = blockIdx.x;
    if (threadIdx.x == 0) nbad = 0;
    __syncthreads();
    const int i = blockIdx.y * NT + threadIdx.x;
    if (i < L) {
        const float v = (float)zdm[b * L + i];
        if (!(v > st[b].lo && v < st[b].hi)) bad[atomicAdd(&nbad, 1)] = i;
    }
    __syncthreads();
    const int n = nbad;
    if (n == 0) return;
    const uint8_t *rows = raw + b * L * (long long)nchan;
    for (int c = 4 * threadIdx.x; c < nchan; c += 4 * NT) {
        unsigned s[4] = {0, 0, 0, 0};
#pragma unroll 4
        for (int k = 0; k < n; k++) {
            const uchar4 v = __ldg(reinterpret_cast<const uchar4 *>(rows + bad[k] * (long long)nchan + c));
            s[0] += v.x;
            s[1] += v.y;
            s[2] += v.z;
            s[3] += v.w;
        }
#pragma unroll
        for (int q = 0; q < 4; q++) atomicSub(sums + b * nchan + c + q, s[q]);
    }
}

/* The chains from block to block, side by side: CTA 0's first lane has the
 * running mean and sigma of the zero-DM sums; lane c of the others the running
 * level of channel column c, in place over its integer sums (below 2^24, exact
 * as floats), with the next CB blocks' sums already on their way.  CTAs of one
 * warp, so that the columns' chains spread over the SMs.  Bound by the chains'
 * latency; apart, with eight blocks read at a time, the two took 40 us for 125
 * blocks of 1024 columns, together 29 us. */
constexpr int CB = 16;
__global__ void __launch_bounds__(32) chains_kernel(const BlockStats *st, long long nblocks,
                                                    float clip_sigma, float *ravg, float *trig,
                                                    int nchan, float *lv)
{
    if (blockIdx.x == 0) {
        __shared__ BlockStats sb[32];
        const int lane = threadIdx.x;
        float running_avg = 0.0f, running_std = 0.0f;
        for (long long b0 = 0; b0 < nblocks; b0 += 32) {
            __syncwarp();
            if (b0 + lane < nblocks) sb[lane] = st[b0 + lane];
            __syncwarp();
            if (lane != 0) continue;
            const int n = (int)min(32ll, nblocks - b0);
            for (int k = 0; k < n; k++) {
                double cur_avg, cur_std;
                if (sb[k].ngood < 1) {
                    cur_avg = (double)running_avg;
                    cur_std = (double)running_std;
                } else {
                    cur_avg = sb[k].mean;
                    cur_std = sb[k].sigma;
                }
                if (b0 + k) {
                    running_avg = (float)(0.9 * (double)running_avg + 0.1 * cur_avg);
                    running_std = (float)(0.9 * (double)running_std + 0.1 * cur_std);
                } else {
                    running_avg = (float)cur_avg;
                    running_std = (float)cur_std;
                }
                ravg[b0 + k] = running_avg;
                trig[b0 + k] = clip_sigma * running_std;
            }
        }
        return;
    }
    const int c = (blockIdx.x - 1) * 32 + threadIdx.x;
    if (c >= nchan) return;
    float run = 0.0f;
    int ng[CB], ngn[CB];
    unsigned sum[CB], sumn[CB];
    auto fetch = [&](long long b0) {
#pragma unroll
        for (int k = 0; k < CB; k++) {
            ngn[k] = 0;
            sumn[k] = 0;
            if (b0 + k < nblocks) {
                ngn[k] = st[b0 + k].ngood;
                sumn[k] = __float_as_uint(lv[(b0 + k) * nchan + c]);
            }
        }
    };
    fetch(0);
    for (long long b0 = 0; b0 < nblocks; b0 += CB) {
#pragma unroll
        for (int k = 0; k < CB; k++) {
            ng[k] = ngn[k];
            sum[k] = sumn[k];
        }
        fetch(b0 + CB);
        double mean[CB];                /* off the running chain */
#pragma unroll
        for (int k = 0; k < CB; k++)
            mean[k] = ng[k] >= 1 ? (double)(float)sum[k] / (double)ng[k] : 0.0;
#pragma unroll
        for (int k = 0; k < CB; k++) {
            const long long b = b0 + k;
            if (b >= nblocks) break;
            const double cur = ng[k] >= 1 ? mean[k] : (double)run;
            run = b ? (float)(0.9 * (double)run + 0.1 * cur) : (float)cur;
            lv[b * nchan + c] = run;
        }
    }
}

}  // namespace ck

/* scratch layout: zero-DM sums, block statistics, running values, count */
static size_t clip_layout(long long nspec, int L, size_t off[5])
{
    const long long nblocks = nspec / L, n = nblocks * L;
    size_t o = 0;
    auto take = [&](size_t bytes) { const size_t at = o; o = (o + bytes + 255) & ~(size_t)255; return at; };
    off[0] = take((size_t)n * sizeof(int));
    off[1] = take((size_t)nblocks * sizeof(ck::BlockStats));
    off[2] = take((size_t)nblocks * sizeof(float));
    off[3] = take((size_t)nblocks * sizeof(float));
    off[4] = take(sizeof(unsigned long long));
    return o;
}

CS_EXPORT size_t cs_clip_scratch_bytes(long long nspec, int L)
{
    if (nspec < 0 || L < 1) return 0;
    size_t off[5];
    return clip_layout(nspec, L, off);
}

static int clip_run(const uint8_t *d_raw, long long nspec, int nchan, int L, float clip_sigma,
                    long long *nclipped, uint8_t *d_flags, float *d_levels, void *d_scratch,
                    size_t scratch_bytes, void *stream, int device, const char *who)
{
    if (!nclipped || nchan < 1 || L < 1 || L > ck::MAX_L || nspec < 0) return -1;
    *nclipped = 0;
    const long long nblocks = nspec / L;     /* a partial last block is never read */
    if (nblocks == 0 || !(clip_sigma > 0.0f)) return 0;
    if (!d_raw) return -1;
    if (cudaSetDevice(device) != cudaSuccess) return -1;
    cudaStream_t st = (cudaStream_t)stream;
    const long long n = nblocks * L;
    const size_t smem = ck::stats_smem(L);
    int nbits = 1;                           /* of a zero-DM sum */
    while (nbits < 31 && ((long long)nchan * 255) >> nbits) nbits++;
    size_t off[5];
    const size_t need = clip_layout(nspec, L, off);
    cudaError_t e = cudaSuccess;
    char *base = (char *)d_scratch;
    const bool own = d_scratch == nullptr;
    if (own) {
        e = cudaMalloc((void **)&base, need);
    } else if (scratch_bytes < need || ((uintptr_t)d_scratch & 255)) {
        fprintf(stderr, "Error: %s: scratch of %zu bytes (256-byte aligned) needed\n", who, need);
        return -1;
    }
    int *zdm = (int *)(base + off[0]);
    ck::BlockStats *bs = (ck::BlockStats *)(base + off[1]);
    float *ravg = (float *)(base + off[2]), *trig = (float *)(base + off[3]);
    unsigned long long *cnt = (unsigned long long *)(base + off[4]), hcnt = 0;
    if (e == cudaSuccess) e = cudaMemsetAsync(cnt, 0, sizeof(unsigned long long), st);
    /* the limit of 48 KB is for this and the kernel's own arrays together.  It is
     * raised to the longest block's need, never to this call's: a thread with other
     * blocks may launch between the two calls */
    if (e == cudaSuccess && smem > 32 * 1024)
        e = cudaFuncSetAttribute((const void *)ck::stats_kernel,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)ck::stats_smem(ck::MAX_L));
    if (e == cudaSuccess) {
        const int vec16 = (nchan % 16 == 0) && (((uintptr_t)d_raw & 15) == 0);
        /* one pass for both sums where the levels are wanted and a warp's
         * lanes can hold a row's columns */
        unsigned *cols = reinterpret_cast<unsigned *>(d_levels);
        const bool fused = d_levels && vec16 && nchan <= 4096;
        if (fused) {
            const dim3 g((unsigned)nblocks, (unsigned)((L + ck::CR - 1) / ck::CR));
            const size_t csm = (size_t)nchan * sizeof(unsigned);
            e = cudaMemsetAsync(cols, 0, (size_t)nblocks * nchan * sizeof(unsigned), st);
            if (nchan <= 512)
                ck::zdm_cols_kernel<1><<<g, ck::NT, csm, st>>>(d_raw, L, nchan, zdm, cols);
            else if (nchan <= 1024)
                ck::zdm_cols_kernel<2><<<g, ck::NT, csm, st>>>(d_raw, L, nchan, zdm, cols);
            else if (nchan <= 2048)
                ck::zdm_cols_kernel<4><<<g, ck::NT, csm, st>>>(d_raw, L, nchan, zdm, cols);
            else
                ck::zdm_cols_kernel<8><<<g, ck::NT, csm, st>>>(d_raw, L, nchan, zdm, cols);
        } else {
            const long long threads = n * 32;
            ck::zdm_kernel<<<(unsigned)((threads + ck::NT - 1) / ck::NT), ck::NT, 0, st>>>(
                d_raw, n, nchan, vec16, zdm);
        }
        ck::stats_kernel<<<(unsigned)nblocks, ck::NT, smem, st>>>(zdm, L, nbits, bs);
        if (d_levels) {
            if (fused) {
                const dim3 g((unsigned)nblocks, (unsigned)((L + ck::NT - 1) / ck::NT));
                ck::fix_cols_kernel<<<g, ck::NT, 0, st>>>(d_raw, L, nchan, zdm, bs, cols);
            } else {
                const dim3 g((unsigned)nblocks, (unsigned)((nchan + ck::NT - 1) / ck::NT));
                ck::chan_sum_kernel<<<g, ck::NT, 0, st>>>(d_raw, L, nchan, zdm, bs, cols);
            }
        }
        ck::chains_kernel<<<1 + (d_levels ? (nchan + 31) / 32 : 0), 32, 0, st>>>(
            bs, nblocks, clip_sigma, ravg, trig, nchan, d_levels);
        ck::decide_kernel<<<(unsigned)((n + ck::NT - 1) / ck::NT), ck::NT, 0, st>>>(
            zdm, n, L, ravg, trig, cnt, d_flags);
        if (e == cudaSuccess)
            e = cudaGetLastError();
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(&hcnt, cnt, sizeof(unsigned long long), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (own) cudaFree(base);
    if (e != cudaSuccess) {
        fprintf(stderr, "Error: %s: %s\n", who, cudaGetErrorString(e));
        return -1;
    }
    *nclipped = (long long)hcnt;
    return 0;
}

CS_EXPORT int cs_clip_count(const uint8_t *d_raw, long long nspec, int nchan, int L,
                            float clip_sigma, long long *nclipped, uint8_t *d_flags,
                            void *d_scratch, size_t scratch_bytes, void *stream, int device)
{
    return clip_run(d_raw, nspec, nchan, L, clip_sigma, nclipped, d_flags, nullptr, d_scratch,
                    scratch_bytes, stream, device, "cs_clip_count");
}

CS_EXPORT int cs_clip_levels(const uint8_t *d_raw, long long nspec, int nchan, int L,
                             float clip_sigma, long long *nclipped, uint8_t *d_flags,
                             float *d_levels, void *d_scratch, size_t scratch_bytes, void *stream,
                             int device)
{
    if (!d_flags || !d_levels) {
        if (nclipped) *nclipped = 0;
        return -1;
    }
    return clip_run(d_raw, nspec, nchan, L, clip_sigma, nclipped, d_flags, d_levels, d_scratch,
                    scratch_bytes, stream, device, "cs_clip_levels");
}
