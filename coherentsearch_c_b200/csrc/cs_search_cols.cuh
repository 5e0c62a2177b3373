/*
 * The search kernel of single spectra for the ladder configurations of
 * cs_search_ws.cuh (nharms 60, 32, 16), built around register blocks of the
 * interpolation.
 *
 * search_ws gives every lane one trial: per (trial, harmonic) 128 B of
 * window, 64 B of weights and 8 B of phase factor go through the load path
 * into its registers, and that path's 128 B a clock bound it (8.05 M trials,
 * nharms 60: 2.7 ms of 4.68).  Two things are shared between trials:
 *
 *   windows   harmonic h moves h * pnum / q bins a trial (at most half a bin
 *             at hidr 0.5), so consecutive trials see almost the same bins;
 *   weights   the trial grid has period q, so trials a multiple of q apart
 *             have the same fractional offsets, a whole number of bins on.
 *
 * A thread therefore takes 4 consecutive trials x 4 columns, D trials apart
 * (D a multiple of 2q and of 16): each bin read serves 4 trials, each weight 4
 * columns, about 70 B a (trial, harmonic) instead of 200.  The 4 trials share
 * one window of NT = 18 or 20 taps that starts at an even bin; their weight
 * rows are shifted inside it and padded with zeros, which leaves each chain
 * the reference's 16 fused multiply-adds in tap order (adding 0 * x between
 * them changes nothing for finite x).  A spectrum with a bin that is not finite
 * is left alone (NOT_FINITE): 0 times such a bin would spoil trials whose own 16
 * taps miss it.  (Skipping the padding in a second loop for such spectra cost
 * every other one 1.5 %: the host runs the kernel for any geometry instead.)
 *
 * Measured: 8.05 M trials at nharms 60 4.68 -> 2.31 ms, 1.0 M 0.70 -> 0.336, 3.0 M
 * at 32 0.474 -> 0.331, 1.1 M at 16 0.219 -> 0.142.  No unit is full (issue slots
 * 63 % busy, 70 % on the fullest scheduler; shared-memory path 47 %, FP32 44 %): at
 * nharms 60 a third of an interpolation warp's time goes into waits for boxes, 60
 * small ones a tile (8 rows of some 200 bytes, 175 cycles each as it runs; 8
 * stages or 10, 5 K steps or 6 are the same); at 32 and 16 the epilogue is as long.
 *
 *   tile      128 trials: 16 consecutive (a phase block) x 8 columns;
 *             row (k * 4 + j) * 8 + cg * 4 + g is trial 4g + k of the phase
 *             block in column 4cg + j, so that the lanes of a warp write an
 *             operand block to consecutive banks.
 *   CTA       persistent, a run of (phase block, column group) tiles, phase
 *             block slowest: its weights (nharms x NT x 16 floats) stay in
 *             shared memory.
 *   windows   a padded copy of the spectrum (pad_amax_kernel); per (tile,
 *             harmonic) one TMA box of 8 rows (the columns, a fixed number of
 *             bins apart) into a ring of stages, four harmonics a stage.
 *   warps     8 (nharms 16: 4) interpolate (a stage each in turn: 4 harmonics x
 *             8 threads) into a shared-memory ring of A operand K steps; 8 run
 *             the boxcar epilogue from tensor memory; 2 issue the TMA boxes; one
 *             finds each row's chunk; one copies each K step (8 harmonics) to
 *             tensor memory on arrival and issues the MMAs.
 *
 * Every wait is bounded; one that gives up sets the session's error flag and
 * a CTA-wide one that the other roles see, copies and MMAs in flight are
 * waited for and tensor memory is freed.
 */
#pragma once

namespace cols {

using wsk::Args;
using wsk::TMEM_COLS;

constexpr int NEPI = 8;                       /* epilogue warps */
constexpr int NTMA = 2;                       /* warps that issue the boxes */
/* The warps of a configuration: interpolation, epilogue, boxes, rows, MMA.  One
 * interpolation warp a scheduler waits for its own loads, rotations and stores
 * (1 M trials at nharms 60: 361 us); two of them hide that (341), with registers
 * moved from the other roles: 640 x 96 are launched, 8 x 32 x 120 + 8 x 32 x 88 +
 * 4 x 32 x 64 are used, the same sum.  Four warps on the boxes would leave 112 and
 * 80: slower (364).  nharms 16 has 4 blocks a tile, one a warp. */
template <class C>
struct Roles {
    static constexpr int NINT = C::NH >= 32 ? 8 : 4;
    static constexpr int TMA = NINT + NEPI, ROW = TMA + NTMA, MMA = ROW + 1;
    static constexpr int NTHREADS = 32 * (MMA + 1);
};
constexpr int TI = 16, TC = 8;                /* consecutive trials, columns of a tile */
/* tensor memory: NACC accumulators, then NAB copies of a tile's A operand (hi:
 * K/2 columns, then lo) */
template <class C>
struct Tm {
    static constexpr int DS = C::NPAD <= 64 ? 64 : 128, AC = C::KPAD, A0 = 384;
    static constexpr int NACC = A0 / DS, NAB = 128 / AC < 4 ? 128 / AC : 4;
};
constexpr int MAX_ACC = 6;
constexpr int NROW = 4;                       /* row-info slots */
/* A operand K steps in the ring.  A warp's block before this one was at most 5
 * steps back, so its slot's use two back is complete: a parity needs that. */
constexpr int NA = 5;
constexpr int A_STEP = 2 * 2 * CS_TILE_M * 16;    /* bytes: hi and lo, two K blocks each */
constexpr int MAX_STG = 10;                   /* most window stages */
constexpr int MIN_STG = 4;                    /* fewest */
constexpr int FRONT = 16;                     /* zero bins before the padded copy */
constexpr int NOT_FINITE = 2;                 /* error flag: no tile was searched */

/* Per phase block, contiguous in global and shared memory:
 *   weights   per block hb of 4 harmonics, harmonic, tap: 16 floats (trials)
 *   gains     per harmonic 16 float2
 *   x0        per harmonic the bin of the padded copy where the box of column
 *             0 starts (even)
 *   goff      per harmonic, a byte each: where group g's window starts in the
 *             box, in 16-byte units */
struct Geo {
    int nh, nblk;                 /* harmonics, blocks of 4 */
    int npb, ncg;                 /* phase blocks, column groups */
    int ntiles;                   /* npb * ncg */
    int D;                        /* trials between columns */
    int total;                    /* trials */
    int nchunks;
    int nstg, stg_bytes;          /* window stages */
    int tab_bytes, g_off, x_off;  /* one phase block's table; its gains and x0 */
    int np[16];                   /* tap pairs of block hb (9 or 10) */
    int bw[16];                   /* box width of block hb, bins */
    int w_off[16];                /* byte offset of block hb's weights */
    int shift[64];                /* bins between columns, per harmonic */
};

struct XArgs {
    Geo g;
    const unsigned char *tab;     /* [npb][tab_bytes] */
    const void *maps;             /* CUtensorMap [nh] */
};

/* Shared memory: B hi | B lo | table | A ring | window stages | row info |
 * barriers */
struct Lay {
    int blo, tab, a, win, row, bar, total;
};

static __host__ __device__ inline Lay layout(const Geo &g, int npad, int kpad)
{
    Lay L;
    L.blo = npad * kpad * 2;
    L.tab = 2 * L.blo;
    L.a = (L.tab + g.tab_bytes + 127) / 128 * 128;
    L.win = L.a + NA * A_STEP;
    L.row = L.win + g.nstg * g.stg_bytes;
    L.bar = L.row + NROW * (CS_TILE_M * 12 + 16);
    L.total = L.bar + 512 + 16 * 16;
    return L;
}

/* Bounded wait without a back-off: try_wait itself suspends the warp, and a
 * sleep's wake-up would add to every hand-off of the rings.  Gives up after
 * CS_WAIT_NS, or when another role has given up (*stop). */
static __device__ __forceinline__ bool wait_bar(uint32_t bar, uint32_t parity,
                                                const volatile int *stop)
{
    if (mbar_try(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    for (int n = 1;; n++) {
        if (mbar_try(bar, parity)) return true;
        if ((n & 15) == 0 && (*stop || global_ns() - t0 > CS_WAIT_NS)) return false;
    }
}

/* The same for a count in shared memory to reach n. */
static __device__ __forceinline__ bool count_wait(const volatile int *count, int n,
                                                  const volatile int *stop)
{
    if (*count >= n) return true;
    const unsigned long long t0 = global_ns();
    for (int i = 1;; i++) {
        if (*count >= n) return true;
        if ((i & 15) == 0 && (*stop || global_ns() - t0 > CS_WAIT_NS)) return false;
    }
}

/* One lane of the warp, known to the compiler as one: what it issues takes its
 * operands from uniform registers without a loop over lanes. */
static __device__ __forceinline__ bool elect()
{
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

static __device__ __forceinline__ void expect_tx(uint32_t bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(bar), "r"(bytes) : "memory");
}

static __device__ __forceinline__ void tma_rows(uint32_t dst, const void *map, int x, uint32_t bar)
{
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3}], [%4];"
                 :: "r"(dst), "l"(map), "r"(x), "r"(0), "r"(bar) : "memory");
}

static __device__ __forceinline__ void bulk_in(uint32_t dst, const void *src, uint32_t bytes,
                                               uint32_t bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1], %2, [%3];"
                 :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

/* 128 rows x 16 bytes of shared memory (8-row groups of 128 bytes) into 4
 * columns of tensor memory; later MMAs of the thread see it. */
static __device__ __forceinline__ void tmem_copy16(uint32_t taddr, uint64_t sdesc)
{
    asm volatile("tcgen05.cp.cta_group::1.128x128b [%0], %1;" :: "r"(taddr), "l"(sdesc) : "memory");
}

/* The spectrum's largest |component| (cs_amax_kernel) and its copy behind
 * FRONT zero bins; the pads are cleared when the buffer is allocated. */
__global__ void __launch_bounds__(256) pad_amax_kernel(const float2 *__restrict__ amps, int namps,
                                                       float2 *__restrict__ pad,
                                                       unsigned *__restrict__ out)
{
    float mx = 0.0f;
    unsigned bad = 0;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < namps; i += gridDim.x * blockDim.x) {
        const float2 a = amps[i];
        pad[FRONT + i] = a;
        mx = fmaxf(mx, fmaxf(fabsf(a.x), fabsf(a.y)));
        /* NaN or Inf, each by itself: a maximum hides a NaN */
        if (!(fabsf(a.x) <= 3.0e38f) || !(fabsf(a.y) <= 3.0e38f)) bad = 1;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        bad |= __shfl_xor_sync(0xffffffffu, bad, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&out[0], __float_as_uint(mx));
        if (bad) atomicOr(&out[1], 1u);
    }
}

/* The tables of every phase block (grid: phase blocks x harmonics). */
__global__ void __launch_bounds__(64) table_kernel(const __grid_constant__ Geo g, const CsHarm *harm,
                                                   const uint16_t *rowtab, const uint8_t *carry,
                                                   const float *W, const float2 *A, int q, int pnum,
                                                   int m, unsigned char *tab)
{
    const int pb = blockIdx.x, h = blockIdx.y + 1, hb = (h - 1) >> 2, hh = (h - 1) & 3;
    __shared__ int srow[TI], sbin[TI];
    const int i = threadIdx.x;
    if (i < TI) {
        const long long tp = (long long)(pb * TI + i) * pnum * h;
        const long long Q = tp / q;
        const int row = harm[h - 1].woff + rowtab[(size_t)(h - 1) * q + (int)(tp - Q * q)];
        srow[i] = row;
        sbin[i] = (int)(harm[h - 1].rfloor0 + Q + carry[row]) + 1 - m / 2 + FRONT;
    }
    __syncthreads();
    unsigned char *t = tab + (size_t)pb * g.tab_bytes;
    const int nt = 2 * g.np[hb];
    const int x0 = sbin[0] & ~1;
    float *w = reinterpret_cast<float *>(t + g.w_off[hb] + hh * nt * TI * 4);
    for (int e = threadIdx.x; e < nt * TI; e += blockDim.x) {
        const int tap = e / TI, tr = e % TI;
        const int k = tap - (sbin[tr] - (sbin[tr & ~3] & ~1));
        w[e] = k >= 0 && k < m ? W[(size_t)srow[tr] * m + k] : 0.0f;
    }
    if (i < TI) reinterpret_cast<float2 *>(t + g.g_off)[(h - 1) * TI + i] = A[srow[i]];
    if (i == 0) {
        unsigned go = 0;
        for (int gr = 0; gr < 4; gr++)
            go |= (unsigned)(((sbin[4 * gr] & ~1) - x0) >> 1) << (8 * gr);
        reinterpret_cast<int *>(t + g.x_off)[h - 1] = x0;
        reinterpret_cast<unsigned *>(t + g.x_off)[64 + h - 1] = go;
    }
}

/* One tap pair of 4 trials x 4 columns. */
struct Pair {
    float4 wa, wb, x[4];
};

static __device__ __forceinline__ void pair_load(Pair &q, const unsigned char *w,
                                                 const unsigned char *v, int pitch, int p)
{
    q.wa = *reinterpret_cast<const float4 *>(w + 128 * p);
    q.wb = *reinterpret_cast<const float4 *>(w + 128 * p + 64);
#pragma unroll
    for (int j = 0; j < 4; j++)
        q.x[j] = *reinterpret_cast<const float4 *>(v + j * pitch + 16 * p);
}

static __device__ __forceinline__ void pair_fma(const Pair &q, float2 (&acc)[4][4])
{
    const float wa[4] = {q.wa.x, q.wa.y, q.wa.z, q.wa.w}, wb[4] = {q.wb.x, q.wb.y, q.wb.z, q.wb.w};
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[k][j] = __ffma2_rn(make_float2(wa[k], wa[k]), make_float2(q.x[j].x, q.x[j].y),
                                   acc[k][j]);
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int j = 0; j < 4; j++)
            acc[k][j] = __ffma2_rn(make_float2(wb[k], wb[k]), make_float2(q.x[j].z, q.x[j].w),
                                   acc[k][j]);
}

/* 4 trials x 4 columns of one harmonic, np tap pairs, the next pair's loads
 * ahead of a pair's multiply-adds (the last load of an even np reads one pair
 * past the rows, inside shared memory, and is not used).
 *
 * The loop stays rolled, here and in the epilogue: with every loop unrolled
 * the roles' straight-line code (60 KB) did not stay in the instruction
 * caches, and waiting for instructions was the largest stall by far (5.1 of
 * 11.2 warps per issue; 6.7 ms for 8.05 M trials at nharms 60 where the first
 * rolled form took 3.9). */
static __device__ __forceinline__ void block16(const unsigned char *w, const unsigned char *v,
                                               int pitch, int np, float2 (&acc)[4][4])
{
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int j = 0; j < 4; j++) acc[k][j] = make_float2(0.0f, 0.0f);
    Pair qa, qb;
    pair_load(qa, w, v, pitch, 0);
    int p = 1;
#pragma unroll 1
    for (; p < np; p += 2) {
        pair_load(qb, w, v, pitch, p);
        pair_fma(qa, acc);
        pair_load(qa, w, v, pitch, p + 1);
        pair_fma(qb, acc);
    }
    if (p == np) pair_fma(qa, acc);
}

/* ------------------------------ epilogue ------------------------------ */
/* W consecutive accumulator columns (W even), not yet waited for. */
template <int W>
static __device__ __forceinline__ void tm_load(uint32_t taddr, float *v)
{
    if constexpr (W >= 16) {
        uint32_t r[16];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 "
                     "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                       "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]),
                       "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                     : "r"(taddr));
#pragma unroll
        for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
        if constexpr (W > 16) tm_load<W - 16>(taddr + 16, v + 16);
    } else if constexpr (W >= 8) {
        uint32_t r[8];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                       "=r"(r[6]), "=r"(r[7])
                     : "r"(taddr));
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
        if constexpr (W > 8) tm_load<W - 8>(taddr + 8, v + 8);
    } else if constexpr (W >= 4) {
        uint32_t r[4];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr));
#pragma unroll
        for (int i = 0; i < 4; i++) v[i] = __uint_as_float(r[i]);
        if constexpr (W > 4) tm_load<W - 4>(taddr + 4, v + 4);
    } else if constexpr (W == 2) {
        uint32_t r[2];
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
                     : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
        v[0] = __uint_as_float(r[0]);
        v[1] = __uint_as_float(r[1]);
    }
}

/* W bins of a K-fold sum of the profile at columns col, col + NK, ... (K = 1:
 * the profile itself), left to right. */
template <int K, int NK, int W>
static __device__ __forceinline__ void fold_bins(uint32_t col, float *v)
{
    float u[K][W];
#pragma unroll
    for (int q = 0; q < K; q++) tm_load<W>(col + q * NK, u[q]);
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < W; i += 2) {
        float2 t = make_float2(u[0][i], u[0][i + 1]);
#pragma unroll
        for (int q = 1; q < K; q++) t = __fadd2_rn(t, make_float2(u[q][i], u[q][i + 1]));
        v[i] = t.x;
        v[i + 1] = t.y;
    }
}

/* The boxcar metric of one NK-bin profile, the K-fold average of the columns
 * from COL0 on, in the reference's expression order: cyclic prefix sums, the
 * largest difference of each width, max of (M_w - w / NK * total) * invsw_w
 * (src/boxcar.c:203-231).  W bins a step of a rolled loop; +infinity stands for
 * the prefixes before the first bin, which keeps windows that are not complete
 * out of the maxima. */
template <int K, int COL0, int NK, int W, class WS>
static __device__ __noinline__ float exact_metric(uint32_t trow, const float *invsw)
{
    constexpr int wmax = WS::wmax;
    static_assert(wmax <= 6 && wmax <= NK && NK % W == 0 && W % 2 == 0, "profile shape");
    const uint32_t col = trow + COL0;
    const float invk = 1.0f / (float)K;
    float mx[WS::n];
    float h[8];                     /* prefixes of the last steps, newest first */
#pragma unroll
    for (int n = 0; n < WS::n; n++) mx[n] = -INFINITY;
    h[0] = 0.0f;
#pragma unroll
    for (int i = 1; i < 8; i++) h[i] = INFINITY;
    auto push = [&](float x) {
#pragma unroll
        for (int i = 7; i > 0; i--) h[i] = h[i - 1];
        h[0] = __fadd_rn(h[0], K == 1 ? x : __fmul_rn(x, invk));
    };
#pragma unroll 1
    for (int c = 0; c < NK; c += W) {
        float v[W];
        fold_bins<K, NK, W>(col + c, v);
#pragma unroll
        for (int i = 0; i < W; i += 2) {
            push(v[i]);
            push(v[i + 1]);
#pragma unroll
            for (int n = 0; n < WS::n; n++) {
                const int w = WS::w(n);
                mx[n] = wsk::fmax3(mx[n], __fsub_rn(h[1], h[w + 1]), __fsub_rn(h[0], h[w]));
            }
        }
    }
    const float tot = h[0];
    if constexpr (wmax > 1) {
        /* the first bins again: step NK + e closes windows of more than e bins */
        constexpr int E = wmax / 2 * 2;
        float v[E];
        fold_bins<K, NK, E>(col, v);
#pragma unroll
        for (int e = 1; e < wmax; e++) {
            push(v[e - 1]);
#pragma unroll
            for (int n = 0; n < WS::n; n++)
                if (WS::w(n) > e) mx[n] = fmaxf(mx[n], __fsub_rn(h[0], h[WS::w(n)]));
        }
    }
    float best = -INFINITY;
#pragma unroll
    for (int n = 0; n < WS::n; n++) {
        const float duty = (float)WS::w(n) / (float)NK;
        best = fmaxf(best, __fmul_rn(__fsub_rn(mx[n], __fmul_rn(duty, tot)), invsw[n]));
    }
    return best;
}

/* The metric, or any value not above `need` where the metric is not above it.
 *
 * A profile's largest bin m1 and largest pair of neighbours m2 bound its longer
 * windows (3 bins: m1 + m2, 4: 2 m2, 6: 3 m2), and noise stays far below the
 * threshold by that bound too: 3 m2 reaches 8 sqrt(6) sigma only where a pair
 * is at 4.6 of its sigma.  So a pass that costs two additions, a sum and two
 * maxima for two bins decides for the warp's 32 rows whether exact_metric has
 * anything to find.  `margin` is more than its rounding errors: each prefix is
 * at most |total| + NK m1 in size, wrong by NK / 2 units in its last place at
 * most, and enters two subtractions.  (nharms 60, 8.05 M trials: the kernel takes
 * 0.35 ms less than with every width summed.) */
template <int K, int COL0, int NK, int W, class WS>
static __device__ __forceinline__ float slot_metric(uint32_t trow, const float *invsw, float need)
{
    static_assert(NK % W == 0 && W % 2 == 0, "chunks");
    const uint32_t col = trow + COL0;
    float m1 = -INFINITY, m2 = -INFINITY, tot = 0.0f, last = -INFINITY, first = 0.0f;
#pragma unroll 1
    for (int c = 0; c < NK; c += W) {
        float v[W];
        fold_bins<K, NK, W>(col + c, v);
        if (c == 0) first = v[0];
#pragma unroll
        for (int i = 0; i < W; i += 2) {
            const float p0 = v[i] + last, p1 = v[i + 1] + v[i];
            tot += p1;
            m1 = wsk::fmax3(m1, v[i], v[i + 1]);
            if (WS::wmax >= 2) m2 = wsk::fmax3(m2, p0, p1);
            last = v[i + 1];
        }
    }
    m2 = fmaxf(m2, first + last);
    const float margin = (fabsf(tot) + NK * fabsf(m1)) * (NK * 2.4e-7f);
    float bound = -INFINITY;
#pragma unroll
    for (int n = 0; n < WS::n; n++) {
        const int w = WS::w(n);
        const float duty = (float)w / (float)NK;
        const float m = w == 1 ? m1 : w == 2 ? m2 : w == 3 ? m1 + m2 : w == 4 ? 2.0f * m2 : 3.0f * m2;
        bound = fmaxf(bound, (m - duty * tot + margin) * invsw[n]);
    }
    bound *= 1.0f / (float)K;
    if (!__any_sync(0xffffffffu, !(bound <= need))) return bound;
    return exact_metric<K, COL0, NK, W, WS>(trow, invsw);
}

/* Threshold one metric of slot S of this row.  thr is the largest float not
 * above the threshold: a float metric exceeds one when it exceeds the other. */
template <int S>
static __device__ __forceinline__ void post(const Args &a, const CsChunk &ch, float m, bool valid,
                                            int ci, int j, int lane, float thr)
{
    const bool hit = valid && m > thr && j < ch.nvalid[S];
    if (__any_sync(0xffffffffu, hit)) wsk::emit(a, hit, ci, S, j, m, lane);
}

using wsk::W5;
using wsk::W4;
using wsk::W3;
using wsk::W2;

/* A row of an accumulator and the trial in it. */
struct Row {
    uint32_t trow;
    int ci, j;
    bool valid;
};

/* The slots of each configuration over the two epilogue groups, about equal in
 * bins x widths.  Each slot runs over up to two tiles before the next one: its
 * code is then fetched once for both. */
template <class C>
static __device__ __forceinline__ void epilogue(int grp, const Row &r0, const Row &r1, int ntile,
                                                const Args &a, int lane, float inv, float thr)
{
    const float need = thr / inv * (thr > 0.0f ? 0.99999f : 1.00001f);
#define SLOT(S, ...)                                                                            \
    _Pragma("unroll 1") for (int u = 0; u < ntile; u++) {                                       \
        const Row r = u ? r1 : r0;                                                              \
        const CsChunk &ch = a.chunks[r.ci];                                                     \
        const float m = slot_metric<__VA_ARGS__>(r.trow, ch.invsw[S], need) * inv;              \
        post<S>(a, ch, m, r.valid, r.ci, r.j, lane, thr);                                       \
    }
    if constexpr (C::NH == 60) {
        if (grp == 0) {
            SLOT(0, 1, 0, 120, 12, W5)
            SLOT(2, 3, 0, 40, 8, W4)
        } else {
            SLOT(1, 2, 0, 60, 12, W4)
            SLOT(3, 4, 0, 30, 10, W4)
            SLOT(4, 5, 0, 24, 8, W4)
            SLOT(5, 6, 0, 20, 4, W4)
        }
    } else if constexpr (C::NH == 32) {
        if (grp == 0) {
            SLOT(0, 1, 0, 64, 8, W5)
            SLOT(5, 1, 96, 10, 10, W2)
        } else {
            SLOT(1, 2, 0, 32, 8, W4)
            SLOT(2, 1, 64, 20, 4, W4)
            SLOT(3, 4, 0, 16, 4, W3)
            SLOT(4, 1, 84, 12, 4, W2)
        }
    } else {
        if (grp == 0) {
            SLOT(0, 1, 0, 32, 8, W5)
        } else {
            SLOT(1, 2, 0, 16, 8, W3)
            SLOT(2, 1, 32, 10, 10, W2)
            SLOT(3, 4, 0, 8, 8, wsk::Widths<2>)
            SLOT(4, 1, 42, 6, 6, wsk::Widths<1>)
            SLOT(5, 1, 48, 4, 4, wsk::Widths<1>)
        }
    }
#undef SLOT
}

/* Rotate by the (scaled) gains, split and store 2 x 4 values of an A block. */
static __device__ __forceinline__ void store_rows(const float2 (&acc)[4][4], float4 gn, uint32_t *ah)
{
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const float2 gk = k ? make_float2(gn.z, gn.w) : make_float2(gn.x, gn.y);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            float2 z;
            z.x = __fsub_rn(__fmul_rn(gk.x, acc[k][j].x), __fmul_rn(gk.y, acc[k][j].y));
            z.y = __fadd_rn(__fmul_rn(gk.x, acc[k][j].y), __fmul_rn(gk.y, acc[k][j].x));
            uint32_t hw, lw;
            wsk::split_hl(z, 1.0f, hw, lw);
            ah[(4 * k + j) * 32] = hw;
            ah[(4 * k + j) * 32 + 1024] = lw;
        }
    }
}

template <class C>
__global__ void __launch_bounds__(Roles<C>::NTHREADS, 1) search_cols(const __grid_constant__ Args a,
                                                           const __grid_constant__ XArgs x)
{
    constexpr int NINT = Roles<C>::NINT, WARP_TMA = Roles<C>::TMA, WARP_ROW = Roles<C>::ROW;
    constexpr int NPAD = C::NPAD, NBLK = C::NH / 4, NKS = (NBLK + 1) / 2;
    constexpr unsigned long long ALL = C::NH == 64 ? ~0ull : (1ull << C::NH) - 1;
    static_assert(NBLK >= NINT, "every interpolation warp has a block in every tile");
    extern __shared__ __align__(1024) unsigned char smem[];
    const Geo &g = x.g;
    const Lay L = layout(g, NPAD, C::KPAD);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = smem_u32(smem);
    const uint32_t bar = sbase + L.bar;
    constexpr int NACC = Tm<C>::NACC, NAB = Tm<C>::NAB;
    const uint32_t wfull = bar, wempty = wfull + 8 * MAX_STG, afull = wempty + 8 * MAX_STG,
                   aempty = afull + 8 * NA, dfull = aempty + 8 * NA, dempty = dfull + 8 * MAX_ACC,
                   rfull = dempty + 8 * MAX_ACC, rempty = rfull + 8 * NROW, tbar = rempty + 8 * NROW,
                   bbar = tbar + 8, drain = bbar + 8;
    volatile int *stop = reinterpret_cast<volatile int *>(smem + L.bar + 496);
    uint32_t *tm_slot = reinterpret_cast<uint32_t *>(smem + L.bar + 500);
    static_assert(8 * (2 * MAX_STG + 2 * NA + 2 * MAX_ACC + 2 * NROW + 3) <= 448, "barriers");
    /* uses of each window stage that its reader has begun with */
    volatile int *used = reinterpret_cast<volatile int *>(smem + L.bar + 448);
    static_assert(NACC >= 3 && NACC <= MAX_ACC, "the epilogue holds two accumulators");
    unsigned long long *row_fill = reinterpret_cast<unsigned long long *>(smem + L.row);
    int *row_ci = reinterpret_cast<int *>(smem + L.row + NROW * CS_TILE_M * 8);
    volatile int *row_all = reinterpret_cast<volatile int *>(smem + L.row + NROW * CS_TILE_M * 12);
    /* pairs, row pitch, weights' offset of a block */
    int4 *blk = reinterpret_cast<int4 *>(smem + L.bar + 512);
    const int tb = (int)(((long long)g.ntiles * blockIdx.x) / gridDim.x);
    const int te = (int)(((long long)g.ntiles * (blockIdx.x + 1)) / gridDim.x);
    const bool finite = a.amax[1] == 0u;
    const int nt = finite ? te - tb : 0;

    if (warp == 0) tmem_alloc(smem_u32(tm_slot), TMEM_COLS);
    if (tid == 0) {
        for (int i = 0; i < g.nstg; i++) {
            mbar_init(wfull + 8 * i, NTMA);
            mbar_init(wempty + 8 * i, 1);
        }
        for (int i = 0; i < NA; i++) {
            mbar_init(afull + 8 * i, 2);
            mbar_init(aempty + 8 * i, 1);
        }
        for (int i = 0; i < NACC; i++) {
            mbar_init(dfull + 8 * i, 1);
            mbar_init(dempty + 8 * i, NEPI);
        }
        for (int i = 0; i < NROW; i++) {
            mbar_init(rfull + 8 * i, 1);
            mbar_init(rempty + 8 * i, NINT + NEPI);
        }
        mbar_init(tbar, 1);
        mbar_init(bbar, 1);
        mbar_init(drain, 1);
        for (int i = 0; i < MAX_STG; i++) used[i] = 0;
        *stop = 0;
        if (!finite) atomicExch(a.err, NOT_FINITE);
        /* the B images, behind the other set-up; the MMA warp waits for them */
        fence_proxy_async();
        expect_tx(bbar, 2u * L.blo);
        for (int o = 0; o < 2 * L.blo; o += 16384)
            bulk_in(sbase + o, reinterpret_cast<const char *>(a.bimg) + o,
                    (uint32_t)min(16384, 2 * L.blo - o), bbar);
    }
    if (tid < NBLK) blk[tid] = make_int4(g.np[tid], g.bw[tid] * 8, g.w_off[tid], 0);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tm_slot;
    if (warp < 4) {
        /* the K padding (harmonics past nharms) of the A copies stays zero */
        const uint32_t ab = tmem + Tm<C>::A0 + ((uint32_t)(warp * 32) << 16);
#pragma unroll
        for (int b = 0; b < NAB; b++)
#pragma unroll
            for (int c = C::NH; c < C::KPAD / 2; c += 4) {
                wsk::tmem_st4(ab + b * C::KPAD + c, 0, 0, 0, 0);
                wsk::tmem_st4(ab + b * C::KPAD + C::KPAD / 2 + c, 0, 0, 0, 0);
            }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
        tc_fence_before();
    }
    __syncthreads();
    tc_fence_after();
    const float scale = operand_scale(a.amax, a.gbound);
    auto fail = [&]() {
        *stop = 1;
        atomicExch(a.err, 1);
    };
    /* slot i of a ring of n: wait for its use number `use` to be complete */
    auto full_wait = [&](uint32_t b, int slot, int use) {
        return wait_bar(b + 8 * slot, use & 1, stop);
    };

    if constexpr (NINT == 8) {      /* by groups of 4 warps, all through here */
        if (warp < NINT) asm volatile("setmaxnreg.inc.sync.aligned.u32 120;");
        else if (warp < WARP_TMA) asm volatile("setmaxnreg.dec.sync.aligned.u32 88;");
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    }
    if (warp < NINT) {
        /* ------------------------- interpolation ------------------------- */
        const int hh = lane >> 3, cg = (lane >> 2) & 1, gr = lane & 3;
        const unsigned char *tab = smem + L.tab;
        const unsigned *goffs = reinterpret_cast<const unsigned *>(tab + g.x_off) + 64;
        const int nunit = nt * NBLK;
        int it = -1, itn = 0, hb = warp, all = 1, pb = tb / g.ncg - 1, loads = 0;
        int pb_end = tb;                     /* first tile past phase block pb */
        int st = warp % g.nstg, round = warp / g.nstg;
        bool ok = true;
        /* what a block needs from shared memory is read while the block before
         * is stored: its rows' shape, and the groups' window offsets */
        int4 b4 = blk[hb];
        unsigned goff = 0;
        for (int n = warp; n < nunit; n += NINT) {
            const int h = 4 * hb + hh;                          /* harmonic - 1 */
            if (itn != it) {
                if (it >= 0 && lane == 0) wsk::mbar_arrive(rempty + 8 * (it % NROW));
                it = itn;
                ok = full_wait(rfull, it % NROW, it / NROW) && ok;
                all = row_all[4 * (it % NROW)];
                if (tb + it >= pb_end) {     /* its table */
                    pb++;
                    pb_end = (pb + 1) * g.ncg;
                    ok = full_wait(tbar, 0, loads++) && ok;
                    goff = goffs[h];
                }
            }
            const int np = b4.x, pitch = b4.y;
            const unsigned char *w = tab + b4.z + hh * np * 128 + gr * 16;
            const unsigned char *v = smem + L.win + st * g.stg_bytes +
                                     (hh * TC + 4 * cg) * pitch +
                                     ((goff >> (8 * gr)) & 0xfu) * 16;
            const int ks = it * NKS + (hb >> 1), as = ks % NA;
            /* the stage's last use first: its reader may be another warp that is
             * behind, and a parity says nothing about a phase two back */
            ok = count_wait(used + st, round, stop) && ok;
            ok = full_wait(wfull, st, round) && ok;
            if (lane == 0) used[st] = round + 1;
            const bool afree = ks < NA || mbar_try(aempty + 8 * as, (ks / NA - 1) & 1);
            const float4 *gp = reinterpret_cast<const float4 *>(tab + g.g_off) + h * 8 + 2 * gr;
            float4 gn[2] = {gp[0], gp[1]};
            float2 acc[4][4];
            block16(w, v, pitch, np, acc);
            if (!__all_sync(0xffffffffu, ok && afree)) {
                if (!afree) ok = full_wait(aempty, as, ks / NA - 1) && ok;
                if (!__all_sync(0xffffffffu, ok)) {
                    fail();
                    break;
                }
            }
            if (lane == 0) wsk::mbar_arrive(wempty + 8 * st);    /* window and table are read */
            /* the next block */
            const bool odd_tail = (NBLK & 1) && hb == NBLK - 1;
            uint32_t *ah = reinterpret_cast<uint32_t *>(smem + L.a + as * A_STEP + (hb & 1) * 2048 +
                                                        (lane & 7) * 16 + hh * 4);
            hb += NINT;
            if (hb >= NBLK) {
                hb -= NBLK;
                itn++;
            }
            st += NINT;
            while (st >= g.nstg) {
                st -= g.nstg;
                round++;
            }
            b4 = blk[hb];
            goff = goffs[4 * hb + hh];
            const unsigned long long *fill = row_fill + (it % NROW) * CS_TILE_M + (lane & 7);
            /* the fp16 operand scale, a power of two, goes in with the gains */
#pragma unroll
            for (int k = 0; k < 2; k++)
                gn[k] = make_float4(gn[k].x * scale, gn[k].y * scale, gn[k].z * scale,
                                    gn[k].w * scale);
#pragma unroll 1
            for (int k2 = 0; k2 < 2; k2++) {
                store_rows(acc, gn[0], ah + 256 * k2);
                gn[0] = gn[1];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    acc[0][j] = acc[2][j];
                    acc[1][j] = acc[3][j];
                }
            }
            if (!all) {
                /* rows whose harmonic is not active */
#pragma unroll 1
                for (int r = 0; r < 16; r++)
                    if (!((fill[8 * r] >> h) & 1ull)) ah[32 * r] = ah[32 * r + 1024] = 0;
            }
            /* the MMA thread has the proxy fence between its wait and its MMAs */
            __syncwarp();
            if (lane == 0) {
                wsk::mbar_arrive(afull + 8 * as);
                if (odd_tail) wsk::mbar_arrive(afull + 8 * as);
            }
        }
    } else if (warp < WARP_TMA) {
        /* --------------------------- epilogue ---------------------------- */
        const int e = warp - NINT, grp = e >> 2, quarter = e & 3;
        const int r = quarter * 32 + lane;
        const float inv_scale = 1.0f / scale, thr = __double2float_rd(a.thresh);
        const int toff = 4 * (r & 3) + (r >> 5) +
                         g.D * (4 * ((r >> 2) & 1) + ((r >> 3) & 3));
        int p = tb / g.ncg, cgi = tb - p * g.ncg;
        for (int it = 0; it < nt; it += 2) {
            const int ntile = min(2, nt - it);
            Row row[2];
            bool ok = true;
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (u < ntile) {
                    const int k = it + u, s = k % NACC, rs = k % NROW;
                    ok = full_wait(rfull, rs, k / NROW) && ok;
                    ok = full_wait(dfull, s, k / NACC) && ok;
                    const int c = row_ci[rs * CS_TILE_M + r];
                    row[u].valid = c >= 0;
                    row[u].ci = max(c, 0);
                    row[u].j = p * TI + cgi * TC * g.D + toff - (int)a.chunks[max(c, 0)].i0;
                    row[u].trow = tmem + (uint32_t)(s * Tm<C>::DS) +
                                  ((uint32_t)(quarter * 32) << 16);
                    if (++cgi == g.ncg) {
                        cgi = 0;
                        p++;
                    }
                } else {
                    row[u] = row[0];
                }
            }
            if (!__all_sync(0xffffffffu, ok)) {
                fail();
                break;
            }
            tc_fence_after();
            epilogue<C>(grp, row[0], row[1], ntile, a, lane, inv_scale, thr);
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                for (int k = it; k < it + ntile; k++) {
                    wsk::mbar_arrive(dempty + 8 * (k % NACC));
                    wsk::mbar_arrive(rempty + 8 * (k % NROW));
                }
        }
    } else if (warp < WARP_ROW) {
        /* ---- window boxes: warp i issues harmonics 2i and 2i + 1 of every
         * block, so that either has seen every stage's last use itself ---- */
        const int me = warp - WARP_TMA;
        int pb = -1, loads = 0;
        int p = tb / g.ncg, cgi = tb - p * g.ncg;
        int n = 0, st = 0, round = 0;
        bool ok = true;
        /* a lane holds what its box of the tile needs, block lane / 2: nothing is
         * computed or read between a stage's wait and its boxes (the two warps
         * were busy all the time: 1 M trials 341 -> 336 us, 1.1 M at nharms 16 174 ->
         * 152) */
        const int mine = lane >> 1, hl = 4 * min(mine, NBLK - 1) + 2 * me + (lane & 1);
        const int *x0 = reinterpret_cast<const int *>(smem + L.tab + g.x_off);
        const char *maps = reinterpret_cast<const char *>(x.maps) + 2 * me * 128;
        const int pitch = blk[min(mine, NBLK - 1)].y;
        const uint32_t dst = sbase + L.win;
        const int step = 2 * TC * g.shift[0] * (hl + 1);     /* floats a column group */
        int xp = 0;
        for (int it = 0; it < nt && ok; it++) {
            if (p != pb) {
                pb = p;
                if (me == 0) {
                    /* the interpolation is done with the last table when every
                     * stage filled so far is free again */
                    for (int k = n > g.nstg ? n - g.nstg : 0; k < n; k++)
                        ok = full_wait(wempty, k % g.nstg, k / g.nstg) && ok;
                    if (ok && lane == 0) {
                        expect_tx(tbar, (uint32_t)g.tab_bytes);
                        const unsigned char *src = x.tab + (size_t)p * g.tab_bytes;
                        for (int o = 0; o < g.tab_bytes; o += 16384)
                            bulk_in(sbase + L.tab + o, src + o,
                                    (uint32_t)min(16384, g.tab_bytes - o), tbar);
                    }
                    __syncwarp();
                }
                ok = full_wait(tbar, 0, loads++) && ok;
                xp = 2 * x0[hl];
            }
            /* a multiple of 4 floats: the box starts on 16 bytes */
            const int xc = (xp + cgi * step) & ~3;
#pragma unroll 1
            for (int hb = 0; hb < NBLK; hb++, n++) {
                if (round > 0) ok = full_wait(wempty, st, round - 1) && ok;
                if (__any_sync(0xffffffffu, !ok)) {
                    ok = false;
                    break;
                }
                const int xa = __shfl_sync(0xffffffffu, xc, 2 * hb);
                const int xb = __shfl_sync(0xffffffffu, xc, 2 * hb + 1);
                const uint32_t rows = __shfl_sync(0xffffffffu, (uint32_t)(TC * pitch), 2 * hb);
                const uint32_t b = wfull + 8 * st, to = dst + st * g.stg_bytes + 2 * me * rows;
                const char *m = maps + hb * 512;
                if (elect()) {
                    expect_tx(b, 2 * rows);
                    tma_rows(to, m, xa, b);
                    tma_rows(to + rows, m + 128, xb, b);
                }
                __syncwarp();
                if (++st == g.nstg) {
                    st = 0;
                    round++;
                }
            }
            if (++cgi == g.ncg) {
                cgi = 0;
                p++;
            }
        }
        if (!ok) fail();
        /* never leave with copies in flight: the last table and the last use of each
         * stage landed.  Not full_wait, which ends when any role has given up */
        if (loads && !mbar_wait(tbar, (loads - 1) & 1)) fail();
        for (int k = n > g.nstg ? n - g.nstg : 0; k < n; k++)
            if (!mbar_wait(wfull + 8 * (k % g.nstg), (k / g.nstg) & 1)) fail();
    } else if (warp == WARP_ROW) {
        /* ------- the chunk and active harmonics of rows lane, lane + 32, .. ------- */
        int p = tb / g.ncg, cgi = tb - p * g.ncg;
        int ci[4] = {-1, -1, -1, -1};
        const int off = 4 * (lane & 3) + g.D * (4 * ((lane >> 2) & 1) + ((lane >> 3) & 3));
        for (int it = 0; it < nt; it++) {
            const int rs = it % NROW;
            bool full = true, ok = true;
            int c[4];
            unsigned long long f[4];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const int t = p * TI + k + cgi * TC * g.D + off;
                f[k] = 0;
                c[k] = -1;
                if (t < g.total) {
                    if (ci[k] < 0) {
                        int lo = 0, hi = g.nchunks - 1;
                        while (lo < hi) {              /* last chunk starting at or before t */
                            const int mid = (lo + hi + 1) >> 1;
                            if (a.chunks[mid].i0 <= t) lo = mid;
                            else hi = mid - 1;
                        }
                        ci[k] = lo;
                    }
                    while (ci[k] + 1 < g.nchunks && a.chunks[ci[k] + 1].i0 <= t) ci[k]++;
                    c[k] = ci[k];
                    f[k] = a.chunks[c[k]].filled;
                }
                full = full && (f[k] & ALL) == ALL;
            }
            if (it >= NROW) ok = full_wait(rempty, rs, it / NROW - 1);
            if (!__all_sync(0xffffffffu, ok)) {
                fail();
                break;
            }
#pragma unroll
            for (int k = 0; k < 4; k++) {
                row_ci[rs * CS_TILE_M + 32 * k + lane] = c[k];
                row_fill[rs * CS_TILE_M + 32 * k + lane] = f[k];
            }
            full = __all_sync(0xffffffffu, full);
            if (lane == 0) row_all[4 * rs] = full ? 1 : 0;
            __syncwarp();
            if (lane == 0) wsk::mbar_arrive(rfull + 8 * rs);
            if (++cgi == g.ncg) {
                cgi = 0;
                p++;
#pragma unroll
                for (int k = 0; k < 4; k++) ci[k] = -1;
            }
        }
    } else {
        /* ----------------------------- MMAs ------------------------------ */
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | ((uint32_t)(NPAD >> 3) << 17) |
                                   ((uint32_t)(CS_TILE_M >> 4) << 24);
            const uint32_t lbo_b = NPAD * 16;
            const uint32_t b_hi = sbase, b_lo = sbase + L.blo;
            bool ok = full_wait(bbar, 0, 0);
            for (int it = 0; it < nt && ok; it++) {
                const int s = it % NACC;
                if (it >= NACC) ok = full_wait(dempty, s, it / NACC - 1);
                /* the A copy is free when the transform that read it is done */
                if (it >= NAB) ok = ok && full_wait(dfull, (it - NAB) % NACC, (it - NAB) / NACC);
                if (!ok) break;
                tc_fence_after();
                const uint32_t d = tmem + (uint32_t)(s * Tm<C>::DS);
                const uint32_t a_hi = tmem + (uint32_t)(Tm<C>::A0 + (it % NAB) * C::KPAD);
                const uint32_t a_lo = a_hi + C::KPAD / 2;
                /* each K step on arrival: copied to tensor memory, which frees its
                 * slot, and its hi * hi; then lo * hi and hi * lo of the whole tile
                 * (the order of search_ws: the same bits) */
                for (int k = 0; k < NKS; k++) {
                    const int ks = it * NKS + k, as = ks % NA;
                    ok = full_wait(afull, as, ks / NA);
                    if (!ok) break;
                    fence_proxy_async();        /* the A step was written by plain stores */
                    tc_fence_after();
                    const uint32_t src = sbase + L.a + as * A_STEP;
                    for (int b = 0; b < 2 && 2 * k + b < NBLK; b++) {
                        tmem_copy16(a_hi + 4 * (2 * k + b), umma_desc(src + b * 2048, 2048, 128));
                        tmem_copy16(a_lo + 4 * (2 * k + b), umma_desc(src + 4096 + b * 2048, 2048, 128));
                    }
                    wsk::mma_f16_ts(d, a_hi + 8 * k,
                                    umma_desc(b_hi + (uint32_t)k * 2 * lbo_b, lbo_b, 128), idesc, k > 0);
                    mma_commit(aempty + 8 * as);
                }
                if (!ok) break;
                for (int k = 0; k < NKS; k++)
                    wsk::mma_f16_ts(d, a_lo + 8 * k,
                                    umma_desc(b_hi + (uint32_t)k * 2 * lbo_b, lbo_b, 128), idesc, 1);
                for (int k = 0; k < NKS; k++)
                    wsk::mma_f16_ts(d, a_hi + 8 * k,
                                    umma_desc(b_lo + (uint32_t)k * 2 * lbo_b, lbo_b, 128), idesc, 1);
                mma_commit(dfull + 8 * s);
            }
            if (!ok) fail();
            /* never leave with the B images on their way, nor free tensor memory
             * under copies and MMAs in flight, whichever role gave up */
            bool landed = mbar_wait(bbar, 0);
            mma_commit(drain);
            landed = mbar_wait(drain, 0) && landed;
            if (!landed) fail();
        }
    }
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        tmem_dealloc(tmem, TMEM_COLS);
    }
}

}  // namespace cols
