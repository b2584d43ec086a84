// vg_range.cuh -- the FP32 iteration kernel: warps on ranges of samples.
//
// Reference: src/vegas/_vegas.pyx (vegas 6.4.1): sampling and map of
// Integrator._random_batch (pyx:1731-1752), the per-hypercube mean and
// variance of Integrator.__call__ (pyx:2136-2193), the training feed
// (pyx:2173, 2196-2197 -> AdaptiveMap.add_training_data pyx:421-464).
//
// Samples of an iteration are ordered by hypercube.  They are divided into
// chunks of 128, the chunks into contiguous ranges of as equal length as
// possible, one per group of 8 warps and in it one per warp.  A chunk is sampled
// with lane l on samples l, l + 32, ... (coalesced reads and writes, one
// sample's values live at a time), its wgt*f left in the warp's shared memory;
// then lane l reduces samples 4l .. 4l+3, so a hypercube is a run over a few
// lanes and one segmented scan by shuffles joins the pieces.  A hypercube that
// continues into the warp's next chunk is carried in registers, the pieces of
// one cut by the ends of the warps' ranges are joined by one warp of 8; only
// those cut by the ends of these groups' ranges leave records for the finalize.
//
// The variance needs no second pass over the samples: sums of d = wf - c and
// d^2 about c = the hypercube's first sample of the range, in float-float
// (about 2^-44 relative), give (n Q - D^2) / (n - 1) -- the reference's formula,
// which is exact for any c.  The cancellation costs about (c - mean)^2 / var, n at the
// most, of the 2^-44, and the samples themselves are FP32.  (Variances of iterations
// against long double, five integrands, dims 1 to 9: 2^-47 to 2^-50, as with two
// passes about the mean.)  Sums of squares beyond 1e30 go to FP64; a hypercube that goes
// on into the next chunk then goes on about its mean, so that Q stays near the
// variance where c was an outlier.
//
// Why this shape.  No barrier of the CTA is inside the loop, so 1024 threads
// share one grid table and one training histogram (64 KB each at dim 8 with
// 1000 increments, which left room for only 8 warps per SM with a CTA of 256
// threads and its block-wide scans), and the loops are not unrolled over a
// thread's samples, so the code fits the instruction cache.
#pragma once
#include <atomic>

#include "vg_tile.cuh"

namespace vg {

constexpr int CHUNK = 128;      // samples per chunk
constexpr int WCAP = 68;        // hypercube starts a chunk can see (two samples each or more), padded
static_assert(CHUNK == BASE_TILE, "tile_h0 gives the first hypercube of each chunk");

constexpr int OPEN = WCAP - 1;  // a chunk sees WCAP - 2 hypercubes at the most

// Per-warp shared memory.  res holds (D, Q) of the hypercubes that end in the
// chunk, the sampling weights dv_y / neval_h use the same space before; its
// last element holds (D, Q) of the one that began before the chunk.
struct WarpBuf {
    float4 res[WCAP];
    float wf[CHUNK];
    int off[WCAP];              // start of each hypercube relative to the chunk
    unsigned int mask[CHUNK / 32];   // bit i: a hypercube after the chunk's first starts at sample i
};

struct RangePlan {
    size_t table, hsum, hcnt, itab, red, recs, warps, total;
};

__host__ __device__ inline RangePlan range_plan(int ntb, int dim, int maxK, int table_smem, int hist_copies,
                                                int tab_len)
{
    RangePlan p;
    size_t o = 0;
    p.table = o;
    if (table_smem) o = (o + sizeof(float2) * (size_t)dim * (maxK + 1) + 15) & ~(size_t)15;
    p.hsum = o;
    o = (o + sizeof(float) * (size_t)dim * (maxK + 1) * hist_copies + 15) & ~(size_t)15;
    p.hcnt = o;
    if (hist_copies) o = (o + sizeof(unsigned int) * (size_t)dim * (maxK + 1) + 15) & ~(size_t)15;
    p.itab = o;
    o = (o + sizeof(float) * (tab_len + 4) + 15) & ~(size_t)15;
    p.red = o;
    o = (o + sizeof(float) * 6 * (ntb / 32) + 15) & ~(size_t)15;
    p.recs = o;
    o += sizeof(RangeRec) * 2 * (ntb / 32);
    p.warps = o;
    o += sizeof(WarpBuf) * (ntb / 32);
    p.total = o;
    return p;
}

// The warps of a CTA work in groups of 8 on one contiguous range each; the groups'
// ranges are dealt to the CTAs in turn, so that every CTA sees several parts of
// the integration region (a ridge sample costs three times as much on the ridge
// as off it; one contiguous range per CTA took 62 us instead of 49 at 1e6
// samples of dim 4).
constexpr int GROUP = 8;
// Records of an iteration of N samples: one pair per group that has any chunk,
// or, where units of `deal` chunks are dealt to the warps (deal > 0), per unit.
__host__ __device__ __forceinline__ int64_t record_count(int64_t N, int64_t ngroups, int deal)
{
    const int64_t c = (N + CHUNK - 1) / CHUNK;
    return deal ? (c + deal - 1) / deal : (c < ngroups ? c : ngroups);
}

// Sums of d = x - c and d^2 in float-float (TwoDiff and TwoProd, error-free).
struct DQ {
    float dh, dl, qh, ql;
    __device__ __forceinline__ void zero() { dh = dl = qh = ql = 0.f; }
    __device__ __forceinline__ void add(float x, float c)
    {
        const float d = __fsub_rn(x, c);
        const float bb = __fsub_rn(d, x);
        const float e = __fsub_rn(__fsub_rn(x, __fsub_rn(d, bb)), __fadd_rn(c, bb));
        vg_ff_add(dh, dl, d);
        dl = __fadd_rn(dl, e);
        const float p = __fmul_rn(d, d);
        const float pe = __fmaf_rn(__fmul_rn(2.f, d), e, __fmaf_rn(d, d, -p));
        vg_ff_add(qh, ql, p);
        ql = __fadd_rn(ql, pe);
    }
    __device__ __forceinline__ void add(const DQ &o)
    {
        ff_add_pair(dh, dl, o.dh, o.dl);
        ff_add_pair(qh, ql, o.qh, o.ql);
    }
    __device__ __forceinline__ DQ up(int off) const
    {
        DQ r;
        r.dh = __shfl_up_sync(0xffffffffu, dh, off);
        r.dl = __shfl_up_sync(0xffffffffu, dl, off);
        r.qh = __shfl_up_sync(0xffffffffu, qh, off);
        r.ql = __shfl_up_sync(0xffffffffu, ql, off);
        return r;
    }
    __device__ __forceinline__ DQ from(int lane) const
    {
        DQ r;
        r.dh = __shfl_sync(0xffffffffu, dh, lane);
        r.dl = __shfl_sync(0xffffffffu, dl, lane);
        r.qh = __shfl_sync(0xffffffffu, qh, lane);
        r.ql = __shfl_sync(0xffffffffu, ql, lane);
        return r;
    }
};

// The sum n c + D of a piece of n samples.
__device__ __forceinline__ void piece_sum(float fn, float c, const DQ &v, float &sh, float &sl)
{
    sh = __fmul_rn(fn, c);
    sl = __fmaf_rn(fn, c, -sh);
    ff_add_pair(sh, sl, v.dh, v.dl);
}

// Where no sample differs from the others, every deviation from the mean is
// below EPSILON |mean| and counts as that (pyx:2156): Q of n such samples.
__device__ __forceinline__ float guard_q(float fn, float sh)
{
    const float thr = (float)VG_EPSILON * fabsf(sh * __frcp_rn(fn));
    return fn * thr * thr;
}

// The next digit of a hypercube's number where it may exceed 31 bits.
static __device__ __noinline__ int wide_digit(int64_t &h, int nstrat)
{
    const int64_t q = h / nstrat;
    const int y0 = (int)(h - q * nstrat);
    h = q;
    return y0;
}

// adapt_to_errors: a hypercube's |variance| trains the map at its last sample.
static __device__ __noinline__ void train_last(const IterArgs &a, int64_t h, double v)
{
    unsigned short b[VG_MAX_DIM];
    last_sample_bins<float>(a, h, b);
    train_hcube(a, b, v);
}

// Running sums of the hypercubes a lane finishes.
struct LaneSums {
    float mh, ml, vh, vl, sh, sl;
};

// Beyond this a sum Q of squares goes to FP64 (also where it is infinite or NaN).
constexpr float BIG_Q = 1e30f;

// D and Q in FP64 of the piece at samples o to oe of the chunk about c; with o < 0 it
// began earlier, and wb.res[OPEN] has the sums of its samples before the chunk.
__device__ __forceinline__ void sums_f64(const WarpBuf &wb, int o, int oe, float c, double &D, double &Q)
{
    D = Q = 0.0;
    if (o < 0) {
        const float4 v = wb.res[OPEN];
        D = vg_ff_value(v.x, v.y);
        Q = vg_ff_value(v.z, v.w);
    }
    for (int i = max(o, 0); i < oe; i++) {
        const double d = (double)wb.wf[i] - (double)c;
        D += d;
        Q = fma(d, d, Q);
    }
}

// A hypercube of n samples whose squares leave the float range, in FP64.
static __device__ __noinline__ double3 finish_big(const WarpBuf &wb, int o, int oe, float c, double beta_half,
                                                  int adaptive, double *sigf_h, int want_var)
{
    const int n = oe - o;
    const double nd = (double)n;
    double S, D = 0.0, Q = 0.0;
    if (o >= 0) {
        S = 0.0;
        for (int i = o; i < oe; i++) S += (double)wb.wf[i];
        const double m = S / nd;
        for (int i = o; i < oe; i++) {
            const double d = (double)wb.wf[i] - m;
            D += d;
            Q = fma(d, d, Q);
        }
    } else {
        sums_f64(wb, o, oe, c, D, Q);
        S = nd * (double)c;
    }
    return finish_f64(S, D, Q, n, beta_half, adaptive, sigf_h, want_var);
}

// A piece of n samples of which those before oe in the chunk are the last, and whose squares
// about c leave the float range: its sums about its mean, which is returned, to
// wb.res[OPEN].  Q is then near the variance and no longer up to n times as large (c an
// outlier), so a piece that goes on stays in the range that its variance has.  One lane.
static __device__ __noinline__ float recentre_big(WarpBuf &wb, int o, int oe, int n, float c)
{
    double D, Q;
    sums_f64(wb, o, oe, c, D, Q);
    const double nd = (double)n;
    const float m = (float)((double)c + D / nd);
    const double t = (double)c - (double)m;
    Q += t * (2.0 * D + nd * t);
    D += nd * t;
    float4 v;
    ff_from_double(D, v.x, v.y);
    ff_from_double(Q, v.z, v.w);
    wb.res[OPEN] = v;
    return m;
}

// One whole hypercube: mean, variance (n Q - D^2) / (n - 1) and sigf =
// |var|^(beta/2) (pyx:2174-2186) into the lane's sums; FP64 only where the
// squares leave the float range.  It is at samples o (< 0: it began earlier) to oe
// of the chunk.
__device__ __forceinline__ void finish_hcube(const IterArgs &a, int64_t h, const WarpBuf &wb, int o, int oe, float c,
                                             const DQ &v, float beta_half_f, LaneSums &s)
{
    const float fn = (float)(oe - o);
    if (!(fabsf(v.qh) < BIG_Q)) {
        const double3 r = finish_big(wb, o, oe, c, a.beta_half, a.adaptive, a.sigf + h, a.train_hc);
        float rh, rl;
        ff_from_double(r.x, rh, rl);
        ff_add_pair(s.mh, s.ml, rh, rl);
        ff_from_double(r.y, rh, rl);
        ff_add_pair(s.vh, s.vl, rh, rl);
        if (!a.train_hc) {
            ff_from_double(r.z, rh, rl);
            ff_add_pair(s.sh, s.sl, rh, rl);
        } else {
            train_last(a, h, r.z);
        }
        return;
    }
    float th, tl, vh, vl;
    piece_sum(fn, c, v, th, tl);
    ff_add_pair(s.mh, s.ml, th, tl);
    const float qh = v.qh == 0.f ? guard_q(fn, th) : v.qh;
    float d2h, d2l;
    ff_mul_f(qh, v.ql, fn, vh, vl);
    ff_sqr(v.dh, v.dl, d2h, d2l);
    ff_add_pair(vh, vl, -d2h, -d2l);
    ff_div_f(vh, vl, fn - 1.f, vh, vl);
    ff_add_pair(s.vh, s.vl, vh, vl);
    if (a.adaptive) {
        const float av = fabsf(vh);
        const float sg = av > 0.f ? vg_ex2_approx(beta_half_f * vg_lg2_approx(av)) : 0.f;
        a.sigf[h] = (double)sg;
        vg_ff_add(s.sh, s.sl, sg);
    }
    if (a.train_hc) train_last(a, h, fabs(vg_ff_value(vh, vl)));
}

// A piece of a hypercube cut by the ends of ranges: samples, sum, squared
// deviations about its mean (float-float).  Joined by Chan et al.'s
// parallel-variance update: Q = Q1 + Q2 + (m2 - m1)^2 n1 n2 / (n1 + n2).
struct Piece {
    float n, sh, sl, qh, ql;
    __device__ __forceinline__ void from(const RangeRec &r)
    {
        n = (float)(r.n < 0 ? -r.n : r.n);
        sh = r.dh;
        sl = r.dl;
        qh = r.qh;
        ql = r.ql;
        if (r.c != r.c) return;
        piece_sum(n, r.c, DQ{r.dh, r.dl, r.qh, r.ql}, sh, sl);
        if (qh == 0.f) {
            qh = guard_q(n, sh);
        } else {
            // Q - D (D / n), at most Q: D^2 would leave the float range before it
            float mh, ml, th, tl;
            ff_div_f(r.dh, r.dl, n, mh, ml);
            ff_mul(r.dh, r.dl, mh, ml, th, tl);
            ff_add_pair(qh, ql, -th, -tl);
        }
    }
    __device__ __forceinline__ RangeRec record(int64_t h, bool spans) const
    {
        return RangeRec{h, spans ? -(int)n : (int)n, __int_as_float(0x7fffffff), sh, sl, qh, ql};
    }
    __device__ __forceinline__ void put_first(const Piece &p)   // p comes before this one
    {
        if (!(p.n > 0.f)) return;
        const float n2 = n + p.n;
        float m1h, m1l, m2h, m2l, wh, wl, ddh, ddl, th, tl;
        ff_div_f(p.sh, p.sl, p.n, m1h, m1l);
        ff_div_f(sh, sl, n, m2h, m2l);
        ff_add_pair(m2h, m2l, -m1h, -m1l);
        const float wph = __fmul_rn(p.n, n);
        const float wpl = __fmaf_rn(p.n, n, -wph);
        ff_div_f(wph, wpl, n2, wh, wl);
        ff_sqr(m2h, m2l, ddh, ddl);
        ff_mul(ddh, ddl, wh, wl, th, tl);
        ff_add_pair(qh, ql, p.qh, p.ql);
        ff_add_pair(qh, ql, th, tl);
        ff_add_pair(sh, sl, p.sh, p.sl);
        n = n2;
    }
    __device__ __forceinline__ Piece up(int off) const
    {
        Piece r;
        r.n = __shfl_up_sync(0xffffffffu, n, off);
        r.sh = __shfl_up_sync(0xffffffffu, sh, off);
        r.sl = __shfl_up_sync(0xffffffffu, sl, off);
        r.qh = __shfl_up_sync(0xffffffffu, qh, off);
        r.ql = __shfl_up_sync(0xffffffffu, ql, off);
        return r;
    }
};

// A cut hypercube, all of its pieces joined: its mean, variance and sigf into
// the sums (s6: mean, variance, sigf in float-float).
static __device__ __noinline__ void finish_cut(const IterArgs &a, int64_t h, const Piece &p, float (&s6)[6])
{
    float vh, vl;
    if (fabsf(p.qh) < BIG_Q) {
        ff_mul_f(p.qh, p.ql, p.n, vh, vl);
        ff_div_f(vh, vl, p.n - 1.f, vh, vl);
    } else {   // squares beyond the float range: this hypercube in FP64
        const double nd = (double)p.n;
        const double v = vg_div_fast(__dmul_rn(nd, vg_ff_value(p.qh, p.ql)), nd - 1.0);
        vh = (float)v;
        vl = (float)(v - (double)vh);
    }
    if (a.train_hc) train_last(a, h, fabs(vg_ff_value(vh, vl)));
    ff_add_pair(s6[0], s6[1], p.sh, p.sl);
    ff_add_pair(s6[2], s6[3], vh, vl);
    if (a.adaptive) {
        const float av = fabsf(vh);
        const float sg = av > 0.f ? vg_ex2_approx((float)a.beta_half * vg_lg2_approx(av)) : 0.f;
        a.sigf[h] = (double)sg;
        vg_ff_add(s6[4], s6[5], sg);
    }
}

// Open pieces across the lanes of a warp (started: the lane's piece begins in
// the lane): each lane gets the piece joined with what came before it.  Returns
// whether it begins in the warp.
__device__ __forceinline__ bool scan_pieces(Piece &cur, bool started)
{
    const int lane = threadIdx.x & 31;
    const unsigned int heads = __ballot_sync(0xffffffffu, started) & (0xffffffffu >> (31 - lane));
    const int dist = heads ? lane - (31 - __clz(heads)) : lane;
    const int maxd = __reduce_max_sync(0xffffffffu, dist);
    for (int off = 1; off <= maxd; off <<= 1) {
        const Piece o = cur.up(off);
        if (dist >= off) cur.put_first(o);
    }
    return heads != 0u;
}

// Hypercubes of one sample or none: the hypercube of the sample b, at h or after it, and
// a length of the chunk there such that it sees no more hypercubes than the warp's
// buffer takes, and none without samples (two that start at the same sample).
struct Windows {
    int64_t h;
    int len;
};
static __device__ __noinline__ Windows few_windows(const IterArgs &a, int64_t b, int64_t N, int64_t h, int len)
{
    const int lane = threadIdx.x & 31;
    auto start = [&](int64_t k) {   // of hypercube k, relative to b
        const int64_t dif = (k <= a.H ? a.offsets[k] : N) - b;
        return dif > CHUNK ? CHUNK + 1 : (dif < -1 ? -1 : (int)dif);
    };
    for (;;) {   // pass those that end at b or before
        const int64_t next = h + 1 + lane;
        const unsigned int m = __ballot_sync(0xffffffffu, next < a.H && start(next) <= 0);
        h += __popc(m);
        if (m != 0xffffffffu) break;
    }
    int cut = len;
    for (int k = 1 + lane; k < WCAP - 1; k += 32) {
        const int s = start(h + k);
        if (s < cut && (k == WCAP - 2 || start(h + k + 1) == s)) cut = s;
    }
    return Windows{h, __reduce_min_sync(0xffffffffu, cut)};
}

// ------------------------------------------------------------------ kernel
constexpr int RF_CHAIN = 8;   // a kernel of its own, launched with vg_launch_pdl

template <bool WIDE>
struct IndexType {
    typedef int type;
};
template <>
struct IndexType<true> {
    typedef int64_t type;
};

// What a body is compiled for.  A sample's code reads few of the run-time
// choices below again and again for each axis; compiled in, they take a third
// of the instructions away (2^20 samples of the 8-d mixture: 37 -> 25 million
// warp instructions).
constexpr int RF_EXACT = 1;   // dim == DIMB
constexpr int RF_TABLE = 2;   // the grid table is in shared memory (else: read through L1)
constexpr int RF_GENERAL = 4; // injected uniforms, 2^31 hypercubes or samples, 2^24 strata on an axis, hypercubes
                              // of fewer than two samples, the table and the histogram in either place

// The work of CTA `rank` of `nranks` on one integral's iteration; its partial
// sums go to a.parts[rank].  deal > 0 (the batched launch): units of `deal`
// chunks are dealt to the CTAs and their warps in turn.  Which samples share a
// CTA's FP32 histogram, and in what order they come, decides how its sums are
// rounded; where a few samples carry a bin (the lattice integrals, Lorentzians
// in 9 dimensions) adapting from iteration to iteration amplifies that a
// thousandfold.  Dealt units add in the order of the samples as a CTA walking
// tile by tile does, so results stay those of such a launch to the atomics'
// noise.
template <int MODE, int KIND, int DIMB, int F>
__device__ __forceinline__ void range_body(const IterArgs &a, const VgParams &prm, unsigned char *smem, int rank,
                                           int nranks, int deal)
{
    constexpr bool NEED_RED = (MODE == MODE_REDUCE || MODE == MODE_FUSED || MODE == MODE_REDUCE_KEPT);
    constexpr bool NEED_MAP = MODE != MODE_REDUCE_KEPT;
    constexpr bool NEED_X = MODE == MODE_POINTS || MODE == MODE_FUSED || MODE == MODE_EVAL;
    constexpr bool GENERAL = F & RF_GENERAL;
    typedef typename IndexType<GENERAL>::type Idx;   // samples and hypercubes
    const int NTB = (int)blockDim.x, NW = NTB >> 5;
    const int dim = (F & RF_EXACT) ? DIMB : a.dim;
    const bool table_smem = NEED_MAP && (GENERAL ? a.table_smem != 0 : bool(F & RF_TABLE));
    const bool wide = GENERAL && a.wide;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int W = a.maxK + 1;
    const RangePlan sp = range_plan(NTB, dim, a.maxK, table_smem, a.hist_smem, a.tab_len);
    float2 *table = reinterpret_cast<float2 *>(smem + sp.table);
    float *hsum = reinterpret_cast<float *>(smem + sp.hsum);
    unsigned int *hcnt = reinterpret_cast<unsigned int *>(smem + sp.hcnt);
    float *itab = reinterpret_cast<float *>(smem + sp.itab);
    float *red = reinterpret_cast<float *>(smem + sp.red);
    RangeRec *s_rec = reinterpret_cast<RangeRec *>(smem + sp.recs);
    WarpBuf &wb = reinterpret_cast<WarpBuf *>(smem + sp.warps)[warp];
    float *win_w = reinterpret_cast<float *>(wb.res);

    // ---- per-CTA setup: histogram, integrand constants; then, once the
    // allocation is done, the grid table
    const int hist = dim * W;   // the last bin of an axis takes what is not counted
    if (NEED_RED && a.train && a.hist_smem) {
        for (int i = tid; i < hist * a.hist_smem; i += NTB) hsum[i] = 0.f;
        for (int i = tid; i < hist; i += NTB) hcnt[i] = 0u;
    }
    VgF32Consts kc;
    if (MODE == MODE_FUSED || MODE == MODE_EVAL) {
        kc = vg_prepare_f32<KIND>(prm, dim);
        vg_fill_table_f32<KIND>(prm, dim, itab, kc);
    }
    if (F & RF_CHAIN) {
        vg_pdl_wait();
        vg_pdl_go();
    }
    if (a.stats->ntiles == 0) return;   // allocation failed: nothing to do
    const int64_t N = a.stats->neval;
    if (NEED_MAP && table_smem)
        for (int i = tid; i < dim * W; i += NTB) table[i] = a.tablef[i];
    __syncthreads();

    const float dv_yf = (float)a.dv_y;
    const float beta_half_f = (float)a.beta_half;
    float *my_hsum = hsum + (a.hist_smem > 1 ? (lane & (a.hist_smem - 1)) * hist : 0);
    int nan_local = 0;
    LaneSums sums = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};

    const unsigned int nchunk = (unsigned int)((N + CHUNK - 1) / CHUNK);
    const unsigned int nrec = (unsigned int)record_count(N, (int64_t)nranks * (NW / GROUP), deal);
    const unsigned int seg = rank + nranks * (warp / GROUP);   // the group's range
    unsigned int seg0 = 0, nsc = 0;                            // its chunks
    if (!deal && seg < nrec) {
        const unsigned int q = nchunk / nrec, m = nchunk - q * nrec;
        seg0 = seg * q + min(seg, m);
        nsc = q + (seg < m);
    }
    // ranges of the group's warps, or units
    const unsigned int nu = deal ? nrec : min(nsc, (unsigned int)GROUP);
    const unsigned int ustep = deal ? nranks * NW : GROUP;
    Idx h_ahead = -1;   // dealt units: the next one's first hypercube, loaded a unit ahead
    for (unsigned int u = deal ? rank + nranks * warp : warp % GROUP; u < nu; u += ustep) {
        RangeRec *rec = deal ? a.rrecs + 2 * (size_t)u : s_rec + 2 * warp;
        unsigned int c0 = u * deal, c1 = c0 + deal;
        if (!deal) {
            const unsigned int q = nsc / nu, m = nsc - q * nu;
            c0 = seg0 + u * q + min(u, m);
            c1 = c0 + q + (u < m);
        }
        const Idx s0 = (Idx)c0 * CHUNK, s1 = c1 < nchunk ? (Idx)c1 * CHUNK : (Idx)N;
        Idx h = h_ahead >= 0 ? h_ahead : (Idx)a.tile_h0[c0];
        if (deal && u + ustep < nu) h_ahead = (Idx)a.tile_h0[(u + ustep) * deal];
        bool cut0 = false, cut_first = false;   // the hypercube started before the range
        bool open = false;
        int n_open = 0;                         // samples of the open hypercube
        float c_open = 0.f;
        DQ v_open;
        v_open.zero();
        int len = CHUNK;
        for (Idx b = s0; b < s1; b += GENERAL ? len : CHUNK) {
            len = (int)(s1 - b < CHUNK ? s1 - b : CHUNK);
            if constexpr (GENERAL)
                if (a.few) {
                    const Windows w = few_windows(a, b, N, h, len);
                    h = w.h;
                    len = w.len;
                }
            // ---- the hypercubes of the chunk
            int nw = 0;
            if (lane < CHUNK / 32) wb.mask[lane] = 0u;
            __syncwarp();
            for (int q = 0; q < 3; q++) {
                const int k = 32 * q + lane;
                // below 2^31 where it is used: a hypercube has at most that many samples
                const Idx dif = (Idx)(h + k <= (Idx)a.H ? a.offsets[h + k] : N) - b;
                const int rel = GENERAL && dif > (Idx)0x7fffffff ? 0x7fffffff : (int)dif;
                const bool in = h + k < (Idx)a.H && rel < len;
                if (k < WCAP) wb.off[k] = rel;
                if (k > 0 && in && rel >= 0) atomicOr(&wb.mask[rel >> 5], 1u << (rel & 31));
                const unsigned int m = __ballot_sync(0xffffffffu, in);
                nw += __popc(m);
                if (m != 0xffffffffu) break;
            }
            if (nw < 1 || nw > WCAP - 2) {   // impossible: counts of 2 or more, or a shortened chunk
                if (lane == 0) a.stats->status = VG_ERR_UNSUPPORTED;
                break;
            }
            __syncwarp();
            for (int k = lane; k < nw; k += 32) win_w[k] = dv_yf / (float)(wb.off[k + 1] - wb.off[k]);
            __syncwarp();

            // ---- sampling: draw, map, evaluate, training histogram
            int before = 0;   // hypercube starts in the words before
#pragma unroll 1
            for (int k = 0; k < CHUNK / 32; k++) {
                // d * W formed anew for each sample: as loop invariants the axes'
                // offsets into table and histogram take 20 registers, spilled
                int Wk = W;
                asm volatile("" : "+r"(Wk));
                const int li = 32 * k + lane;
                const unsigned int m = wb.mask[k];
                const int cur = before + __popc(m & (0xffffffffu >> (31 - lane)));
                before += __popc(m);
                float wf = 0.f;
                if (li < len) {
                    const Idx ig = b + li;
                    float jac = 1.f;
                    float x[DIMB];
                    unsigned int bins[(DIMB + 3) / 4 * 2];   // training bins, 16 bits each (ninc: none)
                    if (NEED_MAP) {
                        unsigned int hh = (unsigned int)(h + cur);
                        int64_t hl = h + cur;
#pragma unroll
                        for (int g = 0; 4 * g < DIMB; g++) {
                            if (4 * g >= dim) break;
                            float u[4];
                            if (GENERAL && a.u != nullptr) {
#pragma unroll
                                for (int q = 0; q < 4; q++)
                                    u[q] = 4 * g + q < dim ? (float)a.u[(size_t)ig * dim + 4 * g + q] : 0.5f;
                            } else {
                                VgUniform<float>::group(a.seed, a.stream, a.itn, (uint64_t)ig, g, u);
                            }
                            // in the batched kernel the arguments are in shared memory:
                            // not loaded ahead for all axes, to be spilled (beside 223 KB
                            // of shared memory L1 holds few of 1024 threads' spills; with
                            // the d * W above, dim 5 to 8: 7.22 -> 6.55 ms of the bucket,
                            // dim 3 and 4: 6.66 -> 5.64)
                            if (!(F & RF_CHAIN)) asm volatile("" ::: "memory");
#pragma unroll
                            for (int q = 0; q < 4; q++) {
                                const int d = 4 * g + q;
                                if (d >= dim) {
                                    if (d < DIMB) x[d] = 0.f;
                                    if (!(d & 1)) bins[d >> 1] = 0u;
                                    continue;
                                }
                                const AxisArgs &ax = a.ax[d];
                                int y0;
                                if (!wide) {
                                    const unsigned int qh = __umulhi(hh << 1, ax.dmul) >> ax.dshift;
                                    y0 = (int)(hh - qh * (unsigned int)ax.nstrat);
                                    hh = qh;
                                } else {
                                    y0 = wide_digit(hl, ax.nstrat);
                                }
                                float yd, yn, yfl;
                                const int iy = sample_y<float>(y0, (float)y0, u[q], ax.nstrat, ax.rstrat, ax.ninc,
                                                               ax.Kf, yd, yn, yfl);
                                // y <= 1 (below 2^24 strata the product y0 + u = nstrat times 1 / nstrat
                                // rounds to 1 at most), so iy <= ninc, and at y = 1 the table's last entry
                                // has x and dy = 0.  (An ordinary load: the batched kernel rewrites
                                // the table at each iteration, and this kernel may be placed while
                                // the allocation still writes it, so the read-only path is not open.)
                                const float2 e = table_smem ? table[d * Wk + iy] : a.tablef[d * Wk + iy];
                                float dy = yn - yfl;
                                if (wide && iy >= ax.ninc) dy = 0.f;
                                if (NEED_X) x[d] = fmaf(e.y, dy, e.x);
                                jac *= e.y * ax.Kf;
                                // the training bin; y = 0 and y = 1 are not counted (pyx:460)
                                const unsigned int bin = yn > 0.f ? (unsigned int)iy : (unsigned int)ax.ninc;
                                if (d & 1) bins[d >> 1] |= bin << 16;
                                else bins[d >> 1] = bin;
                                if (MODE == MODE_POINTS && a.y_out) ((float *)a.y_out)[(size_t)ig * dim + d] = yd;
                            }
                        }
                    } else {
                        // (ordinary loads, for the kernel may be placed while the sampler writes these)
                        jac = ((const float *)a.keep_jac)[ig];
                        if (a.train) {
                            const uint2 *src = reinterpret_cast<const uint2 *>(a.keep_bins + (size_t)ig * a.keep_bstride);
#pragma unroll
                            for (int g = 0; 4 * g < DIMB; g++) {
                                if (4 * g >= dim) break;
                                const uint2 t = src[g];
                                bins[2 * g] = t.x;
                                bins[2 * g + 1] = t.y;
                            }
                        }
                    }
                    if (!(F & RF_CHAIN)) asm volatile("" ::: "memory");
                    // weight, pyx:1748-1749: jac *= dv_y / neval_hcube
                    const float wg = jac * win_w[cur];
                    if (MODE == MODE_POINTS) {
                        float *xo = (float *)a.x_out + (size_t)ig * dim;
                        if (DIMB % 4 == 0 && a.x_vec) {   // dim a multiple of 4, 16-byte aligned rows
#pragma unroll
                            for (int g = 0; 4 * g < DIMB; g++)
                                if (4 * g < dim)
                                    reinterpret_cast<float4 *>(xo)[g] =
                                        make_float4(x[4 * g], x[4 * g + 1], x[4 * g + 2], x[4 * g + 3]);
                        } else {
#pragma unroll
                            for (int d = 0; d < DIMB; d++)
                                if (d < dim) xo[d] = x[d];
                        }
                        if (a.wgt_out) a.wgt_out[ig] = (double)wg;
                        if (a.hc_out) a.hc_out[ig] = h + cur;
                        if (a.keep_jac) {
                            ((float *)a.keep_jac)[ig] = jac;
                            uint2 *dst = reinterpret_cast<uint2 *>(a.keep_bins + (size_t)ig * a.keep_bstride);
#pragma unroll
                            for (int g = 0; 4 * g < DIMB; g++)
                                if (4 * g < dim) dst[g] = make_uint2(bins[2 * g], bins[2 * g + 1]);
                        }
                    } else {
                        float f;
                        if (MODE == MODE_FUSED || MODE == MODE_EVAL)
                            f = vg_eval_f32<KIND, DIMB>(kc, itab, a.tab_len, dim, x, prm.term_count);
                        else
                            f = a.f_f64 ? (float)((const double *)a.f_in)[ig] : ((const float *)a.f_in)[ig];
                        if (MODE == MODE_EVAL) {
                            a.f_eval[ig] = f;
                        } else {
                            if (f != f) nan_local = 1;
                            wf = wg * f;
                            if (a.train) {   // fdv2 = (wgt f neval)^2 into the bins, pyx:2173, 460-463
                                const float t1 = f * (jac * dv_yf);
                                const float fd = t1 * t1;
#pragma unroll
                                for (int d = 0; d < DIMB; d++) {
                                    if (d >= dim) break;
                                    const unsigned int bin = (d & 1) ? bins[d >> 1] >> 16 : bins[d >> 1] & 0xffffu;
                                    if (!GENERAL || a.hist_smem) {
                                        atomicAdd(my_hsum + d * Wk + bin, fd);
                                        atomicAdd(hcnt + d * Wk + bin, 1u);
                                    } else if (bin < (unsigned int)a.ax[d].ninc) {
                                        atomicAdd(&a.sum_f[d * a.ldi + bin], (double)fd);
                                        atomicAdd(&a.n_f[d * a.ldi + bin], 1ull);
                                    }
                                }
                            }
                        }
                    }
                }
                if (NEED_RED) wb.wf[li] = wf;
            }
            __syncwarp();
            if (b == s0) cut_first = cut0 = wb.off[0] < 0;
            const bool ended = wb.off[nw] == len;   // the chunk's last hypercube ends with it
            const int nfin = ended ? nw : nw - 1;
            if (NEED_RED) {
                // ---- (D, Q) of the lane's runs of equal hypercube
                if (!open) {   // nothing carried: a cut first hypercube counts from here
                    c_open = wb.wf[0];
                    v_open.zero();
                }
                const float4 x4 = reinterpret_cast<const float4 *>(wb.wf)[lane];
                const float xv[4] = {x4.x, x4.y, x4.z, x4.w};
                const unsigned int mw = wb.mask[lane >> 3];
                const unsigned int nib = (mw >> ((lane & 7) * 4)) & 15u;
                int kcur = __popc(mw & ((2u << ((lane & 7) * 4)) - 1u));
                for (int q = 0; q < (lane >> 3); q++) kcur += __popc(wb.mask[q]);
                const int nv = len - 4 * lane;
                const int o0 = wb.off[kcur];
                float c = o0 < 0 ? c_open : wb.wf[o0];
                DQ v, vfirst;
                v.zero();
                if (lane == 0) {
                    v = v_open;
                    wb.res[OPEN] = make_float4(v.dh, v.dl, v.qh, v.ql);
                }
                bool started = lane == 0 || (nib & 1u);
                int kfirst = -1;
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    if (j > 0 && (nib >> j & 1u)) {   // a hypercube ends, the next starts
                        if (started) {
                            wb.res[kcur] = make_float4(v.dh, v.dl, v.qh, v.ql);
                        } else {
                            vfirst = v;
                            kfirst = kcur;
                        }
                        started = true;
                        kcur++;
                        c = xv[j];
                        v.zero();
                    }
                    if (j < nv) v.add(xv[j], c);
                }
                // ---- the pieces of a hypercube across lanes: segmented scan
                // of the lanes' last runs, as many steps as the longest
                // hypercube of the chunk needs
                const unsigned int heads = __ballot_sync(0xffffffffu, started);
                const int dist = lane - (31 - __clz(heads & (0xffffffffu >> (31 - lane))));
                const int maxd = __reduce_max_sync(0xffffffffu, nv > 0 ? dist : 0);
                for (int off = 1; off <= maxd; off <<= 1) {
                    const DQ o = v.up(off);
                    if (dist >= off) v.add(o);
                }
                const DQ prev = v.up(1);
                if (kfirst >= 0) {
                    vfirst.add(prev);
                    wb.res[kfirst] = make_float4(vfirst.dh, vfirst.dl, vfirst.qh, vfirst.ql);
                }
                const int last = (len - 1) >> 2;
                const bool next_head = __shfl_down_sync(0xffffffffu, nib, 1) & 1u;
                if (lane < last ? next_head : (lane == last && ended))
                    wb.res[kcur] = make_float4(v.dh, v.dl, v.qh, v.ql);
                const DQ v_next = v.from(last);
                const float c_next = __shfl_sync(0xffffffffu, c, last);
                __syncwarp();
                // ---- the hypercubes that end here, one lane each
                for (int k = lane; k < nfin; k += 32) {
                    const float4 t = wb.res[k];
                    DQ q = {t.x, t.y, t.z, t.w};
                    const int o = wb.off[k], oe = wb.off[k + 1];
                    float ck = o < 0 ? c_open : wb.wf[o];
                    if (k == 0 && cut0) {
                        const int n = (int)(b + oe - s0);
                        if (!(fabsf(q.qh) < BIG_Q)) {
                            ck = recentre_big(wb, o, oe, n, ck);
                            q = DQ{wb.res[OPEN].x, wb.res[OPEN].y, wb.res[OPEN].z, wb.res[OPEN].w};
                        }
                        rec[0] = RangeRec{h, n, ck, q.dh, q.dl, q.qh, q.ql};
                    } else {
                        finish_hcube(a, h + k, wb, o, oe, ck, q, beta_half_f, sums);
                    }
                }
                if (nfin > 0) cut0 = false;   // its first piece is recorded
                open = !ended;
                n_open = len - wb.off[nw - 1];
                v_open = v_next;
                c_open = c_next;
                if (open && !(fabsf(v_next.qh) < BIG_Q)) {
                    if (lane == 0)
                        c_open = recentre_big(wb, wb.off[nw - 1], len, cut0 ? (int)(b + len - s0) : n_open, c_next);
                    __syncwarp();
                    const float4 t = wb.res[OPEN];
                    v_open = DQ{t.x, t.y, t.z, t.w};
                    c_open = __shfl_sync(0xffffffffu, c_open, 0);
                }
            }
            h += nfin;
            __syncwarp();
        }
        if (NEED_RED && lane == 0) {   // records of the hypercubes cut by the range
            const bool spans = open && cut0;
            const DQ &v = v_open;
            if (spans) rec[0] = RangeRec{h, -(int)(s1 - s0), c_open, v.dh, v.dl, v.qh, v.ql};
            else if (!cut_first) rec[0].h = -1;
            if (open && !spans) rec[1] = RangeRec{h, n_open, c_open, v.dh, v.dl, v.qh, v.ql};
            else rec[1].h = -1;
        }
    }

    // ---- epilogue: the CTA's partial sums, NaN flag, histogram flush
    if (NEED_RED) {
        if (nan_local) atomicExch((int *)&a.stats->nan_seen, 1);
        float r6[6] = {sums.mh, sums.ml, sums.vh, sums.vl, sums.sh, sums.sl};
        if (!deal) {
            __syncthreads();
            if (warp % GROUP == 0 && nu > 0) {   // lane l joins the pieces of the l-th warp's range with those before it
                RangeRec H, T;
                H.h = T.h = -1;
                if (lane < (int)nu) {
                    H = s_rec[2 * (warp + lane)];
                    T = s_rec[2 * (warp + lane) + 1];
                }
                Piece cur = {0.f, 0.f, 0.f, 0.f, 0.f}, end = cur;
                const bool h_spans = H.h >= 0 && H.n < 0, h_ends = H.h >= 0 && H.n > 0;
                if (h_spans) cur.from(H);
                if (h_ends) end.from(H);
                if (T.h >= 0) cur.from(T);
                const bool inside = scan_pieces(cur, !h_spans);
                const Piece prev = cur.up(1);
                const bool prev_inside = __shfl_up_sync(0xffffffffu, (int)inside, 1) && lane > 0;
                if (h_ends) {   // a hypercube begun earlier ends in this lane's range
                    if (lane > 0) end.put_first(prev);
                    if (prev_inside) finish_cut(a, H.h, end, r6);
                    else a.rrecs[2 * (size_t)seg] = end.record(H.h, false);
                }
                const unsigned int wrote = __ballot_sync(0xffffffffu, h_ends && !prev_inside);
                if (lane == (int)nu - 1) {   // what is open at the end of the CTA's range
                    const bool spans = h_spans && !inside;
                    const RangeRec o = cur.record(T.h >= 0 ? T.h : H.h, spans);
                    if (spans) a.rrecs[2 * (size_t)seg] = o;
                    else if (!wrote) a.rrecs[2 * (size_t)seg].h = -1;
                    if (!spans && (T.h >= 0 || h_spans)) a.rrecs[2 * (size_t)seg + 1] = o;
                    else a.rrecs[2 * (size_t)seg + 1].h = -1;
                }
            }
        }
        ff_block_reduce6(r6, red);   // a fixed order; its barriers also end the histogram
        if (tid == 0) {
            TilePart p;
            p.mean = VgKSum{ff_pack(r6[0], r6[1]), 0.0};
            p.var = VgKSum{ff_pack(r6[2], r6[3]), 0.0};
            p.sigf = VgKSum{ff_pack(r6[4], r6[5]), 0.0};
            a.parts[rank] = p;
        }
        if (a.train && a.hist_smem) {
            for (int d = 0; d < dim; d++) {
                const int K = a.ninc[d];
                for (int i = tid; i < K; i += NTB) {
                    const unsigned int cnt = hcnt[d * W + i];
                    if (!cnt) continue;
                    float s = 0.f;
                    for (int q = 0; q < a.hist_smem; q++) s += hsum[q * hist + d * W + i];
                    atomicAdd(&a.sum_f[d * a.ldi + i], (double)s);
                    atomicAdd(&a.n_f[d * a.ldi + i], (unsigned long long)cnt);
                }
            }
        }
    }
}

// ---------------------------------------------------------------- finalize
// The iteration's sums by one CTA: the partial sums of the ncta reduction CTAs
// (ngroups groups of warps) and the hypercubes cut by the ends of their ranges (or of the dealt units).
// Each thread takes consecutive records and joins the pieces in them one after
// the other; a segmented scan joins those of a hypercube that goes on through
// several threads' records, so the time follows the logarithm of its length.
// Sums in a fixed order; valid in thread 0.
__device__ __forceinline__ void finalize_ranges(const IterArgs &a, int ncta, int64_t ngroups, int deal,
                                                float (&s6)[6])
{
    __shared__ Piece s_last[32];
    __shared__ int s_head[32];
    __shared__ float s_red[6 * 32];
    const int NTB = (int)blockDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const vg_stats *st = a.stats;
    const int64_t R = st->ntiles ? record_count(st->neval, ngroups, deal) : 0;
#pragma unroll
    for (int i = 0; i < 6; i++) s6[i] = 0.f;
    if (R > 0)
        for (int i = tid; i < ncta; i += NTB) {
            const TilePart p = a.parts[i];
            float h, l;
            ff_unpack(p.mean.s, h, l);
            ff_add_pair(s6[0], s6[1], h, l);
            ff_unpack(p.var.s, h, l);
            ff_add_pair(s6[2], s6[3], h, l);
            ff_unpack(p.sigf.s, h, l);
            ff_add_pair(s6[4], s6[5], h, l);
        }
    const int64_t per = (R + NTB - 1) / NTB;
    const int64_t t0 = tid * per, t1 = t0 + per < R ? t0 + per : R;
    Piece cur = {0.f, 0.f, 0.f, 0.f, 0.f}, first = cur;   // the open piece; the end of one begun earlier
    int64_t hfirst = -1;
    bool started = t0 >= t1;   // what is open (if anything) began in this thread
    for (int64_t t = t0; t < t1; t++) {
        const RangeRec H = a.rrecs[2 * t], T = a.rrecs[2 * t + 1];
        if (H.h >= 0) {
            Piece p;
            p.from(H);
            p.put_first(cur);
            cur = p;
            if (H.n > 0) {
                if (started) {
                    finish_cut(a, H.h, cur, s6);
                } else {
                    first = cur;
                    hfirst = H.h;
                    started = true;
                }
                cur.n = 0.f;
            }
        } else if (t == t0) {
            started = true;   // nothing comes in from before
        }
        if (T.h >= 0) {
            cur.from(T);
            started = true;
        }
    }
    // open pieces across the lanes, then across the warps
    const bool inside = scan_pieces(cur, started);
    if (lane == 31) {
        s_last[warp] = cur;
        s_head[warp] = inside;
    }
    __syncthreads();
    Piece carry = {0.f, 0.f, 0.f, 0.f, 0.f};
    if (warp > 0) {
        carry = s_last[warp - 1];
        for (int w = warp - 1; w > 0 && !s_head[w]; w--) carry.put_first(s_last[w - 1]);
    }
    if (!inside) cur.put_first(carry);
    Piece prev = cur.up(1);
    if (lane == 0) prev = carry;
    if (hfirst >= 0) {
        first.put_first(prev);
        finish_cut(a, hfirst, first, s6);
    }
    ff_block_reduce6(s6, s_red);
}

// ---------------------------------------------------------------- launcher
// Threads per CTA (one CTA per SM) by dimension: as many as the registers of
// one sample's coordinates leave.
__host__ __device__ constexpr int range_threads(int dimb) { return dimb <= 8 ? 1024 : (dimb <= 16 ? 768 : 256); }

template <int MODE, int KIND, int DIMB, int F>
__global__ void __launch_bounds__(range_threads(DIMB), 1)
range_kernel(const __grid_constant__ IterArgs a, const __grid_constant__ VgParams prm)
{
    extern __shared__ __align__(16) unsigned char smem[];
    range_body<MODE, KIND, DIMB, F | RF_CHAIN>(a, prm, smem, blockIdx.x, gridDim.x, 0);
}

// Shared memory of a CTA: the histogram comes first (its copies spread the
// lanes' colliding float adds, which are compare-and-swap loops: 53 cycles
// per warp-wide add on 50 bins, 15 on 1000), then the grid table, then up to 8
// copies of the histogram.
inline RangePlan range_fit(int ntb, int dim, int maxK, int tab_len, int train, int want_table, size_t budget,
                           int *table_smem, int *hist_copies)
{
    int hc = train ? 1 : 0, tb = want_table ? 1 : 0;
    RangePlan p = range_plan(ntb, dim, maxK, tb, hc, tab_len);
    if (p.total > budget && tb) p = range_plan(ntb, dim, maxK, tb = 0, hc, tab_len);
    if (p.total > budget && hc) p = range_plan(ntb, dim, maxK, tb, hc = 0, tab_len);
    while (hc > 0 && hc < 8) {
        const RangePlan q = range_plan(ntb, dim, maxK, tb, 2 * hc, tab_len);
        if (q.total > budget) break;
        hc *= 2;
        p = q;
    }
    *table_smem = tb;
    *hist_copies = hc;
    return p;
}

constexpr size_t RANGE_SMEM = 220 * 1024;

template <int MODE, int KIND, int DIMB, int F>
int launch_range_as(IterArgs &a, const VgParams *prm, size_t smem, cudaStream_t st)
{
    constexpr int NTB = range_threads(DIMB);
    auto kern = range_kernel<MODE, KIND, DIMB, F>;
    static std::atomic<uint64_t> attr{0};   // devices where it is set: once per kernel, always the largest
    int dev = 0;
    VG_CUDA_CHECK(cudaGetDevice(&dev));
    const uint64_t bit = 1ull << (dev & 63);
    if (!(attr.load(std::memory_order_relaxed) & bit)) {
        VG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RANGE_SMEM));
        if (dev < 64) attr.fetch_or(bit, std::memory_order_relaxed);
    }
    // one CTA per SM, fewer where there are fewer chunks
    int64_t grid = vg_num_sms();
    const int64_t chunks = (a.ncap + CHUNK - 1) / CHUNK;
    if (grid > chunks) grid = chunks;
    if (grid < 1) grid = 1;
    a.ncta = (int)grid;
    a.ngroups = grid * (NTB / 32 / GROUP);
    static const VgParams empty = {};
    VG_CUDA_CHECK(vg_launch_pdl(kern, (unsigned)grid, NTB, smem, st, a, prm ? *prm : empty));
    return VG_OK;
}

// The body for this iteration: by exact dimension to 8, where most of the work
// of low-dimensional integrals is per axis; above that by the run-time one.
template <int MODE, int KIND>
int launch_range(IterArgs &a, const VgParams *prm, int tab_len, cudaStream_t st)
{
    constexpr bool NEED_RED = (MODE == MODE_REDUCE || MODE == MODE_FUSED || MODE == MODE_REDUCE_KEPT);
    constexpr bool NEED_MAP = MODE != MODE_REDUCE_KEPT;
    constexpr int T = RF_TABLE, ET = RF_EXACT | RF_TABLE, G = RF_GENERAL;
    a.tab_len = tab_len;
    const int train = NEED_RED && a.train && g_tile_hist != 0;
    const RangePlan p = range_fit(range_threads(a.dim), a.dim, a.maxK, tab_len, train, NEED_MAP && g_tile_table != 0,
                                  RANGE_SMEM, &a.table_smem, &a.hist_smem);
    if (p.total > RANGE_SMEM) return vg_fail(VG_ERR_UNSUPPORTED, "shared memory plan too large");
    if ((!NEED_MAP || a.u == nullptr) && !a.wide && !a.few && (!NEED_RED || !a.train || a.hist_smem)) {
        if (!NEED_MAP || a.table_smem) {
            switch (a.dim) {
            case 1: return launch_range_as<MODE, KIND, 1, ET>(a, prm, p.total, st);
            case 2: return launch_range_as<MODE, KIND, 2, ET>(a, prm, p.total, st);
            case 3: return launch_range_as<MODE, KIND, 3, ET>(a, prm, p.total, st);
            case 4: return launch_range_as<MODE, KIND, 4, ET>(a, prm, p.total, st);
            case 5: return launch_range_as<MODE, KIND, 5, ET>(a, prm, p.total, st);
            case 6: return launch_range_as<MODE, KIND, 6, ET>(a, prm, p.total, st);
            case 7: return launch_range_as<MODE, KIND, 7, ET>(a, prm, p.total, st);
            case 8: return launch_range_as<MODE, KIND, 8, ET>(a, prm, p.total, st);
            }
            if (a.dim <= 16) return launch_range_as<MODE, KIND, 16, T>(a, prm, p.total, st);
        }
        if constexpr (NEED_MAP)
            if (a.dim > 8 && a.dim <= 16) return launch_range_as<MODE, KIND, 16, 0>(a, prm, p.total, st);
    }
    // (64 takes every dimension: the reduction of kept samples has little per axis)
    if constexpr (NEED_MAP) {
        if (a.dim <= 8) return launch_range_as<MODE, KIND, 8, G>(a, prm, p.total, st);
        if (a.dim <= 16) return launch_range_as<MODE, KIND, 16, G>(a, prm, p.total, st);
    }
    return launch_range_as<MODE, KIND, 64, G>(a, prm, p.total, st);
}

}  // namespace vg
