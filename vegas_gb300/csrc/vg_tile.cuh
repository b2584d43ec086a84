// vg_tile.cuh -- the FP64 tile kernel of a vegas+ iteration, and what it
// shares with the FP32 kernel (vg_range.cuh).
//
// Reference: src/vegas/_vegas.pyx (vegas 6.4.1): sampling and map of
// Integrator._random_batch (pyx:1731-1752), the per-hypercube two-pass
// reduction of Integrator.__call__ (pyx:2136-2193), the training feed
// (pyx:2173, 2196-2197 -> AdaptiveMap.add_training_data pyx:421-464).
//
// Samples of an iteration are ordered by hypercube (as in the reference).  A
// tile is NTB*S consecutive samples; thread t owns samples [t*S, t*S+S) of the
// tile.  Reduction modes assign tiles to CTAs statically, the others take them
// from an atomic counter; everything a tile produces is indexed by the tile.
//
// Template parameters: DIMB is a compile-time bound on the dimension (arrays
// stay in registers); S samples per thread; NTB threads per CTA; MODE points /
// reduce / fused; KIND the built-in integrand of the fused mode.
#pragma once
#include <math.h>
#include <string.h>

#include "vg_common.cuh"
#include "vg_integrands.cuh"

namespace vg {

constexpr int NT = 256;          // threads per CTA of the large FP64 tiles
constexpr int BASE_TILE = 128;   // granularity of the tile schedule tile_h0[]
constexpr int MAX_PARTS = 4096;  // partial sums of an iteration (one per CTA)
#define VG_WAIT_ITERS_DEFAULT (1u << 24)   // polls of a bounded wait (vg_set_wait_budget)
extern uint32_t g_wait_iters;
constexpr int ALLOC_NT = 256;    // allocation count / offsets blocks
constexpr int ALLOC_PER = 4;     // hypercubes per thread there

// POINTS: write points for a torch integrand (optionally also keep each
// sample's Jacobian and training bins); REDUCE: read f and reduce,
// regenerating each sample; REDUCE_KEPT: read f and the kept Jacobians and
// bins and reduce (no Philox, no map: a stream over HBM); FUSED: evaluate a
// built-in integrand and reduce in one kernel; EVAL: evaluate a built-in
// integrand and write f (first half of the split path used for expensive
// integrands, followed by a REDUCE launch).
enum { MODE_POINTS = 0, MODE_REDUCE = 1, MODE_FUSED = 2, MODE_EVAL = 3, MODE_REDUCE_KEPT = 4 };

// FP64: partial statistics of a hypercube cut by a tile boundary.
struct TileRec {
    int64_t h;       // hypercube, -1 if the slot is empty
    double n;        // samples of h inside the tile
    double S;        // sum of wf
    double Q;        // sum of squared deviations about S/n (EPSILON-guarded)
    double D;        // sum of deviations (round-off residue: Neely correction)
    int32_t spans;   // head slot only: h also continues past the tile
    int32_t pad;
};

// FP32: a piece of a hypercube cut by the end of a range: n samples (-n where it
// also continues past the range), the sums D of wf - c and Q of their squares in
// float-float; with c = NaN, D is the sum of wf and Q that about the mean.
struct __align__(16) RangeRec {
    int64_t h;       // hypercube, -1 if the slot is empty
    int32_t n;
    float c, dh, dl, qh, ql;
};

struct TilePart {
    VgKSum mean, var, sigf;
};

// One axis for the FP32 sampler: strata and increments as it uses them.  h / nstrat
// = umulhi(2 h, dmul) >> dshift for h < 2^31.
struct __align__(16) AxisArgs {
    unsigned int dmul;
    int dshift, nstrat, ninc;
    float rstrat, Kf;         // 1 / nstrat, ninc
    float pad[2];
};

struct IterArgs {
    int dim;
    int nstrat[VG_MAX_DIM];
    int ninc[VG_MAX_DIM];
    const double *grid, *inc;
    int64_t ldg, ldi;
    int64_t H;
    int64_t ncap;
    double *sigf;
    double beta;
    int adaptive;             // update sigf (pyx:2083, 2183-2186)
    int adaptive_alloc;       // allocate from sigf (pyx:1668)
    int train;                // accumulate training histogram (pyx:2196)
    int train_hc;             // adapt_to_errors: train on each hypercube's variance (pyx:2187-2193)
    double *sum_f;
    unsigned long long *n_f;
    vg_stats *stats;
    int32_t *neval_h;
    int64_t *offsets;
    int64_t *bsum;            // allocation: published block totals / prefixes
    int64_t *tile_h0;         // first hypercube of each BASE_TILE samples
    unsigned long long *counter;  // dynamic tile counter (reset by allocation)
    unsigned int *fin_counter;    // finalize blocks done (reset by allocation)
    unsigned int *alloc_sync;     // single-pass allocation: ticket, epoch, error, count maximum
    TileRec *recs;            // two per FP64 tile
    RangeRec *rrecs;          // FP32: two per CTA or dealt unit (the same memory)
    TilePart *parts;
    int64_t ntiles_cap;       // in BASE_TILE units
    AxisArgs ax[VG_MAX_DIM];  // FP32: what a sample needs of each axis
    int wide;                 // FP32: 2^31 hypercubes or samples or more, or 2^24 strata on an axis
    int x_vec;                // MODE_POINTS: rows of x are 16-byte aligned multiples of 16 bytes
    int64_t neval;
    double neval_frac;
    int64_t min_neval_hcube, max_neval_hcube;
    uint64_t seed;
    uint32_t stream;
    uint32_t itn;
    const double *u;          // injected uniforms [n, dim] or nullptr
    const void *f_in;         // MODE_REDUCE, MODE_REDUCE_KEPT
    void *keep_jac;           // per-sample Jacobian (T): written by MODE_POINTS when set, read by REDUCE_KEPT
    unsigned short *keep_bins;   // per-sample training bins [n, keep_bstride] (0xffff: none), likewise
    int keep_bstride;            // bins per kept sample: dim rounded up to 4 (8-byte aligned rows)
    int f_f64;
    void *x_out, *y_out;      // MODE_POINTS
    float *f_eval;            // MODE_EVAL output / MODE_REDUCE input of the split path
    TilePart *part2;          // finalize: one partial per finalize block
    double *wgt_out;
    int64_t *hc_out;
    float2 *tablef;           // FP32 mode: (x_node, inc) table [dim][maxK+1], built by the allocation
    int table_smem;           // grid table staged in shared memory
    int hist_smem;            // training histogram in shared memory (FP32: copies of it)
    int maxK;
    int tab_len;              // integrand table length (floats)
    int T;                    // tile size of the launched kernel
    int ncta;                 // CTAs of the launched reduction kernel (one partial each)
    int64_t ngroups;          // FP32: groups of warps of that kernel (two records each)
    double dv_y;              // 1 / nhcube (pyx:1639)
    double beta_half;         // beta / 2 (pyx:2185)
    uint32_t wait_iters;      // polls of a bounded wait before it gives up (vg_set_wait_budget)
    int few;                  // hypercubes may have fewer than two samples
};

struct SmemPlan {
    size_t table, hsum, hcnt, bins, win_off, win_n, seg_S, keyF, keyL, P, red, total;
};

template <int NTB>
__host__ __device__ inline SmemPlan smem_plan(int dim, int maxK, int Ttile, int table_smem,
                                              int hist_smem, int bins_smem, int need_red)
{
    SmemPlan p;
    size_t o = 0;
    p.table = o;
    if (table_smem) o = (o + sizeof(double2) * (size_t)dim * (maxK + 1) + 15) & ~(size_t)15;
    p.hsum = o;
    if (hist_smem) o = (o + sizeof(double) * (size_t)dim * maxK + 15) & ~(size_t)15;
    p.hcnt = o;
    if (hist_smem) o = (o + sizeof(unsigned int) * (size_t)dim * maxK + 15) & ~(size_t)15;
    p.bins = o;
    if (bins_smem) o = (o + sizeof(unsigned short) * (size_t)Ttile * dim + 15) & ~(size_t)15;
    p.win_off = o; o = (o + sizeof(int) * (Ttile + 2) + 15) & ~(size_t)15;
    p.win_n = o;   o = (o + sizeof(int) * (Ttile + 2) + 15) & ~(size_t)15;
    p.seg_S = o;   if (need_red) o = (o + sizeof(double) * (Ttile + 2) + 15) & ~(size_t)15;
    p.keyF = o;    if (need_red) o = (o + sizeof(int) * NTB + 15) & ~(size_t)15;
    p.keyL = o;    if (need_red) o = (o + sizeof(int) * NTB + 15) & ~(size_t)15;
    p.P = o;       if (need_red) o = (o + sizeof(double2) * NTB + 15) & ~(size_t)15;
    p.red = o;     if (need_red) o = (o + sizeof(VgKSum) * (NTB / 32) * 3 + 64 + 15) & ~(size_t)15;
    p.total = o;
    return p;
}

// Block-wide exclusive prefix sum of one int64 per thread (warp shuffles,
// then a scan of the warp totals); *total = the block's sum.
__device__ __forceinline__ int64_t block_excl_scan(int64_t v, int64_t *wtot /* one per warp */, int64_t *total)
{
    const int NW = (int)blockDim.x >> 5;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int64_t x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x += y;
    }
    if (lane == 31) wtot[w] = x;
    __syncthreads();
    if (w == 0) {
        int64_t z = lane < NW ? wtot[lane] : 0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, z, off);
            if (lane >= off) z += y;
        }
        if (lane < NW) wtot[lane] = z;
    }
    __syncthreads();
    *total = wtot[NW - 1];
    const int64_t r = (w > 0 ? wtot[w - 1] : 0) + x - v;
    __syncthreads();
    return r;
}

__device__ __forceinline__ int64_t block_max(int64_t v, int64_t *wtot /* one per warp */)
{
    const int NW = (int)blockDim.x >> 5;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const int64_t o = __shfl_xor_sync(0xffffffffu, v, off);
        v = o > v ? o : v;
    }
    if (lane == 0) wtot[w] = v;
    __syncthreads();
    int64_t m = wtot[0];
    for (int i = 1; i < NW; i++) m = wtot[i] > m ? wtot[i] : m;
    __syncthreads();
    return m;
}

// Inclusive segmented scan over the NTB threads of (flag, value2); the result
// for thread t is returned and stored in P[t].
template <int NTB>
__device__ __forceinline__ double2 seg_scan(int flag, double2 v, double2 *P, double2 *wsum,
                                            int *wflag)
{
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int f = flag;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        double ux = __shfl_up_sync(0xffffffffu, v.x, off);
        double uy = __shfl_up_sync(0xffffffffu, v.y, off);
        int uf = __shfl_up_sync(0xffffffffu, f, off);
        if (lane >= off) {
            if (!f) {
                v.x = ux + v.x;
                v.y = uy + v.y;
            }
            f |= uf;
        }
    }
    if (lane == 31) {
        wsum[w] = v;
        wflag[w] = f;
    }
    __syncthreads();
    if (w == 0) {
        const int NW = NTB / 32;
        double2 x = lane < NW ? wsum[lane] : make_double2(0.0, 0.0);
        int g = lane < NW ? wflag[lane] : 1;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            double ux = __shfl_up_sync(0xffffffffu, x.x, off);
            double uy = __shfl_up_sync(0xffffffffu, x.y, off);
            int ug = __shfl_up_sync(0xffffffffu, g, off);
            if (lane >= off) {
                if (!g) {
                    x.x = ux + x.x;
                    x.y = uy + x.y;
                }
                g |= ug;
            }
        }
        if (lane < NW) wsum[lane] = x;
    }
    __syncthreads();
    if (w > 0 && !f) {
        double2 c = wsum[w - 1];
        v.x = c.x + v.x;
        v.y = c.y + v.y;
    }
    P[threadIdx.x] = v;
    __syncthreads();
    return v;
}

// (ah, al) += (bh, bl) in float-float (TwoSum of the heads, tails added,
// renormalised): the FP32 mode's sums.
__device__ __forceinline__ void ff_add_pair(float &ah, float &al, float bh, float bl)
{
    const float s = __fadd_rn(ah, bh);
    const float bb = __fsub_rn(s, ah);
    float e = __fadd_rn(__fsub_rn(ah, __fsub_rn(s, bb)), __fsub_rn(bh, bb));
    e = __fadd_rn(e, __fadd_rn(al, bl));
    ah = __fadd_rn(s, e);
    al = __fsub_rn(e, __fsub_rn(ah, s));
}

// FP32 mode keeps float-float values in the FP64 fields of the tile records
// and partial sums as bit patterns (low word = head, high word = tail), so
// storing and loading them moves integers -- GB300's FP64 pipe is slow, and
// a single warp waits hundreds of cycles per dependent FP64 instruction.
__device__ __forceinline__ double ff_pack(float h, float l)
{
    return __hiloint2double(__float_as_int(l), __float_as_int(h));
}

__device__ __forceinline__ void ff_unpack(double d, float &h, float &l)
{
    h = __int_as_float(__double2loint(d));
    l = __int_as_float(__double2hiint(d));
}

// Block-wide float-float reduction of six floats (three float-float values)
// in a fixed order; the result is valid in thread 0.  scratch: 6 floats per
// warp of shared memory.
__device__ __forceinline__ void ff_warp_reduce6(float (&r6)[6])
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        float o6[6];
#pragma unroll
        for (int i = 0; i < 6; i++) o6[i] = __shfl_down_sync(0xffffffffu, r6[i], off);
#pragma unroll
        for (int i = 0; i < 6; i += 2) ff_add_pair(r6[i], r6[i + 1], o6[i], o6[i + 1]);
    }
}

__device__ __forceinline__ void ff_block_reduce6(float (&r6)[6], float *scratch)
{
    const int tid = threadIdx.x;
    ff_warp_reduce6(r6);
    if ((tid & 31) == 0) {
#pragma unroll
        for (int i = 0; i < 6; i++) scratch[(tid >> 5) * 6 + i] = r6[i];
    }
    __syncthreads();
    if (tid < 32) {
#pragma unroll
        for (int i = 0; i < 6; i++) r6[i] = tid < (int)blockDim.x >> 5 ? scratch[tid * 6 + i] : 0.f;
        ff_warp_reduce6(r6);
    }
    __syncthreads();
}

// (h, l) = (ah, al) * b in float-float (the head's product error by fma).
__device__ __forceinline__ void ff_mul_f(float ah, float al, float b, float &h, float &l)
{
    const float p = __fmul_rn(ah, b);
    float e = __fmaf_rn(ah, b, -p);
    e = __fmaf_rn(al, b, e);
    h = __fadd_rn(p, e);
    l = __fsub_rn(e, __fsub_rn(h, p));
}

// (h, l) = (ah, al) * (bh, bl) in float-float.
__device__ __forceinline__ void ff_mul(float ah, float al, float bh, float bl, float &h, float &l)
{
    const float p = __fmul_rn(ah, bh);
    float e = __fmaf_rn(ah, bh, -p);
    e = __fmaf_rn(ah, bl, e);
    e = __fmaf_rn(al, bh, e);
    h = __fadd_rn(p, e);
    l = __fsub_rn(e, __fsub_rn(h, p));
}

// A double as float-float (exact when it came from one).
__device__ __forceinline__ void ff_from_double(double x, float &h, float &l)
{
    h = (float)x;
    l = (float)(x - (double)h);
}

// (h, l) = (ah, al)^2 in float-float.
__device__ __forceinline__ void ff_sqr(float ah, float al, float &h, float &l)
{
    const float p = __fmul_rn(ah, ah);
    float e = __fmaf_rn(ah, ah, -p);
    e = __fmaf_rn(__fmul_rn(2.f, ah), al, e);
    h = __fadd_rn(p, e);
    l = __fsub_rn(e, __fsub_rn(h, p));
}

// (h, l) = (ah, al) / b in float-float, b a count: head quotient, its remainder by
// fma, one correction term.  The reciprocal is the correctly rounded one, by a Newton
// step on the special-function unit's (as that is, to an ulp, the quotient's error is up
// to twice as large).  The step gives __frcp_rn's bits for every count below 2^31, and
// __frcp_rn itself, whose path is for all floats, took 2 % of the dim-4 ridge's call.
__device__ __forceinline__ void ff_div_f(float ah, float al, float b, float &h, float &l)
{
    float rb;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rb) : "f"(b));
    rb = __fmaf_rn(rb, __fmaf_rn(-b, rb, 1.f), rb);
    const float q1 = __fmul_rn(ah, rb);
    const float r = __fadd_rn(__fmaf_rn(-q1, b, ah), al);
    const float q2 = __fmul_rn(r, rb);
    h = __fadd_rn(q1, q2);
    l = __fsub_rn(q2, __fsub_rn(h, q1));
}

// a / b in double for the FP32 mode's rare FP64 paths: a reciprocal multiply
// refined by one Newton step (GB300 FP64 division is expensive).
__device__ __forceinline__ double vg_div_fast(double a, double b)
{
    double r = (double)__frcp_rn((float)b);
    r = fma(r, fma(-b, r, 1.0), r);
    return a * r;
}

// One sample's y along one axis and its map increment index (pyx:1738-1742,
// 325-330): yd = (y0 + u) / nstrat, yn = yd * K, iy = floor(yn); yfl = the
// floor as T.  FP32 mode: the reciprocal of nstrat and K as float are given,
// the floor's integer comes from the float's bits (0 <= yn < 2^23): no
// float -> int conversion.
template <typename T>
__device__ __forceinline__ int sample_y(int y0, float y0f, T u, int ns, float rns, int K, float Kf, T &yd,
                                        T &yn, T &yfl)
{
    int iy;
    if (sizeof(T) == 8) {
        yd = (T)__ddiv_rn(__dadd_rn((double)y0, (double)u), (double)ns);
        yn = (T)__dmul_rn((double)yd, (double)K);
        iy = (int)floor((double)yn);
        yfl = (T)iy;
    } else {
        yd = (T)__fmul_rn(__fadd_rn(y0f, (float)u), rns);
        yn = (T)__fmul_rn((float)yd, Kf);
        const float fl = floorf((float)yn);
        iy = __float_as_int(fl + 8388608.f) - 0x4B000000;
        yfl = (T)fl;
    }
    return iy;
}

// Training bin of a sample along one axis: its increment, or 0xffff when y
// is 0 or 1 (add_training_data skips those, pyx:460).
template <typename T>
__device__ __forceinline__ unsigned short sample_bin(T yd, int iy, int K)
{
    return (unsigned short)((yd > (T)0 && yd < (T)1 && iy < K) ? iy : 0xffff);
}

// adapt_to_errors: the hypercube's |variance| into the training histogram
// at its last sample's bins, count 1 (pyx:2187-2193).
__device__ __forceinline__ void train_hcube(const IterArgs &a, const unsigned short *bins, double v)
{
    for (int d = 0; d < a.dim; d++) {
        const unsigned short b = bins[d];
        if (b == 0xffff) continue;
        atomicAdd(&a.sum_f[d * a.ldi + b], v);
        atomicAdd(&a.n_f[d * a.ldi + b], 1ull);
    }
}

// The training bins of hypercube h's last sample, regenerated from its
// uniforms exactly as the tile kernels form them (for hypercubes that the
// finalize merges across tiles).
template <typename T>
static __device__ __noinline__ void last_sample_bins(const IterArgs &a, int64_t h, unsigned short *bins)
{
    const int dim = a.dim;
    const int64_t ig = a.offsets[h] + a.neval_h[h] - 1;
    T u[VG_MAX_DIM];
    if (a.u != nullptr) {
        for (int d = 0; d < dim; d++) u[d] = (T)a.u[ig * dim + d];
    } else {
        VgUniform<T>::template draw<VG_MAX_DIM>(a.seed, a.stream, a.itn, (uint64_t)ig, dim, u);
    }
    int64_t hh = h;
    for (int d = 0; d < dim; d++) {
        const int ns = a.nstrat[d];
        const int y0 = (int)(hh % ns);
        hh /= ns;
        const int K = a.ninc[d];
        T yd, yn, yfl;
        const int iy = sample_y<T>(y0, (float)y0, u[d], ns, 1.f / (float)ns, K, (float)K, yd, yn, yfl);
        bins[d] = sample_bin<T>(yd, iy, K);
    }
}

// FP32 mode, rare path: a hypercube whose squared deviations leave the float
// range, finished in FP64.  Returns its (mean, variance, sigf) contributions
// and stores its sigf.
// (With want_var, the third value is |variance| instead: adapt_to_errors.)
static __device__ __noinline__ double3 finish_f64(double Sx, double Dx, double Qx, int nin, double beta_half,
                                                  int adaptive, double *sigf_h, int want_var)
{
    const double nd = (double)nin;
    const double vh = vg_div_fast(__dsub_rn(__dmul_rn(nd, Qx), __dmul_rn(Dx, Dx)), __dsub_rn(nd, 1.));
    double sg = 0.0;
    if (adaptive) {
        sg = vg_pow_fast(fabs(vh), beta_half);
        *sigf_h = sg;
    }
    return make_double3(__dadd_rn(Sx, Dx), vh, want_var ? fabs(vh) : sg);
}

// FP32 mode: the (x_node, inc) table of the grid in FP32, entry K of each
// axis = (grid[K], inc[K-1]) -- built once per iteration by the allocation so
// the tile CTAs copy it instead of converting FP64 nodes themselves.
__device__ __forceinline__ void build_tablef(const IterArgs &a, int64_t first, int64_t stride)
{
    const int W = a.maxK + 1;
    for (int64_t i = first; i < (int64_t)a.dim * W; i += stride) {
        const int d = (int)(i / W), j = (int)(i % W);
        const int K = a.ninc[d];
        float2 e = make_float2(0.f, 1.f);
        if (j < K) e = make_float2((float)a.grid[d * a.ldg + j], (float)a.inc[d * a.ldi + j]);
        else if (j == K) e = make_float2((float)a.grid[d * a.ldg + K], (float)a.inc[d * a.ldi + K - 1]);
        a.tablef[i] = e;
    }
}

// ------------------------------------------------------------------ kernel
// The work of one CTA: reduction modes take tiles first, first + stride, ...
// (static, deterministic); evaluation-only modes take tiles from the atomic
// counter.  The CTA's partial sums go to a.parts[part_slot].  Called by the
// grid-wide tile_kernel (first = blockIdx.x, stride = gridDim.x) and by the
// batched kernel, where G CTAs share an integral (rank, G, rank).
template <int MODE, int KIND, int DIMB, int S, int NTB>
__device__ __forceinline__ void tile_body(const IterArgs &a, const VgParams &prm, unsigned char *smem,
                                          int64_t first, int64_t stride, int64_t part_slot)
{
    constexpr int TT = NTB * S;
    constexpr int KSUB = TT / BASE_TILE;   // base tiles per tile
    const int dim = a.dim;
    const int tid = threadIdx.x;
    constexpr int NEED_RED = (MODE == MODE_REDUCE || MODE == MODE_FUSED || MODE == MODE_REDUCE_KEPT);
    const int use_bins = NEED_RED && (a.train || a.train_hc);   // per-sample bins in shared memory
    const SmemPlan sp = smem_plan<NTB>(dim, a.maxK, TT, a.table_smem, a.hist_smem, use_bins, NEED_RED);
    double2 *table = (double2 *)(smem + sp.table);
    double *hsum = (double *)(smem + sp.hsum);
    unsigned int *hcnt = (unsigned int *)(smem + sp.hcnt);
    unsigned short *sbins = (unsigned short *)(smem + sp.bins);
    int *win_off = (int *)(smem + sp.win_off);
    int *win_n = (int *)(smem + sp.win_n);
    double *seg_S = (double *)(smem + sp.seg_S);
    int *keyF = (int *)(smem + sp.keyF);
    int *keyL = (int *)(smem + sp.keyL);
    double2 *Pv = (double2 *)(smem + sp.P);
    VgKSum *red = (VgKSum *)(smem + sp.red);
    double2 *wsum = (double2 *)red;   // scan scratch (aliases red; used apart)
    int *wflag = (int *)(red + NTB / 32 + 1);
    __shared__ int64_t s_tile;

    const int64_t N = a.stats->neval;
    const int64_t ntiles = (N + TT - 1) / TT;
    const int64_t nbase = (N + BASE_TILE - 1) / BASE_TILE;
    if (a.stats->ntiles == 0) return;   // allocation failed: nothing to do

    // ---- per-CTA setup: grid table, histogram, integrand constants
    if (a.table_smem) {
        for (int d = 0; d < dim; d++) {
            const int K = a.ninc[d];
            for (int i = tid; i <= K; i += NTB)
                table[(size_t)d * (a.maxK + 1) + i] =
                    make_double2(a.grid[d * a.ldg + i], a.inc[d * a.ldi + (i < K ? i : K - 1)]);
        }
    }
    if (use_bins && a.hist_smem) {
        for (int i = tid; i < dim * a.maxK; i += NTB) {
            hsum[i] = 0.0;
            hcnt[i] = 0u;
        }
    }
    const double dv_y = a.dv_y;
    const double beta_half = a.beta_half;
    int nan_local = 0;
    // per-thread running sums over every hypercube this thread finalises
    double acc_m = 0.0, acc_v = 0.0, acc_s = 0.0;
    // The running sums -> one compensated block reduction in a fixed order ->
    // a.parts[slot]; the sums restart from zero.
    auto emit_partial = [&](int64_t slot) {
        __syncthreads();
        VgKSum v3[3] = {{acc_m, 0.0}, {acc_v, 0.0}, {acc_s, 0.0}};
        vg_block_ksum3<NTB>(v3, red);
        if (tid == 0) {
            TilePart p;
            p.mean = v3[0];
            p.var = v3[1];
            p.sigf = v3[2];
            a.parts[slot] = p;
        }
        acc_m = acc_v = acc_s = 0.0;
        __syncthreads();
    };
    int64_t next_static = first;

    for (;;) {
        __syncthreads();
        int64_t tile;
        if (NEED_RED) {
            // reduction modes: fixed tile -> CTA assignment, so the per-CTA
            // partial sums (and hence the result) are deterministic
            tile = next_static;
            next_static += stride;
        } else {
            // evaluation-only modes: dynamic tiles for load balance
            if (tid == 0) s_tile = (int64_t)atomicAdd(a.counter, 1ull);
            __syncthreads();
            tile = s_tile;
        }
        if (tile >= ntiles) break;
        const int64_t tile_start = tile * (int64_t)TT;
        const int tile_len = (int)min((int64_t)TT, N - tile_start);
        const int64_t h0 = a.tile_h0[tile * KSUB];
        const int64_t bnext = (tile + 1) * KSUB;            // base tile after this tile
        const int64_t hnext = bnext < nbase ? a.tile_h0[bnext] : a.H;
        const int64_t hlast = (hnext < a.H) ? hnext : a.H - 1;
        const int nwin = (int)(hlast - h0 + 1);
        if (nwin < 1 || nwin > TT) {   // impossible while every count is >= 2
            if (tid == 0) a.stats->status = VG_ERR_UNSUPPORTED;
            break;
        }
        for (int k = tid; k <= nwin; k += NTB) {
            int64_t h = h0 + k;
            int64_t o = (h <= a.H) ? a.offsets[h] : N;
            int64_t r = o - tile_start;
            win_off[k] = (int)(r < 0 ? 0 : (r > tile_len ? tile_len : r));
            if (k < nwin) win_n[k] = a.neval_h[h];
        }
        __syncthreads();

        // ---- pass 0: draw, map, evaluate the thread's samples
        const int li0 = tid * S;
        int nmine = tile_len - li0;
        nmine = nmine < 0 ? 0 : (nmine > S ? S : nmine);
        int lh = 0;
        if (nmine > 0) {
            int lo = 0, hi = nwin - 1;   // last k with win_off[k] <= li0
            while (lo < hi) {
                int mid = (lo + hi + 1) >> 1;
                if (win_off[mid] <= li0) lo = mid;
                else hi = mid - 1;
            }
            lh = lo;
        }
        int y0[DIMB];
        if (a.H <= 0x7fffffff) {   // 32-bit mixed-radix decode
            int hh = (int)(h0 + lh);
#pragma unroll
            for (int d = 0; d < DIMB; d++) {
                if (d < dim) {
                    const int q = hh / a.nstrat[d];
                    y0[d] = hh - q * a.nstrat[d];
                    hh = q;
                } else {
                    y0[d] = 0;
                }
            }
        } else {
            int64_t hh = h0 + lh;
#pragma unroll
            for (int d = 0; d < DIMB; d++) {
                if (d < dim) {
                    int64_t q = hh / a.nstrat[d];
                    y0[d] = (int)(hh - q * a.nstrat[d]);
                    hh = q;
                } else {
                    y0[d] = 0;
                }
            }
        }
        double xs[S][DIMB];
        double wg[S];   // sampler weight
        int lhs[S];
        int cur = lh;
        // the uniforms of all the thread's samples first (into xs): the
        // draws do not depend on the hypercube walk below, so the S samples'
        // Philox rounds interleave instead of waiting on one another
        // (REDUCE_KEPT reads the kept Jacobians instead)
#pragma unroll
        for (int k = 0; k < S && MODE != MODE_REDUCE_KEPT; k++) {
#pragma unroll
            for (int d = 0; d < DIMB; d++) xs[k][d] = 0.5;
            if (k < nmine) {
                const int64_t ig = tile_start + li0 + k;
                if (a.u != nullptr) {
#pragma unroll
                    for (int d = 0; d < DIMB; d++)
                        if (d < dim) xs[k][d] = (double)a.u[ig * dim + d];
                } else {
                    VgUniform<double>::draw<DIMB>(a.seed, a.stream, a.itn, (uint64_t)ig, dim, xs[k]);
#pragma unroll
                    for (int d = 0; d < DIMB; d++)
                        if (d >= dim) xs[k][d] = 0.5;
                }
            }
        }
#pragma unroll
        for (int k = 0; k < S; k++) {
            lhs[k] = cur;
            wg[k] = 0.0;
            if (k < nmine) {
                const int li = li0 + k;
                while (li >= win_off[cur + 1]) {   // next hypercube: mixed-radix increment
                    cur++;
                    int carry = 1;
#pragma unroll
                    for (int d = 0; d < DIMB; d++) {
                        if (d < dim && carry) {
                            if (++y0[d] < a.nstrat[d]) carry = 0;
                            else y0[d] = 0;
                        }
                    }
                }
                lhs[k] = cur;
                const int64_t ig = tile_start + li;
                const int nh = win_n[cur];
                double jac = 1.0;
                double yv[DIMB];
                unsigned short kbin[DIMB];   // MODE_POINTS: the bins to keep
                if constexpr (MODE == MODE_REDUCE_KEPT) {
                    jac = ((const double *)a.keep_jac)[ig];
                    if (use_bins) {   // rows of 4 bins, one 8-byte load each
                        const uint2 *src = reinterpret_cast<const uint2 *>(a.keep_bins + ig * a.keep_bstride);
                        for (int q = 0; q < dim; q += 4) {
                            const uint2 v = src[q >> 2];
                            const unsigned short b4[4] = {(unsigned short)(v.x & 0xffffu), (unsigned short)(v.x >> 16),
                                                          (unsigned short)(v.y & 0xffffu), (unsigned short)(v.y >> 16)};
                            for (int r = 0; r < 4 && q + r < dim; r++) sbins[(li0 + k) * dim + q + r] = b4[r];
                        }
                    }
                }
#pragma unroll
                for (int d = 0; d < DIMB; d++) {
                    if (d >= dim || MODE == MODE_REDUCE_KEPT) continue;
                    const int K = a.ninc[d];
                    double yd, yn, yfl;
                    const int iy = sample_y<double>(y0[d], 0.f, xs[k][d], a.nstrat[d], 0.f, K, 0.f, yd, yn, yfl);
                    const double dy = yn - yfl;
                    yv[d] = yd;
                    const int clamp = iy >= K;
                    const int ie = clamp ? K : iy;
                    double2 e;
                    if (a.table_smem) {
                        e = table[(size_t)d * (a.maxK + 1) + ie];
                    } else {
                        e.x = a.grid[d * a.ldg + ie];
                        e.y = a.inc[d * a.ldi + (clamp ? K - 1 : ie)];
                    }
                    xs[k][d] = clamp ? e.x : __dadd_rn(e.x, __dmul_rn(e.y, dy));
                    jac = __dmul_rn(jac, __dmul_rn(e.y, (double)K));
                    if (use_bins) sbins[(li0 + k) * dim + d] = sample_bin<double>(yd, iy, K);
                    if (MODE == MODE_POINTS) kbin[d] = sample_bin<double>(yd, iy, K);
                }
                if (MODE == MODE_POINTS && a.keep_bins) {   // rows of 4 bins, one 8-byte store each
                    uint2 *dst = reinterpret_cast<uint2 *>(a.keep_bins + ig * a.keep_bstride);
#pragma unroll
                    for (int q = 0; q < DIMB; q += 4) {
                        if (q >= dim) break;
                        unsigned int w4[4];
#pragma unroll
                        for (int r = 0; r < 4; r++) w4[r] = (q + r < dim && q + r < DIMB) ? kbin[q + r] : 0xffffu;
                        dst[q >> 2] = make_uint2(w4[0] | (w4[1] << 16), w4[2] | (w4[3] << 16));
                    }
                }
                // weight, pyx:1748-1749: jac *= dv_y / neval_hcube
                wg[k] = __dmul_rn(jac, __ddiv_rn(dv_y, (double)nh));
                if (MODE == MODE_POINTS) {
                    double *xo = (double *)a.x_out;
#pragma unroll
                    for (int d = 0; d < DIMB; d++)
                        if (d < dim) xo[ig * dim + d] = xs[k][d];
                    if (a.y_out) {
                        double *yo = (double *)a.y_out;
#pragma unroll
                        for (int d = 0; d < DIMB; d++)
                            if (d < dim) yo[ig * dim + d] = yv[d];
                    }
                    if (a.wgt_out) a.wgt_out[ig] = (double)wg[k];
                    if (a.hc_out) a.hc_out[ig] = h0 + cur;
                    if (a.keep_jac) ((double *)a.keep_jac)[ig] = jac;
                }
            }
        }
        if (MODE == MODE_POINTS) continue;

        double fv[S];
        if (MODE == MODE_FUSED) {
#pragma unroll
            for (int k = 0; k < S; k++) fv[k] = vg_eval_f64<KIND, DIMB>(prm, dim, xs[k]);
        } else {
#pragma unroll
            for (int k = 0; k < S; k++) {
                fv[k] = 0.0;
                if (k < nmine) {
                    const int64_t ig = tile_start + li0 + k;
                    fv[k] = a.f_f64 ? (double)((const double *)a.f_in)[ig]
                                    : (double)((const float *)a.f_in)[ig];
                }
            }
        }
        double wf[S];   // wgt * f, pyx:2143
#pragma unroll
        for (int k = 0; k < S; k++) {
            wf[k] = 0.0;
            if (k >= nmine) continue;
            if (fv[k] != fv[k]) nan_local = 1;
            wf[k] = __dmul_rn(wg[k], fv[k]);
            if (use_bins && a.train) {
                // fdv2 = (wgt*f*neval)^2, pyx:2173; |fdv2| into the bins, pyx:460-463
                const double t1 = __dmul_rn(wf[k], (double)win_n[lhs[k]]);
                const double fd = __dmul_rn(t1, t1);
                for (int d = 0; d < dim; d++) {
                    const unsigned short b = sbins[(li0 + k) * dim + d];
                    if (b == 0xffff) continue;
                    if (a.hist_smem) {
                        atomicAdd(&hsum[d * a.maxK + b], fd);
                        atomicAdd(&hcnt[d * a.maxK + b], 1u);
                    } else {
                        atomicAdd(&a.sum_f[d * a.ldi + b], fd);
                        atomicAdd(&a.n_f[d * a.ldi + b], 1ull);
                    }
                }
            }
        }

        // ---- pass 1: per-run sums of wf; segmented scan across threads
        const int has = nmine > 0;
        const int fk = has ? lhs[0] : 0x7fffffff;
        const int lk = has ? lhs[nmine - 1] : 0x7fffffff;
        double fsum = 0.0, lsum = 0.0;
#pragma unroll
        for (int k = 0; k < S; k++) {
            if (k < nmine && lhs[k] == fk) fsum += (double)wf[k];
            if (k < nmine && lhs[k] == lk) lsum += (double)wf[k];
        }
        keyF[tid] = fk;
        keyL[tid] = lk;
        __syncthreads();
        const int prevL = tid > 0 ? keyL[tid - 1] : -1;
        const int nextF = tid < NTB - 1 ? keyF[tid + 1] : -2;
        const int flag = (tid == 0) || (lk != prevL);
        double2 Pi = seg_scan<NTB>(flag, make_double2(lsum, 0.0), Pv, wsum, wflag);
        const double carry1 = (tid > 0 && prevL == fk && has) ? Pv[tid - 1].x : 0.0;
        const int ends_last = has && (lk != nextF);
        if (has && lk != fk) seg_S[fk] = fsum + carry1;
        if (ends_last) seg_S[lk] = Pi.x;
        __syncthreads();

        // ---- pass 2: deviations about the hypercube mean (pyx:2154-2171)
        double2 dq_first = make_double2(0.0, 0.0), dq_last = make_double2(0.0, 0.0);
        {
            int k = 0;
            while (k < nmine) {
                const int key = lhs[k];
                int k1 = k;
                double Sloc = 0.0;
                while (k1 < nmine && lhs[k1] == key) Sloc += (double)wf[k1++];
                const int nin = win_off[key + 1] - win_off[key];
                const bool is_first = (key == fk), is_last = (key == lk);
                const double Sseg = (is_first || is_last) ? seg_S[key] : Sloc;
                const double m = __ddiv_rn(Sseg, (double)nin);
                const double thr = __dmul_rn(VG_EPSILON, fabs(m));
                double Dr = 0.0, Qr = 0.0;
                for (int q = k; q < k1; q++) {
                    const double dwf = __dsub_rn((double)wf[q], m);
                    if (fabs(dwf) < thr) {
                        Qr = __dadd_rn(Qr, __dmul_rn(thr, thr));
                    } else {
                        Qr = __dadd_rn(Qr, __dmul_rn(dwf, dwf));
                        Dr = __dadd_rn(Dr, dwf);
                    }
                }
                if (is_first) dq_first = make_double2(Dr, Qr);
                if (is_last) dq_last = make_double2(Dr, Qr);
                if (!is_first && !is_last) {   // hypercube wholly inside this thread
                    const double nd = (double)nin;
                    const double vh = __ddiv_rn(__dsub_rn(__dmul_rn(nd, Qr), __dmul_rn(Dr, Dr)),
                                                __dsub_rn(nd, 1.));
                    acc_m += __dadd_rn(Sseg, Dr);
                    acc_v += vh;
                    if (a.adaptive) {
                        const double sg = pow(fabs(vh), beta_half);
                        a.sigf[h0 + key] = sg;
                        acc_s += sg;
                    }
                    if (a.train_hc) train_hcube(a, sbins + (size_t)(win_off[key + 1] - 1) * dim, fabs(vh));
                }
                k = k1;
            }
        }
        __syncthreads();
        double2 Pq = seg_scan<NTB>(flag, dq_last, Pv, wsum, wflag);
        const double2 carry2 =
            (tid > 0 && prevL == fk && has) ? Pv[tid - 1] : make_double2(0.0, 0.0);
#pragma unroll
        for (int which = 0; which < 2; which++) {
            int key;
            double2 dq;
            if (which == 0) {
                if (!(has && lk != fk)) continue;
                key = fk;
                dq = make_double2(dq_first.x + carry2.x, dq_first.y + carry2.y);
            } else {
                if (!ends_last) continue;
                key = lk;
                dq = Pq;
            }
            const int64_t h = h0 + key;
            const int nin = win_off[key + 1] - win_off[key];
            const int nh = win_n[key];
            const double Sseg = seg_S[key];
            const int64_t ostart = a.offsets[h];
            const bool starts_before = ostart < tile_start;
            const bool ends_after = ostart + nh > tile_start + tile_len;
            if (!starts_before && !ends_after) {
                const double nd = (double)nin;
                const double vh = __ddiv_rn(__dsub_rn(__dmul_rn(nd, dq.y), __dmul_rn(dq.x, dq.x)),
                                            __dsub_rn(nd, 1.));
                acc_m += __dadd_rn(Sseg, dq.x);
                acc_v += vh;
                if (a.adaptive) {
                    const double sg = pow(fabs(vh), beta_half);
                    a.sigf[h] = sg;
                    acc_s += sg;
                }
                if (a.train_hc) train_hcube(a, sbins + (size_t)(win_off[key + 1] - 1) * dim, fabs(vh));
            } else {
                TileRec r;
                r.h = h;
                r.n = (double)nin;
                r.S = Sseg;
                r.Q = dq.y;
                r.D = dq.x;
                r.spans = (starts_before && ends_after) ? 1 : 0;
                r.pad = 0;
                a.recs[2 * tile + (starts_before ? 0 : 1)] = r;
            }
        }
        if (tid == 0) {   // empty record slots
            const int64_t o0 = a.offsets[h0];
            if (!(o0 < tile_start)) a.recs[2 * tile].h = -1;
            int lastkey = nwin - 1;
            while (lastkey > 0 && win_off[lastkey] >= tile_len) lastkey--;
            const int64_t hL = h0 + lastkey;
            const bool tail = (a.offsets[hL] + a.neval_h[hL] > tile_start + tile_len) &&
                              !(hL == h0 && o0 < tile_start);
            if (!tail) a.recs[2 * tile + 1].h = -1;
        }
    }

    // ---- epilogue: partial sums (unless written per tile), NaN flag,
    // histogram flush
    if (NEED_RED) {
        emit_partial(part_slot);
        if (nan_local) atomicExch((int *)&a.stats->nan_seen, 1);
        if (use_bins && a.hist_smem) {
            __syncthreads();
            for (int d = 0; d < dim; d++) {
                const int K = a.ninc[d];
                for (int i = tid; i < K; i += NTB) {
                    const unsigned int c = hcnt[d * a.maxK + i];
                    if (c) {
                        atomicAdd(&a.sum_f[d * a.ldi + i], hsum[d * a.maxK + i]);
                        atomicAdd(&a.n_f[d * a.ldi + i], (unsigned long long)c);
                    }
                }
            }
        }
    }
}

template <int MODE, int KIND, int DIMB, int S, int NTB>
__global__ void __launch_bounds__(NTB, 1) tile_kernel(const __grid_constant__ IterArgs a,
                                                   const __grid_constant__ VgParams prm)
{
    extern __shared__ __align__(16) unsigned char smem[];
    vg_pdl_wait();
    vg_pdl_go();
    tile_body<MODE, KIND, DIMB, S, NTB>(a, prm, smem, blockIdx.x, gridDim.x, blockIdx.x);
}

// ---------------------------------------------------------------- launcher
// Tuning (vg_set_tile_tuning): grid table / histogram in shared memory (-1
// automatic, 0 off, 1 on where it fits).
extern int g_tile_table, g_tile_hist;

template <int MODE, int KIND, int DIMB, int S, int NTB>
int launch_tile_as(IterArgs &a, const VgParams *prm, cudaStream_t st, int stage)
{
    constexpr int TT = NTB * S;
    const int dim = a.dim;
    a.tab_len = 0;
    a.T = TT;
    constexpr int NEED_RED = (MODE == MODE_REDUCE || MODE == MODE_FUSED || MODE == MODE_REDUCE_KEPT);
    const int bins = NEED_RED && (a.train || a.train_hc);
    const size_t budget = 200 * 1024;
    a.table_smem = g_tile_table < 0 ? stage : g_tile_table;
    a.hist_smem = NEED_RED && a.train && (g_tile_hist < 0 ? stage : g_tile_hist);
    SmemPlan p = smem_plan<NTB>(dim, a.maxK, TT, a.table_smem, a.hist_smem, bins, NEED_RED);
    if (p.total > budget && a.hist_smem) {
        a.hist_smem = 0;
        p = smem_plan<NTB>(dim, a.maxK, TT, a.table_smem, a.hist_smem, bins, NEED_RED);
    }
    if (p.total > budget) {
        a.table_smem = 0;
        p = smem_plan<NTB>(dim, a.maxK, TT, a.table_smem, a.hist_smem, bins, NEED_RED);
    }
    if (p.total > 220 * 1024) return vg_fail(VG_ERR_UNSUPPORTED, "shared memory plan too large");
    auto kern = tile_kernel<MODE, KIND, DIMB, S, NTB>;
    static size_t attr_bytes = 0;   // largest dynamic shared memory enabled so far
    if (p.total > attr_bytes) {
        VG_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)p.total));
        attr_bytes = p.total;
    }
    int per_sm = 0;
    VG_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NTB, p.total));
    if (per_sm < 1) per_sm = 1;
    int64_t grid = (int64_t)vg_num_sms() * per_sm;
    const int64_t tcap = (a.ncap + TT - 1) / TT;
    if (grid > tcap) grid = tcap;
    if (grid < 1) grid = 1;
    if (NEED_RED && grid > MAX_PARTS) grid = MAX_PARTS;
    a.ncta = (int)grid;
    static const VgParams empty = {};
    VG_CUDA_CHECK(vg_launch_pdl(kern, (unsigned)grid, NTB, p.total, st, a, prm ? *prm : empty));
    return VG_OK;
}

template <int MODE, int KIND, int DIMB, int S>
int launch_tile(IterArgs &a, const VgParams *prm, cudaStream_t st)
{
    // Fewer large tiles than SMs: tiles of 128 samples instead, four times as
    // many, so that the FP64 work (19 cycles per warp instruction and SM) spreads
    // over more SMs; a CTA then has too few samples to stage the grid or a
    // histogram for.  1e4 evaluations at dim 4: 75 us on 18 SMs before.
    // (Not where hypercubes may have one sample or none: a tile takes as many
    // hypercubes as samples.)
    if (MODE != MODE_POINTS && !a.few && (a.ncap + NT * S - 1) / (NT * S) < vg_num_sms())
        return launch_tile_as<MODE, KIND, DIMB, 1, BASE_TILE>(a, prm, st, 0);
    return launch_tile_as<MODE, KIND, DIMB, S, NT>(a, prm, st, 1);
}

int finalize_launch(IterArgs &a, cudaStream_t st, int fast, vg_stats *rec);
int launch_reduce(IterArgs &a, int f64, cudaStream_t st);
int launch_reduce_kept(IterArgs &a, int f64, cudaStream_t st);
// IterArgs of one integral (pointers into its workspace) and its adapt scratch grid
int fill_iter_args(IterArgs &a, const vg_integrator *it, uint32_t itn, const double *u);
void scratch_grid(const vg_integrator *it, double **new_grid, double **new_inc);

}  // namespace vg
