// vg_adapt.cuh -- AdaptiveMap.adapt for one axis as a block-level device
// function (src/vegas/_vegas.pyx:467-594: average of the training data,
// 3-tap smoothing, normalisation, damping ((1-f)/-ln f)^alpha, regrid).
// The adapt kernel runs it with 1024 threads per axis, the batched kernel with
// the threads of its CTA.
#pragma once
#include <cooperative_groups.h>

#include "vg_common.cuh"

namespace vgadapt {

struct AdaptArgs {
    int dim;
    int old_ninc[VG_MAX_DIM];
    int new_ninc[VG_MAX_DIM];
    const double *grid, *inc;
    int64_t ldg, ldi;
    const double *sum_f;
    const unsigned long long *n_f;
    double alpha;
    double *new_grid, *new_inc;
    int64_t ldg_new, ldi_new;
    int max_old;      // length of the shared avg_f buffer (pyx:533)
    int sequential;   // one block walks all axes, carrying avg_f (pyx:533 semantics)
    int fast;         // FP32 mode: MUFU transcendentals and reciprocal multiplies
    int zero_hist;    // clear sum_f / n_f once read (the end of an iteration)
};

// ((1 - v) / -ln v)^alpha of the damping step (pyx:560-562), FP32-mode path:
// 1 - v and the exponent split in double, logs/exps on the MUFU.
__device__ __forceinline__ double damp_fast(double v, double alpha)
{
    const double one_m = 1.0 - v;
    float lnv;
    if (one_m < 0.25) lnv = log1pf((float)(v - 1.0));
    else lnv = vg_log2_split(v) * 0.69314718055994531f;
    const float q = (float)one_m / (-lnv);
    return (double)vg_ex2_approx((float)alpha * vg_lg2_approx(q));
}

// a / b in double with one Newton step on a float reciprocal (FP32 mode).
__device__ __forceinline__ double div_fast(double a, double b)
{
    double r = (double)__frcp_rn((float)b);
    r = fma(r, fma(-b, r, 1.0), r);
    return a * r;
}

// The threads that work on one axis: a whole CTA, or a set of GROUP_NT of its
// threads with a barrier of their own, so that a CTA adapts several axes at once.
struct WholeCta {
    __device__ __forceinline__ int t() const { return threadIdx.x; }
    __device__ __forceinline__ int n() const { return blockDim.x; }
    __device__ __forceinline__ void sync() const { __syncthreads(); }
};
constexpr int GROUP_NT = 256;
struct PartOfCta {
    __device__ __forceinline__ int t() const { return threadIdx.x % GROUP_NT; }
    __device__ __forceinline__ int n() const { return GROUP_NT; }
    __device__ __forceinline__ void sync() const
    {
        asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / GROUP_NT), "n"(GROUP_NT) : "memory");
    }
};

// Block-wide inclusive prefix sum of v[0..n) in place (FP64, fixed order):
// per-thread sequential over a contiguous chunk, then a scan of the chunk
// totals by warp shuffles (within each warp, then over the warp totals) --
// few FP64 instructions per thread (GB300 issues FP64 at a low rate).
template <typename CTA>
static __device__ void block_inclusive_scan(const CTA cta, double *v, int n, double *part /* >= 32 */)
{
    const int NT = cta.n(), NW = NT >> 5;
    const int t = cta.t(), lane = t & 31, w = t >> 5;
    const int per = (n + NT - 1) / NT;
    const int b = t * per, e = min(n, b + per);
    double s = 0.0;
    for (int i = b; i < e; i++) {
        s = __dadd_rn(s, v[i]);
        v[i] = s;
    }
    double x = s;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x = __dadd_rn(x, y);
    }
    if (lane == 31) part[w] = x;
    cta.sync();
    if (w == 0) {
        double z = lane < NW ? part[lane] : 0.0;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const double y = __shfl_up_sync(0xffffffffu, z, off);
            if (lane >= off) z = __dadd_rn(z, y);
        }
        if (lane < NW) part[lane] = z;
    }
    cta.sync();
    double ex = __shfl_up_sync(0xffffffffu, x, 1);   // exclusive prefix within the warp
    if (lane == 0) ex = 0.0;
    if (t > 0) {
        const double carry = (w > 0) ? __dadd_rn(part[w - 1], ex) : ex;
        for (int i = b; i < e; i++) v[i] = __dadd_rn(v[i], carry);
    }
    cta.sync();
}

// Sum of v[0..n) in a fixed order; result broadcast to all threads.
template <typename CTA>
static __device__ double block_sum(const CTA cta, const double *v, int n, double *part /* >= 33 */)
{
    const int NT = cta.n(), NW = NT >> 5;
    const int t = cta.t(), lane = t & 31, w = t >> 5;
    double s = 0.0;
    for (int i = t; i < n; i += NT) s = __dadd_rn(s, v[i]);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, off));
    if (lane == 0) part[w] = s;
    cta.sync();
    if (w == 0) {
        double z = lane < NW ? part[lane] : 0.0;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) z = __dadd_rn(z, __shfl_xor_sync(0xffffffffu, z, off));
        if (lane == 0) part[32] = z;
    }
    cta.sync();
    const double r = part[32];
    cta.sync();
    return r;
}

// FP32 block reductions (max, sum) over the first red_nt threads; f = shared
// scratch of >= 33 floats.  Result broadcast to all threads.
template <bool MAX, typename CTA>
__device__ float block_reduce_f(const CTA cta, float v, float *f, int red_nt)
{
    const int NW = red_nt >> 5;
    const int t = cta.t(), lane = t & 31, w = t >> 5;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float o = __shfl_xor_sync(0xffffffffu, v, off);
        v = MAX ? fmaxf(v, o) : v + o;
    }
    if (lane == 0 && w < NW) f[w] = v;
    cta.sync();
    if (w == 0) {
        float z = lane < NW ? f[lane] : 0.f;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float o = __shfl_xor_sync(0xffffffffu, z, off);
            z = MAX ? fmaxf(z, o) : z + o;
        }
        if (lane == 0) f[32] = z;
    }
    cta.sync();
    const float r = f[32];
    cta.sync();
    return r;
}

// FP32 mode: the normalised, damped weight of a smoothed average sf; rmx the
// reciprocal of the largest one, sp the sum of all times rmx.
__device__ __forceinline__ double damped_weight_fast(float sf, float rmx, float sp, double alpha)
{
    const float rs = sp > 0.f ? 1.f / sp : 0.f;
    const float vf = sf * rmx * rs;
    double v;
    if (sp > 0.f && vf >= 1.17549435e-38f && vf < 0.99999f) {
        const float one_m = 1.f - vf;
        const float lnv = one_m < 0.25f ? log1pf(-one_m) : vg_lg2_approx(vf) * 0.69314718f;
        const float q = one_m / (-lnv);
        v = (double)vg_ex2_approx((float)alpha * vg_lg2_approx(q));
    } else {
        v = sp > 0.f ? (double)sf * (double)rmx * (double)rs + VG_TINY : VG_TINY;
        if (v > 0 && v <= 0.99999999) v = damp_fast(v, alpha);
    }
    return v;
}

// FP32 mode, alpha > 0 with training data: the weights of one axis (average,
// 3-tap smoothing, normalisation, damping; pyx:539-562) in FP32 on the MUFU,
// written to avg[] as doubles.  The FP32 sum is formed by SUM_NT threads, so that
// it does not depend on the size of the CTA that adapts.  A normalised weight outside the float range
// (or within 1e-5 of 1) is formed and damped in FP64, so tiny weights keep
// the reference's ((1 - v) / -ln v)^alpha.  The cumulative sums and the new
// nodes (regrid) stay FP64.
template <int SUM_NT, typename CTA>
__device__ void adapt_weights_fast(const CTA cta, const AdaptArgs &a, int d, int K, double *avg, double *tmp,
                                   double *part)
{
    const int t = cta.t(), NT = cta.n();
    float *af = reinterpret_cast<float *>(tmp);   // [K] averages
    float *sf = af + K;                           // [K] smoothed (tmp holds 2K floats)
    float *pf = reinterpret_cast<float *>(part);
    for (int i = t; i < K; i += NT) {
        const unsigned long long c = a.n_f[d * a.ldi + i];
        af[i] = c ? (float)div_fast(a.sum_f[d * a.ldi + i], (double)c) : 0.f;
        if (a.zero_hist) {
            const_cast<double *>(a.sum_f)[d * a.ldi + i] = 0.0;
            const_cast<unsigned long long *>(a.n_f)[d * a.ldi + i] = 0ull;
        }
    }
    cta.sync();
    float mx = 0.f;
    for (int i = t; i < K; i += NT) {
        float v;
        if (i == 0) v = fmaf(7.f, af[0], af[1]);
        else if (i == K - 1) v = fmaf(7.f, af[K - 1], af[K - 2]);
        else v = fmaf(6.f, af[i], af[i - 1] + af[i + 1]);
        v = fabsf(v) * 0.125f;
        sf[i] = v;
        mx = fmaxf(mx, v);
    }
    mx = block_reduce_f<true>(cta, mx, pf, NT);
    const float rmx = mx > 0.f ? 1.f / mx : 0.f;   // sum of values scaled by the max: no overflow
    float sp = 0.f;
    const int sum_nt = SUM_NT > 0 ? SUM_NT : NT;
    if (t < sum_nt)
        for (int i = t; i < K; i += sum_nt) sp += sf[i] * rmx;
    sp = block_reduce_f<false>(cta, sp, pf, sum_nt);
    for (int i = t; i < K; i += NT) {
        avg[i] = damped_weight_fast(sf[i], rmx, sp, a.alpha);
    }
    cta.sync();
}

// One axis of AdaptiveMap.adapt.  avg (length >= max_old) holds the carried
// avg_f values on entry, the final ones on exit.  With gs / is (shared
// memory, max_old + 1 and max_old doubles) the axis' old nodes and
// increments are staged there first, so new_grid / new_inc may be the grid
// itself (adapt in place).
template <int SUM_NT = 0, typename CTA = WholeCta>
__device__ void adapt_axis(const AdaptArgs &a, int d, double *avg, double *tmp, double *part,
                           double *gs = nullptr, double *is = nullptr, const CTA cta = CTA())
{
    const int K = a.old_ninc[d];
    const int Kn = a.new_ninc[d];
    const int t = cta.t(), NT = cta.n();
    const double alpha = a.alpha;
    if (alpha > 0 && K > 1 && a.fast && a.sum_f != nullptr) {
        adapt_weights_fast<SUM_NT>(cta, a, d, K, avg, tmp, part);
    } else if (alpha != 0 && K > 1) {
        if (a.sum_f != nullptr) {
            for (int i = t; i < K; i += NT) {
                const unsigned long long c = a.n_f[d * a.ldi + i];
                if (a.fast) {
                    avg[i] = c ? div_fast(a.sum_f[d * a.ldi + i], (double)c) : 0.0;
                } else {
                    const double nf = __dadd_rn((double)c, VG_TINY);
                    avg[i] = (nf > 0) ? __ddiv_rn(a.sum_f[d * a.ldi + i], nf) : 0.0;
                }
                if (a.zero_hist) {
                    const_cast<double *>(a.sum_f)[d * a.ldi + i] = 0.0;
                    const_cast<unsigned long long *>(a.n_f)[d * a.ldi + i] = 0ull;
                }
            }
            cta.sync();
        }
        if (alpha > 0) {
            // smoothing, pyx:548-553
            for (int i = t; i < K; i += NT) {
                double v;
                if (i == 0) v = __dadd_rn(__dmul_rn(7., avg[0]), avg[1]);
                else if (i == K - 1) v = __dadd_rn(__dmul_rn(7., avg[K - 1]), avg[K - 2]);
                else v = __dadd_rn(__dadd_rn(__dmul_rn(6., avg[i]), avg[i - 1]), avg[i + 1]);
                tmp[i] = __dmul_rn(fabs(v), 0.125);   // == v / 8 exactly
            }
            cta.sync();
            double s = block_sum(cta, tmp, K, part);
            // normalise + damp, pyx:554-562
            const double rs = (s > 0) ? 1.0 / s : 0.0;
            for (int i = t; i < K; i += NT) {
                double v;
                if (a.fast) {
                    v = (s > 0) ? tmp[i] * rs + VG_TINY : VG_TINY;
                    if (v > 0 && v <= 0.99999999) v = damp_fast(v, alpha);
                } else {
                    v = (s > 0) ? __dadd_rn(__ddiv_rn(tmp[i], s), VG_TINY) : VG_TINY;
                    if (v > 0 && v <= 0.99999999) v = pow(__ddiv_rn(-(1 - v), log(v)), alpha);
                }
                avg[i] = v;
            }
            cta.sync();
        }
    }
    // regrid, pyx:563-587: new node i sits where the running sum of avg_f
    // reaches i*f_ninc; found by a block scan + binary search per node.
    double *P = tmp;
    const double *gd = a.grid + d * a.ldg;
    const double *id = a.inc + d * a.ldi;
    for (int i = t; i < K; i += NT) {
        P[i] = avg[i];
        if (gs != nullptr) {
            gs[i] = gd[i];
            is[i] = id[i];
        }
    }
    if (gs != nullptr && t == 0) gs[K] = gd[K];
    cta.sync();
    if (gs != nullptr) {
        gd = gs;
        id = is;
    }
    block_inclusive_scan(cta, P, K, part);
    const double total = P[K - 1];
    const double f_ninc = a.fast ? div_fast(total, (double)Kn) : __ddiv_rn(total, (double)Kn);
    double *ng = a.new_grid + d * a.ldg_new;
    for (int i = t; i <= Kn; i += NT) {
        double v;
        if (i == 0) v = gd[0];
        else if (i == Kn) v = gd[K];
        else {
            const double target = __dmul_rn((double)i, f_ninc);
            // first j with P[j] >= target; P and target are >= 0, so their
            // IEEE bit patterns order like the values (integer compares)
            const long long tb = __double_as_longlong(target);
            int lo = 0, hi = K - 1;
            while (lo < hi) {
                int mid = (lo + hi) >> 1;
                if (__double_as_longlong(P[mid]) < tb) lo = mid + 1;
                else hi = mid;
            }
            int j = lo;
            double acc = __dsub_rn(P[j], target);
            const double q = a.fast ? div_fast(acc, avg[j]) : __ddiv_rn(acc, avg[j]);
            v = __dsub_rn(gd[j + 1], __dmul_rn(q, id[j]));
        }
        ng[i] = v;
    }
    cta.sync();
    double *ni = a.new_inc + d * a.ldi_new;
    for (int i = t; i < Kn; i += NT) ni[i] = __dsub_rn(ng[i + 1], ng[i]);
    cta.sync();
}

// ----------------------------------------------------------- cluster form
// The same for one axis by a cluster of CLUSTER CTAs of CLUSTER_NT threads, in
// place: thread t of CTA c has increment and node i = c * CLUSTER_NT + t, and
// cluster memory holds what the others need.  For alpha > 0 with training data
// and at most CLUSTER * CLUSTER_NT - 1 increments.  The sums are formed in the
// order of adapt_axis with 1024 threads, so the results are the same bits.
constexpr int CLUSTER = 8, CLUSTER_NT = 128;
constexpr int CLUSTER_MAX = CLUSTER * CLUSTER_NT - 1;

struct ClusterSmem {
    double P[CLUSTER * CLUSTER_NT];         // cumulative weights of the whole axis
    double gs[CLUSTER * CLUSTER_NT], is[CLUSTER * CLUSTER_NT];   // its old nodes and increments
    double avg[CLUSTER_NT];                 // this CTA's weights
    double node[CLUSTER_NT];                // its new nodes
    double near[CLUSTER_NT + 2];            // its averages and the neighbours'
    double wtot[CLUSTER_NT / 32], wsum[CLUSTER_NT / 32];
    float wmax[CLUSTER_NT / 32], wsumf[CLUSTER_NT / 32];
};

static __device__ __forceinline__ void adapt_axis_cluster(const AdaptArgs &a, int d)
{
    namespace cg = cooperative_groups;
    __shared__ ClusterSmem s;
    constexpr int NW = CLUSTER_NT / 32;
    cg::cluster_group cl = cg::this_cluster();
    const int c = (int)cl.block_rank(), t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int i = c * CLUSTER_NT + t, gw = c * NW + w;
    const int K = a.old_ninc[d];
    double *gd = a.new_grid + d * a.ldg;   // the grid itself
    double *id = a.new_inc + d * a.ldi;
    double *sum_f = const_cast<double *>(a.sum_f) + d * a.ldi;
    unsigned long long *n_f = const_cast<unsigned long long *>(a.n_f) + d * a.ldi;
    for (int j = t; j <= K; j += CLUSTER_NT) {
        s.gs[j] = gd[j];
        if (j < K) s.is[j] = id[j];
    }
    auto average = [&](int j) -> double {   // pyx:539-547
        if (j < 0 || j >= K) return 0.0;
        const unsigned long long n = n_f[j];
        if (a.fast) return n ? (double)(float)div_fast(sum_f[j], (double)n) : 0.0;
        return __ddiv_rn(sum_f[j], __dadd_rn((double)n, VG_TINY));
    };
    s.near[t + 1] = average(i);
    if (t == 0) s.near[0] = average(i - 1);
    if (t == CLUSTER_NT - 1) s.near[CLUSTER_NT + 1] = average(i + 1);
    __syncthreads();
    const double am = s.near[t], a0 = s.near[t + 1], ap = s.near[t + 2];
    double v = 0.0;   // the weight
    if (a.fast) {
        // adapt_weights_fast: smoothing, normalisation and damping in FP32
        float sf = 0.f;
        if (i < K) {
            if (i == 0) sf = fmaf(7.f, (float)a0, (float)ap);
            else if (i == K - 1) sf = fmaf(7.f, (float)a0, (float)am);
            else sf = fmaf(6.f, (float)a0, (float)am + (float)ap);
            sf = fabsf(sf) * 0.125f;
        }
        float mx = sf;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        if (lane == 0) s.wmax[w] = mx;
        cl.sync();   // also: every CTA has read its averages and staged the axis
        mx = cl.map_shared_rank(s.wmax, lane / NW)[lane % NW];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float rmx = mx > 0.f ? 1.f / mx : 0.f;
        float sp = 0.f;
        if (i < K) sp += sf * rmx;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sp = sp + __shfl_xor_sync(0xffffffffu, sp, off);
        if (lane == 0) s.wsumf[w] = sp;
        cl.sync();
        sp = cl.map_shared_rank(s.wsumf, lane / NW)[lane % NW];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) sp = sp + __shfl_xor_sync(0xffffffffu, sp, off);
        if (i < K) v = damped_weight_fast(sf, rmx, sp, a.alpha);
    } else {
        double sm = 0.0;
        if (i < K) {
            if (i == 0) sm = __dadd_rn(__dmul_rn(7., a0), ap);
            else if (i == K - 1) sm = __dadd_rn(__dmul_rn(7., a0), am);
            else sm = __dadd_rn(__dadd_rn(__dmul_rn(6., a0), am), ap);
            sm = __dmul_rn(fabs(sm), 0.125);
        }
        double z = sm;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) z = __dadd_rn(z, __shfl_xor_sync(0xffffffffu, z, off));
        if (lane == 0) s.wsum[w] = z;
        cl.sync();   // also: every CTA has read its averages and staged the axis
        z = cl.map_shared_rank(s.wsum, lane / NW)[lane % NW];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) z = __dadd_rn(z, __shfl_xor_sync(0xffffffffu, z, off));
        if (i < K) {   // normalise + damp, pyx:554-562
            v = (z > 0) ? __dadd_rn(__ddiv_rn(sm, z), VG_TINY) : VG_TINY;
            if (v > 0 && v <= 0.99999999) v = pow(__ddiv_rn(-(1 - v), log(v)), a.alpha);
        }
    }
    if (i < K) {
        sum_f[i] = 0.0;
        n_f[i] = 0ull;
    }
    // cumulative weights of the whole axis, into every CTA
    s.avg[t] = v;
    double x = v;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, x, off);
        if (lane >= off) x = __dadd_rn(x, y);
    }
    if (lane == 31) s.wtot[w] = x;
    double ex = __shfl_up_sync(0xffffffffu, x, 1);
    if (lane == 0) ex = 0.0;
    cl.sync();
    double z = cl.map_shared_rank(s.wtot, lane / NW)[lane % NW];
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const double y = __shfl_up_sync(0xffffffffu, z, off);
        if (lane >= off) z = __dadd_rn(z, y);
    }
    const double before = __shfl_sync(0xffffffffu, z, gw > 0 ? gw - 1 : 0);
    const double P = i > 0 ? __dadd_rn(v, gw > 0 ? __dadd_rn(before, ex) : ex) : v;
    for (int r = 0; r < CLUSTER; r++) cl.map_shared_rank(s.P, r)[i] = P;
    cl.sync();
    // regrid, pyx:563-587
    const double total = s.P[K - 1];
    const double f_ninc = a.fast ? div_fast(total, (double)K) : __ddiv_rn(total, (double)K);
    auto node = [&](int n) -> double {
        if (n == 0) return s.gs[0];
        if (n >= K) return s.gs[K];
        const double target = __dmul_rn((double)n, f_ninc);
        const long long tb = __double_as_longlong(target);
        int lo = 0, hi = K - 1;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (__double_as_longlong(s.P[mid]) < tb) lo = mid + 1;
            else hi = mid;
        }
        const double acc = __dsub_rn(s.P[lo], target);
        const double wgt = cl.map_shared_rank(s.avg, lo / CLUSTER_NT)[lo % CLUSTER_NT];
        const double q = a.fast ? div_fast(acc, wgt) : __ddiv_rn(acc, wgt);
        return __dsub_rn(s.gs[lo + 1], __dmul_rn(q, s.is[lo]));
    };
    const double mine = node(i);
    s.node[t] = mine;
    const double last = t == CLUSTER_NT - 1 ? node(i + 1) : 0.0;
    __syncthreads();
    if (i <= K) gd[i] = mine;
    if (i < K) id[i] = __dsub_rn(t == CLUSTER_NT - 1 ? last : s.node[t + 1], mine);
    cl.sync();   // no CTA ends while another reads its weights
}

}  // namespace vgadapt
