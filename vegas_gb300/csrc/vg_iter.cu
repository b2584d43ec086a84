// vg_iter.cu -- one vegas+ iteration on the GPU.
//
// Reference: src/vegas/_vegas.pyx (vegas 6.4.1), Integrator._random_batch
// (pyx:1636-1765) and the batch loop of Integrator.__call__ (pyx:2096-2197).
//
// Layout of an iteration (all device-resident, no host round trip; each kernel
// is launched while the one before it drains):
//   1. alloc_kernel: neval_h[h] from sigf (pyx:1692-1706), exclusive scan ->
//      offsets[h], neval_hcube_range, the schedule tile_h0[t] (first hypercube
//      of each 128 samples); without adaptive allocation the offsets are
//      products.  FP32 mode: also the grid as an FP32 table.
//   2. the iteration kernel over all samples (ordered by hypercube, as in the
//      reference): Philox uniforms (or injected ones), y = (y0 + u)/nstrat, the
//      map y -> x, J, the integrand (fused built-in or read from an array),
//      wf = wgt*f, the training histogram of fdv2 = (wf*n_h)^2 and the
//      per-hypercube mean and variance with the reference's EPSILON
//      round-off guard.  FP32: warps on ranges of samples (vg_range.cuh); FP64:
//      CTAs on tiles (vg_tile.cuh).  Hypercubes cut by the ends of ranges or
//      tiles leave partial records (count, sum, sum of squared deviations).
//   3. tail_kernel: one block (FP64: a few) merges the partial records with
//      Chan's parallel variance formula and sums the partials into the
//      iteration's mean / var / sum_sigf, while clusters of 8 CTAs adapt one
//      axis each (finalize and adapt are separate kernels where the caller
//      asks for one of them, or an axis has more increments than a cluster's
//      threads).
// The iteration kernels' instantiations per integrand are spread over
// vg_fused_*.cu and vg_dropin.cu.
#include <math.h>
#include <string.h>

#include <cooperative_groups.h>

#include "vg_adapt.cuh"
#include "vg_range.cuh"

namespace {
using namespace vg;

// ======================================================== allocation
// Allocation, pyx:1692-1706, in one pass over the hypercubes: block b
// (numbered by the order in which blocks start, so it only waits on blocks
// already running) counts neval_h for its ALLOC_NT * ALLOC_PER hypercubes,
// publishes its total, looks back over its predecessors' published totals
// for its offset (decoupled look-back: a predecessor that already knows its
// inclusive prefix ends the walk), publishes its inclusive prefix, and writes
// offsets[h] and the tile schedule.  The last block writes the iteration's
// totals and resets the pass for the next iteration.  Published words hold
// (epoch, state, value) so nothing has to be cleared between iterations;
// every wait is bounded and a timeout is reported as VG_ERR_TIMEOUT with no
// tiles scheduled.  With build_table the grid also builds the FP32 grid table.
struct AllocSync {
    unsigned int ticket, epoch, err, pad;
    unsigned long long maxacc;
};

constexpr int FLAG_AGG = 1, FLAG_INC = 2;

__device__ __forceinline__ unsigned long long flag_word(unsigned int epoch, int state, int64_t v)
{
    return ((unsigned long long)(epoch & 0x3fffffu) << 42) | ((unsigned long long)state << 40) |
           ((unsigned long long)v & ((1ull << 40) - 1));
}

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long *p)
{
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

__device__ __forceinline__ void st_release_u64(unsigned long long *p, unsigned long long v)
{
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// The iteration's totals, by the thread that has them.
__device__ __forceinline__ void alloc_totals(const IterArgs &a, int64_t N, int64_t mxn, unsigned int err)
{
    vg_stats *st = a.stats;
    st->neval = N;
    // neval_hcube_range starts at [mnh, mnh] and every count is >= mnh
    // (pyx:1681, 1701-1704)
    st->range_lo = a.min_neval_hcube;
    st->range_hi = a.adaptive_alloc ? (mxn > a.min_neval_hcube ? mxn : a.min_neval_hcube) : a.min_neval_hcube;
    int64_t ntiles = (N + BASE_TILE - 1) / BASE_TILE;
    if (err) {
        st->status = VG_ERR_TIMEOUT;
        ntiles = 0;
    } else if (N > a.ncap || ntiles + 1 > a.ntiles_cap) {
        st->status = VG_ERR_MEMORY;
        ntiles = 0;
    } else {
        st->status = VG_OK;
        a.tile_h0[ntiles] = a.H;   // sentinel
    }
    a.offsets[a.H] = N;
    st->ntiles = ntiles;
    st->nan_seen = 0;
    *a.counter = 0ull;
    *a.fin_counter = 0u;
}

// offsets[h] and the tiles whose first sample falls in [run, run + n).
__device__ __forceinline__ void place_hcube(const IterArgs &a, int64_t h, int64_t run, int64_t n)
{
    a.offsets[h] = run;
    for (int64_t tt = (run + BASE_TILE - 1) / BASE_TILE; tt * BASE_TILE < run + n && tt < a.ntiles_cap; tt++)
        a.tile_h0[tt] = h;
}

__global__ void __launch_bounds__(ALLOC_NT) alloc_kernel(const __grid_constant__ IterArgs a, int64_t nblk, int build_table)
{
    __shared__ int64_t wtot[ALLOC_NT / 32], wmax[ALLOC_NT / 32];
    __shared__ double s_nsf;
    __shared__ int64_t s_prefix;
    __shared__ unsigned int s_b, s_epoch;
    AllocSync *sy = reinterpret_cast<AllocSync *>(a.alloc_sync);
    unsigned long long *flags = reinterpret_cast<unsigned long long *>(a.bsum);
    const int t = threadIdx.x;
    vg_pdl_wait();
    vg_pdl_go();
    if (!a.adaptive_alloc) {
        // as many in every hypercube: offsets are products, and no block has to
        // know of another (2e5 evaluations of dim 6, 85 blocks:
        // an iteration of 39 us became one of 35)
        const int64_t n = (int64_t)((double)a.neval / (double)a.H);
        if (build_table)
            build_tablef(a, (int64_t)blockIdx.x * ALLOC_NT + t, (int64_t)gridDim.x * ALLOC_NT);
        for (int k = 0; k < ALLOC_PER; k++) {
            const int64_t h = ((int64_t)blockIdx.x * ALLOC_PER + k) * ALLOC_NT + t;
            if (h >= a.H) break;
            a.neval_h[h] = (int32_t)n;
            place_hcube(a, h, h * n, n);
        }
        if (blockIdx.x == 0 && t == 0) {
            a.stats->neval_sigf = 0.0;
            alloc_totals(a, a.H * n, n, 0u);
        }
        return;
    }
    if (t == 0) {
        s_b = atomicAdd(&sy->ticket, 1u);
        s_epoch = *(volatile unsigned int *)&sy->epoch;
        const double sum_sigf = a.stats->sum_sigf;
        s_nsf = sum_sigf > 0 ? __ddiv_rn(__dmul_rn(a.neval_frac, (double)a.neval), sum_sigf) : 0.0;
        if (s_b == 0) a.stats->neval_sigf = s_nsf;
    }
    if (build_table)
        build_tablef(a, (int64_t)blockIdx.x * ALLOC_NT + t, (int64_t)gridDim.x * ALLOC_NT);
    __syncthreads();
    const int64_t b = (int64_t)(s_b % (unsigned int)nblk);
    const unsigned int epoch = s_epoch;
    const double nsf = s_nsf;
    const int64_t mx = a.max_neval_hcube > a.min_neval_hcube ? a.max_neval_hcube : a.min_neval_hcube;
    // counts of this thread's ALLOC_PER consecutive hypercubes
    const int64_t h0 = (b * ALLOC_NT + t) * ALLOC_PER;
    int64_t loc[ALLOC_PER];
    int64_t sum = 0, m = 0;
#pragma unroll
    for (int k = 0; k < ALLOC_PER; k++) {
        const int64_t h = h0 + k;
        int64_t n = 0;
        if (h < a.H) {
            n = (int64_t)__dmul_rn(a.sigf[h], nsf) + a.min_neval_hcube;
            if (n > mx) n = mx;
        }
        loc[k] = n;
        sum += n;
        m = n > m ? n : m;
    }
    if (h0 + ALLOC_PER <= a.H) {   // 16-byte aligned: h0 is a multiple of 4
        *reinterpret_cast<int4 *>(a.neval_h + h0) = make_int4((int)loc[0], (int)loc[1], (int)loc[2], (int)loc[3]);
    } else {
#pragma unroll
        for (int k = 0; k < ALLOC_PER; k++)
            if (h0 + k < a.H) a.neval_h[h0 + k] = (int32_t)loc[k];
    }
    // the block's exclusive scan and maximum, with one barrier
    const int lane = t & 31, warp = t >> 5;
    int64_t run = sum;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, run, off);
        if (lane >= off) run += y;
        const int64_t z = __shfl_xor_sync(0xffffffffu, m, off);
        m = z > m ? z : m;
    }
    if (lane == 31) {
        wtot[warp] = run;
        wmax[warp] = m;
    }
    run -= sum;
    __syncthreads();
    int64_t tot = 0, bm = 0;
#pragma unroll
    for (int w = 0; w < ALLOC_NT / 32; w++) {
        if (w == warp) run += tot;
        tot += wtot[w];
        bm = wmax[w] > bm ? wmax[w] : bm;
    }
    // warp 0: publish the block total, then look back 32 predecessors at a
    // time (each lane waits for one published word; the nearest inclusive
    // prefix ends the walk)
    if (t < 32) {
        if (lane == 0) {
            atomicMax(&sy->maxacc, (unsigned long long)bm);
            __threadfence();
            st_release_u64(&flags[b], flag_word(epoch, b == 0 ? FLAG_INC : FLAG_AGG, tot));
        }
        __syncwarp();
        int64_t prefix = 0;
        int ok = 1;
        for (int64_t hi = b - 1; hi >= 0; hi -= 32) {
            const int64_t p = hi - lane;
            int64_t v = 0;
            int inc = 1;   // before block 0: an inclusive prefix of 0
            if (p >= 0) {
                unsigned long long w = 0;
                uint32_t i = 0;
                const uint32_t budget = a.wait_iters;
                for (; i < budget; i++) {
                    w = ld_acquire_u64(&flags[p]);
                    if ((unsigned int)(w >> 42) == (epoch & 0x3fffffu) && ((w >> 40) & 3u) != 0) break;
                    if (i >= 64) __nanosleep(64);
                }
                if (i == budget) ok = 0;   // gave up: reported below, the walk goes on
                v = (int64_t)(w & ((1ull << 40) - 1));
                inc = ((w >> 40) & 3u) == (unsigned)FLAG_INC;
            }
            const unsigned int incm = __ballot_sync(0xffffffffu, inc);
            const int first = incm ? __ffs(incm) - 1 : 32;
            int64_t c = lane <= first ? v : 0;
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
            prefix += c;
            if (incm) break;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (lane == 0) {
            if (b > 0) {
                if (!ok) atomicOr(&sy->err, 1u);
                __threadfence();
                st_release_u64(&flags[b], flag_word(epoch, FLAG_INC, prefix + tot));
            }
            s_prefix = prefix;
        }
    }
    __syncthreads();
    run += s_prefix;
#pragma unroll
    for (int k = 0; k < ALLOC_PER; k++) {
        const int64_t h = h0 + k;
        if (h >= a.H) break;
        place_hcube(a, h, run, loc[k]);
        run += loc[k];
    }
    if (b == nblk - 1 && t == 0) {   // every other block has published: totals, reset
        __threadfence();
        alloc_totals(a, s_prefix + tot, (int64_t)*(volatile unsigned long long *)&sy->maxacc,
                     *(volatile unsigned int *)&sy->err);
        sy->maxacc = 0ull;
        sy->err = 0u;
        sy->epoch = epoch + 1u;
        sy->ticket = 0u;
    }
}

// FP32 mode: the grid as an FP32 (x_node, inc) table for the tile CTAs.
__global__ void tablef_kernel(IterArgs a)
{
    build_tablef(a, (int64_t)blockIdx.x * blockDim.x + threadIdx.x, (int64_t)gridDim.x * blockDim.x);
}

// ========================================================== finalize
// FP64 mode.
// Stage 1 (one thread per tile, FIN_NT tiles per block): the tile's
// partial sums plus, for a tile whose last hypercube continues into later
// tiles, the Chan et al. merge of that hypercube's partial records; a
// fixed-order block reduction gives one partial per block.
// Stage 2 (one block): those partials in block order -> iteration mean, var,
// sum_sigf (compensated FP64), and the constant-integrand reset.
constexpr int FIN_NT = 128;      // threads per finalize block, one tile each (the tail kernel's CTAs)

// The iteration's results from the stats fields (mean, var, sum_sigf) and
// the constant-integrand reset (pyx:2209-2215); thread 0 has the sums.
__device__ __forceinline__ void finalize_store(const IterArgs &a, double mean, double var, double ss, int *reset,
                                               vg_stats *rec)
{
    if (threadIdx.x == 0) {
        vg_stats *st = a.stats;
        st->mean = mean;
        st->var = var;
        *reset = 0;
        st->sigf_reset = 0;
        if (a.adaptive) {
            if (ss > 0) {
                st->sum_sigf = ss;
            } else {   // integrand looks constant: even distribution
                st->sum_sigf = (double)a.H;
                st->sigf_reset = 1;
                *reset = 1;
            }
        }
        if (rec != nullptr) *rec = *st;   // the caller's copy (pinned host memory)
    }
    __syncthreads();
    if (*reset)
        for (int64_t h = threadIdx.x; h < a.H; h += blockDim.x) a.sigf[h] = 1.0;
}

// FP32 mode: one CTA.
constexpr int FIN32_NT = 256;
__device__ __forceinline__ void finalize32(const IterArgs &a, vg_stats *rec)
{
    __shared__ int s_reset;
    float s6[6];
    finalize_ranges(a, a.ncta, a.ngroups, 0, s6);
    finalize_store(a, vg_ff_value(s6[0], s6[1]), vg_ff_value(s6[2], s6[3]), vg_ff_value(s6[4], s6[5]), &s_reset, rec);
}

__global__ void __launch_bounds__(FIN32_NT) finalize32_kernel(const __grid_constant__ IterArgs a, vg_stats *rec)
{
    vg_pdl_wait();
    vg_pdl_go();
    finalize32(a, rec);
}

// Stage 1, and stage 2 in the block that finishes last (a counter the
// allocation resets; the partials are read back in block order, so the
// result does not depend on which block that is).  Block `block` of `nblocks`.
__device__ __forceinline__ void finalize64(const IterArgs &a, int block, int nblocks, vg_stats *rec)
{
    __shared__ VgKSum red[3 * (FIN_NT / 32)];
    __shared__ int s_last, s_reset;
    const vg_stats *st = a.stats;
    const int64_t N = st->neval;
    const int64_t ntiles = st->ntiles ? (N + a.T - 1) / a.T : 0;
    const int64_t nwork = ntiles > a.ncta ? ntiles : a.ncta;
    const int64_t nblk = (nwork + FIN_NT - 1) / FIN_NT;
    if (block < nblk) {
        const double beta_half = a.beta_half;
        VgKSum cm = {0.0, 0.0}, cv = {0.0, 0.0}, cs = {0.0, 0.0};
        const int64_t t = (int64_t)block * FIN_NT + threadIdx.x;
        if (t < a.ncta && ntiles > 0) {   // partial sums of the reduction CTA t
            const TilePart p = a.parts[t];
            cm = p.mean;
            cv = p.var;
            cs = p.sigf;
        }
        if (t < ntiles) {   // a hypercube starting in tile t and cut by its end
            const TileRec r = a.recs[2 * t + 1];
            if (r.h >= 0) {
                double n = r.n, Sx = r.S, Q = r.Q, D = r.D;
                for (int64_t t2 = t + 1; t2 < ntiles; t2++) {
                    const TileRec q = a.recs[2 * t2];
                    if (q.h != r.h) break;
                    const double n2 = n + q.n;
                    const double delta = q.S / q.n - Sx / n;   // Chan et al. merge
                    Q = Q + q.Q + delta * delta * (n * q.n / n2);
                    Sx += q.S;
                    D += q.D;
                    n = n2;
                    if (!q.spans) break;
                }
                const double num = __dsub_rn(__dmul_rn(n, Q), __dmul_rn(D, D));
                const double vh = __ddiv_rn(num, __dsub_rn(n, 1.));
                if (a.train_hc) {   // adapt_to_errors: train at the hypercube's last sample
                    unsigned short b[VG_MAX_DIM];
                    last_sample_bins<double>(a, r.h, b);
                    train_hcube(a, b, fabs(vh));
                }
                cm.add(__dadd_rn(Sx, D));
                cv.add(vh);
                if (a.adaptive) {
                    const double sg = pow(fabs(vh), beta_half);
                    a.sigf[r.h] = sg;
                    cs.add(sg);
                }
            }
        }
        VgKSum v3[3] = {cm, cv, cs};
        vg_block_ksum3<FIN_NT>(v3, red);
        if (nblocks == 1) {   // nothing to wait for
            finalize_store(a, v3[0].value(), v3[1].value(), v3[2].value(), &s_reset, rec);
            return;
        }
        if (threadIdx.x == 0) {
            TilePart p;
            p.mean = v3[0];
            p.var = v3[1];
            p.sigf = v3[2];
            a.part2[block] = p;
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = (atomicAdd(a.fin_counter, 1u) == (unsigned int)nblocks - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) *a.fin_counter = 0u;
    VgKSum t3[3] = {{0.0, 0.0}, {0.0, 0.0}, {0.0, 0.0}};
    for (int64_t b = threadIdx.x; b < nblk; b += FIN_NT) {
        const TilePart p = a.part2[b];
        t3[0].merge(p.mean);
        t3[1].merge(p.var);
        t3[2].merge(p.sigf);
    }
    vg_block_ksum3<FIN_NT>(t3, red);
    finalize_store(a, t3[0].value(), t3[1].value(), t3[2].value(), &s_reset, rec);
}

__global__ void __launch_bounds__(FIN_NT) finalize64_kernel(const __grid_constant__ IterArgs a, vg_stats *rec)
{
    vg_pdl_wait();
    vg_pdl_go();
    finalize64(a, blockIdx.x, gridDim.x, rec);
}

// The end of an iteration in one launch: the iteration's sums, and the map's
// adapt, which needs only the training histogram.  A cluster of 8 CTAs per
// axis adapts, 128 of the axis' increments each: the FP64 work per increment
// (damping in FP64 mode; the cumulative sum, the search for each new node and
// its interpolation in both) is spread over 8 SMs, whose FP64 pipes take 19
// cycles per warp instruction; one CTA of 1024 threads per axis took 53 us
// in FP64 and 18 us in FP32 at 1000 increments.  The clusters after them
// finalize (FP32: one CTA; FP64: 128 tiles per CTA).
__global__ void __cluster_dims__(vgadapt::CLUSTER, 1, 1) __launch_bounds__(FIN_NT)
tail_kernel(const __grid_constant__ IterArgs a, const __grid_constant__ vgadapt::AdaptArgs ad, int f64, int nfin,
            vg_stats *rec)
{
    vg_pdl_wait();
    vg_pdl_go();
    const int b = (int)blockIdx.x - ad.dim * vgadapt::CLUSTER;
    if (b < 0) vgadapt::adapt_axis_cluster(ad, blockIdx.x / vgadapt::CLUSTER);
    else if (b < nfin) {
        if (f64) finalize64(a, b, nfin, rec);
        else finalize32(a, rec);
    }
}

// ================================================================ host
struct WorkLayout {
    size_t neval_h, offsets, bsum, tile_h0, counter, recs, parts, part2, feval, newgrid,
        newinc, tablef, total;
    int64_t nblk, ntiles_cap, ncap, rec_cap, part_cap;
};

inline size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

inline int64_t neval_cap(const vg_integrator *it)
{
    // sum_h min(max, int(sigf_h*nsf) + mnh) <= neval_frac*neval + H*mnh (+ rounding)
    const int64_t H = it->nhcube;
    const int64_t avg = (int64_t)((double)it->neval / (double)H);
    const int64_t mnh = it->min_neval_hcube > avg ? it->min_neval_hcube : avg;
    const double adaptive = it->neval_frac * (double)it->neval;
    return (int64_t)(adaptive * (1.0 + 1e-9)) + 64 + H * mnh;
}

WorkLayout layout(const vg_integrator *it, int64_t ncap)
{
    WorkLayout L;
    const int64_t H = it->nhcube;
    L.nblk = (H + ALLOC_NT * ALLOC_PER - 1) / (ALLOC_NT * ALLOC_PER);
    L.ntiles_cap = (ncap + BASE_TILE - 1) / BASE_TILE + 1;
    size_t o = 0;
    L.neval_h = o; o = align256(o + sizeof(int32_t) * H);
    L.offsets = o; o = align256(o + sizeof(int64_t) * (H + 1));
    L.bsum = o;    o = align256(o + sizeof(int64_t) * L.nblk);
    L.tile_h0 = o; o = align256(o + sizeof(int64_t) * (L.ntiles_cap + 1));
    L.counter = o; o = align256(o + 16 + sizeof(AllocSync));
    // FP64: two records per tile of 256 or more samples (or 128); FP32: per group or dealt unit
    const int f64 = it->precision == VG_F64;
    const int64_t small = L.ntiles_cap < 1024 ? L.ntiles_cap : 1024;   // tiles of 128 where there are few
    const int64_t tiles = (ncap + 255) / 256 + 1 > small ? (ncap + 255) / 256 + 1 : small;
    L.part_cap = L.ntiles_cap < MAX_PARTS ? L.ntiles_cap : (int64_t)MAX_PARTS;
    if (L.part_cap < 1024) L.part_cap = 1024;   // the batched launch's groups of CTAs, whatever the integral's size
    const int64_t units = L.ntiles_cap + 1;
    L.rec_cap = f64 ? tiles : (units > L.part_cap ? units : L.part_cap);
    const int64_t fin = L.rec_cap > L.part_cap ? L.rec_cap : L.part_cap;
    L.recs = o;    o = align256(o + (f64 ? sizeof(TileRec) : sizeof(RangeRec)) * 2 * L.rec_cap);
    L.parts = o;   o = align256(o + sizeof(TilePart) * L.part_cap);
    L.part2 = o;   o = align256(o + sizeof(TilePart) * (fin / FIN_NT + 2));
    L.feval = o;   o = align256(o + sizeof(float) * ncap);
    L.ncap = ncap;
    L.newgrid = o; o = align256(o + sizeof(double) * it->dim * it->ldg);
    L.newinc = o;  o = align256(o + sizeof(double) * it->dim * it->ldi);
    int64_t maxK = 1;
    for (int d = 0; d < it->dim; d++) maxK = it->ninc[d] > maxK ? it->ninc[d] : maxK;
    L.tablef = o;  o = align256(o + sizeof(float2) * it->dim * (maxK + 1));
    L.total = o;
    return L;
}

int fill_args(IterArgs &a, const vg_integrator *it, uint32_t itn, const double *u)
{
    memset(&a, 0, sizeof(a));
    if (it->dim < 1 || it->dim > VG_MAX_DIM) return vg_fail(VG_ERR_UNSUPPORTED, "dim");
    if (!it->work || !it->stats) return vg_fail(VG_ERR_VALUE, "missing workspace/stats");
    a.dim = it->dim;
    int maxK = 1;
    for (int d = 0; d < it->dim; d++) {
        if (it->nstrat[d] < 1 || it->ninc[d] < 1 || it->ninc[d] > 65534)
            return vg_fail(VG_ERR_VALUE, "bad geometry (ninc must be in 1..65534)");
        a.nstrat[d] = (int)it->nstrat[d];
        a.ninc[d] = (int)it->ninc[d];
        AxisArgs &x = a.ax[d];
        x.nstrat = a.nstrat[d];
        x.ninc = a.ninc[d];
        x.Kf = (float)a.ninc[d];
        x.rstrat = 1.f / (float)a.nstrat[d];
        int sh = 0;   // 2^sh >= nstrat: h * (dmul * nstrat - 2^(31+sh)) < 2^(31+sh) for h < 2^31
        while (((int64_t)1 << sh) < a.nstrat[d]) sh++;
        x.dshift = sh;
        x.dmul = (unsigned int)((((uint64_t)1 << (31 + sh)) + (uint64_t)a.nstrat[d] - 1) / (uint64_t)a.nstrat[d]);
        a.wide |= a.nstrat[d] >= (1 << 24);
        maxK = a.ninc[d] > maxK ? a.ninc[d] : maxK;
        if (it->ninc[d] + 1 > it->ldg || it->ninc[d] > it->ldi)
            return vg_fail(VG_ERR_VALUE, "grid arrays too small");
    }
    a.maxK = maxK;
    a.grid = it->grid;
    a.inc = it->inc;
    a.ldg = it->ldg;
    a.ldi = it->ldi;
    a.H = it->nhcube;
    a.wide |= it->nhcube > 0x7fffffff;
    a.ncap = neval_cap(it);
    a.wide |= a.ncap > 0x7fffffff - 4096;
    WorkLayout L = layout(it, a.ncap);
    if (it->work_bytes < L.total)
        return vg_fail(VG_ERR_VALUE, "workspace too small: %zu < %zu", it->work_bytes, L.total);
    char *w = (char *)it->work;
    a.sigf = it->sigf;
    a.beta = it->beta;
    // adapt_to_errors: uniform allocation, no sigf, the map trained on each
    // hypercube's variance (pyx:1659, 1675, 2187-2196, 2209)
    const int ate = it->adapt_to_errors ? 1 : 0;
    a.adaptive_alloc = (it->beta > 0 && it->nhcube > 1 && !ate) ? 1 : 0;
    a.adaptive = (a.adaptive_alloc && it->adapt) ? 1 : 0;
    a.few = (a.adaptive_alloc ? (double)it->min_neval_hcube : (double)it->neval / (double)it->nhcube) < 2.0;
    a.train = (it->adapt && it->alpha > 0 && !ate) ? 1 : 0;
    a.train_hc = (ate && it->adapt) ? 1 : 0;
    a.sum_f = it->sum_f;
    a.n_f = (unsigned long long *)it->n_f;
    a.stats = it->stats;
    a.neval_h = (int32_t *)(w + L.neval_h);
    a.offsets = (int64_t *)(w + L.offsets);
    a.bsum = (int64_t *)(w + L.bsum);
    a.tile_h0 = (int64_t *)(w + L.tile_h0);
    a.counter = (unsigned long long *)(w + L.counter);
    a.fin_counter = (unsigned int *)(w + L.counter + sizeof(unsigned long long));
    a.alloc_sync = (unsigned int *)(w + L.counter + 16);
    a.recs = (TileRec *)(w + L.recs);
    a.rrecs = (RangeRec *)(w + L.recs);
    a.parts = (TilePart *)(w + L.parts);
    a.part2 = (TilePart *)(w + L.part2);
    a.f_eval = (float *)(w + L.feval);
    a.tablef = (float2 *)(w + L.tablef);
    a.ntiles_cap = L.ntiles_cap;
    a.neval = it->neval;
    a.neval_frac = it->neval_frac;
    a.min_neval_hcube = it->min_neval_hcube;
    a.max_neval_hcube = it->max_neval_hcube;
    a.seed = it->seed;
    a.stream = it->stream_id;
    a.itn = itn;
    a.u = u;
    a.dv_y = 1.0 / (double)it->nhcube;
    a.beta_half = it->beta / 2.0;
    a.wait_iters = g_wait_iters;
    return VG_OK;
}

}  // namespace

namespace vg {
// CTAs of the FP64 finalize: the tiles of the launched kernel, bounded by the capacity.
static int64_t finalize_blocks(const IterArgs &a)
{
    const int64_t tcap = (a.ncap + a.T - 1) / a.T;
    const int64_t nwork = tcap > a.ncta ? tcap : a.ncta;
    return (nwork + FIN_NT - 1) / FIN_NT;
}

int finalize_launch(IterArgs &a, cudaStream_t st, int fast, vg_stats *rec)
{
    if (fast) VG_CUDA_CHECK(vg_launch_pdl(finalize32_kernel, 1, FIN32_NT, 0, st, a, rec));
    else VG_CUDA_CHECK(vg_launch_pdl(finalize64_kernel, (unsigned)finalize_blocks(a), FIN_NT, 0, st, a, rec));
    return VG_OK;
}

int launch_points(IterArgs &a, int f64, cudaStream_t st);
int launch_reduce(IterArgs &a, int f64, cudaStream_t st);
int launch_fused(IterArgs &a, int kind, const VgParams &P, int tab_len, int f64, cudaStream_t st);

int fill_iter_args(IterArgs &a, const vg_integrator *it, uint32_t itn, const double *u)
{
    return fill_args(a, it, itn, u);
}

void scratch_grid(const vg_integrator *it, double **new_grid, double **new_inc)
{
    WorkLayout L = layout(it, neval_cap(it));
    char *w = (char *)it->work;
    *new_grid = (double *)(w + L.newgrid);
    *new_inc = (double *)(w + L.newinc);
}
}  // namespace vg

// ====================================================================== ABI
extern "C" int64_t vg_neval_cap(const vg_integrator *it) { return neval_cap(it); }

extern "C" size_t vg_workspace_bytes(const vg_integrator *it, int64_t ncap)
{
    if (it == nullptr || it->dim < 1 || it->dim > VG_MAX_DIM) {   // layout() reads ninc[0 .. dim)
        vg_fail(VG_ERR_VALUE, "vg_workspace_bytes: dim outside 1..%d", VG_MAX_DIM);
        return 0;
    }
    if (ncap <= 0) ncap = neval_cap(it);
    return layout(it, ncap).total;
}

extern "C" int vg_allocate(const vg_integrator *it, void *stream)
{
    VG_RANGE("vg_allocate");
    vg_clear_error();
    IterArgs a;
    int rc = fill_args(a, it, 0, nullptr);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    WorkLayout L = layout(it, a.ncap);
    // the FP32 grid table is built by the counting grid, or alone when that
    // grid has too few threads for it
    const int64_t ntab = (int64_t)a.dim * (a.maxK + 1);
    const int table_in_count = (it->precision == VG_F32) && ntab <= L.nblk * ALLOC_NT;
    VG_CUDA_CHECK(vg_launch_pdl(alloc_kernel, (unsigned)L.nblk, ALLOC_NT, 0, st, a, L.nblk, table_in_count));
    if (it->precision == VG_F32 && !table_in_count) {
        tablef_kernel<<<(unsigned)((ntab + 255) / 256), 256, 0, st>>>(a);
        VG_LAUNCH_CHECK();
    }
    return VG_OK;
}

// Clears the single-pass allocation's published block words and its
// ticket / epoch for a workspace that other geometries have used (the
// static scratch of vg_iteration_noalloc).
int vg_alloc_sync_reset(const vg_integrator *it, void *stream)
{
    WorkLayout L = layout(it, neval_cap(it));
    char *w = (char *)it->work;
    cudaStream_t st = (cudaStream_t)stream;
    VG_CUDA_CHECK(cudaMemsetAsync(w + L.bsum, 0, sizeof(int64_t) * (size_t)L.nblk, st));
    VG_CUDA_CHECK(cudaMemsetAsync(w + L.counter, 0, 16 + sizeof(AllocSync), st));
    return VG_OK;
}

static int reset_counter(IterArgs &a, cudaStream_t st)
{
    VG_CUDA_CHECK(cudaMemsetAsync(a.counter, 0, sizeof(unsigned long long), st));
    return VG_OK;
}

extern "C" int vg_sample(const vg_integrator *it, uint32_t itn, const double *u, void *x, void *y,
                         double *wgt, int64_t *hcube, int64_t n_cap, void *stream)
{
    VG_RANGE("vg_sample");
    vg_clear_error();
    IterArgs a;
    int rc = fill_args(a, it, itn, u);
    if (rc) return rc;
    if (n_cap < a.ncap) return vg_fail(VG_ERR_VALUE, "output capacity %lld < %lld",
                                       (long long)n_cap, (long long)a.ncap);
    a.x_out = x;
    a.y_out = y;
    a.wgt_out = wgt;
    a.hc_out = hcube;
    a.train = 0;
    a.train_hc = 0;
    a.adaptive = 0;
    a.x_vec = (a.dim % 4 == 0) && ((uintptr_t)x & 15) == 0;
    cudaStream_t st = (cudaStream_t)stream;
    if (it->precision == VG_F64 && (rc = reset_counter(a, st))) return rc;   // FP64 tiles are taken from a counter
    return vg::launch_points(a, it->precision == VG_F64, st);
}

extern "C" int vg_reduce(const vg_integrator *it, uint32_t itn, const double *u, const void *f,
                         int f_dtype, void *stream)
{
    VG_RANGE("vg_reduce");
    vg_clear_error();
    IterArgs a;
    int rc = fill_args(a, it, itn, u);
    if (rc) return rc;
    a.f_in = f;
    a.f_f64 = (f_dtype == VG_F64);
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = vg::launch_reduce(a, it->precision == VG_F64, st))) return rc;   // static tiles
    return vg::finalize_launch(a, st, it->precision == VG_F32, nullptr);
}

// An iteration record set to zero but for the carried sum_sigf.
__global__ void stats_reset_kernel(vg_stats *st, double sum_sigf)
{
    if (threadIdx.x == 0) {
        vg_stats z;
        memset(&z, 0, sizeof(z));
        z.sum_sigf = sum_sigf;
        *st = z;
    }
}

extern "C" int vg_stats_reset(vg_stats *stats, double sum_sigf, void *stream)
{
    vg_clear_error();
    if (stats == nullptr) return vg_fail(VG_ERR_VALUE, "vg_stats_reset: no record");
    stats_reset_kernel<<<1, 32, 0, (cudaStream_t)stream>>>(stats, sum_sigf);
    VG_LAUNCH_CHECK();
    return VG_OK;
}

// The kept-sample buffer of vg_sample_keep / vg_reduce_kept: per sample its
// Jacobian (the precision's float type), then its training bins (16-bit per
// axis, rows padded to a multiple of 4 axes so that each 4 bins move as one
// 8-byte word).
static int keep_bstride(const vg_integrator *it) { return (it->dim + 3) & ~3; }

static size_t keep_jac_bytes(const vg_integrator *it, int64_t ncap)
{
    const size_t t = it->precision == VG_F64 ? sizeof(double) : sizeof(float);
    return (t * (size_t)ncap + 255) & ~(size_t)255;
}

extern "C" size_t vg_keep_bytes(const vg_integrator *it, int64_t n_cap)
{
    if (it == nullptr || it->dim < 1 || it->dim > VG_MAX_DIM) {
        vg_fail(VG_ERR_VALUE, "vg_keep_bytes: dim outside 1..%d", VG_MAX_DIM);
        return 0;
    }
    if (n_cap <= 0) n_cap = neval_cap(it);
    return keep_jac_bytes(it, n_cap) + sizeof(unsigned short) * (size_t)keep_bstride(it) * (size_t)n_cap;
}

static int keep_args(IterArgs &a, const vg_integrator *it, void *keep, size_t keep_bytes)
{
    if (keep == nullptr) return vg_fail(VG_ERR_VALUE, "kept-sample buffer missing");
    if (keep_bytes < vg_keep_bytes(it, a.ncap))
        return vg_fail(VG_ERR_VALUE, "kept-sample buffer too small: %zu < %zu", keep_bytes,
                       vg_keep_bytes(it, a.ncap));
    a.keep_jac = keep;
    a.keep_bins = (unsigned short *)((char *)keep + keep_jac_bytes(it, a.ncap));
    a.keep_bstride = keep_bstride(it);
    return VG_OK;
}

extern "C" int vg_sample_keep(const vg_integrator *it, uint32_t itn, const double *u, void *x, void *y,
                              double *wgt, int64_t *hcube, int64_t n_cap, void *keep, size_t keep_bytes,
                              void *stream)
{
    VG_RANGE("vg_sample_keep");
    vg_clear_error();
    IterArgs a;
    int rc = fill_args(a, it, itn, u);
    if (rc) return rc;
    if (n_cap < a.ncap) return vg_fail(VG_ERR_VALUE, "output capacity %lld < %lld",
                                       (long long)n_cap, (long long)a.ncap);
    if ((rc = keep_args(a, it, keep, keep_bytes))) return rc;
    a.x_out = x;
    a.y_out = y;
    a.wgt_out = wgt;
    a.hc_out = hcube;
    a.train = 0;
    a.train_hc = 0;
    a.adaptive = 0;
    a.x_vec = (a.dim % 4 == 0) && ((uintptr_t)x & 15) == 0;
    cudaStream_t st = (cudaStream_t)stream;
    if (it->precision == VG_F64 && (rc = reset_counter(a, st))) return rc;   // FP64 tiles are taken from a counter
    return vg::launch_points(a, it->precision == VG_F64, st);
}

extern "C" int vg_reduce_kept(const vg_integrator *it, uint32_t itn, const double *u, const void *f, int f_dtype,
                              const void *keep, size_t keep_bytes, void *stream)
{
    VG_RANGE("vg_reduce_kept");
    vg_clear_error();
    IterArgs a;
    int rc = fill_args(a, it, itn, u);   // itn, u: the finalize regenerates a cut hypercube's last sample
                                         // under adapt_to_errors
    if (rc) return rc;
    if ((rc = keep_args(a, it, const_cast<void *>(keep), keep_bytes))) return rc;
    a.f_in = f;
    a.f_f64 = (f_dtype == VG_F64);
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = vg::launch_reduce_kept(a, it->precision == VG_F64, st))) return rc;   // static tiles
    return vg::finalize_launch(a, st, it->precision == VG_F32, nullptr);
}

static unsigned long long *g_term_count = nullptr;
namespace vg {
uint32_t g_wait_iters = VG_WAIT_ITERS_DEFAULT;
int g_eval_split = 0;
int g_tile_table = -1, g_tile_hist = -1;
}

// Tuning of the iteration kernels: grid table and training histogram in
// shared memory (-1 automatic, 0 off, 1 on where it fits).  s_dim4, samples
// per thread of an earlier FP32 kernel, is checked and has no effect.
extern "C" int vg_set_tile_tuning(int s_dim4, int table_smem, int hist_smem)
{
    if (s_dim4 != 0 && s_dim4 != 2 && s_dim4 != 4) return vg_fail(VG_ERR_VALUE, "s_dim4 %d", s_dim4);
    if (table_smem < -1 || table_smem > 1 || hist_smem < -1 || hist_smem > 1)
        return vg_fail(VG_ERR_VALUE, "shared-memory policy");
    vg::g_tile_table = table_smem;
    vg::g_tile_hist = hist_smem;
    return VG_OK;
}

// Polls of the bounded device-side waits (allocation look-back; four times
// as many for the batched launch's group barriers) before they give up and
// report VG_ERR_TIMEOUT; a negative value restores the default.  Read when
// an iteration's arguments are filled (vg_allocate, vg_iterate, ...,
// vg_batch_prepare).
extern "C" int vg_set_wait_budget(int64_t iters)
{
    vg::g_wait_iters = iters < 0 ? VG_WAIT_ITERS_DEFAULT
                                 : (iters > 0xffffffffll ? 0xffffffffu : (uint32_t)iters);
    return VG_OK;
}

// Tuning: how FP32 iterations of the ridge run -- 0 automatic, 1 the single
// fused kernel, 2 split into EVAL (writes f) + REDUCE.
extern "C" int vg_set_eval_split(int policy)
{
    if (policy < 0 || policy > 2) return vg_fail(VG_ERR_VALUE, "split policy %d", policy);
    vg::g_eval_split = policy;
    return VG_OK;
}

// Instrumentation: while set, the FP32 ridge adds the number of Gaussian
// terms it evaluates to *count (device); NULL turns it off.
extern "C" int vg_set_term_counter(unsigned long long *count)
{
    g_term_count = count;
    return VG_OK;
}

// Validate the parameters of a built-in integrand and fill P (including its
// host-precomputed FP32 constants); tab_len = length of its per-CTA table.
int vg_build_params(int kind, int dim, const double *params, int nparams, VgParams *Pp, int *tab_len_out)
{
    if (nparams < 0 || nparams > VG_MAX_PARAMS) return vg_fail(VG_ERR_VALUE, "too many params");
    VgParams &P = *Pp;
    memset(&P, 0, sizeof(P));
    P.n = nparams;
    for (int i = 0; i < nparams; i++) P.p[i] = params[i];
    int need = 0, tab_len = 0;
    switch (kind) {
    case VG_F_GAUSS: need = 3; break;
    case VG_F_RIDGE:
        need = 2;
        if (nparams >= 2 && (params[0] < 1 || params[0] > 16384))
            return vg_fail(VG_ERR_VALUE, "ridge M out of range 1..16384");
        tab_len = nparams >= 1 ? (int)params[0] : 0;
        break;
    case VG_F_LORENTZ: need = 2 * dim; tab_len = 4 * dim; break;
    case VG_F_MIXTURE:
        need = nparams >= 1 ? 2 + (int)params[0] * dim : 1;
        if (nparams >= 1 && (params[0] < 1 || params[0] * dim > VG_MAX_PARAMS - 2))
            return vg_fail(VG_ERR_VALUE, "mixture size out of range");
        tab_len = nparams >= 1 ? (int)params[0] * dim : 0;
        break;
    case VG_F_LATTICE: need = 2; break;
    case VG_F_CONST: need = 1; break;
    default: return vg_fail(VG_ERR_VALUE, "unknown integrand kind %d", kind);
    }
    if (nparams < need) return vg_fail(VG_ERR_VALUE, "integrand needs %d parameters", need);
    vg_prepare_f32_host(P, kind, dim);
    P.term_count = (kind == VG_F_RIDGE) ? g_term_count : nullptr;
    *tab_len_out = tab_len;
    return VG_OK;
}

extern "C" int vg_fused_iteration(const vg_integrator *it, uint32_t itn, const double *u, int kind,
                                  const double *params, int nparams, void *stream)
{
    VG_RANGE("vg_fused_iteration");
    vg_clear_error();
    IterArgs a;
    int rc = fill_args(a, it, itn, u);
    if (rc) return rc;
    VgParams P;   // copied into the kernel arguments at launch
    int tab_len = 0;
    if ((rc = vg_build_params(kind, it->dim, params, nparams, &P, &tab_len))) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    if ((rc = vg::launch_fused(a, kind, P, tab_len, it->precision == VG_F64, st))) return rc;
    return vg::finalize_launch(a, st, it->precision == VG_F32, nullptr);
}

// forward declaration: one full iteration (below)
extern "C" int vg_end_iteration(const vg_integrator *it, void *stream);

int vg_adapt_launch(int dim, const int64_t *old_ninc, const int64_t *new_ninc, const double *grid,
                    const double *inc, int64_t ldg, int64_t ldi, const double *sum_f,
                    const uint64_t *n_f, double alpha, double *new_grid, double *new_inc,
                    int64_t ldg_new, int64_t ldi_new, cudaStream_t st, int fast, int zero_hist);
int vg_adapt_in_place_ok(int max_old);
int vg_adapt_cluster_args(vgadapt::AdaptArgs &a, int dim, const int64_t *ninc, double *grid, double *inc, int64_t ldg,
                          int64_t ldi, double *sum_f, uint64_t *n_f, double alpha, int fast);

extern "C" int vg_end_iteration(const vg_integrator *it, void *stream)
{
    VG_RANGE("vg_end_iteration");
    vg_clear_error();
    cudaStream_t st = (cudaStream_t)stream;
    if (!(it->adapt && it->alpha > 0)) return VG_OK;
    int64_t kmin = it->ninc[0], kmax = it->ninc[0];
    for (int d = 1; d < it->dim; d++) {
        kmin = it->ninc[d] < kmin ? it->ninc[d] : kmin;
        kmax = it->ninc[d] > kmax ? it->ninc[d] : kmax;
    }
    if (kmin > 1 && vg_adapt_in_place_ok((int)kmax))   // one kernel: adapt in place, clear the histogram
        return vg_adapt_launch(it->dim, it->ninc, it->ninc, it->grid, it->inc, it->ldg, it->ldi, it->sum_f,
                               it->n_f, it->alpha, it->grid, it->inc, it->ldg, it->ldi, st,
                               it->precision == VG_F32, 1);
    WorkLayout L = layout(it, neval_cap(it));
    if (it->work_bytes < L.total) return vg_fail(VG_ERR_VALUE, "workspace too small");
    char *w = (char *)it->work;
    double *ng = (double *)(w + L.newgrid);
    double *ni = (double *)(w + L.newinc);
    int rc = vg_adapt_launch(it->dim, it->ninc, it->ninc, it->grid, it->inc, it->ldg, it->ldi,
                             it->sum_f, it->n_f, it->alpha, ng, ni, it->ldg, it->ldi, st,
                             it->precision == VG_F32, 0);
    if (rc) return rc;
    VG_CUDA_CHECK(cudaMemcpyAsync(it->grid, ng, sizeof(double) * it->dim * it->ldg,
                                  cudaMemcpyDeviceToDevice, st));
    VG_CUDA_CHECK(cudaMemcpyAsync(it->inc, ni, sizeof(double) * it->dim * it->ldi,
                                  cudaMemcpyDeviceToDevice, st));
    VG_CUDA_CHECK(cudaMemsetAsync(it->sum_f, 0, sizeof(double) * it->dim * it->ldi, st));
    VG_CUDA_CHECK(cudaMemsetAsync(it->n_f, 0, sizeof(uint64_t) * it->dim * it->ldi, st));
    return VG_OK;
}

// One full vegas+ iteration = vg_allocate + vg_fused_iteration +
// vg_end_iteration, enqueued by one call: allocation, tiles, and one kernel
// that finalizes and adapts (adapt_to_errors, whose finalize adds to the
// training histogram, and maps the cluster form does not take adapt after the
// finalize).  rec: a copy of the iteration's record goes there.
static int iterate(const vg_integrator *it, uint32_t itn, int kind, const double *params, int nparams, vg_stats *rec,
                   cudaStream_t st)
{
    int rc = vg_allocate(it, st);
    if (rc) return rc;
    vg_clear_error();
    IterArgs a;
    if ((rc = fill_args(a, it, itn, nullptr))) return rc;
    VgParams P;   // copied into the kernel arguments at launch
    int tab_len = 0;
    if ((rc = vg_build_params(kind, it->dim, params, nparams, &P, &tab_len))) return rc;
    const int f64 = it->precision == VG_F64;
    if ((rc = vg::launch_fused(a, kind, P, tab_len, f64, st))) return rc;
    vgadapt::AdaptArgs ad;
    if (!(it->adapt && it->alpha > 0) || it->adapt_to_errors ||
        !vg_adapt_cluster_args(ad, it->dim, it->ninc, it->grid, it->inc, it->ldg, it->ldi, it->sum_f, it->n_f, it->alpha,
                               !f64)) {
        if ((rc = vg::finalize_launch(a, st, !f64, rec))) return rc;
        return vg_end_iteration(it, st);
    }
    const int nfin = f64 ? (int)finalize_blocks(a) : 1;
    const int C = vgadapt::CLUSTER;
    const unsigned grid = (unsigned)(C * (it->dim + (nfin + C - 1) / C));
    // placed early, its CTAs would all wait on the few SMs that come free first
    // and share their FP64 pipes there: an ordinary launch
    tail_kernel<<<grid, FIN_NT, 0, st>>>(a, ad, f64, nfin, rec);
    VG_LAUNCH_CHECK();
    return VG_OK;
}

extern "C" int vg_iterate(const vg_integrator *it, uint32_t itn, int kind, const double *params, int nparams,
                          void *stream)
{
    VG_RANGE("vg_iterate");
    return iterate(it, itn, kind, params, nparams, nullptr, (cudaStream_t)stream);
}

extern "C" int vg_iterate_record(const vg_integrator *it, uint32_t itn, int kind, const double *params, int nparams,
                                 vg_stats *rec, void *stream)
{
    VG_RANGE("vg_iterate_record");
    return iterate(it, itn, kind, params, nparams, rec, (cudaStream_t)stream);
}
