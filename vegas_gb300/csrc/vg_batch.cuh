// vg_batch.cuh -- many independent vegas+ integrals in one persistent launch.
//
// One CTA runs one integral at a time, all of its iterations back to back:
// allocation of evaluations to hypercubes (pyx:1692-1706), the fused body of
// the single-integral kernel over all of the integral's samples (sampling, map,
// integrand, per-hypercube mean and variance, training histogram), the merge of
// hypercubes cut by the ends of ranges or tiles and the
// iteration sums (finalize), AdaptiveMap.adapt (pyx:467-594), and at the end
// the weighted average over the iterations after the warm-up ones
// (RAvg.add, pyx:2392-2410) -- in the arithmetic of the single-integral
// path.  CTAs take integrals from an atomic queue in an order given by the
// host (largest first), so nothing crosses CTAs and the launch needs no
// grid-wide synchronisation.
#pragma once
#include "vg_adapt.cuh"
#include "vg_range.cuh"

namespace vgbatch {
using namespace vg;

struct BatchJob {
    IterArgs a;                  // per-integral arguments (its own workspace)
    vgadapt::AdaptArgs ad;       // adapt: grid -> scratch grid of the workspace
    double *out;                 // [nitn][3] iteration mean, variance, evaluations
    double *res;                 // [4] weighted mean, sdev, chi2, dof
    unsigned int *sync;          // group barrier counter (group mode)
    int bucket;                  // dimension bucket: 0 (dim <= 4), 1 (<= 8), 2 (<= 16)
    int adapt;                   // adapt the map after each iteration: axes at a time (0: not)
    unsigned long long *stamp;   // instrumentation (or nullptr): [0] start, [1] end (globaltimer ns), [2] SM
};

__device__ __forceinline__ unsigned long long vg_globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ unsigned int vg_smid()
{
    unsigned int r;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(r));
    return r;
}

// Barrier of the G CTAs working on one integral (group mode; the launch is
// cooperative, so they are co-resident).  Thread 0 releases this CTA's
// writes, arrives, and waits (at most 4 wait_iters polls) until all G
// arrived `round` times.
// Returns false when the wait gave up.
__device__ __forceinline__ bool group_barrier(unsigned int *ctr, unsigned int target, uint32_t wait_iters)
{
    __shared__ int s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(ctr, 1u);
        int ok = 0;
        const uint64_t budget = 4ull * wait_iters;
        for (uint64_t i = 0; i < budget; i++) {
            unsigned int v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ctr) : "memory");
            if (v >= target) {
                ok = 1;
                break;
            }
            __nanosleep(256);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0;
}

// Shared memory of an axis' adaptation: weights, cumulative sums, partial sums
// (block_sum takes 33).
__host__ __device__ constexpr size_t adapt_group_doubles(int max_old) { return 2 * (size_t)max_old + 34; }

constexpr int APER = 4;          // hypercubes per thread and pass of the allocation
constexpr int F64_S = 2;         // samples per thread of the FP64 tiles

// Chunks of 128 samples in a unit: one where a CTA has the integral to itself
// (its warps then stay together in the sample order), four in a group of CTAs.
__device__ __forceinline__ int deal_chunks(int G) { return G > 1 ? 4 : 1; }

// The arguments of the CTA's integral.  The functions that are not inlined into
// the kernel name this variable and the dynamic shared memory themselves: through
// a pointer parameter every access to the arguments, the grid table and the
// histogram would be a generic one (the 16-dimensional lattice took 5 % longer).
__device__ __forceinline__ IterArgs &job_args()
{
    __shared__ IterArgs sa;
    return sa;
}

// Allocation of one iteration by one CTA: neval_h, offsets, tile heads,
// totals in the integral's stats (the three allocation kernels' work).
static __device__ __noinline__ void cta_alloc(int64_t *scan /* one per warp */)
{
    const IterArgs &a = job_args();
    const int tid = threadIdx.x, NTB = (int)blockDim.x;
    build_tablef(a, tid, NTB);   // the FP32 grid table of this iteration
    vg_stats *st = a.stats;
    const double sum_sigf = st->sum_sigf;
    const double nsf = (a.beta > 0 && sum_sigf > 0)
                           ? __ddiv_rn(__dmul_rn(a.neval_frac, (double)a.neval), sum_sigf)
                           : 0.0;
    const int64_t mx = a.max_neval_hcube > a.min_neval_hcube ? a.max_neval_hcube : a.min_neval_hcube;
    const int64_t avg = (int64_t)((double)a.neval / (double)a.H);
    int64_t run = 0, mxn = 0;
    if (!a.adaptive_alloc) {   // as many in every hypercube: offsets are products
        for (int64_t h = tid; h < a.H; h += NTB) {
            const int64_t off = h * avg;
            a.neval_h[h] = (int32_t)avg;
            a.offsets[h] = off;
            for (int64_t tt = (off + BASE_TILE - 1) / BASE_TILE; tt * BASE_TILE < off + avg; tt++)
                if (tt < a.ntiles_cap) a.tile_h0[tt] = h;
        }
        run = a.H * avg;
        __syncthreads();   // the sentinel below comes after the tiles
    }
    for (int64_t base = a.adaptive_alloc ? 0 : a.H; base < a.H; base += (int64_t)NTB * APER) {
        int64_t loc[APER];
        int64_t s = 0;
#pragma unroll
        for (int k = 0; k < APER; k++) {
            const int64_t h = base + (int64_t)tid * APER + k;
            int64_t n = 0;
            if (h < a.H) {
                n = (int64_t)__dmul_rn(a.sigf[h], nsf) + a.min_neval_hcube;
                if (n > mx) n = mx;
                mxn = n > mxn ? n : mxn;
            }
            loc[k] = n;
            s += n;
        }
        int64_t total;
        int64_t off = run + block_excl_scan(s, scan, &total);
#pragma unroll
        for (int k = 0; k < APER; k++) {
            const int64_t h = base + (int64_t)tid * APER + k;
            if (h >= a.H) break;
            const int64_t n = loc[k];
            a.neval_h[h] = (int32_t)n;
            a.offsets[h] = off;
            for (int64_t tt = (off + BASE_TILE - 1) / BASE_TILE; tt * BASE_TILE < off + n; tt++)
                if (tt < a.ntiles_cap) a.tile_h0[tt] = h;
            off += n;
        }
        run += total;
    }
    if (a.adaptive_alloc) mxn = block_max(mxn, scan);
    if (tid == 0) {
        const int64_t N = run;
        int64_t ntiles = (N + BASE_TILE - 1) / BASE_TILE;
        a.offsets[a.H] = N;
        st->neval = N;
        st->neval_sigf = nsf;
        st->range_lo = a.min_neval_hcube;
        st->range_hi = a.adaptive_alloc ? (mxn > a.min_neval_hcube ? mxn : a.min_neval_hcube)
                                        : a.min_neval_hcube;
        if (N > a.ncap || ntiles + 1 > a.ntiles_cap) {
            st->status = VG_ERR_MEMORY;
            ntiles = 0;
        } else {
            st->status = VG_OK;
            a.tile_h0[ntiles] = a.H;
        }
        st->ntiles = ntiles;
        st->nan_seen = 0;
        *a.counter = 0ull;
    }
    __syncthreads();
}

// Iteration sums of one integral by one CTA: the partial sums of the group's
// CTAs plus the Chan et al. merge of every hypercube cut by the ends of the
// warps' ranges (the finalize kernels' work); sum_sigf and the constant-integrand
// reset (pyx:2209-2215).
static __device__ __noinline__ void cta_finalize(int ngroup, int *flag)
{
    const IterArgs &a = job_args();
    const int tid = threadIdx.x, NTB = (int)blockDim.x;
    vg_stats *st = a.stats;
    float s6[6];
    finalize_ranges(a, ngroup, (int64_t)ngroup * (NTB / 32 / GROUP), deal_chunks(ngroup), s6);
    if (tid == 0) {
        st->mean = vg_ff_value(s6[0], s6[1]);
        st->var = vg_ff_value(s6[2], s6[3]);
        st->sigf_reset = 0;
        *flag = 0;
        if (a.adaptive) {
            const double ss = vg_ff_value(s6[4], s6[5]);
            if (ss > 0) {
                st->sum_sigf = ss;
            } else {
                st->sum_sigf = (double)a.H;
                st->sigf_reset = 1;
                *flag = 1;
            }
        }
    }
    __syncthreads();
    if (*flag)
        for (int64_t h = tid; h < a.H; h += NTB) a.sigf[h] = 1.0;
    __syncthreads();
}

// FP64 mode: the hypercube whose first piece is the tail record of tile t,
// merged in FP64 with its pieces in the following tiles (Chan et al.'s
// parallel-variance update, the FP64 finalize's formulas); adds its mean,
// variance and sigf to the compensated sums and stores its sigf.
static __device__ __noinline__ void merge_cut_f64(const IterArgs &a, int64_t t, int64_t ntiles, VgKSum &cm,
                                                  VgKSum &cv, VgKSum &cs)
{
    const TileRec r = a.recs[2 * t + 1];
    if (r.h < 0) return;
    double n = r.n, Sx = r.S, Q = r.Q, D = r.D;
    for (int64_t t2 = t + 1; t2 < ntiles; t2++) {
        const TileRec q = a.recs[2 * t2];
        if (q.h != r.h) break;
        const double n2 = n + q.n;
        const double delta = q.S / q.n - Sx / n;
        Q = Q + q.Q + delta * delta * (n * q.n / n2);
        Sx += q.S;
        D += q.D;
        n = n2;
        if (!q.spans) break;
    }
    const double num = __dsub_rn(__dmul_rn(n, Q), __dmul_rn(D, D));
    const double vh = __ddiv_rn(num, __dsub_rn(n, 1.));
    cm.add(__dadd_rn(Sx, D));
    cv.add(vh);
    if (a.adaptive) {
        const double sg = pow(fabs(vh), a.beta_half);
        a.sigf[r.h] = sg;
        cs.add(sg);
    }
}

// FP64 mode (the parity configuration of the batched launch): the group
// CTAs' FP64 partials plus the merged cut hypercubes, compensated FP64 sums
// in a fixed order; sum_sigf and the constant-integrand reset as
// cta_finalize.
static __device__ __noinline__ void cta_finalize_f64(const IterArgs &a, int ngroup, VgKSum *red, int *flag)
{
    const int tid = threadIdx.x;
    vg_stats *st = a.stats;
    const int64_t N = st->neval;
    const int64_t ntiles = st->ntiles ? (N + a.T - 1) / a.T : 0;
    VgKSum cm = {0.0, 0.0}, cv = {0.0, 0.0}, cs = {0.0, 0.0};
    if (tid < ngroup && ntiles > 0) {
        const TilePart p = a.parts[tid];
        cm = p.mean;
        cv = p.var;
        cs = p.sigf;
    }
    for (int64_t t = tid; t < ntiles; t += NT) merge_cut_f64(a, t, ntiles, cm, cv, cs);
    VgKSum v3[3] = {cm, cv, cs};
    vg_block_ksum3<NT>(v3, red);
    if (tid == 0) {
        st->mean = v3[0].value();
        st->var = v3[1].value();
        st->sigf_reset = 0;
        *flag = 0;
        if (a.adaptive) {
            const double ss = v3[2].value();
            if (ss > 0) {
                st->sum_sigf = ss;
            } else {
                st->sum_sigf = (double)a.H;
                st->sigf_reset = 1;
                *flag = 1;
            }
        }
    }
    __syncthreads();
    if (*flag)
        for (int64_t h = tid; h < a.H; h += NT) a.sigf[h] = 1.0;
    __syncthreads();
}

// End of iteration: adapt the map, copy the new grid back, clear the training
// histogram (vg_end_iteration's work).  An axis is a chain of FP64 sums, scans
// and searches, bound by their latency with 256 threads as with 1024, so the
// CTA adapts an axis per 256 threads at a time.  (Only an axis of a single
// increment would use the weights that pyx:533 carries from axis to axis, and
// its nodes are fixed.)  Of a group of G CTAs each adapts some of the axes
// (16 axes and 9 CTAs on each of 16 lattice integrals: 4.32 -> 4.08 ms).
static __device__ __noinline__ void cta_adapt(const BatchJob &J, int rank, int G)
{
    extern __shared__ __align__(16) unsigned char smem[];
    const IterArgs &a = job_args();
    const int tid = threadIdx.x, NTB = (int)blockDim.x;
    const vgadapt::AdaptArgs &ad = J.ad;
    const int ng = J.adapt, grp = tid / vgadapt::GROUP_NT, step = ng * G;
    if (grp < ng) {
        double *avg = (double *)smem + (size_t)grp * adapt_group_doubles(ad.max_old);
        double *tmp = avg + ad.max_old;
        double *part = tmp + ad.max_old;
        const vgadapt::PartOfCta part_of_cta;
        for (int i = part_of_cta.t(); i < ad.max_old; i += vgadapt::GROUP_NT) avg[i] = 1.0;
        part_of_cta.sync();
        for (int d = rank * ng + grp; d < ad.dim; d += step)
            vgadapt::adapt_axis<vgadapt::GROUP_NT>(ad, d, avg, tmp, part, nullptr, nullptr, part_of_cta);
    }
    __syncthreads();
    for (int d = rank * ng; d < ad.dim; d += d % ng == ng - 1 ? step - ng + 1 : 1) {   // this CTA's axes
        const int K = ad.old_ninc[d];
        double *g = const_cast<double *>(ad.grid) + d * ad.ldg;
        double *inc = const_cast<double *>(ad.inc) + d * ad.ldi;
        for (int i = tid; i <= K; i += NTB) g[i] = ad.new_grid[d * ad.ldg_new + i];
        for (int i = tid; i < K; i += NTB) {
            inc[i] = ad.new_inc[d * ad.ldi_new + i];
            a.sum_f[d * a.ldi + i] = 0.0;
            a.n_f[d * a.ldi + i] = 0ull;
        }
    }
    __syncthreads();
}

// Weighted average of iterations [nwarm, nitn) (RAvg, pyx:2392-2410):
// mean = sum(m/v)/sum(1/v), sdev = sum(1/v)^-1/2, chi2 = sum((m-mean)^2/v).
static __device__ __noinline__ void cta_ravg(const BatchJob &J, int nitn, int nwarm)
{
    if (threadIdx.x != 0) return;
    double sw = 0.0, swm = 0.0;
    int cnt = 0;
    for (int i = nwarm; i < nitn; i++) {
        const double m = J.out[3 * i], v = J.out[3 * i + 1];
        if (v > 0) {
            sw += 1.0 / v;
            swm += m / v;
        }
        cnt++;
    }
    const double mean = sw > 0 ? swm / sw : 0.0;
    double chi2 = 0.0;
    for (int i = nwarm; i < nitn; i++) {
        const double m = J.out[3 * i], v = J.out[3 * i + 1];
        if (v > 0) chi2 += (m - mean) * (m - mean) / v;
    }
    J.res[0] = mean;
    J.res[1] = sw > 0 ? 1.0 / sqrt(sw) : 0.0;
    J.res[2] = chi2;
    J.res[3] = (double)(cnt > 0 ? cnt - 1 : 0);
}

// The fused body of one integral, compiled for its dimension.
template <int KIND, int DIM, int F>
static __device__ __noinline__ void cta_range(const VgParams &prm, int rank, int G)
{
    extern __shared__ __align__(16) unsigned char smem[];
    range_body<MODE_FUSED, KIND, DIM, F>(job_args(), prm, smem, rank, G, deal_chunks(G));
}

template <int KIND, int DIMB>
__device__ __forceinline__ void range_dispatch(const VgParams &prm, int rank, int G)
{
    const IterArgs &a = job_args();
    constexpr int ET = RF_EXACT | RF_TABLE;
    if (a.wide || a.few || (a.train && !a.hist_smem) || (DIMB <= 8 && !a.table_smem))
        return cta_range<KIND, DIMB, RF_GENERAL>(prm, rank, G);
    if constexpr (DIMB == 4) {
        if (a.dim == 4) cta_range<KIND, 4, ET>(prm, rank, G);
        else if (a.dim == 3) cta_range<KIND, 3, ET>(prm, rank, G);
        else if (a.dim == 2) cta_range<KIND, 2, ET>(prm, rank, G);
        else cta_range<KIND, 1, ET>(prm, rank, G);
    } else if constexpr (DIMB == 8) {
        if (a.dim == 8) cta_range<KIND, 8, ET>(prm, rank, G);
        else if (a.dim == 7) cta_range<KIND, 7, ET>(prm, rank, G);
        else if (a.dim == 6) cta_range<KIND, 6, ET>(prm, rank, G);
        else cta_range<KIND, 5, ET>(prm, rank, G);
    } else {
        if (a.table_smem) cta_range<KIND, DIMB, RF_TABLE>(prm, rank, G);
        else cta_range<KIND, DIMB, 0>(prm, rank, G);
    }
}

// The persistent kernel of one dimension bucket (every integral it takes has
// dim <= DIMB): sampling, map and evaluation in T (float; double in the
// FP64 parity configuration), at most MAXT threads per CTA (the number of
// threads and of CTAs per SM is picked by the autotuner per bucket).
//
// Queue mode (group <= 1): each CTA takes whole integrals from the queue.
// Group mode (group = G >= 2, cooperative launch): CTA c works on integral
// order[c / G] as rank c % G; rank 0 allocates and finalizes, all G
// ranks share the samples and the axes to adapt, with three group barriers per
// iteration (four under adapt_to_errors).
template <typename T, int KIND, int DIMB, int MAXT>
__global__ void __launch_bounds__(MAXT, 1) batch_kernel(const BatchJob *__restrict__ jobs,
                                                   const VgParams *__restrict__ params,
                                                   const int *__restrict__ order, int njobs, int nitn,
                                                   int nwarm, uint32_t itn0, unsigned int *queue,
                                                   int group, int *status)
{
    extern __shared__ __align__(16) unsigned char smem[];
    IterArgs &sa = job_args();
    __shared__ int64_t scan[MAXT / 32];
    __shared__ VgKSum red[3 * (MAXT / 32)];
    __shared__ int s_q, s_flag;
    const int tid = threadIdx.x, NTB = (int)blockDim.x;
    const int G = group > 1 ? group : 1;
    const int rank = G > 1 ? (int)(blockIdx.x % G) : 0;
    bool first = true;
    for (;;) {
        int q;
        if (G > 1) {
            if (!first) break;
            q = (int)(blockIdx.x / G);
        } else {
            if (tid == 0) s_q = (int)atomicAdd(queue, 1u);
            __syncthreads();
            q = s_q;
            __syncthreads();
        }
        first = false;
        if (q >= njobs) break;
        const int j = order[q];
        const BatchJob &J = jobs[j];
        if (J.stamp != nullptr && tid == 0 && rank == 0) {
            J.stamp[0] = vg_globaltimer();
            J.stamp[2] = vg_smid();
        }
        {
            const int nw = (int)(sizeof(IterArgs) / 4);
            const uint32_t *src = reinterpret_cast<const uint32_t *>(&J.a);
            uint32_t *dst = reinterpret_cast<uint32_t *>(&sa);
            for (int i = tid; i < nw; i += NTB) dst[i] = src[i];
        }
        __syncthreads();
        unsigned int rounds = 0;
        bool ok = true;
        for (int it = 0; it < nitn && ok; it++) {
            if (tid == 0) sa.itn = itn0 + (uint32_t)it;
            __syncthreads();
            if (rank == 0) cta_alloc(scan);
            if (G > 1 && !(ok = group_barrier(J.sync, (unsigned)G * ++rounds, sa.wait_iters))) break;
            if (sa.stats->ntiles > 0) {
                if constexpr (sizeof(T) == 8)
                    tile_body<MODE_FUSED, KIND, DIMB, F64_S, MAXT>(sa, params[j], smem, rank, G, rank);
                else
                    range_dispatch<KIND, DIMB>(params[j], rank, G);
            }
            __syncthreads();
            if (G > 1 && !(ok = group_barrier(J.sync, (unsigned)G * ++rounds, sa.wait_iters))) break;
            if (rank == 0) {
                if constexpr (sizeof(T) == 8) cta_finalize_f64(sa, G, red, &s_flag);
                else cta_finalize(G, &s_flag);
                if (tid == 0) {
                    J.out[3 * it] = sa.stats->mean;
                    J.out[3 * it + 1] = sa.stats->var;
                    J.out[3 * it + 2] = (double)sa.stats->neval;
                }
            }
            // adapt_to_errors: the finalize still trains the map on the hypercubes
            // cut by ranges, and the other ranks are not to read or clear before
            if (G > 1 && J.adapt && sa.train_hc &&
                !(ok = group_barrier(J.sync, (unsigned)G * ++rounds, sa.wait_iters))) break;
            if (J.adapt) cta_adapt(J, rank, G);
            __syncthreads();
            if (G > 1 && J.adapt && !(ok = group_barrier(J.sync, (unsigned)G * ++rounds, sa.wait_iters))) break;
        }
        if (!ok) {
            if (tid == 0) atomicExch(status, VG_ERR_TIMEOUT);
            break;
        }
        if (rank == 0) cta_ravg(J, nitn, nwarm);
        __syncthreads();
        if (J.stamp != nullptr && tid == 0 && rank == 0) J.stamp[1] = vg_globaltimer();
    }
}

// Launch (queue mode, or cooperative for co-resident groups) and occupancy
// of one instantiation; the bucket files dispatch to these.
template <typename T, int KIND, int DIMB, int MAXT>
int launch_one(int ntb, const BatchJob *jobs, const VgParams *prm, const int *order, int njobs, int nitn, int nwarm,
               uint32_t itn0, unsigned int *queue, size_t smem, int grid, int group, int *status, cudaStream_t st)
{
    auto k = batch_kernel<T, KIND, DIMB, MAXT>;
    if (group > 1) {
        void *args[] = {(void *)&jobs, (void *)&prm, (void *)&order, (void *)&njobs, (void *)&nitn, (void *)&nwarm,
                        (void *)&itn0, (void *)&queue, (void *)&group, (void *)&status};
        VG_CUDA_CHECK(cudaLaunchCooperativeKernel((const void *)k, dim3((unsigned)grid), dim3(ntb), args, smem, st));
        return VG_OK;
    }
    k<<<grid, ntb, smem, st>>>(jobs, prm, order, njobs, nitn, nwarm, itn0, queue, group, status);
    VG_LAUNCH_CHECK();
    return VG_OK;
}

// sets the kernel's shared-memory attribute (outside any stream capture): always
// all that the kernel may have, so that plans of one batch do not lower another's
template <typename T, int KIND, int DIMB, int MAXT>
int occupancy_one(int ntb, size_t smem, int *per_sm)
{
    auto k = batch_kernel<T, KIND, DIMB, MAXT>;
    int dev = 0, most = 0;
    cudaFuncAttributes fa;
    VG_CUDA_CHECK(cudaGetDevice(&dev));
    VG_CUDA_CHECK(cudaDeviceGetAttribute(&most, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev));
    VG_CUDA_CHECK(cudaFuncGetAttributes(&fa, k));
    VG_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, most - (int)fa.sharedSizeBytes));
    VG_CUDA_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k, ntb, smem));
    return VG_OK;
}

// Configurations of each bucket: threads per CTA and CTAs per SM.
struct BucketConfig {
    int ntb, minb;
};
constexpr int NCONFIG = 3;
constexpr int NBUCKET = 3;
constexpr int BUCKET_DIM[NBUCKET] = {4, 8, 16};
// FP64 parity configuration (cfg VG_BATCH_CFG_F64): Lorentzian products of
// dim <= 8 (buckets 0 and 1 share the one instantiation), the large tiles of
// the single-integral FP64 kernel, one CTA per SM.
constexpr BucketConfig F64_CONFIG = {NT, 1};
constexpr int F64_DIMB = 8;
constexpr BucketConfig BUCKET_CONFIGS[NBUCKET][NCONFIG] = {
    {{1024, 1}, {512, 2}, {256, 4}},   // dim <= 4
    {{512, 2}, {1024, 1}, {768, 1}},   // dim <= 8
    {{768, 1}, {512, 1}, {256, 2}},    // dim <= 16
};

// One bucket's launch and occupancy for configuration cfg (instantiated by
// the bucket's own translation unit, vg_batch_b<DIMB>.cu).
template <int KIND, int DIMB>
int bucket_launch(int cfg, const BatchJob *jobs, const VgParams *prm, const int *order, int njobs, int nitn,
                  int nwarm, uint32_t itn0, unsigned int *queue, size_t smem, int grid, int group, int *status,
                  cudaStream_t st)
{
    constexpr int b = DIMB == 4 ? 0 : (DIMB == 8 ? 1 : 2);
    return launch_one<float, KIND, DIMB, range_threads(DIMB)>(BUCKET_CONFIGS[b][cfg].ntb, jobs, prm, order, njobs, nitn,
                                                              nwarm, itn0, queue, smem, grid, group, status, st);
}

template <int KIND, int DIMB>
int bucket_occupancy(int cfg, size_t smem, int *per_sm)
{
    constexpr int b = DIMB == 4 ? 0 : (DIMB == 8 ? 1 : 2);
    return occupancy_one<float, KIND, DIMB, range_threads(DIMB)>(BUCKET_CONFIGS[b][cfg].ntb, smem, per_sm);
}

// The entry points of each bucket's translation unit.
#define VG_BATCH_BUCKET_ENTRY(DIMB)                                                                             \
    int launch_b##DIMB(int kind, int cfg, const BatchJob *jobs, const VgParams *prm, const int *order,          \
                       int njobs, int nitn, int nwarm, uint32_t itn0, unsigned int *queue, size_t smem,         \
                       int grid, int group, int *status, cudaStream_t st)                                       \
    {                                                                                                           \
        if (kind == VG_F_LATTICE)                                                                               \
            return bucket_launch<VG_F_LATTICE, DIMB>(cfg, jobs, prm, order, njobs, nitn, nwarm, itn0, queue,    \
                                                     smem, grid, group, status, st);                            \
        return bucket_launch<VG_F_LORENTZ, DIMB>(cfg, jobs, prm, order, njobs, nitn, nwarm, itn0, queue, smem,  \
                                                 grid, group, status, st);                                      \
    }                                                                                                           \
    int occupancy_b##DIMB(int kind, int cfg, size_t smem, int *per_sm)                                          \
    {                                                                                                           \
        if (kind == VG_F_LATTICE) return bucket_occupancy<VG_F_LATTICE, DIMB>(cfg, smem, per_sm);               \
        return bucket_occupancy<VG_F_LORENTZ, DIMB>(cfg, smem, per_sm);                                         \
    }

}  // namespace vgbatch
