// vg_array.cu -- per-hypercube reduction of array-valued integrands.
//
// Reference: Integrator.__call__, src/vegas/_vegas.pyx:2136-2193 (the loops
// over fcn_size s): per hypercube, per component c the sums
//     sum_wf[c]  = sum_j wgt_j f_jc
//     dwf_c      = wgt_j f_jc - sum_wf[c]/n;  |dwf_c| < EPSILON |mean_c| ->
//                  sum_dwf2[c,c] += (EPSILON |mean_c|)^2 and dwf_c = 0
//                  (which removes it from the off-diagonal products)
//     sum_dwf[c] += dwf_c;  sum_dwf2[c,t] += dwf_c dwf_t  (t < c, correlated)
// and the iteration totals mean[c] += sum_wf[c] + sum_dwf[c] (Neely),
// var[c,t] += (n sum_dwf2[c,t] - sum_dwf[c] sum_dwf[t]) / (n - 1).
// sigf and the training histogram come from component 0 only (pyx:2173,
// 2181-2186): the scalar reduction (vg_reduce on column 0) does those.
//
// FP64 throughout, bound by the FP64 pipe (19 cycles per warp instruction and
// SM): a warp takes 32 neighbouring hypercubes, one per lane, so that each FP64
// instruction serves 32 samples; hypercubes of more than SMALL_N samples are
// then taken by the whole warp one after the other.  (One warp per hypercube
// spent most of its time in the warp sums: 5 FP64 adds of 32 lanes for each of
// s + s(s+1)/2 sums of typically 8 samples.  3e5 samples of 4 correlated
// components in dim 3: 900 us, and 730 us for the sum over the warps by one
// thread per value; see below for the sums now.)  Per-lane totals in a fixed
// order, summed over the CTA and then over the CTAs with Neumaier compensation
// -- deterministic.  Uncorrelated components are independent, so more than 16
// of them are reduced 16 at a time (one pair of launches per group of columns).
#include <string.h>

#include "vg_tile.cuh"

namespace {

constexpr int AW = 8;              // warps per CTA
constexpr int ANT = AW * 32;

struct ArrArgs {
    int64_t H;
    const int64_t *offsets;
    const int32_t *neval_h;
    const double *wgt;
    const void *f;
    int f64;
    int s;                         // components in this launch
    int c0, ld;                    // first column of this launch, row length of f
    double *parts;                 // [CTAs][nval]
    int nval;
};

__device__ __forceinline__ double fval(const ArrArgs &a, int64_t j, int c)
{
    const int64_t i = j * a.ld + a.c0 + c;
    return a.f64 ? ((const double *)a.f)[i] : (double)((const float *)a.f)[i];
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}

constexpr int SMALL_N = 24;        // samples of a hypercube that one lane reduces

// The sums of one hypercube.
template <int SM, bool CORR>
struct ArrSums {
    static constexpr int NP = CORR ? SM * (SM + 1) / 2 : SM;
    double sw[SM], sd[SM], q[NP];

    // samples j0, j0 + step, ... of the n at off: sum of wgt f (pyx:2143)
    __device__ __forceinline__ void pass1(const ArrArgs &a, int64_t off, int n, int j0, int step)
    {
#pragma unroll
        for (int c = 0; c < SM; c++) sw[c] = 0.0;
        for (int j = j0; j < n; j += step) {
            const double w = a.wgt[off + j];
#pragma unroll
            for (int c = 0; c < SM; c++)
                if (c < a.s) sw[c] = __dadd_rn(sw[c], __dmul_rn(w, fval(a, off + j, c)));
        }
    }
    // deviations from the mean and their products (pyx:2149-2172)
    __device__ __forceinline__ void pass2(const ArrArgs &a, int64_t off, int n, int j0, int step)
    {
        double mc[SM], thr[SM];
#pragma unroll
        for (int c = 0; c < SM; c++) {
            mc[c] = __ddiv_rn(sw[c], (double)n);
            thr[c] = __dmul_rn(VG_EPSILON, fabs(mc[c]));
            sd[c] = 0.0;
        }
#pragma unroll
        for (int p = 0; p < NP; p++) q[p] = 0.0;
        for (int j = j0; j < n; j += step) {
            const double w = a.wgt[off + j];
            double d[SM];
#pragma unroll
            for (int c = 0; c < SM; c++) {
                d[c] = 0.0;
                if (c >= a.s) continue;
                double dv = __dsub_rn(__dmul_rn(w, fval(a, off + j, c)), mc[c]);
                const int qi = CORR ? c * (c + 1) / 2 + c : c;
                if (fabs(dv) < thr[c]) {
                    q[qi] = __dadd_rn(q[qi], __dmul_rn(thr[c], thr[c]));
                    dv = 0.0;
                } else {
                    q[qi] = __dadd_rn(q[qi], __dmul_rn(dv, dv));
                }
                sd[c] = __dadd_rn(sd[c], dv);
                d[c] = dv;
                if (CORR) {
#pragma unroll
                    for (int t = 0; t < SM; t++)
                        if (t < c) q[c * (c + 1) / 2 + t] = __dadd_rn(q[c * (c + 1) / 2 + t], __dmul_rn(dv, d[t]));
                }
            }
        }
    }
    // the hypercube's mean and (co)variance added to M and V
    __device__ __forceinline__ void add_to(const ArrArgs &a, int n, double (&M)[SM], double (&V)[NP]) const
    {
        const double nd = (double)n, n1 = __dsub_rn(nd, 1.);
#pragma unroll
        for (int c = 0; c < SM; c++) {
            if (c >= a.s) continue;
            M[c] = __dadd_rn(M[c], __dadd_rn(sw[c], sd[c]));
#pragma unroll
            for (int t = 0; t < SM; t++) {
                if (t > c || (!CORR && t < c)) continue;
                const int p = CORR ? c * (c + 1) / 2 + t : c;
                V[p] = __dadd_rn(V[p], __ddiv_rn(__dsub_rn(__dmul_rn(nd, q[p]), __dmul_rn(sd[c], sd[t])), n1));
            }
        }
    }
};

template <int SM, bool CORR>
__global__ void __launch_bounds__(ANT) array_hcube_kernel(ArrArgs a)
{
    constexpr int NP = ArrSums<SM, CORR>::NP;
    __shared__ double s_part[AW][SM + NP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t gw = (int64_t)blockIdx.x * AW + warp;
    const int64_t nw = (int64_t)gridDim.x * AW;
    double M[SM], V[NP];
#pragma unroll
    for (int c = 0; c < SM; c++) M[c] = 0.0;
#pragma unroll
    for (int p = 0; p < NP; p++) V[p] = 0.0;
    for (int64_t h0 = gw * 32; h0 < a.H; h0 += nw * 32) {
        const int64_t h = h0 + lane;
        const int64_t off = h < a.H ? a.offsets[h] : 0;
        const int n = h < a.H ? a.neval_h[h] : 0;
        ArrSums<SM, CORR> s;
        if (n > 0 && n <= SMALL_N) {
            s.pass1(a, off, n, 0, 1);
            s.pass2(a, off, n, 0, 1);
            s.add_to(a, n, M, V);
        }
        for (unsigned int big = __ballot_sync(0xffffffffu, n > SMALL_N); big; big &= big - 1) {
            const int k = __ffs(big) - 1;
            const int64_t ok = __shfl_sync(0xffffffffu, off, k);
            const int nk = __shfl_sync(0xffffffffu, n, k);
            s.pass1(a, ok, nk, lane, 32);
#pragma unroll
            for (int c = 0; c < SM; c++) s.sw[c] = warp_sum(s.sw[c]);
            s.pass2(a, ok, nk, lane, 32);
#pragma unroll
            for (int c = 0; c < SM; c++) s.sd[c] = warp_sum(s.sd[c]);
#pragma unroll
            for (int p = 0; p < NP; p++) s.q[p] = warp_sum(s.q[p]);
            if (lane == k) s.add_to(a, nk, M, V);
        }
    }
#pragma unroll
    for (int c = 0; c < SM; c++) M[c] = warp_sum(M[c]);
#pragma unroll
    for (int p = 0; p < NP; p++) V[p] = warp_sum(V[p]);
    if (lane == 0) {
#pragma unroll
        for (int c = 0; c < SM; c++) s_part[warp][c] = M[c];
#pragma unroll
        for (int p = 0; p < NP; p++) s_part[warp][SM + p] = V[p];
    }
    __syncthreads();
    for (int v = threadIdx.x; v < a.nval; v += ANT) {   // value v: component v, or pair v - s
        const int i = v < a.s ? v : SM + v - a.s;
        VgKSum k = {0.0, 0.0};
        for (int w = 0; w < AW; w++) k.add(s_part[w][i]);
        a.parts[(int64_t)blockIdx.x * a.nval + v] = k.value();
    }
}

// Fixed-order compensated sum of the CTAs' partials, one warp per value (CTA),
// unpacked into mean[s] and the s x s (co)variance matrix.
// Components c0 .. c0+s-1 of an s_all-component integrand; the first launch
// (zero = 1) clears the entries off the diagonal.
__global__ void __launch_bounds__(32) array_total_kernel(const double *__restrict__ parts, int np, int nval, int s,
                                                         int corr, int c0, int s_all, int zero,
                                                         double *__restrict__ mean_out, double *__restrict__ var_out)
{
    const int v = blockIdx.x, lane = threadIdx.x;
    if (zero && !corr)
        for (int i = v * 32 + lane; i < s_all * s_all; i += nval * 32)
            if (i / s_all != i % s_all) var_out[i] = 0.0;
    VgKSum k = {0.0, 0.0};
    for (int w = lane; w < np; w += 32) k.add(parts[(int64_t)w * nval + v]);
    k = vg_block_ksum<32>(k, nullptr);
    if (lane != 0) return;
    const double tot = k.value();
    if (v < s) {
        mean_out[c0 + v] = tot;
    } else if (corr) {
        int p = v - s, c = 0;
        while ((c + 1) * (c + 2) / 2 <= p) c++;
        const int t = p - c * (c + 1) / 2;
        var_out[c * s + t] = tot;
        var_out[t * s + c] = tot;
    } else {
        const int c = c0 + v - s;
        var_out[(int64_t)c * s_all + c] = tot;
    }
}

template <int SM, bool CORR>
int launch_array(const ArrArgs &A, int grid, int corr, int s_all, double *mean_out, double *var_out, cudaStream_t st)
{
    array_hcube_kernel<SM, CORR><<<grid, ANT, 0, st>>>(A);
    VG_LAUNCH_CHECK();
    array_total_kernel<<<A.nval, 32, 0, st>>>(A.parts, grid, A.nval, A.s, corr, A.c0, s_all, A.c0 == 0, mean_out,
                                              var_out);
    VG_LAUNCH_CHECK();
    return VG_OK;
}

}  // namespace

// mean_out[s]; var_out[s*s] (correlated: full symmetric matrix; else the
// diagonal in var_out[c*s + c], zeros elsewhere).
extern "C" int vg_reduce_array(const vg_integrator *it, const void *f, int f_dtype, int s, int correlate,
                               const double *wgt, double *mean_out, double *var_out, void *work,
                               size_t work_bytes, void *stream)
{
    VG_RANGE("vg_reduce_array");
    vg_clear_error();
    vg::IterArgs a;
    int rc = vg::fill_iter_args(a, it, 0, nullptr);
    if (rc) return rc;
    if (s < 1) return vg_fail(VG_ERR_VALUE, "s < 1");
    if (correlate && s > 6)
        return vg_fail(VG_ERR_UNSUPPORTED, "array integrands: s <= 6 correlated components");
    const int np = correlate ? s * (s + 1) / 2 : s;
    const int nval = s + np;
    // two CTAs per SM, fewer where there are fewer hypercubes
    int64_t grid = (it->nhcube + ANT - 1) / ANT;
    const int most = vg_num_sms() * 2;
    if (grid > most) grid = most;
    const size_t need = sizeof(double) * (size_t)most * nval;
    if (work_bytes < need) return vg_fail(VG_ERR_VALUE, "array workspace %zu < %zu", work_bytes, need);
    ArrArgs A;
    A.H = it->nhcube;
    A.offsets = a.offsets;
    A.neval_h = a.neval_h;
    A.wgt = wgt;
    A.f = f;
    A.f64 = (f_dtype == VG_F64);
    A.ld = s;
    cudaStream_t st = (cudaStream_t)stream;
    const int g = (int)grid;
    if (correlate) {
        A.s = s;
        A.c0 = 0;
        A.parts = (double *)work;
        A.nval = nval;
        switch (s) {   // registers follow the pairs of components
        case 1: return launch_array<1, true>(A, g, 1, s, mean_out, var_out, st);
        case 2: return launch_array<2, true>(A, g, 1, s, mean_out, var_out, st);
        case 3: return launch_array<3, true>(A, g, 1, s, mean_out, var_out, st);
        case 4: return launch_array<4, true>(A, g, 1, s, mean_out, var_out, st);
        case 5: return launch_array<5, true>(A, g, 1, s, mean_out, var_out, st);
        default: return launch_array<6, true>(A, g, 1, s, mean_out, var_out, st);
        }
    }
    for (int c0 = 0; c0 < s; c0 += 16) {   // groups of 16 independent columns
        const int sc = s - c0 < 16 ? s - c0 : 16;
        A.s = sc;
        A.c0 = c0;
        A.nval = 2 * sc;
        A.parts = (double *)work + (size_t)most * 2 * c0;
        if (sc <= 4) rc = launch_array<4, false>(A, g, 0, s, mean_out, var_out, st);
        else if (sc <= 8) rc = launch_array<8, false>(A, g, 0, s, mean_out, var_out, st);
        else rc = launch_array<16, false>(A, g, 0, s, mean_out, var_out, st);
        if (rc) return rc;
    }
    return VG_OK;
}

extern "C" size_t vg_reduce_array_work_bytes(int s, int correlate)
{
    const int np = correlate ? s * (s + 1) / 2 : s;
    return sizeof(double) * (size_t)vg_num_sms() * 2 * (s + np);
}
