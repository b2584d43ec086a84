// vg_dropin.cu -- tile-kernel instantiations of the drop-in (torch integrand)
// path: MODE_POINTS writes x (and optionally y, weights, hypercubes, and the
// kept Jacobians and training bins) for the integrand; MODE_REDUCE reads the
// integrand values back and reduces, regenerating each sample;
// MODE_REDUCE_KEPT reduces from the kept Jacobians and bins instead.
#include "vg_range.cuh"

namespace vg {

int launch_points(IterArgs &a, int f64, cudaStream_t st)
{
    if (f64) {
        if (a.dim <= 8) return launch_tile<MODE_POINTS, 0, 8, 1>(a, nullptr, st);
        return launch_tile<MODE_POINTS, 0, 64, 1>(a, nullptr, st);
    }
    return launch_range<MODE_POINTS, 0>(a, nullptr, 0, st);
}

int launch_reduce(IterArgs &a, int f64, cudaStream_t st)
{
    if (f64) {
        if (a.dim <= 8) return launch_tile<MODE_REDUCE, 0, 8, 2>(a, nullptr, st);
        return launch_tile<MODE_REDUCE, 0, 64, 1>(a, nullptr, st);
    }
    return launch_range<MODE_REDUCE, 0>(a, nullptr, 0, st);
}

int launch_reduce_kept(IterArgs &a, int f64, cudaStream_t st)
{
    if (f64) {
        if (a.dim <= 8) return launch_tile<MODE_REDUCE_KEPT, 0, 8, 2>(a, nullptr, st);
        return launch_tile<MODE_REDUCE_KEPT, 0, 64, 1>(a, nullptr, st);
    }
    return launch_range<MODE_REDUCE_KEPT, 0>(a, nullptr, 0, st);
}

}  // namespace vg

// Samples per thread that the FP32 drop-in kernels were once compiled for:
// the kernels have one shape now, so valid values are accepted and do nothing.
extern "C" int vg_set_dropin_tuning(int s_points, int s_reduce)
{
    if (s_points != 0 && s_points != 2 && s_points != 4 && s_points != 8)
        return vg_fail(VG_ERR_VALUE, "s_points %d", s_points);
    if (s_reduce != 0 && s_reduce != 2 && s_reduce != 4) return vg_fail(VG_ERR_VALUE, "s_reduce %d", s_reduce);
    return VG_OK;
}

#include "vg_fused.cuh"

namespace vg {
int launch_fused(IterArgs &a, int kind, const VgParams &P, int tab_len, int f64, cudaStream_t st)
{
    switch (kind) {
    case VG_F_GAUSS: return launch_fused_gauss(a, P, tab_len, f64, st);
    case VG_F_RIDGE: return launch_fused_ridge(a, P, tab_len, f64, st);
    case VG_F_LORENTZ: return launch_fused_lorentz(a, P, tab_len, f64, st);
    case VG_F_MIXTURE: return launch_fused_mixture(a, P, tab_len, f64, st);
    case VG_F_LATTICE: return launch_fused_lattice(a, P, tab_len, f64, st);
    default: return launch_fused_const(a, P, tab_len, f64, st);
    }
}
}  // namespace vg
