"""Iteration kernels at the edges of their tiles and dispatch rules.

The reduction of one iteration (mean, variance, sigf; _vegas.pyx:2136-2193) and
the training histogram (pyx:421-464) of the FP32 and FP64 kernels against the
oracle's loops in FP64 on the kernel's own samples; the routes that one
iteration can take (grid table and histogram in shared memory or not, samples
regenerated or kept) against each other; array-valued reductions around the
hypercube size that changes lanes; the end of an iteration in one kernel against
the separate kernels; the flow's pass over many rows against its pass over few,
and its gradient in a captured graph against the same call outside.

Tolerances.  FP32: the kernel forms wgt*f in FP32, as the oracle is given it
here, and sums in float-float: 2^-44 per addition over at most 2^18 samples
leaves 2e-8 of the mean; the variance (n Q - D^2)/(n - 1) cancels to no less
than 1e-3 of n Q with these integrands, so 1e-5.  sigf goes through
ex2/lg2.approx: 2e-5 for its exponents below 2^6.  FP64: 1e-12 of the mean,
1e-9 of the variance after the same cancellation.  A bin of the FP32 histogram
adds at most 1600 terms in any order: 1600 * 2^-24 = 1e-4.
"""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
import vegas_gb300 as vg
from vegas_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _f(x):
    return torch.exp(-3.0 * ((x - 0.4) ** 2).sum(dim=1)) + 0.1 * x[:, 0]


def _integrator(nstrat, neval, precision, peak):
    I = vg.Integrator(len(nstrat) * [[0, 1]], neval=neval, nstrat=nstrat, precision=precision, seed=11,
                      beta=0.75 if peak else 0.0)
    if peak and I.nhcube > 1:   # nearly all evaluations in one hypercube, the others at the minimum
        s = np.full(I.nhcube, 1e-12)
        s[I.nhcube // 2] = 1.0
        I._sigf.copy_(torch.from_numpy(s).to(I.device))
        I.sum_sigf = float(s.sum())
    return I


def _iteration(I, kept=False):
    """One iteration's reduction: record, sigf, histogram, and what the oracle needs."""
    L = N.load()
    it, ncap = I._struct()
    I.map.sum_f.zero_()
    I.map.n_f.zero_()
    I._allocate(it)
    n = int(I._read_stats().neval)
    keep = I._keep_buffer(it, ncap) if kept else None
    x, _, w, _ = I._points(it, ncap, 3, None, keep=keep)
    f = torch.zeros(ncap, dtype=x.dtype, device=x.device)
    f[:n] = _f(x[:n])
    fdt = N.VG_F64 if x.dtype == torch.float64 else N.VG_F32
    s0 = I._sigf.clone()
    stream = N.stream_ptr(I.device)
    if kept:
        N.check(L.vg_reduce_kept(ctypes.byref(it), 3, None, N.ptr(f), fdt, N.ptr(keep), keep.numel(), stream))
    else:
        N.check(L.vg_reduce(ctypes.byref(it), 3, None, N.ptr(f), fdt, stream))
    st = I._read_stats()
    assert st.status == 0 and not st.nan_seen
    sigf = I.sigf.copy()
    I._sigf.copy_(s0)
    return dict(st=st, sigf=sigf, sum_f=I.map.sum_f.cpu().numpy(), n_f=I.map.n_f.cpu().numpy(), n=n,
                nh=I._neval_h_host(), wf=(w[:n].to(x.dtype) * f[:n]).cpu().numpy())


SHAPES = [
    ([63], 126, False), ([64], 128, False), ([65], 130, False),              # a chunk of 128 samples, 2 per hypercube
    ([511], 1022, False), ([512], 1024, False), ([513], 1026, False),        # a group of 8 warps' chunks
    ([1], 5000, False),                                                      # one hypercube
    ([2], 127, False), ([3, 5, 2, 4], 60000, True),                          # one hypercube in many warps' ranges
    ([40, 40], 40000, True), ([3] * 5, 30000, False), ([4] * 8, 131072, False), ([2] * 9, 5000, True),
    ([2] * 16, 131072, False), ([2, 3] + [1] * 15, 20000, False),            # above 16 dimensions
    ([5, 7, 3], 76500, False), ([5, 7, 3], 79500, False),                    # FP64: small tiles, large tiles
]


@pytest.mark.parametrize('precision', ['fp32', 'fp64'])
@pytest.mark.parametrize('nstrat,neval,peak', SHAPES)
def test_reduction_matches_oracle(nstrat, neval, peak, precision):
    I = _integrator(nstrat, neval, precision, peak)
    adaptive = I.beta > 0 and I.nhcube > 1
    s0 = I.sigf.copy()
    for kept in (False, True):
        r = _iteration(I, kept)
        assert int(r['nh'].sum()) == r['n']
        if peak and I.nhcube > 1:
            assert r['nh'].max() > 20 * np.median(r['nh'])
        mean, var, sigf, ss, _ = O.reduce(r['nh'], r['wf'], np.ones(r['n']), beta=I.beta, adaptive=adaptive, sigf=s0)
        t = (2e-8, 1e-5, 2e-5) if precision == 'fp32' else (1e-12, 1e-9, 1e-9)
        st = r['st']
        assert abs(st.mean - mean[0]) <= t[0] * abs(mean[0])
        assert abs(st.var - var[0, 0]) <= t[1] * var[0, 0]
        if adaptive:
            np.testing.assert_allclose(r['sigf'], sigf, rtol=t[2])
            assert abs(st.sum_sigf - ss) <= t[2] * ss
        # every sample trains one bin of each axis (but y = 0, at 2^-24 a sample)
        total = r['n_f'].sum(axis=1)
        assert np.all(total <= r['n']) and np.all(total >= r['n'] - 2)


@pytest.mark.parametrize('nstrat,neval,peak', SHAPES)
def test_routes_agree_fp32(nstrat, neval, peak):
    L = N.load()
    I = _integrator(nstrat, neval, 'fp32', peak)
    ref = _iteration(I)
    for table, hist in ((0, -1), (-1, 0), (0, 0)):
        N.check(L.vg_set_tile_tuning(0, table, hist))
        try:
            for kept in (False, True):
                r = _iteration(I, kept)
                assert abs(r['st'].mean - ref['st'].mean) <= 2e-8 * abs(ref['st'].mean)
                assert abs(r['st'].var - ref['st'].var) <= 1e-5 * ref['st'].var
                np.testing.assert_allclose(r['sigf'], ref['sigf'], rtol=2e-5)
                assert np.array_equal(r['n_f'], ref['n_f'])
                assert np.max(np.abs(r['sum_f'] - ref['sum_f'])) <= 1e-4 * np.max(ref['sum_f'])
        finally:
            N.check(L.vg_set_tile_tuning(0, -1, -1))


def _columns(x, s):
    g = torch.exp(-5.0 * ((x - 0.45) ** 2).sum(dim=1))
    return torch.stack([g * x[:, k % x.shape[1]] ** k for k in range(s)], dim=1)


@pytest.mark.parametrize('s,correlate', [(s, True) for s in range(1, 7)] + [(s, False) for s in (1, 2, 3, 4, 5, 6, 9)])
def test_array_reduction_around_the_lane_size(s, correlate):
    """Hypercubes of 5 to 38 samples in one iteration: one lane reduces up to 24, a
    warp the larger ones."""
    I = vg.Integrator(2 * [[0, 1]], neval=7000, nstrat=[19, 17], precision='fp64', seed=8,
                      correlate_integrals=correlate)
    H = I.nhcube
    sg = 1e-9 + (np.arange(H) % 39) / 39.0
    I._sigf.copy_(torch.from_numpy(sg).to(I.device))
    I.sum_sigf = float(sg.sum())
    it, ncap = I._struct()
    I._allocate(it)
    n = int(I._read_stats().neval)
    nh = I._neval_h_host()
    assert {23, 24, 25}.issubset(set(nh.tolist())) and nh.min() < 8 and nh.max() > 32
    x, _, w, _ = I._points(it, ncap, 1, None)
    f = torch.zeros((ncap, s), dtype=torch.float64, device=x.device)
    f[:n] = _columns(x[:n], s)
    mean, var = I._reduce_array(it, f, N.VG_F64, w)
    rm, rv, _, _, _ = O.reduce(nh, w[:n].cpu().numpy(), f[:n].cpu().numpy(), adaptive=False)
    np.testing.assert_allclose(mean, rm, rtol=1e-12)
    if correlate:
        np.testing.assert_allclose(var, rv, rtol=1e-9, atol=1e-12 * np.abs(rv).max())
    else:
        np.testing.assert_allclose(np.diag(var), np.diag(rv), rtol=1e-9)


@pytest.mark.parametrize('precision', ['fp32', 'fp64'])
@pytest.mark.parametrize('ninc', [2, 3, 127, 128, 129, 1022, 1023, 1024, 1500])
def test_iteration_in_one_call_matches_separate_kernels(ninc, precision):
    """vg_iterate_record (adapt beside the finalize, by clusters up to 1023
    increments) against allocate, fused iteration and end of iteration."""
    L = N.load()
    f = vg.Gaussian(a=20.0, c=0.45, dim=3)
    p = f.params(3)
    out = []
    for one_call in (True, False):
        I = vg.Integrator(3 * [[0, 1]], neval=30000, nstrat=[1, 2, 1], maxinc_axis=ninc, precision=precision, seed=4)
        I.map.adapt(ninc=ninc)
        it, ncap = I._struct()
        s = N.stream_ptr(I.device)
        if one_call:
            I._put_sum_sigf()
            host = I._records_host(1)
            N.check(L.vg_iterate_record(ctypes.byref(it), 1, int(f.kind), N.dbl_array(p), len(p), host.data_ptr(), s))
            torch.cuda.synchronize()
            rec = N.VgStats.from_buffer_copy(host[0].numpy())
            st = I._read_stats()
            for k in ('mean', 'var', 'neval', 'sum_sigf', 'status', 'range_lo', 'range_hi'):
                assert getattr(rec, k) == getattr(st, k)
        else:
            I._allocate(it)
            N.check(L.vg_fused_iteration(ctypes.byref(it), 1, None, int(f.kind), N.dbl_array(p), len(p), s))
            N.check(L.vg_end_iteration(ctypes.byref(it), s))
            st = I._read_stats()
        assert st.status == 0 and int(max(I.map.ninc)) == ninc
        assert not I.map.sum_f.any() and not I.map.n_f.any()   # cleared for the next iteration
        out.append((st.mean, st.var, st.sum_sigf, I.map.grid, I.map.inc))
    a, b = out
    # the same samples and sums; the histogram's order of addition is free
    t = 1e-4 if precision == 'fp32' else 1e-11
    for k in range(3):
        assert abs(a[k] - b[k]) <= 1e-12 * abs(b[k])
    np.testing.assert_allclose(a[3], b[3], rtol=0, atol=t)
    np.testing.assert_allclose(a[4], b[4], rtol=0, atol=t)


@pytest.mark.parametrize('K', [16, 32])
@pytest.mark.parametrize('dim', [2, 5, 8, 16])
def test_flow_pass_of_many_rows_matches_few(dim, K):
    """More than one 128-row tile per SM takes the pass with two groups of warps;
    the rows are independent, so the pass over few rows at a time gives the
    same but for BF16 roundings that may flip (z 2e-3, logdet 2e-2 as against the
    oracle; nearly all rows to 1e-5)."""
    from vegas_gb300.flow import Flow
    import flow_oracle as F
    fl = Flow(dim, K=K)
    fl.set_theta(F.init_theta(dim, 6, K, 128, seed=2, out_scale=0.5))
    tiles = torch.cuda.get_device_properties(0).multi_processor_count
    g = torch.Generator(device='cuda').manual_seed(dim)
    u = torch.rand((tiles * 128 + 129, dim), generator=g, device='cuda')
    for run in (fl.sample, fl.density):
        parts = [run(c.contiguous()) for c in u.split(5000)]
        zr, lr = torch.cat([p[0] for p in parts]), torch.cat([p[1] for p in parts])
        for n in (tiles * 128, tiles * 128 + 1, tiles * 128 + 127, tiles * 128 + 128, tiles * 128 + 129):
            z, ld = run(u[:n].contiguous())
            assert float((z - zr[:n]).abs().max()) <= 2e-3
            assert float((ld - lr[:n]).abs().max()) <= 2e-2
            assert float((ld - lr[:n]).abs().median()) <= 1e-5


@pytest.mark.parametrize('n', [130, 19457, 40001])
def test_flow_gradient_in_a_graph_matches_outside(n):
    """The weight gradients run on a forked stream, under capture on the caller's
    own: the same sums but for the order of the FP32 atomics."""
    from vegas_gb300.flow import Flow
    import flow_oracle as F
    fl = Flow(5, K=32)
    fl.set_theta(F.init_theta(5, 6, 32, 128, seed=3, out_scale=0.5))
    g = torch.Generator(device='cuda').manual_seed(n)
    z = torch.rand((n, 5), generator=g, device='cuda')
    w = torch.rand(n, generator=g, device='cuda')
    fl.grad.zero_()
    fl.accumulate_grad(z, w)
    torch.cuda.synchronize()
    want = fl.grad.clone()
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        with torch.cuda.graph(graph, stream=side):
            fl.accumulate_grad(z, w)
    fl.grad.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert float((fl.grad - want).norm()) <= 1e-5 * float(want.norm())
