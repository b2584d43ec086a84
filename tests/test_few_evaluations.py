"""Hypercubes of fewer than two evaluations (callers of the C interface set
min_neval_hcube, or neval of the order of nhcube): points, weights and sums against the
counts that the allocation made.

A hypercube of one has no variance, so the record's is not looked at where a count is 1
(nor the FP64 mode's sigf, which are all 1 when their sum is NaN); hypercubes without
evaluations add nothing and keep their sigf.  Tolerances as in
test_iteration_kernels.py.
"""
import ctypes

import numpy as np
import pytest
import torch

import vegas_gb300 as vg
from vegas_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _counts(kind, H, rng):
    if kind == 'some ones':
        return rng.integers(1, 5, H)
    if kind == 'run of ones':        # longer than a tile of 128 samples, shorter than one of 512
        n = rng.integers(2, 5, H)
        n[300:500] = 1
        return n
    if kind == 'ones':
        return np.ones(H, np.int64)
    if kind == 'some none':
        return rng.choice([0, 2, 3, 7], H)
    if kind == 'long gaps':          # more without evaluations on end than a chunk sees
        n = rng.integers(2, 6, H)
        for k in range(5, H, 400):
            n[k:k + 150] = 0
        n[:70] = 0
        n[-90:] = 0
        return n
    n = np.where(rng.random(H) < 0.9, 0, rng.integers(2, 4, H))
    n[H // 2] = 3000                 # and one over many chunks
    return n


@pytest.mark.parametrize('precision', ['fp32', 'fp64'])
@pytest.mark.parametrize('kind', ['some ones', 'run of ones', 'some none', 'ones', 'long gaps', 'one large'])
@pytest.mark.parametrize('nstrat', [[40, 50], [7, 5, 6, 4, 5]])
def test_counts_below_two(nstrat, kind, precision):
    if precision == 'fp64' and kind not in ('some ones', 'run of ones'):
        pytest.skip('the FP64 tiles take no more hypercubes than samples')
    L = N.load()
    H = int(np.prod(nstrat))
    want = _counts(kind, H, np.random.default_rng(H))
    I = vg.Integrator(len(nstrat) * [[0, 1]], neval=8 * H, nstrat=nstrat, seed=3, precision=precision, alpha=0.0,
                      max_neval_hcube=5000)
    I.min_neval_hcube = 0
    I._sigf.copy_(torch.from_numpy(want + 0.5).to(I.device))
    I.sum_sigf = I.neval_frac * I.neval       # counts = int(sigf)
    it, ncap = I._struct()
    I._allocate(it)
    n = int(I._read_stats().neval)
    nh = I._neval_h_host()
    assert np.array_equal(nh, want) and n == want.sum()
    for kept in (False, True):
        keep = I._keep_buffer(it, ncap) if kept else None
        x, _, w, hc = I._points(it, ncap, 3, None, want_hc=True, keep=keep)
        h = np.repeat(np.arange(H), want)
        assert I._read_stats().status == 0
        assert np.array_equal(hc[:n].cpu().numpy(), h)
        np.testing.assert_allclose(w[:n].cpu().numpy(), 1.0 / H / want[h], rtol=1e-6)
        xs = x[:n].double().cpu().numpy()
        q = h.copy()
        for d, k in enumerate(nstrat):        # inside its hypercube
            assert np.abs(xs[:, d] * k - q % k - 0.5).max() <= 0.5 + 1e-5
            q //= k
        f = torch.zeros(ncap, dtype=x.dtype, device=x.device)
        f[:n] = torch.exp(-3.0 * ((x[:n] - 0.4) ** 2).sum(dim=1)) + 0.1 * x[:n, 0]
        fdt = N.VG_F64 if precision == 'fp64' else N.VG_F32
        s0 = I._sigf.clone()
        args = (N.ptr(f), fdt) + ((N.ptr(keep), keep.numel()) if kept else ()) + (N.stream_ptr(I.device),)
        N.check((L.vg_reduce_kept if kept else L.vg_reduce)(ctypes.byref(it), 3, None, *args))
        st = I._read_stats()
        sigf = I.sigf.copy()
        I._sigf.copy_(s0)
        assert st.status == 0
        wf = (w[:n].to(x.dtype) * f[:n]).double().cpu().numpy()
        S = np.bincount(h, wf, H)
        assert abs(st.mean - S.sum()) <= 2e-8 * abs(S.sum())
        two = want >= 2
        dev = wf - (S / np.maximum(want, 1))[h]
        var = np.bincount(h, dev ** 2, H)[two] * (want / np.maximum(want - 1.0, 1.0))[two]
        if not (want == 1).any():
            assert abs(st.var - var.sum()) <= 1e-5 * var.sum()
        if precision == 'fp64':
            continue
        np.testing.assert_allclose(sigf[two], var ** (I.beta / 2), rtol=2e-5)
        np.testing.assert_array_equal(sigf[want == 0], (want + 0.5)[want == 0])
