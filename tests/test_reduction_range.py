"""Reductions of FP32 iterations whose squares come near or leave the float range.

A few samples X times larger than the others, each the first of its hypercube, of
its chunk of 128 or of its warp's range: the sums about a hypercube's first sample
are then as large as they get, (n - 1) X^2 for a piece of n samples where the
variance is near X^2.  Up to X = 5e18 (X^2 = 2.5e37) the variances are floats, so they
have to come out, in hypercubes within a chunk, over several chunks of one warp and
over the ranges of many warps.

Tolerances: float-float sums, 2^-44 an addition and n 2^-44 where the first sample
is the outlier, n <= 5000: 3e-10 of the variance; 1e-6 is allowed, 2e-8 of the mean
and 2e-5 of sigf (ex2 and lg2 by the special-function unit) as for other integrands.
"""
import ctypes

import numpy as np
import pytest
import torch

import oracle as O
import vegas_gb300 as vg
from vegas_gb300 import _native as N

pytestmark = pytest.mark.gpu


def _reduce(I, values, kept):
    """One iteration's record and sigf for f = values(x, weights, counts), and the oracle's."""
    L = N.load()
    it, ncap = I._struct()
    I._allocate(it)
    n = int(I._read_stats().neval)
    keep = I._keep_buffer(it, ncap) if kept else None
    x, _, w, _ = I._points(it, ncap, 3, None, keep=keep)
    nh = I._neval_h_host()
    f = torch.zeros(ncap, dtype=torch.float32, device=x.device)
    f[:n] = values(x[:n], w[:n].float(), nh)
    s0 = I._sigf.clone()
    stream = N.stream_ptr(I.device)
    if kept:
        N.check(L.vg_reduce_kept(ctypes.byref(it), 3, None, N.ptr(f), N.VG_F32, N.ptr(keep), keep.numel(), stream))
    else:
        N.check(L.vg_reduce(ctypes.byref(it), 3, None, N.ptr(f), N.VG_F32, stream))
    st = I._read_stats()
    sigf = I.sigf.copy()
    I._sigf.copy_(s0)
    wf = (w[:n].float() * f[:n]).cpu().numpy()
    return st, sigf, nh, wf


@pytest.mark.parametrize('kept', [False, True])
@pytest.mark.parametrize('X', [1e16, 3e17, 5e18])
@pytest.mark.parametrize('nstrat,neval,beta,every', [
    ([64], 1024, 0.75, None),       # whole hypercubes in a chunk
    ([1], 5000, 0.0, 128 * 8),      # one hypercube over the ranges of many warps
    ([2], 127, 0.0, None),
    ([7], 9000, 0.75, None),
    ([3, 5, 2, 4], 60000, 0.75, None),
    ([4000], 1400000, 0.75, None),  # over several chunks of one warp's range
    ([120], 1400000, 0.75, 128 * 999),
])
def test_outliers_near_the_float_range(nstrat, neval, beta, every, X, kept):
    I = vg.Integrator(len(nstrat) * [[0, 1]], neval=neval, nstrat=nstrat, seed=5, beta=beta, alpha=0.0)

    def values(x, w, nh):
        wf = w * (1.0 + x[:, 0])
        first = np.concatenate([[0], np.cumsum(nh)[:-1]])
        at = np.arange(0, x.shape[0], every) if every else first[::max(1, len(first) // 8)]
        wf[torch.from_numpy(at.astype(np.int64)).to(x.device)] = X
        return wf / w

    st, sigf, nh, wf = _reduce(I, values, kept)
    adaptive = I.beta > 0 and I.nhcube > 1
    mean, var, want, ss, _ = O.reduce(nh, wf, np.ones(len(wf)), beta=I.beta, adaptive=adaptive,
                                      sigf=np.ones(I.nhcube))
    assert st.status == 0 and var[0, 0] > X * X
    assert abs(st.mean - mean[0]) <= 2e-8 * abs(mean[0])
    assert abs(st.var - var[0, 0]) <= 1e-6 * var[0, 0]
    if adaptive:
        np.testing.assert_allclose(sigf, want, rtol=2e-5)
        assert abs(st.sum_sigf - ss) <= 2e-5 * ss
