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


def _divide(a, b):
    """a / b as float-float: quotient by the correctly rounded reciprocal, corrected once."""
    r = np.float32(1) / np.float32(b)
    q1 = np.float32(np.float32(a) * r)
    q2 = np.float32(np.float32(float(a) - float(q1) * b) * r)
    return float(q1) + float(q2)


def test_variance_divides_by_the_rounded_reciprocal():
    """One hypercube of n small whole numbers, 0 the first and the sum of each chunk of 128:
    n Q is a whole number below 2^24 and exact on every way to the variance n Q / (n - 1),
    whose bits are then those of the division.  (A reciprocal to an ulp is another float
    for one whole number in eight, and its quotient's error up to twice as large.)"""
    rng = np.random.default_rng(2)
    for n in range(129, 801):
        I = vg.Integrator([[0, 1]], neval=n, nstrat=[1], maxinc_axis=2, seed=n, beta=0.0, alpha=0.0)
        want = np.zeros(n, np.float32)

        def values(x, w, nh):
            w0 = np.float32(w[0].item())
            q = np.arange(1, 6).astype(np.float32)   # those that are products of floats and the weight
            f = np.stack([q / w0, np.nextafter(q / w0, np.float32(100)), np.nextafter(q / w0, np.float32(0))])
            hit = (f * w0 == q).any(axis=0)
            f = f[(f * w0 == q).argmax(axis=0), np.arange(len(q))]
            out = np.zeros(n, np.float32)
            for b in range(0, n, 128):
                m = (min(n, b + 128) - b - 1) // 2   # pairs after the first
                pick = rng.choice(np.flatnonzero(hit), m)
                want[b + 1:b + 1 + m], out[b + 1:b + 1 + m] = q[pick], f[pick]
                want[b + 1 + m:b + 1 + 2 * m], out[b + 1 + m:b + 1 + 2 * m] = -q[pick], -f[pick]
            return torch.from_numpy(out).to(x.device)

        st, _, nh, wf = _reduce(I, values, False)
        assert list(nh) == [n] and np.array_equal(wf, want)
        num = n * int((want.astype(np.int64) ** 2).sum())
        assert st.status == 0 and 0 < num < 2 ** 24
        assert st.var == _divide(num, n - 1), n
