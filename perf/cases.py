"""Performance cases of vegas_gb300: what users of the framework have it do.

Four ways in: ``Integrator`` on a built-in integrand (evaluated inside the
iteration kernels), ``Integrator`` on a torch batch integrand, ``BatchIntegrator``
(many integrals in one launch), and the learned proposal (``Flow``,
``FlowIntegrator``).  The integrands and sizes are those of ``bench.py`` and the
tests, over the range from a 10^4-evaluation integral to 10^7 evaluations an
iteration.

The runs are such that the same seed gives the same numbers.  Where the
allocation of evaluations follows FP32 variances through many iterations it does
not: sums in another order move an evaluation from one hypercube to another, and
every later sample of the iteration with it.  So FP32 runs of many iterations
have beta = 0, or a map and strata that no longer adapt, or start anew.

``exact`` follows the same random numbers through the same algorithm in 64 bits
with plain torch (below, ``_vegas64`` and ``_flow64``).
"""
import math

import numpy as np
import torch

import vegas_gb300 as vg
from vegas_gb300.batch import BatchIntegrator
from vegas_gb300.flow import Flow
from vegas_gb300.flow_vegas import FlowIntegrator


def listed():
    return [
        # the tutorial-sized integral, FP64 throughout, 10 adapting iterations in one call: launch latency
        dict(name='gauss4_f64_1e4', path='integrate', integrand='gauss', dim=4, neval=10000, nitn=10,
             precision='fp64', mode='vegas+'),
        # a middling integral without adaptive stratification (beta = 0): sampling, training histogram, adapt
        dict(name='lorentz6_classic', path='integrate', integrand='lorentz', dim=6, neval=200003, nitn=10,
             precision='fp32', mode='classic'),
        # the benchmark's integrand and size, the dim-4 ridge of 1000 Gaussians at 1e6 evaluations: production
        # iterations on a saved map and saved strata, nothing adapting any more
        dict(name='ridge4_frozen', path='integrate', integrand='ridge', dim=4, neval=1000000, nitn=10,
             precision='fp32', mode='frozen'),
        # the same of the 8-d mixture of Gaussians
        dict(name='mixture8_frozen', path='integrate', integrand='mixture', dim=8, neval=1 << 20, nitn=10,
             precision='fp32', mode='frozen'),
        # a user's own torch integrand, 1e7 evaluations an iteration, from a new Integrator
        dict(name='torch4_1e7', path='torch', integrand='gauss', dim=4, neval=10000000, nitn=2, values=1),
        # an array-valued torch integrand (a density and its moments) with its covariances
        dict(name='torch3_moments', path='torch', integrand='gauss', dim=3, neval=300007, nitn=2, values=4),
        # many independent integrals of mixed dimension and size in one launch, as that launch's integrals adapt
        # from iteration to iteration
        dict(name='batch_lorentz', path='batch', integrand='lorentz', njobs=1024, dmin=3, dmax=9,
             nmin=10000, nmax=250000, nitn=4),
        # a parameter scan of the lattice path integral: few large integrals, groups of CTAs on each
        dict(name='batch_lattice', path='batch', integrand='lattice', njobs=16, dmin=16, dmax=16,
             nmin=1000000, nmax=1000000, nitn=2),
        # the flow as a sampler: one iteration's points
        dict(name='flow_sample8', path='flow_sample', dim=8, K=32, rows=1 << 20),
        # the flow's density at given points, at the largest dimension, a ragged number of rows
        dict(name='flow_density16', path='flow_density', dim=16, K=32, rows=100003),
        # loss and gradient of one training batch (forward and backward)
        dict(name='flow_grad8', path='flow_grad', dim=8, K=32, rows=1 << 15),
        # flow-augmented vegas: iterations with a trained, frozen flow
        dict(name='flow_integrate8', path='flow_integrate', integrand='mixture', dim=8, neval=1 << 18, nitn=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(['f64', 'classic', 'frozen', 'ridge', 'torch', 'moments', 'batch', 'lattice', 'flow_sample',
                       'flow_density', 'flow_grad', 'flow_integrate'])
    peaks = ['gauss', 'lorentz']
    if path == 'f64':
        return dict(path='integrate', integrand=rng.choice(peaks), dim=rng.randint(2, 6),
                    neval=_log(rng, 5000, 100000), nitn=10, precision='fp64', mode='vegas+')
    if path == 'classic':
        return dict(path='integrate', integrand=rng.choice(peaks), dim=rng.randint(2, 6),
                    neval=_log(rng, 20000, 2000000), nitn=10, precision='fp32', mode=path)
    if path == 'frozen':
        return dict(path='integrate', integrand=rng.choice(peaks + ['mixture']), dim=rng.randint(2, 10),
                    neval=_log(rng, 10000, 2000000), nitn=10, precision='fp32', mode=path)
    if path == 'ridge':
        return dict(path='integrate', integrand='ridge', dim=rng.randint(3, 5), neval=_log(rng, 30000, 1500000),
                    nitn=10, precision='fp32', mode='frozen')
    if path in ('torch', 'moments'):
        return dict(path='torch', integrand=rng.choice(peaks + ['mixture']), dim=rng.randint(2, 8),
                    neval=_log(rng, 30000, 8000000 if path == 'torch' else 500000), nitn=2,
                    values=1 if path == 'torch' else rng.randint(2, 5))
    if path == 'batch':
        return dict(path='batch', integrand='lorentz', njobs=_log(rng, 256, 1000), dmin=3, dmax=9, nmin=10000,
                    nmax=_log(rng, 100000, 250000), nitn=rng.randint(2, 4))
    if path == 'lattice':
        n = _log(rng, 300000, 1000000)
        return dict(path='batch', integrand='lattice', njobs=rng.randint(8, 16), dmin=16, dmax=16, nmin=n, nmax=n,
                    nitn=2)
    if path in ('flow_sample', 'flow_density'):
        return dict(path=path, dim=rng.randint(2, 16), K=32, rows=_log(rng, 500, 500000))
    if path == 'flow_grad':
        return dict(path=path, dim=rng.randint(2, 16), K=32, rows=_log(rng, 1000, 32768))
    return dict(path=path, integrand='mixture', dim=rng.randint(3, 10), neval=_log(rng, 30000, 262144), nitn=2)


# ------------------------------------------------------------------- inputs
def _problem(case, seed):
    """The integrand's parameters and the integration box."""
    r = np.random.RandomState(seed % (1 << 31))
    dim, kind = case['dim'], case['integrand']
    if kind == 'gauss':
        return dict(kind=kind, a=100.0, c=float(r.uniform(0.4, 0.6)), lo=0.0, hi=1.0)
    if kind == 'lorentz':
        return dict(kind=kind, c=r.uniform(0.2, 0.8, dim), w=np.exp(r.uniform(np.log(0.03), np.log(0.1), dim)),
                    lo=0.0, hi=1.0)
    if kind == 'mixture':
        return dict(kind=kind, centers=r.uniform(0.15, 0.85, (4, dim)), sigma=0.05, lo=0.0, hi=1.0)
    return dict(kind='ridge', M=1000, s=0.01, lo=0.0, hi=1.0)


def _builtin(p, dim):
    if p['kind'] == 'gauss':
        return vg.Gaussian(a=p['a'], c=p['c'], dim=dim)
    if p['kind'] == 'lorentz':
        return vg.LorentzianProduct(p['c'], p['w'])
    if p['kind'] == 'mixture':
        return vg.GaussianMixture(p['centers'], sigma=p['sigma'])
    return vg.Ridge(M=p['M'], s=p['s'])


def _density(p, x):
    """The integrand in torch at x[n, dim], in x's type."""
    dim = x.shape[1]
    if p['kind'] == 'gauss':
        return (p['a'] / math.pi) ** (dim / 2.0) * torch.exp(-p['a'] * ((x - p['c']) ** 2).sum(dim=1))
    if p['kind'] == 'lorentz':
        c, w = (torch.as_tensor(p[k], dtype=x.dtype, device=x.device) for k in 'cw')
        return torch.prod((w / math.pi) / ((x - c) ** 2 + w ** 2), dim=1)
    if p['kind'] == 'ridge':
        c = (torch.arange(p['M'], dtype=x.dtype, device=x.device) + 0.5) / p['M']
        m = x.mean(dim=1, keepdim=True)
        f = torch.cat([torch.exp(-dim * (q - c) ** 2 / (2 * p['s'] ** 2)).sum(dim=1) for q in m.split(1 << 16)])
        return f * torch.exp(-((x - m) ** 2).sum(dim=1) / (2 * p['s'] ** 2)) \
            * (2 * math.pi * p['s'] ** 2) ** (-0.5 * dim) / p['M']
    f = torch.zeros_like(x[:, 0])
    for c in p['centers']:
        f += torch.exp(-((x - torch.as_tensor(c, dtype=x.dtype, device=x.device)) ** 2).sum(dim=1)
                       / (2 * p['sigma'] ** 2))
    return f * (2 * math.pi * p['sigma'] ** 2) ** (-0.5 * dim) / len(p['centers'])


def _values(p, x, s):
    """f, or [f, f x_0, f x_1, ...] with s components."""
    f = _density(p, x)
    if s == 1:
        return f
    return torch.stack([f] + [f * x[:, (k - 1) % x.shape[1]] ** (1 + (k - 1) // x.shape[1]) for k in range(1, s)],
                       dim=1)


def _saved_state(p, dim, nstrat, ninc, seed):
    """A map and strata weights as an adapted run leaves them: nodes dense where the integrand's marginals are,
    sigf following the integrand over the hypercubes."""
    r = np.random.RandomState((seed + 1) % (1 << 31))
    t = np.linspace(p['lo'], p['hi'], 4001)
    grid = []
    for d in range(dim):
        if p['kind'] == 'gauss':
            q = np.exp(-p['a'] * (t - p['c']) ** 2)
        elif p['kind'] == 'lorentz':
            q = 1.0 / ((t - p['c'][d]) ** 2 + p['w'][d] ** 2)
        elif p['kind'] == 'mixture':
            q = sum(np.exp(-(t - c[d]) ** 2 / (2 * p['sigma'] ** 2)) for c in p['centers'])
        else:
            q = np.ones_like(t)
        q = 0.2 + 0.8 * q / q.mean()
        cdf = np.concatenate([[0.0], np.cumsum(0.5 * (q[1:] + q[:-1]))])
        g = np.interp(np.linspace(0.0, 1.0, int(ninc[d]) + 1), cdf / cdf[-1], t)
        g[0], g[-1] = p['lo'], p['hi']
        grid.append(g)
    H = int(np.prod(nstrat))
    h = torch.arange(H, device='cuda')
    x = torch.empty((H, dim), dtype=torch.float64, device='cuda')
    jac = torch.ones(H, dtype=torch.float64, device='cuda')
    for d in range(dim):
        y = ((h % int(nstrat[d])).double() + 0.5) / int(nstrat[d]) * int(ninc[d])
        h = h // int(nstrat[d])
        i = y.long()
        g = torch.from_numpy(grid[d]).cuda()
        x[:, d] = g[i] + (g[i + 1] - g[i]) * (y - i)
        jac *= (g[i + 1] - g[i]) * int(ninc[d])
    w = _density(dict(p, s=0.03) if p['kind'] == 'ridge' else p, x) * jac   # a hypercube is wider than the ridge
    w = w.cpu().numpy()
    sigf = (w / w.mean() + 0.05) ** 0.75 * np.exp(0.4 * r.standard_normal(H))
    return grid, sigf / H


def _flow_theta(dim, nlayers, K, hidden, seed):
    """Parameters of a flow in mid-training: layer by layer W1, b1, W2, b2, W3, b3."""
    r = np.random.RandomState(seed % (1 << 31))
    out = []
    for A, B in _masks(dim, nlayers):
        dA, P = max(len(A), 1), len(B) * (2 * K + 1)
        out += [r.normal(0, math.sqrt(2.0 / dA), hidden * dA), r.normal(0, 0.1, hidden),
                r.normal(0, math.sqrt(2.0 / hidden), hidden * hidden), r.normal(0, 0.1, hidden),
                r.normal(0, 0.5 / math.sqrt(hidden), P * hidden), r.normal(0, 0.1, P)]
    return np.concatenate(out).astype(np.float32)


def _rows(case, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    z = torch.rand((case['rows'], case['dim']), generator=g, device='cuda', dtype=torch.float32)
    w = torch.exp(torch.randn(case['rows'], generator=g, device='cuda', dtype=torch.float32))
    return z, w / w.mean()


def _batch_problem(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    dims = r.randint(case['dmin'], case['dmax'] + 1, case['njobs'])
    nevals = np.exp(r.uniform(np.log(case['nmin']), np.log(case['nmax']), case['njobs'])).astype(np.int64)
    if case['integrand'] == 'lattice':
        lam = np.exp(r.uniform(math.log(0.01), 0.0, case['njobs']))
        return [vg.LatticeAction(a=0.5, lam=v) for v in lam], nevals, dims
    return [vg.LorentzianProduct(r.uniform(0.2, 0.8, d), np.exp(r.uniform(np.log(0.01), np.log(0.1), d)))
            for d in dims], nevals, dims


def prepare(case, seed):
    path = case['path']
    if path == 'integrate':
        dim, p = case['dim'], _problem(case, seed)
        f = _builtin(p, dim)
        box = dim * [[p['lo'], p['hi']]]
        args = dict(neval=case['neval'], precision=case['precision'], seed=seed)
        if case['mode'] == 'classic':
            integ = vg.Integrator(box, beta=0.0, **args)
        elif case['mode'] == 'frozen':
            integ = vg.Integrator(box, adapt=False, **args)
            grid, sigf = _saved_state(p, dim, integ.nstrat, integ.map.ninc, seed)
            integ.set(map=vg.AdaptiveMap(grid), sigf=sigf)
        else:
            integ = vg.Integrator(box, **args)
        return dict(path=path, integ=integ, f=f, nitn=case['nitn'],
                    dtype=np.float64 if case['precision'] == 'fp64' else np.float32)
    if path == 'torch':
        p = _problem(case, seed)
        if 'c' in p and not np.isscalar(p['c']):     # a user's integrand holds its constants on the GPU
            p = dict(p, **{k: torch.tensor(p[k], dtype=torch.float32, device='cuda') for k in 'cw'})
        if 'centers' in p:
            p = dict(p, centers=torch.tensor(p['centers'], dtype=torch.float32, device='cuda'))
        s = case['values']

        @vg.lbatchintegrand
        def f(x):
            return _values(p, x, s)

        return dict(path=path, f=f, box=case['dim'] * [[p['lo'], p['hi']]], neval=case['neval'], nitn=case['nitn'],
                    seed=seed, values=s)
    if path == 'batch':
        fs, nevals, dims = _batch_problem(case, seed)
        lim = (-5.0, 5.0) if case['integrand'] == 'lattice' else (0.0, 1.0)
        b = BatchIntegrator(fs, nevals, nitn=case['nitn'], nwarm=0, beta=0.0, seed=seed, variant=(1, 1, 0), dims=dims,
                            limits=lim)
        for _ in range(max(1, 8 // case['nitn'])):
            b.run()                  # warm-up iterations, as before any result that is kept
        return dict(path=path, batch=b)
    if path == 'flow_integrate':
        p = _problem(case, seed)
        fi = FlowIntegrator(case['dim'] * [[p['lo'], p['hi']]], neval=case['neval'], beta=0.0, seed=seed, plain_itn=1,
                            grace=10 ** 9)
        fi.flow.set_theta(_flow_theta(case['dim'], 6, 32, 128, seed))
        f = _builtin(p, case['dim'])
        fi(f, nitn=2, train=False)   # the plain iteration, and the first with the flow
        return dict(path=path, integ=fi, f=f, nitn=case['nitn'])
    flow = Flow(case['dim'], K=case['K'])
    flow.set_theta(_flow_theta(case['dim'], flow.nlayers, case['K'], flow.hidden, seed))
    z, w = _rows(case, seed)
    return dict(path=path, flow=flow, z=z, w=w)


# ---------------------------------------------------------------------- run
def _itns(r, dtype):
    return {'mean': np.array([g.mean for g in r.itn_results], dtype),
            'sdev': np.array([g.sdev for g in r.itn_results], dtype),
            'average': np.array([r.mean, r.sdev], dtype)}


def run(s):
    path = s['path']
    if path == 'integrate':
        integ = s['integ']
        r = integ(s['f'], nitn=s['nitn'])
        return dict(_itns(r, s['dtype']), grid=integ.map.grid_tensor)
    if path == 'torch':
        integ = vg.Integrator(s['box'], neval=s['neval'], seed=s['seed'])
        r = integ(s['f'], nitn=s['nitn'])
        itns = [np.atleast_1d(np.asarray(g, dtype=object)) for g in r.itn_results]
        return {'mean': [np.array([v.mean for v in g], np.float32) for g in itns],
                'sdev': [np.array([v.sdev for v in g], np.float32) for g in itns],
                'grid': integ.map.grid_tensor}
    if path == 'batch':
        res = s['batch'].run()
        return {'mean': res[:, 0].astype(np.float32), 'sdev': res[:, 1].astype(np.float32)}
    if path == 'flow_integrate':
        return _itns(s['integ'](s['f'], nitn=s['nitn'], train=False), np.float32)
    flow = s['flow']
    if path == 'flow_sample':
        z, ld = flow.sample(s['z'])
        return {'z': z, 'logdet': ld}
    if path == 'flow_density':
        z, ld = flow.density(s['z'])
        return {'zhat': z, 'logdet': ld}
    flow.grad.zero_()
    flow.loss.zero_()
    flow.accumulate_grad(s['z'], s['w'])
    return {'grad': flow.grad, 'loss': flow.loss.float()}


# --------------------------------------------------------------------- work
def _eval_flops(kind, dim):
    """Operations of one evaluation: drawing and mapping the point, the integrand, the sums."""
    draw_map = 25 * dim + 9 * dim
    f = {'gauss': 3 * dim + 3, 'lorentz': 6 * dim, 'mixture': 4 * (3 * dim + 3), 'ridge': 3 * dim + 4 * 100,
         'lattice': 8 * dim + 2}[kind]
    return draw_map + f + 46


def work(case):
    path = case['path']
    if path in ('integrate', 'torch', 'flow_integrate'):
        n, dim = case['neval'] * case['nitn'], case['dim']
        flops = n * _eval_flops(case['integrand'], dim)
        # strata weights read and written, two evaluations a hypercube at the least
        nbytes = case['nitn'] * 16.0 * (0.125 * case['neval'] if path == 'integrate' else 1) + 16.0 * 1000 * dim
        if path == 'torch':
            nbytes += n * 4.0 * (2 * dim + 2 * case['values'])     # points and values out and in again
        if path == 'flow_integrate':
            flops += n * _flow_flops(dim, 32)
            nbytes += n * 4.0 * 2
        return {'bytes': nbytes, 'flops': float(flops)}
    if path == 'batch':
        dim = 0.5 * (case['dmin'] + case['dmax'])
        lo, hi = case['nmin'], case['nmax']
        n = case['njobs'] * case['nitn'] * (lo if lo == hi else (hi - lo) / math.log(hi / lo))
        return {'bytes': 16.0 * 0.125 * n, 'flops': n * _eval_flops(case['integrand'], dim)}
    rows, dim, K = case['rows'], case['dim'], case['K']
    flops, nbytes = rows * _flow_flops(dim, K), rows * 4.0 * (2 * dim + 1)
    if path == 'flow_grad':
        flops, nbytes = 3 * flops, rows * 4.0 * (dim + 1) + 8.0 * 6 * (128 * 128 + 128 * dim * (2 * K + 1) / 2)
    return {'bytes': nbytes, 'flops': float(flops)}


def _flow_flops(dim, K, nlayers=6, hidden=128):
    return sum(2 * hidden * (len(A) + hidden + len(B) * (2 * K + 1)) + len(B) * 12 * K for A, B in _masks(dim, nlayers))


# -------------------------------------------------------------------- exact
def _mul32(a, b):
    """High and low 32 bits of a * b, a a constant and b an int64 tensor, both below 2^32."""
    lo, hi = (a & 0xffff) * b, (a >> 16) * b
    t = hi + (lo >> 16)
    return t >> 16, ((t & 0xffff) << 16) | (lo & 0xffff)


def _philox(i, c2, c3, seed):
    """Philox4x32-10 (Salmon et al., SC'11) of the counters (i, c2, c3) with the key `seed`."""
    c = [i & 0xffffffff, i >> 32, torch.full_like(i, c2), torch.full_like(i, c3)]
    k0, k1 = seed & 0xffffffff, (seed >> 32) & 0xffffffff
    for _ in range(10):
        h0, l0 = _mul32(0xD2511F53, c[0])
        h1, l1 = _mul32(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k0, l1, h0 ^ c[3] ^ k1, l0]
        k0, k1 = (k0 + 0x9E3779B9) & 0xffffffff, (k1 + 0xBB67AE85) & 0xffffffff
    return c


def _uniforms(n, dim, seed, itn, wide):
    """u[n, dim]: 53 bits of two words an axis, or 24 bits of one."""
    i = torch.arange(n, device='cuda')
    u = torch.empty((n, dim), dtype=torch.float64, device='cuda')
    for g in range(-(-dim // (2 if wide else 4))):
        w = _philox(i, itn, (0x80 if wide else 0) | g, seed)
        if wide:
            v = [((w[0] << 21) | (w[1] >> 11)) * 2.0 ** -53, ((w[2] << 21) | (w[3] >> 11)) * 2.0 ** -53]
        else:
            v = [(x >> 8) * 2.0 ** -24 for x in w]
        for k, x in enumerate(v):
            if g * len(v) + k < dim:
                u[:, g * len(v) + k] = x
    return u


def _sizes(dim, neval, beta, maxinc=1000, neval_frac=0.75):
    """Strata and increments of the axes, and the least evaluations of a hypercube (vegas _vegas.pyx:1346-1407)."""
    nf = neval_frac if beta > 0 else 0.0
    base = (1 - nf) * neval / 2.0
    ns = max(1, int(math.exp(math.log(base) / dim)))
    d = max(0, int((math.log(base) - dim * math.log(ns)) / math.log(1 + 1.0 / ns)))
    nstrat = [ns + 1 if k < d else ns for k in range(dim)]
    ni = min(maxinc, int(neval / 10.0))
    ninc = []
    for k in range(dim):
        if ni >= nstrat[k]:
            ninc.append(ni // nstrat[k] * nstrat[k])
        elif nstrat[k] <= maxinc:
            ninc.append(nstrat[k])
        else:
            nstrat[k] = nstrat[k] // ni * ni
            ninc.append(ni)
    H = int(np.prod(nstrat))
    return nstrat, ninc, max(2, int((1 - nf) * neval / H)) if H > 1 else neval


def _vegas64(p, dim, neval, nitn, seed, wide, beta=0.75, alpha=0.5, adapt=True, saved=None, values=1):
    """nitn iterations of vegas+ in 64 bits: per iteration the means and (co)variances, and the last grid."""
    nstrat, ninc, least = _sizes(dim, neval, beta)
    H, K = int(np.prod(nstrat)), max(ninc)
    grid = [torch.linspace(p['lo'], p['hi'], k + 1, dtype=torch.float64, device='cuda') for k in ninc]
    sigf = torch.ones(H, dtype=torch.float64, device='cuda')
    if saved is not None:
        grid = [torch.from_numpy(g).cuda() for g in saved[0]]
        sigf = torch.from_numpy(saved[1]).cuda()
    out = []
    for itn in range(1, nitn + 1):
        if beta > 0 and H > 1:
            n_h = (sigf * (0.75 * neval / sigf.sum())).long() + least
            n_h = torch.clamp(n_h, max=max(50000, least))
        else:
            n_h = torch.full((H,), neval // H, dtype=torch.int64, device='cuda')
        n = int(n_h.sum())
        h = torch.repeat_interleave(torch.arange(H, device='cuda'), n_h)
        u = _uniforms(n, dim, seed, itn, wide)
        x = torch.empty_like(u)
        jac = torch.ones(n, dtype=torch.float64, device='cuda')
        bins, q = [], h.clone()
        for d in range(dim):
            y = ((q % nstrat[d]).double() + u[:, d]) / nstrat[d] * ninc[d]
            q = q // nstrat[d]
            i = torch.clamp(y.long(), max=ninc[d] - 1)
            inc = grid[d][1:] - grid[d][:-1]
            x[:, d] = grid[d][i] + inc[i] * (y - i)
            jac *= inc[i] * ninc[d]
            bins.append(i)
        del u, q
        f = _values(p, x, values).reshape(n, values)
        wf = f * (jac / H / n_h[h])[:, None]

        def per_cube(v):
            return torch.zeros((H, v.shape[1]), dtype=torch.float64, device='cuda').index_add_(0, h, v)

        S = per_cube(wf)
        mean = S.sum(0)
        dev = wf - (S / n_h[:, None])[h]
        first = (n_h * per_cube(dev[:, :1] ** 2)[:, 0] - per_cube(dev[:, :1])[:, 0] ** 2) / (n_h - 1)
        cov = torch.stack([torch.stack([((dev[:, a] * dev[:, b]) * (n_h / (n_h - 1.0))[h]).sum()
                                        for b in range(values)]) for a in range(values)])
        out.append((mean.cpu().numpy(), cov.cpu().numpy()))
        if not adapt:
            continue
        if beta > 0 and H > 1:
            sigf = first.abs() ** (beta / 2)
        t = (wf[:, 0] * n_h[h]) ** 2
        for d in range(dim):
            k = ninc[d]
            a = torch.zeros(k, dtype=torch.float64, device='cuda').index_add_(0, bins[d], t) \
                / torch.clamp(torch.bincount(bins[d], minlength=k).double(), min=1.0)
            if k == 1:
                continue
            b = a.clone()
            b[1:-1] = (6 * a[1:-1] + a[:-2] + a[2:]) / 8
            b[0], b[-1] = (7 * a[0] + a[1]) / 8, (7 * a[-1] + a[-2]) / 8
            b = b / b.sum() + 1e-257
            b = torch.where(b <= 0.99999999, ((b - 1) / torch.log(b)) ** alpha, b)
            c = torch.cumsum(b, 0)
            want = torch.arange(1, k, device='cuda') * (c[-1] / k)
            j = torch.clamp(torch.searchsorted(c, want), max=k - 1)
            g = grid[d]
            grid[d] = torch.cat([g[:1], g[j + 1] - (c[j] - want) / b[j] * (g[j + 1] - g[j]), g[-1:]])
    whole = torch.zeros((dim, K + 1), dtype=torch.float64, device='cuda')
    for d in range(dim):
        whole[d, :ninc[d] + 1] = grid[d]
    return out, whole


def _average(means, variances, weighted):
    if weighted:
        w = 1.0 / variances
        return np.array([(w * means).sum() / w.sum(), math.sqrt(1.0 / w.sum())])
    return np.array([means.mean(), math.sqrt(variances.sum()) / len(means)])


def _masks(dim, nlayers):
    """(conditioning, transformed) coordinates of each coupling layer, by the bits of their indexes."""
    bits = max(1, int(math.ceil(math.log2(dim)))) if dim > 1 else 1
    out = []
    for l in range(nlayers):
        B = [i for i in range(dim) if (i >> ((l // 2) % bits) & 1) == l % 2]
        A = [i for i in range(dim) if i not in B]
        out.append((A, B) if A and B else ([], list(range(dim))))
    return out


def _flow64(theta, z, dim, K, inverse, nlayers=6, hidden=128):
    """The coupling flow in 64 bits: z and the sum of the log densities of its splines (piecewise-quadratic
    coupling transforms, Mueller et al., "Neural Importance Sampling", ACM TOG 2019)."""
    layers, o = [], 0
    for A, B in _masks(dim, nlayers):
        dA, P = max(len(A), 1), len(B) * (2 * K + 1)
        L = []
        for shape in ((hidden, dA), (hidden,), (hidden, hidden), (hidden,), (P, hidden), (P,)):
            m = int(np.prod(shape))
            L.append(theta[o:o + m].reshape(shape))
            o += m
        layers.append((A, B, L))
    logdet = torch.zeros_like(z[:, 0])
    for A, B, (W1, b1, W2, b2, W3, b3) in (reversed(layers) if inverse else layers):
        a = z[:, A] if A else torch.zeros_like(z[:, :1])
        t = torch.relu(torch.relu(a @ W1.T + b1) @ W2.T + b2) @ W3.T + b3
        t = t.reshape(z.shape[0], len(B), 2 * K + 1)
        W = 1e-3 + (1 - K * 1e-3) * torch.softmax(t[..., :K], -1)
        V = torch.exp(t[..., K:])
        area = 0.5 * (V[..., :-1] + V[..., 1:]) * W
        V = V / area.sum(-1, keepdim=True)
        nought = torch.zeros_like(W[..., :1])
        E = torch.cat([nought, torch.cumsum(W, -1)], -1)
        C = torch.cat([nought, torch.cumsum(area / area.sum(-1, keepdim=True), -1)], -1)
        zb = z[:, B].unsqueeze(-1)
        i = torch.searchsorted((C if inverse else E)[..., 1:-1].contiguous().detach(), zb.detach().contiguous(),
                               right=True)
        w, e, v0, v1, c = (torch.gather(q, -1, i + k) for q, k in ((W, 0), (E, 0), (V, 0), (V, 1), (C, 0)))
        if inverse:
            r, m = (zb - c) / w, v1 - v0
            s = 2 * r / (v0 + torch.sqrt(torch.clamp(v0 * v0 + 2 * m * r, min=0.0)))
            new = e + s * w
        else:
            s, m = (zb - e) / w, v1 - v0
            new = c + w * (s * v0 + 0.5 * s * s * m)
        z = z.clone()
        z[:, B] = new.squeeze(-1)
        logdet = logdet + torch.log(v0 + s * m).squeeze(-1).sum(1)
    return z, logdet


def exact(case, seed):
    path = case['path']
    if path == 'integrate':
        dim, p, frozen = case['dim'], _problem(case, seed), case['mode'] == 'frozen'
        beta = 0.0 if case['mode'] == 'classic' else 0.75
        nstrat, ninc, _ = _sizes(dim, case['neval'], beta)
        out, grid = _vegas64(p, dim, case['neval'], case['nitn'], seed, case['precision'] == 'fp64', beta=beta,
                             adapt=not frozen, saved=_saved_state(p, dim, nstrat, ninc, seed) if frozen else None)
        m, v = np.array([o[0][0] for o in out]), np.array([o[1][0, 0] for o in out])
        return {'mean': m, 'sdev': np.sqrt(v), 'average': _average(m, v, not frozen), 'grid': grid}
    if path == 'torch':
        # the second iteration's allocation follows FP32 variances: the first has a value
        out, _ = _vegas64(_problem(case, seed), case['dim'], case['neval'], 1, seed, False, values=case['values'])
        return {'mean': [out[0][0], None], 'sdev': [np.sqrt(np.diag(out[0][1])), None], 'grid': None}
    if path in ('batch', 'flow_integrate'):
        return None
    theta = torch.from_numpy(_flow_theta(case['dim'], 6, case['K'], 128, seed)).cuda().double()
    z, w = _rows(case, seed)
    if path == 'flow_grad':
        theta.requires_grad_(True)
        _, ld = _flow64(theta, z.double(), case['dim'], case['K'], False)
        loss = -(w.double() * ld).sum()
        loss.backward()
        return {'grad': theta.grad, 'loss': loss.detach().reshape(1)}
    parts = [_flow64(theta, q.double(), case['dim'], case['K'], path == 'flow_sample') for q in z.split(1 << 17)]
    return {'z' if path == 'flow_sample' else 'zhat': torch.cat([a for a, _ in parts]),
            'logdet': torch.cat([b for _, b in parts])}
