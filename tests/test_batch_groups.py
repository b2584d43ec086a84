"""Groups of CTAs on one integral against one CTA on it, after adapting.

Iterations after the first read the grid table that the launch itself rebuilt, in
a group on other SMs than those that adapted the axes; a table or an axis left
behind gives samples and weights that agree with one another, so nothing shows in
pulls against the closed form.  Here the second iteration's record and the grids
are compared with those of the same integrals without groups.

Tolerances.  The first iteration has the same samples and float-float sums: 1e-6.
The groups' FP32 histograms add in another order, at most 1600 * 2^-24 = 1e-4 of a
bin and, roundings being random, about 40 * 2^-24 = 2e-6; the damping
((1 - f) / -ln f)^0.5 at bins of f <= 0.1 makes a fifth of that of a weight.  A node
stands where the weights' sum reaches its share of their total: at most 2e-5 of 1000
increments, 0.02 of one where its weight is the average, 0.1 of one where it is a
fifth of that.  The next iteration's samples shift by a fortieth of that, 0.0005 of
an increment of 1e-3 beside a width of 0.03 or more, and their weights by 4e-7: 2e-5 an
axis at the most, 3e-4 of a sample over 16 axes.  2e-3 of the mean and 4e-3 of the
variance are allowed.  An axis that was not adapted is off by many increments, a
stale table by a standard deviation.
"""
import numpy as np
import pytest

import vegas_gb300 as vg

pytestmark = pytest.mark.gpu


def _lorentz(dim, n, seed):
    rng = np.random.default_rng(seed)
    return [vg.LorentzianProduct(rng.uniform(0.2, 0.8, dim), np.exp(rng.uniform(np.log(0.03), np.log(0.1), dim)))
            for _ in range(n)]


@pytest.mark.parametrize('kind,dim,variant,group', [
    ('lorentz', 16, 0, 3),    # the table is read from global memory, and 3 does not divide the axes
    ('lattice', 12, 0, 2),
    ('lorentz', 8, 0, 3),     # two CTAs per SM leave no room for the table
    ('lorentz', 4, 2, 5),     # four CTAs per SM, more CTAs than axes
    ('lorentz', 7, 1, 2),     # four axes at a time in a CTA
])
def test_groups_agree_after_adapting(kind, dim, variant, group):
    from vegas_gb300.batch import BatchIntegrator
    lattice = kind == 'lattice'
    lo, hi = (-5.0, 5.0) if lattice else (0.0, 1.0)
    fs = [vg.LatticeAction(0.5, lam) for lam in (0.02, 0.1, 0.7)] if lattice else _lorentz(dim, 3, dim)

    def run(nitn, g):
        B = BatchIntegrator(fs, [100003, 150000, 120001], nitn=nitn, nwarm=0, beta=0.0, seed=31, variant=variant,
                            dims=[dim] * 3, limits=(lo, hi), group=g)
        B.run()
        assert B.group == g
        return B

    a, b = run(1, 1), run(1, group)
    for j in range(3):   # the grids after one iteration
        ga, gb = (x.state(j)['grid'].cpu().numpy() for x in (a, b))
        assert np.abs(ga - gb).max() <= 0.1 * (hi - lo) / a.ninc[j].min()
        for d, k in enumerate(a.ninc[j]):   # every axis was adapted
            assert np.abs(ga[d, :k + 1] - np.linspace(lo, hi, k + 1)).max() > (hi - lo) / 100
    oa, ob = run(2, 1).iterations(), run(2, group).iterations()
    assert np.array_equal(oa[:, :, 2], ob[:, :, 2])
    np.testing.assert_allclose(ob[:, 0, :2], oa[:, 0, :2], rtol=1e-6)
    np.testing.assert_allclose(ob[:, 1, 0], oa[:, 1, 0], rtol=2e-3)
    np.testing.assert_allclose(ob[:, 1, 1], oa[:, 1, 1], rtol=4e-3)


@pytest.mark.parametrize('dim,variant,group', [(16, 0, 3), (8, 0, 3), (4, 2, 5), (7, 1, 2)])
def test_groups_agree_when_adapting_to_errors(dim, variant, group):
    """adapt_to_errors (a field of the C record): the finalize adds the hypercubes cut by
    ranges to the training histogram that the group's other CTAs then adapt from.  The
    variances are float-float and the sums FP64; their averages are rounded to FP32,
    6e-8, so 6e-8 of 1000 increments is the most that a node moves where its weight is the
    average: a thousandth of an increment is allowed."""
    from vegas_gb300.batch import BatchIntegrator
    runs = []
    for g in (1, group):
        B = BatchIntegrator(_lorentz(dim, 3, dim), [100003, 150000, 120001], nitn=1, nwarm=0, beta=0.0, seed=31,
                            variant=variant, group=g)
        for it in B.its:
            it.adapt_to_errors = 1
        B.set_variant(variant)
        B.run()
        runs.append(B)
    a, b = runs
    np.testing.assert_allclose(b.iterations()[:, 0], a.iterations()[:, 0], rtol=1e-6)
    for j in range(3):
        ga, gb = (x.state(j)['grid'].cpu().numpy() for x in (a, b))
        assert np.abs(ga - gb).max() <= 1e-3 / a.ninc[j].min()
        for d, k in enumerate(a.ninc[j]):
            assert np.abs(ga[d, :k + 1] - np.linspace(0.0, 1.0, k + 1)).max() > 0.01
