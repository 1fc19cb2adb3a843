"""chi^2 and its gradient at the edges of the register kernel: one and the most
levels it holds, one more (the shared-memory kernel), fewer points than threads,
a partial last pass, and frequencies whose squares leave the range of the
Newton reciprocal."""
import numpy as np
import pytest

import dmfted
import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nbath,L,scale", [
    (1, 1, 1.0), (1, 129, 1.0), (4, 100, 1.0), (8, 257, 1.0), (9, 1000, 1.0), (13, 128, 1.0),
    (16, 300, 1.0), (17, 300, 1.0), (5, 200, 1e16), (5, 200, 1e-16),
])
def test_chi2_and_gradient_match_oracle(nbath, L, scale):
    rng = np.random.default_rng(nbath * 1000 + L)
    wm = scale * np.pi / 100.0 * (2.0 * np.arange(1, L + 1) - 1.0)
    e = scale * rng.uniform(-1.0, 1.0, nbath)
    v = scale * (0.5 + rng.uniform(-0.1, 0.1, nbath))
    g = (v ** 2 / (1j * wm[:, None] - e)).sum(axis=1)
    g = g + 1e-3 * scale * (rng.normal(size=L) + 1j * rng.normal(size=L))
    w = 1.0 / wm
    a = np.concatenate([e, v]) * (1.0 + 0.05 * rng.normal(size=(3, 2 * nbath)))
    s = dmfted.EDSolver(dmfted.default_params(norb=1, nbath=3, lmats=16, lreal=0))
    chi2, grad = s.chi2_delta_batch(a, wm, g, w)
    assert np.array_equal(chi2, s.chi2_delta_batch(a, wm, g, w, grad=False))
    for i in range(3):
        c, d = O.chi2_delta(a[i], wm, g, w)
        # 64-bit sums of L terms, each to a few ulp
        assert abs(chi2[i] - c) <= 1e-12 * abs(c)
        assert np.abs(grad[i] - d).max() <= 1e-12 * np.abs(d).max()
    s.close()


def test_fit_batch_takes_an_odd_number_of_points():
    rng = np.random.default_rng(2)
    L, nbath = 201, 4
    wm = np.pi / 100.0 * (2.0 * np.arange(1, L + 1) - 1.0)
    e, v = rng.uniform(-1.0, 1.0, nbath), 0.5 + rng.uniform(-0.1, 0.1, nbath)
    g = (v ** 2 / (1j * wm[:, None] - e)).sum(axis=1)
    w = 1.0 / wm
    a = np.concatenate([e, v]) * (1.0 + 0.01 * rng.normal(size=(3, 2 * nbath)))
    s = dmfted.EDSolver(dmfted.default_params(norb=1, nbath=nbath, lmats=16, lreal=0))
    am, c2, _ = s.cg_fit_batch(a, wm, g, w, scheme=dmfted.CG_DELTA)
    start = s.chi2_delta_batch(a, wm, g, w, grad=False)
    for i in range(3):
        # the minimiser's chi^2 is that of its parameters, and below the start's
        assert abs(c2[i] - O.chi2_delta(am[i], wm, g, w)[0]) <= 1e-12 * start[i]
        assert c2[i] < 0.1 * start[i]
    s.close()
