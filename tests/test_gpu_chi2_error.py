"""The register kernel of chi^2 and its gradient is no further from extended
precision than the shared-memory kernel: the same sets through both (levels of
zero coupling, which add nothing, take them past the register kernel's range)."""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

import dmfted

pytestmark = pytest.mark.gpu

SETS, LEVELS = 1024, range(1, 17)
X = np.longdouble


def exact(a, wm, g, w):
    nb = a.shape[1] // 2
    e, v = a[:, :nb, None].astype(X), a[:, nb:, None].astype(X)
    inv = 1 / (e * e + wm.astype(X) ** 2)
    re, im = -e * inv, -wm.astype(X) * inv
    rr = g.real.astype(X) - (v * v * re).sum(axis=1)
    ri = g.imag.astype(X) - (v * v * im).sum(axis=1)
    chi2 = ((rr * rr + ri * ri) / w.astype(X)).sum(axis=1)
    rr, ri = (rr / w.astype(X))[:, None], (ri / w.astype(X))[:, None]
    de = -2 * v[:, :, 0] ** 2 * (rr * (re * re - im * im) + 2 * ri * re * im).sum(axis=2)
    dv = -4 * v[:, :, 0] * (rr * re + ri * im).sum(axis=2)
    return chi2, np.concatenate([de, dv], axis=1)


def inputs(nb, points):
    rng = np.random.default_rng(nb * 10000 + points)
    wm = np.pi / 100.0 * (2.0 * np.arange(1, points + 1) - 1.0)
    e, v = rng.uniform(-1.0, 1.0, nb), 0.5 + rng.uniform(-0.1, 0.1, nb)
    g = (v ** 2 / (1j * wm[:, None] - e)).sum(axis=1)
    g = g + 1e-4 * (rng.normal(size=points) + 1j * rng.normal(size=points))
    a = np.concatenate([e, v]) + 0.05 * rng.normal(size=(SETS, 2 * nb))
    return a, wm, g, 1.0 / wm


def test_errors_no_larger_than_the_shared_memory_kernels():
    cases = [(nb, points) for nb in LEVELS for points in (200, 700, 1500)]

    def reference(case):  # in parts that stay small
        a, *rest = inputs(*case)
        parts = [exact(p, *rest) for p in np.split(a, 16)]
        return [np.concatenate(q) for q in zip(*parts)]

    with ThreadPoolExecutor(8) as pool:
        refs = list(pool.map(reference, cases))
    errors = []
    with dmfted.EDSolver(dmfted.default_params(norb=1, nbath=3, lmats=16, lreal=0)) as s:
        for case, ref in zip(cases, refs):
            nb = case[0]
            a, *rest = inputs(*case)
            pad = np.zeros((SETS, 17 - nb))
            wide = np.concatenate([a[:, :nb], pad + 0.5, a[:, nb:], pad], axis=1)
            keep = list(range(nb)) + list(range(17, 17 + nb))
            c, g = s.chi2_delta_batch(a, *rest)
            cw, gw = s.chi2_delta_batch(wide, *rest)
            errors.append([np.sqrt(float(((o - r) ** 2).sum() / (r ** 2).sum()))
                           for o, r in ((c, ref[0]), (cw, ref[0]), (g, ref[1]),
                                        (gw[:, keep], ref[1]))])
    c, cw, g, gw = np.mean(errors, axis=0)
    # unit roundoffs of the norm; the two kernels take as many roundings per term
    assert c <= cw and g <= gw, (c, cw, g, gw)
