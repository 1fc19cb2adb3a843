"""The one-row form of the lean H*v (odd row counts, vectors off the two-element
boundary) against the oracle, at the edges of its tiles: row counts below, at and
above the block size, a partial last tile, two vectors back to back."""
import numpy as np
import pytest

import dmfted
import oracle as O

pytestmark = pytest.mark.gpu


def product(s, x):
    """H x on device vectors (nvec rows of x), in x's precision."""
    import torch
    d = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    y = torch.empty_like(d)
    torch.cuda.synchronize()
    lib = dmfted.lib()
    f = lib.dmfted_hxv_device_f64 if x.dtype == np.float64 else lib.dmfted_hxv_device_f32
    assert f(s.ctx, d.data_ptr(), y.data_ptr(), x.shape[0]) == 0, lib.dmfted_last_error()
    torch.cuda.synchronize()
    return y.cpu().numpy()


def solver(nbath, nup, ndw):
    m = O.seeded_model(11, nbath=nbath, u=2.0)
    s = dmfted.EDSolver(dmfted.default_params(norb=1, nbath=nbath, uloc=[2.0], beta=100.0, lmats=16,
                                              lreal=0))
    s.set_bath(m.bath_array())
    s.setup_hv_sector(s.sector_index(nup, ndw))
    return m, s


@pytest.mark.parametrize("nbath,nup,ndw", [
    (6, 3, 2),    # 35 x 21
    (6, 7, 3),    # one row
    (10, 3, 4),   # 165 x 330
    (10, 4, 3),   # 330 x 165: even rows, the second vector's base is even too
    (11, 4, 5),   # 495 x 792
    (12, 5, 2),   # 1287 x 78
])
def test_odd_rows_match_oracle(nbath, nup, ndw):
    m, s = solver(nbath, nup, ndw)
    hm = O.build_sector(nbath + 1, nup, ndw)
    x = np.random.default_rng(3).normal(size=(2, hm.size))
    ref = O.hxv(m, hm, x[0] + 1j * x[1], nthreads=4)
    ref = np.stack([ref.real, ref.imag])
    # the bars of the product tests: 1e-13 (FP64) and 2e-6 (FP32) of the largest
    scale = np.abs(ref).max()
    assert np.abs(product(s, x) - ref).max() <= 1e-13 * scale
    assert np.abs(product(s, x.astype(np.float32)) - ref).max() <= 2e-6 * scale
    s.close()


def test_an_infinite_element_reaches_only_the_rows_it_couples_to():
    _, s = solver(6, 3, 2)
    n, i = 35 * 21, 311
    e = np.zeros((1, n))
    e[0, i] = 1.0
    coupled = product(s, e)[0] != 0.0
    e[0, i] = np.inf
    assert np.array_equal(~np.isfinite(product(s, e)[0]), coupled)
    s.close()
