"""The large CTA of the lean H*v (768 threads, one tile per SM), which takes the
half-filled sector of 16 sites over from the kernel with the columns in global
memory: the product of that sector digit for digit and the fused Lanczos step
against the global kernel, and the form forced on smaller sectors against the
oracle (rows below, near and above two per thread, partial last tiles)."""
import ctypes as C

import numpy as np
import pytest

import dmfted
import oracle as O

pytestmark = pytest.mark.gpu

GLOBAL, LARGE = "3", "4"


def solver(monkeypatch, kern, nbath, **kw):
    monkeypatch.setenv("DMFTED_HXV_KERNEL", kern)
    m = O.seeded_model(11, nbath=nbath, u=3.0)
    s = dmfted.EDSolver(dmfted.default_params(norb=1, nbath=nbath, uloc=[3.0], beta=100.0,
                                              lmats=256, lreal=0, **kw))
    s.set_bath(m.bath_array())
    return m, s


def product(s, x):
    import torch
    y = torch.empty_like(x)
    torch.cuda.synchronize()
    lib = dmfted.lib()
    f = lib.dmfted_hxv_device_f64 if x.dtype == torch.float64 else lib.dmfted_hxv_device_f32
    dmfted._ck(f(s.ctx, x.data_ptr(), y.data_ptr(), 1))
    torch.cuda.synchronize()
    return y


def test_half_filled_sector_of_16_sites_repeats_the_global_kernel(monkeypatch):
    import torch
    dim, steps = 12870 ** 2, 3
    gen = torch.Generator("cuda").manual_seed(1)
    x = torch.randn(dim, dtype=torch.float64, device="cuda", generator=gen)
    out = []
    for kern in ("0", GLOBAL):
        _, s = solver(monkeypatch, kern, 15)
        isec = s.sector_index(8, 8)
        assert s.sector_dim(isec) == dim
        s.setup_hv_sector(isec)
        y, y32 = product(s, x), product(s, x.float())
        work = torch.empty(2 * dim, dtype=torch.float64, device="cuda")
        a, b = (torch.empty(steps, dtype=torch.float64, device="cuda") for _ in range(2))
        used = torch.empty(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        dmfted._ck(dmfted.lib().dmfted_lanc_tridiag_noalloc(
            s.ctx, isec, C.c_void_p(x.data_ptr()), steps,
            *(C.c_void_p(t.data_ptr()) for t in (work, a, b, used))))
        out.append((y, y32, a.cpu().numpy(), b.cpu().numpy()))
        del work
        s.close()
    (y, y32, a, b), (z, z32, ga, gb) = out
    assert torch.equal(y, z) and torch.equal(y32, z32)
    # the same elements, summed compensated over other splits
    assert np.abs(a - ga).max() <= 1e-13 * np.abs(ga).max()
    assert np.abs(b - gb).max() <= 1e-13 * np.abs(gb).max()


@pytest.mark.parametrize("nbath,nup,ndw", [
    (7, 4, 4),    # 70 x 70: a partial last tile in FP32
    (11, 5, 4),   # 792 x 495: a partial last tile in both precisions
    (12, 6, 6),   # 1716 rows: two passes of 1536
])
def test_forced_on_smaller_sectors_matches_oracle(monkeypatch, nbath, nup, ndw):
    import torch
    m, s = solver(monkeypatch, LARGE, nbath)
    s.setup_hv_sector(s.sector_index(nup, ndw))
    hm = O.build_sector(nbath + 1, nup, ndw)
    x = np.random.default_rng(3).normal(size=hm.size)
    ref = O.hxv(m, hm, x.astype(complex), nthreads=4).real
    # the bars of the product tests: 1e-13 (FP64) and 2e-6 (FP32) of the largest
    scale, d = np.abs(ref).max(), torch.from_numpy(x).cuda()
    assert np.abs(product(s, d).cpu().numpy() - ref).max() <= 1e-13 * scale
    assert np.abs(product(s, d.float()).cpu().numpy() - ref).max() <= 2e-6 * scale
    s.close()


@pytest.mark.parametrize("precision", [dmfted.FP64, dmfted.MIXED])
def test_forced_solve_matches_default_kernels(monkeypatch, precision):
    # both precisions' Lanczos steps; the bars of the same test of the global kernel
    out = []
    for kern in ("0", LARGE):
        m, s = solver(monkeypatch, kern, 9, precision=precision, lanc_nstates_sector=1)
        s.ed_solve(m.bath_array(), sectors=[s.sector_index(5, 5)])
        out.append((s.egs(), s.ed_get_gimp_matsubara()))
        s.close()
    assert abs(out[0][0] - out[1][0]) <= 1e-12 * abs(out[0][0])
    assert np.abs(out[0][1] - out[1][1]).max() <= 1e-10
