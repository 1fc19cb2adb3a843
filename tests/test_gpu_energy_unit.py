"""The dense branch's eigenvalues do not depend on the unit of energy: scaling
every energy by a power of two is exact in FP64, so the Sturm counts have to
give the scaled eigenvalues also where eight steps of the leading minors would
leave the range of FP64 (|H| below about 1e-38)."""
import numpy as np
import pytest

import dmfted

pytestmark = pytest.mark.gpu


def ground_energy(scale, nup, ndw):
    rng = np.random.default_rng(5)
    e, v = rng.uniform(-1.0, 1.0, 5), 0.5 + rng.uniform(-0.1, 0.1, 5)
    p = dmfted.default_params(norb=1, nbath=5, nspin=1, uloc=[2.0 * scale], beta=100.0 / scale,
                              lmats=16, lreal=0, gs_threshold=1e-9 * scale,
                              lanc_dim_threshold=512, lanc_nstates_sector=4)
    with dmfted.EDSolver(p) as s:
        s.ed_solve(np.concatenate([e, v]) * scale, sectors=[s.sector_index(nup, ndw)])
        return s.egs() / scale


@pytest.mark.parametrize("nup,ndw", [(1, 1), (2, 2), (3, 3)])  # 36, 225 and 400 states
@pytest.mark.parametrize("power", [-40, -120, -140, -200])
def test_ground_energy_scales_with_the_unit(power, nup, ndw):
    one = ground_energy(1.0, nup, ndw)
    # the multisection stops within 4.4e-16 of the value
    assert abs(ground_energy(2.0 ** power, nup, ndw) - one) <= 1e-14 * abs(one)
