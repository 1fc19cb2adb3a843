"""Batched jobs whose vectors stay on chip (one CTA or a cluster) against the
grid-wide path on the same problems, at the shapes where the work split has its
edges: a row count that does not divide the block, more up than down words and
the reverse (up words are always the rows), a single row, chains that need one to
four CTAs (test_gpu_chain_kernels.py holds those that need sixteen)."""
import os

import numpy as np
import pytest

import dmfted

pytestmark = pytest.mark.gpu


def solve(env, norb, nbath, nspin, sectors, total=1, lmats=128, seed=31):
    rng = np.random.default_rng(seed)
    e = rng.uniform(-1.0, 1.0, (nspin, norb, nbath))
    v = 0.5 + rng.uniform(-0.1, 0.1, (nspin, norb, nbath))
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        p = dmfted.default_params(norb=norb, nbath=nbath, nspin=nspin, uloc=[2.5] * norb,
                                  ust=1.5 if norb > 1 else 0.0, jh=0.5 if norb > 1 else 0.0,
                                  beta=40.0, lmats=lmats, lreal=0, lanc_nstates_total=total)
        with dmfted.EDSolver(p) as s:
            idx = None if sectors is None else [s.sector_index(*n) for n in sectors]
            s.ed_solve(np.concatenate([e.reshape(-1), v.reshape(-1)]), sectors=idx)
            en, _, z = s.eigenspace()
            return en, z, s.ed_get_gimp_matsubara()
    finally:
        for k, val in old.items():
            os.environ.pop(k) if val is None else os.environ.__setitem__(k, val)


@pytest.mark.parametrize("cluster", ["1", "2", "8"])
@pytest.mark.parametrize("norb,nbath,nspin,sector", [
    (1, 8, 1, (3, 6)),   # 84 x 84
    (1, 8, 2, (6, 4)),   # 84 x 126, chains with more up words too
    (1, 6, 1, (0, 3)),   # a single up word; the hole chains do not exist
    (1, 10, 1, (4, 4)),  # the hole chains (54,450 states) need 4 CTAs and more
    (2, 4, 2, (4, 3)),   # two orbitals, up to eight hops a word
])
def test_onchip_chains_match_the_grid_path(norb, nbath, nspin, sector, cluster):
    # the bars of the batched path against the grid path (test_gpu_batch.py)
    grid = solve({"DMFTED_BATCH_MAX_DIM": "0"}, norb, nbath, nspin, [sector])
    chip = solve({"DMFTED_BATCH_CLUSTER_GF": cluster, "DMFTED_BATCH_CLUSTER_MIN": "8"},
                 norb, nbath, nspin, [sector])
    assert np.allclose(chip[0], grid[0], rtol=0, atol=1e-10 * np.abs(grid[0]).max())
    assert np.abs(chip[2] - grid[2]).max() <= 1e-9
