"""The two kernels of the batched Green's-function chains -- vectors on chip
(k_chains_onchip) and in L2 (k_batch_chains) -- against each other and across
the cluster sizes: chains with spin exchange and pair hopping (always through
L2), without (either kernel), solves whose chains split between both, and the
largest chains a cluster of 16 holds."""
import os

import numpy as np
import pytest

import dmfted

pytestmark = pytest.mark.gpu


def solve(env, norb, nbath, nspin, sectors, total=1, jhflag=0, seed=31, reps=0):
    rng = np.random.default_rng(seed)
    e = rng.uniform(-1.0, 1.0, (nspin, norb, nbath))
    v = 0.5 + rng.uniform(-0.1, 0.1, (nspin, norb, nbath))
    two = norb > 1
    old = {k: os.environ.get(k) for k in env}
    os.environ.update(env)
    try:
        p = dmfted.default_params(norb=norb, nbath=nbath, nspin=nspin, uloc=[2.5] * norb,
                                  ust=1.5 if two else 0.0, jh=0.5 if two else 0.0, jhflag=jhflag,
                                  jx=0.3 * jhflag, jp=0.2 * jhflag, beta=40.0, lmats=128, lreal=0,
                                  lanc_nstates_total=total)
        with dmfted.EDSolver(p) as s:
            idx = None if sectors is None else [s.sector_index(*n) for n in sectors]
            bath = np.concatenate([e.reshape(-1), v.reshape(-1)])
            s.ed_solve(bath, sectors=idx)
            g, n = s.ed_get_gimp_matsubara(), s.launch_count()
            if not reps:
                return g, n
            times = []
            for _ in range(reps):
                s.ed_solve(bath, sectors=idx)
                times.append(s.timings()["gf_ms"])
            return min(times)
    finally:
        for k, val in old.items():
            os.environ.pop(k) if val is None else os.environ.__setitem__(k, val)


# the same eigenvectors, chains with compensated sums over other splits: the bar
# of the cluster sizes against one CTA (test_gpu_batch.py)
BAR = 1e-11


@pytest.mark.parametrize("cluster", ["1", "2", "4", "8", "16"])
@pytest.mark.parametrize("jhflag", [0, 1])
def test_chains_through_l2_match_across_cluster_sizes(jhflag, cluster):
    base = {"DMFTED_CHAINS_ONCHIP": "0", "DMFTED_BATCH_CLUSTER_MIN": "8",
            "DMFTED_BATCH_CLUSTER_EIGS": "1"}
    args = (2, 2, 2, None, 16, jhflag)
    one, _ = solve(dict(base, DMFTED_BATCH_CLUSTER_GF="1"), *args)
    many, _ = solve(dict(base, DMFTED_BATCH_CLUSTER_GF=cluster), *args)
    assert np.abs(many - one).max() <= BAR
    if not jhflag:  # the same solve on chip
        chip, _ = solve({"DMFTED_BATCH_CLUSTER_GF": cluster, "DMFTED_BATCH_CLUSTER_MIN": "8",
                         "DMFTED_BATCH_CLUSTER_EIGS": "1"}, *args)
        assert np.abs(chip - one).max() <= BAR


@pytest.mark.parametrize("nbath,sector", [
    (11, (4, 2)),  # the particle chain (5, 2) has 792 rows (L2), the hole chain (3, 2) 220
    (11, (5, 2)),  # (6, 2) through L2, (4, 2) on chip: 495 rows
    (10, (5, 4)),  # the hole chains: 330 x 330 (108,900 states, a cluster of 16)
    (12, (4, 3)),  # the hole chain: 286 x 286
])
def test_chains_split_between_the_kernels(nbath, sector):
    mixed, n_mixed = solve({}, 1, nbath, 1, [sector])
    l2, n_l2 = solve({"DMFTED_CHAINS_ONCHIP": "0"}, 1, nbath, 1, [sector])
    assert np.abs(mixed - l2).max() <= BAR
    # a device that holds no cluster of 16: the largest chains go through L2
    eight, _ = solve({"DMFTED_CHAINS_ONCHIP": "8"}, 1, nbath, 1, [sector])
    assert np.abs(eight - l2).max() <= BAR
    if sector[1] == 2:  # one launch each for the two kernels
        assert n_mixed == n_l2 + 1


def test_split_chains_run_at_once():
    # one list after the other takes 1.5 times as long as both chains through L2
    split, l2 = (solve(env, 1, 11, 1, [(4, 2)], reps=9)
                 for env in ({}, {"DMFTED_CHAINS_ONCHIP": "0"}))
    assert split <= 1.25 * l2
