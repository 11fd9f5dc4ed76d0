"""The device exchange (one warp per sample) against the library's host-side
exchange (parallel_tempering.cu:316-352) fed the same energies and drand48
state: permutation, counters and betas equal after every step, for few and
for more than 32 replicas per temperature and for samples too large to be
staged in shared memory.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("NT,nrep,samples", [(2, 1, 1), (5, 3, 4), (7, 32, 1), (3, 33, 2), (4, 70, 1), (2, 2100, 1)])
def test_exchange_matches_host(NT, nrep, samples):
    import cuda_pspin_b200 as ps
    R = NT * nrep
    cfgs = [ps.default_config(N=8, nrep=R, seed=70 + k) for k in range(samples)]
    with ps.Engine(cfgs) as eng:
        _, betas = ps.temperature_schedule(NT, 0.3, 1.5, True)
        eng.pt_init(NT, nrep, betas, 1)
        perm = np.tile(np.arange(R, dtype=np.int32), (samples, 1))
        drand = np.array([((int(c.seed) + 5000) << 16) | 0x330E for c in cfgs], np.uint64)
        acc, prop = np.zeros((samples, NT - 1), np.int64), np.zeros((samples, NT - 1), np.int64)
        off = np.arange(samples, dtype=np.int64) * R
        for _ in range(6):
            eng.pt_run(1)
            E = eng.get_results()[0]
            ps.exchange_host(betas, E, off, perm, drand, acc, prop)
            for k in range(samples):
                p, a, n = eng.pt_get(k)
                assert np.array_equal(p, perm[k]) and np.array_equal(a, acc[k]) and np.array_equal(n, prop[k])
