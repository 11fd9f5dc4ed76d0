"""Lists of dense samples built on the device: the chain (whose bits depend on
every list's order and parts), the FP64 energies (the quartet table's order) and
the list-resident sweep (the neighbour masks) equal those of an engine whose lists
the host makes (generic_lists), bit for bit.
"""
import hashlib
import json
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden", "fc_chains.json")


def _run(ps, cfgs, generic, **opts):
    opts = ps.make_options(generic_lists=generic, **opts)
    with ps.Engine(cfgs, ps.PSPIN_DENSE, opts) as eng:
        eng.fill_betas(2.0)
        E0 = eng.get_results()[0]
        e2, e4 = eng.split_energies()
        eng.sweep(2)
        return [np.concatenate([a.ravel() for a in eng.get_spins()]), E0, e2, e4, *eng.get_results()]


@pytest.mark.parametrize("shape", [dict(warps_per_unit=8, cluster_size=1), dict(warps_per_unit=4, cluster_size=8)])
@pytest.mark.parametrize("kw", [dict(N=5, nrep=3, fmc_mode=2, gamma=2.0), dict(N=12, nrep=33, fmc_mode=2, gamma=0.3),
                                dict(N=33, nrep=5, fmc_mode=2, gamma=0.1), dict(N=40, nrep=8, fmc_mode=2, gamma=0.004),
                                dict(N=24, nrep=5, fmc_mode=1, gamma=2.0), dict(N=70, nrep=4, fmc_mode=2, gamma=0.9),
                                dict(N=32, nrep=4, fmc_mode=2, gamma=0.1, alpha=0.0, alpha0=0.0),
                                dict(N=72, nrep=2, fmc_mode=2, gamma=1e-9)])
def test_device_lists_equal_host_lists(kw, shape):
    import cuda_pspin_b200 as ps
    cfg = ps.default_config(seed=23, T=0.5, **kw)
    for a, b in zip(_run(ps, cfg, False, **shape), _run(ps, cfg, True, **shape)):
        np.testing.assert_array_equal(a, b)


def test_mixed_batch():
    """Fully connected and masked samples in one engine."""
    import cuda_pspin_b200 as ps
    cfgs = [ps.default_config(N=n, nrep=4, seed=30 + n, fmc_mode=f, gamma=0.2) for n, f in ((9, 0), (21, 2), (16, 0), (34, 2))]
    opts = dict(warps_per_unit=2, cluster_size=2)
    whole = _run(ps, cfgs, False, **opts)
    at = 0
    rep = 0
    for c in cfgs:
        one = _run(ps, [c], False, **opts)
        np.testing.assert_array_equal(whole[0][at:at + 4 * c.N], one[0])
        for a, b in zip(whole[1:], one[1:]):
            np.testing.assert_array_equal(a[rep:rep + 4], b)
        at += 4 * c.N
        rep += 4


@pytest.mark.parametrize("kw", [dict(N=14, nrep=40, fmc_mode=2, gamma=0.02), dict(N=24, nrep=20, fmc_mode=1, gamma=1.0)])
def test_neighbours_of_resident_moves(kw):
    """Commuting moves of the list-resident sweep (one warp takes them in order)."""
    import cuda_pspin_b200 as ps
    cfg = ps.default_config(seed=11, T=0.5, **kw)
    ref = _run(ps, cfg, True, warps_per_unit=1, cluster_size=-1)
    for warps in (1, 8):
        for a, b in zip(_run(ps, cfg, False, warps_per_unit=warps, cluster_size=-1), ref):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("key", sorted(json.load(open(GOLDEN))))
def test_fully_connected_chain_is_pinned(key):
    """Digests of amplitudes after three sweeps and of the first energies, recorded
    with lists made on the host (they have no generic twin of the same order)."""
    import cuda_pspin_b200 as ps
    N, R, warps, cluster = map(int, key.split(","))
    cfg = ps.default_config(N=N, nrep=R, seed=40 + N, T=0.5)
    with ps.Engine(cfg, ps.PSPIN_DENSE, ps.make_options(warps_per_unit=warps, cluster_size=cluster)) as eng:
        eng.fill_betas(2.0)
        E0 = eng.get_results()[0]
        eng.sweep(3)
        s = np.ascontiguousarray(eng.get_spins()[0])
    assert hashlib.md5(s.tobytes() + E0.tobytes()).hexdigest() == json.load(open(GOLDEN))[key]
