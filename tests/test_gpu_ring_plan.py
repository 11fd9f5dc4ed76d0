"""How a move's chains are spread over CTAs does not change the chain: a
sample alone (few units: many CTAs, at most four chains each, or one CTA)
and the same sample among enough others to fill the machine (16 chains per
CTA) give the same amplitudes, energies and counters bit for bit, for every
block shape, list format and number of replicas per lane.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warps,cluster,lanes", [(1, 1, 1), (2, 1, 3), (8, 1, 1), (8, 1, 2), (4, 2, 1), (1, 4, 3), (8, 2, 3),
                                                 (2, 16, 1), (4, 8, 2), (8, 4, 3)])
@pytest.mark.parametrize("kw", [dict(N=12, nrep=33, fmc_mode=0), dict(N=21, nrep=70, fmc_mode=2, gamma=0.15),
                                dict(N=40, nrep=40, fmc_mode=1, gamma=1.0, sparse=True)])
def test_plan_does_not_change_the_chain(warps, cluster, lanes, kw):
    import cuda_pspin_b200 as ps
    kw = dict(kw)
    variant = ps.PSPIN_SPARSE if kw.pop("sparse", False) else ps.PSPIN_DENSE
    out = []
    for copies in (1, 90):
        cfgs = [ps.default_config(seed=50 + k, T=0.5, **kw) for k in range(copies)]
        opts = ps.make_options(warps_per_unit=warps, cluster_size=cluster, replicas_per_lane=lanes, disorder_stream=True)
        with ps.Engine(cfgs, variant, opts) as eng:
            eng.fill_betas(2.0)
            eng.sweep(3)
            E, acc, prop = eng.get_results()
            R = cfgs[0].nrep
            out.append((eng.get_spins()[0], E[:R], acc[:R], prop[:R]))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[0][2].sum() > 0


@pytest.mark.parametrize("kw", [dict(N=12, nrep=33, fmc_mode=2, gamma=0.3), dict(N=33, nrep=40, fmc_mode=2, gamma=0.1),
                                dict(N=40, nrep=8, fmc_mode=2, gamma=0.004), dict(N=64, nrep=20, fmc_mode=2, gamma=0.1),
                                dict(N=24, nrep=5, fmc_mode=1, gamma=2.0), dict(N=70, nrep=4, fmc_mode=2, gamma=0.9)])
@pytest.mark.parametrize("warps,cluster,lanes", [(8, 1, 1), (2, 16, 1), (8, 2, 3), (4, 1, 2)])
def test_tiles_equal_records(kw, warps, cluster, lanes):
    """A masked sample's lists as dense tiles (few and many terms per group,
    groups longer than 32 terms, columns of one and of eight) and as per-term
    records (generic_lists) give the same chain bit for bit."""
    import cuda_pspin_b200 as ps
    out = []
    for generic in (False, True):
        c = ps.default_config(seed=17, T=0.5, **kw)
        opts = ps.make_options(warps_per_unit=warps, cluster_size=cluster, replicas_per_lane=lanes, generic_lists=generic)
        with ps.Engine(c, ps.PSPIN_DENSE, opts) as eng:
            eng.fill_betas(2.0)
            eng.sweep(2)
            E, acc, prop = eng.get_results()
            out.append((eng.get_spins()[0], E, acc, prop))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[0][2].sum() > 0


@pytest.mark.parametrize("samples,Ns,NT,nrep,freq,warps,cluster,lanes", [
    (1, (12,), 4, 8, 1, 2, 1, 1),              # one block, one replica per lane
    (3, (8, 17, 12), 6, 5, 2, 8, 1, 2),        # ragged blocks, exchange every second sweep
    (200, (8, 11, 20, 9), 3, 4, 1, 8, 2, 3),   # more blocks than run at once: tasks from the queue
    (170, (6, 14), 2, 40, 3, 8, 4, 3),         # the same with 40 columns, a cluster of many CTAs
])
def test_steps_in_one_launch_equal_single_steps(samples, Ns, NT, nrep, freq, warps, cluster, lanes):
    """PT steps inside one launch (exchange by the sweep kernel's deciders,
    units in tasks) equal one launch per step with the exchange kernel: states,
    counters, betas by their effect, permutations; across resyncs and partial
    steps."""
    import cuda_pspin_b200 as ps
    out = []
    for graph_steps in (0, -1):
        cfgs = [ps.default_config(N=Ns[k % len(Ns)], nrep=NT * nrep, seed=80 + k) for k in range(samples)]
        opts = ps.make_options(warps_per_unit=warps, cluster_size=cluster, replicas_per_lane=lanes,
                               graph_steps=graph_steps, resync_every=11)
        with ps.Engine(cfgs, ps.PSPIN_DENSE, opts) as eng:
            _, betas = ps.temperature_schedule(NT, 0.3, 1.5, True)
            eng.pt_init(NT, nrep, betas, freq)
            for n in (1, 7, 9):
                eng.pt_run(n)
            pt = [eng.pt_get(k) for k in range(samples)]
            out.append([np.concatenate([a.ravel() for a in eng.get_spins()]), *eng.get_results(),
                        np.stack([p[0] for p in pt]), np.stack([p[1] for p in pt]), np.stack([p[2] for p in pt])])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[0][5].sum() > 0


@pytest.mark.parametrize("samples,N,NT,nrep,freq,fmc", [(1, 96, 2, 3, 1, 1), (3, 64, 8, 8, 2, 0), (2, 48, 5, 17, 1, 1)])
@pytest.mark.parametrize("warps", [2, 8])
def test_resident_steps_in_one_launch_equal_single_steps(samples, N, NT, nrep, freq, fmc, warps):
    """List-resident blocks of one sample as a cluster that exchanges inside the
    launch (one block, two, three with a ragged last) equal one launch and one
    exchange kernel per step, and one-warp blocks."""
    import cuda_pspin_b200 as ps
    out = []
    for graph_steps, w in ((0, warps), (-1, warps), (-1, 1)):
        cfgs = [ps.default_config(N=N, nrep=NT * nrep, seed=60 + k, fmc_mode=fmc) for k in range(samples)]
        for c in cfgs:
            c.gamma = 1.0 if fmc == 1 else 0.0
        opts = ps.make_options(warps_per_unit=w, cluster_size=-1, graph_steps=graph_steps, resync_every=11,
                               disorder_stream=True)
        with ps.Engine(cfgs, ps.PSPIN_SPARSE, opts) as eng:
            _, betas = ps.temperature_schedule(NT, 0.3, 1.5, True)
            eng.pt_init(NT, nrep, betas, freq)
            for n in (1, 7, 9):
                eng.pt_run(n)
            pt = [eng.pt_get(k) for k in range(samples)]
            out.append([np.concatenate([a.ravel() for a in eng.get_spins()]), *eng.get_results(),
                        np.stack([p[0] for p in pt]), np.stack([p[1] for p in pt]), np.stack([p[2] for p in pt])])
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
    assert out[0][5].sum() > 0
