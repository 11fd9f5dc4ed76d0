"""Two-pass sweeps (recording and learned proposal): how a replica block's
chains are spread over CTAs, and the format of its lists (dense tiles or
groups), do not change the chain -- bit for bit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KW = [dict(N=12, nrep=33, fmc_mode=0), dict(N=21, nrep=40, fmc_mode=2, gamma=0.15), dict(N=40, nrep=8, fmc_mode=2, gamma=0.05)]


def _run(ps, cfgs, proposal, **opts):
    with ps.Engine(cfgs, ps.PSPIN_DENSE, ps.make_options(**opts)) as eng:
        eng.fill_betas(2.0)
        if proposal == ps.PROPOSAL_LEARNED:
            eng.learn_init(5)
        eng.set_proposal(proposal)
        eng.sweep(3)
        E, acc, prop = eng.get_results()
        R = cfgs[0].nrep
        return eng.get_spins()[0], E[:R], acc[:R], prop[:R]


@pytest.mark.parametrize("proposal", ["PROPOSAL_PLAIN_FIELDS", "PROPOSAL_LEARNED"])
@pytest.mark.parametrize("warps,cluster", [(1, 1), (2, 1), (8, 1), (4, 2), (1, 4), (8, 2), (2, 16), (8, 4)])
@pytest.mark.parametrize("kw", KW)
def test_plan_does_not_change_the_chain(proposal, warps, cluster, kw):
    """One sample alone (up to 8 CTAs per block), among a few (3 to 7, CTAs with an
    uneven share) and among enough to fill the machine (the block shape's own)."""
    import cuda_pspin_b200 as ps
    out = []
    for copies in (1, 11, 26, 90):
        cfgs = [ps.default_config(seed=50 + k, T=0.5, **kw) for k in range(copies)]
        out.append(_run(ps, cfgs, getattr(ps, proposal), warps_per_unit=warps, cluster_size=cluster))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
    assert out[0][2].sum() > 0


@pytest.mark.parametrize("proposal", ["PROPOSAL_PLAIN_FIELDS", "PROPOSAL_LEARNED"])
@pytest.mark.parametrize("kw", KW[1:] + [dict(N=70, nrep=4, fmc_mode=2, gamma=0.9)])
@pytest.mark.parametrize("copies", [1, 80])
def test_tiles_equal_groups(proposal, kw, copies):
    import cuda_pspin_b200 as ps
    if kw["N"] == 70 and copies > 1:
        copies = 4
    out = []
    for generic in (False, True):
        cfgs = [ps.default_config(seed=17 + k, T=0.5, **kw) for k in range(copies)]
        out.append(_run(ps, cfgs, getattr(ps, proposal), warps_per_unit=8, cluster_size=1, generic_lists=generic))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[0][2].sum() > 0
