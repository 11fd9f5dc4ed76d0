"""Two-pass sweeps of block shapes with many CTAs: with few blocks every chain's sum
goes to the other CTAs, with full SMs the sums of the shape's CTAs, on as few CTAs as
hold the chains -- the same chain bit for bit, and an abort leaves the state alone.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(ps, copies, warps, cluster, proposal, **opts):
    cfgs = [ps.default_config(N=16 + 5 * (k % 2), nrep=40, seed=70 + k, T=0.5, fmc_mode=0) for k in range(copies)]
    eng = ps.Engine(cfgs, ps.PSPIN_DENSE, ps.make_options(warps_per_unit=warps, cluster_size=cluster, resync_every=-1, **opts))
    eng.fill_betas(2.0)
    eng.learn_init(5)
    eng.set_proposal(proposal)
    return eng


@pytest.mark.parametrize("proposal", [1, 2])
@pytest.mark.parametrize("warps,cluster", [(4, 2), (4, 4), (8, 2), (8, 4), (4, 8), (2, 8), (1, 16), (2, 16)])
def test_full_machine_equals_one_sample(warps, cluster, proposal):
    import cuda_pspin_b200 as ps
    out = []
    for copies in (2, 18, 100):
        with _engine(ps, copies, warps, cluster, proposal) as eng:
            eng.sweep(3)
            E, acc, prop = eng.get_results()
            out.append((*eng.get_spins()[:2], E[:80], acc[:80], prop[:80]))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
    assert out[0][3].sum() > 0


@pytest.mark.parametrize("stall", [1, 9])
def test_an_abort_with_group_sums_keeps_the_state(stall):
    import cuda_pspin_b200 as ps
    with _engine(ps, 100, 8, 4, 1, wait_limit_clocks=2_000_000, test_stall_move=stall) as eng:
        before = [np.concatenate([a.ravel() for a in eng.get_spins()]), *eng.get_results()]
        with pytest.raises(ps.PspinError) as ei:
            eng.sweep(2)
        assert ei.value.code == ps.PSPIN_ERR_TIMEOUT
        for a, b in zip(before, [np.concatenate([a.ravel() for a in eng.get_spins()]), *eng.get_results()]):
            np.testing.assert_array_equal(a, b)
