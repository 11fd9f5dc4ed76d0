"""A wait that runs out in a launch whose replica blocks run as several tasks, or as
a cluster of blocks that exchange: every block keeps its state from before the
launch, with PT its permutation, counters and betas too.

The waits are made to run out by the test option test_stall_move, within about a
millisecond each; no GPU fault or endless wait is involved.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STALL_CLOCKS = 2_000_000        # ~1 ms at 1.9 GHz


def _state(eng, samples, pt):
    E, acc, prop = eng.get_results()
    out = [np.concatenate([a.ravel() for a in eng.get_spins()]), E, acc, prop]
    for k in range(samples if pt else 0):
        out += [x.copy() for x in eng.pt_get(k)]
    return out


def _engine(ps, Ns, samples, NT, nrep, stall, pt, sparse=False, **opts):
    cfgs = [ps.default_config(N=Ns[k % len(Ns)], nrep=NT * nrep, seed=40 + k, fmc_mode=1 if sparse else 0)
            for k in range(samples)]
    for c in cfgs:
        c.gamma = 1.0 if sparse else c.gamma
    eng = ps.Engine(cfgs, ps.PSPIN_SPARSE if sparse else ps.PSPIN_DENSE,
                    ps.make_options(resync_every=-1, wait_limit_clocks=STALL_CLOCKS, test_stall_move=stall,
                                    disorder_stream=sparse, **opts))
    _, betas = ps.temperature_schedule(NT, 0.3, 1.5, True)
    if pt:
        eng.pt_init(NT, nrep, betas, 1)
    else:
        eng.set_betas(np.tile(np.repeat(betas, nrep), samples))
    return eng


@pytest.mark.parametrize("pt", [False, True])
@pytest.mark.parametrize("Ns,samples,warps,cluster,lanes,stall", [
    ((8,), 200, 8, 1, 3, 1),             # four moves a sweep, the last of three tasks holds two sweeps
    ((8,), 200, 8, 4, 3, 6),             # on clusters
    ((8, 20), 200, 8, 2, 3, 5),          # samples of uneven size
    ((8,), 200, 8, 1, 3, 8),             # at the launch's last move
    ((8, 20), 200, 8, 1, 3, 15),         # only the larger samples' last tasks have that many moves
])
def test_a_queued_launch_keeps_the_state_from_before_it(ps, Ns, samples, warps, cluster, lanes, stall, pt):
    NT, nrep, sweeps = 24, 4, 6
    opts = dict(warps_per_unit=warps, cluster_size=cluster, replicas_per_lane=lanes)
    with _engine(ps, Ns, samples, NT, nrep, stall, pt, **opts) as eng:
        run = eng.pt_run if pt else eng.sweep
        before = _state(eng, samples, pt)
        with pytest.raises(ps.PspinError) as ei:
            run(sweeps)
        assert ei.value.code == ps.PSPIN_ERR_TIMEOUT, str(ei.value)
        after = _state(eng, samples, pt)
        steps = np.repeat([Ns[k % len(Ns)] // 2 for k in range(samples)], NT * nrep)
        reached = steps * 2 >= stall                     # the stall is a move of these samples' last task
        assert np.array_equal(before[3][reached], after[3][reached])
        assert np.array_equal(before[1][reached], after[1][reached])
        if reached.all():
            for a, b in zip(before, after):
                np.testing.assert_array_equal(a, b)
        e2, e4 = eng.split_energies()                    # the context works, energies and amplitudes agree
        np.testing.assert_allclose(after[1], e2 + e4, rtol=0, atol=1e-4 * np.abs(e2 + e4).max())


@pytest.mark.parametrize("pt", [False, True])
def test_a_stall_beyond_the_launch_changes_nothing(ps, pt):
    out = []
    for stall in (0, 1000):
        opts = dict(warps_per_unit=8, cluster_size=2, replicas_per_lane=3)
        with _engine(ps, (8, 12), 200, 12, 4, stall, pt, **opts) as eng:
            (eng.pt_run if pt else eng.sweep)(7)
            out.append(_state(eng, 200, pt))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[0][2].sum() > 0


@pytest.mark.parametrize("warps", [2, 8])
@pytest.mark.parametrize("samples,N,NT,nrep,stall,pt", [
    (1, 96, 24, 4, 1, True), (3, 64, 24, 4, 70, True),       # three blocks a sample: one of a cluster gives up
    (2, 48, 10, 17, 144, True),                              # six, a ragged last, at the launch's last move
    (2, 48, 4, 8, 100, True), (3, 96, 10, 4, 33, False),     # one block; blocks of their own
])
def test_resident_blocks_of_a_sample_abort_together(ps, samples, N, NT, nrep, stall, pt, warps):
    with _engine(ps, (N,), samples, NT, nrep, stall, pt, sparse=True, warps_per_unit=warps, cluster_size=-1) as eng:
        before = _state(eng, samples, pt)
        with pytest.raises(ps.PspinError) as ei:
            (eng.pt_run if pt else eng.sweep)(6)
        assert ei.value.code == ps.PSPIN_ERR_TIMEOUT, str(ei.value)
        for a, b in zip(before, _state(eng, samples, pt)):
            np.testing.assert_array_equal(a, b)


def test_a_short_copy_limit_does_not_end_resident_moves(ps):
    """Waits for earlier moves and for other blocks are not copies: a limit of a few
    clocks leaves them alone."""
    out = []
    for limit in (0, 50):
        cfgs = [ps.default_config(N=96, nrep=96, seed=3, fmc_mode=1)]
        cfgs[0].gamma = 1.0
        opts = ps.make_options(warps_per_unit=8, cluster_size=-1, disorder_stream=True, wait_limit_clocks=limit)
        with ps.Engine(cfgs, ps.PSPIN_SPARSE, opts) as eng:
            _, betas = ps.temperature_schedule(24, 0.3, 1.5, True)
            eng.pt_init(24, 4, betas, 1)
            eng.pt_run(20)
            out.append(_state(eng, 1, True))
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("pt", [False, True])
@pytest.mark.parametrize("samples,warps,cluster,lanes", [(1, 8, 1, 1), (1, 2, 16, 1), (2, 8, 4, 3), (60, 8, 1, 3)])
@pytest.mark.parametrize("stall", [1, 7, 24])            # the first move, one between, the last
def test_every_block_of_a_launch_gives_up_at_any_move(ps, samples, warps, cluster, lanes, stall, pt):
    """One task a block, on one CTA and on clusters."""
    opts = dict(warps_per_unit=warps, cluster_size=cluster, replicas_per_lane=lanes)
    with _engine(ps, (8,), samples, 6, 4, stall, pt, **opts) as eng:
        before = _state(eng, samples, pt)
        for _ in range(2):
            with pytest.raises(ps.PspinError) as ei:
                (eng.pt_run if pt else eng.sweep)(6)
            assert ei.value.code == ps.PSPIN_ERR_TIMEOUT, str(ei.value)
            for a, b in zip(before, _state(eng, samples, pt)):
                np.testing.assert_array_equal(a, b)
