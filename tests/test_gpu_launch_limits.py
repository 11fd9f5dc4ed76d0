"""Limits of one sweep launch: how many sweeps pspin_pt_run puts into it, and block
shapes near the shared-memory limit.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("freq,nsweeps,launches", [(1, 300, 2), (100, 600, 3), (300, 900, 3)])
def test_a_launch_holds_at_most_256_sweeps_or_one_step(freq, nsweeps, launches):
    """The length of a launch, and with it the number of its moves (31 bits), is
    bounded by its sweeps, not by its PT steps: 256 sweeps, or one step."""
    import cuda_pspin_b200 as ps
    NT, nrep = 2, 3
    c = ps.default_config(N=8, nrep=NT * nrep, seed=5)
    with ps.Engine(c, ps.PSPIN_DENSE, ps.make_options(resync_every=-1)) as eng:
        _, betas = ps.temperature_schedule(NT, 0.3, 1.5, True)
        eng.pt_init(NT, nrep, betas, freq)
        eng.get_profile()
        eng.pt_run(nsweeps)
        assert eng.get_profile()[1] == launches
        perm, acc, prop = eng.pt_get(0)
        assert np.all(prop == nsweeps // freq * nrep)
        assert np.all(eng.get_results()[2] == nsweeps * 4)


@pytest.mark.parametrize("N,NT,nrep,lanes", [(288, 24, 4, 3), (291, 24, 4, 3), (437, 16, 4, 2), (880, 8, 4, 1)])
def test_steps_whose_exchange_does_not_fit_the_launch(N, NT, nrep, lanes):
    """Block shapes that hold a sample's amplitudes but not the exchange's arrays
    beside them run one step a launch, with the same results."""
    import cuda_pspin_b200 as ps
    out = []
    for graph_steps in (0, -1):
        c = ps.default_config(N=N, nrep=NT * nrep, seed=7, fmc_mode=1)
        c.gamma = 1.0
        opts = ps.make_options(warps_per_unit=1, cluster_size=1, replicas_per_lane=lanes, graph_steps=graph_steps,
                               disorder_stream=True)
        with ps.Engine(c, ps.PSPIN_SPARSE, opts) as eng:
            _, betas = ps.temperature_schedule(NT, 0.3, 1.5, True)
            eng.pt_init(NT, nrep, betas, 1)
            eng.pt_run(3)
            out.append([eng.get_spins()[0], *eng.get_results(), *eng.pt_get(0)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
    assert out[0][2].sum() > 0


@pytest.mark.parametrize("N,warps,cluster,lanes,fits", [(291, 1, 1, 3, True), (292, 1, 1, 3, False), (439, 1, 1, 2, True),
                                                        (440, 1, 1, 2, False), (211, 2, 16, 3, True), (212, 2, 16, 3, False),
                                                        (234, 8, 4, 3, True), (235, 8, 4, 3, False)])
def test_the_largest_N_of_a_block_shape_is_accepted_and_runs(N, warps, cluster, lanes, fits):
    """What set-up accepts by the sizes alone, the sweep runs; the next N is refused."""
    import cuda_pspin_b200 as ps
    c = ps.default_config(N=N, nrep=8, seed=7, fmc_mode=1)
    c.gamma = 1.0
    opts = ps.make_options(warps_per_unit=warps, cluster_size=cluster, replicas_per_lane=lanes, disorder_stream=True)
    if not fits:
        with pytest.raises(ps.PspinError):
            ps.Engine(c, ps.PSPIN_SPARSE, opts)
        return
    with ps.Engine(c, ps.PSPIN_SPARSE, opts) as eng:
        eng.fill_betas(1.0)
        eng.sweep(1)
        assert np.all(eng.get_results()[2] == N // 2)


def _resident(ps, warps):
    c = ps.default_config(N=512, nrep=128, seed=11, fmc_mode=1)
    c.gamma = 1.0
    opts = ps.make_options(warps_per_unit=warps, cluster_size=-1, disorder_stream=True)
    return ps.Engine(c, ps.PSPIN_SPARSE, opts)


def test_a_list_resident_run_allocates_nothing(ps):
    """The workspace of prepared moves (57 MB here) is made with the engine, given
    back with it, and made again where a checkpoint brings the shape."""
    import torch
    free = lambda: torch.cuda.mem_get_info()[0]
    _, betas = ps.temperature_schedule(32, 0.3, 1.5, True)
    for _ in range(2):                      # (the first round loads kernels as well)
        start = free()
        with _resident(ps, 8) as eng:
            eng.pt_init(32, 4, betas, 1)
            before = free()
            assert start - before > 50 << 20
            eng.pt_run(3)
            eng.sweep(2)
            after = free()
        end = free()
    assert before - after < 4 << 20
    assert start - end < 4 << 20


def test_a_checkpoint_of_a_list_resident_shape_runs_on(ps, tmp_path):
    _, betas = ps.temperature_schedule(32, 0.3, 1.5, True)
    out = []
    with _resident(ps, 8) as eng:
        eng.pt_init(32, 4, betas, 1)
        eng.pt_run(3)
        eng.checkpoint_save(str(tmp_path / "c.bin"))
        eng.pt_run(4)
        out.append([eng.get_spins()[0], *eng.get_results(), *eng.pt_get(0)])
    with _resident(ps, 1) as eng:           # made with one warp: no workspace
        eng.pt_init(32, 4, betas, 1)
        eng.checkpoint_load(str(tmp_path / "c.bin"))
        eng.pt_run(4)
        out.append([eng.get_spins()[0], *eng.get_results(), *eng.pt_get(0)])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("warps,launches", [(1, 2), (8, 3)])
def test_every_launch_is_counted(ps, warps, launches):
    """A list-resident sweep of several warps prepares its moves in a launch of its
    own: prepare, sweep, sweep counter."""
    _, betas = ps.temperature_schedule(32, 0.3, 1.5, True)
    with _resident(ps, warps) as eng:
        eng.get_profile()
        eng.sweep(1)
        assert eng.get_profile()[2] == launches
        eng.pt_init(32, 4, betas, 1)
        eng.pt_run(2)
        assert eng.get_profile()[2] == (2 if warps == 1 else 1) * launches
