"""List-resident sweeps of many blocks run in batches of commuting moves, of few as a
dataflow: the same chain bit for bit as one warp per block, and as single samples.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(ps, samples, Ns, R, fmc, variant, warps, NT, out):
    cfgs = [ps.default_config(N=Ns[k % len(Ns)], nrep=R, seed=200 + k, fmc_mode=fmc, T=0.5) for k in range(samples)]
    for c in cfgs:
        c.gamma = {0: c.gamma, 1: 1.0, 2: 0.3}[fmc]
    opts = ps.make_options(warps_per_unit=warps, cluster_size=-1, resync_every=-1, disorder_stream=variant == ps.PSPIN_SPARSE)
    with ps.Engine(cfgs, variant, opts) as eng:
        if NT:
            _, betas = ps.temperature_schedule(NT, 0.3, 1.5, True)
            eng.pt_init(NT, R // NT, betas, 2)
        else:
            eng.fill_betas(1.5)
        for n in (1, 4, 9):
            (eng.pt_run if NT else eng.sweep)(n)
        eng.get_profile()
        eng.sweep(20)
        launches = eng.get_profile()[2]
        E, acc, prop = eng.get_results()
        state = [np.concatenate([a.ravel() for a in eng.get_spins()]), E, acc, prop]
        for k in range(samples if NT else 0):
            state += [x.copy() for x in eng.pt_get(k)]
        out.append(state)
    return launches


@pytest.mark.parametrize("NT", [0, 8])
@pytest.mark.parametrize("Ns,R,fmc,sparse", [((12, 30, 17), 96, 1, True),       # one-entry groups
                                             ((33, 8), 40, 0, True),            # quartets drawn from all of them
                                             ((12, 9), 72, 0, False),           # fully connected tiles
                                             ((14, 12), 96, 2, False)])         # masked tiles or records
def test_the_form_does_not_change_the_chain(Ns, R, fmc, sparse, NT):
    import cuda_pspin_b200 as ps
    variant = ps.PSPIN_SPARSE if sparse else ps.PSPIN_DENSE
    out, launches = [], {}
    for warps in (1, 2, 8):
        launches[warps] = _run(ps, 170, Ns, R, fmc, variant, warps, NT, out)
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
    assert out[0][2].sum() > 0
    assert launches[8] == 2                     # batched: nothing prepared
    few = []                                    # of two warps: a dataflow, prepared
    assert _run(ps, 2, Ns, R, fmc, variant, 2, NT, few) == 3
    n0 = sum(Ns[k % len(Ns)] * R for k in range(2))
    np.testing.assert_array_equal(few[0][0], out[0][0][:n0])
    for q in (2, 3):
        np.testing.assert_array_equal(few[0][q], out[0][q][:2 * R])
    np.testing.assert_array_equal(few[0][1], out[0][1][:2 * R])


@pytest.mark.parametrize("N,warps,sweeps,launches", [(32, 4, 9, 2), (34, 4, 9, 3), (64, 8, 9, 2), (66, 8, 9, 3), (16, 2, 9, 3),
                                                     (64, 2, 2, 2), (66, 2, 2, 3), (128, 8, 1, 2), (130, 8, 1, 3), (96, 1, 1, 2)])
def test_forms_at_their_bounds(N, warps, sweeps, launches):
    """Few blocks: batched at N <= 8 warps from four warps on, and up to 64 moves a
    launch; the state is the one-warp chain's."""
    import cuda_pspin_b200 as ps
    out = []
    for w in (warps, 1):
        c = ps.default_config(N=N, nrep=40, seed=4, fmc_mode=1, T=0.5)
        c.gamma = 1.0
        with ps.Engine(c, ps.PSPIN_SPARSE, ps.make_options(warps_per_unit=w, cluster_size=-1, resync_every=-1,
                                                           disorder_stream=True)) as eng:
            eng.fill_betas(1.5)
            eng.get_profile()
            eng.sweep(sweeps)
            if w == warps:
                assert eng.get_profile()[2] == launches
            out.append([eng.get_spins()[0], *eng.get_results()])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
