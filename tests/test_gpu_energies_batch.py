"""The FP64 energies of a sample are its own: the same bits alone and among
other samples, whatever the number of CTAs that a table is summed on.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw", [dict(N=48, nrep=96, fmc_mode=0), dict(N=64, nrep=40, fmc_mode=0),
                                dict(N=56, nrep=33, fmc_mode=2, gamma=0.2)])
def test_energies_do_not_depend_on_the_batch(kw):
    import cuda_pspin_b200 as ps
    out = []
    for others in (0, 1, 60):
        cfgs = [ps.default_config(seed=9, T=0.5, **kw)]
        cfgs += [ps.default_config(N=10 + k % 7, nrep=70, seed=100 + k, T=0.5) for k in range(others)]
        with ps.Engine(cfgs, ps.PSPIN_DENSE, ps.make_options()) as eng:
            R = kw["nrep"]
            e2, e4 = eng.split_energies()
            created = eng.get_results()[0][:R]
            eng.set_spins(eng.get_spins())
            out.append((e2[:R], e4[:R], created, eng.get_results()[0][:R]))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)
