"""Device scratch of the overlap analysis: calls of several threads, of sizes
below and above what the pool keeps between calls, give the serial counts; and
the engine's configurations read back exactly as they were set.
"""
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_calls_of_several_threads():
    from cuda_pspin_b200 import analysis
    rng = np.random.default_rng(3)
    sizes = [(1, 2, 2, 5), (4, 3, 2, 16), (30, 24, 4, 96), (3, 2, 3, 64)]     # snapshots, temperatures, replicas, sites
    data = [rng.standard_normal((s, t, r, n, 2)) for s, t, r, n in sizes]
    serial = [(analysis.overlap_histograms(d), analysis.ifo_histograms(d)) for d in data]
    with ThreadPoolExecutor(4) as pool:
        again = list(pool.map(lambda d: (analysis.overlap_histograms(d), analysis.ifo_histograms(d)), data * 3))

    def flat(x):
        return np.concatenate([np.ravel(np.asarray(v, float)) for v in _leaves(x)])

    for k, got in enumerate(again):
        assert np.array_equal(flat(got), flat(serial[k % len(data)]), equal_nan=True)


def _leaves(x):
    if isinstance(x, (tuple, list)):
        for v in x:
            yield from _leaves(v)
    elif isinstance(x, dict):
        for v in x.values():
            yield from _leaves(v)
    elif x is not None:
        yield x


def test_configurations_read_back():
    import cuda_pspin_b200 as ps
    rng = np.random.default_rng(4)
    cfgs = [ps.default_config(N=n, nrep=r, seed=9 + n) for n, r in ((8, 3), (11, 5))]
    with ps.Engine(cfgs) as eng:
        want = [(rng.standard_normal((r, n)).astype(np.float32) + 1j * rng.standard_normal((r, n)).astype(np.float32))
                .astype(np.complex64).astype(np.complex128) for n, r in ((8, 3), (11, 5))]
        eng.set_spins(want)
        got = eng.get_spins()
    for g, w in zip(got, want):
        assert g.dtype == np.complex128 and g.flags.c_contiguous and g.flags.writeable
        assert np.array_equal(g, w)
