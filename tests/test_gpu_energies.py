"""FP64 energies (pspin_split_energies): the run-factored table sum, cut over
several CTAs per replica block, against a direct FP64 evaluation of
mc.cu:323-405 on the same amplitudes and couplings.

Cases sit where the kernel changes path: one warp's worth of entries and many
CTAs per table, tables in q order (dense) and in selection order (sparse),
the channels' conjugations, ragged replica blocks, and amplitudes upcast in
shared memory (N <= 192) or at each use (above).  Bound: 40 roundings of
FP64 against the sum of |terms|.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CHANNELS = (((0, 1), (2, 3)), ((0, 3), (1, 2)), ((0, 2), (1, 3)))


def quartets(N):
    return np.array([(i, j, k, l) for l in range(3, N) for k in range(2, l) for j in range(1, k) for i in range(j)])


def e4_terms(a, q, ch, g):
    out = np.zeros((a.shape[0], len(q)))
    for c, (u, v) in enumerate(CHANNELS):
        m = ch == c
        z = a[:, q[m, u[0]]] * a[:, q[m, u[1]]] * np.conj(a[:, q[m, v[0]]] * a[:, q[m, v[1]]])
        out[:, m] = -z.real * g[m]
    return out


@pytest.mark.parametrize("N,R,fmc,sparse", [(5, 1, 0, False), (12, 33, 2, False), (24, 40, 1, False), (48, 70, 0, False),
                                            (16, 8, 0, True), (193, 5, 1, True), (260, 35, 1, True)])
def test_split_energies(N, R, fmc, sparse):
    import cuda_pspin_b200 as ps
    c = ps.default_config(N=N, nrep=R, seed=31 + N, fmc_mode=fmc)
    if fmc:
        c.gamma = 0.2 if fmc == 2 else 1.0
    with ps.Engine(c, ps.PSPIN_SPARSE if sparse else ps.PSPIN_DENSE, ps.make_options(disorder_stream=sparse)) as eng:
        e2, e4 = eng.split_energies()
        E = eng.get_results()[0]
        a = eng.get_spins()[0]
        g2, g4, mask = eng.couplings(0, dense_g4=not sparse)
        if sparse:
            rec, g = eng.sparse_quartets(0)
            q, ch = rec[:, :4], rec[:, 4]
        else:
            q, ch, g = quartets(N), np.zeros(0, int), g4
            keep = [(mask >> k) & 1 == 1 for k in range(3)]
            ch = np.concatenate([np.full(m.sum(), k) for k, m in enumerate(keep)])
            g = np.concatenate([g4[m] for m in keep])
            q = np.concatenate([q[m] for m in keep])
        i, j = np.triu_indices(N, 1)
        t2 = -(g2[i, j] * (a[:, i] * np.conj(a[:, j])).real)
        t4 = e4_terms(a, q, ch, g)
        if not eng.info(0).h2_active:
            t2[:] = 0.0
        tol = 40 * 2.3e-16
        assert np.all(np.abs(e2 - t2.sum(1)) <= tol * np.abs(t2).sum(1))
        assert np.all(np.abs(e4 - t4.sum(1)) <= tol * np.abs(t4).sum(1))
        assert np.array_equal(E, e2 + e4)
