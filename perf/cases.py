"""The work a user of the engine has it do, as measurable cases.

Every case goes through the package's public entry points the way the drivers
and the studies of this repository do: a parallel-tempering (PT) or plain
Monte Carlo run up to the next save point and the state that is written
there, the host-side exchange loop of the reference's driver pattern, the
FP64 energies, the learned proposal and its training, the set-up of a
sample, and the overlap analysis of saved configurations.

Block shapes (warps per CTA, CTAs per replica block, replicas per lane) are
given where a long run would keep the autotuner's pick, and left at 0 (the
engine's defaults, what the command-line drivers run with) elsewhere.  The
chain depends on the first two (they fix the summation order of the fields),
so they belong to the case.
"""
import math

import numpy as np
import torch

import cuda_pspin_b200 as ps
from cuda_pspin_b200 import analysis

GAMMA = 0.1                          # FMC width of the uniform-frequency configurations
TMIN, TMAX = 0.2, 1.6                # geometric temperature ladder of the configurations
MIX = (24, 32, 48, 64)               # sizes of the batched benchmark


def listed():
    return [
        # the smallest call: one small sample, the reference's driver loop (betas in, one
        # sweep, results out, exchange on the host) once; launches and copies count
        dict(name="host_loop_n16", kind="host_loop", N=16, samples=1, NT=4, nrep=2, fmc=0, steps=1,
             warps=0, cluster=0, lanes=0),
        # one sample, FMC uniform N=32, 20 temperatures x 4: a plain PT run to its next save point
        dict(name="pt_fmc_n32", kind="pt", N=32, samples=1, NT=20, nrep=4, fmc=2, sweeps=64,
             warps=4, cluster=8, lanes=1),
        # one sample, FMC uniform N=64, 24 x 4, with the drivers' default options
        dict(name="pt_fmc_n64_default", kind="pt", N=64, samples=1, NT=24, nrep=4, fmc=2, sweeps=32,
             warps=0, cluster=0, lanes=0),
        # one sparse sample, comb N=512, 32 x 4, lists resident in shared memory
        dict(name="pt_sparse_n512", kind="pt_sparse", N=512, samples=1, NT=32, nrep=4, fmc=1, sweeps=64,
             warps=8, cluster=-1, lanes=0),
        # plain Monte Carlo at one temperature, N=128 fully connected, 64 replicas
        dict(name="mc_fc_n128", kind="mc", N=128, samples=1, R=64, fmc=0, sweeps=2,
             warps=2, cluster=16, lanes=1),
        # many samples of one FMC size (the learned study's and the disorder averages' shape)
        dict(name="pt_fmc_n64_batch", kind="pt", N=64, samples=64, NT=24, nrep=4, fmc=2, sweeps=32,
             warps=8, cluster=4, lanes=3),
        # the batched benchmark: 256 fully connected samples of uneven N, 24 x 4
        dict(name="pt_fc_batch", kind="pt", N=0, samples=256, NT=24, nrep=4, fmc=0, sweeps=64,
             warps=8, cluster=2, lanes=3),
        # FP64 two- and four-body energies of a batch (energy_split.txt at every save point)
        dict(name="energies_fc_batch", kind="energies", N=0, samples=16, R=96, fmc=0, warps=0, cluster=0, lanes=0),
        # PT with the learned proposal
        dict(name="pt_learned_n64", kind="pt_learned", N=64, samples=8, NT=24, nrep=4, fmc=2, sweeps=4,
             warps=8, cluster=2, lanes=0),
        # training of the proposal network on recorded moves: forward, backward, Adam
        dict(name="learn_train", kind="train", N=16, samples=1, NT=8, nrep=4, fmc=0, steps=16, batch=4096,
             warps=0, cluster=0, lanes=0),
        # set-up of one sample: disorder, masks, site lists, amplitudes, energies
        dict(name="setup_fmc_n48", kind="setup", N=48, samples=1, R=96, fmc=2, warps=0, cluster=0, lanes=0),
        # overlap distributions of one run's saved configurations (host arrays)
        dict(name="analysis_n64", kind="analysis", N=64, NT=24, nrep=4, nsnap=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same kinds, sizes spread over their ranges."""
    kind = rng.choice(["host_loop", "pt", "pt", "pt_batch", "pt_batch", "pt_sparse", "mc", "energies", "pt_learned",
                       "train", "setup", "analysis"])
    NT, nrep = rng.randint(4, 24), rng.randint(2, 4)
    plain = rng.choice([(0, 0, 0), (8, 1, 1), (4, 2, 1), (4, 8, 1), (8, 4, 1), (8, 2, 3), (8, 4, 3), (8, 2, 2)])
    shape = dict(zip(("warps", "cluster", "lanes"), plain))
    if kind == "host_loop":
        return dict(kind=kind, N=rng.randint(12, 40), samples=_log_int(rng, 1, 16), NT=NT, nrep=nrep,
                    fmc=rng.choice([0, 2]), steps=rng.randint(1, 4), warps=0, cluster=0, lanes=0)
    if kind == "pt":
        return dict(kind=kind, N=rng.randint(20, 72), samples=1, NT=NT, nrep=nrep, fmc=rng.choice([0, 2]),
                    sweeps=rng.randint(8, 48), **shape)
    if kind == "pt_batch":
        batch = dict(zip(("warps", "cluster", "lanes"),
                         rng.choice([(0, 0, 0), (8, 1, 1), (4, 2, 1), (8, 2, 3), (8, 4, 3), (8, 2, 2)])))
        return dict(kind="pt", N=rng.choice([0, rng.randint(20, 64)]), samples=_log_int(rng, 4, 64), NT=NT, nrep=nrep,
                    fmc=rng.choice([0, 2]), sweeps=rng.randint(8, 32), **batch)
    if kind == "pt_sparse":
        return dict(kind=kind, N=rng.randint(96, 512), samples=_log_int(rng, 1, 8), NT=NT, nrep=nrep, fmc=1,
                    sweeps=rng.randint(8, 64), warps=rng.choice([1, 2, 4, 8]), cluster=-1, lanes=0)
    if kind == "mc":
        w, c = rng.choice([(2, 16), (4, 8), (8, 4), (0, 0)])
        return dict(kind=kind, N=rng.randint(64, 120), samples=1, R=rng.randint(16, 96), fmc=0,
                    sweeps=rng.randint(1, 4), warps=w, cluster=c, lanes=rng.choice([1, 2] if c else [0]))
    if kind == "energies":
        return dict(kind=kind, N=rng.choice([0, rng.randint(16, 64)]), samples=_log_int(rng, 1, 16),
                    R=rng.randint(8, 128), fmc=rng.choice([0, 2]), warps=0, cluster=0, lanes=0)
    if kind == "pt_learned":
        return dict(kind=kind, N=rng.randint(24, 56), samples=_log_int(rng, 1, 8), NT=NT, nrep=nrep,
                    fmc=rng.choice([0, 2]), sweeps=rng.randint(2, 4), warps=8, cluster=rng.choice([1, 2]), lanes=0)
    if kind == "train":
        return dict(kind=kind, N=rng.randint(12, 20), samples=1, NT=8, nrep=4, fmc=0,
                    steps=rng.randint(4, 32), batch=_log_int(rng, 512, 8192), warps=0, cluster=0, lanes=0)
    if kind == "setup":
        return dict(kind=kind, N=rng.randint(16, 56), samples=_log_int(rng, 1, 4), R=rng.randint(8, 96),
                    fmc=rng.choice([0, 2]), warps=0, cluster=0, lanes=0)
    return dict(kind="analysis", N=rng.randint(12, 96), NT=NT, nrep=nrep, nsnap=_log_int(rng, 4, 64))


def _sizes(case):
    if case["N"]:
        return [case["N"]] * case["samples"]
    return [MIX[(k * 2654435761 >> 7) % 4] for k in range(case["samples"])]


def _replicas(case):
    return case["R"] if "R" in case else case["NT"] * case["nrep"]


def _engine(case, seed, **options):
    variant = ps.PSPIN_SPARSE if case["kind"] == "pt_sparse" else ps.PSPIN_DENSE
    cfgs = []
    for k, N in enumerate(_sizes(case)):
        c = ps.default_config(N=N, nrep=_replicas(case), seed=1000 + 4096 * (seed % (1 << 28)) + k, fmc_mode=case["fmc"], T=0.5)
        if case["fmc"]:
            c.gamma = 1.0 if case["fmc"] == 1 else GAMMA
        cfgs.append(c)
    return ps.Engine(cfgs, variant, ps.make_options(warps_per_unit=case["warps"], cluster_size=case["cluster"],
                                                    replicas_per_lane=case["lanes"], **options))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "analysis":
        rng = np.random.default_rng(seed)
        # correlated replicas about a common configuration per temperature: overlaps of all sizes
        shape = (case["nsnap"], case["NT"], case["nrep"], case["N"], 2)
        common = rng.standard_normal((1, case["NT"], 1, case["N"], 2))
        mix = np.linspace(0.0, 0.95, case["NT"])[None, :, None, None, None]
        a = mix * common + np.sqrt(1.0 - mix ** 2) * rng.standard_normal(shape)
        s["configs"] = a * np.sqrt(case["N"] / (a ** 2).sum((-1, -2), keepdims=True))
        return s
    if kind == "setup":
        s["seed"] = seed
        return s
    s["eng"] = eng = _engine(case, seed, disorder_stream=kind == "pt_sparse")
    if kind == "mc":
        eng.fill_betas(2.0)
    elif kind == "energies":
        s["spins"] = eng.get_spins()
    else:
        _, betas = ps.temperature_schedule(case["NT"], TMIN, TMAX, True)
        eng.pt_init(case["NT"], case["nrep"], betas, 1)
        if kind == "host_loop":
            S, R, NT = case["samples"], _replicas(case), case["NT"]
            s["sched"] = betas
            s["betas"] = np.tile(np.repeat(betas, case["nrep"]), S)
            s["off"] = np.arange(S, dtype=np.int64) * R
            s["perm"] = np.tile(np.arange(R, dtype=np.int32), (S, 1))
            s["drand"] = np.array([((int(c.seed) + 5000 & 0xFFFFFFFF) << 16) | 0x330E for c in eng.cfgs], np.uint64)
            s["acc"], s["prop"] = np.zeros((S, NT - 1), np.int64), np.zeros((S, NT - 1), np.int64)
        elif kind in ("pt_learned", "train"):
            eng.learn_init(seed=1 + seed % 1000, capacity=1 << 16, record_prob=1.0)
            if kind == "train":
                eng.set_proposal(ps.PROPOSAL_PLAIN_FIELDS)
                eng.pt_run(64)             # one replica block: its moves enter the ring in order
                eng.set_proposal(ps.PROPOSAL_PLAIN)
            else:
                eng.set_proposal(ps.PROPOSAL_LEARNED)
    return s


def _state(eng):
    """What a save point writes: energies, counters, amplitudes (one array over all samples)."""
    E, acc, prop = eng.get_results()
    spins = eng.get_spins()
    return {"E": E, "accepted": acc, "proposed": prop,
            "spins": spins[0] if len(spins) == 1 else np.concatenate([a.reshape(-1) for a in spins])}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "analysis":
        pq = analysis.overlap_histograms(s["configs"])
        ifo, exp_ifo = analysis.ifo_histograms(s["configs"])
        return {"parisi": pq, "ifo": ifo, "exp_ifo": exp_ifo}
    if kind == "setup":
        with _engine(case, s["seed"]) as eng:
            out = [eng.couplings(k) for k in range(case["samples"])]
            return {"couplings": out, **_state(eng)}
    eng = s["eng"]
    if kind == "energies":
        eng.set_spins(s["spins"])
        e2, e4 = eng.split_energies()
        return {"e2": e2, "e4": e4, "E": eng.get_results()[0]}
    if kind == "train":
        loss = eng.learn_train(case["steps"], case["batch"], 1e-3)
        return {"loss": loss, "weights": eng.learn_params()}
    if kind == "host_loop":
        for _ in range(case["steps"]):
            eng.set_betas(s["betas"])
            eng.sweep(1)
            E, acc, prop = eng.get_results()
            ps.exchange_host(s["sched"], E, s["off"], s["perm"], s["drand"], s["acc"], s["prop"], s["betas"])
        return {"E": E, "accepted": acc, "proposed": prop, "perm": s["perm"].copy(), "betas": s["betas"].copy(),
                "ex_acc": s["acc"].copy(), "spins": np.concatenate([a.reshape(-1) for a in eng.get_spins()])}
    if kind == "mc":
        eng.sweep(case["sweeps"])
        return _state(eng)
    eng.pt_run(case["sweeps"])
    pt = [eng.pt_get(k) for k in range(case["samples"])]
    return {"perm": np.stack([p[0] for p in pt]), "ex_acc": np.stack([p[1] for p in pt]), **_state(eng)}


def _c4(N):
    return N * (N - 1) * (N - 2) * (N - 3) // 24


def _quartets(case, N):
    """Active (quartet, channel) pairs of one sample (expected, for the FMC ones)."""
    if case["kind"] == "pt_sparse":
        return N
    return _c4(N) * (0.34 if case["fmc"] == 2 else 1.0)


def work(case):
    kind = case["kind"]
    if kind == "analysis":
        n = case["nsnap"] * case["NT"] * case["nrep"] * case["N"]
        return {"bytes": 16.0 * n, "flops": 2.0 * n * (4 + 4 * (case["nrep"] - 1))}
    if kind == "train":
        # 6426 weights, three products of the network per record and step; the records are read each step
        return {"bytes": 44.0 * case["batch"] * case["steps"] + 8.0 * 6426 * case["steps"],
                "flops": 6.0 * 6400 * case["batch"] * case["steps"]}
    R, by, fl = _replicas(case), 0.0, 0.0
    for N in _sizes(case):
        q = _quartets(case, N)
        state = 8.0 * N * R + 24.0 * R
        if kind == "setup":
            by += 9.0 * _c4(N) + 16.0 * 4 * q + 16.0 * N * R
            fl += 20.0 * q * R
        elif kind == "energies":
            by += 8.0 * q + 2 * state
            fl += 20.0 * q * R                     # one product of four amplitudes per quartet and replica
        else:
            sweeps = case["steps"] if kind == "host_loop" else case["sweeps"]
            terms = (N // 2) * 2 * (4.0 * q / N)   # field terms of the moves' two sites, per replica and sweep
            by += 4.0 * 4 * q + 2 * state          # every coupling of the site lists once, the state in and out
            fl += sweeps * R * (4.0 * terms + 64.0 * (N // 2)) * (2 if kind == "pt_learned" else 1)
    return {"bytes": by, "flops": fl}


def exact(case, seed):
    """The FP64 energies from the couplings and amplitudes; chains, trained weights and counts
    have no value that is not their own."""
    if case["kind"] == "energies":
        with _engine(case, seed) as eng:           # the disorder and the amplitudes: the case's inputs
            spins = eng.get_spins()
            inputs = [eng.couplings(k) for k in range(case["samples"])]
        e2, e4 = [], []
        for a, (g2, g4, mask) in zip(spins, inputs):
            N = a.shape[1]
            a = torch.from_numpy(a.astype(np.complex64).astype(np.complex128)).cuda()
            g2 = torch.from_numpy(np.triu(g2, 1)).cuda().to(torch.complex128)
            e2.append(-((a @ g2) * a.conj()).sum(1).real)
            total = torch.zeros(len(a), dtype=torch.float64, device="cuda")
            k4 = torch.combinations(torch.arange(N), 4)
            key = k4[:, 3] * (k4[:, 3] - 1) * (k4[:, 3] - 2) * (k4[:, 3] - 3) // 24 + \
                k4[:, 2] * (k4[:, 2] - 1) * (k4[:, 2] - 2) // 6 + k4[:, 1] * (k4[:, 1] - 1) // 2 + k4[:, 0]
            k4 = k4[torch.argsort(key)].cuda()
            g4, mask = torch.from_numpy(g4).cuda(), torch.from_numpy(mask).cuda()
            for ch, (u, c) in enumerate((((0, 1), (2, 3)), ((0, 3), (1, 2)), ((0, 2), (1, 3)))):
                at = torch.nonzero(mask & (1 << ch)).flatten()
                for part in at.split(1 << 16):
                    q = k4[part]
                    z = a[:, q[:, u[0]]] * a[:, q[:, u[1]]] * (a[:, q[:, c[0]]] * a[:, q[:, c[1]]]).conj()
                    total -= z.real @ g4[part]
            e4.append(total)
        e2, e4 = torch.cat(e2).cpu().numpy(), torch.cat(e4).cpu().numpy()
        return {"e2": e2, "e4": e4, "E": e2 + e4}
    return None
