"""Performance cases: the work a user of this framework has it do, through the
binding's public classes (Job, Batch, SpJob, SpBatch of eagb.py).

Three kinds of work:

  "sp"     a sample-packed job (64 samples per word, any L): one bin of the
           cadence, then what a run keeps of it -- the average energies, the
           tempering state and, where the bin ends with a checkpoint, the spins;
  "ms"     a job in the reference's multispin layout (L, Lz multiples of 8):
           the same with the temperature history, every bin with a checkpoint;
  "spbatch", "msbatch"   many jobs of different tubes advanced together;
  "corr"   the correlation functions of the plane overlaps of a configuration.

A bin moves its job on, as in a run: the same state can be run again and again.
"""
import importlib.util
import os
import random

import numpy as np

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
_spec = importlib.util.spec_from_file_location("eagb", os.path.join(ROOT, "ea-lcd-mc_gb300", "eagb.py"))
eagb = importlib.util.module_from_spec(_spec)
_spec.loader.exec_module(eagb)

PBC, OBC = 0, 1
# operations of the update: 32-bit operations of one random triple (six Philox
# calls, 24 threshold searches) and of one updated spin word
OPS_TRIPLE, OPS_WORD = 6 * 100 + 24 * 6, 60


def listed():
    return [
        # the smallest job: a cube-section tube of 864 sites, tempering every
        # sweep, no cluster moves -- a chain of short launches
        {"name": "sp_L6", "kind": "sp", "L": 6, "Lz": 24, "bc": PBC, "nt": 12, "nrep": 2, "nwords": 1,
         "itmax": 64, "houfr": 1, "cluster": False, "spins": True},
        # odd sizes in everything: odd L and Lz (three colours), an odd number
        # of temperatures and of replicas, moves every 8 sweeps
        {"name": "sp_L7_odd", "kind": "sp", "L": 7, "Lz": 21, "bc": PBC, "nt": 13, "nrep": 3, "nwords": 3,
         "itmax": 4, "houfr": 8, "cluster": True, "spins": True},
        # an ordinary production job: 64 samples of a 12 x 12 x 48 tube with a
        # cluster move every 10 sweeps
        {"name": "sp_L12", "kind": "sp", "L": 12, "Lz": 48, "bc": OBC, "nt": 24, "nrep": 4, "nwords": 1,
         "itmax": 10, "houfr": 10, "cluster": True, "spins": True},
        # the same tube for 4096 samples: the wide job of a disorder average
        {"name": "sp_L12_4096", "kind": "sp", "L": 12, "Lz": 48, "bc": OBC, "nt": 24, "nrep": 4, "nwords": 64,
         "itmax": 10, "houfr": 10, "cluster": True, "spins": False},
        # the large tube, 64 samples, a move every 5 sweeps
        {"name": "sp_L24", "kind": "sp", "L": 24, "Lz": 192, "bc": OBC, "nt": 32, "nrep": 4, "nwords": 1,
         "itmax": 10, "houfr": 5, "cluster": True, "spins": True},
        # many small tubes of different shapes at once (a serving mix)
        {"name": "sp_batch", "kind": "spbatch", "Ls": "8,10,12", "ratios": "2,4", "nts": "16,24", "nrep": 2,
         "nwords": 1, "itmax": 4, "houfr": 10, "cluster": True},
        # the smallest multispin job: two samples of an 8 x 8 x 16 tube
        {"name": "ms_L8", "kind": "ms", "L": 8, "Lz": 16, "bc": PBC, "nt": 8, "nrep": 4, "ns": 2,
         "itmax": 20, "houfr": 4, "cluster": True},
        # an ordinary multispin job with cluster moves
        {"name": "ms_L16", "kind": "ms", "L": 16, "Lz": 64, "bc": OBC, "nt": 24, "nrep": 4, "ns": 8,
         "itmax": 10, "houfr": 10, "cluster": True},
        # sweeps and tempering alone, the shipped set of 40 temperatures
        {"name": "ms_L16_nocluster", "kind": "ms", "L": 16, "Lz": 48, "bc": OBC, "nt": 40, "nrep": 8, "ns": 16,
         "itmax": 50, "houfr": 1, "cluster": False},
        # the large tube as one reference process takes it: 31 samples, 8
        # replicas, a move every 5 sweeps
        {"name": "ms_L24", "kind": "ms", "L": 24, "Lz": 192, "bc": OBC, "nt": 32, "nrep": 8, "ns": 31,
         "itmax": 100, "houfr": 5, "cluster": True},
        # 36 multispin jobs of different tubes in one batch, four samples each
        {"name": "ms_batch", "kind": "msbatch", "Ls": "8,16", "ratios": "2,4,8", "nts": "16,24,32", "nrep": 4,
         "ns": 4, "itmax": 2, "houfr": 10, "cluster": True},
        # analysis of a configuration: correlation functions at every distance
        {"name": "corr_L12", "kind": "corr", "L": 12, "Lz": 48, "bc": OBC, "nt": 24, "nrep": 4, "nwords": 1, "r": 4,
         "dmax": 47},
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def _sweeps(rng, spins, houfr, low, high):
    """Iterations of a bin worth low..high spin updates."""
    return max(1, min(64, int(low * (high / low) ** rng.random() / (spins * houfr))))


def draw(rng):
    kind = rng.choice(["sp", "sp", "sp", "ms", "ms", "ms", "spbatch", "msbatch", "corr"])
    if kind == "sp":
        while True:
            L = rng.randint(4, 24)
            Lz = min(192, max(4, _log_int(rng, L, 8 * L)))
            nt, nrep = rng.randint(5, 32), rng.choice([2, 2, 3, 4, 4, 5, 6])
            nwords = rng.choice([1, 1, 1, 2, 3]) if rng.random() < 0.6 else _log_int(rng, 2, 64)
            words = L * L * Lz * nt * nrep * nwords
            if words <= 15e6:
                break
        cluster = rng.random() < 0.75
        houfr = rng.randint(4, 12) if cluster else 1
        return {"kind": "sp", "L": L, "Lz": Lz, "bc": rng.choice([PBC, OBC]), "nt": nt, "nrep": nrep,
                "nwords": nwords, "itmax": _sweeps(rng, 64 * words, houfr, 2e8, 1.2e10), "houfr": houfr,
                "cluster": cluster, "spins": nwords <= 4}
    if kind == "ms":
        while True:
            L = rng.choice([8, 8, 16, 16, 24])
            Lz = 8 * _log_int(rng, 1, 24)
            nt, nrep, ns = rng.randint(5, 32), rng.choice([2, 4, 4, 8]), rng.randint(1, 31)
            spins = L * L * Lz * nt * nrep * ns
            if spins <= 4e8:
                break
        cluster = nrep >= 4 and rng.random() < 0.75
        houfr = rng.randint(2, 10) if cluster else 1
        return {"kind": "ms", "L": L, "Lz": Lz, "bc": rng.choice([PBC, OBC]), "nt": nt, "nrep": nrep, "ns": ns,
                "itmax": _sweeps(rng, spins, houfr, 2e8, 1e10), "houfr": houfr, "cluster": cluster}
    if kind == "spbatch":
        Ls = sorted(rng.sample(range(5, 15), rng.randint(2, 3)))
        return {"kind": kind, "Ls": ",".join(map(str, Ls)), "ratios": rng.choice(["1,2", "2,3", "2,4", "3", "4"]),
                "nts": ",".join(map(str, sorted(rng.sample(range(8, 25), 2)))), "nrep": rng.choice([2, 3, 4]),
                "nwords": rng.randint(1, 2), "itmax": rng.randint(1, 2), "houfr": rng.randint(5, 10),
                "cluster": rng.random() < 0.8}
    if kind == "msbatch":
        return {"kind": kind, "Ls": rng.choice(["8", "8,16", "16"]), "ratios": rng.choice(["1,2", "2,4", "3,5", "4"]),
                "nts": ",".join(map(str, sorted(rng.sample(range(8, 33), 2)))), "nrep": rng.choice([4, 8]),
                "ns": rng.randint(1, 6), "itmax": 1, "houfr": rng.randint(3, 10), "cluster": rng.random() < 0.8}
    L, nrep = rng.randint(4, 16), rng.choice([2, 4, 5, 6, 8])
    Lz = _log_int(rng, 8, 96)
    return {"kind": "corr", "L": L, "Lz": Lz, "bc": rng.choice([PBC, OBC]), "nt": rng.randint(5, 24), "nrep": nrep,
            "nwords": rng.randint(1, 3), "r": 2 * rng.randint(1, nrep // 2), "dmax": rng.randint(Lz // 2, Lz - 1)}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _temperatures(nt):
    """betas and thresholds of nt temperatures: a shipped set of that size, or
    nt temperatures spread over the 32 of the [0.7, 1.6] set."""
    golden = os.path.join(ROOT, "tests", "golden")
    if nt == 40:
        d = np.load(os.path.join(golden, "lut_shipped_N40.npz"))
        return d["betas"], d["cum"]
    d = np.load(os.path.join(golden, "lut_T07_16_N32.npz"))
    k = np.round(np.linspace(0, 31, nt)).astype(int)
    return d["betas"][k], d["cum"][k]


def _ints(text):
    return [int(x) for x in text.split(",")]


def _masters(rng):
    return tuple(rng.getrandbits(63) | 1 for _ in range(4))


def _sp_job(c, rng, jobid=0):
    betas, cum = _temperatures(c["nt"])
    return eagb.SpJob(c["L"], c["Lz"], betas, cum, nrep=c["nrep"], nwords=c["nwords"], bc=c["bc"],
                      seeds=_masters(rng), jobid=jobid)


def _ms_job(c, rng, jobid=0, alone=True):
    """A multispin job whose generators and couplings are those of a new run;
    the spin words of the start are random, as a new run's are."""
    betas, cum = _temperatures(c["nt"])
    g = eagb.geom(c["L"], c["Lz"], c["nt"], c["nrep"], c["ns"], c["bc"])
    job = eagb.Job(g)
    if not alone:
        job.set_rng_sms(0)   # the jobs of a batch share every SM
    job.set_temperatures(betas, cum)
    m = _masters(rng)
    sJ, _, sMC = eagb.host_seeds(m, c["ns"], c["nrep"])
    gen, pt = eagb.host_generators(sMC, c["ns"], m[3])
    job.set_generators(gen, pt)
    nrng = np.random.default_rng(rng.getrandbits(63))
    n = c["nt"] * job.half * c["nrep"]
    for s in range(c["ns"]):
        job.set_spins(s, nrng.integers(0, 1 << 64, n, np.uint64), nrng.integers(0, 1 << 64, n, np.uint64))
        job.set_couplings(s, eagb.host_init_couplings(g, int(sJ[s]))[1])
    job.set_permutations(None)
    job.set_counter(0, jobid)
    return job


def _corr_spins(c, seed):
    """Configurations as a run leaves them: replicas that agree more and more
    from the hottest slot (last) to the coldest (first)."""
    rng = np.random.default_rng(seed)
    V, nt = c["L"] * c["L"] * c["Lz"], c["nt"]
    base = rng.integers(0, 1 << 64, (c["nwords"], V, 1, 1), np.uint64)
    shape = (c["nwords"], V, c["nrep"], nt)
    noise = rng.integers(0, 1 << 64, shape, np.uint64)
    for k in range(1, 4):   # a spin differs with probability 1/2, 1/4, 1/8, 1/16
        cold = nt - (k * nt) // 4
        noise[..., :cold] &= rng.integers(0, 1 << 64, shape[:3] + (cold,), np.uint64)
    return base ^ noise


class State:
    def __init__(self, case):
        self.case, self.jobs, self.batch = case, [], None
        self.cad = dict(itmax=case.get("itmax", 1), houfr=case.get("houfr", 1), mesfr=1, ptfr=1,
                        cluster=case.get("cluster", False))

    def __del__(self):
        if self.batch is not None:
            self.batch.close()
        for j in self.jobs:
            j.close()


def _shapes(case):
    return [dict(case, L=L, Lz=r * L, bc=bc, nt=nt) for L in _ints(case["Ls"]) for r in _ints(case["ratios"])
            for bc in (PBC, OBC) for nt in _ints(case["nts"])]


def prepare(case, seed):
    s = State(case)
    rng = random.Random(seed)
    kind = case["kind"]
    if kind == "sp":
        s.jobs = [_sp_job(case, rng)]
    elif kind == "ms":
        s.jobs = [_ms_job(case, rng)]
    elif kind == "spbatch":
        s.jobs = [_sp_job(c, rng, k) for k, c in enumerate(_shapes(case))]
        s.batch = eagb.SpBatch(s.jobs)
    elif kind == "msbatch":
        s.jobs = [_ms_job(c, rng, k, alone=False) for k, c in enumerate(_shapes(case))]
        s.batch = eagb.Batch(s.jobs)
    else:
        s.jobs = [_sp_job(case, rng)]
        s.jobs[0].set_spins(_corr_spins(case, seed))
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def _ms_spins(job):
    return [x.view(np.int64) for smp in range(job.g.nsamples) for x in job.get_spins(smp)]


def run(s):
    kind = s.case["kind"]
    if kind == "sp":
        job = s.jobs[0]
        out = {"avg": job.run_bin(**s.cad)}
        E, perm, acc, M = job.tempering()
        out.update(E=E, perm=perm, acc=acc.view(np.int32), swaps=M.view(np.int64))
        if s.case["spins"]:
            out["spins"] = job.get_spins().view(np.int64)
        return out
    if kind == "ms":
        job = s.jobs[0]
        avg, hist = job.run_bin(**s.cad)
        return {"avg": avg, "hist": hist, "spins": _ms_spins(job)}
    if kind == "spbatch":
        s.batch.run_bin(**s.cad)
        return {"avg": np.concatenate([j.bin_results().reshape(-1) for j in s.jobs]),
                "E": np.concatenate([j.tempering()[0].reshape(-1) for j in s.jobs]),
                "spins": np.concatenate([j.get_spins().reshape(-1) for j in s.jobs]).view(np.int64)}
    if kind == "msbatch":
        s.batch.run_bin(**s.cad)
        got = [j.bin_results() for j in s.jobs]
        return {"avg": np.concatenate([a.reshape(-1) for a, _ in got]),
                "hist": np.concatenate([h.reshape(-1) for _, h in got]),
                "spins": np.concatenate([w for j in s.jobs for w in _ms_spins(j)])}
    return s.jobs[0].plane_correlations(s.case["r"], s.case["dmax"])


def work(case):
    """Each spin word read and written once a bin, the couplings and thresholds
    read once, the results written; operations of the updates (random triples
    are shared by the words, or the samples, of a job)."""
    kind = case["kind"]
    if kind == "corr":
        n = case["L"] ** 2 * case["Lz"] * case["r"] * case["nt"] * case["nwords"]
        c = 64 * case["nwords"] * case["nt"] * (case["dmax"] + 1)
        return {"bytes": 8.0 * n + 72.0 * c, "flops": 2.0 * n + 18.0 * c * case["Lz"] * (case["r"] // 2)}
    total = {"bytes": 0.0, "flops": 0.0}
    for c in _shapes(case) if "batch" in kind else [case]:
        V, G = c["L"] ** 2 * c["Lz"], c["nrep"] * c["nt"]
        sweeps = c["itmax"] * c["houfr"]
        if kind.startswith("sp"):
            words, triples, J = V * G * c["nwords"], V * G, 48.0 * V * c["nwords"]
            outs = 64 * G * c["nwords"] * 18
        else:
            words, triples, J = V // 64 * G * c["ns"], V // 64 * G, 0.75 * V * c["ns"]
            outs = G * c["ns"] * 26
        total["bytes"] += 16.0 * words + J + 2048.0 * c["nt"] + outs
        total["flops"] += float(sweeps) * (triples * OPS_TRIPLE + words * OPS_WORD)
    return total


def exact(case, seed):
    """The correlation functions in 64 bits from the same spins; a simulation
    of many sweeps has no other value than its own."""
    if case["kind"] != "corr":
        return None
    L, Lz, r, nw, nt = case["L"], case["Lz"], case["r"], case["nwords"], case["nt"]
    S = _corr_spins(case, seed).reshape(nw, Lz, L * L, case["nrep"], nt)
    q = np.empty((nw, 64, r // 2, nt, Lz))
    for k in range(r // 2):
        x = S[:, :, :, 2 * k] ^ S[:, :, :, 2 * k + 1]                       # [nw][Lz][L^2][nt]
        for b in range(64):
            n = ((x >> np.uint64(b)) & np.uint64(1)).sum(axis=2, dtype=np.int64)   # [nw][Lz][nt]
            q[:, b, k] = 1.0 - 2.0 * n.transpose(0, 2, 1) / (L * L)
    f = np.stack([q, q ** 3, np.sign(q)], -1)                              # [nw][64][pair][nt][Lz][3]
    C = np.empty((nw * 64, nt, case["dmax"] + 1, 3, 3))
    for d in range(case["dmax"] + 1):
        a, b = (f, np.roll(f, -d, axis=4)) if case["bc"] == PBC else (f[..., :Lz - d, :], f[..., d:, :])
        C[:, :, d] = np.einsum("wskbzp,wskbzq->wsbpq", a, b).reshape(nw * 64, nt, 3, 3) / (r // 2 * a.shape[4])
    return C
