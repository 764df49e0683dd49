"""The workloads this engine is measured on: what a user has it do, through its
public entry points, over the range of sizes, models, precisions and output
paths that are used in earnest.  Sizes follow the repository's own workloads
(the benchmark's dim 12, T 10,000 tables, the 100,000-run dim 2, T 1,000 table,
the ragged 60-pair batch, the smoke shape) and generic odd ones.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

from __graft_entry__ import load_package

jne = load_package()

PS = [0.01, 0.05, 0.1, 0.5, 0.9, 0.95, 0.99]  # the quantiles of the published tables


def listed():
    return [
        # the smoke shape: a handful of runs by the engine's default (FP64) precision, results in host memory;
        # one call's latency
        dict(name="smoke_fp64", kind="host", model=1, dim=3, steps=1000, runs=8, precision=0),
        # one small table (model 0, dim 2, T 1,000, 100,000 runs), results left on the device
        dict(name="table_dim2", kind="device", model=0, dim=2, steps=1000, runs=100_000, precision=1),
        # the headline table: dim 12, T 10,000, 200,000 runs of one model
        dict(name="table_dim12", kind="device", model=4, dim=12, steps=10_000, runs=200_000, precision=1),
        # an odd middle shape, results in host memory
        dict(name="odd_dim7_host", kind="host", model=3, dim=7, steps=2503, runs=30_011, precision=1),
        # the plain FP64 form of the headline table
        dict(name="fp64_dim12", kind="device", model=4, dim=12, steps=10_000, runs=10_000, precision=0),
        # an FP64 table of middle dim with an odd number of runs
        dict(name="fp64_dim5", kind="device", model=3, dim=5, steps=1000, runs=50_001, precision=0),
        # finite-sample critical values: paths of 100 observations (below the mixed kernel's shortest path)
        dict(name="short_paths", kind="host", model=2, dim=6, steps=100, runs=20_011, precision=1),
        # all five models of one (dim, T) in one pass over the paths, as the simulation driver runs them
        dict(name="five_models", kind="models", dim=12, steps=2000, runs=40_000, precision=1),
        # the ragged batch over all 60 (model, dim) pairs, captured once and replayed
        dict(name="ragged60_plan", kind="plan", pairs=60, mix=4, runs_lo=100, runs_hi=10_000),
        # eigenvalues of increments the caller brings (host matrices), FP64
        dict(name="increments_fp64", kind="increments", model=2, dim=4, steps=1000, runs=2000, precision=0),
        # critical values of a finished table: trace and largest-eigenvalue quantiles of 10^6 runs on the device
        dict(name="quantiles_1m", kind="quantiles", k=12, runs=1_000_000),
        # a simulation to its .dat file, then the file read back and its quantiles taken
        dict(name="simulation_file", kind="simulation", model=2, dim=5, steps=1000, runs=200_000, precision=1),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["host", "device", "device", "device", "models", "plan", "batch", "increments", "quantiles",
                       "simulation", "sink", "pack"])
    if kind in ("plan", "batch"):
        lo = _log_uniform(rng, 10, 300)
        return dict(kind=kind, pairs=rng.randint(2, 60), mix=rng.randint(1, 10**6), runs_lo=lo,
                    runs_hi=lo * rng.randint(2, 33))
    if kind == "quantiles":
        return dict(kind=kind, k=rng.randint(1, 13), runs=_log_uniform(rng, 10, 1_000_000))
    if kind == "pack":
        return dict(kind=kind, k=rng.randint(1, 13), runs=_log_uniform(rng, 10, 1_000_000),
                    seed_first=_log_uniform(rng, 1, 2**31))
    c = dict(kind=kind, dim=rng.randint(1, 12), precision=rng.choice([0, 1, 1]))
    if kind != "models":
        c["model"] = rng.randint(0, 4)
    c["steps"] = _log_uniform(rng, 40 if kind != "sink" else 256, 20_000)
    if rng.random() < 0.3:
        c["steps"] = rng.choice([100, 250, 500, 1000, 5000, 10_000])
    # 32-step tiles of path in all: at most those of the largest table of the precision
    tiles = (200_000 if c["precision"] == 1 and c["steps"] >= 256 else 5_000) * 313
    if kind in ("host", "simulation", "sink", "models"):
        tiles //= 4
    if kind == "increments":
        tiles = 1_000_000 // c["dim"]
    cap = max(2, min(300_000, tiles // ((c["steps"] + 31) // 32)))
    c["runs"] = _log_uniform(rng, min(cap, 8), cap)
    return c


def _requests(case, base_seed):
    """The requests of a ragged batch: (model, dim) pairs in order, T from {1000, 5000, 10000}, runs log-uniform."""
    rng = np.random.default_rng(case["mix"])
    every = [(m, d) for m in range(5) for d in range(1, 13)]
    if case["pairs"] < len(every):
        every = [every[i] for i in sorted(rng.choice(len(every), case["pairs"], replace=False))]
    return [dict(model=m, dim=d, steps=int(rng.choice([1000, 5000, 10_000])), base_seed=base_seed,
                 n_runs=int(np.exp(rng.uniform(np.log(case["runs_lo"]), np.log(case["runs_hi"]))))) for m, d in every]


def _device_eigs(k, runs, seed):
    """Descending positive rows, spread like the eigenvalues of a simulation."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    e = torch.rand((runs, k), generator=g, dtype=torch.float64, device="cuda")
    scale = torch.arange(1, k + 1, dtype=torch.float64, device="cuda")
    return torch.sort(-torch.log1p(-e) * scale, dim=1, descending=True).values.contiguous()


def _base_seed(seed):
    return (int(seed) * 0x9E3779B97F4A7C15 + 0x4A4F48) % 2**62


class _State:
    pass


def prepare(case, seed):
    s = _State()
    s.case, s.base, s.kind = case, _base_seed(seed), case["kind"]
    s.eng = jne.Engine(0)
    s.seed_first = 1 + int(seed) % 1000
    if s.kind == "device":
        s.out = torch.empty((case["runs"], jne.eigen_count(case["model"], case["dim"])), dtype=torch.float64,
                            device="cuda")
    elif s.kind in ("plan", "batch"):
        s.reqs = _requests(case, s.base)
        s.out = [torch.empty((r["n_runs"], jne.eigen_count(r["model"], r["dim"])), dtype=torch.float64, device="cuda")
                 for r in s.reqs]
        s.ptrs = [o.data_ptr() for o in s.out]
        if s.kind == "plan":
            s.plan = s.eng.plan(s.reqs, s.ptrs)
    elif s.kind == "increments":
        s.dB = _increments(case, seed)
    elif s.kind == "quantiles":
        s.eigs = _device_eigs(case["k"], case["runs"], seed)
    elif s.kind == "pack":
        s.eigs = _device_eigs(case["k"], case["runs"], seed)
        n = jne.record_bytes(case["seed_first"], case["runs"], case["k"])
        s.out = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    return s


def _increments(case, seed):
    rng = np.random.default_rng(int(seed))
    return rng.standard_normal((case["runs"], case["steps"], case["dim"])) / math.sqrt(case["steps"])


def run(s):
    c, eng = s.case, s.eng
    if s.kind == "host":
        return eng.eigs_seeded(c["model"], c["dim"], c["steps"], s.seed_first, c["runs"], precision=c["precision"],
                               base_seed=s.base)
    if s.kind == "device":
        eng.eigs_seeded_device(c["model"], c["dim"], c["steps"], s.seed_first, c["runs"], s.out.data_ptr(),
                               precision=c["precision"], base_seed=s.base)
        return s.out
    if s.kind == "models":
        outs = eng.eigs_seeded_models(range(5), c["dim"], c["steps"], s.seed_first, c["runs"],
                                      precision=c["precision"], base_seed=s.base)
        return [outs[m] for m in range(5)]
    if s.kind == "plan":
        s.plan.launch()
        return s.out
    if s.kind == "batch":
        eng.run_batch(s.reqs, s.ptrs)
        return s.out
    if s.kind == "increments":
        return eng.eigs_from_increments(c["model"], s.dB, precision=c["precision"])
    if s.kind == "quantiles":
        return [np.array(eng.percentiles_device(s.eigs.data_ptr(), c["runs"], c["k"], stat, PS))
                for stat in ("trace", "maxeig")]
    if s.kind == "pack":
        eng.pack_records_device(c["seed_first"], c["runs"], c["k"], s.eigs.data_ptr(), s.out.data_ptr(), s.out.numel())
        return s.out
    data_dir = tempfile.mkdtemp(prefix="jne_")
    try:
        if s.kind == "simulation":
            sim = jne.EigenvalueSimulation(c["model"], c["dim"], c["steps"], c["runs"], data_dir=data_dir,
                                           precision=c["precision"], base_seed=s.base, engine=eng)
            sim.run_simulation_quiet()
            rec = sim.read_data()
        else:  # "sink": a batch streamed into its simulation file, records packed on the GPU
            eng.run_batch_to_dat([dict(model=c["model"], dim=c["dim"], steps=c["steps"], n_runs=c["runs"],
                                       precision=c["precision"], base_seed=s.base)], data_dir)
            rec = jne.read_dat(os.path.join(data_dir, os.listdir(data_dir)[0]))[0]
    finally:
        shutil.rmtree(data_dir, ignore_errors=True)
    return [rec.seeds.astype(np.int64), rec.eigs, np.array(jne.percentiles(rec.eigs, "trace", PS)),
            np.array(jne.percentiles(rec.eigs, "maxeig", PS))]


def _gram_flops(model, dim, steps, runs):
    """The Gram contraction: k (k + 1) / 2 entries of S11 and k dim of S10, one multiply-add per step each."""
    k = dim + 1 if model in (1, 3) else dim
    return float(runs) * steps * k * (k + 1 + 2 * dim)


def work(case):
    kind = case["kind"]
    if kind == "quantiles":
        return {"bytes": 8.0 * case["k"] * case["runs"] + 16 * len(PS), "flops": 2.0 * case["k"] * case["runs"]}
    if kind == "pack":
        return {"bytes": 8.0 * case["k"] * case["runs"] + jne.record_bytes(case["seed_first"], case["runs"], case["k"]),
                "flops": 0.0}
    if kind in ("plan", "batch"):
        reqs = [(r["model"], r["dim"], r["steps"], r["n_runs"]) for r in _requests(case, 0)]
    elif kind == "models":
        reqs = [(m, case["dim"], case["steps"], case["runs"]) for m in range(5)]
    else:
        reqs = [(case["model"], case["dim"], case["steps"], case["runs"])]
    nbytes = sum(8.0 * n * jne.eigen_count(m, d) for m, d, _, n in reqs)
    if kind == "increments":
        nbytes += 8.0 * case["runs"] * case["steps"] * case["dim"]
    return {"bytes": nbytes, "flops": sum(_gram_flops(*r) for r in reqs)}


# ---- the same values in 64 bits, in plain torch ----
MOST_NORMALS = 5e9


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors that hold 32-bit words."""
    def mul(a, m):  # high and low words of a * m
        lo = (a & 0xFFFF) * m
        mid = (a >> 16) * m + (lo >> 16)
        return mid >> 16, ((mid & 0xFFFF) << 16) | (lo & 0xFFFF)

    for _ in range(10):
        h0, l0 = mul(c0, 0xD2511F53)
        h1, l1 = mul(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = h1 ^ c1 ^ k0, l1, h0 ^ c3 ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return c0, c1, c2, c3


def _normals(base_seed, dim, steps, seed_first, runs):
    """(runs, steps, dim) normals of the counter-based stream, the transform in 64 bits."""
    nq = (dim + 3) // 4
    dev = dict(dtype=torch.int64, device="cuda")
    shape = (runs, steps, nq)
    s = torch.arange(1, steps + 1, **dev).view(1, -1, 1).expand(shape)
    j = torch.arange(nq, **dev).view(1, 1, -1).expand(shape)
    seed = torch.arange(seed_first, seed_first + runs, **dev).view(-1, 1, 1).expand(shape)
    zero = torch.zeros((), **dev)
    w = _philox(s, j, seed, zero, base_seed & 0xFFFFFFFF, (base_seed >> 32) ^ (0x4A4E0000 | dim))
    z = []
    for a, b in ((w[0], w[1]), (w[2], w[3])):
        m, e = torch.frexp(a.double())  # the radius word's leading 24 bits
        u = torch.ldexp(torch.trunc(m * 2.0**24), e.double() - 24.0)
        u = ((u + 0.5) * 2.0**-32).float().double()
        r = torch.sqrt(-2.0 * torch.log(u))
        th = 2.0 * math.pi * (((b >> 9).double() + 0.5) * 2.0**-23) - math.pi
        z += [r * torch.cos(th), r * torch.sin(th)]
    return torch.stack(z, dim=3).reshape(runs, steps, 4 * nq)[:, :, :dim]


def _eigs(model, dB):
    """Eigenvalues of the pencil (S10' S10, S11) of each run, descending: the dense definition."""
    runs, steps, dim = dB.shape
    B = torch.zeros_like(dB)
    torch.cumsum(dB[:, :-1], dim=1, out=B[:, 1:]) if steps > 1 else None
    y = (torch.arange(1, steps + 1, dtype=torch.float64, device=dB.device) / steps).view(1, -1, 1).expand(runs, -1, 1)
    if model == 0:
        F = B
    elif model == 1:
        F = torch.cat([B, torch.ones_like(y)], dim=2)
    elif model in (2, 3):
        rows = B[:, :, : dim - 1] if model == 2 else B
        F = torch.cat([rows - rows.mean(dim=1, keepdim=True), y - 0.5], dim=2)
    else:
        F = torch.cat([B[:, :, : dim - 1], y * y], dim=2)
        X = torch.cat([torch.ones_like(y[:1]), y[:1] - y[:1].mean()], dim=2)[0]
        q, _ = torch.linalg.qr(X)
        F = F - q @ (q.T @ F)
    s11 = F.transpose(1, 2) @ F / steps
    s10 = dB.transpose(1, 2) @ F
    E = torch.linalg.solve_triangular(torch.linalg.cholesky(s11), s10.transpose(1, 2), upper=False)
    return torch.linalg.eigvalsh(E @ E.transpose(1, 2)).abs().sort(dim=1, descending=True).values


def _blocks(runs, steps, dim):
    per = max(1, int(3e7 // (steps * (dim + 3))))
    return [(a, min(per, runs - a)) for a in range(0, runs, per)]


def _exact_seeded(models, dim, steps, base_seed, seed_first, runs):
    got = {m: [] for m in models}
    for a, n in _blocks(runs, steps, dim):
        dB = _normals(base_seed, dim, steps, seed_first + a, n) / math.sqrt(steps)
        for m in models:
            got[m].append(_eigs(m, dB))
    return [torch.cat(got[m]) for m in models]


def _quantiles(v):
    """Linear interpolation at rank p (n - 1) of the sorted values."""
    v = np.sort(v)
    out = []
    for p in PS:
        rank = p * (len(v) - 1)
        lo, hi = math.floor(rank), math.ceil(rank)
        out.append(v[lo] if lo == hi else v[lo] * (1.0 - (rank - lo)) + v[hi] * (rank - lo))
    return np.array(out)


def exact(case, seed):
    kind, base, first = case["kind"], _base_seed(seed), 1 + int(seed) % 1000
    if kind == "pack":  # bytes, not computed numbers
        return None
    if kind == "quantiles":
        e = _device_eigs(case["k"], case["runs"], seed).cpu().numpy()
        return [_quantiles(e.sum(axis=1)), _quantiles(e.max(axis=1))]
    if kind in ("plan", "batch"):
        reqs = _requests(case, base)
        if sum(float(r["n_runs"]) * r["steps"] * r["dim"] for r in reqs) > MOST_NORMALS:
            return None
        return [_exact_seeded([r["model"]], r["dim"], r["steps"], base, 1, r["n_runs"])[0] for r in reqs]
    if float(case["runs"]) * case["steps"] * case["dim"] > MOST_NORMALS:
        return None
    shape = (case["dim"], case["steps"], base)
    if kind == "models":
        return [v.cpu().numpy() for v in _exact_seeded(range(5), *shape, first, case["runs"])]
    if kind == "device":
        return _exact_seeded([case["model"]], *shape, first, case["runs"])[0]
    if kind == "host":
        return _exact_seeded([case["model"]], *shape, first, case["runs"])[0].cpu().numpy()
    if kind == "increments":
        dB = torch.from_numpy(_increments(case, seed)).cuda()
        return torch.cat([_eigs(case["model"], dB[a:a + n]) for a, n in _blocks(*dB.shape)]).cpu().numpy()
    e = _exact_seeded([case["model"]], *shape, 1, case["runs"])[0].cpu().numpy()
    return [None, e, _quantiles(e.sum(axis=1)), _quantiles(e.max(axis=1))]
