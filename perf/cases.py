"""Performance cases of the ALTO library, through its public entry points.

Each case is one thing a user's program has the library do over and over:
MTTKRPs of a tensor it has encoded (AltoTensor.mttkrp), building a tensor
and using it once (create_alto), CP-ALS (cpd_alto), pushing time slices into
a CP-stream session (CPStream.push), serving many streams at once (Server)
and cutting a tensor into time slices (Slicer).  Inputs are power-law or
uniform coordinates with the value distributions of the benchmark
workloads, made on the GPU from a seed.

listed() are fixed points of the ranges, draw() gives others; prepare()
makes what a program holds before the call, run() is one pass, exact() the
same result in float64 without this library, work() the bytes and
operations no implementation can avoid.

The library keeps factors in float32 on the device and hands some of them
out as float64 arrays; such outputs are returned rounded back to float32,
the precision they have.
"""
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "alto-stream_b200"))

import alto_b200 as A  # noqa: E402
from alto_b200 import synth  # noqa: E402


def listed():
    return [
        # The smallest call: a toy tensor's MTTKRP of every mode; launches and latency.
        dict(name="mttkrp-tiny", kind="mttkrp", dims="300x400x500", nnz=20000, rank=16, zipf="0,0,0", dtype="f32"),
        # The plain CP-ALS configuration's tensor (1000^3, 1M uniform nonzeros), its MTTKRP alone.
        dict(name="mttkrp-cube-1m", kind="mttkrp", dims="1000x1000x1000", nnz=1000000, rank=16, zipf="0,0,0",
             dtype="f32"),
        # A ragged four-mode tensor at a rank chosen at run time (no specialised kernel).
        dict(name="mttkrp-ragged-r10", kind="mttkrp", dims="40009x13007x1031x61", nnz=3000017, rank=10,
             zipf="1.1,1.1,0,0", dtype="f32"),
        # The headline: the power-law three-mode shape with a 65-bit key at rank 32, at 40M nonzeros.
        dict(name="mttkrp-power-40m", kind="mttkrp", dims="4800000x1800000x1800000", nnz=40000000, rank=32,
             zipf="1.2,1.2,1.2", dtype="f32"),
        # The five-mode shape at rank 64 with bfloat16 factor storage.
        dict(name="mttkrp-five-bf16", kind="mttkrp", dims="100000x100000x10000x1000x100", nnz=12000000, rank=64,
             zipf="1.1,1.1,0,0,0", dtype="bf16"),
        # A tensor that is built, used once per mode and dropped: encoding and the first (untuned) MTTKRPs.
        dict(name="build-8m", kind="build", dims="1200000x450000x450000", nnz=8000000, rank=16, zipf="1.2,1.2,1.2"),
        # Plain CP-ALS: 1000^3, 1M nonzeros, rank 16, twenty iterations.
        dict(name="cpals-cube-1m", kind="cpals", dims="1000x1000x1000", nnz=1000000, rank=16, zipf="0,0,0",
             iters=20, dtype="f32"),
        # CP-ALS at rank 64 on a five-mode power-law tensor, float32 storage.
        dict(name="cpals-five-r64", kind="cpals", dims="20000x20000x5000x1000x100", nnz=5000000, rank=64,
             zipf="1.1,1.1,0,0,0", iters=8, dtype="f32"),
        # CP-stream with a non-negativity ADMM constraint at rank 16: host slices of the streaming configuration.
        dict(name="stream-nonneg-r16", kind="stream", dims="100000x100000x10000", nnz=200000, rank=16,
             zipf="1.1,1.1,1.1", nonneg=True, device=False, inner=10, slices=4),
        # CP-stream unconstrained at rank 32 on long modes: slices that are already on the device.
        dict(name="stream-free-r32", kind="stream", dims="120011x30011x9001", nnz=400009, rank=32,
             zipf="1.1,1.1,1.1", nonneg=False, device=True, inner=10, slices=5),
        # Serving: twelve independent streams of mixed ranks, constraints and sizes, their slices arriving together.
        dict(name="serve-12", kind="serve", streams=12, lo=1000, hi=30000, nnz=50000, inner=10, slices=3),
        # The stream slicer over a whole four-mode tensor of 200 time steps, cut into batches of steps.
        dict(name="slicer-10m", kind="slicer", dims="200x100000x100000x10000", nnz=10000000, zipf="0,1.1,1.1,1.1",
             steps=4),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["mttkrp", "mttkrp", "mttkrp", "build", "cpals", "stream", "stream", "serve", "slicer"])
    if kind == "serve":
        return dict(kind=kind, streams=rng.randint(4, 12), lo=1000, hi=_log(rng, 4000, 30000),
                    nnz=_log(rng, 10000, 50000), inner=rng.choice([5, 10]), slices=3)
    if kind == "stream":
        dims = [_log(rng, 5000, 120000), _log(rng, 2000, 100000), _log(rng, 1000, 10000)]
        return dict(kind=kind, dims=_x(dims), nnz=_log(rng, 20000, 400000), rank=rng.choice([8, 16, 32]),
                    zipf="1.1,1.1,1.1", nonneg=rng.random() < 0.5, device=rng.random() < 0.5,
                    inner=rng.choice([5, 10]), slices=4)
    if kind == "slicer":
        dims = [_log(rng, 50, 300), _log(rng, 5000, 100000), _log(rng, 5000, 100000), _log(rng, 1000, 10000)]
        return dict(kind=kind, dims=_x(dims), nnz=_log(rng, 300000, 10000000), zipf="0,1.1,1.1,1.1",
                    steps=rng.randint(3, 6))
    n = rng.choice([3, 3, 4, 5])
    tops = {3: (3000000, 1200000, 1200000), 4: (100000, 40000, 5000, 300), 5: (60000, 60000, 8000, 1000, 100)}[n]
    dims = [_log(rng, max(20, t // 100), t) for t in tops]
    zipf = rng.choice([("1.1", "1.1", "0", "0", "0"), ("0", "0", "0", "0", "0")])[:n] if n > 3 else \
        rng.choice([("1.2", "1.2", "1.2"), ("0", "0", "0")])
    space = 1.0
    for d in dims:
        space *= d
    most = min(20000000, space / 50)
    if kind == "cpals":
        return dict(kind=kind, dims=_x([min(d, 5000) for d in dims]),
                    nnz=_log(rng, 200000, min(3000000, max(most, 400000))), rank=rng.choice([8, 16, 32, 64]), zipf=",".join(zipf), iters=rng.randint(4, 10),
                    dtype=rng.choice(["f32", "bf16"]))
    if kind == "build":
        return dict(kind=kind, dims=_x(dims), nnz=_log(rng, 50000, min(8000000, most)),
                    rank=rng.choice([8, 16, 32]), zipf=",".join(zipf))
    return dict(kind=kind, dims=_x(dims), nnz=_log(rng, 20000, most), rank=rng.choice([8, 10, 16, 24, 32, 64]),
                zipf=",".join(zipf), dtype=rng.choice(["f32", "f32", "bf16"]))


# ------------------------------------------------------------------ inputs

def _x(dims):
    return "x".join(str(d) for d in dims)


def _dims(case):
    return [int(d) for d in case["dims"].split("x")]


def _draw(dims, nnz, zipf, seed):
    """nnz distinct coordinates (int64 [N, nnz], random order) and their generator.

    A mode of exponent s > 0 draws ranks from the power law x^-s over its
    length (the continuous law's inverse, cut to whole ranks) and spreads
    them over the labels by a multiplication modulo the length; 0 is uniform.
    Every step gives the same result each time it runs."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    keys = torch.empty(0, dtype=torch.int64, device="cuda")
    for _ in range(64):
        key = 0
        for m, (d, z) in enumerate(zip(dims, zipf)):
            x = torch.rand(nnz + 1024, generator=g, device="cuda", dtype=torch.float64)
            if z:
                r = ((x * ((d + 1.0) ** (1 - z) - 1) + 1) ** (1 / (1 - z))).long().clamp_(1, d) - 1
                step = 2654435761 + 2 * m
                while np.gcd(step, d) != 1:
                    step += 1
                x = (r * step + seed) % d
            else:
                x = (x * d).long().clamp_(max=d - 1)
            key = key * d + x  # (distinct modulo 2^64: the product of the lengths is below that)
        keys = torch.unique(torch.cat([keys, key]))
        if keys.numel() >= nnz:
            break
    keys = keys[torch.argsort(torch.rand(keys.numel(), generator=g, device="cuda", dtype=torch.float64))[:nnz]]
    idx = torch.empty((len(dims), keys.numel()), dtype=torch.int64, device="cuda")
    high = keys < 0  # a key past 2^63 reads as key - 2^64
    for m in range(len(dims) - 1, -1, -1):
        d = dims[m]
        # floor division of the unsigned key: 2^64 = q d + r
        q, r = divmod(1 << 64, d)
        lo = keys.div(d, rounding_mode="floor")
        idx[m] = keys - lo * d + high * r
        over = idx[m].div(d, rounding_mode="floor")
        idx[m] -= over * d
        keys = lo + over + high * (q if q < 1 << 63 else q - (1 << 64))
        high = keys < 0
    return idx, g


def _coo(case, seed, values="uniform"):
    """(dims, [int64 index tensors], float32 values) on the GPU."""
    dims = _dims(case)
    idx, g = _draw(dims, case["nnz"], [float(z) for z in case["zipf"].split(",")], seed)
    if values == "lognormal":
        vals = torch.randn(idx.shape[1], generator=g, device="cuda").exp_()
    else:
        vals = torch.rand(idx.shape[1], generator=g, device="cuda")
    return dims, [idx[m].contiguous() for m in range(len(dims))], vals


def _factors(dims, rank, seed, dtype=torch.float32):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed * 7 + 1)
    return [(torch.rand((d, rank), generator=g, device="cuda") * 2 - 1).to(dtype) for d in dims]


def _model(dims, rank, seed):
    """Initial host model: values in [-3, 3], random sign, as the driver draws them."""
    flat = synth.init_values(sum(dims) * rank, seed=seed).astype(np.float32).astype(np.float64)
    out, at = [], 0
    for d in dims:
        out.append(flat[at:at + d * rank].reshape(d, rank))
        at += d * rank
    return out


def _slices(dims, nnz, zipf, rank, count, seed, device):
    """`count` slices of one time step each over the spatial `dims`.  A
    nonzero lies inside one of `rank` communities (row i belongs to i mod
    rank), so the streams have the components that a model of them finds."""
    out = []
    for k in range(count):
        idx, g = _draw(dims, nnz, zipf, seed * 1009 + k)
        vals = torch.rand(idx.shape[1], generator=g, device="cuda")
        for m in range(1, len(dims)):
            c = idx[m] - idx[m] % rank + idx[0] % rank
            idx[m] = torch.where(c < dims[m], c, c - rank)
        n = idx.shape[1]
        cols = torch.zeros((len(dims) + 1, n), dtype=torch.int64, device="cuda")
        cols[1:] = idx
        vals = torch.floor(vals * 6) + 1  # small counts
        if device:
            out.append(([c.to(torch.int32).contiguous() for c in cols], vals))
        else:
            out.append((cols.cpu().numpy().astype(np.uint64), vals.double().cpu().numpy()))
    return out


def _warm(dims, rank, seed):
    """Initial model of a stream, near its communities (a session that is resumed)."""
    rng = np.random.default_rng(seed)
    rows = np.concatenate([np.arange(d) for d in [1] + dims])
    U = 0.1 * rng.standard_normal((len(rows), rank))
    U[np.arange(len(rows)), rows % rank] += 1.0 + rng.random(len(rows))
    return U.ravel()


def _streams(case, seed):
    """The serving case's streams: spatial dims log-uniform, a rank and a constraint each."""
    rng = np.random.default_rng(case["streams"] * 1000 + case["inner"])  # (shapes are the case's, data the seed's)
    out = []
    for k in range(case["streams"]):
        dims = [int(round(case["lo"] * (case["hi"] / case["lo"]) ** rng.random())) for _ in range(3)]
        nnz = int(np.clip(rng.lognormal(np.log(case["nnz"]), 0.7), 10000, 4 * case["nnz"]))
        rank = (8, 16, 32)[k % 3]
        out.append(dict(dims=dims, rank=rank, nonneg=bool(k % 2), inner=case["inner"],
                        slices=_slices(dims, nnz, [1.1] * 3, rank, case["slices"], seed * 31 + k, False),
                        init=_warm(dims, rank, seed * 31 + k)))
    return out


def _one_stream(case, seed):
    dims = _dims(case)
    zipf = [float(z) for z in case["zipf"].split(",")]
    return dict(dims=dims, rank=case["rank"], nonneg=case["nonneg"], inner=case["inner"],
                slices=_slices(dims, case["nnz"], zipf, case["rank"], case["slices"], seed, case["device"]),
                init=_warm(dims, case["rank"], seed))


FORGETTING = 0.95


def prepare(case, seed):
    kind = case["kind"]
    if kind == "mttkrp":
        dims, idx, vals = _coo(case, seed, "lognormal")
        t = A.create_alto(dims, idx, vals)
        dt = torch.bfloat16 if case["dtype"] == "bf16" else torch.float32
        F = _factors(dims, case["rank"], seed, dt)
        t.autotune(F, case["rank"])
        out = [torch.empty((d, case["rank"]), dtype=torch.float32, device="cuda") for d in dims]
        return dict(kind=kind, t=t, F=F, rank=case["rank"], out=out)
    if kind == "build":
        dims, idx, vals = _coo(case, seed, "lognormal")
        return dict(kind=kind, dims=dims, idx=idx, vals=vals.double(), F=_factors(dims, case["rank"], seed),
                    rank=case["rank"])
    if kind == "cpals":
        dims, idx, vals = _coo(case, seed)
        return dict(kind=kind, t=A.create_alto(dims, idx, vals), U=_model(dims, case["rank"], seed),
                    lam=np.ones(case["rank"]), rank=case["rank"], iters=case["iters"],
                    storage=A.BF16 if case["dtype"] == "bf16" else A.F32)
    if kind == "stream":
        s = _one_stream(case, seed)
        h = A.CPStream(4, 0, s["rank"], constraint=A.NONNEG if s["nonneg"] else A.UNCONSTRAINED,
                       forgetting=FORGETTING, max_inner=s["inner"], epsilon=0.0)
        dims = [1] + s["dims"]
        h.push(dims, *s["slices"][0], init_vals=s["init"])
        return dict(kind=kind, h=h, dims=dims, slices=s["slices"][1:])
    if kind == "serve":
        streams = _streams(case, seed)
        srv = A.Server(80 << 30)
        sids = [srv.open(4, 0, s["rank"], [1] + s["dims"], max(len(x[1]) for x in s["slices"]),
                         constraint=A.NONNEG if s["nonneg"] else A.UNCONSTRAINED, forgetting=FORGETTING,
                         max_inner=s["inner"], epsilon=0.0) for s in streams]
        for sid, s in zip(sids, streams):
            srv.submit(sid, [1] + s["dims"], *s["slices"][0], init_vals=s["init"])
        srv.drain()
        return dict(kind=kind, srv=srv, sids=sids, streams=streams)
    dims, idx, vals = _coo(case, seed)
    return dict(kind=kind, dims=dims, idx=idx, vals=vals.double(), steps=case["steps"])


def run(state):
    kind = state["kind"]
    if kind == "mttkrp":
        t, F, R = state["t"], state["F"], state["rank"]
        return [t.mttkrp(m, F, R, out=o) for m, o in enumerate(state["out"])]
    if kind == "build":
        t = A.create_alto(state["dims"], state["idx"], state["vals"])
        out = [t.mttkrp(m, state["F"], state["rank"]) for m in range(len(state["dims"]))]
        t.close()
        return out
    if kind == "cpals":
        U, lam, fits, _ = A.cpd_alto(state["t"], state["U"], state["lam"], state["rank"], state["iters"], 0.0,
                                     fit_mode=A.FIT_EXACT, storage=state["storage"])
        return [u.astype(np.float32) for u in U] + [lam.astype(np.float32), fits.astype(np.float32)]
    if kind == "stream":
        h = state["h"]
        for idx, vals in state["slices"]:
            h.push(state["dims"], idx, vals)
        out = [h.factor(m, d).astype(np.float32) for m, d in enumerate(state["dims"]) if m]
        return out + [h.factor(0, 1 << 16)[-len(state["slices"]):].astype(np.float32)]
    if kind == "serve":
        srv, last = state["srv"], []
        for k in range(1, len(state["streams"][0]["slices"])):
            for sid, s in zip(state["sids"], state["streams"]):
                srv.submit(sid, [1] + s["dims"], *s["slices"][k])
        srv.drain()
        for sid in state["sids"]:
            last += [srv.factor(sid, m).astype(np.float32) for m in (1, 2, 3)]
        return last
    s = A.Slicer(state["dims"], state["idx"], state["vals"], 0)
    n = s.cut_all(nnz_threshold=1 << 62, timeslice_limit=state["steps"])
    cuts = np.array([[b.nnz, *b.dims.tolist()] for b in (s.batch(k) for k in range(n))], np.int64)
    idx, vals = s.tensor().tensors()
    for x in (*idx, vals):
        x.slicer = s  # the views live as long as the slicer
    labels = []
    for m in range(1, len(state["dims"])):
        labels.append(np.full(state["dims"][m], -1, np.int64))
        seen = s.iperm(m)
        labels[-1][:len(seen)] = seen
    return [*idx, vals, cuts, *labels]


# ------------------------------------------------------------------- exact

def _mttkrp64(idx, vals, F, mode):
    out = torch.zeros(F[mode].shape, dtype=torch.float64, device="cuda")
    step = max(1, (1 << 26) // F[0].shape[1])
    for a in range(0, vals.numel(), step):
        p = vals[a:a + step].double()[:, None].expand(-1, F[0].shape[1])
        for m, f in enumerate(F):
            if m != mode:
                p = p * f[idx[m][a:a + step]].double()
        out.index_add_(0, idx[mode][a:a + step], p)
    return out


def _hadamard(mats):
    p = mats[0].clone()
    for m in mats[1:]:
        p = p * m
    return p


def _stream64(s):
    """Factors after all slices, and the time rows: CP-stream in float64."""
    R, N, dims = s["rank"], 4, [1] + s["dims"]
    eye = torch.eye(R, dtype=torch.float64, device="cuda")
    init = torch.from_numpy(s["init"].astype(np.float32)).double().cuda()
    U, at = [], 0
    for d in dims:
        U.append(init[at:at + d * R].reshape(d, R).clone())
        at += d * R
    U[0].zero_()
    for m in (1, 2, 3):
        U[m] /= U[m].square().sum(0).clamp_min(1e-12).sqrt()
    P = [torch.zeros_like(u) for u in U]
    Gt = torch.zeros_like(eye)
    rows = []
    for cols, vals in s["slices"]:
        idx = [torch.as_tensor(np.asarray(c).astype(np.int64) if isinstance(c, np.ndarray) else c).cuda().long()
               for c in cols]
        v = torch.as_tensor(vals).cuda().double()
        G = [None] + [U[m].T @ U[m] for m in (1, 2, 3)]
        C = [None] + [P[m].T @ U[m] for m in (1, 2, 3)]
        dual = [torch.zeros_like(u) for u in U]
        for _ in range(s["inner"]):
            U[0] = torch.linalg.solve(_hadamard(G[1:]) + 1e-12 * eye, _mttkrp64(idx, v, U, 0).T).T
            old = Gt
            Gt = Gt + U[0].T @ U[0]
            for j in (1, 2, 3):
                others = [m for m in (1, 2, 3) if m != j]
                rhs = P[j] @ (old * _hadamard([C[m] for m in others])) + _mttkrp64(idx, v, U, j)
                Phi = Gt * _hadamard([G[m] for m in others])
                if s["nonneg"]:
                    U[j], dual[j] = _admm64(U[j], dual[j], rhs, Phi, eye)
                else:
                    U[j] = torch.linalg.solve(Phi + 1e-12 * eye, rhs.T).T
                G[j], C[j] = U[j].T @ U[j], P[j].T @ U[j]
        Gt = Gt * FORGETTING
        P = [u.clone() for u in U]
        rows.append(U[0].clone())
    return U, torch.cat(rows)


def _admm64(x, u, rhs, Phi, eye):
    rho = Phi.trace() / Phi.shape[0]
    W = torch.linalg.inv(Phi + rho * eye)
    x0 = x
    z = (rhs + rho * (x + u)) @ W
    x = (z - u).clamp_min(0)
    for k in range(25):
        y = x - z
        u = u + y
        z = (rhs + rho * (x + u)) @ W
        moved = (x - x0).square().sum() if k == 0 else 0.0 * rho
        pres, pnorm, dnorm = y.square().sum(), x.square().sum(), u.square().sum()
        x = (z - u).clamp_min(0)
        tol = float(np.float32(1e-6))
        if pres <= tol * pnorm and moved <= tol * dnorm:
            break
    return x, u


def _cpals64(case, seed):
    dims, idx, vals = _coo(case, seed)
    R = case["rank"]
    U = [torch.from_numpy(u).cuda() for u in _model(dims, R, seed)]
    G = [u.T @ u for u in U]
    eye = torch.eye(R, dtype=torch.float64, device="cuda")
    norm = vals.double().square().sum()
    fits = []
    for it in range(case["iters"]):
        for j in range(len(dims)):
            M = _mttkrp64(idx, vals, U, j)
            V = _hadamard([G[m] for m in range(len(dims)) if m != j])
            U[j] = torch.linalg.solve(V + 1e-3 * eye, M.T).T
            lam = U[j].square().sum(0).clamp_min(1e-12).sqrt() if it == 0 else U[j].amax(0).clamp_min(1.0)
            U[j] = U[j] / lam
            G[j] = U[j].T @ U[j]
        inner = (U[-1] * M * lam).sum()
        model = ((lam[:, None] * lam[None, :]) * _hadamard(G)).sum().abs()
        fits.append(((norm + model - 2 * inner).clamp_min(0).sqrt() / norm.sqrt()).reshape(1))
    return U + [lam, torch.cat(fits)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("mttkrp", "build"):
        dims, idx, vals = _coo(case, seed, "lognormal")
        F = _factors(dims, case["rank"], seed, torch.bfloat16 if case.get("dtype") == "bf16" else torch.float32)
        return [_mttkrp64(idx, vals, F, m) for m in range(len(dims))]
    if kind == "cpals":
        if case["dtype"] == "bf16":  # the rounding of the stored factors is the caller's choice
            return None
        return _cpals64(case, seed)
    if kind == "stream":
        U, rows = _stream64(_one_stream(case, seed))
        return U[1:] + [rows[1:]]
    if kind == "serve":
        out = []
        for s in _streams(case, seed):
            out += _stream64(s)[0][1:]
        return out
    return None  # sorted and relabelled indices: whole numbers


# -------------------------------------------------------------------- work

def _mttkrp_work(dims, nnz, R, fbytes):
    """All modes: the key and value of every nonzero once, each factor and output once."""
    key = 8 if sum(max(0, (d - 1).bit_length()) for d in dims) <= 64 else 16
    b = sum(nnz * (key + 4) + R * fbytes * (sum(dims) - d) + 4 * R * d for d in dims)
    return b, float(nnz) * R * len(dims) * len(dims)


def _stream_work(dims, nnz, R, inner, slices, nonneg):
    """Per inner iteration and mode: the MTTKRP, the row solves and the Grams."""
    mb, mf = _mttkrp_work([1] + dims, nnz, R, 4)
    rows = sum(dims)
    b = mb + rows * R * (12 + 8 + (24 if nonneg else 0))
    f = mf + rows * R * R * 2 * (4 + (2 if nonneg else 0))
    return inner * slices * b, inner * slices * f


def work(case):
    kind = case["kind"]
    if kind == "serve":
        mid = int((case["lo"] * case["hi"]) ** 0.5)
        b, f = _stream_work([mid] * 3, case["nnz"], 16, case["inner"], case["slices"] - 1, True)
        return {"bytes": b * case["streams"], "flops": f * case["streams"]}
    dims, nnz = _dims(case), case["nnz"]
    if kind == "slicer":
        return {"bytes": nnz * (8 * len(dims) + 8 + 4 * len(dims) + 8), "flops": 0}
    R = case["rank"]
    if kind == "stream":
        b, f = _stream_work(dims, nnz, R, case["inner"], case["slices"] - 1, case["nonneg"])
        return {"bytes": b, "flops": f}
    b, f = _mttkrp_work(dims, nnz, R, 2 if case.get("dtype") == "bf16" else 4)
    if kind == "build":
        return {"bytes": b + nnz * (8 * len(dims) + 8), "flops": f}
    if kind == "cpals":
        it = case["iters"]
        return {"bytes": it * (b + sum(dims) * R * 12) + sum(dims) * R * 16,
                "flops": it * (f + sum(dims) * R * R * 4)}
    return {"bytes": b, "flops": f}
