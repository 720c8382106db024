"""Workloads of the framework as a user's program calls it, for timing and checking.

A case is a dict of plain values:

* ``kind``: what one pass does
    - ``mttkrp``: the MTTKRP of every mode in order, following the plan, into device buffers
      (what a CP-ALS sweep spends its time on);
    - ``als``: a whole CP-ALS run from seeded start factors, factors and lambda read back;
    - ``batch``: CP-ALS sweeps of many small tensors in one captured graph;
    - ``build``: an engine built on a tensor in device memory (sort, trees, walk schedules) and its
      first MTTKRP;
    - ``host_mttkrp``, ``host_als``: the AdaTM C entry points on host FP64 buffers.
* ``dims`` ("1000x1000x1000"), ``nnz`` (coordinates drawn; duplicates are summed), ``alpha`` (Zipf
  exponent of every mode's indices, 0 = uniform), ``lognormal`` (values lognormal(0,1), else U(0,1)),
  ``rank``, ``plan`` ("learned", "analytic": memoized; "allmode", "twomode", "onemode": SPLATT's plain
  allocations), ``bf16`` (BF16 factor rows), ``iters``, ``count`` (tensors of a batch).

The engines compute in FP32 (rows of FP32 factors, FP32 partial sums); the FP64 containers that the
entry points fill are returned as the FP32 values that they hold to that precision. BF16 engines keep
BF16-valued factors, but their MTTKRPs are FP32 sums as well.

Sizes are such that every slice of every mode holds nonzeros (a tensor is cleaned of empty slices
before it is decomposed), so its dims do not depend on the seed.
"""
import math
import os

import numpy as np
import torch

import adatm_b200 as A

HERE = os.path.dirname(os.path.abspath(A.__file__))
MASK = (1 << 64) - 1


def _case(name, kind, dims, nnz, alpha, rank, plan, bf16=False, lognormal=False, iters=0, count=0):
    return {"name": name, "kind": kind, "dims": dims, "nnz": nnz, "alpha": alpha, "rank": rank,
            "plan": plan, "bf16": bf16, "lognormal": lognormal, "iters": iters, "count": count}


def listed():
    return [
        # one MTTKRP call of a C program on a small tensor: latency, copies and conversions
        _case("host_mttkrp_3mode_100k_r10", "host_mttkrp", "300x200x100", 100_000, 1.1, 10, "analytic"),
        # a small decomposition on the device: every kernel is a few microseconds
        _case("als_4mode_20k_r16", "als", "60x50x40x30", 20_000, 0.0, 16, "analytic", iters=3),
        # the benchmark's plain 3rd-order tensor, its ten iterations
        _case("als_3mode_1m_r16", "als", "1000x1000x1000", 1_000_000, 0.0, 16, "learned", iters=10),
        # a C program's cpd_als_iterate_adaptive: host FP64 factors in and out, three iterations
        _case("host_als_4mode_2m_r24", "host_als", "2000x1500x500x300", 2_000_000, 0.0, 24, "analytic",
              iters=3),
        # many small tensors swept together (the batched workload at tensor sizes of its lower half),
        # one captured sweep
        _case("batch_16_r16", "batch", "", 0, 0.0, 16, "analytic", iters=1, count=16),
        # a plain single-tree allocation (root, internal and leaf MTTKRPs), odd dims and rank
        _case("mttkrp_3mode_3m_onemode_r17", "mttkrp", "1777x333x4999", 3_000_000, 1.0, 17, "onemode"),
        # one tree per mode, a wide rank that fills no power of two
        _case("mttkrp_4mode_4m_allmode_r100", "mttkrp", "8000x3001x700x64", 4_000_000, 1.2, 100,
              "allmode"),
        # the highest order supported: long memo chains, hypersparse lower levels
        _case("mttkrp_8mode_3m_r32", "mttkrp", "3000x2500x2000x1500x800x400x200x60", 3_000_000, 1.3, 32,
              "learned"),
        # the benchmark's 4th-order tensor
        _case("mttkrp_4mode_20m_r32", "mttkrp", "5000x5000x2000x500", 20_000_000, 1.1, 32, "learned"),
        # the benchmark's 5th-order tensor with BF16 factor rows
        _case("mttkrp_5mode_50m_r64_bf16", "mttkrp", "20000x10000x5000x1000x200", 50_000_000, 1.2, 64,
              "learned", bf16=True, lognormal=True),
        # the benchmark's headline: the 6th-order tensor
        _case("mttkrp_6mode_100m_r32", "mttkrp", "50000x20000x10000x2000x500x100", 100_000_000, 1.3, 32,
              "learned"),
        # a new tensor: trees and schedules built, then the first MTTKRP on them
        _case("build_5mode_5m_r32", "build", "8000x6000x5000x1000x200", 5_000_000, 1.2, 32, "analytic"),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _most(nnz, alpha, hi):
    """The largest dim up to `hi` that `nnz` draws fill: 25 or more expected in its least likely slice."""
    if not alpha:
        return max(2, min(hi, nnz // 25))
    p = np.arange(1, hi + 1, dtype=np.float64) ** -alpha
    return max(2, int(np.searchsorted(-p / np.cumsum(p), -25.0 / nnz, side="right")))


def draw(rng):
    kind = rng.choice(["mttkrp"] * 6 + ["als", "host_mttkrp", "host_als", "build"])
    order = rng.randint(3, 8)
    rank = _log_uniform(rng, 6, 128)
    if kind in ("als", "host_als"):
        # sparse tensors with uniform indices and one sweep: well conditioned, so the factors say
        # something about each step of it
        order = rng.randint(3, 5)
        rank = _log_uniform(rng, 6, 32)
        nnz = _log_uniform(rng, 20_000, 2_000_000)
        alpha = 0.0
        top = _most(nnz, alpha, 5000)
        dims = [_log_uniform(rng, min(top, 200), top) for _ in range(order)]
        nnz = min(nnz, math.prod(dims) // 200)
    else:
        most = {"mttkrp": 20_000_000, "build": 5_000_000, "host_mttkrp": 500_000}[kind]
        nnz = min(_log_uniform(rng, 10_000, most), 640_000_000 // rank)
        alpha = rng.choice([0.0, round(rng.uniform(1.0, 1.6), 2)])
        top = _most(nnz, alpha, 100_000)
        dims = [_log_uniform(rng, min(top, 50), top) for _ in range(order)]
    plan = "analytic"
    if kind in ("mttkrp", "build"):
        plan = rng.choice(["learned", "learned", "analytic", "allmode", "twomode", "onemode"])
    return {"kind": kind, "dims": "x".join(map(str, dims)), "nnz": nnz, "alpha": alpha, "rank": rank,
            "plan": plan, "bf16": kind == "mttkrp" and rng.random() < 0.3,
            "lognormal": rng.random() < 0.3 and kind == "mttkrp",
            "iters": 1 if kind in ("als", "host_als") else 0, "count": 0}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

_MODEL = None


def _model():
    global _MODEL
    if _MODEL is None:
        _MODEL = A.PlanModel.load(os.path.join(HERE, "planner_data", "plan_model.npz"))
    return _MODEL


def _dims(case):
    return [int(d) for d in case["dims"].split("x")]


def _batch_specs(case):
    """Dims and nnz of a batch's tensors: like the batched workload, uneven orders and sizes."""
    rng = np.random.default_rng(12345)
    specs = []
    for _ in range(case["count"]):
        order = int(rng.integers(3, 6))
        nnz = int(round(math.exp(rng.uniform(math.log(2e4), math.log(5e5)))))
        top = _most(nnz, 0.0, 20_000)
        dims = [int(round(math.exp(rng.uniform(math.log(200), math.log(top))))) for _ in range(order)]
        specs.append((dims, min(nnz, math.prod(dims) // 200)))
    return specs


def _generate(case, seed):
    return A.Tensor.generate(_dims(case), case["nnz"], alpha=case["alpha"] or None,
                             value_kind=1 if case["lognormal"] else 0, seed=seed)


def _plan(case, t):
    if case["plan"] == "learned":
        return A.plan_learned(t, case["rank"], _model())[0]
    if case["plan"] == "analytic":
        return A.plan_analytic(t, case["rank"])[0]
    return A.plan_splatt(t, {"onemode": A.CSF_ONEMODE, "twomode": A.CSF_TWOMODE,
                             "allmode": A.CSF_ALLMODE}[case["plan"]])


def _buffers(dims, rank):
    ldr = (rank + 3) // 4 * 4
    return [torch.zeros((d, ldr), dtype=torch.float64, device="cuda") for d in dims]


def _host_factors(dims, rank, seed):
    rng = np.random.default_rng(seed)
    return [rng.random((d, rank), dtype=np.float32).astype(np.float64) for d in dims]


def prepare(case, seed):
    rank, kind = case["rank"], case["kind"]
    st = {"case": case, "seed": seed}
    if kind == "batch":
        st["engines"], st["tensors"] = [], []
        for k, (dims, nnz) in enumerate(_batch_specs(case)):
            t = A.Tensor.generate(dims, nnz, seed=seed * 1000 + k)
            st["tensors"].append(t)
            st["engines"].append(A.Engine(t, rank, A.plan_analytic(t, rank)[0]))
        st["batch"] = A.BatchSweep(st["engines"])
        return st
    t = _generate(case, seed)
    _, _, dims = t.info()
    plan = _plan(case, t)
    if kind in ("host_mttkrp", "host_als"):
        inds, vals, dims = t.download()
        groups = plan["groups"]
        st["csf"] = A.csf_alloc_adaptive(inds, vals, dims, groups)
        st["rcsf"] = A.rcsf_alloc_adaptive(st["csf"], rank, groups)
        st["groups"] = groups
        st["use"] = A.decide_use_csfs(len(dims), groups, len(st["csf"]))
        st["mats"] = _host_factors(dims, rank, seed)
        return st
    st["tensor"], st["plan"] = t, plan
    st["out"] = _buffers(dims, rank)
    torch.cuda.synchronize()  # the buffers are zeroed on torch's stream, the engine has its own
    if kind != "build":
        st["engine"] = A.Engine(t, rank, plan, bf16=case["bf16"])
        st["engine"].init_factors(seed)
    return st


def _f32(x):
    return torch.from_numpy(x).to(torch.float32)


def run(st):
    case, kind = st["case"], st["case"]["kind"]
    rank = case["rank"]
    if kind == "mttkrp":
        # the buffers' last readers ran on torch's stream; the engine's calls end with its own
        torch.cuda.current_stream().synchronize()
        e = st["engine"]
        for m, b in enumerate(st["out"]):
            e.mttkrp_into(m, b.data_ptr())
        return [b[:, :rank].float() for b in st["out"]]
    if kind == "build":
        torch.cuda.current_stream().synchronize()
        e = A.Engine(st["tensor"], rank, st["plan"])
        e.init_factors(st["seed"])
        e.mttkrp_into(0, st["out"][0].data_ptr())
        e.free()
        return st["out"][0][:, :rank].float()
    if kind == "als":
        e = st["engine"]
        e.init_factors(st["seed"])
        r = e.als(case["iters"])
        mats, lam = e.get_factors()
        return {"factors": [_f32(m) for m in mats], "lambda": _f32(lam), "fit": _f32(r["trace"])}
    if kind == "batch":
        for e in st["engines"]:
            e.init_factors(st["seed"])
        st["batch"].begin()
        st["batch"].time_sweeps(case["iters"])
        return [_f32(np.concatenate(e.get_factors()[0])) for e in st["engines"]]
    uc, ut = st["use"]
    if kind == "host_mttkrp":
        return _f32(A.mttkrp_csf_adaptive(st["csf"], st["rcsf"], st["mats"], 0, st["groups"], uc, ut))
    r = A.cpd_als_iterate_adaptive(st["csf"], st["rcsf"], st["groups"], uc, ut, st["mats"],
                                   case["iters"], 0.0)
    return {"factors": [_f32(m) for m in r["factors"]], "lambda": _f32(r["lambda"]),
            "fit": _f32(np.array([r["fit"]]))}


def work(case):
    """Nonzeros read once (leaf index and value; the drawn count, as if none were duplicates), every
    factor read once, every result written once (FP32); one multiply and add per nonzero and column
    for each pass over the tensor that an MTTKRP sequence cannot share (one)."""
    rank = case["rank"]
    if case["kind"] == "batch":
        specs, sweeps = _batch_specs(case), case["iters"]
    else:
        specs, sweeps = [(_dims(case), case["nnz"])], max(1, case["iters"])
    nnz, rows = sum(n for _, n in specs), sum(sum(d) for d, _ in specs)
    if case["kind"] == "build":  # the coordinates in, one tree's worth of them out
        order = len(specs[0][0])
        return {"bytes": nnz * (4.0 * order + 8) + nnz * 8.0 + 8.0 * rows * rank, "flops": 2.0 * nnz * rank}
    width = 2.0 if case["bf16"] else 4.0
    return {"bytes": sweeps * (8.0 * nnz + (width + 4.0) * rows * rank), "flops": sweeps * 2.0 * nnz * rank}


# ---------------------------------------------------------------------------
# the same in FP64 with torch alone
# ---------------------------------------------------------------------------

def _signed(v):
    v &= MASK
    return v - (1 << 64) if v >> 63 else v


def _mix(z):
    """splitmix64's output function on int64 tensors (wrapping products, logical shifts)."""
    z = z + _signed(0x9E3779B97F4A7C15)
    z = (z ^ ((z >> 30) & ((1 << 34) - 1))) * _signed(0xBF58476D1CE4E5B9)
    z = (z ^ ((z >> 27) & ((1 << 37) - 1))) * _signed(0x94D049BB133111EB)
    return z ^ ((z >> 31) & ((1 << 33) - 1))


def _u01(key, first, n):
    z = _mix(torch.arange(first, first + n, device="cuda") + _signed(key))
    return ((z >> 11) & ((1 << 53) - 1)).double() * (1.0 / 9007199254740992.0)


def _key(x):
    z = (x + 0x9E3779B97F4A7C15) & MASK
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & MASK
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & MASK
    return z ^ (z >> 31)


def _draws(dims, nnz, alpha, lognormal, seed):
    """The drawn coordinates (one int32 tensor per mode, empty slices dropped), their values and the
    dims that are left; duplicates stay apart (every sum over nonzeros is the same)."""
    keys = [_key((seed * 0x100000001B3 + 0x1000 + m) & MASK) for m in range(len(dims) + 2)]
    idx, left = [], []
    for m, d in enumerate(dims):
        u = _u01(keys[m], 0, nnz)
        if alpha:
            p = np.cumsum(np.arange(1, d + 1, dtype=np.float64) ** -alpha)
            cdf = torch.from_numpy(p / p[-1]).cuda()
            cdf[-1] = 1.0
            k = torch.searchsorted(cdf, u, right=True).clamp_(max=d - 1)
        else:
            k = (u * d).long().clamp_(max=d - 1)
        used = torch.bincount(k, minlength=d) > 0
        idx.append((torch.cumsum(used, 0) - 1)[k].int())
        left.append(int(used.sum()))
        del u, k
    u = _u01(keys[len(dims)], 0, nnz)
    if lognormal:
        v = _u01(keys[len(dims) + 1], 0, nnz)
        u = torch.exp(torch.sqrt(-2.0 * torch.log(1.0 - u)) * torch.cos(2.0 * math.pi * v))
    return idx, u, left


def _seeded_factors(dims, rank, seed, bf16):
    out = []
    for m, d in enumerate(dims):
        f = _u01(_key((seed * 0x100000001B3 + m) & MASK), 0, d * rank).float()
        out.append((f.bfloat16() if bf16 else f).double().reshape(d, rank))
    return out


def _mttkrps(idx, vals, mats, modes):
    rank = mats[0].shape[1]
    out = {m: torch.zeros_like(mats[m]) for m in modes}
    step = max(1, 120_000_000 // rank)
    for a in range(0, len(vals), step):
        part = [i[a:a + step].long() for i in idx]
        rows = [f[i] for f, i in zip(mats, part)]
        for m in modes:
            x = vals[a:a + step, None].expand(-1, rank).contiguous()
            for k, r in enumerate(rows):
                if k != m:
                    x *= r
            out[m].index_add_(0, part[m], x)
    return [out[m] for m in modes]


def _als(idx, vals, dims, mats, iters, unit):
    """CP-ALS as SPLATT runs it; `unit`: factors scaled to unit columns at the end."""
    key = torch.zeros_like(idx[0], dtype=torch.int64)
    for i, d in zip(idx, dims):
        key = key * d + i
    norm = torch.zeros(int(key.max()) + 1, device="cuda", dtype=torch.float64) if key.max() < 1 << 28 else None
    if norm is None:
        uniq, inv = torch.unique(key, return_inverse=True)
        norm = torch.zeros(len(uniq), device="cuda", dtype=torch.float64)
        key = inv
    norm = norm.index_add_(0, key, vals).square().sum()
    rank = mats[0].shape[1]
    mats = list(mats)
    grams = [f.T @ f for f in mats]
    trace, lam = [], None
    for it in range(iters):
        for m in range(len(dims)):
            v = torch.ones(rank, rank, dtype=torch.float64, device="cuda")
            for k, g in enumerate(grams):
                if k != m:
                    v = v * g
            prod = _mttkrps(idx, vals, mats, [m])[0]
            f = torch.linalg.solve(v, prod.T).T
            lam = f.norm(dim=0) if it == 0 else f.max(dim=0).values.clamp(min=1.0)
            mats[m] = f / lam
            grams[m] = mats[m].T @ mats[m]
        had = torch.ones(rank, rank, dtype=torch.float64, device="cuda")
        for g in grams:
            had = had * g
        est = (lam @ had @ lam).abs()
        inner = (lam * (mats[-1] * prod).sum(dim=0)).sum()
        trace.append(float(1 - torch.sqrt(norm + est - 2 * inner) / torch.sqrt(norm)))
    if unit:
        for m, f in enumerate(mats):
            n = f.norm(dim=0)
            lam = lam * n
            mats[m] = f / n
        trace = trace[-1:]
    return {"factors": mats, "lambda": lam, "fit": torch.tensor(trace, dtype=torch.float64)}


def exact(case, seed):
    rank, kind = case["rank"], case["kind"]
    if kind == "batch":
        out = []
        for k, (dims, nnz) in enumerate(_batch_specs(case)):
            idx, vals, dims = _draws(dims, nnz, 0.0, False, seed * 1000 + k)
            r = _als(idx, vals, dims, _seeded_factors(dims, rank, seed, False), case["iters"], False)
            out.append(torch.cat(r["factors"]))
        return out
    idx, vals, dims = _draws(_dims(case), case["nnz"], case["alpha"], case["lognormal"], seed)
    if kind in ("host_mttkrp", "host_als"):
        mats = [torch.from_numpy(f).cuda() for f in _host_factors(dims, rank, seed)]
    else:
        mats = _seeded_factors(dims, rank, seed, case["bf16"])
    if kind in ("als", "host_als"):
        return _als(idx, vals, dims, mats, case["iters"], kind == "host_als")
    if kind == "mttkrp":
        return _mttkrps(idx, vals, mats, list(range(len(dims))))
    return _mttkrps(idx, vals, mats, [0])[0]
