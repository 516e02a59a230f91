"""Timing cases of the Laplace FMM engine: the calls a program makes, over the range of its use.

Every case is one call sequence through the public Python binding:

* "fmm": new positions into a context that the program keeps, one solve, the
  results on the device (an MD or n-body step, a served request).
* "batch": many independent systems of uneven sizes in one call.
* "direct": the FP64 direct sum over sampled targets that every accuracy check makes
  (host arrays, as the program that verifies a solve has them).

Both precisions run: FP64 (the plain method) and mixed.  Orders, acceptance
parameters and leaf sizes are those of the benchmark, the tests and the example
driver: P from 4 to 12, theta from 0.35 to 0.5, ncrit 32 to 128.
"""
import importlib
import math

import numpy as np
import torch

fmm = importlib.import_module("exafmm-beta_b200")
datasets = importlib.import_module("exafmm-beta_b200.datasets")

MAX_EXACT_PAIRS = 6.0e10  # pairs the 64-bit direct sum takes in a few seconds


def listed():
    return [
        # the smallest served request, plain method: launches and latency are all of it
        dict(name="cube_1k_fp64_p6", kind="fmm", dist="cube", n=1000, P=6, theta=0.4, ncrit=64, mixed=False, images=0),
        # a small served request or chain step of odd size, mixed precision
        dict(name="sphere_7k_mixed_p10", kind="fmm", dist="sphere", n=7019, P=10, theta=0.4, ncrit=64, mixed=True,
             images=0),
        # the example driver's own configuration, plain method
        dict(name="cube_100k_fp64_p10", kind="fmm", dist="cube", n=100000, P=10, theta=0.4, ncrit=64, mixed=False,
             images=0),
        # the same in mixed precision: an ordinary served request
        dict(name="cube_100k_mixed_p10", kind="fmm", dist="cube", n=100000, P=10, theta=0.4, ncrit=64, mixed=True,
             images=0),
        # a served request of low order and ragged size, adaptive tree
        dict(name="plummer_300k_mixed_p6", kind="fmm", dist="plummer", n=300007, P=6, theta=0.4, ncrit=64, mixed=True,
             images=0),
        # a large adaptive solve, plain method
        dict(name="plummer_1m_fp64_p8", kind="fmm", dist="plummer", n=1000003, P=8, theta=0.35, ncrit=64, mixed=False,
             images=0),
        # the largest: the benchmark's adaptive solve
        dict(name="plummer_4m_mixed_p8", kind="fmm", dist="plummer", n=4194304, P=8, theta=0.35, ncrit=128, mixed=True,
             images=0),
        # a periodic box of ordinary MD size, plain method
        dict(name="water_36k_fp64_p8_images3", kind="fmm", dist="water", n=36000, P=8, theta=0.4, ncrit=64,
             mixed=False, images=3),
        # the benchmark's periodic water box
        dict(name="water_1m_mixed_p10_images3", kind="fmm", dist="water", n=999999, P=10, theta=0.4, ncrit=128,
             mixed=True, images=3),
        # many uneven systems in one call (the batched workload)
        dict(name="batch_128_mixed_p10", kind="batch", count=128, lo=2000, hi=200000, P=10, theta=0.4, ncrit=128,
             mixed=True),
        # the accuracy check of a large solve: strided targets against every body
        dict(name="direct_4k_of_1m", kind="direct", nt=4096, ns=1000003),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choices(["fmm", "periodic", "batch", "direct"], [6, 2, 2, 1])[0]
    mixed = rng.random() < 0.5
    P = rng.choice([4, 6, 8, 8, 10, 10, 12])
    theta = rng.choice([0.35, 0.4, 0.4, 0.5])
    ncrit = rng.choice([32, 64, 64, 128])
    # sizes whose solve costs no more than the largest listed one's
    hi = (1500000 if mixed else 300000) if P <= 8 else (400000 if mixed else 100000)
    if kind == "fmm":
        return dict(kind="fmm", dist=rng.choice(["cube", "sphere", "plummer"]), n=_log(rng, 1000, hi), P=P,
                    theta=theta, ncrit=ncrit, mixed=mixed, images=0)
    if kind == "periodic":
        return dict(kind="fmm", dist="water", n=3 * _log(rng, 1000, hi // 6), P=P, theta=rng.choice([0.4, 0.5]),
                    ncrit=ncrit, mixed=mixed, images=rng.choice([1, 2, 3]))
    if kind == "batch":
        return dict(kind="batch", count=rng.randrange(8, 97), lo=2000, hi=_log(rng, 10000, 100000 if mixed else 40000),
                    P=rng.choice([6, 8, 10]), theta=0.4, ncrit=rng.choice([64, 128]), mixed=mixed)
    return dict(kind="direct", nt=_log(rng, 100, 4096), ns=_log(rng, 10000, 1000000))


# ---------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _bodies(dist, n, seed):
    """(n, 4) float64 on the GPU (x, y, z, charge), and the edge of the box."""
    if dist == "water":
        x, edge = datasets.water_box(n // 3, seed=seed)
        return torch.from_numpy(np.ascontiguousarray(x)).cuda(), edge
    g = _gen(seed)
    x = torch.empty((n, 4), dtype=torch.float64, device="cuda")
    if dist == "cube":  # uniform in [-1, 1]^3, zero net charge
        x.uniform_(-1.0, 1.0, generator=g)
        x[:, 3] -= x[:, 3].mean()
        return x, 2.0
    v = torch.randn((n, 3), dtype=torch.float64, device="cuda", generator=g)
    v /= v.norm(dim=1, keepdim=True)
    u = torch.rand(n, dtype=torch.float64, device="cuda", generator=g)
    if dist == "sphere":  # unit sphere's surface, charges U[-1, 1]
        x[:, :3] = v
        x[:, 3] = 2.0 * u - 1.0
        return x, 2.0
    # Plummer sphere by the inverse CDF, cut off at 20 core radii, equal charges
    top = (1.0 + 20.0 ** -2) ** -1.5
    r = 1.0 / torch.sqrt((u * top).clamp_min(1e-30) ** (-2.0 / 3.0) - 1.0)
    x[:, :3] = v * r[:, None]
    x[:, 3] = 1.0 / n
    return x, 40.0


def _sizes(case):
    """The batch's sizes: log-uniform in [lo, hi], the same for every seed."""
    r = np.random.default_rng(case["count"] * 1000003 + case["hi"])
    return [int(v) for v in np.exp(r.uniform(math.log(case["lo"]), math.log(case["hi"]), case["count"]))]


def _systems(case, seed):
    return [_bodies("sphere" if i % 2 else "cube", n, seed * 4099 + i)[0] for i, n in enumerate(_sizes(case))]


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "direct":
        src = _bodies("plummer", case["ns"], seed)[0].cpu().numpy()
        s["sources"] = src
        s["targets"] = np.ascontiguousarray(src[datasets.strided_sample(case["ns"], case["nt"])])
        return s
    precision = fmm.MIXED if case["mixed"] else fmm.FP64
    if kind == "batch":
        s["x"] = torch.cat(_systems(case, seed))
        s["sizes"] = _sizes(case)
        s["out"] = torch.zeros_like(s["x"])
        off = np.concatenate([[0], np.cumsum(s["sizes"])])[:-1] * 32
        s["in_ptrs"] = [s["x"].data_ptr() + int(o) for o in off]
        s["out_ptrs"] = [s["out"].data_ptr() + int(o) for o in off]
        s["batch"] = fmm.Batch(P=case["P"], theta=case["theta"], ncrit=case["ncrit"], precision=precision, workers=3,
                               forest=3)
    else:
        s["x"], edge = _bodies(case["dist"], case["n"], seed)
        s["out"] = torch.zeros_like(s["x"])
        s["fmm"] = fmm.Fmm(P=case["P"], theta=case["theta"], ncrit=case["ncrit"], images=case["images"], cycle=edge,
                           precision=precision)
    torch.cuda.synchronize()  # the engine reads these on a stream of its own
    return s


def run(state):
    kind = state["case"]["kind"]
    if kind == "direct":
        r = fmm.direct(state["targets"], state["sources"])
    elif kind == "batch":
        state["batch"].solve_device(state["sizes"], state["in_ptrs"], state["out_ptrs"])
        r = state["out"]
    else:
        f = state["fmm"]
        f.set_bodies_device(state["x"].data_ptr(), len(state["x"]))
        f.solve()
        f.results_device(state["out"].data_ptr())
        r = state["out"]
    return {"potential": r[:, 0], "gradient": r[:, 1:]}


# ---------------------------------------------------------------- what a pass needs
def _fmm_flops(n, P, ncrit):
    """Near field: 27 neighbor leaves of ncrit / 2 bodies, 20 operations a pair.  Far field: 189
    translations a leaf cell, 4 P^3 operations each (the cost of a translation by rotations)."""
    leaf = ncrit / 2
    return n * 27 * min(leaf, n) * 20 + (n / leaf) * 189 * 4.0 * P ** 3


def work(case):
    kind = case["kind"]
    if kind == "direct":
        return {"bytes": 32.0 * case["ns"] + 64.0 * case["nt"], "flops": 20.0 * case["ns"] * case["nt"]}
    if kind == "batch":
        n = sum(_sizes(case))
        return {"bytes": 64.0 * n, "flops": _fmm_flops(n, case["P"], case["ncrit"])}
    return {"bytes": 64.0 * case["n"], "flops": _fmm_flops(case["n"], case["P"], case["ncrit"])}


def tolerance(case):
    # Measured as the difference between a solve and the solve of the same bodies with their
    # coordinates permuted (another orientation of every expansion, other sums), times four.
    if case["kind"] == "direct":
        return {"rel": 1e-13, "max": 1e-11}
    if not case["mixed"]:
        # the lattice's image sums cancel strongly in the periodic potential
        return {"rel": 5e-11} if case.get("images") else {"rel": 1e-13}
    return {"rel": 2.5e-6, "max": 2e-5}


# ---------------------------------------------------------------- the 64-bit answer
def _direct64(targets, sources):
    nt, ns = len(targets), len(sources)
    out = torch.zeros((nt, 4), dtype=torch.float64, device=targets.device)
    rows = max(1, min(nt, 1 << 12))
    cols = max(1, (1 << 26) // rows)
    for a in range(0, nt, rows):
        t = targets[a:a + rows]
        for b in range(0, ns, cols):
            s = sources[b:b + cols]
            d = [t[:, k, None] - s[None, :, k] for k in range(3)]
            r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
            inv = torch.where(r2 > 0, r2.rsqrt(), torch.zeros_like(r2))
            q = inv * s[None, :, 3]
            out[a:a + rows, 0] += q.sum(1)
            q *= inv * inv
            for k in range(3):
                out[a:a + rows, 1 + k] -= (q * d[k]).sum(1)
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "direct":
        s = _bodies("plummer", case["ns"], seed)[0]
        idx = torch.from_numpy(datasets.strided_sample(case["ns"], case["nt"])).cuda()
        r = _direct64(s[idx], s)
    elif kind == "batch":
        if sum(float(n) * n for n in _sizes(case)) > MAX_EXACT_PAIRS:
            return None
        r = torch.cat([_direct64(x, x) for x in _systems(case, seed)])
    else:
        if case["images"] or float(case["n"]) ** 2 > MAX_EXACT_PAIRS:
            return None
        x = _bodies(case["dist"], case["n"], seed)[0]
        r = _direct64(x, x)
    if kind == "direct":
        r = r.cpu().numpy()
    return {"potential": r[:, 0], "gradient": r[:, 1:]}
