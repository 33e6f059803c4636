"""The work that a program using this engine has it do, as measurable cases.

A case is one request through the public Python interface: load (or build) a
filtered complex, reduce it, and take its pairs and essential simplices.
`listed` names the cases, `draw` gives further ones of the same ranges,
`prepare` makes what a program holds before the call, `run` is one request.

Sizes follow the benchmark's and the workloads' configurations (2,000-point,
100,000-point and 300-20,000-point Rips complexes, mean degree 8-40;
lower-star grids of 16^3 to 96^3; batches of 200-5,000-point clouds) and the
smoke test.  The complexes of one program are reduced on one context, so every
state shares one Engine, and results land in buffers that the program keeps.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from specseqplusplus_b200 import Engine, Params, gen
from specseqplusplus_b200.engine import reduce_noalloc

_engine = None


def _the_engine():
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


# What a program passes to reduce(): the reference's defaults, the benchmark's
# setting for grids, the 100,000-point configuration's (edge collapse and guided
# clearing), and what the autotuner settles on for batches of Rips complexes.
_PARAMS = {
    "default": {},
    "grid": {"model": 1, "max_iteration": 10, "level1_capacity": 32, "level2_capacity": 8192},
    "collapse": {"model": 3, "max_iteration": 100, "level1_capacity": 100, "level2_capacity": 250},
    "tuned": {"ss_block_size": 1 << 30, "growth": 1.0, "level1_capacity": 64, "level2_capacity": 8192},
}


def _params(case) -> Params:
    return Params(**_PARAMS[case["params"]], dualize=case.get("dualize", 0),
                  representatives=case.get("representatives", 0))


def _radius(npts: int, space_dim: int, degree: float) -> float:
    return gen.rips_radius_for_degree(npts, space_dim, degree)


def _cloud(npts: int, space_dim: int, seed: int) -> np.ndarray:
    return np.random.default_rng(seed).random((npts, space_dim), dtype=np.float32)


def _field(gx: int, gy: int, gz: int, sigma: float, seed: int) -> torch.Tensor:
    """Gaussian noise smoothed by a Gaussian of `sigma` voxels, [gz, gy, gx] on the GPU (element-wise sums in
    64 bits, so that the same seed gives the same field)."""
    f = torch.from_numpy(np.random.default_rng(seed).standard_normal((gz, gy, gx))).cuda()
    half = int(4 * sigma + 0.5)
    for axis in range(3):
        n = f.shape[axis]
        at = torch.arange(n, device=f.device)
        out = torch.zeros_like(f)
        for k in range(-half, half + 1):
            i = (at + k) % (2 * n)  # reflected at both ends
            out += math.exp(-0.5 * (k / sigma) ** 2) * f.index_select(axis, torch.where(i < n, i, 2 * n - 1 - i))
        f = out
    f = (f / f.std()).float().contiguous()
    torch.cuda.synchronize()  # the engine reads it on a stream of its own
    return f


def _matrix(case, seed: int):
    """The boundary matrix of the case's complex, in host memory."""
    e = _the_engine()
    if case["kind"] == "grid":
        e.load_lowerstar(_field(case["gx"], case["gy"], case["gz"], case["sigma"], seed), 3)
    else:
        r = _radius(case["npts"], case["space_dim"], case["degree"])
        e.load_rips(_cloud(case["npts"], case["space_dim"], seed), r, case["maxdim"])
    return e.input_matrix()


def _batch(case, seed: int) -> list:
    """Point clouds of uneven size: log-uniform in 200-5,000 points, half in the plane (dimension <= 2), half in
    space (dimension <= 3), mean degree 8-40."""
    out = []
    for i in range(case["count"]):
        # the sizes are the case's, the points the seed's
        size = np.random.default_rng(4_000_012 + i)
        n = int(round(math.exp(size.uniform(math.log(200), math.log(5000)))))
        d = 2 if i % 2 == 0 else 3
        out.append(("rips", _cloud(n, d, seed * 1_000_003 + i), _radius(n, d, float(size.uniform(8.0, 40.0))), d))
    return out


def _columns(case) -> int:
    """Columns of the case's complex: a grid's exactly, a cloud's as an upper bound (half as many again as uniform
    points without a border would give, for the mean numbers of cliques in a ball of `degree` neighbours)."""
    if case["kind"] == "grid":
        g = [case["gx"], case["gy"], case["gz"]]
        total = 1
        for steps, ways in (((1, 0, 0), 1), ((0, 1, 0), 1), ((0, 0, 1), 1), ((1, 1, 0), 3), ((1, 0, 1), 3),
                            ((0, 1, 1), 3), ((1, 1, 1), 13)):
            # chains of vertices from (0, 0, 0) to `steps`: 1 over one axis, 3 over two, 13 over three
            total += ways * math.prod(n - k for n, k in zip(g, steps))
        return total + math.prod(g) - 1
    d, k = case["space_dim"], case["degree"]
    three, four = (0.59, 0.3) if d == 2 else (0.47, 0.15)
    per_point = 1 + k / 2 + three * k * k / 6 + (four * k ** 3 / 24 if case["maxdim"] >= 3 else 0)
    return int(1.5 * case["npts"] * per_point) + 1000


def _buffers(columns: int, essentials: int, pinned: bool):
    """Room for the results: a column is in one pair at most."""
    return [torch.full((n,), -1, dtype=torch.int64, pin_memory=pinned).numpy()
            for n in (2 * (columns // 2), essentials)]


def listed() -> list[dict]:
    return [
        # the smallest requests, where launches and synchronisations count: the smoke test's complex, and the
        # 2,000-point configuration with the reference's defaults (radius 0.08), from host arrays
        {"name": "rips 400 host", "kind": "rips", "npts": 400, "space_dim": 3, "degree": 9.77, "maxdim": 3,
         "source": "host", "params": "default"},
        {"name": "rips 2000 host", "kind": "rips", "npts": 2000, "space_dim": 3, "degree": 4.29, "maxdim": 3,
         "source": "host", "params": "default"},
        # an ordinary point cloud in the plane, built on the device, reduced as cohomology
        {"name": "cloud 5000 dual", "kind": "rips", "npts": 5000, "space_dim": 2, "degree": 24.0, "maxdim": 2,
         "source": "input", "params": "default", "dualize": 1},
        # a small point cloud in space whose representative cycles are wanted afterwards
        {"name": "cloud 1200 cycles", "kind": "rips", "npts": 1200, "space_dim": 3, "degree": 16.0, "maxdim": 3,
         "source": "input", "params": "default", "representatives": 1},
        # the largest point clouds of the serving mix (mean degree 24), as a matrix already on the device
        {"name": "rips 20000 mode 2", "kind": "rips", "npts": 20000, "space_dim": 3, "degree": 24.0, "maxdim": 3,
         "source": "device", "params": "tuned", "dualize": 2},
        # the 100,000-point configuration (radius 0.016): edge collapse and guided clearing
        {"name": "rips 100000 collapse", "kind": "rips", "npts": 100000, "space_dim": 3, "degree": 1.716, "maxdim": 3,
         "source": "device", "params": "collapse"},
        # scalar fields: a small ragged one built on the device, a middle one from host arrays, the benchmark's
        # 64^3 on the device, and the largest of the serving mix with the reference's defaults
        {"name": "field 21x24x19", "kind": "grid", "gx": 21, "gy": 24, "gz": 19, "sigma": 1.5, "source": "input",
         "params": "default"},
        {"name": "grid 32 host", "kind": "grid", "gx": 32, "gy": 32, "gz": 32, "sigma": 2.0, "source": "host",
         "params": "default"},
        {"name": "grid 64", "kind": "grid", "gx": 64, "gy": 64, "gz": 64, "sigma": 2.0, "source": "device",
         "params": "grid"},
        {"name": "grid 93", "kind": "grid", "gx": 93, "gy": 93, "gz": 93, "sigma": 2.5, "source": "device",
         "params": "default"},
        # a batch of uneven point clouds, built and reduced together
        {"name": "batch 64", "kind": "batch", "count": 64, "params": "tuned", "dualize": 2},
        # the call that allocates nothing, for callers that own all of the device's memory
        {"name": "rips 700 noalloc", "kind": "noalloc", "npts": 700, "space_dim": 3, "degree": 8.0, "maxdim": 3},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["rips", "rips", "grid", "grid", "collapse", "batch", "noalloc"])
    if kind == "grid":
        g = _log(rng, 16, 80)
        size = [max(3, round(g * rng.uniform(0.8, 1.2))) for _ in range(3)]
        return {"kind": "grid", "gx": size[0], "gy": size[1], "gz": size[2], "sigma": round(rng.uniform(1.0, 3.0), 2),
                "source": rng.choice(["host", "input", "device"]), "params": rng.choice(["default", "grid", "tuned"])}
    if kind == "batch":
        return {"kind": "batch", "count": _log(rng, 8, 64), "params": "tuned", "dualize": rng.choice([0, 2])}
    if kind == "noalloc":
        return {"kind": "noalloc", "npts": _log(rng, 200, 2000), "space_dim": 3,
                "degree": round(rng.uniform(4.0, 10.0), 2), "maxdim": 3}
    d = rng.choice([2, 3])
    if kind == "collapse":
        n = _log(rng, 1000, 100000)
        return {"kind": "rips", "npts": n, "space_dim": d, "maxdim": 3, "params": "collapse",
                "degree": round(rng.uniform(1.5, 2.5 if n > 20000 else 8.0), 2), "source": rng.choice(["input", "device"])}
    n = _log(rng, 300, 20000)
    case = {"kind": "rips", "npts": n, "space_dim": d, "degree": round(rng.uniform(8.0, 24.0), 2), "maxdim": d,
            "source": rng.choice(["host", "input", "device"]), "params": rng.choice(["default", "tuned"]),
            "dualize": rng.choice([0, 1, 2] if n <= 5000 else [0, 2])}
    if n <= 5000 and case["dualize"] == 0:
        case["representatives"] = rng.choice([0, 1])
    return case


def prepare(case, seed):
    s = {"case": case, "engine": _the_engine()}
    if case["kind"] == "batch":
        s["requests"] = _batch(case, seed)
        s["params"] = _params(case)
        columns = sum(_columns({"kind": "rips", "npts": len(p), "space_dim": d, "maxdim": d,
                                "degree": len(p) * r ** d * (math.pi if d == 2 else 4 * math.pi / 3)})
                      for _, p, r, d in s["requests"])
        s["pairs"], s["essentials"] = _buffers(columns, columns, False)
        return s
    if case["kind"] == "noalloc":
        m = _matrix(dict(case, kind="rips"), seed)
        s["device"] = [torch.from_numpy(x).cuda() for x in (m.dims, m.col_ptr, m.rows)]
        s["size"] = (m.ncols, m.nnz)
        s["pairs"] = torch.full((_columns(case), 2), -1, dtype=torch.int64, device="cuda")
        s["npairs"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        return s
    s["params"] = _params(case)
    columns = _columns(case)
    # a grid is contractible: one essential vertex
    s["pairs"], s["essentials"] = _buffers(columns, 1 if case["kind"] == "grid" else columns,
                                           case["source"] == "device")
    if case["source"] == "input":
        if case["kind"] == "grid":
            s["input"] = _field(case["gx"], case["gy"], case["gz"], case["sigma"], seed)
        else:
            s["input"] = torch.from_numpy(_cloud(case["npts"], case["space_dim"], seed)).cuda()
            s["radius"] = _radius(case["npts"], case["space_dim"], case["degree"])
        return s
    m = _matrix(case, seed)
    if case["source"] == "host":
        s["host"] = m
    else:
        s["device"] = [torch.from_numpy(x).cuda() for x in (m.dims, m.col_ptr, m.rows)]
        s["ncols"] = m.ncols
    return s


def run(s):
    case, e = s["case"], s["engine"]
    if case["kind"] == "noalloc":
        d = s["device"]
        reduce_noalloc(*s["size"], d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr(), s["pairs"].data_ptr(),
                       s["npairs"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return {"pairs": s["pairs"], "npairs": s["npairs"]}
    if case["kind"] == "batch":
        e.load_built_batch(s["requests"])
        e.reduce(s["params"])
        at = [0, 0]
        counts = np.zeros((case["count"], 2), dtype=np.int64)
        for i, (pairs, essentials) in enumerate(e.batch_results()):  # one table of all complexes' results
            s["pairs"][at[0]:at[0] + pairs.size] = pairs.reshape(-1)
            s["essentials"][at[1]:at[1] + essentials.size] = essentials
            at = [at[0] + pairs.size, at[1] + essentials.size]
            counts[i] = len(pairs), len(essentials)
        return {"pairs": s["pairs"], "essentials": s["essentials"], "counts": counts}
    if case["source"] == "input":
        if case["kind"] == "grid":
            e.load_lowerstar(s["input"], 3)
        else:
            e.load_rips(s["input"], s["radius"], case["maxdim"])
    elif case["source"] == "host":
        e.load_csc(s["host"])
    else:
        d = s["device"]
        e.load_csc_device(s["ncols"], d[0].data_ptr(), d[1].data_ptr(), d[2].data_ptr())
    e.reduce(s["params"])
    e.pairs(s["pairs"])
    e.essentials(s["essentials"])
    return {"pairs": s["pairs"], "essentials": s["essentials"]}


def work(case):
    """The input as it is handed over, read once, and the results, written once; no floating-point work."""
    s = prepare(case, 1)
    given = list(s.get("device", ()))
    if "host" in s:
        given += [s["host"].dims, s["host"].col_ptr, s["host"].rows]
    if "input" in s:
        given.append(s["input"])
    given += [r[1] for r in s.get("requests", ())]
    got = sum(8 * int((x != -1).sum()) for x in run(s).values())  # what was written of the buffers
    return {"bytes": float(sum(x.nbytes for x in given) + got), "flops": 0.0}


def exact(case, seed):
    return None  # pairs and essentials are whole numbers: they stay equal
