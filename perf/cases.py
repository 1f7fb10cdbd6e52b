"""The work a user has this library do, as timed cases.

A case is one call of a public entry point on one set of inputs:

  wrapper  VariantDBSCAN(eps, minpts, x, y): the drop-in for the reference's
           Python function (host arrays in, host labels out)
  replay   Context.run_device(graph=True): the same dataset shape again and
           again, replayed as one CUDA graph
  noalloc  vdb_run_noalloc: one variant in device memory, nothing allocated
  batch    Context.run on many datasets of uneven sizes (host arrays)
  request  Context.run(table="border"): one request of a serving loop, labels
           only, host arrays, a table budget per worker
  device   Context.run_device: one dataset already on the device

Point sets follow the benchmark workloads (variantdbscan_gb300.synthetic):
longitude [0, 360), latitude [-90, 90], Gaussian blobs plus uniform
background, optionally on a 0.01 degree lattice.  They are drawn on the GPU so
that millions of points take no time to make.

Outputs are labels (whole numbers, one per point and variant) and the counts
of neighbour pairs and clusters: all of them integers that have to come out
equal, so no output has a 64-bit reference value to be near to.
"""
import ctypes
import math

import numpy as np
import torch

import variantdbscan_gb300 as v

SWEEP = "0.1,0.2,0.4,0.8"
SWEEP_MINPTS = "4,16,64,256"


def _case(name, api, n, points, eps, minpts, **more):
    c = {"name": name, "api": api, "n": n, "points": points, "eps": eps, "minpts": minpts,
         "mbb": 70, "table": "all", "precision": "mixed", "budget_mib": 0, "datasets": 1}
    c.update(more)
    return c


def listed():
    return [
        # smallest call: a few thousand points (the size of the test fixtures),
        # one variant; launches and waits are all there is
        _case("wrapper_3k", "wrapper", 3001, "single", "0.5", "10"),
        # the plain single-variant workload of the benchmark
        _case("wrapper_50k", "wrapper", 50000, "single", "0.5", "10"),
        # the same, resident on the device and called over and over
        _case("replay_50k", "replay", 50000, "single", "0.5", "10"),
        # latency-bound callers that may not allocate
        _case("noalloc_20k", "noalloc", 20000, "single", "0.5", "10"),
        # a parameter scan over a small dataset: 16 variants in one call
        _case("wrapper_60k_x16", "wrapper", 60013, "sweep", SWEEP, SWEEP_MINPTS),
        # uneven datasets in one call (the multi-dataset batch, its lower sizes)
        _case("batch_24", "batch", 200000, "mixture", "0.05:1.5", "4:128", datasets=24),
        # one request of the serving loop: labels only, many variants
        _case("request_400k_x12", "request", 400009, "mixture", "0.05:1.5", "4:128",
              table="border", budget_mib=19200, variants=12),
        # every distance in FP64, for callers that want no FP32 filter
        _case("fp64_100k", "device", 100003, "sweep", SWEEP, "4,64", precision="fp64"),
        # sparse data: a few points per cell, no blobs
        _case("uniform_1m", "device", 999983, "uniform", "0.05,0.1,0.2", "3,6"),
        # points on a 0.01 degree lattice (many pairs at exactly eps), tables
        # built in row chunks under a budget
        _case("lattice_2m", "device", 2000000, "lattice", "0.05,0.1,0.25,0.5", "8,32",
              budget_mib=4096),
        # the variant sweep with every table row written
        _case("sweep_1m", "device", 1000000, "sweep", SWEEP, SWEEP_MINPTS),
        # the full variant sweep, labels only
        _case("labels_2m", "device", 2000000, "sweep", SWEEP, SWEEP_MINPTS, table="border"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed ranges: any entry point, sizes log-uniform."""
    api = rng.choice(["wrapper", "wrapper", "replay", "noalloc", "batch", "request", "device",
                      "device", "device"])
    eps1 = "%.3g" % math.exp(rng.uniform(math.log(0.1), math.log(0.8)))
    mp1 = str(rng.randint(4, 64))
    if api == "wrapper":
        if rng.random() < 0.5:
            return _unnamed(api, _log_int(rng, 1000, 200000), "single", eps1, mp1,
                            mbb=rng.choice([1, 10, 70]))
        return _unnamed(api, _log_int(rng, 5000, 200000), "sweep", SWEEP, SWEEP_MINPTS)
    if api == "replay":
        return _unnamed(api, _log_int(rng, 3000, 200000), "single", eps1, mp1)
    if api == "noalloc":
        return _unnamed(api, _log_int(rng, 1000, 24000), "single", "0.5", mp1)
    if api == "batch":
        return _unnamed(api, _log_int(rng, 30000, 200000), "mixture", "0.05:1.5", "4:128",
                        datasets=rng.randint(4, 32))
    if api == "request":
        return _unnamed(api, _log_int(rng, 20000, 800000), "mixture", "0.05:1.5", "4:128",
                        table="border", budget_mib=19200, variants=rng.randint(1, 16))
    points = rng.choice(["sweep", "uniform", "lattice", "mixture"])
    if points == "uniform":
        return _unnamed(api, _log_int(rng, 50000, 1500000), points, "0.05,0.1,0.2", "3,6")
    if points == "lattice":
        return _unnamed(api, _log_int(rng, 50000, 2000000), points, "0.05,0.1,0.25,0.5", "8,32",
                        budget_mib=4096)
    if points == "mixture":
        return _unnamed(api, _log_int(rng, 20000, 600000), points, "0.05:1.5", "4:128",
                        variants=rng.randint(1, 12))
    if rng.random() < 0.3:
        return _unnamed(api, _log_int(rng, 20000, 200000), points, SWEEP, "4,64",
                        precision="fp64")
    table = rng.choice(["all", "border"])
    return _unnamed(api, _log_int(rng, 50000, 1000000), points, SWEEP, SWEEP_MINPTS, table=table)


def _unnamed(*a, **k):
    c = _case("", *a, **k)
    del c["name"]
    return c


# --------------------------------------------------------------------- inputs

def _shape(points, rng):
    """Blob weights, their sigma range, background share and lattice step."""
    if points == "single":
        return np.full(8, 1 / 8), 0.5, 3.0, 0.20, 0
    if points == "sweep":
        return rng.dirichlet(np.ones(64)), 0.2, 2.0, 0.10, 0
    if points == "lattice":
        return np.full(256, 1 / 256), 0.05, 0.5, 0.30, 100
    if points == "mixture":
        nb = int(rng.integers(4, 33))
        return np.full(nb, 1 / nb), 0.2, 3.0, float(rng.uniform(0.05, 0.30)), 0
    return np.zeros(1), 1.0, 1.0, 1.0, 0


def _points(n, points, seed):
    rng = np.random.default_rng(seed)
    w, lo, hi, bg, steps = _shape(points, rng)
    nb = len(w)
    c = torch.from_numpy(np.stack([rng.uniform(0, 360, nb), rng.uniform(-90, 90, nb),
                                   rng.uniform(lo, hi, nb)])).cuda()
    g = torch.Generator(device="cuda")
    g.manual_seed(int(rng.integers(1 << 31)))
    u = torch.rand((3, n), generator=g, device="cuda", dtype=torch.float64)
    x, y = u[0] * 360, u[1] * 180 - 90
    if bg < 1.0:
        edges = torch.from_numpy(np.cumsum(w)).cuda()
        which = torch.searchsorted(edges, torch.rand(n, generator=g, device="cuda",
                                                     dtype=torch.float64)).clamp_(max=nb - 1)
        z = torch.randn((2, n), generator=g, device="cuda", dtype=torch.float64)
        s = c[2][which]
        blob = u[2] >= bg
        x = torch.where(blob, torch.remainder(c[0][which] + z[0] * s, 360.0), x)
        y = torch.where(blob, (c[1][which] + z[1] * s).clamp_(-90, 90), y)
    if steps:
        x = torch.round(x * steps) / steps
        y = torch.round(y * steps) / steps
        x = torch.where(x >= 360, x - 360, x)
    return x.contiguous(), y.contiguous()


def _sizes(case):
    """Points and variants of a batch's datasets: sizes evenly spread in the
    logarithm over [10000, n], 4 to 12 variants."""
    k, top = case["datasets"], math.log(case["n"] / 10000)
    return [(int(10000 * math.exp(top * (i + 0.5) / k)) | 1, 4 + 5 * i % 9) for i in range(k)]


def _variants(case, rng, nv=0):
    """(eps, minpts): the grid of two lists, or random ones for "lo:hi" ranges."""
    if ":" in case["eps"]:
        lo, hi = (float(t) for t in case["eps"].split(":"))
        a, b = (int(t) for t in case["minpts"].split(":"))
        nv = nv or int(case["variants"])
        return (np.exp(rng.uniform(math.log(lo), math.log(hi), nv)),
                rng.integers(a, b + 1, nv).astype(np.uint32))
    eps = [float(t) for t in case["eps"].split(",")]
    mp = [int(t) for t in case["minpts"].split(",")]
    e, m = np.meshgrid(eps, mp, indexing="ij")
    return e.ravel().astype(np.float64), m.ravel().astype(np.uint32)


def _noalloc():
    lib = v.load_library()
    fn = lib.vdb_run_noalloc
    fn.restype = ctypes.c_int
    fn.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_uint32, ctypes.c_double,
                   ctypes.c_uint32, ctypes.c_int32, ctypes.c_void_p, ctypes.c_void_p]
    return fn


def prepare(case, seed):
    rng = np.random.default_rng([seed, 77])
    api, n = case["api"], case["n"]
    s = {"case": case}
    if api == "batch":
        items = []
        for i, (m, nv) in enumerate(_sizes(case)):
            x, y = _points(m, case["points"], [seed, i])
            items.append(v.BatchItem(x.cpu().numpy(), y.cpu().numpy(),
                                     *_variants(case, rng, nv), mbb_size=case["mbb"]))
        s.update(items=items, ctx=v.Context())
        return s
    x, y = _points(n, case["points"], [seed, 0])
    eps, mp = _variants(case, rng)
    s.update(eps=eps, minpts=mp)
    if api in ("wrapper", "request"):
        s.update(x=x.cpu().numpy(), y=y.cpu().numpy())
        if api == "request":
            s.update(ctx=v.Context())
        return s
    s.update(x=x, y=y, labels=torch.zeros((len(eps), n), dtype=torch.int32, device="cuda"))
    if api == "noalloc":
        s.update(fn=_noalloc())
    else:
        s.update(ctx=v.Context())
    torch.cuda.synchronize()  # the library's own streams read these
    return s


def _host(labels):
    return labels.view(np.int32)


def _counts(st):
    return {"pairs": int(st["pairs"]), "clusters": int(st["clusters"])}


def run(state):
    c = state["case"]
    api = c["api"]
    if api == "wrapper":
        return _host(v.VariantDBSCAN(state["eps"], state["minpts"], state["x"], state["y"],
                                     c["mbb"]))
    if api == "noalloc":
        rc = state["fn"](state["x"].data_ptr(), state["y"].data_ptr(), c["n"],
                         float(state["eps"][0]), int(state["minpts"][0]), c["mbb"],
                         state["labels"].data_ptr(), None)
        if rc != v.VDB_OK:
            raise v.VDBError(rc)
        return state["labels"]
    if api == "batch":
        out, st = state["ctx"].run(state["items"])
        return {"labels": [_host(t) for t in out], **_counts(st)}
    if api == "request":
        item = v.BatchItem(state["x"], state["y"], state["eps"], state["minpts"], c["mbb"])
        out, st = state["ctx"].run([item], budget=c["budget_mib"] << 20, streams=1,
                                   table=c["table"])
        return {"labels": _host(out[0]), **_counts(st)}
    st = state["ctx"].run_device(state["x"].data_ptr(), state["y"].data_ptr(), c["n"],
                                 state["eps"], state["minpts"], state["labels"].data_ptr(),
                                 mbb_size=c["mbb"], precision=c["precision"],
                                 budget=c["budget_mib"] << 20, table=c["table"],
                                 graph=api == "replay")
    return {"labels": state["labels"], **_counts(st)}


# ----------------------------------------------------------------------- work

def _pairs(n, points, eps):
    """Expected neighbour pairs (self included) of one epsilon: points of one
    Gaussian blob are within eps with probability 1 - exp(-eps^2 / 4 sigma^2);
    all others are taken as uniform over the box."""
    w2 = {"single": 1 / 8, "sweep": 2 / 65, "lattice": 1 / 256, "mixture": 1 / 13,
          "uniform": 0.0}[points]
    lo, hi, bg = {"single": (0.5, 3.0, 0.2), "sweep": (0.2, 2.0, 0.1),
                  "lattice": (0.05, 0.5, 0.3), "mixture": (0.2, 3.0, 0.175),
                  "uniform": (1.0, 1.0, 1.0)}[points]
    sig = np.linspace(lo, hi, 64)
    same = (1 - bg) ** 2 * w2
    near = float(np.mean(1 - np.exp(-eps * eps / (4 * sig * sig))))
    return n + float(n) * n * (same * near + (1 - same) * math.pi * eps * eps / (360 * 180))


def work(case):
    """Coordinates in, labels out, and the neighbour tables' 16-bit entries
    where the call has every row written (32-bit for noalloc); five
    operations for the distance of each pair within eps."""
    ranges = ":" in case["eps"]
    if case["api"] == "batch":
        sets = _sizes(case)
    else:
        sets = [(case["n"], case["variants"] if ranges else
                 len(case["eps"].split(",")) * len(case["minpts"].split(",")))]
    entry = 0 if case["table"] == "border" else 4 if case["api"] == "noalloc" else 2
    b = f = 0.0
    for m, nv in sets:
        if ranges:  # every variant has an epsilon of its own
            lo, hi = (float(t) for t in case["eps"].split(":"))
            eps = [lo * (hi / lo) ** ((i + 0.5) / nv) for i in range(nv)]
        else:
            eps = [float(t) for t in case["eps"].split(",")]
        p = sum(_pairs(m, case["points"], e) for e in eps)
        b += 16 * m + 4 * m * nv + entry * p
        f += 5 * p / 2
    return {"bytes": b, "flops": f}


def exact(case, seed):
    """Every output is a whole number (see above)."""
    return None
