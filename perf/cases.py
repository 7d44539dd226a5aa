"""Performance cases of the sketch-ingest and connectivity-query path: what users of this package
have it do, through its public entry points.

    listed()             the cases that are measured by name
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  the inputs and handles a program has in hand before the call
    run(state)           one pass: the calls a program makes, and what they answer
    work(case)           bytes one pass cannot do without

Every output is whole numbers or bytes (labels, component counts, rounds, sketch bytes), so two
implementations agree exactly or not at all; there is no value of a computed real number.

Kinds of cases:
  stream    a new graph stream is sketched from empty sketches and queried once at its end
  segment   a stream goes on: a segment of updates is folded into a live handle, then queried.
            An update is a toggle, so a second pass over the same state takes the segment out again
  point     the smallest request: a few updates from host memory, then one pair's connectivity
  driver    GraphSketchDriver over a stream held in host memory, as a reference program uses it
  batches   the reference's worker contract: one apply_update_batch call per vertex
  noalloc   records folded into sketches that the caller owns, without allocation
  many      many independent graphs through one batch handle
  serving   one tick of the tenant server: update batches of many tenants, then some queries
"""
import ctypes
import math

import numpy as np
import torch

import graphzeppelin_b200 as gz
from graphzeppelin_b200 import _lib
from graphzeppelin_b200.serve import SketchServer

SKETCH_SEED = 0x5EED5EED


def listed():
    return [
        # a service answers "are a and b connected" right after a handful of updates
        dict(name="point_v1024", kind="point", vertices=1024, base=20000, records=16, graph="planted",
             components=8),
        # the reference's test fixture size (1024 vertices, 8,528 updates) through the driver
        dict(name="driver_v1024", kind="driver", vertices=1024, records=8528, graph="planted",
             components=8),
        # worker threads of a host gutter hand over one batch per vertex
        dict(name="batches_v2048", kind="batches", vertices=2048, records=600000, graph="planted",
             components=16),
        # a live graph takes a request-sized batch from host memory and is queried
        dict(name="segment_v65536", kind="segment", vertices=65536, base=1000000, records=4096,
             graph="powerlaw", source="host"),
        # an ordinary sparse graph of a size that is no power of two, records in device memory
        dict(name="stream_v50021", kind="stream", vertices=50021, records=3000017, graph="planted",
             components=37, source="device"),
        # the benchmark's dense stream: 2^17 vertices, about 1.4e8 updates in device memory
        dict(name="stream_v131072", kind="stream", vertices=131072, records=140000000, graph="planted",
             components=64, source="device"),
        # the same vertices fed from page-locked host memory, a quarter of that stream
        dict(name="host_v131072", kind="stream", vertices=131072, records=36000001, graph="planted",
             components=64, source="host"),
        # a large power-law graph with a query after each tenth of its stream: the second tenth
        dict(name="segment_v1048576", kind="segment", vertices=1048576, base=12800000, records=12800000,
             graph="powerlaw", source="device"),
        # CubeSketch, the reference's other sketch (its L0_SAMPLING build)
        dict(name="cube_v5003", kind="stream", vertices=5003, records=1000003, graph="planted",
             components=11, source="device", algorithm="cube"),
        # a plugin that owns its sketches folds a chunk of records into them
        dict(name="noalloc_v50000", kind="noalloc", vertices=50000, base=2000000, records=1500001,
             graph="powerlaw"),
        # many graphs of uneven size (a tenth to a quarter of the benchmark's batch)
        dict(name="many_g128", kind="many", graphs=128, log2_v_min=8.0, log2_v_max=16.0, degree_min=8.0,
             degree_max=256.0),
        # one serving tick: 17 tenants' update batches (about 2^19 records), four of them queried
        dict(name="serving_t17", kind="serving", tenants=17, queried=4, log2_v_min=10.0, log2_v_max=18.0,
             records=524288),
    ]


def draw(rng):
    def log(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["point", "driver", "batches", "segment", "segment", "stream", "stream", "stream",
                       "cube", "noalloc", "many", "serving"])
    if kind == "point":
        v = log(64, 1 << 17)
        return dict(kind=kind, vertices=v, base=min(20 * v, 2000000), records=log(1, 256),
                    graph=rng.choice(["planted", "powerlaw"]), components=rng.randint(1, 8))
    if kind == "driver":
        v = log(300, 32768)
        return dict(kind=kind, vertices=v, records=v * rng.randint(4, 32) + rng.randint(0, 99),
                    graph=rng.choice(["planted", "powerlaw"]), components=rng.randint(1, 16))
    if kind == "batches":
        v = log(512, 8192)
        return dict(kind=kind, vertices=v, records=v * rng.randint(16, 300) + rng.randint(0, 99),
                    graph="planted", components=rng.randint(1, 16))
    if kind == "segment":
        v = log(4096, 1 << 20)
        return dict(kind=kind, vertices=v, base=v * rng.randint(4, 20), records=log(1024, 12 * v + 2048),
                    graph="powerlaw", source=rng.choice(["host", "device"]))
    if kind in ("stream", "cube"):
        v = log(1024, 1 << 18) if kind == "stream" else log(512, 8192)
        per = rng.uniform(math.log(6), math.log(500 if kind == "stream" else 200))
        c = dict(kind="stream", vertices=v, records=min(int(v * math.exp(per)), 60000000, v * (v - 1) // 4),
                 graph=rng.choice(["planted", "planted", "powerlaw"]), components=rng.randint(1, 64),
                 source=rng.choice(["host", "device", "device"]))
        if kind == "cube":
            c["algorithm"] = "cube"
        return c
    if kind == "noalloc":
        return dict(kind=kind, vertices=log(1000, 200000), base=log(1000, 2000000),
                    records=log(1000, 1 << 21), graph=rng.choice(["planted", "powerlaw"]),
                    components=rng.randint(1, 16))
    if kind == "many":
        lo = rng.uniform(6, 10)
        return dict(kind=kind, graphs=log(8, 160), log2_v_min=lo, log2_v_max=lo + rng.uniform(2, 6),
                    degree_min=8.0, degree_max=rng.uniform(16, 256))
    t = rng.randint(2, 40)
    return dict(kind="serving", tenants=t, queried=rng.randint(1, min(t, 8)),
                log2_v_min=rng.uniform(8, 11), log2_v_max=rng.uniform(14, 18), records=log(2000, 1 << 21))


# ------------------------------------------------------------------------------------------------
# inputs, made on the GPU
# ------------------------------------------------------------------------------------------------

def _pack(u, v, kind):
    """Packed 9-byte records {u8 type, u32 src, u32 dst} as a flat uint8 tensor on the GPU."""
    n = u.numel()
    out = torch.empty((n, 9), dtype=torch.uint8, device="cuda")
    out[:, 0] = kind
    out[:, 1:5] = u.to(torch.int32).view(torch.uint8).view(n, 4)
    out[:, 5:9] = v.to(torch.int32).view(torch.uint8).view(n, 4)
    return out.view(-1)


def _rand(gen, n):
    return torch.rand(n, generator=gen, device="cuda", dtype=torch.float64)


def _flip(gen, u, v):
    swap = torch.rand(u.numel(), generator=gen, device="cuda") < 0.5
    return torch.where(swap, v, u), torch.where(swap, u, v)


def _planted(gen, vertices, components, n):
    """n updates of a planted-components graph: the inserts of distinct edges inside the components
    (about 5 in 6 updates), and random pairs inserted and later deleted again, shuffled."""
    used = vertices - vertices // 50  # an id space has gaps: some ids have no edge that stays
    k = max(1, min(components, vertices // 4))
    churn = n // 12
    edges = n - 2 * churn
    extra = used - 2 * k
    cuts = torch.sort((_rand(gen, k - 1) * (extra + 1)).long())[0]
    ends = torch.cat([cuts, torch.tensor([extra], device="cuda")])
    sizes = torch.diff(ends, prepend=torch.zeros(1, dtype=torch.long, device="cuda")) + 2
    first = torch.cumsum(sizes, 0) - sizes
    perm = torch.randperm(vertices, generator=gen, device="cuda")
    pairs = sizes * (sizes - 1) // 2
    upto = torch.cumsum(pairs, 0)
    total = int(upto[-1])
    if edges < total < 5 * edges:  # dense: distinct pairs, each with the same chance
        p = min(1.0, edges / total * 1.002 + 100.0 / total)
        idx = torch.nonzero(torch.rand(total, generator=gen, device="cuda") < p).view(-1)
        idx = idx[torch.randperm(idx.numel(), generator=gen, device="cuda")[:edges]]
    else:  # sparse: hardly any pair is drawn twice (where one is, its second update deletes it)
        idx = (_rand(gen, edges) * total).long()
    if idx.numel() < edges:
        idx = torch.cat([idx, (_rand(gen, edges - idx.numel()) * total).long()])
    comp = torch.searchsorted(upto, idx, right=True)
    local = idx - (upto - pairs)[comp]
    hi = ((1.0 + torch.sqrt(1.0 + 8.0 * local.double())) / 2.0).long()
    hi -= (hi * (hi - 1) // 2 > local).long()
    hi += ((hi + 1) * hi // 2 <= local).long()
    lo = local - hi * (hi - 1) // 2
    eu, ev = perm[first[comp] + lo], perm[first[comp] + hi]
    cu = (_rand(gen, churn) * vertices).long()
    cv = (cu + 1 + (_rand(gen, churn) * (vertices - 1)).long()) % vertices
    u, v = _flip(gen, torch.cat([eu, cu, cu]), torch.cat([ev, cv, cv]))
    at = torch.randperm(n, generator=gen, device="cuda")
    kind = torch.zeros(n, dtype=torch.uint8, device="cuda")
    kind[torch.maximum(at[edges:edges + churn], at[edges + churn:])] = 1
    su, sv = torch.empty_like(u), torch.empty_like(v)
    su[at], sv[at] = u, v
    return _pack(su, sv, kind)


def _powerlaw(gen, vertices, n, exponent=2.1, cap=16384.0):
    """n updates of a Chung-Lu power-law graph: both endpoints drawn by weight (rank)^(-1/(exponent-1)),
    no vertex above `cap` expected updates; repeated pairs toggle."""
    used = vertices - vertices // 50  # an id space has gaps
    w = torch.arange(1, used + 1, device="cuda", dtype=torch.float64) ** (-1.0 / (exponent - 1.0))
    for _ in range(8):
        w = torch.clamp(w * (2.0 * n / w.sum()), max=max(cap, 4.0 * n / used))
    cdf = torch.cumsum(w, 0)
    cdf /= cdf[-1].clone()
    ids = torch.randperm(vertices, generator=gen, device="cuda")
    a = torch.searchsorted(cdf, _rand(gen, n), right=True).clamp(max=used - 1)
    b = torch.searchsorted(cdf, _rand(gen, n), right=True).clamp(max=used - 1)
    u, v = ids[a], ids[torch.where(a == b, (b + 1) % used, b)]
    kind = (torch.rand(n, generator=gen, device="cuda") < 0.15).to(torch.uint8)
    return _pack(u, v, kind)


def _records(case, gen, n):
    if case["graph"] == "planted":
        return _planted(gen, case["vertices"], case["components"], n)
    return _powerlaw(gen, case["vertices"], n)


def _pinned(records):
    out = torch.empty(records.numel(), dtype=torch.uint8, pin_memory=True)
    out.copy_(records)
    return out


def _handle(case, seed):
    return gz.CCSketchAlg(case["vertices"], SKETCH_SEED + seed,
                          sketch_algorithm=case.get("algorithm", "cameo"))


def _spread(n, step):
    """n numbers spread evenly over [0, 1) in a mixed order (the same for every seed)."""
    return (0.5 + np.arange(n) * step) % 1.0


def _sizes(case, n):
    """Vertices per graph or tenant: log-uniform over the case's range."""
    lo, hi = case["log2_v_min"], case["log2_v_max"]
    return np.exp2(lo + (hi - lo) * _spread(n, 0.6180339887)).astype(np.int64)


def _many_counts(case, sizes):
    """Updates per graph: a mean degree uniform over the case's range, and a tenth of churn."""
    lo, hi = case["degree_min"], case["degree_max"]
    degree = lo + (hi - lo) * _spread(sizes.size, 0.7548776662)
    return np.maximum(16, sizes * degree / 2 * 1.2).astype(np.int64)


def _serving_counts(case):
    """Updates per tenant: request batches of 1k to 64k records, scaled to the tick's total."""
    share = 1 / 64 + (1 - 1 / 64) * _spread(case["tenants"], 0.7548776662)
    return np.maximum(1, case["records"] * share / share.sum()).astype(np.int64)


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    s = {"kind": kind}
    if kind in ("stream", "segment", "point"):
        s["alg"] = alg = _handle(case, seed)
        if case.get("base"):
            base = _records(case, gen, case["base"])
            torch.cuda.synchronize()
            alg.ingest_records_device(base.data_ptr(), case["base"])
            alg.flush()
            alg.connected_components()
        rec = _records(case, gen, case["records"])
        if kind == "point":
            s["records"] = rec.cpu().numpy()
            s["pair"] = tuple(int(x) for x in rng.integers(0, case["vertices"], 2))
        elif case["source"] == "host":
            s["pinned"] = _pinned(rec)
            s["records"] = s["pinned"].numpy()
        else:
            s["device"], s["n"] = rec, case["records"]
    elif kind == "driver":
        rec = _records(case, gen, case["records"]).cpu().numpy()
        s["alg"] = _handle(case, seed)
        s["stream"] = gz.Stream(case["vertices"], rec.view(gz.RECORD_DTYPE))
    elif kind == "batches":
        rec = _records(case, gen, case["records"]).cpu().numpy().view(gz.RECORD_DTYPE)
        src = np.concatenate([rec["src"], rec["dst"]])
        dst = np.concatenate([rec["dst"], rec["src"]])
        order = np.argsort(src, kind="stable")
        src, dst = src[order], np.ascontiguousarray(dst[order])
        cuts = np.flatnonzero(np.diff(src)) + 1
        starts = np.concatenate([[0], cuts])
        s["batches"] = list(zip(src[starts].tolist(), np.split(dst, cuts)))
        s["alg"] = _handle(case, seed)
    elif kind == "noalloc":
        s["lib"] = _lib.load()
        s["V"], s["seed"], s["n"] = case["vertices"], SKETCH_SEED + seed, case["records"]
        s["sketches"] = torch.zeros(case["vertices"] * _sketch_bytes(case["vertices"]), dtype=torch.uint8,
                                    device="cuda")
        s["device"] = _records(case, gen, case["base"])
        torch.cuda.synchronize()
        _fold(s, case["base"])
        s["device"] = _records(case, gen, case["records"])
    elif kind == "many":
        sizes = _sizes(case, case["graphs"])
        counts = _many_counts(case, sizes)
        comps = rng.integers(1, 17, sizes.size)
        s["device"] = torch.cat([_planted(gen, int(v), int(k), int(n)) for v, k, n in zip(sizes, comps, counts)])
        s["offsets"] = np.concatenate([[0], np.cumsum(counts)]).astype(np.uint64)
        s["batch"] = gz.CCSketchBatch(sizes, [SKETCH_SEED + seed + i for i in range(sizes.size)])
    elif kind == "serving":
        t = case["tenants"]
        sizes = _sizes(case, t)
        counts = _serving_counts(case).tolist()
        need = sum(int(v) * _sketch_bytes(int(v)) + (1 << 20) for v in sizes)
        s["server"] = srv = SketchServer(need + (64 << 20), 1 << 20)
        srv.set_query_snapshot(False)
        s["tenants"] = [srv.admit(int(v), SKETCH_SEED + seed + i) for i, v in enumerate(sizes)]
        loads = [_pinned(_powerlaw(gen, int(v), 6 * n, exponent=2.3)) for v, n in zip(sizes, counts)]
        srv.ingest_segments(s["tenants"], [x.numpy() for x in loads])
        s["pinned"] = [_pinned(_powerlaw(gen, int(v), n, exponent=2.3)) for v, n in zip(sizes, counts)]
        s["segments"] = [x.numpy() for x in s["pinned"]]
        s["queried"] = s["tenants"][:case["queried"]]
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------------

def _answer(alg):
    cc = alg.connected_components()
    return {"labels": cc.parent_arr, "components": cc.size(), "rounds": alg.last_query_rounds}


def _fold(s, n):
    rc = s["lib"].gz_ingest_records_noalloc(ctypes.c_void_p(s["sketches"].data_ptr()), s["V"], s["seed"], 1.0,
                                            ctypes.c_void_p(s["device"].data_ptr()), n, None)
    if rc:
        raise RuntimeError(_lib.last_error())


def run(s):
    kind = s["kind"]
    if kind in ("stream", "segment"):
        alg = s["alg"]
        if kind == "stream":
            alg.clear()
        if "device" in s:
            alg.ingest_records_device(s["device"].data_ptr(), s["n"])
        else:
            alg.ingest_records(s["records"])
        return _answer(alg)
    if kind == "point":
        s["alg"].ingest_records(s["records"])
        connected = s["alg"].point_query(*s["pair"])
        return dict(_answer(s["alg"]), connected=connected)  # the answer is cached by now
    if kind == "driver":
        alg = s["alg"]
        alg.clear()
        driver = gz.GraphSketchDriver(alg, gz.BinaryFileStream(stream=s["stream"]))
        driver.process_stream_until(gz.END_OF_STREAM)
        driver.prep_query(gz.CONNECTIVITY)
        return dict(_answer(alg), sketches=alg.dump_sketches())
    if kind == "batches":
        alg = s["alg"]
        alg.clear()
        for src, dsts in s["batches"]:
            alg.apply_update_batch(0, src, dsts)
        alg.flush()
        return _answer(alg)
    if kind == "noalloc":
        _fold(s, s["n"])
        return s["sketches"]
    if kind == "many":
        b = s["batch"]
        b.clear()
        b.ingest_device(s["device"].data_ptr(), s["offsets"])
        res = b.connected_components()
        # the graphs' labels are views of one array, graph after graph
        return {"labels": res.labels[0].base, "components": res.num_cc, "rounds": res.rounds,
                "status": res.status}
    srv = s["server"]
    srv.ingest_segments(s["tenants"], s["segments"])
    ticket = srv.query_submit(s["queried"])
    return [list(x) for x in srv.query_wait(ticket, s["queried"])]


# ------------------------------------------------------------------------------------------------
# work
# ------------------------------------------------------------------------------------------------

def _geometry(v, algorithm="cameo"):
    """(columns, buckets per column, columns per sample) of one vertex sketch."""
    b = int(math.ceil(math.log2(math.ceil(v * (v - 1) / 2))) + 1)
    if algorithm == "cube":
        return 7 * max(18, math.ceil(math.log2(v) / (math.log2(3) - 1))), b, 7
    return max(18, math.ceil(math.log2(v) / (1 - math.log2(1.2)))), b, 1


def _sketch_bytes(v, algorithm="cameo"):
    c, b, _ = _geometry(v, algorithm)
    return (c * b + 1) * 12


def _graph_work(v, n, fresh, query, algorithm="cameo"):
    """Records read once; sketches written once (from empty), or the buckets that the records touch
    read and written; a query reads one sample of every vertex and writes the labels."""
    c, b, cps = _geometry(v, algorithm)
    if fresh:
        moved = v * (c * b + 1) * 12
    else:
        moved = 2 * min(2 * n * (c + 1), v * (c * b + 1)) * 12
    asked = v * (cps * b + 1) * 12 + 4 * v if query else 0
    return 9 * n + moved + asked


def work(case):
    kind = case["kind"]
    if kind in ("stream", "driver", "batches"):
        v, a = case["vertices"], case.get("algorithm", "cameo")
        more = v * _sketch_bytes(v, a) if kind == "driver" else 0  # the sketches it writes out
        return {"bytes": _graph_work(v, case["records"], True, True, a) + more, "flops": 0}
    if kind in ("segment", "point", "noalloc"):
        return {"bytes": _graph_work(case["vertices"], case["records"], False, kind != "noalloc"), "flops": 0}
    if kind == "many":
        sizes = _sizes(case, case["graphs"])
        each = zip(sizes.tolist(), _many_counts(case, sizes).tolist())
        return {"bytes": sum(_graph_work(v, n, True, True) for v, n in each), "flops": 0}
    each = zip(_sizes(case, case["tenants"]).tolist(), _serving_counts(case).tolist())
    return {"bytes": sum(_graph_work(v, n, False, i < case["queried"]) for i, (v, n) in enumerate(each)),
            "flops": 0}
