"""The workloads gary_b200 is timed on, each through the calls a user's program makes.

listed()            the named cases
draw(rng)           another case of the ranges they stand for
prepare(case, s)    what the program holds before the call, made from seed s
run(state)          one pass; returns the whole result
work(case)          the bytes one pass cannot do without
exact(case, s)      the result by plain torch, where that is quick

Sizes come from this repository: the RMAT scales and edge factors of bench.py
and the tests, the README's example graph, the Zipf(1.2) pair microbench and
the uneven batch of Barabasi-Albert and RMAT graphs of gary_b200.batch.
"""
from __future__ import annotations

import math

import torch

import gary_b200 as gb
from gary_b200 import batch as gbatch
from gary_b200 import setops as so

ZIPF_S = 1.2


def listed():
    return [
        # The example of the package's docstring: a graph small enough that the
        # call itself (launches, copy back, wait) is most of the time.
        {"name": "triangles_er_16k", "kind": "count", "pattern": 3, "graph": "er", "n": 16384, "m": 131072},
        # An ordinary graph, counted again and again on a resident handle.
        {"name": "triangles_rmat20", "kind": "count", "pattern": 3, "graph": "rmat", "scale": 20, "ef": 16},
        # The headline workload of bench.py, the largest of all.
        {"name": "triangles_rmat24_ef32", "kind": "count", "pattern": 3, "graph": "rmat", "scale": 24, "ef": 32},
        # The two other patterns at the size bench.py's pattern workload is profiled on.
        {"name": "four_cycles_rmat22", "kind": "count", "pattern": 4, "graph": "rmat", "scale": 22, "ef": 16},
        {"name": "four_cliques_rmat22", "kind": "count", "pattern": 5, "graph": "rmat", "scale": 22, "ef": 16},
        # Many uneven graphs in one captured launch, replayed.
        {"name": "batch_128_graphs", "kind": "batch", "graphs": 128, "n_lo": 1000, "n_hi": 200000, "captured": True},
        # The set-operation microbench: per-pair counts of a large batch, ...
        {"name": "intersect_counts_1m", "kind": "intersect", "pairs": 1 << 20, "nmax": 65536, "overlap": 0.1,
         "variant": "auto", "lists": False, "bounded": False},
        # ... and the intersections themselves for a smaller, odd one.
        {"name": "intersect_lists_50k", "kind": "intersect", "pairs": 50001, "nmax": 65536, "overlap": 0.5,
         "variant": "auto", "lists": True, "bounded": False},
        # Membership of many keys in one sorted list (a vertex list, an id table).
        {"name": "search_4m_keys", "kind": "search", "len": 4 << 20, "keys": 4 << 20, "cache": 1024},
        # End to end from the host: copy, orient, plan, count, free.
        {"name": "upload_and_count_rmat20", "kind": "upload", "scale": 20, "ef": 16, "dag": True},
        # An edge list on the device into a symmetric CSR.
        {"name": "csr_from_edges_rmat20", "kind": "csr", "graph": "rmat", "scale": 20, "ef": 16, "distinct": 0.9},
        # Byte planes of an id array, split and joined again.
        {"name": "planes_64m_words", "kind": "planes", "words": (64 << 20) + 3, "word_bytes": 4, "plane_bytes": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _odd(rng, lo, hi):
    return rng.randrange(lo, hi + 1, 2)


def draw(rng):
    kind = rng.choice(["count", "count", "count", "batch", "intersect", "intersect", "search", "upload", "csr",
                       "planes"])
    if kind == "count":
        pattern = rng.choice([3, 3, 4, 5])
        if rng.random() < 0.5:
            n = _log_int(rng, 2000, 2000000)
            return {"kind": "count", "pattern": pattern, "graph": "er", "n": n, "m": n * rng.randint(3, 24) + rng.randint(0, 9)}
        return {"kind": "count", "pattern": pattern, "graph": "rmat", "scale": rng.randint(12, 22 if pattern == 3 else 20),
                "ef": _odd(rng, 3, 23)}
    if kind == "batch":
        return {"kind": "batch", "graphs": _log_int(rng, 8, 128), "n_lo": rng.choice([200, 1000]),
                "n_hi": rng.choice([20000, 200000]), "captured": rng.random() < 0.5}
    if kind == "intersect":
        lists = rng.random() < 0.4
        return {"kind": "intersect", "pairs": _log_int(rng, 1000, 1 << 20), "nmax": rng.choice([4096, 65536]),
                "overlap": rng.choice([0.0, 0.1, 0.25, 0.5]),
                "variant": rng.choice(["auto", "auto", "auto", "merge", "search"]), "lists": lists,
                "bounded": not lists and rng.random() < 0.3}
    if kind == "search":
        return {"kind": "search", "len": _log_int(rng, 1000, 32 << 20), "keys": _log_int(rng, 1000, 32 << 20),
                "cache": rng.choice([0, 256, 1024, 8192])}
    if kind == "upload":
        return {"kind": "upload", "scale": rng.randint(12, 21), "ef": _odd(rng, 3, 23), "dag": rng.random() < 0.5}
    if kind == "csr":
        if rng.random() < 0.5:
            n = _log_int(rng, 2000, 2000000)
            return {"kind": "csr", "graph": "er", "n": n, "m": n * rng.randint(2, 24) + rng.randint(0, 9), "distinct": 0.9}
        scale = rng.randint(12, 21)
        return {"kind": "csr", "graph": "rmat", "scale": scale, "ef": _odd(rng, 3, 23), "distinct": 0.4 if scale < 16 else 0.7}
    wb = rng.choice([4, 8])
    return {"kind": "planes", "words": _log_int(rng, 1000, 64 << 20), "word_bytes": wb,
            "plane_bytes": rng.choice([1, 2] if wb == 4 else [1, 2, 4])}


# ---- inputs -------------------------------------------------------------------
def _rand(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _edges(case, seed):
    """(src, dst, n) on the device, as sampled: loops and repeats included."""
    if case["graph"] == "er":
        g = _rand(seed)
        e = torch.randint(case["n"], (2, case["m"]), generator=g, device="cuda", dtype=torch.int32)
        return e[0].contiguous(), e[1].contiguous(), case["n"]
    src, dst = gb.gen_rmat_device(case["scale"], seed, case["ef"] << case["scale"])
    return src, dst, 1 << case["scale"]


def _edge_list(case, seed):
    """As _edges, with the stated share of distinct edges and the rest repeats
    of them (some reversed, some loops), so that the CSR's size follows from
    the case."""
    src, dst, n = _edges(case, seed)
    g = _rand(seed)
    m, d = src.numel(), int(src.numel() * case["distinct"])
    s, t = src.long(), dst.long()
    key = torch.unique((torch.minimum(s, t) * n + torch.maximum(s, t))[s != t])
    if key.numel() < d:
        raise ValueError(f"{key.numel()} distinct edges sampled, {d} wanted")
    key = key[torch.randperm(key.numel(), generator=g, device="cuda")[:d]]
    key = torch.cat([key, key[torch.randint(d, (m - d,), generator=g, device="cuda")]])
    a, b = key // n, key % n
    b[d:] = torch.where(torch.rand(m - d, generator=g, device="cuda") < 0.05, a[d:], b[d:])
    flip = torch.rand(m, generator=g, device="cuda") < 0.5
    order = torch.randperm(m, generator=g, device="cuda")
    return (torch.where(flip, b, a).to(torch.int32)[order].contiguous(),
            torch.where(flip, a, b).to(torch.int32)[order].contiguous(), n)


class _DeviceArray:
    """A device pointer of the library as an array interface (for torch.as_tensor)."""

    def __init__(self, ptr, count, typestr):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 3}


def _csr_tensors(csr):
    n, nnz = csr.shape()
    p, i = csr.device_ptrs()
    idx = torch.as_tensor(_DeviceArray(i, nnz, "<i4"), device="cuda") if nnz else torch.empty(0, dtype=torch.int32, device="cuda")
    return torch.as_tensor(_DeviceArray(p, n + 1, "<i8"), device="cuda"), idx


def _pinned(t):
    return torch.empty(t.shape, dtype=t.dtype, pin_memory=True).copy_(t)


def _zipf(nmax):
    w = [k ** -ZIPF_S for k in range(1, nmax + 1)]
    h = sum(w)
    return [x / h for x in w]


def _list_room(case):
    """Ids set aside for the intersections of a batch: 1.5 times what the
    shorter lists of its pairs hold on average, and 20 of the longest."""
    mean_min, tail = 0.0, 1.0
    for p in _zipf(case["nmax"]):
        mean_min += tail * tail
        tail -= p
    return int(1.5 * case["pairs"] * mean_min) + 20 * case["nmax"]


def _search_inputs(case, seed):
    g = _rand(seed)
    # sorted distinct ids with random gaps; half of the keys are members
    lst = torch.cumsum(torch.randint(1, 64, (case["len"],), generator=g, device="cuda"), 0)
    member = lst[torch.randint(case["len"], (case["keys"],), generator=g, device="cuda")]
    other = torch.randint(int(lst[-1]) + 1, (case["keys"],), generator=g, device="cuda")
    pick = torch.rand(case["keys"], generator=g, device="cuda") < 0.5
    return lst.to(torch.int32), torch.where(pick, member, other).to(torch.int32)


def _plane_words(case, seed):
    # neighbour ids with a skew, so that high-order planes repeat as they do in real lists
    g = _rand(seed)
    r = torch.rand(case["words"], generator=g, device="cuda")
    ids = (r * r * (1 << 24)).to(torch.int32)
    return ids if case["word_bytes"] == 4 else ids.to(torch.int64) * 0x10001


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("count", "upload"):
        with gb.csr_from_edges_device(*_edges(dict(case, graph=case.get("graph", "rmat")), seed)) as csr:
            ptr, idx = _csr_tensors(csr)
            n = csr.shape()[0]
            if kind == "count":
                return {"kind": kind, "graph": gb.Graph.upload(ptr, idx, n), "pattern": case["pattern"]}
            if case["dag"]:  # every edge once, in the row of its larger endpoint
                rows = torch.repeat_interleave(torch.arange(n, device="cuda", dtype=torch.int32), ptr[1:] - ptr[:-1])
                keep = idx < rows
                idx = idx[keep]
                ptr = torch.zeros_like(ptr)
                torch.cumsum(torch.bincount(rows[keep], minlength=n), 0, out=ptr[1:])
            return {"kind": kind, "ptr": _pinned(ptr), "idx": _pinned(idx), "n": n,
                    "flags": gb.GARY_INPUT_DAG if case["dag"] else 0}
    if kind == "batch":
        specs = gbatch.make_specs(case["graphs"], seed, case["n_lo"], case["n_hi"])
        b = gbatch.Batch.build(specs)
        stream = torch.cuda.Stream()
        return {"kind": kind, "batch": b, "stream": stream, "exec": b.capture(stream) if case["captured"] else None}
    if kind == "intersect":
        b = so.PairBatch.generate(seed, 0, case["pairs"], so.zipf_table(case["nmax"], ZIPF_S), case["overlap"])
        word = lambda: torch.zeros(1, dtype=torch.int64, device="cuda")  # noqa: E731
        state = {"kind": kind, "pairs": b, "variant": so.VARIANTS[case["variant"]], "lists": case["lists"], "bound": None,
                 "counts": torch.empty(case["pairs"], dtype=torch.int64, device="cuda"), "queue": word(), "total": word()}
        if case["lists"]:
            # pair i fills a prefix of its slot, the rest of the buffer stays 0
            room = _list_room(case)
            off = torch.zeros(case["pairs"] + 1, dtype=torch.int64, device="cuda")
            torch.cumsum(torch.minimum(b.la, b.lb).long(), 0, out=off[1:])
            if int(off[-1]) > room:
                raise ValueError(f"the lists need {int(off[-1])} ids, {room} are set aside")
            state["outputs"] = (torch.zeros(room, dtype=torch.int32, device="cuda"), off)
        if case["bounded"]:
            state["bound"] = torch.randint(so.RANGE, (case["pairs"],), generator=_rand(seed), device="cuda", dtype=torch.int32)
        return state
    if kind == "search":
        lst, keys = _search_inputs(case, seed)
        return {"kind": kind, "list": lst, "keys": keys, "cache": case["cache"]}
    if kind == "csr":
        src, dst, n = _edge_list(case, seed)
        return {"kind": kind, "src": src, "dst": dst, "n": n, "csr": None}
    return {"kind": kind, "words": _plane_words(case, seed), "word_bytes": case["word_bytes"], "plane_bytes": case["plane_bytes"]}


# ---- one pass -------------------------------------------------------------------
def run(s):
    kind = s["kind"]
    if kind == "count":
        return s["graph"].count(s["pattern"])
    if kind == "upload":
        with gb.Graph.upload(s["ptr"], s["idx"], s["n"], s["flags"]) as g:
            return g.count(gb.GARY_PATTERN_TRIANGLE)
    if kind == "batch":
        if s["exec"] is None:
            counts, total = s["batch"].count()
            return {"counts": counts.view("int64"), "total": total}
        s["exec"].launch(s["stream"])
        return {"counts": s["exec"].counts, "total": s["exec"].total}
    if kind == "intersect":
        if s["bound"] is not None:
            counts, total = so.intersect_num(s["pairs"], s["bound"], variant=s["variant"])
            return {"counts": counts, "total": total}
        if s["lists"]:
            counts, total, out, _ = so.intersect(s["pairs"], s["variant"], True, counts=s["counts"], queue=s["queue"],
                                                 total=s["total"], outputs=s["outputs"])
            return {"counts": counts, "total": total, "ids": out}
        counts, total = so.intersect(s["pairs"], s["variant"], counts=s["counts"], queue=s["queue"], total=s["total"])
        return {"counts": counts, "total": total}
    if kind == "search":
        found, count = so.search(s["list"], s["keys"], s["cache"])
        return {"found": found, "count": count}
    if kind == "csr":
        if s["csr"] is not None:
            s["csr"].free()
        s["csr"] = gb.csr_from_edges_device(s["src"], s["dst"], s["n"])
        ptr, idx = _csr_tensors(s["csr"])
        return {"ptr": ptr, "idx": idx}
    planes = gb.planes_split(s["words"], s["plane_bytes"])
    return {"planes": planes, "words": gb.planes_join(planes, s["word_bytes"])}


# ---- what a pass cannot do without ------------------------------------------------
def _graph_size(case):
    """(vertices, sampled edges) of a graph case."""
    if case.get("graph") == "er":
        return case["n"], case["m"]
    return 1 << case["scale"], case["ef"] << case["scale"]


def work(case):
    kind = case["kind"]
    if kind == "count":  # every oriented list once
        n, m = _graph_size(case)
        return {"bytes": 4 * m + 8 * n + 8, "flops": 0}
    if kind == "upload":  # the host arrays once
        n, m = _graph_size(case)
        return {"bytes": (4 if case["dag"] else 8) * m + 8 * n + 16, "flops": 0}
    if kind == "csr":  # the edge list in, offsets and both directions out
        n, m = _graph_size(case)
        return {"bytes": 8 * m + 8 * m + 8 * n + 8, "flops": 0}
    if kind == "batch":  # mean vertex count of the log-uniform law, about 8.5 edges each
        lo, hi = case["n_lo"], case["n_hi"]
        n = case["graphs"] * (hi - lo) / math.log(hi / lo)
        return {"bytes": n * (8.5 * 4 + 8) + 8 * case["graphs"], "flops": 0}
    if kind == "intersect":  # mean list length of Zipf(ZIPF_S) on [1, nmax]
        mean = sum(k * p for k, p in enumerate(_zipf(case["nmax"]), 1))
        return {"bytes": case["pairs"] * (2 * mean * 4 + 32), "flops": 0}
    if kind == "search":
        return {"bytes": 4 * case["len"] + 5 * case["keys"] + 8, "flops": 0}
    return {"bytes": 4 * case["words"] * case["word_bytes"], "flops": 0}


# ---- the same result by plain torch -----------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind == "count":
        if case["graph"] != "er" or case["n"] > 16384 or case["pattern"] == 5:
            return None
        src, dst, n = _edges(case, seed)
        a = torch.zeros((n, n), dtype=torch.float64, device="cuda")
        a[src.long(), dst.long()] = 1
        a[dst.long(), src.long()] = 1
        a.fill_diagonal_(0)
        paths = a @ a  # paths of length 2 between every pair
        if case["pattern"] == 3:
            return int((paths * a).sum()) // 6
        paths.fill_diagonal_(0)
        return int((paths * (paths - 1)).sum()) // 8
    if kind == "intersect" and not case["lists"]:
        s = prepare(case, seed)
        b, bound = s["pairs"], s["bound"]
        if int(b.a_off[-1]) > 200_000_000:
            return None

        def keys(off, length, ids):  # pair << 32 | id of every id that counts, in order
            length = length.long()
            pair = torch.repeat_interleave(torch.arange(b.npairs, device="cuda"), length)
            at = torch.arange(pair.numel(), device="cuda") - (torch.cumsum(length, 0) - length)[pair] + off[pair]
            v = ids[at].long()
            k = (pair << 32) | v
            return k if bound is None else k[v < bound[pair]]

        ka, kb = keys(b.a_off, b.la, b.a), keys(b.b_off, b.lb, b.b)
        at = torch.searchsorted(kb, ka).clamp_(max=max(kb.numel() - 1, 0))
        hit = kb[at] == ka if kb.numel() else torch.zeros_like(ka, dtype=torch.bool)
        counts = torch.bincount(ka[hit] >> 32, minlength=b.npairs)
        return {"counts": counts, "total": counts.sum().reshape(1)}
    if kind == "search":
        lst, keys = _search_inputs(case, seed)
        at = torch.searchsorted(lst, keys).clamp_(max=case["len"] - 1)
        found = (lst[at] == keys).to(torch.uint8)
        return {"found": found, "count": found.sum(dtype=torch.int64).reshape(1)}
    if kind == "csr":
        src, dst, n = _edge_list(case, seed)
        s, d = torch.cat([src, dst]).long(), torch.cat([dst, src]).long()
        key = torch.unique((s * n + d)[s != d])
        ptr = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
        torch.cumsum(torch.bincount(key // n, minlength=n), 0, out=ptr[1:])
        return {"ptr": ptr, "idx": (key % n).to(torch.int32)}
    if kind == "planes":
        w = _plane_words(case, seed)
        wb, pb = case["word_bytes"], case["plane_bytes"]
        dt = {1: torch.uint8, 2: torch.int16, 4: torch.int32}[pb]
        by = w.view(torch.uint8).reshape(-1, wb)
        return {"planes": [by[:, j * pb:(j + 1) * pb].contiguous().view(dt).reshape(-1) for j in range(wb // pb)], "words": w}
    return None
