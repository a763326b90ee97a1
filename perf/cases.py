"""The work that is timed when this library's speed is compared from one change to the next.

A case is one piece of work that a program gives to `trove_gb300`, called the way such a program calls it and with the
library's own choice of kernels (nothing is tuned beforehand).  Struct widths are those of the benchmark and of the
tests: 4 to 64 bytes in steps of 4, wider rows (68 to 256 bytes) and widths that are no multiple of 4.

Kinds:
  small    copy, gather and scatter of one small array: launches and latency count
  copy     a contiguous copy, whole arrays or views that start `src_at` / `dst_at` structs into a buffer
  exit     the early-exit copy through the device API (warp-contiguous or block interface)
  gather   dst[i] = src[idx[i]]
  scatter  dst[idx[i]] = src[i], idx a permutation
  layout   array of structs -> structure of arrays -> array of structs
  batch    many uneven arrays in one captured persistent launch
  serve    a burst of requests to the server, each result copied out, then released
"""
import math
import random

import torch

import trove_gb300 as tg

BATCH_WIDTHS = (4, 12, 20, 36, 64)
SERVE_WIDTHS = (8, 12, 16, 28, 64)


def listed():
    return [
        # a few thousand records picked and put back, many times a second: a simulation's small groups
        {"name": "small_28B", "kind": "small", "width": 28, "n": 4097},
        # part of a vertex buffer (float3) copied to the front of another one: the two start at different alignments
        {"name": "copy_view_12B", "kind": "copy", "width": 12, "n": (1 << 22) + 3, "src_at": 1, "dst_at": 0},
        # the benchmark's sweep: a kernel that loads a struct, may leave early, and stores it (5 % of warps diverge)
        {"name": "exit_warp_12B", "kind": "exit", "width": 12, "n": (1 << 30) // 12, "modulus": 625, "path": "warp"},
        {"name": "exit_block_44B", "kind": "exit", "width": 44, "n": (1 << 30) // 44, "modulus": 625, "path": "block"},
        # the benchmark's random gather: particles reordered by a permutation
        {"name": "gather_perm_24B", "kind": "gather", "width": 24, "n": 1 << 24, "src_n": 1 << 24, "pattern": "perm",
         "path": "auto"},
        # the same through coalesced_ptr (a user's kernel), where half of the indices come in runs (a neighbour list)
        {"name": "gather_ptr_runs_36B", "kind": "gather", "width": 36, "n": (1 << 23) + 5, "src_n": 1 << 23,
         "pattern": "runs", "path": "coalesced"},
        # rows wider than a struct kernel holds: an embedding table, repeated rows
        {"name": "gather_rows_200B", "kind": "gather", "width": 200, "n": (1 << 21) + 1, "src_n": 1 << 21,
         "pattern": "uniform", "path": "auto"},
        # packed records of a width that is no multiple of 4 bytes
        {"name": "gather_packed_13B", "kind": "gather", "width": 13, "n": 1 << 22, "src_n": 1 << 22,
         "pattern": "uniform", "path": "auto"},
        # narrow records put to their places (a sort's last step), destination larger than the L2 cache
        {"name": "scatter_12B", "kind": "scatter", "width": 12, "n": 1 << 24, "dst_n": 1 << 24},
        # records to and from one array for each field, a number of structs that is no multiple of anything
        {"name": "layout_28B", "kind": "layout", "width": 28, "n": (1 << 24) + 7},
        # the benchmark's mixed batch, an eighth of its arrays
        {"name": "batch_512", "kind": "batch", "count": 512, "lo": 1 << 10, "hi": 1 << 22},
        # the benchmark's serving stream: a burst of requests in flight at once
        {"name": "serve_64", "kind": "serve", "count": 64, "lo": 1 << 8, "hi": 1 << 20},
    ]


def log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))))


def draw(rng):
    kind = rng.choice(("small", "copy", "exit", "exit", "gather", "gather", "gather", "scatter", "layout", "batch",
                       "serve"))
    width = 4 * rng.randint(1, 16)
    most = (1 << 29) // width  # 512 MB to an array at most
    if kind == "small":
        return {"kind": kind, "width": width, "n": log_int(rng, 33, 1 << 16)}
    if kind == "copy":
        width = rng.choice((width, width, rng.randint(1, 256)))
        at = rng.choice(((0, 0), (1, 0), (rng.randint(0, 9), rng.randint(0, 9))))
        return {"kind": kind, "width": width, "n": log_int(rng, 1 << 10, (1 << 29) // width), "src_at": at[0],
                "dst_at": at[1]}
    if kind == "exit":
        return {"kind": kind, "width": width, "n": log_int(rng, 1 << 14, (1 << 30) // width), "modulus": 625,
                "path": rng.choice(("warp", "block"))}
    if kind in ("gather", "scatter"):
        path = "auto"
        form = rng.choice(("struct", "struct", "struct", "wide", "packed"))
        if form == "wide":
            width = 4 * rng.randint(17, 64)
        elif form == "packed":
            width = 4 * rng.randint(0, 15) + rng.randint(1, 3)
        elif kind == "gather":
            path = rng.choice(("auto", "auto", "coalesced"))
        n = log_int(rng, 1 << 12, min(1 << 24, (1 << 29) // width))
        if kind == "scatter":
            return {"kind": kind, "width": width, "n": n, "dst_n": n}
        return {"kind": kind, "width": width, "n": n, "src_n": n,
                "pattern": rng.choice(("perm", "uniform", "runs", "identity")), "path": path}
    if kind == "layout":
        return {"kind": kind, "width": width, "n": log_int(rng, 1 << 12, most)}
    if kind == "batch":
        count = log_int(rng, 16, 384)
        lo = 1 << rng.randint(8, 12)
        return {"kind": kind, "count": count, "lo": lo, "hi": lo << rng.randint(2, 9)}
    return {"kind": kind, "count": rng.randint(4, 96), "lo": 1 << 8, "hi": 1 << rng.randint(12, 19)}


# ---- inputs ---------------------------------------------------------------------


def generator(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def payload(nbytes, g):
    """Random bytes in a buffer of whole 32-bit words (seen as bytes)."""
    words = torch.randint(-(1 << 31), 1 << 31, ((nbytes + 3) // 4,), dtype=torch.int32, device="cuda", generator=g)
    return words.view(torch.uint8)


def indices(pattern, n, src_n, g):
    if pattern == "identity":
        return torch.arange(n, dtype=torch.int64, device="cuda").remainder_(src_n).to(torch.int32)
    if pattern == "perm":
        return torch.randperm(n, device="cuda", generator=g).to(torch.int32)
    idx = torch.randint(0, src_n, (n,), dtype=torch.int32, device="cuda", generator=g)
    if pattern == "runs" and src_n > 32:  # each group of 32 outputs: a run of consecutive structs, or single ones
        groups = (n + 31) // 32
        start = torch.randint(0, src_n - 31, (groups, 1), dtype=torch.int32, device="cuda", generator=g)
        run = (start + torch.arange(32, dtype=torch.int32, device="cuda")).reshape(-1)[:n]
        single = torch.rand((groups, 1), device="cuda", generator=g).lt(0.5).expand(groups, 32).reshape(-1)[:n]
        idx = torch.where(single, idx, run)
    return idx


def lengths(case):
    rng = random.Random(17)
    return rng, [log_int(rng, case["lo"], case["hi"]) for _ in range(case["count"])]


def batch_plan(case):
    """(op, width, n) of each array of a batch: the case's own, whatever the seed of its contents."""
    rng, ns = lengths(case)
    ops = [rng.choices((tg.OP_COPY, tg.OP_GATHER, tg.OP_SCATTER), (5, 4, 1))[0] for _ in ns]
    return list(zip(ops, [rng.choice(BATCH_WIDTHS) for _ in ns], ns))


def serve_plan(case):
    """(op, width, n) of each request of a burst."""
    rng, ns = lengths(case)
    return [(rng.choice((tg.OP_COPY, tg.OP_GATHER)), rng.choice(SERVE_WIDTHS), n) for n in ns]


def offsets(sizes, step=256):
    """Start of each of the arrays in one buffer, and the buffer's size."""
    at, starts = 0, []
    for s in sizes:
        starts.append(at)
        at += (s + step - 1) // step * step
    return starts, at


def prepare(case, seed):
    g = generator(seed)
    kind = case["kind"]
    state = {"case": dict(case)}
    if kind in ("small", "gather", "scatter"):
        w, n = case["width"], case["n"]
        src_n = case.get("src_n", n)
        state["src"] = payload(src_n * w, g)
        state["idx"] = indices(case.get("pattern", "perm"), n, src_n, g)
        state["dst"] = torch.zeros(n * w, dtype=torch.uint8, device="cuda")
        if kind == "small":
            state["copied"] = torch.zeros_like(state["dst"])
            state["back"] = torch.zeros_like(state["dst"])
    elif kind == "copy":
        w, n = case["width"], case["n"]
        state["src"] = payload((n + case["src_at"]) * w, g)[case["src_at"] * w:]
        state["dst"] = torch.zeros((n + case["dst_at"]) * w, dtype=torch.uint8, device="cuda")[case["dst_at"] * w:]
    elif kind == "exit":
        state["src"] = payload(case["n"] * case["width"], g)
        state["dst"] = torch.zeros(case["n"] * case["width"], dtype=torch.uint8, device="cuda").view(torch.int32)
    elif kind == "layout":
        state["src"] = payload(case["n"] * case["width"], g)
        state["soa"] = torch.zeros(case["n"] * case["width"], dtype=torch.uint8, device="cuda").view(torch.int32)
        state["dst"] = torch.zeros_like(state["soa"])
    elif kind == "batch":
        plan = batch_plan(case)
        data_at, data_size = offsets([w * n for _, w, n in plan])
        idx_at, idx_size = offsets([n if op != tg.OP_COPY else 0 for op, _, n in plan])
        state["src"] = payload(data_size, g)
        state["dst"] = torch.zeros(data_size, dtype=torch.uint8, device="cuda").view(torch.int32)
        state["idx"] = torch.zeros(idx_size, dtype=torch.int32, device="cuda")
        tasks = []
        for (op, w, n), at, ia in zip(plan, data_at, idx_at):
            t = {"op": op, "width": w, "n": n, "src": state["src"].data_ptr() + at,
                 "dst": state["dst"].data_ptr() + at}
            if op != tg.OP_COPY:
                state["idx"][ia:ia + n] = indices("uniform" if op == tg.OP_GATHER else "perm", n, n, g)
                t.update(idx=state["idx"].data_ptr() + 4 * ia, bound=n)
            tasks.append(t)
        state["batch"] = tg.Batch(tasks)
        side = torch.cuda.Stream()
        state["batch"].capture(side)
        side.synchronize()
    else:
        plan = serve_plan(case)
        out_at, out_size = offsets([w * n for _, w, n in plan])
        src_at, src_size = offsets([w * n for _, w, n in plan])
        state["src"] = payload(src_size, g)
        idx_at, idx_size = offsets([n if op == tg.OP_GATHER else 0 for op, _, n in plan])
        state["idx"] = torch.zeros(max(idx_size, 1), dtype=torch.int32, device="cuda")
        state["out"] = torch.zeros(out_size, dtype=torch.uint8, device="cuda")
        state["out_at"] = out_at
        state["requests"] = []
        for (op, w, n), at, ia in zip(plan, src_at, idx_at):
            r = {"op": op, "width": w, "n": n, "src": state["src"].data_ptr() + at, "src_n": n}
            if op == tg.OP_GATHER:
                state["idx"][ia:ia + n] = indices("uniform", n, n, g)
                r["idx"] = state["idx"].data_ptr() + 4 * ia
            state["requests"].append(tg.make_request(r))
        state["server"] = tg.Server(max(out_size, 1 << 20))
    return state


# ---- one pass --------------------------------------------------------------------


def run(state):
    case = state["case"]
    kind = case["kind"]
    w, n = case.get("width"), case.get("n")
    if kind == "small":
        tg.copy(state["copied"], state["src"], n, w)
        tg.gather(state["dst"], state["src"], n, state["idx"], n, w)
        tg.scatter(state["back"], n, state["dst"], state["idx"], n, w)
        return [state["copied"], state["dst"], state["back"]]
    if kind == "copy":
        tg.copy(state["dst"], state["src"], n, w)
    elif kind == "exit":
        tg.copy_exit(state["dst"], state["src"], n, w, case["modulus"], path=case["path"])
    elif kind == "gather":
        tg.gather(state["dst"], state["src"], case["src_n"], state["idx"], n, w, path=case["path"])
    elif kind == "scatter":
        tg.scatter(state["dst"], case["dst_n"], state["src"], state["idx"], n, w)
    elif kind == "layout":
        tg.aos_to_soa(state["soa"], state["src"], n, w)
        tg.soa_to_aos(state["dst"], state["soa"], n, w)
        return [state["soa"], state["dst"]]
    elif kind == "batch":
        state["batch"].launch()
    else:
        server, out = state["server"], state["out"].data_ptr()
        ids = [server.submit(r) for r in state["requests"]]
        for rid, r, at in zip(ids, state["requests"], state["out_at"]):
            tg.copy(out + at, server.wait(rid).dst, r.n, r.width)
        torch.cuda.current_stream().synchronize()  # the results have been copied out: their memory can go back
        for rid in ids:
            server.release(rid)
        return state["out"]
    return state["dst"]


def exact(case, seed):
    """Nothing here is a computed number: every output is bytes moved, and has to be equal."""
    return None


def work(case):
    """Bytes read and written once; the indices' 4 bytes each."""
    kind = case["kind"]
    if kind == "batch":
        plan = batch_plan(case)
        return {"bytes": sum(2 * w * n + (0 if op == tg.OP_COPY else 4 * n) for op, w, n in plan), "flops": 0}
    if kind == "serve":  # each result is written by the server, and copied out by its user
        plan = serve_plan(case)
        return {"bytes": sum(4 * w * n + (4 * n if op == tg.OP_GATHER else 0) for op, w, n in plan), "flops": 0}
    w, n = case["width"], case["n"]
    moved = 2 * w * n
    if kind == "small":
        return {"bytes": 3 * moved + 8 * n, "flops": 0}
    if kind == "exit":
        return {"bytes": moved - w * n // case["modulus"], "flops": 0}
    if kind == "layout":
        return {"bytes": 2 * moved, "flops": 0}
    if kind in ("gather", "scatter"):
        return {"bytes": moved + 4 * n, "flops": 0}
    return {"bytes": moved, "flops": 0}
