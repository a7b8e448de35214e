"""What this library's users run, as cases that can be timed and compared.

Every case goes through the public entry points of the `b200kv` package on device tensors, as an engine calls them:
decode attention over a paged latent cache (dense, sharded, sparse, any page size and head count), the indexer in
front of the sparse form, the prefill side (the producer of the appended rows; append and gather), and the batched
engine driver. `draw` spreads the same kinds over their ranges. Lengths are a function of the case, values of the
seed: latent rows and queries are N(0, 1) bf16 as everywhere in this repository.
"""
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "ascend-moe-engine_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import b200kv  # noqa: E402

LATENT, ROPE, ROW = b200kv.LATENT_DIM, b200kv.ROPE_DIM, b200kv.ROW_DIM
INDEX_DIM = 128
SCALE = 1.0 / 24.0  # 1 / sqrt(576)


def _decode(name, **over):
    """Decode attention. `graph`: the layers' calls captured once and replayed each step, as a serving loop does (and as
    this repository's benchmark does); otherwise one call after the other from Python."""
    case = {"name": name, "kind": "decode", "seqs": 1, "lo": 129, "hi": 129, "heads": 64, "block": 64, "layers": 1, "fused_rows": True,
            "append": False, "quant": False, "stable": True, "graph": False, "q_gain": 1.0}
    case.update(over)
    return case


def listed():
    return [
        # One user, a short prompt: the model's 43 layers of one decode step, the append inside each launch.
        _decode("step_1x129_43layers", layers=43, append=True, graph=True),
        # The engine driver serving a few short requests: admission, chunked prefill, decode steps with the output quantised,
        # release. Small calls one after the other, each step's result read before the next begins.
        {"name": "serve_5x400", "kind": "serve", "seqs": 5, "lo": 100, "hi": 700, "block": 128, "layers": 3, "steps": 4, "chunk": 256},
        # The headline configuration: 32 sequences at context 4,096, the append inside the launch.
        _decode("step_32x4096", seqs=32, lo=4096, hi=4096, layers=2, append=True, graph=True),
        # A full machine: 256 sequences of 512 .. 32,768 tokens, the two caches, the output quantised for the next GEMM.
        _decode("ragged_256", seqs=256, lo=512, hi=32768, fused_rows=False, quant=True),
        # One long document.
        _decode("long_1x262144", seqs=1, lo=262144, hi=262144),
        # A cache with pages of 16 tokens, which many engines use.
        _decode("pages16_16x4096", seqs=16, lo=300, hi=4096, block=16),
        # A quarter of the 64 heads, as one rank of four in tensor parallelism has them.
        _decode("heads16_32x2048", seqs=32, lo=200, hi=2048, heads=16),
        # One rank's share of a long context over eight: its shard's partial, then the merge of the eight.
        {"name": "shard_32768_of_8", "kind": "shard", "seqs": 1, "shard": 32768, "world": 8, "block": 64, "layers": 2, "graph": True},
        # A sparse layer for a few users: index scores, the 512 best of some 4,000 tokens, attention over them.
        {"name": "sparse_4x4096", "kind": "sparse", "seqs": 4, "lo": 3500, "hi": 4096, "index_heads": 64, "top": 512, "block": 64, "layers": 3,
         "attend": True, "graph": True},
        # The indexer on one long document, many selected.
        {"name": "indexer_1x131072", "kind": "sparse", "seqs": 1, "lo": 131072, "hi": 131072, "index_heads": 64, "top": 2048, "block": 64,
         "layers": 2, "attend": False, "graph": True},
        # Prefill, write side: RMSNorm + rotary + paged write of a large batch of prompt tokens.
        {"name": "producer_49157", "kind": "producer", "tokens": 49157, "fused_rows": False, "copies": False},
        # Chunked prefill: the chunk's rows appended, then every sequence's history gathered.
        {"name": "chunk_64x256", "kind": "chunk", "seqs": 64, "lo": 257, "hi": 2048, "chunk": 256, "block": 64, "fused_rows": False},
    ]


def _log(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _lens_range(rng, seqs, most_tokens, longest, shortest=1):
    hi = _log(rng, shortest, max(shortest, min(longest, most_tokens // seqs)))
    return (hi if rng.random() < 0.4 else max(1, hi // rng.choice([2, 4, 16]))), hi


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "any", "any", "shard", "sparse", "sparse", "producer", "chunk", "serve"])
    if kind in ("decode", "any"):
        seqs = _log(rng, 1, 256 if kind == "decode" else 64)
        lo, hi = _lens_range(rng, seqs, 2_000_000 if kind == "decode" else 24_000, 262_144 if kind == "decode" else 8192)
        case = _decode("", seqs=seqs, lo=lo, hi=hi, fused_rows=rng.random() < 0.5, q_gain=rng.choice([1.0 / 24.0, 1.0, 1.0, 3.0]))
        if kind == "decode":
            small = seqs * hi <= 262_144
            case.update(block=rng.choice([64, 64, 128, 256]), append=rng.random() < 0.4 and small, quant=rng.random() < 0.3,
                        stable=rng.random() < 0.7, layers=rng.choice([1, 2, 3]) if small else 1, graph=rng.random() < 0.4)
        else:
            case["heads"], case["block"] = rng.choice([(64, 1), (64, 8), (64, 16), (64, 32), (64, 48), (64, 96), (8, 64), (16, 64), (16, 16),
                                                       (32, 64), (32, 128), (128, 64)])
        del case["name"]
        return case
    if kind == "shard":
        return {"kind": "shard", "seqs": rng.choice([1, 1, 2, 5]), "shard": _log(rng, 1, 65_536), "world": rng.choice([2, 3, 4, 8]),
                "block": rng.choice([64, 128]), "layers": rng.choice([1, 2, 4]), "graph": rng.random() < 0.5}
    if kind == "sparse":
        # One document of any length, or several short sequences. (Positions come back in the order of their scores, so one score
        # that is off by rounding can move many of them: larger batches are compared score by score in the tests.)
        seqs = rng.choice([1, _log(rng, 2, 64)])
        lo, hi = _lens_range(rng, seqs, 262_144 if seqs == 1 else 128 * (148 // seqs) * seqs, 262_144, 16)
        return {"kind": "sparse", "seqs": seqs, "lo": lo, "hi": hi, "index_heads": rng.choice([16, 32, 64, 64]),
                "top": rng.choice([64, 256, 512, 1024, 2048, 1337]), "block": rng.choice([64, 128]), "layers": rng.choice([1, 2]),
                "attend": rng.random() < 0.7, "graph": rng.random() < 0.5}
    if kind == "producer":
        return {"kind": "producer", "tokens": _log(rng, 1, 131_072), "fused_rows": rng.random() < 0.5, "copies": rng.random() < 0.3}
    if kind == "serve":
        seqs = _log(rng, 1, 32)
        lo, hi = _lens_range(rng, seqs, 16_384, 4096)
        return {"kind": "serve", "seqs": seqs, "lo": lo, "hi": hi, "block": rng.choice([64, 128]), "layers": rng.choice([1, 2, 3]),
                "steps": rng.choice([1, 2, 5]), "chunk": rng.choice([64, 256, 1024])}
    seqs = _log(rng, 1, 300)
    lo, hi = _lens_range(rng, seqs, 160_000, 65_536, 2)
    return {"kind": "chunk", "seqs": seqs, "lo": lo, "hi": hi, "chunk": _log(rng, 1, 512), "block": rng.choice([64, 64, 128, 16, 32]),
            "fused_rows": rng.random() < 0.5}


# ---- inputs ---------------------------------------------------------------------------------------------------------
def _lens(case):
    r = np.random.RandomState(case["seqs"] * 7919 + case["lo"] * 31 + case["hi"])
    return r.randint(case["lo"], case["hi"] + 1, case["seqs"]).astype(np.int32)


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _normal(g, *shape):
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.bfloat16)


def _tables(lens, block, seed):
    """Block tables over a shuffled pool with a few blocks to spare: (table [n, columns] int32, blocks)."""
    need = (lens.astype(np.int64) + block - 1) // block
    blocks = int(need.sum()) + 5
    order = np.random.RandomState((int(seed) + 77) & 0x7FFFFFFF).permutation(blocks).astype(np.int32)
    table = np.zeros((len(lens), max(1, int(need.max()))), dtype=np.int32)
    at = 0
    for b, n in enumerate(need):
        table[b, :n] = order[at:at + n]
        at += int(n)
    return table, blocks


def _pools(g, layers, rows, fused_rows):
    """A layer-major cache: latent [layers, rows, 512] and rope [layers, rows, 64] as the caller holds them, and each layer's
    view; fused rows keep both in one 576-wide array."""
    if fused_rows:
        both = _normal(g, layers, rows, ROW)
        return both[..., :LATENT], both[..., LATENT:], [b200kv.pool_view(both[i]) for i in range(layers)]
    latent, rope = _normal(g, layers, rows, LATENT), _normal(g, layers, rows, ROPE)
    return latent, rope, [b200kv.pool_view(latent[i], rope[i]) for i in range(layers)]


def _empty(*shape, dtype=torch.bfloat16):
    return torch.empty(shape, dtype=dtype, device="cuda")


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _slots(table, lens, back, block):
    """Pool rows of every sequence's last `back[b]` positions, sequence after sequence."""
    out = []
    for b, n in enumerate(lens):
        t = np.arange(int(n) - int(back[b]), int(n))
        out.append(table[b][t // block].astype(np.int64) * block + t % block)
    return np.concatenate(out).astype(np.int32)


def _with_graph(state, step):
    """Captures `step` the way a serving loop captures its decode step; the replay is then the whole step."""
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        step(state)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        graph.capture_begin()
        out = step(state)
        graph.capture_end()
    torch.cuda.current_stream().wait_stream(side)
    state["graph"], state["graph_out"] = graph, out


def _angles(positions):
    """Rotary angles of the positions, [n, 64] with the two halves alike."""
    at = torch.as_tensor(np.asarray(positions), device="cuda", dtype=torch.float32)
    angle = at[:, None] * (10000.0 ** (-torch.arange(32, device="cuda", dtype=torch.float32) / 32))[None, :]
    return torch.cat([angle, angle], dim=1)


def _prepare_serve(case, g, state):
    lens, n, layers, steps, block = _lens(case), case["seqs"], case["layers"], case["steps"], case["block"]
    columns = (int(lens.max()) + steps + block - 1) // block
    need = int(((lens.astype(np.int64) + steps + block - 1) // block).sum())
    state["engine"] = b200kv.Engine(layers=layers, max_seqs=n, num_blocks=need + 3, block_size=block, max_blocks_per_seq=columns,
                                    max_step_tokens=n * case["chunk"], scale=SCALE)
    seqs, done, first = list(range(n)), np.zeros(n, dtype=np.int64), 0
    chunks, owner, positions = [], [], []  # the prefill steps; every appended row's sequence and position, in step order
    while (done < lens).any():
        ids = [b for b in seqs if done[b] < lens[b]]
        grow = [int(min(case["chunk"], lens[b] - done[b])) for b in ids]
        chunks.append((ids, grow, first))
        for b, k in zip(ids, grow):
            owner += [b] * k
            positions += list(range(int(done[b]), int(done[b]) + k))
            done[b] += k
        first += sum(grow)
    for t in range(steps):
        owner += seqs
        positions += [int(lens[b]) + t for b in seqs]
    angle = _angles(positions)
    total = len(positions)
    state.update(seqs=seqs, chunks=chunks, host_lens=lens, owner=np.array(owner), kv_a=_normal(g, layers, total, ROW),
                 gamma=1.0 + 0.1 * _normal(g, layers, LATENT), cos=angle.cos().bfloat16(), sin=angle.sin().bfloat16(),
                 q=_normal(g, steps, layers, n, 64, ROW), out=_empty(steps, layers, n, 64, LATENT),
                 quant=(_empty(steps, layers, n, 64 * LATENT, dtype=torch.uint8),
                        _empty(steps, layers, n, 64 * LATENT // 32, dtype=torch.uint8)))
    return state


def prepare(case, seed):
    g = _gen(seed)
    state = {"case": case, "status": b200kv.new_status()}
    kind = case["kind"]
    if kind in ("decode", "shard", "sparse"):
        n, layers, heads = case["seqs"], case["layers"], case.get("heads", 64)
        lens = np.full(n, case["shard"], dtype=np.int32) if kind == "shard" else _lens(case)
        table, blocks = _tables(lens, case["block"], seed)
        rows = blocks * case["block"]
        state.update(table=_dev(table), lens=_dev(lens), host_table=table, host_lens=lens,
                     ws=_empty(b200kv.decode_workspace_bytes(n, heads), dtype=torch.uint8))
        if case.get("attend", True):
            state["latent"], state["rope"], state["views"] = _pools(g, layers, rows, case.get("fused_rows", True))
            state.update(q=_normal(g, layers, n, heads, ROW) * case.get("q_gain", 1.0), out=_empty(layers, n, heads, LATENT),
                         lse=_empty(layers, n, heads, dtype=torch.float32))
    if kind == "decode":
        state.update(new=None, quant=None)
        if case["append"]:
            state["new"] = (_normal(g, layers, n, LATENT), _normal(g, layers, n, ROPE))
        if case["quant"]:
            state["quant"] = (_empty(layers, n, heads, LATENT, dtype=torch.uint8), _empty(layers, n, heads, LATENT // 32, dtype=torch.uint8))
        step = _decode_step
    elif kind == "shard":
        # The rank's own shard is the first of the context; the other ranks' partials are what an all-gather brings.
        l_sum = (torch.rand((layers, case["world"], n, 64), generator=g, device="cuda") * 0.8 + 0.2) * case["shard"]
        o_sum = torch.randn((*l_sum.shape, LATENT), generator=g, device="cuda") * l_sum[..., None] / math.sqrt(case["shard"])
        state.update(begin=_dev(np.zeros(n, dtype=np.int32)), part_o=o_sum, part_l=l_sum,
                     part_m=torch.rand(l_sum.shape, generator=g, device="cuda"))
        step = _shard_step
    elif kind == "sparse":
        heads = case["index_heads"]
        state.update(index_q=_normal(g, layers, n, heads, INDEX_DIM).to(torch.float8_e4m3fn).view(torch.uint8),
                     index_q_scale=torch.rand((layers, n, heads), generator=g, device="cuda") * 0.02 + 0.01,
                     weights=_normal(g, layers, n, heads).abs(),
                     keys=_normal(g, layers, rows, INDEX_DIM).to(torch.float8_e4m3fn).view(torch.uint8),
                     key_scale=torch.rand((layers, rows), generator=g, device="cuda") * 0.02 + 0.01)
        if case["attend"]:
            state["rows"] = _empty(layers, n, case["top"], dtype=torch.int32)
        step = _sparse_step
    elif kind == "producer":
        tokens = case["tokens"]
        rows = (tokens + 63) // 64 * 64 + 320
        latent, rope, views = _pools(g, 1, rows, case["fused_rows"])
        # Prompt tokens land in blocks of 64 consecutive rows, the blocks in any order.
        order = np.random.RandomState((int(seed) + 5) & 0x7FFFFFFF).permutation(rows // 64)
        slots = (order[:, None] * 64 + np.arange(64)[None, :]).reshape(-1)[:tokens].astype(np.int32)
        angle = _angles(np.arange(tokens))
        state.update(latent=latent[0], rope=rope[0], view=views[0], slots=_dev(slots), kv_a=_normal(g, tokens, ROW),
                     gamma=1.0 + 0.1 * _normal(g, LATENT), cos=angle.cos().bfloat16(), sin=angle.sin().bfloat16(), copies=None)
        if case["copies"]:
            state["copies"] = (_empty(tokens, LATENT), _empty(tokens, ROPE), _empty(tokens, dtype=torch.float32))
        return state
    elif kind == "chunk":
        lens = _lens(case)
        table, blocks = _tables(lens, case["block"], seed)
        back = np.minimum(lens, case["chunk"])
        latent, rope, views = _pools(g, 1, blocks * case["block"], case["fused_rows"])
        total = int(lens.sum())
        offsets = np.concatenate([[0], np.cumsum(lens.astype(np.int64))[:-1]])
        state.update(latent=latent[0], rope=rope[0], view=views[0], table=_dev(table), lens=_dev(lens), offsets=_dev(offsets),
                     slots=_dev(_slots(table, lens, back, case["block"])), total=total, host_table=table, host_lens=lens,
                     new=(_normal(g, int(back.sum()), LATENT), _normal(g, int(back.sum()), ROPE)),
                     out=(_empty(total, LATENT), _empty(total, ROPE)))
        return state
    elif kind == "serve":
        return _prepare_serve(case, g, state)
    else:
        raise ValueError(kind)
    if case["graph"]:
        _with_graph(state, step)
    return state


# ---- one pass -------------------------------------------------------------------------------------------------------
def _decode_step(s):
    case = s["case"]
    for i, view in enumerate(s["views"]):
        b200kv.mla_decode(s["q"][i], view, s["table"], s["lens"], case["block"], SCALE, out=s["out"][i], lse=s["lse"][i],
                          workspace=s["ws"], status=s["status"], new_rows=(s["new"][0][i], s["new"][1][i]) if s["new"] else None,
                          stable_tables=case["stable"], quantised=(s["quant"][0][i], s["quant"][1][i]) if s["quant"] else None)
    return {"out": s["out"], "lse": s["lse"], "quant": list(s["quant"] or ()), "pool": [s["latent"], s["rope"]] if s["new"] else []}


def _shard_step(s):
    n = s["case"]["seqs"]
    for i, view in enumerate(s["views"]):
        o, m, l = s["part_o"][i], s["part_m"][i], s["part_l"][i]
        b200kv.mla_decode(s["q"][i], view, s["table"], s["lens"], s["case"]["block"], SCALE, kv_begin=s["begin"],
                          partial=(o[0], m[0], l[0]), workspace=s["ws"], status=s["status"], stable_tables=True)
        b200kv.lse_merge(o.flatten(1, 2), m.flatten(1), l.flatten(1), s["out"][i], s["lse"][i])
    return {"out": s["out"], "lse": s["lse"]}


def _sparse_step(s):
    case, index, count = s["case"], [], []
    for i in range(case["layers"]):
        rows = s["rows"][i] if case["attend"] else None
        picked, n_picked = b200kv.indexer_topk(s["index_q"][i], s["index_q_scale"][i], s["weights"][i], s["keys"][i], s["key_scale"][i],
                                               s["table"], s["lens"], case["block"], case["hi"], case["top"], status=s["status"],
                                               rows_out=rows)
        if case["attend"]:
            b200kv.mla_decode(s["q"][i], s["views"][i], None, n_picked, 1, SCALE, out=s["out"][i], lse=s["lse"][i], workspace=s["ws"],
                              status=s["status"], row_index=rows)
        index.append(picked)
        count.append(n_picked)
    return {"index": index, "count": count, "out": s["out"] if case["attend"] else None, "lse": s["lse"] if case["attend"] else None}


def _serve(s):
    case, engine, seqs = s["case"], s["engine"], s["seqs"]
    for seq in seqs:
        engine.admit(seq)
    for ids, grow, first in s["chunks"]:
        engine.begin_step(ids, grow)
        n = int(sum(grow))
        for i in range(case["layers"]):
            engine.layer_append(i, s["kv_a"][i][first:first + n], s["gamma"][i], s["cos"][first:first + n], s["sin"][first:first + n])
        engine.end_step()
        torch.cuda.current_stream().synchronize()  # the driver takes a step's result before it begins the next
    first, n = int(s["host_lens"].sum()), case["seqs"]
    for t in range(case["steps"]):
        engine.begin_step(seqs)
        for i in range(case["layers"]):
            engine.layer_append(i, s["kv_a"][i][first:first + n], s["gamma"][i], s["cos"][first:first + n], s["sin"][first:first + n])
            engine.layer_attend(i, s["q"][t][i], s["out"][t][i], s["quant"][0][t][i], s["quant"][1][t][i])
        engine.end_step()
        torch.cuda.current_stream().synchronize()
        first += n
    for seq in seqs:
        engine.release(seq)
    return {"out": s["out"], "quant": list(s["quant"])}


def run(state):
    if "graph" in state:
        state["graph"].replay()
        return state["graph_out"]
    kind = state["case"]["kind"]
    if kind == "decode":
        return _decode_step(state)
    if kind == "shard":
        return _shard_step(state)
    if kind == "sparse":
        return _sparse_step(state)
    if kind == "serve":
        return _serve(state)
    if kind == "producer":
        latent_out, rope_out, rstd = state["copies"] or (None, None, None)
        b200kv.append_fused(state["view"], state["kv_a"], state["gamma"], state["cos"], state["sin"], state["slots"], latent_out=latent_out,
                            rope_out=rope_out, rstd_out=rstd, status=state["status"])
        return {"latent": state["latent"], "rope": state["rope"], "copies": list(state["copies"] or ())}
    b200kv.append(state["view"], state["new"][0], state["new"][1], state["slots"], status=state["status"])
    b200kv.gather(state["view"], state["table"], state["lens"], state["case"]["block"], state["out"][0], state["out"][1], state["offsets"],
                  state["total"], status=state["status"])
    return {"latent": state["out"][0], "rope": state["out"][1], "pool": [state["latent"], state["rope"]]}


# ---- what a pass cannot do without ----------------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind == "decode":
        tokens, rows = int(_lens(case).sum()), case["seqs"] * case["heads"]
        moved = tokens * ROW * 2 + rows * (ROW * 2 + LATENT * 2 + 4) + (case["seqs"] * ROW * 4 if case["append"] else 0)
        moved += rows * (LATENT + LATENT // 32) if case["quant"] else 0
        return {"bytes": case["layers"] * moved, "flops": case["layers"] * 2 * tokens * case["heads"] * (ROW + LATENT)}
    if kind == "shard":
        tokens, rows = case["seqs"] * case["shard"], case["seqs"] * 64
        moved = tokens * ROW * 2 + rows * (ROW * 2 + case["world"] * (LATENT + 2) * 4 + LATENT * 2 + 4)
        return {"bytes": case["layers"] * moved, "flops": case["layers"] * 2 * tokens * 64 * (ROW + LATENT)}
    if kind == "sparse":
        lens = _lens(case).astype(np.int64)
        tokens, kept = int(lens.sum()), int(np.minimum(lens, case["top"]).sum())
        moved = tokens * (INDEX_DIM + 4) + case["seqs"] * case["index_heads"] * (INDEX_DIM + 6) + case["seqs"] * case["top"] * 4
        flops = 2 * tokens * case["index_heads"] * INDEX_DIM
        if case["attend"]:
            moved += kept * ROW * 2 + case["seqs"] * 64 * (ROW * 2 + LATENT * 2 + 4) + case["seqs"] * case["top"] * 4
            flops += 2 * kept * 64 * (ROW + LATENT)
        return {"bytes": case["layers"] * moved, "flops": case["layers"] * flops}
    if kind == "serve":
        lens = _lens(case).astype(np.int64)
        appended = int(lens.sum()) + case["steps"] * case["seqs"]
        attended = sum(int((lens + t + 1).sum()) for t in range(case["steps"]))
        rows = case["steps"] * case["seqs"] * 64
        moved = appended * (2 * ROW * 2 + 2 * ROPE * 2 + 4) + attended * ROW * 2 + rows * (ROW * 2 + LATENT * 3 + LATENT // 32)
        return {"bytes": case["layers"] * moved, "flops": case["layers"] * 2 * attended * 64 * (ROW + LATENT)}
    if kind == "producer":
        return {"bytes": case["tokens"] * (2 * ROW * 2 + 2 * ROPE * 2 + 4 + (ROW * 2 + 4 if case["copies"] else 0)), "flops": case["tokens"] * 4 * ROW}
    lens = _lens(case).astype(np.int64)
    return {"bytes": int(2 * ROW * 2 * (lens.sum() + np.minimum(lens, case["chunk"]).sum())), "flops": 0}


def tolerance(case):
    kind = case["kind"]
    if kind == "chunk":
        return "exact"
    if kind == "producer":  # bf16 results of 32-bit arithmetic: another order of the sum of squares moves a few last places
        return {"rel": 1e-3, "max": 0.02}
    if kind == "sparse":  # positions between scores that differ by rounding only may change places
        return {"rel": 0.02, "max": 0.5, "differ": 0.005}
    # bf16 outputs of weights that are bf16 where the tensor cores take them; a quantised byte flips with its value
    return {"rel": 0.01, "max": 0.1, "differ": 0.01}


# ---- the same in 64 bits --------------------------------------------------------------------------------------------
def _attend64(q, latent, rope, rows, lo=0):
    """q [heads, 576], the sequence's pool rows: (out [heads, 512], lse [heads]) in 64 bits."""
    k, r = latent[rows].double(), rope[rows].double()
    q = q.double()
    s = (q[:, :LATENT] @ k.T + q[:, LATENT:] @ r.T) * SCALE
    lse = torch.logsumexp(s, dim=1)
    return torch.exp(s - lse[:, None]) @ k, lse


def _rows_of(state, b, block):
    t = np.arange(int(state["host_lens"][b]))
    return _dev(state["host_table"][b][t // block].astype(np.int64) * block + t % block)


def _produced64(kv_a, gamma, cos, sin):
    """The producer's rows in 64 bits: (latent, rope, reciprocal RMS)."""
    x = kv_a.double()
    rstd = 1.0 / torch.sqrt(x[:, :LATENT].square().mean(dim=1) + 1e-6)
    a, b, c, n = x[:, LATENT:LATENT + 32], x[:, LATENT + 32:], cos.double(), sin.double()
    return (x[:, :LATENT] * rstd[:, None] * gamma.double(),
            torch.cat([a * c[:, :32] - b * n[:, :32], b * c[:, 32:] + a * n[:, 32:]], dim=1), rstd)


def exact(case, seed):
    s = prepare({**case, "graph": False}, seed)
    kind = case["kind"]
    n, layers = case.get("seqs"), range(case.get("layers", 1))
    if kind == "decode":
        if case["append"]:
            last = _dev(_slots(s["host_table"], s["host_lens"], np.ones(n, dtype=np.int64), case["block"]).astype(np.int64))
            s["latent"][:, last] = s["new"][0]
            s["rope"][:, last] = s["new"][1]
        rows = [_rows_of(s, b, case["block"]) for b in range(n)]
        both = [[_attend64(s["q"][i][b], s["latent"][i], s["rope"][i], rows[b]) for b in range(n)] for i in layers]
        return {"out": torch.stack([torch.stack([o for o, _ in x]) for x in both]), "lse": torch.stack([torch.stack([e for _, e in x]) for x in both]),
                "quant": [None] * (2 if case["quant"] else 0), "pool": [s["latent"].double(), s["rope"].double()] if s["new"] else []}
    if kind == "shard":
        out, lse = torch.empty(s["out"].shape, dtype=torch.float64, device="cuda"), torch.empty(s["lse"].shape, dtype=torch.float64, device="cuda")
        for i in layers:
            for b in range(n):
                o, e = _attend64(s["q"][i][b], s["latent"][i], s["rope"][i], _rows_of(s, b, case["block"]))
                l, m = s["part_l"][i, 1:, b].double(), s["part_m"][i, 1:, b].double()
                each = torch.cat([e[None], m + l.log()])
                lse[i, b] = torch.logsumexp(each, dim=0)
                w = torch.exp(each - lse[i, b])
                out[i, b] = o * w[0][:, None] + (s["part_o"][i, 1:, b].double() / l[..., None] * w[1:, :, None]).sum(0)
        return {"out": out, "lse": lse}
    if kind == "sparse":
        if not case["attend"]:
            return None  # positions only: nothing that has a value in 64 bits
        out, lse = [], []
        for i in layers:
            for b in range(n):
                rows = _rows_of(s, b, case["block"])
                dot = s["index_q"][i][b].view(torch.float8_e4m3fn).double() @ s["keys"][i][rows].view(torch.float8_e4m3fn).double().T
                dot = torch.relu(dot * s["index_q_scale"][i][b].double()[:, None] * s["key_scale"][i][rows].double()[None, :])
                best = torch.topk((dot * s["weights"][i][b].double()[:, None]).sum(0), min(case["top"], len(rows))).indices
                o, e = _attend64(s["q"][i][b], s["latent"][i], s["rope"][i], rows[best])
                out.append(o)
                lse.append(e)
        return {"index": None, "count": None, "out": torch.stack(out).view(s["out"].shape), "lse": torch.stack(lse).view(s["lse"].shape)}
    if kind == "serve":
        out = torch.empty(s["out"].shape, dtype=torch.float64, device="cuda")
        prompt = int(s["host_lens"].sum())
        for i in layers:
            latent, rope, _ = _produced64(s["kv_a"][i], s["gamma"][i], s["cos"], s["sin"])
            latent, rope = latent.bfloat16(), rope.bfloat16()  # as the cache keeps them
            for t in range(case["steps"]):
                seen = s["owner"][:prompt + (t + 1) * n]
                for b in range(n):
                    out[t, i, b] = _attend64(s["q"][t][i][b], latent, rope, _dev(np.flatnonzero(seen == b)))[0]
        return {"out": out, "quant": [None, None]}
    if kind == "producer":
        latent, rope, rstd = _produced64(s["kv_a"], s["gamma"], s["cos"], s["sin"])
        pool = [s["latent"].double(), s["rope"].double()]
        pool[0][s["slots"].long()] = latent
        pool[1][s["slots"].long()] = rope
        return {"latent": pool[0], "rope": pool[1], "copies": [latent, rope, rstd] if case["copies"] else []}
    s["latent"][s["slots"].long()] = s["new"][0]
    s["rope"][s["slots"].long()] = s["new"][1]
    rows = torch.cat([_rows_of(s, b, case["block"]) for b in range(case["seqs"])])
    return {"latent": s["latent"][rows].double(), "rope": s["rope"][rows].double(), "pool": [s["latent"].double(), s["rope"].double()]}
