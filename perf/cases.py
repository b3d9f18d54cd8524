"""The calls a user of this package makes, over the sizes they make them at, for timing and comparison.

``listed()`` names representative cases and ``draw(rng)`` gives more of the same ranges; ``prepare`` makes what a
program holds before the call (inputs, caches, workspaces, operator objects), ``run`` is one pass through the public
operators, ``work`` the bytes and operations that pass cannot do without. Everything is BF16 with head dimension 128
and four query heads per KV head (32 / 8 heads unless a case holds a shard), the geometry the operators exist for;
the two-tile study also takes FP16.
"""
from __future__ import annotations

import functools
import math

import torch

from tilecadence_b200 import cuda_runtime

DIM, GROUP, HIDDEN = 128, 4, 2560
TILE_TOKENS = 64      # the two-tile study's fixed sequence length
MOST_CACHED = 4 * 32768          # rows of KV cache of the largest decode step
MOST_PREFILL = 32768 ** 2        # batch * tokens^2 of the largest prefill


def listed():
    return [
        # A chat turn's first answer tokens: one short sequence, where launches and the call path are everything.
        {"name": "decode_b1_511", "kind": "decode", "batch": 1, "capacity": 4096, "cached": 511, "ragged": False},
        # One long conversation in a cache with room to grow (the benchmark's single-sequence decode step).
        {"name": "decode_b1_8192", "kind": "decode", "batch": 1, "capacity": 32768, "cached": 8192, "ragged": False},
        # Long-context serving, four sequences at the end of a full cache (the benchmark's bandwidth-bound step).
        {"name": "decode_b4_32767", "kind": "decode", "batch": 4, "capacity": 32768, "cached": 32767, "ragged": False},
        # Continuous batching: sequences of very different lengths in a paged cache with a shuffled block table.
        {"name": "paged_b16_ragged", "kind": "paged", "batch": 16, "capacity": 8192, "cached": 8000, "ragged": True,
         "page": 64},
        # A small batch whose rotary embedding is left to the decode launch, lengths apart from each other.
        {"name": "rope_b8_ragged", "kind": "rope", "batch": 8, "capacity": 4096, "cached": 3333, "ragged": True},
        # A token through four layers of a model, projection and attention of each, captured once and replayed.
        {"name": "layers4_b4_4096", "kind": "layers", "batch": 4, "capacity": 4352, "cached": 4096, "layers": 4},
        # A short prompt of odd length: less than one wave of query tiles.
        {"name": "prefill_b1_333", "kind": "prefill", "batch": 1, "tokens": 333, "packed": False},
        # A batch of ordinary prompts, Q, K and V as views of one packed projection output.
        {"name": "prefill_b4_2048_packed", "kind": "prefill", "batch": 4, "tokens": 2048, "packed": True},
        # The benchmark's headline prefill.
        {"name": "prefill_b1_8192", "kind": "prefill", "batch": 1, "tokens": 8192, "packed": False},
        # The longest prompt the operator takes.
        {"name": "prefill_b1_32768", "kind": "prefill", "batch": 1, "tokens": 32768, "packed": False},
        # What one of eight GPUs holds of a long prompt split by KV head, ragged against the tile, key splits automatic.
        {"name": "prefill_shard_h4_8001", "kind": "shard", "batch": 1, "tokens": 8001, "heads": 4},
        # The generated two-tile kernel at the size its own benchmark times (192 heads, FP16).
        {"name": "two_tile_h192", "kind": "two_tile", "batch": 1, "heads": 192, "half": True},
    ]


def _spread(rng, low, high):
    """A whole number between low and high, even over its logarithm."""
    return max(low, min(high, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "paged", "rope", "layers", "prefill", "prefill", "prefill", "shard", "two_tile"))
    if kind in ("decode", "paged", "rope"):
        batch = rng.choice((1, 1, 2, 3, 4, 8, 16, 24, 32))
        cached = _spread(rng, 100, min(32767, MOST_CACHED // batch))
        case = {"kind": kind, "batch": batch, "capacity": min(32768, -(-(cached + 1) // 256) * 256), "cached": cached,
                "ragged": batch > 1 and rng.random() < 0.7}
        if kind == "paged":
            case["page"] = rng.choice((64, 128, 256))
        return case
    if kind == "layers":
        batch = rng.choice((1, 2, 3, 4, 8))
        cached = _spread(rng, 100, min(16384, 32768 // batch))
        return {"kind": kind, "batch": batch, "capacity": -(-(cached + 1) // 256) * 256, "cached": cached,
                "layers": rng.choice((2, 3, 4))}
    if kind == "two_tile":
        return {"kind": kind, "batch": rng.choice((1, 2, 4)), "heads": _spread(rng, 8, 192), "half": rng.random() < 0.5}
    batch = rng.choice((1, 1, 4))
    tokens = _spread(rng, 128, int(math.sqrt(MOST_PREFILL // batch)))
    if kind == "shard":
        return {"kind": kind, "batch": batch, "tokens": tokens, "heads": rng.choice((4, 8, 16))}
    return {"kind": kind, "batch": batch, "tokens": tokens, "packed": rng.random() < 0.5}


def _lengths(case):
    """Cached rows of each sequence: all the same, or from the longest down to a sixteenth of it, out of order."""
    if not case.get("ragged"):
        return [case["cached"]] * case["batch"]
    golden = (math.sqrt(5) - 1) / 2
    return [max(1, int(case["cached"] * 16.0 ** -((b * golden) % 1.0))) for b in range(case["batch"])]


@functools.cache
def _library():
    return cuda_runtime.default_library()


def _ops(phase, heads=32):
    return cuda_runtime.ops_for(_library(), phase, heads)


def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _source(seed):
    generator = torch.Generator(device=_device()).manual_seed(seed)

    def normal(*shape, scale=1.0, dtype=torch.bfloat16):
        values = torch.randn(shape, generator=generator, device=_device(), dtype=dtype)
        return values if scale == 1.0 else values.mul_(scale)

    return generator, normal


def _rope_tables(positions):
    """cos and sin, FP32 [positions, 64], of the usual rotary frequencies (base 1e6)."""
    frequency = 1e6 ** (-torch.arange(0, DIM, 2, device=_device(), dtype=torch.float64) / DIM)
    angle = torch.arange(positions, device=_device(), dtype=torch.float64)[:, None] * frequency
    return angle.cos().float().contiguous(), angle.sin().float().contiguous()


def _decode_buffers(ops, batch, capacity, heads=32):
    """Preallocated O, LSE and split workspace of a decode step."""
    out = torch.empty((batch, 1, heads, DIM), device=_device(), dtype=torch.bfloat16)
    lse = torch.empty((batch, heads, 1), device=_device(), dtype=torch.float32)
    spec = ops.indexed_workspace_spec(batch, capacity, heads // GROUP, _device().index)
    return [out, lse] + [torch.empty(n, device=_device(), dtype=torch.float32) for n in spec[1:3]]


def prepare(case, seed):
    generator, normal = _source(seed)
    kind, batch = case["kind"], case["batch"]
    state = {"kind": kind}
    if kind in ("decode", "paged", "rope"):
        ops = state["ops"] = _ops("decode")
        old = torch.tensor(_lengths(case), device=_device(), dtype=torch.int32)
        rows = (batch, case["capacity"])
        if kind == "paged":
            pages = -(-case["capacity"] // case["page"])
            pool = batch * pages + 8
            rows = (pool, case["page"])
            table = torch.randperm(pool, generator=generator, device=_device())[:batch * pages]
            state["table"] = table.view(batch, pages).to(torch.int32)
        kcache, vcache = normal(*rows, 8, DIM), normal(*rows, 8, DIM)
        q, knew, vnew = normal(batch, 1, 32, DIM), normal(batch, 1, 8, DIM), normal(batch, 1, 8, DIM)
        capacity = pages * case["page"] if kind == "paged" else case["capacity"]
        state["args"] = [q, kcache, vcache, knew, vnew, old, *_decode_buffers(ops, batch, capacity), 0, 1, True]
        if kind == "rope":
            state["tables"] = _rope_tables(case["capacity"])
    elif kind == "layers":
        state["graph"], state["results"], state["held"] = _capture_layers(case, normal)
    elif kind in ("prefill", "shard"):
        heads, tokens = case.get("heads", 32), case["tokens"]
        ops = state["ops"] = _ops("prefill", heads)
        if case.get("packed"):
            qkv = normal(batch, tokens, heads + heads // 2, DIM)
            q, k, v = qkv.split((heads, heads // GROUP, heads // GROUP), dim=2)
        else:
            q, k, v = (normal(batch, tokens, n, DIM) for n in (heads, heads // GROUP, heads // GROUP))
        out = torch.empty((batch, tokens, heads, DIM), device=_device(), dtype=torch.bfloat16)
        lse = torch.empty((batch, heads, tokens), device=_device(), dtype=torch.float32)
        if kind == "shard":
            workspace = torch.empty(ops.key_split_workspace_bytes(q), device=_device(), dtype=torch.uint8)
            state["args"] = [q, k, v, out, lse, workspace, 1, DIM ** -0.5]
        else:
            empty = torch.empty(0, device=_device(), dtype=torch.float32)
            state["args"] = [q, k, v, out, lse, empty, empty, 0, 1, DIM ** -0.5, True]
    else:
        state["ops"] = _ops("exchange")
        dtype, shape = torch.float16 if case["half"] else torch.bfloat16, (batch, TILE_TOKENS, case["heads"], DIM)
        q, k, v = (normal(*shape, dtype=dtype) for _ in range(3))
        lse = torch.empty((batch, case["heads"], TILE_TOKENS), device=_device(), dtype=torch.float32)
        state["args"] = [q, k, v, torch.empty_like(q), lse, None, False]
    return state


def _capture_layers(case, normal):
    """One new token per sequence through `layers` layers: every layer projects (its own weights, head norms, rotary
    embedding) and attends over its own cache. The calls carry the promises that hold in such a chain: a layer's
    projection writes no cache, and two kernels back another layer's cache was in use."""
    batch, capacity, layers = case["batch"], case["capacity"], case["layers"]
    project, decode = _ops("project"), _ops("decode")
    cos, sin = _rope_tables(capacity)
    old = torch.full((batch,), case["cached"], device=_device(), dtype=torch.int32)
    plan = []
    for _ in range(layers):
        weights = normal(48 * DIM, HIDDEN, scale=HIDDEN ** -0.5)
        norms = [1 + normal(DIM, scale=0.1) for _ in range(2)]
        caches = [normal(batch, capacity, 8, DIM) for _ in range(2)]
        x = normal(batch, HIDDEN)
        token = [torch.empty((batch, 1, n, DIM), device=_device(), dtype=torch.bfloat16) for n in (32, 8, 8)]
        plan.append((weights, norms, caches, x, token, _decode_buffers(decode, batch, capacity)))

    def step():
        for weights, norms, caches, x, (q, knew, vnew), buffers in plan:
            project.forward_out(x, weights, old, q, knew, vnew, q_norm_weight=norms[0], k_norm_weight=norms[1],
                                rope_cos=cos, rope_sin=sin, release_early=True)
            decode.forward_out(q, *caches, knew, vnew, old, *buffers, 0, 1, True, cache_stable=True)

    stream = torch.cuda.Stream(_device())
    stream.wait_stream(torch.cuda.current_stream(_device()))
    with torch.cuda.stream(stream):
        step()
        stream.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            step()
    results = [[token, caches, buffers[:2]] for _, _, caches, _, token, buffers in plan]
    return graph, results, (plan, cos, sin, old)


def run(state):
    kind = state["kind"]
    if kind == "layers":
        state["graph"].replay()
        return state["results"]
    args = state["args"]
    if kind == "decode":
        state["ops"].forward_out(*args)
    elif kind == "paged":
        state["ops"].indexed_forward_out(*args, block_table=state["table"])
    elif kind == "rope":
        state["ops"].rope_forward_out(*args, *state["tables"])
    elif kind == "prefill":
        state["ops"].forward_out(*args)
        return args[3:5]
    elif kind == "shard":
        state["ops"].key_split_forward_out(*args)
        return args[3:5]
    else:
        state["ops"].forward_out(*args)
        return args[3:5]
    return [args[6], args[7], args[1], args[2]]  # O, LSE and both caches with the appended rows


def _decode_work(lengths, heads=32):
    """One decode step: K and V of every visible row and the new row, Q, O and LSE; QK^T and PV over those rows."""
    seen, kv_heads, batch = sum(n + 1 for n in lengths), heads // GROUP, len(lengths)
    moved = seen * kv_heads * DIM * 2 * 2 + batch * (2 * heads * DIM * 2 + heads * 4 + 2 * kv_heads * DIM * 2)
    return moved, 4 * seen * heads * DIM


def work(case):
    kind, batch = case["kind"], case["batch"]
    if kind in ("decode", "paged", "rope"):
        moved, flops = _decode_work(_lengths(case))
        if kind == "rope":
            moved += batch * DIM * 4
        elif kind == "paged":
            moved += sum(-(-(n + 1) // case["page"]) for n in _lengths(case)) * 4
    elif kind == "layers":
        rows = 48 * DIM
        moved, flops = _decode_work([case["cached"]] * batch)
        moved += rows * HIDDEN * 2 + batch * (HIDDEN + rows) * 2
        flops += 2 * rows * HIDDEN * batch
        moved, flops = moved * case["layers"], flops * case["layers"]
    elif kind == "two_tile":
        elements = batch * TILE_TOKENS * case["heads"] * DIM
        moved = 4 * elements * 2 + batch * case["heads"] * TILE_TOKENS * 4
        flops = 4 * elements * TILE_TOKENS
    else:
        heads, tokens = case.get("heads", 32), case["tokens"]
        moved = batch * tokens * (2 * heads + heads // 2) * DIM * 2 + batch * heads * tokens * 4
        flops = 4 * batch * heads * DIM * tokens * (tokens + 1) // 2
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """O is rounded to the 16-bit type, and so are the probabilities ahead of PV: against FP64 the operators are off by
    2.2e-3 (BF16) and 2.6e-4 (FP16) in the 2-norm, by up to 0.055 and 0.001 of the root mean square in one value (early
    causal rows average few values and stand far above it). LSE agrees to 1e-7. About four times that is allowed."""
    if case["kind"] == "two_tile" and case["half"]:
        return {"rel": 1.1e-3, "max": 5e-3}
    return {"rel": 8e-3, "max": 0.2}


def _attend(q, k, v, visible, scale):
    """Attention in 64 bits of [rows, 128] queries over [keys, 128]: row r sees the first visible[r] keys (all: None)."""
    scores = (q @ k.T).mul_(scale)
    if visible is not None:
        seen = torch.arange(k.size(0), device=k.device)[None, :] < visible[:, None]
        scores.masked_fill_(~seen, -math.inf)
    lse = scores.logsumexp(-1)
    return scores.sub_(lse[:, None]).exp_() @ v, lse


def _rotate(x, cos, sin):
    """Rotate-half embedding of x [batch, 1, heads, 128] by the tables' rows cos, sin [batch, 64]."""
    (lo, hi), (c, s) = x.double().chunk(2, -1), (t.double()[:, None, None, :] for t in (cos, sin))
    return torch.cat([lo * c - hi * s, hi * c + lo * s], -1)


def _exact_decode(q, knew, vnew, kcache, vcache, old, table=None):
    """O, LSE and the caches after one decode step: the caches keep their type, everything computed is in 64 bits."""
    out, lse, caches = torch.empty_like(q, dtype=torch.float64), [], [kcache.clone(), vcache.clone()]
    for b, rows in enumerate(old.tolist()):
        seen = []
        for cache, new in zip(caches, (knew, vnew)):
            if table is None:
                cache[b, rows], sequence = new[b, 0].to(cache.dtype), cache[b]
            else:
                page, row = divmod(rows, cache.size(1))
                cache[table[b, page], row] = new[b, 0]
                sequence = cache[table[b, :page + 1].long()].flatten(0, 1)
            seen.append(torch.cat([sequence[:rows].double(), new[b].double()]))
        parts = [_attend(q[b, 0, h * GROUP:(h + 1) * GROUP].double(), seen[0][:, h], seen[1][:, h], None, DIM ** -0.5)
                 for h in range(kcache.size(2))]
        out[b, 0] = torch.cat([o for o, _ in parts])
        lse.append(torch.cat([l for _, l in parts]))
    return [out, torch.stack(lse)[:, :, None], *caches]


def _exact_layers(state):
    plan, cos, sin, old = state["held"]
    results = []
    for weights, norms, caches, x, _, _ in plan:
        y = (x.double() @ weights.double().T).view(x.size(0), 1, 48, DIM)
        q, k, v = y.split((32, 8, 8), dim=2)
        at = old.long()
        q, k = (_rotate(t * (t.pow(2).mean(-1, keepdim=True) + 1e-6).rsqrt() * norm.double(), cos[at], sin[at])
                for t, norm in ((q, norms[0]), (k, norms[1])))
        out, lse, kcache, vcache = _exact_decode(q, k, v, *caches, old)
        results.append([[q, k, v], [kcache, vcache], [out, lse]])
    return results


def exact(case, seed):
    """What `run` returns for these inputs, computed in 64 bits by plain torch."""
    state = prepare(case, seed)
    kind = case["kind"]
    if kind == "layers":
        return _exact_layers(state)
    args = state["args"]
    if kind in ("decode", "paged", "rope"):
        q, kcache, vcache, knew, vnew, old = args[:6]
        if kind == "rope":
            cos, sin = (t[old.long()] for t in state["tables"])
            q, knew = _rotate(q, cos, sin), _rotate(knew, cos, sin)
        return _exact_decode(q, knew, vnew, kcache, vcache, old, state.get("table"))
    q, k, v = args[:3]
    batch, tokens, heads, _ = q.shape
    group, causal = heads // k.size(2), kind != "two_tile"
    out = torch.empty(q.shape, device=q.device, dtype=torch.float64)
    lse = torch.empty((batch, heads, tokens), device=q.device, dtype=torch.float64)
    step = 2048
    for b in range(batch):
        for h in range(heads):
            keys, values = (t[b, :, h // group].double() for t in (k, v))
            for at in range(0, tokens, step):
                end = min(at + step, tokens)
                last = end if causal else tokens
                visible = torch.arange(at + 1, end + 1, device=q.device) if causal else None
                out[b, at:end, h], lse[b, h, at:end] = _attend(q[b, at:end, h].double(), keys[:last], values[:last],
                                                               visible, DIM ** -0.5)
    return [out, lse]
