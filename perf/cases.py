"""The work a user of this package has it do, as measurable cases.

A case is one pass through the public entry points: the decode step of one or several attention layers
(``SparseDecodeContext.decode_step``, its CUDA-graph replay, ``torch.ops.hashattn.decode_step``,
``decode_step_host``, ``decode_step_rows``) or the key-hash build of a prompt (``hash_prefill``). Sizes are those of
the package's own configurations and tests (32 query / 8 kv heads of 128, 1 kv-head where the heads are cut over 8
GPUs, contexts from a few hundred to 131072 tokens), or odd ones in between.

``listed()`` names the cases, ``draw()`` gives more of the same ranges. A decode case holds the caches of ``layers``
attention layers, visited one after the other as the layers of a model are.
"""
import importlib.util
import math
import os
import random
import sys

import torch


def _package():
    """The package directory's name is no identifier: it is imported as ``hashattention_b200``."""
    if "hashattention_b200" not in sys.modules:
        root = os.path.join(os.getcwd(), "hashattention-1.0_b200")
        spec = importlib.util.spec_from_file_location("hashattention_b200", os.path.join(root, "__init__.py"),
                                                      submodule_search_locations=[root])
        module = importlib.util.module_from_spec(spec)
        sys.modules["hashattention_b200"] = module
        spec.loader.exec_module(module)
    return sys.modules["hashattention_b200"]


ha = _package()
from hashattention_b200 import synthetic  # noqa: E402

DEVICE = torch.device("cuda:0")
GROUP, DIM = 4, 128
INIT, RECENT = 128, 128
HIDDEN_MACS = 128 * 128 + 128 * 128 + 128 * 32  # multiply-adds of one hash function


def _decode(name, call, batch, low, high, kv_heads=8, heavy=1.0 / 32, mode="simple", weights="bf16", layers=1, rows=1):
    case = dict(kind="decode", call=call, batch=batch, low=low, high=high, kv_heads=kv_heads, heavy=heavy, mode=mode,
                weights=weights, layers=layers, rows=rows)
    return dict(case, name=name) if name else case


def _prefill(name, batch, low, high, kv_heads=8, weights="bf16", tail=0):
    case = dict(kind="prefill", batch=batch, low=low, high=high, kv_heads=kv_heads, weights=weights, tail=tail)
    return dict(case, name=name) if name else case


def listed():
    return [
        # ---- decode steps: one new token per sequence
        # a short chat turn, one sequence, called step by step: all latency and launches
        _decode("short_eager", "eager", 1, 701, 701),
        # one 4K sequence under the model host: the registered operator on fp32 hash weights (what load_usa gives) and
        # the quarter budget that host's documentation configures
        _decode("host_model_4k_op_f32", "op", 1, 4096, 4096, heavy=0.25, weights="f32"),
        # one 32K sequence, the layers of a token replayed as one CUDA graph
        _decode("single_32k_graph", "graph", 1, 32768, 32768, layers=4),
        # one GPU's share of a model cut over 8 GPUs: one kv-head, a batch of 8 at 32K and a little
        _decode("shard_b8_33k_graph", "graph", 8, 33001, 33001, kv_heads=1, layers=4),
        # a serving batch of odd lengths whose q / k / v and output live in pinned host memory
        _decode("batch4_ragged_host", "host", 4, 7000, 24001, heavy=1.0 / 16),
        # long context: the largest uniform batch
        _decode("long_128k_graph", "graph", 4, 131072, 131072, layers=2),
        # a large ragged serving batch over scattered pages: the largest decode step
        _decode("batch32_ragged_graph", "graph", 32, 16384, 65536, heavy=1.0 / 16),
        # the depth rule (every candidate close to the best one), variable set sizes
        _decode("depth_rule_graph", "graph", 3, 9001, 15000, mode="depth", layers=2),
        # speculative / chunked decode: 16 new tokens for each of 2 sequences in one call
        _decode("chunk16_eager", "eager", 2, 20011, 20011, rows=16),
        # ---- key-hash build after (a piece of) the prompt has been prefilled
        # four 128K prompts: the largest build
        _prefill("prefill_4x128k", 4, 131072, 131072),
        # one odd-sized prompt on fp32 hash weights
        _prefill("prefill_20k_f32", 1, 20011, 20011, weights="f32"),
        # chunked prefill: the newest 1000 tokens of each of 6 growing prompts
        _prefill("prefill_tail_1000", 6, 3000, 30000, tail=1000),
    ]


def _log_uniform(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kv_heads = rng.choice([1, 2, 4, 8, 8, 8])
    batch = _log_uniform(rng, 1, 32)
    high = _log_uniform(rng, 500, 131072)
    low = high if rng.random() < 0.4 else max(300, high - rng.randrange(high // 2 + 1))
    weights = "f32" if rng.random() < 0.3 else "bf16"
    if rng.random() < 0.3:
        batch = min(batch, max(1, 524288 // high))
        tail = rng.choice([0, 0, 129, 512, 2048])
        return _prefill(None, batch, low, high, kv_heads, weights, tail if tail < low else 0)
    heavy = rng.choice([1.0 / 32, 1.0 / 32, 1.0 / 16, 1.0 / 8, 1.0 / 4, 512.0])
    call = rng.choice(["eager", "graph", "graph", "graph", "host", "op"])
    rows = 1
    if call == "eager" and rng.random() < 0.5:
        rows, batch = rng.choice([2, 5, 8, 32]), min(batch, 3)
        high = min(high, 40000)
        low = min(low, high)
    mode = "depth" if rng.random() < 0.15 else "simple"
    if mode == "depth":  # its sets have no fixed size: the index buffers cover the whole sequence
        high = min(high, 32768)
        low = min(low, high)
    batch = min(batch, max(1, 1300000 // high))
    while batch > 1 and _decode_bytes(_decode(None, call, batch, low, high, kv_heads, heavy, mode, weights, 1, rows)) > 1.4e9:
        batch -= 1
    layers = 1
    if call == "graph":
        one = _decode_bytes(_decode(None, call, batch, low, high, kv_heads, heavy, mode, weights, 1, rows))
        layers = 4 if one < 60e6 else 2 if one < 400e6 else 1
        if batch * high * kv_heads * 512 * layers > 6e9:
            layers = 1
    return _decode(None, call, batch, low, high, kv_heads, heavy, mode, weights, layers, rows)


def _lengths(case):
    """The cached lengths of the sequences: part of the case, so that another seed changes values and not sizes."""
    rng = random.Random(case["batch"] * 1000003 + case["low"] * 31 + case["high"])
    return [rng.randint(case["low"], case["high"]) for _ in range(case["batch"])]


def _budget(case):
    if case["mode"] == "depth":
        return ha.Budget(INIT, case["heavy"], RECENT, "depth", 6)
    return ha.Budget(INIT, case["heavy"], RECENT)


def _decode_bytes(case):
    """What a pass reads and writes at least: every token's codes once per sequence, the attended K / V rows (sink and
    recent rows once per kv-head, heavy rows once per query head), the hash weights of both sides, q, k, v and out.
    A chunk's rows share the codes and the edge rows; each of them has its own heavy rows."""
    lens, hq = _lengths(case), case["kv_heads"] * GROUP
    one = synthetic.algorithmic_bytes(lens, hq, case["kv_heads"], INIT, RECENT, case["heavy"])
    heavy_rows = 0
    for S in lens:
        hb = int(case["heavy"]) if case["heavy"] > 1.0 else int(S * case["heavy"])
        heavy_rows += 512 * hq * min(hb, max(0, S - INIT - RECENT))
    weights = 2 * hq * (HIDDEN_MACS * (2 if case["weights"] == "bf16" else 4) + 288 * 4)
    new = len(lens) * case["rows"] * DIM * 2 * (2 * hq + 2 * case["kv_heads"])
    # the depth rule's sets are no larger than the budget's plus the ties at its end: the budget stands for them
    return case["layers"] * (one["hash"] + one["kv"] + (case["rows"] - 1) * heavy_rows + weights + new)


def work(case):
    lens, hq = _lengths(case), case["kv_heads"] * GROUP
    if case["kind"] == "prefill":
        tokens = sum(min(S, case["tail"]) if case["tail"] else S for S in lens)
        return {"bytes": tokens * case["kv_heads"] * (DIM * 2 + GROUP * 4) +
                hq * (HIDDEN_MACS * (2 if case["weights"] == "bf16" else 4) + 288 * 4),
                "flops": 2.0 * HIDDEN_MACS * hq * tokens}
    rows = len(lens) * case["rows"]
    attended = 0
    for S in lens:
        hb = int(case["heavy"]) if case["heavy"] > 1.0 else int(S * case["heavy"])
        attended += min(S, INIT + RECENT) + min(hb, max(0, S - INIT - RECENT))
    flops = 2.0 * HIDDEN_MACS * 2 * hq * rows + 4.0 * DIM * hq * attended * case["rows"]
    return {"bytes": _decode_bytes(case), "flops": case["layers"] * flops}


def tolerance(case):
    # Codes are signs of sums with fp32 accuracy: a word may differ where one of its 32 sums is within rounding of zero.
    # Against a 64-bit evaluation, of 262144 words 3 differ with bf16 weights and 19 with fp32 ones.
    codes = 5e-5 if case["weights"] == "bf16" else 3e-4
    if case["kind"] == "prefill":
        return {"rel": 0.0, "max": 0.0, "differ": codes}
    # bf16 results of fp32 sums: against a 64-bit softmax over the same rows the 2-norm is off by 5e-5 and a value by at
    # most its last bit. A key code that differs (above) can swap one of a head's rows for another one of equal score,
    # which is what the norm's allowance is for.
    return {"rel": 2e-3, "max": 0.03, "differ": codes}


def _layer(case, lens, seed):
    kv_heads = case["kv_heads"]
    cache = ha.PagedHashKVCache(len(lens), kv_heads, max(lens), DEVICE, shuffle_seed=seed)
    synthetic.fill_cache_on_device(cache, lens, seed=seed)
    usa = synthetic.make_usa(kv_heads * GROUP, DIM, seed=seed, bf16=case["weights"] == "bf16")
    return cache, usa.packed(DEVICE)


def _new_rows(rows, kv_heads, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    q = torch.randn(rows, kv_heads * GROUP, DIM, generator=gen, device=DEVICE).bfloat16()
    k = torch.randn(rows, kv_heads, DIM, generator=gen, device=DEVICE)
    k[..., list(synthetic.OUTLIER_CHANNELS)] *= synthetic.OUTLIER_SCALE
    v = torch.randn(rows, kv_heads, DIM, generator=gen, device=DEVICE).bfloat16()
    return q, k.bfloat16(), v


def prepare(case, seed):
    """Filled caches (key codes built), hash weights and contexts, and the new token's q / k / v; for the graph call the
    captured graph of the token, for the host call the pinned buffers."""
    lens = _lengths(case)
    if case["kind"] == "prefill":
        cache, weights = _layer(case, lens, seed)
        ctx = ha.SparseDecodeContext(cache, ha.Budget(INIT, 1.0 / 32, RECENT), weights)
        first = None
        if case["tail"]:
            ctx.hash_prefill()  # the pieces in front have their codes already
            first = torch.tensor([max(0, S - case["tail"]) for S in lens], dtype=torch.int32, device=DEVICE)
        return {"case": case, "ctx": ctx, "first": first}

    state = {"case": case, "layers": []}
    for l in range(case["layers"]):
        cache, weights = _layer(case, lens, seed * 8 + l)
        ctx = ha.SparseDecodeContext(cache, _budget(case), weights)
        ctx.hash_prefill()
        q, k, v = _new_rows(len(lens) * case["rows"], case["kv_heads"], seed * 8 + l)
        if case["rows"] > 1:
            # the chunk's tokens are the last ones of the sequence
            cache.seq_lens -= case["rows"]
            chunk = ha.ChunkRows(cache, case["rows"])
            chunk.advance()
            ctx = ha.SparseDecodeContext(chunk, _budget(case), weights)
        state["layers"].append((ctx, q, k, v))
    if case["call"] == "graph":
        outs = [torch.empty_like(q) for _, q, _, _ in state["layers"]]
        side, graph = torch.cuda.Stream(DEVICE), torch.cuda.CUDAGraph()
        side.wait_stream(torch.cuda.current_stream(DEVICE))
        with torch.cuda.stream(side):
            for (ctx, q, k, v), out in zip(state["layers"], outs):
                ctx.decode_step(q, k, v, out=out)
            side.synchronize()
            with torch.cuda.graph(graph, stream=side):
                for (ctx, q, k, v), out in zip(state["layers"], outs):
                    ctx.decode_step(q, k, v, out=out)
        torch.cuda.current_stream(DEVICE).wait_stream(side)
        state["graph"], state["outs"] = graph, outs
    elif case["call"] == "host":
        (ctx, q, k, v), = state["layers"]
        buf = ha.HostStepBuffers(ctx)
        buf.q_host.copy_(q)
        buf.k_host.copy_(k)
        buf.v_host.copy_(v)
        ha.decode_step_host(ctx, buf, use_graph=True)  # records the graph the later steps replay
        state["buf"] = buf
    return state


def run(state):
    """One pass. Returns, per layer, the attention output, the query codes, the numbers of selected tokens and the
    cache the step has appended to; a key-hash build returns the code pages. (The selected indices are a set whose
    order is not part of the interface; the attention output follows from them.)"""
    case = state["case"]
    if case["kind"] == "prefill":
        state["ctx"].hash_prefill(state["first"])
        return state["ctx"].cache.hash_pages
    if case["call"] == "graph":
        state["graph"].replay()
        outs = state["outs"]
    elif case["call"] == "host":
        outs = [ha.decode_step_host(state["layers"][0][0], state["buf"], use_graph=True)]
    elif case["call"] == "op":
        outs = [ha.decode_step_op(ctx, q, k, v) for ctx, q, k, v in state["layers"]]
    elif case["rows"] > 1:
        outs = [ctx.decode_step_rows(q, k, v) for ctx, q, k, v in state["layers"]]
    else:
        outs = [ctx.decode_step(q, k, v) for ctx, q, k, v in state["layers"]]
    return [(out, ctx.q_codes, ctx.sel_cnt, ctx.cache.hash_pages, ctx.cache.k_pages, ctx.cache.v_pages)
            for out, (ctx, _, _, _) in zip(outs, state["layers"])]
