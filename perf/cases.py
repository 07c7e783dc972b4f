"""The work an inference engine has this library do, as cases that can be timed.

Three kinds of pass over a paged INT2/INT4 KV cache, all through the public entry points:

  decode    `PagedDecodeWrapper.run()` over the layers of a model, after one `plan()`
  step      a whole decode step: the step's plan, then per layer the append of one new token per
            request and the decode; eager (`plan()`) or with a captured graph (`update()` and one
            replay)
  append    the cache writer on a chunk of prompt tokens (`append`), or on whole pages where K is
            quantized per channel (`append_page_groups`)
  readback  `dequantize()` of a batch into bf16 rows

Shapes are those of this repository's benchmark workloads (bench.py) and tests: 32/8 heads x 128
(INT2 and INT4), 64/8 x 64 with 256 requests of very different lengths, 16/2 x 256 with K per
channel over a page, contexts of a few hundred to 131,072 tokens. Request lengths are quantiles of
the stated distribution, dealt to the requests in an order that the seed picks, so that a case's
work does not depend on the seed; pages are scattered over the pool; K has per-channel magnitudes
with outliers (log-normal), and q = e4m3(8 q) as the benchmark has it.
"""
import math

import numpy as np
import torch

from foscar_b200 import PagedDecodeWrapper, QuantKVLayout
from foscar_b200.wrapper import graph_workspace_bytes

PAGE = 64
Q_SCALE = 8.0
#: Tokens written by one append while a cache is filled (bounds the bf16 staging).
FILL_TOKENS = 1 << 18
#: Packed bytes of a drawn decode or step at most (the largest listed case has somewhat more).
MOST_BYTES = 1_600_000_000


def _decode(name, bits, batch, hq, hkv, d, lo, hi, dist="uniform", layers=1, k_channel=False,
            q_len=1):
    return dict(name=name, kind="decode", bits=bits, batch=batch, hq=hq, hkv=hkv, d=d, lo=lo,
                hi=hi, dist=dist, layers=layers, k_channel=k_channel, q_len=q_len,
                k_group=d, scale_bf16=False)


def _step(name, bits, batch, hq, hkv, d, lo, hi, layers, graph):
    return dict(name=name, kind="step", bits=bits, batch=batch, hq=hq, hkv=hkv, d=d, lo=lo, hi=hi,
                dist="uniform", layers=layers, graph=graph, k_channel=False, q_len=1, k_group=d,
                scale_bf16=False)


def _cache(name, kind, bits, hkv, d, tokens, requests, k_channel=False):
    return dict(name=name, kind=kind, bits=bits, hkv=hkv, d=d, tokens=tokens, requests=requests,
                k_channel=k_channel, k_group=d, scale_bf16=False, clip=False)


def listed():
    return [
        # A serving batch of mixed context lengths, the benchmark's default workload.
        _decode("decode-int2-mixed", 2, 32, 32, 8, 128, 4096, 32768),
        # The same batch for an engine that keeps four bits.
        _decode("decode-int4-mixed", 4, 32, 32, 8, 128, 4096, 32768),
        # Long documents: every request at the same long context.
        _decode("decode-int2-long", 2, 16, 32, 8, 128, 100352, 100352),
        # One interactive request with a ragged context: the launch's latency, layer after layer.
        _decode("decode-int2-single", 2, 1, 32, 8, 128, 32731, 32731, layers=8),
        # Many requests from one page to 131,072 tokens, eight query heads per KV head.
        _decode("decode-d64-skewed", 2, 256, 64, 8, 64, 64, 131072, dist="loguniform"),
        # head_dim 256 with K quantized per channel over a page.
        _decode("decode-d256-channel", 4, 64, 16, 2, 256, 256, 65536, dist="loguniform",
                k_channel=True),
        # A speculative step: two query tokens per request share one pass over the cache.
        _decode("decode-int2-two-tokens", 2, 16, 32, 8, 128, 8192, 16384, q_len=2),
        # A short eager step (a small batch just after its prompts): host work and launches count.
        _step("step-eager-small", 4, 2, 32, 8, 128, 128, 1024, layers=4, graph=False),
        # A step of an engine that replays a captured graph.
        _step("step-graph", 2, 24, 32, 8, 128, 512, 8192, layers=4, graph=True),
        # A chunk of prompt tokens of several requests, quantized and written.
        _cache("append-prompt-int2", "append", 2, 8, 128, 32768, 5),
        # Whole pages with K per channel, the last page of every request partly filled.
        _cache("append-pages-d256", "append", 4, 2, 256, 32768, 7, k_channel=True),
        # A batch read back into bf16 rows (prefix reuse by a bf16 prefill kernel).
        _cache("readback-int4", "readback", 4, 8, 128, 65000, 16),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the ranges the listed ones stand for."""
    kind = rng.choice(["decode", "decode", "decode", "decode", "step", "step", "append", "append",
                       "readback"])
    bits = rng.choice([2, 4])
    scale_bf16 = rng.random() < 0.2
    hq, hkv, d = rng.choice([(32, 8, 128), (32, 8, 128), (32, 4, 128), (64, 8, 64), (16, 2, 256),
                             (12, 4, 128), (8, 8, 64)])
    k_channel = d == 256 and rng.random() < 0.5
    # K in two groups of 64 channels is stored with bf16 records
    k_group = 64 if d == 128 and rng.random() < 0.15 else d
    scale_bf16 = not k_channel and (scale_bf16 or k_group < d)
    if kind in ("append", "readback"):
        return dict(kind=kind, bits=bits, hkv=hkv, d=d, tokens=_logint(rng, 700, 90000),
                    requests=rng.randint(1, 24), k_channel=k_channel, k_group=k_group,
                    scale_bf16=scale_bf16,
                    clip=kind == "append" and not k_channel and rng.random() < 0.2)
    if kind == "step":
        case = dict(kind="step", bits=bits, batch=_logint(rng, 1, 64), hq=hq, hkv=hkv, d=d,
                    lo=_logint(rng, 64, 1024), hi=0, dist="uniform", layers=rng.randint(2, 4),
                    graph=rng.random() < 0.5, k_channel=False, q_len=1, k_group=k_group,
                    scale_bf16=scale_bf16)
        case["hi"] = case["lo"] + _logint(rng, 1, 8192)
    else:
        case = dict(kind="decode", bits=bits, batch=_logint(rng, 1, 128), hq=hq, hkv=hkv, d=d,
                    lo=_logint(rng, 64, 65536), hi=0,
                    dist=rng.choice(["uniform", "loguniform"]), layers=1, k_channel=k_channel,
                    q_len=1 if k_channel or k_group < d or rng.random() < 0.8 else 2,
                    k_group=k_group, scale_bf16=scale_bf16)
        case["hi"] = min(131072, case["lo"] + _logint(rng, 1, 65536))
    while _packed_bytes(case) > MOST_BYTES:
        case["batch"] -= (case["batch"] + 3) // 4
    return case


# -- sizes ----------------------------------------------------------------------------------------

def _lengths(case):
    """The requests' lengths, shortest first: quantiles of the case's distribution."""
    if "tokens" in case:      # a chunk of tokens split over its requests unevenly
        n = case["requests"]
        shares = np.arange(1, n + 1, dtype=np.float64)
        cuts = np.round(np.cumsum(shares) / shares.sum() * case["tokens"]).astype(np.int64)
        return np.maximum(np.diff(np.concatenate([[0], cuts])), 1)
    at = (np.arange(case["batch"]) + 0.5) / case["batch"]
    lo, hi = case["lo"], case["hi"]
    if case["dist"] == "loguniform":
        return np.round(np.exp(math.log(lo) + at * (math.log(hi) - math.log(lo)))).astype(np.int64)
    return np.round(lo + at * (hi - lo)).astype(np.int64)


def _token_head_bytes(case):
    """Packed bytes of one token of one KV head: K and V codes and the scale records."""
    d = case["d"]
    width = 2 if case["scale_bf16"] else 4
    if case["k_channel"]:    # the V pair, and the page's channel pairs spread over its tokens
        records = (2 + 2 * d / PAGE) * 4
    else:
        records = (2 + 2 * d // case["k_group"]) * width
    return 2 * d * case["bits"] / 8 + records


def _packed_bytes(case):
    return float(_lengths(case).sum()) * case["hkv"] * _token_head_bytes(case) \
        * case.get("layers", 1)


def work(case):
    lens, d, hkv = _lengths(case), case["d"], case["hkv"]
    pages = int(sum(-(-int(n) // PAGE) for n in lens))
    if case["kind"] in ("append", "readback"):
        rows = float(lens.sum()) * hkv * 2 * d * 2
        return {"bytes": rows + _packed_bytes(case) + 8.0 * pages,
                "flops": float(lens.sum()) * hkv * 2 * d * 4}
    cols = case["batch"] * case["q_len"] * case["hq"]
    layers = case["layers"]
    moved = _packed_bytes(case) + layers * (cols * d * (1 + 2) + cols * 4 + 4.0 * pages)
    if case["kind"] == "step":
        moved += layers * case["batch"] * hkv * (2 * d * 2 + _token_head_bytes(case))
    flops = 4.0 * float(lens.sum()) * case["hq"] * case["q_len"] * d * layers
    return {"bytes": moved, "flops": flops}


def tolerance(case):
    """Appended bytes and read-back rows are exact. A decode rounds its weights to about eight
    bits and its output to bf16: measured against 64-bit attention over the same cache the output
    is off by 1.7e-3 to 3.3e-3 (2-norm; the largest difference 0.01 to 0.053 of the root mean
    square) and the lse by 1e-4 of its size."""
    if case["kind"] in ("append", "readback"):
        return "exact"
    return {"rel": 1.2e-2, "max": 0.22}


# -- inputs ---------------------------------------------------------------------------------------

def _paging(case, seed):
    """(lengths, indptr, page ids) of the requests on a scattered pool."""
    rng = np.random.default_rng(seed)
    lens = rng.permutation(_lengths(case))
    pages = -(-lens // PAGE)
    indptr = np.concatenate([[0], np.cumsum(pages)]).astype(np.int32)
    return lens, indptr, rng.permutation(int(pages.sum())).astype(np.int32)


def _slots(lens, indptr, indices):
    """Slot of every token of the batch, request after request (int64)."""
    request = np.repeat(np.arange(len(lens)), lens)
    position = np.arange(int(lens.sum())) - np.repeat(np.cumsum(lens) - lens, lens)
    page = indices[indptr[request] + position // PAGE].astype(np.int64)
    return page * PAGE + position % PAGE


def _layout(case):
    return QuantKVLayout.create(
        bits=case["bits"], head_dim=case["d"], num_kv_heads=case["hkv"], device="cuda",
        k_quant=("channel", PAGE) if case["k_channel"] else ("token", case["k_group"]),
        scale_dtype=torch.bfloat16 if case["scale_bf16"] else None)


def _new_cache(layout, pages):
    buffer = torch.zeros(pages * layout.bytes_per_page(), dtype=torch.uint8, device="cuda")
    return layout.bind(buffer, pages)


def _kv(case, tokens, gen, magnitude):
    shape = (tokens, case["hkv"], case["d"])
    k = torch.randn(shape, device="cuda", dtype=torch.bfloat16, generator=gen) * magnitude
    return k, torch.randn(shape, device="cuda", dtype=torch.bfloat16, generator=gen)


def _magnitude(case, gen):
    return torch.exp(torch.randn(1, case["hkv"], case["d"], device="cuda", generator=gen)).to(
        torch.bfloat16)


def _page_rows(case, lens, indptr, indices):
    """Whole pages of the batch for append_page_groups: page ids and valid tokens (int32)."""
    valid = np.full(len(indices), PAGE, dtype=np.int32)
    valid[indptr[1:] - 1] = lens - (np.diff(indptr) - 1) * PAGE
    return torch.from_numpy(indices).cuda(), torch.from_numpy(valid).cuda()


def _fill(case, cache, lens, indptr, indices, gen):
    """Write every token of the batch through the cache's own writer."""
    magnitude = _magnitude(case, gen)
    if case["k_channel"]:
        pages, valid = _page_rows(case, lens, indptr, indices)
        step = FILL_TOKENS // PAGE
        for a in range(0, len(indices), step):
            n = min(step, len(indices) - a)
            k, v = _kv(case, n * PAGE, gen, magnitude)
            cache.append_page_groups(k, v, pages[a:a + n], valid[a:a + n])
        return
    slots = torch.from_numpy(_slots(lens, indptr, indices)).cuda()
    for a in range(0, slots.numel(), FILL_TOKENS):
        part = slots[a:a + FILL_TOKENS]
        k, v = _kv(case, part.numel(), gen, magnitude)
        cache.append(k, v, part)


def _query(case, gen):
    shape = (case["batch"], case["hq"], case["d"])
    if case["q_len"] > 1:
        shape = (shape[0], case["q_len"], *shape[1:])
    q = torch.randn(shape, device="cuda", generator=gen) * Q_SCALE
    return q.clamp(-448, 448).to(torch.float8_e4m3fn)


def _prepare_decode(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    layout = _layout(case)
    lens, indptr, indices = _paging(case, seed)
    layers = []
    for _ in range(case["layers"]):
        cache = _new_cache(layout, len(indices))
        _fill(case, cache, lens, indptr, indices, gen)
        q = _query(case, gen)
        layer = dict(cache=cache, q=q,
                     out=torch.empty(q.shape, dtype=torch.bfloat16, device="cuda"),
                     lse=torch.empty(q.shape[:-1], dtype=torch.float32, device="cuda"))
        if case["kind"] == "step":     # the step's new token of every request, its last position
            layer["k"], layer["v"] = _kv(case, case["batch"], gen, _magnitude(case, gen))
        layers.append(layer)
    return dict(kind=case["kind"], hq=case["hq"], layout=layout, layers=layers,
                sm_scale=case["d"] ** -0.5 / Q_SCALE,
                lens=torch.from_numpy(lens.astype(np.int32)), indptr=torch.from_numpy(indptr),
                indices=torch.from_numpy(indices).cuda())


def _prepare_step(case, seed):
    state = _prepare_decode(case, seed)
    lens, indptr = state["lens"].long(), state["indptr"].long()
    last = state["indices"].cpu()[indptr[:-1] + (lens - 1) // PAGE].long()
    state["slots"] = (last * PAGE + (lens - 1) % PAGE).cuda()
    state["outputs"] = [(x["out"], x["cache"].k_codes, x["cache"].v_codes, x["cache"].scales)
                        for x in state["layers"]]
    if not case["graph"]:
        state["graph"] = None
        state["wrapper"] = PagedDecodeWrapper(
            torch.empty(64 << 20, dtype=torch.uint8, device="cuda"))
        return state
    batch, most = case["batch"], int(lens.max())
    table = torch.zeros(batch, -(-most // PAGE), dtype=torch.int32, device="cuda")
    for b in range(batch):
        row = state["indices"][indptr[b]:indptr[b + 1]]
        table[b, :row.numel()] = row
    room = graph_workspace_bytes(batch, case["hq"], state["layout"], max_kv_len=most)
    w = PagedDecodeWrapper(torch.empty(room, dtype=torch.uint8, device="cuda"),
                           use_cuda_graph=True)
    w.plan(page_table=table, seq_lens=state["lens"].cuda(), num_qo_heads=case["hq"],
           layout=state["layout"], max_kv_len=most, sm_scale=state["sm_scale"])
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph):
        _layers_of_a_step(w, state)
    state.update(wrapper=w, graph=graph, table=table, step_lens=state["lens"].numpy())
    return state


def _prepare_cache(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    layout = _layout(case)
    lens, indptr, indices = _paging(case, seed)
    cache = _new_cache(layout, len(indices))
    state = dict(kind=case["kind"], cache=cache, clip=None, pages=None)
    if case["kind"] == "readback":
        _fill(case, cache, lens, indptr, indices, gen)
        starts = np.cumsum(lens) - lens
        rows = (int(lens.sum()), case["hkv"], case["d"])
        state.update(k=torch.empty(rows, dtype=torch.bfloat16, device="cuda"),
                     v=torch.empty(rows, dtype=torch.bfloat16, device="cuda"),
                     indptr=torch.from_numpy(indptr).cuda(),
                     indices=torch.from_numpy(indices).cuda(),
                     lens=torch.from_numpy(lens.astype(np.int32)).cuda(),
                     starts=torch.from_numpy(starts).cuda())
        return state
    magnitude = _magnitude(case, gen)
    if case["k_channel"]:
        state["pages"], state["valid"] = _page_rows(case, lens, indptr, indices)
        state["k"], state["v"] = _kv(case, len(indices) * PAGE, gen, magnitude)
    else:
        state["slots"] = torch.from_numpy(_slots(lens, indptr, indices)).cuda()
        state["k"], state["v"] = _kv(case, int(lens.sum()), gen, magnitude)
        state["clip"] = 0.99 if case["clip"] else None
    state["outputs"] = (cache.k_codes, cache.v_codes, cache.scales,
                        cache.v_page_max.view(torch.int32), cache.v_max_hist.view(torch.int32))
    return state


def prepare(case, seed):
    if case["kind"] == "decode":
        state = _prepare_decode(case, seed)
        state["wrapper"] = PagedDecodeWrapper(
            torch.empty(256 << 20, dtype=torch.uint8, device="cuda"))
        state["wrapper"].plan(state["indptr"], state["indices"], state["lens"], case["hq"],
                              state["layout"], sm_scale=state["sm_scale"],
                              q_len_per_req=case["q_len"])
        return state
    if case["kind"] == "step":
        return _prepare_step(case, seed)
    return _prepare_cache(case, seed)


# -- one pass -------------------------------------------------------------------------------------

def _layers_of_a_step(wrapper, state):
    for layer in state["layers"]:
        layer["cache"].append(layer["k"], layer["v"], state["slots"])
        wrapper.run(layer["q"], layer["cache"], out=layer["out"])


def run(state):
    if state["kind"] == "decode":
        wrapper = state["wrapper"]
        for layer in state["layers"]:
            wrapper.run(layer["q"], layer["cache"], out=layer["out"], lse=layer["lse"])
        return [(layer["out"], layer["lse"]) for layer in state["layers"]]
    if state["kind"] == "step":
        wrapper = state["wrapper"]
        if state["graph"] is None:
            wrapper.plan(state["indptr"], state["indices"], state["lens"], state["hq"],
                         state["layout"], sm_scale=state["sm_scale"])
            _layers_of_a_step(wrapper, state)
        else:
            wrapper.update(state["step_lens"])
            state["graph"].replay()
        return state["outputs"]
    cache = state["cache"]
    if state["kind"] == "readback":
        cache.dequantize(state["k"], state["v"], state["indptr"], state["indices"],
                         state["lens"], state["starts"])
        return state["k"], state["v"]
    if state["pages"] is not None:
        cache.append_page_groups(state["k"], state["v"], state["pages"], state["valid"])
    else:
        cache.append(state["k"], state["v"], state["slots"], k_clip=state["clip"],
                     v_clip=state["clip"])
    return state["outputs"]
