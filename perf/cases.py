"""The work that users of this framework have it do, as cases that can be timed and compared.

A case is one step of a serving or chat program on the KV-cache path, through the public entry
points of orinmllm_b200.capi: a decode step (RoPE, append of the new token, attention over the
cache), the prefill of prompts in chunks, or the fork of sequences that share blocks.
"""
import math

import numpy as np
import torch

from orinmllm_b200 import capi

D, BS = 128, 16  # head size, tokens per block
THETA, EPS = 1e6, 1e-6
DTYPES = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}


def decode(name, q, kv, dtype, batch, lo, hi, layers, call, norm=False, layout="paged", shared=0):
    """One decode step of `batch` sequences with lo..hi cached tokens over `layers` layers.
    call: "eager" = append and attention launched layer by layer; "planned" = the same with the
    step's plan; "fused" = one launch per layer; "graph" = the planned step as a CUDA graph."""
    return dict(name=name, kind="decode", q=q, kv=kv, dtype=dtype, batch=batch, lo=lo, hi=hi, layers=layers, call=call,
                norm=norm, layout=layout, shared=shared)


def prefill(name, q, kv, dtype, batch, lo, hi, chunk, norm=False):
    """The prompts of `batch` sequences, lo..hi tokens each, through one layer in chunks."""
    return dict(name=name, kind="prefill", q=q, kv=kv, dtype=dtype, batch=batch, lo=lo, hi=hi, chunk=chunk, norm=norm)


def fork(name, kv, dtype, pairs, layers):
    """Copy-on-write of `pairs` shared blocks in every layer, with their reference counts."""
    return dict(name=name, kind="fork", kv=kv, dtype=dtype, pairs=pairs, layers=layers)


def listed():
    return [
        # one chat on the reference's own fp32 contiguous cache (Qwen2.5-1.5B heads and layers)
        decode("chat_f32_ctx512", 12, 2, "f32", 1, 512, 512, 28, "eager", layout="contiguous"),
        # one chat in production: Qwen3-8B heads and layers, the step replayed as a CUDA graph
        decode("chat_graph_ctx2000", 32, 8, "f16", 1, 2000, 2000, 36, "graph", norm=True),
        # a few short requests, every layer of the step in one launch
        decode("few_fused_bs8", 12, 2, "f16", 8, 64, 1024, 28, "fused"),
        # the headline serving batch: Qwen3-8B heads, 64 requests of 128..4096 tokens
        decode("serve_32x8_bs64", 32, 8, "f16", 64, 128, 4096, 4, "planned", norm=True),
        # the same batch at the Qwen2.5-7B heads (seven query heads per KV head), bf16
        decode("serve_28x4_bs64", 28, 4, "bf16", 64, 128, 4096, 4, "planned"),
        # long-context serving: 8k..32k tokens a request, all launched by hand
        decode("long_ctx_bs16", 32, 8, "f16", 16, 8192, 32768, 1, "eager", norm=True),
        # one very long document
        decode("one_seq_131072", 32, 8, "f16", 1, 131072, 131072, 2, "planned"),
        # requests that share a 1024-token system prompt through the prefix cache
        decode("prefix_shared_bs256", 32, 8, "f16", 256, 1280, 1408, 2, "planned", norm=True, shared=1024),
        # batched prompts as the scheduler feeds them: 4 x 2048 tokens in chunks of 512
        prefill("prefill_4x2048_chunk512", 28, 4, "bf16", 4, 2048, 2048, 512),
        # one short question of odd length, all at once: time to first token
        prefill("prefill_1x777", 32, 8, "f16", 1, 777, 777, 1024, norm=True),
        # one long document in chunks of 2048
        prefill("prefill_1x16384_chunk2048", 32, 8, "bf16", 1, 16384, 16384, 2048, norm=True),
        # 255 requests part from a common partly filled block
        fork("fork_255_blocks", 8, "f16", 255, 36),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    """One more case of the same ranges.  Head layouts are those of the listed cases and of the
    repository's parity tests."""
    kind = rng.choices(["decode", "prefill", "fork"], [7, 4, 1])[0]
    q, kv = rng.choice([(32, 8), (32, 8), (28, 4), (12, 2), (16, 2), (40, 8), (64, 8), (14, 2), (8, 8)])
    norm = rng.random() < 0.5
    if kind == "fork":
        return {k: v for k, v in fork("", kv, rng.choice(["f16", "bf16"]), _log_int(rng, 1, 255), rng.choice([2, 28, 36])).items() if k != "name"}
    if kind == "prefill":
        dtype = rng.choices(["f16", "bf16", "f32"], [5, 5, 1])[0]
        batch = rng.choice([1, 1, 2, 4, 8])
        top = 400 if dtype == "f32" else 9000 // batch
        hi = _log_int(rng, 20, top)
        lo = hi if rng.random() < 0.5 else max(1, int(hi * rng.uniform(0.2, 1.0)))
        c = prefill("", q, kv, dtype, batch, lo, hi, rng.choice([256, 512, 1024, 2048]), norm)
        return {k: v for k, v in c.items() if k != "name"}
    dtype = rng.choices(["f16", "bf16", "f32"], [5, 4, 1])[0]
    call = rng.choice(["eager", "planned", "fused", "graph"])
    batch = _log_int(rng, 1, 256)
    layout = "contiguous" if batch == 1 and rng.random() < 0.4 else "paged"
    tokens = (1_000_000 if dtype == "f32" else 2_000_000) // (batch * kv)  # per sequence, as many as the largest case holds
    hi = _log_int(rng, 16, min(131072, max(64, tokens)))
    lo = max(1, int(hi * rng.choice([0.03, 0.25, 1.0])))
    room = tokens / max(hi, 1)
    layers = 28 if room > 100 else (4 if room > 4 else 1)
    shared = 0
    if layout == "paged" and batch > 4 and lo > 64 and rng.random() < 0.25:
        shared = int(lo * rng.uniform(0.3, 0.9)) // BS * BS
    c = decode("", q, kv, dtype, batch, lo, hi, layers, call, norm and call != "fused", layout, shared)
    return {k: v for k, v in c.items() if k != "name"}


def _lengths(case):
    """lo..hi, evenly spread: the work of a case does not depend on the seed (the order does)."""
    n, lo, hi = case["batch"], case["lo"], case["hi"]
    return [lo + int((hi - lo) * (i + 0.5) / n) for i in range(n)]


def _sin_cos(max_pos):
    sin = torch.empty(max_pos * D, device="cuda", dtype=torch.float32)
    cos = torch.empty_like(sin)
    capi.sin_cos_cache(sin, cos, D, max_pos, THETA)
    return sin, cos


def _place(lens, rng, shared=0):
    """Block table int32 [batch, widest] of a seeded random placement in a pool 1.25 times the
    need; the first `shared` tokens of all sequences lie in the same blocks."""
    sb = shared // BS
    own = [-(-n // BS) - sb for n in lens]
    blocks = math.ceil((sb + sum(own)) * 1.25)
    ids = rng.permutation(blocks).astype(np.int32)
    table = np.zeros((len(lens), sb + max(own)), np.int32)
    table[:, :sb] = ids[:sb]
    at = sb
    for i, n in enumerate(own):
        table[i, sb:sb + n] = ids[at:at + n]
        at += n
    return table, blocks


def _new_rows(layers, rows, q, kv, dtype, gen):
    """q, k and v rows of every layer as the projections leave them: one buffer per tensor, and the
    pristine values that each pass starts from (RoPE works in place)."""
    n_q, n_k = layers * rows * q * D, layers * rows * kv * D
    fresh = torch.randn(n_q + n_k, generator=gen, device="cuda", dtype=dtype)
    qk = torch.empty_like(fresh)
    v = torch.randn(layers, rows, kv * D, generator=gen, device="cuda", dtype=dtype)
    return dict(fresh=fresh, qk=qk, q=list(qk[:n_q].view(layers, rows, q * D)),
                k=list(qk[n_q:].view(layers, rows, kv * D)), v=list(v))


def _norms(gen):
    return [1 + 0.2 * torch.randn(D, generator=gen, device="cuda") for _ in range(2)]


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    dtype = DTYPES[case["dtype"]]
    code = capi.dtype_code(dtype)
    kv = case["kv"]
    if case["kind"] == "fork":
        n = case["pairs"]
        blocks = 2 * n + 2
        ids = torch.from_numpy(rng.permutation(blocks).astype(np.int32)).cuda()
        shape = (case["layers"], blocks, kv, BS, D)
        return dict(case=case, n=n, blocks=blocks, layout=capi.layout_paged(code, kv, D, BS, blocks),
                    kp=torch.randn(shape, generator=gen, device="cuda", dtype=dtype),
                    vp=torch.randn(shape, generator=gen, device="cuda", dtype=dtype),
                    stride=blocks * kv * BS * D, src=ids[:n], dst=ids[n:2 * n], ids=ids[:2 * n].contiguous(),
                    # a source gives one reference back, its copy takes one
                    deltas=torch.cat([torch.full((n,), -1), torch.full((n,), 1)]).to(torch.int32).cuda(),
                    counts=torch.full((blocks,), 1 << 30, dtype=torch.int32, device="cuda"),
                    errors=torch.zeros(1, dtype=torch.int32, device="cuda"))
    lens = _lengths(case)
    if case["kind"] == "prefill":
        return _prepare_prefill(case, lens, dtype, code, gen, rng)
    lens = [lens[i] for i in rng.permutation(len(lens))]
    layers, batch = case["layers"], case["batch"]
    if case["layout"] == "contiguous":
        blocks = -(-(lens[0] + 1) // BS)
        layout = capi.layout_contiguous(code, kv, D, BS, blocks)
        shape, table, width = (layers, blocks * BS, kv * D), None, 0
        slots = np.asarray(lens, np.int64)
    else:
        table, blocks = _place([n + 1 for n in lens], rng, case["shared"])
        layout = capi.layout_paged(code, kv, D, BS, blocks)
        shape, width = (layers, blocks, kv, BS, D), table.shape[1]
        slots = np.asarray([int(table[i, n // BS]) * BS + n % BS for i, n in enumerate(lens)], np.int64)
        table = torch.from_numpy(table).cuda()
    s = _new_rows(layers, batch, case["q"], kv, dtype, gen)
    sin, cos = _sin_cos(max(lens) + 1)
    wsb = capi.decode_workspace_bytes(batch, case["q"], kv, D)
    s.update(case=case, layout=layout, width=width, table=table, sin=sin, cos=cos, batch=batch, wsb=wsb,
             kp=torch.randn(shape, generator=gen, device="cuda", dtype=dtype),
             vp=torch.randn(shape, generator=gen, device="cuda", dtype=dtype),
             pos=torch.tensor(lens, dtype=torch.int32, device="cuda"), slots=torch.from_numpy(slots).cuda(),
             out=torch.zeros(layers, batch, case["q"] * D, device="cuda", dtype=dtype), norms=_norms(gen),
             ws=torch.empty(wsb, dtype=torch.uint8, device="cuda"), scale=1 / math.sqrt(D))
    s.update(kps=list(s["kp"]), vps=list(s["vp"]), outs=list(s["out"]), plan=None)
    capi.workspace_init(s["ws"], wsb)
    if case["call"] in ("planned", "graph"):
        s["plan"] = torch.zeros(capi.decode_plan_bytes(), dtype=torch.uint8, device="cuda")
    if case["call"] == "graph":
        _decode_step(s)  # first use sets the kernels up
        torch.cuda.synchronize()
        s["graph"] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(s["graph"]):
            _decode_step(s)
    return s


def _prepare_prefill(case, lens, dtype, code, gen, rng):
    kv, chunk = case["kv"], case["chunk"]
    table, blocks = _place(lens, rng)
    steps, done = [], [0] * len(lens)
    while any(d < n for d, n in zip(done, lens)):  # every unfinished prompt gives its next chunk
        live = [i for i, n in enumerate(lens) if done[i] < n]
        take = [min(chunk, lens[i] - done[i]) for i in live]
        pos = np.concatenate([np.arange(done[i], done[i] + t) for i, t in zip(live, take)])
        seq = np.repeat(live, take)
        slots = table[seq, pos // BS].astype(np.int64) * BS + pos % BS
        steps.append(dict(n=len(pos), rows=len(live), cu=np.concatenate([[0], np.cumsum(take)]).astype(np.int32),
                          start=np.asarray([done[i] for i in live], np.int32),
                          pos=torch.from_numpy(pos.astype(np.int32)).cuda(), slots=torch.from_numpy(slots).cuda(),
                          table=torch.from_numpy(table[live]).cuda()))
        for i, t in zip(live, take):
            done[i] += t
    total = sum(lens)
    s = _new_rows(1, total, case["q"], kv, dtype, gen)
    shape = (blocks, kv, BS, D)
    wsb = capi.prefill_workspace_bytes(max(st["n"] for st in steps), case["q"], kv, D)
    sin, cos = _sin_cos(max(lens))
    s.update(case=case, steps=steps, layout=capi.layout_paged(code, kv, D, BS, blocks), width=table.shape[1], sin=sin, cos=cos,
             kp=torch.randn(shape, generator=gen, device="cuda", dtype=dtype),
             vp=torch.randn(shape, generator=gen, device="cuda", dtype=dtype), norms=_norms(gen),
             out=torch.zeros(total, case["q"] * D, device="cuda", dtype=dtype), scale=1 / math.sqrt(D),
             ws=torch.empty(wsb, dtype=torch.uint8, device="cuda"), wsb=wsb)
    capi.workspace_init(s["ws"], wsb)
    at = 0
    for st in steps:
        a, b = at, at + st["n"]
        st.update(q=s["q"][0][a:b], k=s["k"][0][a:b], v=s["v"][0][a:b], out=s["out"][a:b])
        at = b
    return s


def _append(s, q, k, v, pos, kp, vp, slots, n):
    case = s["case"]
    if case["norm"]:
        capi.norm_rope_append(q, k, v, case["q"], s["norms"][0], s["norms"][1], EPS, pos, s["sin"], s["cos"], kp, vp,
                              s["layout"], slots, n)
    else:
        capi.rope_append(q, k, v, case["q"], pos, s["sin"], s["cos"], kp, vp, s["layout"], slots, n)


def _decode_step(s):
    case, b, h = s["case"], s["batch"], s["case"]["q"]
    s["qk"].copy_(s["fresh"])  # the projections' results
    if s["plan"] is not None:
        capi.decode_plan(s["plan"], s["plan"].numel(), s["layout"], s["table"], s["width"], s["pos"], 1, b, h)
    for q, k, v, kp, vp, out in zip(s["q"], s["k"], s["v"], s["kps"], s["vps"], s["outs"]):
        if case["call"] == "fused":
            capi.rope_append_decode(out, q, k, v, s["sin"], s["cos"], kp, vp, s["layout"], s["table"], s["width"], s["pos"], b, h,
                                    s["scale"], s["ws"], s["wsb"])
            continue
        _append(s, q, k, v, s["pos"], kp, vp, s["slots"], b)
        if s["plan"] is not None:
            capi.paged_decode_planned(out, q, kp, vp, s["layout"], s["table"], s["width"], s["pos"], 1, b, h, s["scale"],
                                      s["ws"], s["wsb"], s["plan"])
        else:
            capi.paged_decode(out, q, kp, vp, s["layout"], s["table"], s["width"], s["pos"], 1, b, h, s["scale"], s["ws"],
                              s["wsb"])


def run(s):
    kind = s["case"]["kind"]
    if kind == "fork":
        capi.cow_copy_blocks(s["kp"], s["vp"], s["layout"], s["case"]["layers"], s["stride"], s["src"], s["dst"], s["n"])
        capi.refcount_update(s["counts"], s["blocks"], s["ids"], s["deltas"], 2 * s["n"], s["errors"])
        return dict(k=s["kp"], v=s["vp"], counts=s["counts"], errors=s["errors"])
    if kind == "decode":
        if s["case"]["call"] == "graph":
            s["graph"].replay()
        else:
            _decode_step(s)
    else:
        s["qk"].copy_(s["fresh"])
        for st in s["steps"]:
            _append(s, st["q"], st["k"], st["v"], st["pos"], s["kp"], s["vp"], st["slots"], st["n"])
            capi.paged_prefill(st["out"], st["q"], s["kp"], s["vp"], s["layout"], st["table"], s["width"], st["cu"], st["start"],
                               st["rows"], s["case"]["q"], s["scale"], s["ws"], s["wsb"])
    return dict(out=s["out"], k=s["kp"], v=s["vp"])


def work(case):
    e = 4 if case["dtype"] == "f32" else 2
    kv = case["kv"]
    if case["kind"] == "fork":
        return {"bytes": 4 * case["pairs"] * case["layers"] * kv * BS * D * e, "flops": 0}
    lens, q = _lengths(case), case["q"]
    row = (q + 2 * kv) * D * e + 2 * kv * D * e + q * D * e  # q, k, v in; k, v into the pool; the output
    if case["kind"] == "prefill":
        return {"bytes": sum(lens) * row, "flops": sum(4 * q * D * (n * (n + 1) // 2) for n in lens)}
    cached = sum(lens) - case["shared"] * (case["batch"] - 1)
    return {"bytes": case["layers"] * (cached * 2 * kv * D * e + case["batch"] * row),
            "flops": case["layers"] * sum(4 * q * D * (n + 1) for n in lens)}


def tolerance(case):
    """Fork: bytes.  Attention: see TOL; the sums are fp32 and the results rounded once."""
    return "exact" if case["kind"] == "fork" else TOL[case["dtype"]]


# Four times the 2-norm error seen between these outputs and the same path in 64 bits (f16 2.1e-4,
# bf16 1.7e-3: the rounding of the stored results; f32 2.0e-7).  The largest single differences seen
# are 4.9e-4, 3.9e-3 and 8.4e-7; "max" leaves room for a query or key element, rounded to the other
# side by another order of the norm's sum, in a short sequence.
TOL = {"f16": {"rel": 1e-3, "max": 4e-3}, "bf16": {"rel": 7e-3, "max": 3e-2}, "f32": {"rel": 1e-6, "max": 1e-5}}


def _exact_append(s, q, k, v, pos, kp, vp, slots):
    """The step's rows normalised, rotated and stored in 64 bits: q [n, heads, D]; kp and vp
    [slots, heads, D] take the new rows.  The sin / cos tables are inputs as they stand."""
    def rotated(x, heads, w):
        x = x.double().view(-1, heads, D)
        if s["case"]["norm"]:
            x = w.double() * x / torch.sqrt((x * x).mean(-1, keepdim=True) + EPS)
        at = pos.long()
        sin, cos = (t.view(-1, D)[at, ::2].double().unsqueeze(1) for t in (s["sin"], s["cos"]))
        lo, hi = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([lo * cos - hi * sin, lo * sin + hi * cos], -1)
    kp[slots] = rotated(k, s["case"]["kv"], s["norms"][1])
    vp[slots] = v.double().view(-1, s["case"]["kv"], D)
    return rotated(q, s["case"]["q"], s["norms"][0])


def _exact_attention(q, k, v, start, kv, dtype):
    """q [n, heads, D] at positions start.. over k and v [tokens, kv, D]; q and k enter rounded to
    the type that the path holds them in."""
    n, heads = q.shape[:2]
    q, k = (x.to(dtype).double() for x in (q, k))
    hidden = torch.arange(len(k), device="cuda") > start + torch.arange(n, device="cuda").unsqueeze(1)
    out = []
    for h, group in enumerate(q.transpose(0, 1).chunk(kv)):  # the query heads of KV head h
        scores = (group @ k[:, h].T / math.sqrt(D)).masked_fill_(hidden, -math.inf)
        out.append(torch.softmax(scores, -1) @ v[:, h])
    return torch.cat(out).transpose(0, 1).reshape(n, heads * D)


def exact(case, seed):
    """What run returns, in 64 bits; a fork's outputs are bytes."""
    if case["kind"] == "fork":
        return None
    s = prepare(dict(case, call="eager") if case["kind"] == "decode" else case, seed)
    s["qk"].copy_(s["fresh"])
    kv, dtype, out = case["kv"], DTYPES[case["dtype"]], torch.zeros_like(s["out"], dtype=torch.float64)
    paged = case.get("layout") != "contiguous"
    # pools as [layer, slot, head, D]
    kps, vps = (t.double().view(-1, t.shape[-4], kv, BS, D).transpose(2, 3).reshape(-1, t.shape[-4] * BS, kv, D) if paged
                else t.double().view(t.shape[0], -1, kv, D) for t in (s["kp"], s["vp"]))

    def keys(table_row, n):
        at = torch.arange(n, device="cuda")
        return at if table_row is None else table_row[at // BS].long() * BS + at % BS
    if case["kind"] == "decode":
        for i in range(case["layers"]):
            q = _exact_append(s, s["q"][i], s["k"][i], s["v"][i], s["pos"], kps[i], vps[i], s["slots"])
            for b, n in enumerate(s["pos"].tolist()):
                at = keys(s["table"][b] if paged else None, n + 1)
                out[i, b] = _exact_attention(q[b:b + 1], kps[i][at], vps[i][at], n, kv, dtype)[0]
    else:
        row = 0
        for st in s["steps"]:
            q = _exact_append(s, st["q"], st["k"], st["v"], st["pos"], kps[0], vps[0], st["slots"])
            for r, start in enumerate(st["start"].tolist()):
                a, b = st["cu"][r:r + 2].tolist()
                at = keys(st["table"][r], start + b - a)
                out[row + a:row + b] = _exact_attention(q[a:b], kps[0][at], vps[0][at], start, kv, dtype)
            row += st["n"]

    def stored(pools, like):
        if paged:
            pools = pools.view(len(pools), -1, BS, kv, D).transpose(2, 3)
        return pools.reshape(like.shape)
    return dict(out=out, k=stored(kps, s["kp"]), v=stored(vps, s["vp"]))
