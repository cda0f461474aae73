"""Launches that follow each other on a stream may become resident before their predecessor has
ended: each has to see everything that was before it, whoever wrote it."""
import math

import pytest

from tests import kvtest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("batch,ctx", [(1, 40), (3, 700), (48, 300)])
@pytest.mark.parametrize("captured", [False, True])
def test_a_chain_of_steps_sees_what_came_before(native_libs, dtype, batch, ctx, captured):
    """Twelve decode steps in a row whose inputs are made by torch kernels and copies between the
    launches, lengths, slots and plan included; equal, bit for bit, to the same with a wait after
    every launch."""
    import torch
    from orinmllm_b200 import capi
    h, kv, steps = 8, 2, 12
    dt = kvtest.torch_dtype(dtype)
    width = -(-(ctx + steps) // 16)
    blocks = batch * width
    lay = capi.layout_paged(capi.dtype_code(dt), kv, 128, 16, blocks)
    gen = torch.Generator(device="cuda").manual_seed(7)
    table = torch.randperm(blocks, generator=gen, device="cuda").to(torch.int32).view(batch, width)
    pools0 = [torch.randn(blocks, kv, 16, 128, generator=gen, device="cuda").to(dt) for _ in range(2)]
    rows = [[torch.randn(batch, n * 128, generator=gen, device="cuda").to(dt) for n in (h, kv, kv)] for _ in range(steps)]
    sin, cos = (torch.empty(width * 16 * 128, device="cuda") for _ in range(2))
    capi.sin_cos_cache(sin, cos, 128, width * 16, 1e6)
    nbytes = capi.decode_workspace_bytes(batch, h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    plan = torch.zeros(capi.decode_plan_bytes(), dtype=torch.uint8, device="cuda")
    at = torch.arange(batch, device="cuda")

    def run(wait):
        kp, vp = (p.clone() for p in pools0)
        pos = torch.full((batch,), ctx, dtype=torch.int32, device="cuda")
        outs = torch.zeros(steps, batch, h * 128, device="cuda", dtype=dt)
        q, k, v = (torch.empty_like(t) for t in rows[0])
        slots = torch.empty(batch, dtype=torch.int64, device="cuda")

        def chain():
            for i in range(steps):
                for dst, src in zip((q, k, v), rows[i]):
                    dst.copy_(src)
                if i:
                    q.add_(outs[i - 1])  # a step's input depends on the output before it
                slots.copy_(table[at, (pos // 16).long()].long() * 16 + pos % 16)
                wait()
                capi.decode_plan(plan, plan.numel(), lay, table, width, pos, 1, batch, h)
                wait()
                capi.rope_append(q, k, v, h, pos, sin, cos, kp, vp, lay, slots, batch)
                wait()
                capi.paged_decode_planned(outs[i], q, kp, vp, lay, table, width, pos, 1, batch, h, 1 / math.sqrt(128), ws,
                                          nbytes, plan)
                wait()
                pos.add_(1)
        return chain, outs, kp, vp, pos

    capi.workspace_init(ws, nbytes)
    chain, want, wkp, wvp, _ = run(torch.cuda.synchronize)
    chain()
    chain, outs, kp, vp, pos = run(lambda: None)
    if captured:
        chain()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            chain()
        for p, p0 in zip((kp, vp), pools0):
            p.copy_(p0)
        pos.fill_(ctx)
        outs.zero_()
        graph.replay()
    else:
        chain()
    torch.cuda.synchronize()
    assert capi.workspace_status(ws) == 0
    assert torch.equal(outs, want) and torch.equal(kp, wkp) and torch.equal(vp, wvp)


@pytest.mark.parametrize("dtype", ["f16", "f32"])
def test_inputs_written_by_the_launch_before(native_libs, dtype):
    """The norm weights of a rotation and the new rows of a fused step are written by the chained launch
    right in front of it (an append whose "pool" they are), other values every time: the results are
    those with a wait after every launch."""
    import torch
    from orinmllm_b200 import capi
    h, kv, batch, steps = 8, 2, 3, 40
    dt = kvtest.torch_dtype(dtype)
    gen = torch.Generator(device="cuda").manual_seed(11)
    lay = capi.layout_paged(capi.dtype_code(dt), kv, 128, 16, 64)
    rows = {t: capi.layout_contiguous(capi.dtype_code(t), 1, 128, 16, 0) for t in (dt, torch.float32)}
    table = torch.randperm(64, generator=gen, device="cuda")[:batch * 16].to(torch.int32).view(batch, 16)
    pos = torch.tensor([5, 100, 200], dtype=torch.int32, device="cuda")
    at = torch.arange(batch, device="cuda")
    slots = table[at, (pos // 16).long()].long() * 16 + pos % 16
    sin, cos = (torch.empty(256 * 128, device="cuda") for _ in range(2))
    capi.sin_cos_cache(sin, cos, 128, 256, 1e6)
    weights = torch.rand(steps, 2, 128, generator=gen, device="cuda") + 0.5
    fresh = torch.randn(steps, batch * (h + 2 * kv), 128, generator=gen, device="cuda").to(dt)
    pools0 = [torch.randn(64, kv, 16, 128, generator=gen, device="cuda").to(dt) for _ in range(2)]
    nbytes = capi.decode_workspace_bytes(batch, h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)

    def run(wait):
        kp, vp = (p.clone() for p in pools0)
        outs = torch.zeros(steps, batch, h * 128, device="cuda", dtype=dt)
        w = torch.zeros(2, 128, device="cuda")
        x = torch.zeros(batch * (h + 2 * kv), 128, device="cuda", dtype=dt)
        q, k, v = x[:batch * h], x[batch * h:batch * (h + kv)], x[batch * (h + kv):]
        torch.cuda.synchronize()
        for i in range(steps):
            capi.append(x, None, rows[dt], fresh[i], None, num_tokens=len(x))
            wait()
            if i % 2:
                capi.rope_append_decode(outs[i], q, k, v, sin, cos, kp, vp, lay, table, 16, pos, batch, h, 1 / math.sqrt(128),
                                        ws, nbytes)
            else:
                capi.append(w, None, rows[torch.float32], weights[i], None, num_tokens=2)
                wait()
                capi.norm_rope_append(q, k, v, h, w[0], w[1], 1e-6, pos, sin, cos, kp, vp, lay, slots, batch)
                wait()
                capi.append(outs[i].view(-1, 128), None, rows[dt], q, None, num_tokens=len(q))
            wait()
        torch.cuda.synchronize()
        return outs, kp, vp

    want = run(torch.cuda.synchronize)
    for got, ref in zip(run(lambda: None), want):
        assert torch.equal(got, ref)
    assert capi.workspace_status(ws) == 0
