"""Decode attention of 16-bit caches where the matrix-instruction kernel can go wrong: edges of its
16-token tiles, every number of query heads per KV head around its eight rows, strided caches whose
memory ends inside a block, and a workspace that launches of other types share.  Reference: the same
attention in fp64."""
import math

import numpy as np
import pytest

from tests import kvtest

pytestmark = pytest.mark.gpu
LENS = [1, 2, 15, 16, 17, 31, 32, 33, 47, 48, 49, 129, 255, 777]


def _reference(q, k, v):
    """q [heads, 128]; k, v [tokens, kv_heads, 128]"""
    import torch
    mul = q.shape[0] // k.shape[1]
    kk, vv = (x.double().repeat_interleave(mul, 1) for x in (k, v))
    p = torch.softmax(torch.einsum("hd,thd->ht", q.double(), kk) / math.sqrt(128), -1)
    return torch.einsum("ht,thd->hd", p, vv)


def _check(out, ref, dtype, what):
    kvtest.assert_attention_close(out.float().cpu().numpy(), ref.float().cpu().numpy(), what, dtype)


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("heads", [(1, 1), (6, 3), (6, 2), (5, 1), (8, 1), (9, 1), (32, 2), (34, 2)])
@pytest.mark.parametrize("planned", [False, True])
def test_tiles_and_heads_per_kv_head(native_libs, dtype, heads, planned):
    import torch
    from orinmllm_b200 import capi
    h, kv = heads
    dt = kvtest.torch_dtype(dtype)
    gen = torch.Generator(device="cuda").manual_seed(3)
    lens = LENS * 40 if planned else LENS  # (a plan is for launches of many blocks)
    width = -(-max(lens) // 16)
    blocks = len(lens) * width
    table = torch.randperm(blocks, generator=gen, device="cuda").to(torch.int32).view(len(lens), width)
    kp, vp = (torch.randn(blocks, kv, 16, 128, generator=gen, device="cuda").to(dt) for _ in range(2))
    for b, n in enumerate(lens):  # what lies past a sequence's end must not matter
        if n % 16:
            kp[table[b, n // 16], :, n % 16:] = float("nan")
            vp[table[b, n // 16], :, n % 16:] = float("nan")
    q = torch.randn(len(lens), h * 128, generator=gen, device="cuda").to(dt)
    out = torch.full_like(q, float("nan"))
    lay = capi.layout_paged(capi.dtype_code(dt), kv, 128, 16, blocks)
    nbytes = capi.decode_workspace_bytes(len(lens), h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    lens_dev = torch.tensor(lens, dtype=torch.int32, device="cuda")
    plan = None
    if planned:
        plan = torch.zeros(capi.decode_plan_bytes(), dtype=torch.uint8, device="cuda")
        capi.decode_plan(plan, plan.numel(), lay, table, width, lens_dev, 0, min(len(lens), 512), h)
    for _ in range(2):
        n = min(len(lens), 512)
        capi.paged_decode_planned(out, q, kp, vp, lay, table, width, lens_dev, 0, n, h, 1 / math.sqrt(128), ws, nbytes, plan)
        assert capi.workspace_status(ws) == 0
        for b in range(n) if not planned else range(0, n, 37):
            at = torch.arange(lens[b], device="cuda")
            ids = table[b, at // 16].long()
            ref = _reference(q[b].view(h, 128), kp[ids, :, at % 16], vp[ids, :, at % 16])
            _check(out[b].view(h, 128), ref, dtype, f"{dtype} {heads} len {lens[b]}")


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("length", [1, 15, 16, 17, 130, 511, 2049])
def test_strided_cache_that_ends_inside_a_block(native_libs, dtype, length):
    import torch
    from orinmllm_b200 import capi
    h, kv = 28, 4
    dt = kvtest.torch_dtype(dtype)
    gen = torch.Generator(device="cuda").manual_seed(length)
    k, v = (torch.randn(length, kv * 128, generator=gen, device="cuda").to(dt) for _ in range(2))
    q = torch.randn(1, h * 128, generator=gen, device="cuda").to(dt)
    out = torch.full_like(q, float("nan"))
    lay = capi.layout_contiguous(capi.dtype_code(dt), kv, 128, 16, 0)
    nbytes = capi.decode_workspace_bytes(1, h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    for fixed in (False, True):
        lens = None if fixed else torch.tensor([length], dtype=torch.int32, device="cuda")
        capi.paged_decode(out, q, k, v, lay, None, 0, lens, length if fixed else 0, 1, h, 1 / math.sqrt(128), ws, nbytes)
        assert capi.workspace_status(ws) == 0
        ref = _reference(q.view(h, 128), k.view(length, kv, 128), v.view(length, kv, 128))
        _check(out.view(h, 128), ref, dtype, f"strided {dtype} {length}")


def test_small_weights_keep_their_precision(native_libs):
    """One key holds the row's maximum and thousands of others 2^-18 of its weight each, whose sum
    carries a tenth of the output: their weights may not be lost to the 16-bit terms."""
    import torch
    from orinmllm_b200 import capi
    n = 32768
    for dtype, bound in (("f16", 2.0 ** -10), ("bf16", 2.0 ** -7)):  # the output's own rounding, twice
        dt = kvtest.torch_dtype(dtype)
        q = torch.zeros(1, 128, device="cuda", dtype=dt)
        q[0, 0] = 1
        k = torch.zeros(n, 128, device="cuda", dtype=dt)
        k[0, 0] = 18 * math.log(2) * math.sqrt(128)
        v = torch.zeros(n, 128, device="cuda", dtype=dt)
        v[1:] = 1
        lay = capi.layout_contiguous(capi.dtype_code(dt), 1, 128, 16, n // 16)
        nbytes = capi.decode_workspace_bytes(1, 1, 1)
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        capi.workspace_init(ws, nbytes)
        out = torch.full_like(q, float("nan"))
        capi.paged_decode(out, q, k, v, lay, None, 0, None, n, 1, 1, 1 / math.sqrt(128), ws, nbytes)
        ref = _reference(q.view(1, 128), k.view(n, 1, 128), v.view(n, 1, 128))
        err = ((out.double() - ref) / ref).abs().max().item()
        assert err <= bound, f"{dtype}: {err:.2e} > {bound:.2e}"


@pytest.mark.parametrize("heads", [(4, 4), (4, 2), (6, 2), (8, 2), (7, 1), (8, 1)])
def test_types_share_one_workspace(native_libs, heads):
    """Long sequences (two levels of assembly) in f16, f32 and bf16 in turn on one workspace, in the line
    of blocks: every launch leaves its pieces in the workspace's slots."""
    import torch
    from orinmllm_b200 import capi
    h, kv = heads
    gen = torch.Generator(device="cuda").manual_seed(5)
    n = 30000
    nbytes = capi.decode_workspace_bytes(1, h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    k, v = (torch.randn(n, kv * 128, generator=gen, device="cuda") for _ in range(2))
    q = torch.randn(1, h * 128, generator=gen, device="cuda")
    lib = capi.lib()
    lib.kpx_internal_set_decode_cluster(0)
    try:
        for dtype in ("f16", "f32", "bf16", "f32", "f16"):
            dt = kvtest.torch_dtype(dtype)
            kd, vd, qd = (x.to(dt) for x in (k, v, q))
            out = torch.full_like(qd, float("nan"))
            before = ws.clone()
            lay = capi.layout_contiguous(capi.dtype_code(dt), kv, 128, 16, n // 16)
            capi.paged_decode(out, qd, kd, vd, lay, None, 0, None, n, 1, h, 1 / math.sqrt(128), ws, nbytes)
            assert capi.workspace_status(ws) == 0
            # (a piece of one head is half a KB; several hundred warps left one)
            assert (ws != before).sum().item() > 100 * 512, "the launch did not use the workspace"
            ref = _reference(qd.view(h, 128), kd.view(n, kv, 128), vd.view(n, kv, 128))
            _check(out.view(h, 128), ref, dtype, f"shared workspace {dtype}")
    finally:
        lib.kpx_internal_set_decode_cluster(24)
