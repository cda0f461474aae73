"""Small decode launches, one cluster of CTAs per item: every cluster size and CTA width that the
dispatch can choose, shares of no, one and many blocks per warp, with and without the new token, and
the line of 1 block to the limit where the other form takes over.  Reference: fp64 attention; the
fused step's pool rows are compared bit for bit with the two-launch path's."""
import math

import pytest

from tests import kvtest

pytestmark = pytest.mark.gpu


def _attend(q, k, v):
    import torch
    mul = q.shape[0] // k.shape[1]
    kk, vv = (x.double().repeat_interleave(mul, 1) for x in (k, v))
    p = torch.softmax(torch.einsum("hd,thd->ht", q.double(), kk) / math.sqrt(128), -1)
    return torch.einsum("ht,thd->hd", p, vv)


@pytest.mark.parametrize("dtype", ["f16", "bf16", "f32"])
@pytest.mark.parametrize("heads,batch,longest", [
    ((8, 1), 1, 1), ((8, 1), 1, 129), ((6, 2), 1, 2100), ((12, 2), 1, 9001), ((32, 8), 1, 3000), ((28, 4), 2, 1025),
    ((16, 8), 3, 640), ((9, 1), 20, 500), ((32, 8), 18, 333), ((32, 8), 21, 190), ((32, 8), 60, 70), ((64, 8), 75, 40),
    ((4, 4), 130, 33)])
@pytest.mark.parametrize("fused", [False, True])
def test_forms_of_a_small_launch(native_libs, dtype, heads, batch, longest, fused):
    import torch
    from orinmllm_b200 import capi
    h, kv = heads
    dt = kvtest.torch_dtype(dtype)
    gen = torch.Generator(device="cuda").manual_seed(batch)
    lens = [longest if i == 0 else int(torch.randint(0, longest + 1, (1,), generator=gen, device="cuda")) for i in range(batch)]
    width = longest // 16 + 1
    blocks = batch * width
    table = torch.randperm(blocks, generator=gen, device="cuda").to(torch.int32).view(batch, width)
    kp, vp = (torch.randn(blocks, kv, 16, 128, generator=gen, device="cuda").to(dt) for _ in range(2))
    pos = torch.tensor(lens, dtype=torch.int32, device="cuda")
    at = torch.arange(batch, device="cuda")
    ends = table[at, (pos // 16).long()].long()
    for b, n in enumerate(lens):  # what lies past a sequence's end must not matter
        kp[ends[b], :, n % 16:] = float("nan")
        vp[ends[b], :, n % 16:] = float("nan")
    q, k, v = (torch.randn(batch, n * 128, generator=gen, device="cuda").to(dt) for n in (h, kv, kv))
    lay = capi.layout_paged(capi.dtype_code(dt), kv, 128, 16, blocks)
    nbytes = capi.decode_workspace_bytes(batch, h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    out = torch.full_like(q, float("nan"))
    if fused:
        sin, cos = (torch.empty((longest + 1) * 128, device="cuda") for _ in range(2))
        capi.sin_cos_cache(sin, cos, 128, longest + 1, 1e6)
        want_k, want_v, q2, k2 = kp.clone(), vp.clone(), q.clone(), k.clone()
        capi.rope_append(q2, k2, v, h, pos, sin, cos, want_k, want_v, lay, ends * 16 + pos % 16, batch)
        capi.rope_append_decode(out, q, k, v, sin, cos, kp, vp, lay, table, width, pos, batch, h, 1 / math.sqrt(128), ws, nbytes)
        bits = torch.int32 if dtype == "f32" else torch.int16
        assert torch.equal(kp.view(bits), want_k.view(bits)) and torch.equal(vp.view(bits), want_v.view(bits))
        q = q2
    else:
        capi.paged_decode(out, q, kp, vp, lay, table, width, pos, 0, batch, h, 1 / math.sqrt(128), ws, nbytes)
    assert capi.workspace_status(ws) == 0
    for b in range(0, batch, 1 if batch < 25 else 7):
        n = lens[b] + fused
        got = out[b].view(h, 128)
        if n == 0:
            assert torch.equal(got, torch.zeros_like(got))
            continue
        t = torch.arange(n, device="cuda")
        ids = table[b, t // 16].long()
        ref = _attend(q[b].view(h, 128), kp[ids, :, t % 16], vp[ids, :, t % 16])
        kvtest.assert_attention_close(got.float().cpu().numpy(), ref.float().cpu().numpy(),
                                      f"{dtype} {heads} batch {batch} length {lens[b]}", dtype)
