"""RoPE: tables and weights on and off 16-byte boundaries take different forms of the kernel, and so do calls of
few and of many tokens (one or two tokens a CTA, an odd number of them); the bits are the same."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float16", "bfloat16", "float32"])
@pytest.mark.parametrize("tokens", [1, 65, 400, 1399, 1401, 5000])
@pytest.mark.parametrize("norm", [True, False], ids=["norm", "plain"])
def test_same_bits(native_libs, dtype, tokens, norm):
    import torch
    from orinmllm_b200 import capi
    H, HKV, D, BS = 12, 2, 128, 16
    dt = getattr(torch, dtype)
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    blocks = tokens // BS + 2
    lay = capi.layout_paged(capi.dtype_code(dt), HKV, D, BS, blocks)
    max_pos = 700
    tables = torch.empty(2, max_pos * D, device="cuda")
    capi.sin_cos_cache(tables[0], tables[1], D, max_pos, 1e6)
    weights = 1 + 0.2 * torch.randn(2, D, generator=gen, device="cuda")
    rows = [torch.randn(tokens, n * D, generator=gen, device="cuda").to(dt) for n in (H, HKV, HKV)]
    pos = torch.randint(0, max_pos, (tokens,), generator=gen, device="cuda", dtype=torch.int32)
    slots = torch.randperm(blocks * BS, generator=gen, device="cuda")[:tokens]
    slots[::7] = -1  # rotated, not stored

    def moved(x, by):  # the same values, `by` floats behind an aligned address
        room = torch.empty(x.numel() + 4, device="cuda")
        room[by:by + x.numel()] = x
        return room[by:by + x.numel()]

    def run(by, chunk):
        q, k, v = (x.clone() for x in rows)
        kp = torch.zeros(blocks, HKV, BS, D, device="cuda", dtype=dt)
        vp = torch.zeros_like(kp)
        sin, cos, qw, kw = (moved(x, by) for x in (tables[0], tables[1], weights[0], weights[1]))
        for a in range(0, tokens, chunk):
            b = min(tokens, a + chunk)
            what = q[a:b], k[a:b], v[a:b], H
            where = pos[a:b], sin, cos, kp, vp, lay, slots[a:b], b - a
            if norm:
                capi.norm_rope_append(*what, qw, kw, 1e-6, *where)
            else:
                capi.rope_append(*what, *where)
        torch.cuda.synchronize()
        return q, k, kp, vp
    want = run(1, 64)
    for by, chunk in ((0, tokens), (1, tokens), (0, 64)):
        for x, y in zip(want, run(by, chunk)):
            assert torch.equal(x, y)
