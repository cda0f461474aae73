"""RoPE of many tokens (a CTA per one or two of them) with arguments left out: the bits are those of the same call in
small chunks, which take the flat form."""
import pytest

pytestmark = pytest.mark.gpu
H, HKV, D, BS = 12, 2, 128, 16


@pytest.mark.parametrize("tokens", [400, 1401])
@pytest.mark.parametrize("what", ["k_weight_only", "q_weight_only", "no_q", "no_k", "no_v", "no_slots", "no_positions"])
@pytest.mark.parametrize("norm", [True, False], ids=["norm", "plain"])
def test_same_bits_with_arguments_left_out(native_libs, tokens, what, norm):
    import torch
    from orinmllm_b200 import capi
    if not norm and what.endswith("only"):
        pytest.skip("no weights")
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    blocks = tokens // BS + 2
    lay = capi.layout_paged(capi.KPX_F16, HKV, D, BS, blocks)
    base = 37 if what == "no_positions" else 5
    sin, cos = (torch.empty((tokens + base + 700) * D, device="cuda") for _ in range(2))
    capi.sin_cos_cache(sin, cos, D, tokens + base + 700, 1e6)
    qw, kw = 1 + 0.2 * torch.randn(2, D, generator=gen, device="cuda")
    if what == "k_weight_only":
        qw = None
    if what == "q_weight_only":
        kw = None
    rows = [torch.randn(tokens, n * D, generator=gen, device="cuda").half() for n in (H, HKV, HKV)]
    pos = torch.randint(0, 700, (tokens,), generator=gen, device="cuda", dtype=torch.int32)
    slots = torch.randperm(blocks * BS, generator=gen, device="cuda")[:tokens]
    slots[::7] = -1  # rotated, not stored

    def run(chunk):
        q, k, v = (x.clone() for x in rows)
        kp = torch.zeros(blocks, HKV, BS, D, device="cuda", dtype=torch.float16)
        vp = torch.zeros_like(kp)
        for a in range(0, tokens, chunk):
            b = min(tokens, a + chunk)
            has_k, has_v = what not in ("no_k",), what not in ("no_v", "no_k", "no_slots")
            stores = what not in ("no_k", "no_slots")
            args = (None if what == "no_q" else q[a:b], k[a:b] if has_k else None, v[a:b] if has_v else None, H)
            where = (None if what == "no_positions" else pos[a:b], sin, cos, kp if stores else None, vp if has_v else None,
                     lay, slots[a:b] if stores else None, b - a)
            shift = base + a if what == "no_positions" else base
            if norm:
                capi.norm_rope_append(*args, qw, kw, 1e-6, *where, pos_base=shift)
            else:
                capi.rope_append(*args, *where, pos_base=shift)
        torch.cuda.synchronize()
        return q, k, kp, vp
    want, got = run(64), run(tokens)
    for x, y, z in zip(want, got, rows + [None]):
        assert torch.equal(x, y)
    assert torch.equal(got[0], rows[0]) == (what == "no_q") and torch.equal(got[1], rows[1]) == (what == "no_k")
