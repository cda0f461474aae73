"""Decode attention of 16-bit caches at the ends of what fp32 arithmetic can hold, in every form of the
launch: infinities and NaN in V, the last bits of the weights, the rounding of long sums, products
beyond 2^128.  Reference: the same attention in fp64."""
import math

import pytest

from tests import kvtest

pytestmark = pytest.mark.gpu

# form: (cluster knob, entry, tokens, heads): one cluster per item; the line of blocks; its small
# CTAs; items cut into so many pieces that they are assembled in two levels
FORMS = {"cluster": (24, "paged_decode", 300, (8, 2)), "cluster_of_many": (24, "paged_decode", 4000, (7, 1)),
         "line": (0, "paged_decode", 300, (8, 2)), "overlapped": (0, "paged_decode_overlapped", 3000, (32, 8)),
         "two_levels": (0, "paged_decode", 40000, (4, 1)), "fused": (24, None, 300, (8, 2)),
         "fused_line": (0, None, 3000, (28, 4))}


def decode(form, q, k, v, scale):
    """q [heads, 128] over k and v [tokens, kv heads, 128], a strided cache; in the fused forms the
    last token is the new one, at position 0 of the rotation (sin 0, cos 1)."""
    import torch
    from orinmllm_b200 import capi
    knob, entry, _, _ = FORMS[form]
    n, kv = k.shape[:2]
    h = q.shape[0]
    lay = capi.layout_contiguous(capi.dtype_code(k.dtype), kv, 128, 16, -(-n // 16))
    nbytes = capi.decode_workspace_bytes(1, h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    out = torch.full_like(q, float("nan"))
    lib = capi.lib()
    try:
        lib.kpx_internal_set_decode_cluster(knob)
        if knob == 0:
            lib.kpx_internal_set_decode_small(0 if entry == "paged_decode_overlapped" else 12, 12, 4)
        if entry:
            getattr(capi, entry)(out, q, k, v, lay, None, 0, torch.tensor([n], dtype=torch.int32, device="cuda"), 0, 1, h,
                                 scale, ws, nbytes)
        else:
            sin = torch.zeros(n * 128, device="cuda")
            kp, vp = (torch.cat([x[:-1], torch.full_like(x[:1], float("nan"))]) for x in (k, v))
            pos = torch.tensor([n - 1], dtype=torch.int32, device="cuda")
            capi.rope_append_decode(out, q, k[-1].contiguous(), v[-1].contiguous(), sin, torch.ones_like(sin), kp, vp, lay, None,
                                    0, pos, 1, h, scale, ws, nbytes)
        torch.cuda.synchronize()
    finally:
        lib.kpx_internal_set_decode_cluster(24)
        lib.kpx_internal_set_decode_small(12, 12, 4)
    assert capi.workspace_status(ws) == 0
    return out


def reference(q, k, v, scale):
    import torch
    mul = q.shape[0] // k.shape[1]
    kk, vv = (x.double().repeat_interleave(mul, 1) for x in (k, v))
    p = torch.softmax(torch.einsum("hd,thd->ht", q.double(), kk) * scale, -1)
    out = (p.T.unsqueeze(-1) * vv).sum(0)
    return out


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("form", FORMS)
def test_infinities_in_v(native_libs, dtype, form):
    """An infinite element of V makes the output infinite wherever its weight is not 0 (the largest
    weights, whose second 16-bit term is 0, and weights below 2^-50, whose first fp16 term would
    be), infinities of both signs make it NaN, and the other elements are as ever."""
    import torch
    dt = kvtest.torch_dtype(dtype)
    n, (h, kv) = FORMS[form][2:]
    gen = torch.Generator(device="cuda").manual_seed(n)
    q = torch.zeros(h, 128, device="cuda", dtype=dt)
    q[:, 0] = 1
    k = torch.zeros(n, kv, 128, device="cuda", dtype=dt)
    k[:, :, 0] = -3 * torch.rand(n, kv, generator=gen, device="cuda").to(dt)  # scores -0.27 .. 0
    at = [0, n // 3, n // 2, n - 2, n - 1]
    k[at[0], :, 0] = 0                                    # among the largest weights
    k[at[2], :, 0] = -60 * math.log(2) * math.sqrt(128)   # 2^-60 of the largest
    v = torch.randn(n, kv, 128, generator=gen, device="cuda").to(dt)
    inf = float("inf")
    for i, t in enumerate(at):
        v[t, :, 10 + i] = inf
        v[t, :, 20 + i] = -inf
    v[at[1], :, 30], v[at[3], :, 30] = inf, -inf
    v[at[2], :, 31], v[at[4], :, 31] = inf, -inf
    v[at[1], :, 32] = float("nan")
    got, ref = decode(form, q, k, v, 1 / math.sqrt(128)).double(), reference(q, k, v, 1 / math.sqrt(128))
    assert ref.isinf().sum() == 10 * h and ref.isnan().sum() == 3 * h
    assert torch.equal(got.isnan(), ref.isnan())
    assert torch.equal(torch.where(ref.isinf(), got, 0.), torch.where(ref.isinf(), ref, 0.))
    finite = ref.isfinite()
    kvtest.assert_attention_close(got[finite].float().cpu().numpy(), ref[finite].float().cpu().numpy(), f"{dtype} {form}", dtype)


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("form", FORMS)
def test_weights_keep_their_bits(native_libs, dtype, form):
    """Three tokens of weights 1, 1 and w, and V such that the output is what is left of w beyond the
    two 16-bit terms nearest to it: 2^-17 of w for bf16.  Bound: ex2.approx errs by 2^-22, the score
    and three roundings of the sums by 2^-24 each, against a sum of weights of at least 2."""
    import torch
    dt = kvtest.torch_dtype(dtype)
    n, (h, kv) = FORMS[form][2:]
    mul = h // kv
    gen = torch.Generator(device="cuda").manual_seed(n)
    q = torch.zeros(h, 128, device="cuda", dtype=dt)
    q[:, 0] = (0.2 + 5 * torch.rand(h, generator=gen, device="cuda")).to(dt)
    q[:, 1] = 1
    k = torch.zeros(n, kv, 128, device="cuda", dtype=dt)
    k[:, :, 1] = -4000  # weight 0
    at = [n // 32 * 16 + i for i in range(3)]  # (of one block: what is cut apart is added up in fp32)
    k[at, :, 1] = 0
    k[at[2], :, 0] = -1
    scale = 0.125
    w = torch.exp(-q[:, 0].double() * scale)
    first = w.to(dt)
    second = (w - first.double()).to(dt)
    v = torch.randn(n, kv, 128, generator=gen, device="cuda").to(dt)
    heads = torch.arange(h, device="cuda")
    j, d = heads // mul, heads % mul  # head d of KV head j looks at dimension d
    v[at[0], j, d], v[at[1], j, d], v[at[2], j, d] = -first, -second, 1
    got, ref = decode(form, q, k, v, scale).double(), reference(q, k, v, scale)
    err = (got - ref)[heads, d].abs().max().item()
    assert err <= (2.0 ** -22 + 4 * 2.0 ** -24) / 2, f"{dtype} {form}: {err:.2e}"


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("entry", ["paged_decode", "paged_decode_overlapped"])
def test_long_sums_are_rounded_not_cut_off(native_libs, dtype, entry):
    """V of two neighbouring values in about equal shares: outputs near the middle between the two show
    to which side their sums err.  Two hundred tiles a warp, each cut off by half of 2^-24 on
    average, would take 6e-6 off; sums rounded to nearest err by sqrt(200) * 2^-25 or so."""
    import torch
    from orinmllm_b200 import capi
    dt = kvtest.torch_dtype(dtype)
    h, kv, n, batch = 32, 8, 32768, 16
    gen = torch.Generator(device="cuda").manual_seed(3)
    step = 2.0 ** (-10 if dtype == "f16" else -7)
    kp = torch.randn(n // 16, kv, 16, 128, generator=gen, device="cuda").to(dt)
    vp = (1 + step * (torch.rand(n // 16, kv, 16, 128, generator=gen, device="cuda") < 0.5)).to(dt)
    table = torch.arange(n // 16, dtype=torch.int32, device="cuda").expand(batch, -1).contiguous()  # all share their blocks
    q = (torch.randn(batch, h * 128, generator=gen, device="cuda") * 0.2).to(dt)
    out = torch.empty_like(q)
    lay = capi.layout_paged(capi.dtype_code(dt), kv, 128, 16, n // 16)
    nbytes = capi.decode_workspace_bytes(batch, h, kv)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    lens = torch.full((batch,), n, dtype=torch.int32, device="cuda")
    getattr(capi, entry)(out, q, kp, vp, lay, table, n // 16, lens, 0, batch, h, 1 / math.sqrt(128), ws, nbytes)
    k, v = (x.transpose(1, 2).reshape(n, kv, 128) for x in (kp, vp))
    told = 0
    for b in (0, 7, 15):
        ref = torch.cat([torch.softmax(q[b].view(kv, 4, 128)[j].double() @ k[:, j].double().T / math.sqrt(128), -1) @ v[:, j].double()
                         for j in range(kv)])
        from_middle = ref - (1 + step / 2)
        clear = from_middle.abs() > 2e-6
        got = out[b].view(h, 128).double()
        want = torch.where(from_middle > 0, 1 + step, 1.0)
        wrong = clear & (got != want)
        told += (clear & (from_middle.abs() < 5e-6)).sum().item()
        assert not wrong.any(), f"{dtype} {entry}: {wrong.sum().item()} of {clear.sum().item()} fell to the wrong side"
    assert told > 100  # outputs close enough to the middle to tell


@pytest.mark.parametrize("dtype", ["f16", "bf16"])
@pytest.mark.parametrize("form", FORMS)
def test_products_beyond_fp32_before_the_scale(native_libs, dtype, form):
    """bf16 rows may be so large that q . k passes 2^128 while the scaled score does not."""
    import torch
    dt = kvtest.torch_dtype(dtype)
    n, (h, kv) = FORMS[form][2:]
    gen = torch.Generator(device="cuda").manual_seed(n)
    big = 2.0 ** 63 if dtype == "bf16" else 2.0 ** 15
    q = torch.zeros(h, 128, device="cuda", dtype=dt)
    q[:, :8] = big
    k = torch.zeros(n, kv, 128, device="cuda", dtype=dt)
    k[:, :, :8] = (big * (0.5 + 0.5 * torch.rand(n, kv, 8, generator=gen, device="cuda"))).to(dt)
    v = torch.randn(n, kv, 128, generator=gen, device="cuda").to(dt)
    scale = 2.0 ** -126 if dtype == "bf16" else 2.0 ** -30
    got, ref = decode(form, q, k, v, scale), reference(q, k, v, scale)
    kvtest.assert_attention_close(got.float().cpu().numpy(), ref.float().cpu().numpy(), f"{dtype} {form}", dtype)
