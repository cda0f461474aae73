"""Bounded waits of the tensor-core prefill kernel when the second CTA of a pair lacks a tile: its bytes are counted on
barriers of the first, except those of a last tile of V, which it waits for itself."""
import numpy as np
import pytest

from tests import kvtest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cta", [0, 1])
@pytest.mark.parametrize("tile,tokens,start", [(0, 300, 212), (1, 300, 212), (2, 300, 212), (1, 100, 0)],
                         ids=["first_k_tile", "first_v_tile", "second_k_tile", "last_v_tile"])
def test_the_call_returns_and_the_next_one_is_right(native_libs, cta, tile, tokens, start):
    import torch
    from orinmllm_b200 import capi
    H, HKV, D, BS = 8, 2, 128, 16
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    blocks = -(-(start + tokens) // BS)
    kp, vp = (torch.randn((blocks, HKV, BS, D), generator=gen, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn((tokens, H * D), generator=gen, device="cuda", dtype=torch.bfloat16)
    table = torch.randperm(blocks, generator=gen, device="cuda").to(torch.int32).view(1, blocks)
    lay = capi.layout_paged(capi.KPX_BF16, HKV, D, BS, blocks)
    nbytes = capi.prefill_workspace_bytes(tokens, H, HKV, D)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)

    def call():
        out = torch.full_like(q, float("nan"))
        capi.paged_prefill(out, q, kp, vp, lay, table, blocks, np.array([0, tokens], np.int32), np.array([start], np.int32), 1,
                           H, 1 / np.sqrt(D), ws, nbytes)
        torch.cuda.synchronize()  # the kernel has returned
        return out

    lib = capi.lib()
    lib.kpx_internal_set_prefill_split(0)  # whole units: the first CTAs have a second tile
    try:
        good = call()
        assert capi.workspace_status(ws) == 0 and torch.isfinite(good).all()
        lib.kpx_internal_set_prefill_fault(3000, cta | tile << 16)
        try:
            broken = call()
        finally:
            lib.kpx_internal_set_prefill_fault(0, -1)
        assert capi.workspace_status(ws) == capi.KPX_ERR_DEVICE_TIMEOUT
        assert torch.isnan(broken).any()
        again = call()
    finally:
        lib.kpx_internal_set_prefill_split(-1)
    assert capi.workspace_status(ws) == 0
    assert torch.equal(again, good)
    ref = kvtest.storage_to_f32(kvtest.from_device(good, "bf16"), "bf16")
    k, v = (x[table[0].long()].transpose(1, 2).reshape(-1, HKV, D)[:start + tokens].double() for x in (kp, vp))
    k, v = (x.repeat_interleave(H // HKV, 1) for x in (k, v))
    hidden = torch.arange(start + tokens, device="cuda") > start + torch.arange(tokens, device="cuda")[:, None]
    scores = torch.einsum("nhd,thd->hnt", q.double().view(tokens, H, D), k) / np.sqrt(D)
    want = torch.einsum("hnt,thd->nhd", torch.softmax(scores.masked_fill(hidden, -np.inf), -1), v).reshape(tokens, -1)
    kvtest.assert_attention_close(ref, want.cpu().numpy().astype(np.float32), "prefill after a timed-out call", "bf16")
