"""Short prompts through the tensor-core prefill kernel, many times: up to 64 keys in a unit's last tile leave CTA 1
of a pair without keys to fetch, so that it runs beside the others without being waited for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
D, BS = 128, 16


@pytest.mark.parametrize("batch,tokens,start", [(64, 16, 0), (32, 16, 0), (48, 16, 128), (40, 7, 250)])
def test_thousands_of_calls(native_libs, batch, tokens, start):
    import torch
    from orinmllm_b200 import capi
    H, HKV = 32, 8
    gen = torch.Generator(device="cuda").manual_seed(batch)
    width = -(-(start + tokens) // BS)
    blocks = batch * width
    table = torch.randperm(blocks, generator=gen, device="cuda").to(torch.int32).view(batch, width)
    kp, vp = (torch.randn((blocks, HKV, BS, D), generator=gen, device="cuda", dtype=torch.float16) for _ in range(2))
    q = torch.randn((batch * tokens, H * D), generator=gen, device="cuda", dtype=torch.float16)
    lay = capi.layout_paged(capi.KPX_F16, HKV, D, BS, blocks)
    nbytes = capi.prefill_workspace_bytes(batch * tokens, H, HKV, D)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    cu = (np.arange(batch + 1) * tokens).astype(np.int32)
    starts = np.full(batch, start, np.int32)

    def calls(n):
        out = torch.full_like(q, float("nan"))
        for _ in range(n):
            capi.paged_prefill(out, q, kp, vp, lay, table, width, cu, starts, batch, H, 1 / np.sqrt(D), ws, nbytes)
        assert capi.workspace_status(ws) == 0
        return out

    first = calls(1)
    assert torch.isfinite(first).all()
    for _ in range(60):
        assert torch.equal(calls(500), first)
