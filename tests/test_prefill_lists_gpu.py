"""Work lists of tensor-core prefill calls: the longest that travel as a kernel parameter of either size, the
shortest that do not, and a captured call, whose list is gone on the host when the graph is replayed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
D, BS, H = 128, 16, 8  # 8/8 heads: up to 256 tokens of a sequence are eight units


def _prompts(torch, capi, batch, tokens, start):
    gen = torch.Generator(device="cuda").manual_seed(batch)
    width = -(-(start + tokens) // BS)
    blocks = batch * width
    table = torch.randperm(blocks, generator=gen, device="cuda").to(torch.int32).view(batch, width)
    kp, vp = (torch.randn((blocks, H, BS, D), generator=gen, device="cuda", dtype=torch.bfloat16) for _ in range(2))
    q = torch.randn((batch, tokens, H * D), generator=gen, device="cuda", dtype=torch.bfloat16)
    lay = capi.layout_paged(capi.KPX_BF16, H, D, BS, blocks)
    nbytes = capi.prefill_workspace_bytes(batch * tokens, H, H, D)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)

    def call(out, first, last):
        n = last - first
        capi.paged_prefill(out[first:last], q[first:last], kp, vp, lay, table[first:last], width,
                           (np.arange(n + 1) * tokens).astype(np.int32), np.full(n, start, np.int32), n, H,
                           1 / np.sqrt(D), ws, nbytes)
    return q, ws, call


@pytest.mark.parametrize("batch", [44, 45, 120, 121, 130])  # 352, 360, 960, 968 and 1040 units: the last two in one and in two parts
def test_lists_of_every_length(native_libs, batch):
    import torch
    from orinmllm_b200 import capi
    q, ws, call = _prompts(torch, capi, batch, 70, 100)
    together, alone = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    lib = capi.lib()
    lib.kpx_internal_set_prefill_split(0)  # whole units: the same bits however they are dealt
    try:
        call(together, 0, batch)
        for i in range(batch):
            call(alone, i, i + 1)
    finally:
        lib.kpx_internal_set_prefill_split(-1)
    assert capi.workspace_status(ws) == 0
    assert torch.isfinite(together).all() and torch.equal(together, alone)


@pytest.mark.parametrize("batch", [20, 100, 140])  # lists in parameters of both sizes, and in the work area
def test_a_captured_call_carries_its_list(native_libs, batch):
    import torch
    from orinmllm_b200 import capi
    q, ws, call = _prompts(torch, capi, batch, 70, 100)
    want, out = torch.full_like(q, float("nan")), torch.full_like(q, float("nan"))
    call(want, 0, batch)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        call(out, 0, batch)
    other = torch.empty_like(q)
    call(other, 0, max(1, batch // 2))  # host memory is used again
    for _ in range(3):
        out.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert torch.equal(out, want)
    assert capi.workspace_status(ws) == 0
    del graph
