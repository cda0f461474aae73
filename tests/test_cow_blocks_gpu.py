"""Copy-on-write of blocks: every layout, sizes around a CTA's share, pairs that are skipped."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("contiguous", [False, True])
@pytest.mark.parametrize("dtype,kv,hs,bs", [("float16", 8, 128, 16), ("float32", 1, 64, 3), ("bfloat16", 3, 128, 16),
                                            ("float16", 1, 8, 1), ("float32", 5, 192, 16), ("float16", 2, 128, 32)])
def test_copies_exactly_the_pairs(native_libs, contiguous, dtype, kv, hs, bs):
    import torch
    from orinmllm_b200 import capi
    dt = getattr(torch, dtype)
    layers, blocks = 3, 41
    gen = torch.Generator(device="cuda").manual_seed(1)
    shape = (layers, blocks, bs, kv, hs) if contiguous else (layers, blocks, kv, bs, hs)
    kp, vp = (torch.randn(shape, generator=gen, device="cuda").to(dt) for _ in range(2))
    lay = (capi.layout_contiguous if contiguous else capi.layout_paged)(capi.dtype_code(dt), kv, hs, bs, blocks)
    src = torch.tensor([0, 7, -1, 5, 9, 40, 3], dtype=torch.int32, device="cuda")
    dst = torch.tensor([20, 21, 22, -1, 9, 23, 24], dtype=torch.int32, device="cuda")
    want = [p.clone() for p in (kp, vp)]
    for p in want:
        for s, d in zip(src.tolist(), dst.tolist()):
            if s >= 0 and d >= 0:
                p[:, d] = p[:, s]
    capi.cow_copy_blocks(kp, vp, lay, layers, blocks * kv * bs * hs, src, dst, len(src))
    assert torch.equal(kp, want[0]) and torch.equal(vp, want[1])
