"""Tensor-core prefill: groups of query heads packed into 128-row items, two items a unit, several units a
cluster.  Sizes at the edges: items with unused rows, a unit of one item, units of one key tile in a row, a
work list beyond what travels as a parameter, a group of 128 heads (one token an item) and of 129."""
import numpy as np
import pytest

from tests import kvtest

pytestmark = pytest.mark.gpu
D, BS = 128, 16


def _call(capi, torch, dtype, q_heads, kv_heads, lens, starts, seed, v_edit=None):
    rng = np.random.default_rng(seed)
    ends = [s + n for s, n in zip(starts, lens)]
    blocks = [-(-e // BS) for e in ends]
    ids = rng.permutation(sum(blocks) + 3).astype(np.int32)
    table = np.zeros((len(lens), max(blocks)), np.int32)
    at = 0
    for i, b in enumerate(blocks):
        table[i, :b] = ids[at:at + b]
        at += b
    shape = (len(ids), kv_heads, BS, D)
    kp = kvtest.to_storage(rng.standard_normal(shape).astype(np.float32), dtype)
    vp = kvtest.to_storage(rng.standard_normal(shape).astype(np.float32), dtype)
    if v_edit:
        v_edit(vp, table)
    q = kvtest.to_storage(rng.standard_normal((sum(lens), q_heads * D)).astype(np.float32), dtype)
    dq, dk, dv = (kvtest.to_device(x, dtype) for x in (q, kp, vp))
    out = torch.full_like(dq, float("nan"))
    lay = capi.layout_paged(capi.dtype_code(kvtest.torch_dtype(dtype)), kv_heads, D, BS, len(ids))
    nbytes = capi.prefill_workspace_bytes(sum(lens), q_heads, kv_heads, D)
    ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    capi.workspace_init(ws, nbytes)
    cu = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    capi.paged_prefill(out, dq, dk, dv, lay, torch.from_numpy(table).cuda(), table.shape[1], cu,
                       np.asarray(starts, np.int32), len(lens), q_heads, 1 / np.sqrt(D), ws, nbytes)
    assert capi.workspace_status(ws) == 0
    return q, kp, vp, table, cu, out


def _reference(torch, dtype, q_heads, kv_heads, q, kp, vp, table, cu, lens, starts):
    """The same in fp64 by plain torch on the GPU."""
    def wide(x):
        return kvtest.to_device(x, dtype).double()
    qd, kd, vd = wide(q).view(-1, q_heads, D), wide(kp), wide(vp)
    outs = []
    for i, (n, s) in enumerate(zip(lens, starts)):
        idx = torch.from_numpy(table[i, :-(-(s + n) // BS)].astype(np.int64)).cuda()
        k = kd[idx].transpose(1, 2).reshape(-1, kv_heads, D)[:s + n]
        v = vd[idx].transpose(1, 2).reshape(-1, kv_heads, D)[:s + n]
        mul = q_heads // kv_heads
        hidden = torch.arange(s + n, device="cuda") > s + torch.arange(n, device="cuda")[:, None]
        scores = torch.einsum("nhd,thd->hnt", qd[cu[i]:cu[i + 1]], k.repeat_interleave(mul, 1)) / np.sqrt(D)
        w = torch.softmax(scores.masked_fill(hidden, -np.inf), -1)
        outs.append(torch.einsum("hnt,thd->nhd", w, v.repeat_interleave(mul, 1)).reshape(n, -1))
    return torch.cat(outs).cpu().numpy().astype(np.float32)


@pytest.mark.parametrize("dtype,q_heads,kv_heads,lens,starts", [
    ("f16", 8, 8, [1, 127, 129, 300], [0, 5, 130, 0]),      # 128 tokens an item
    ("bf16", 6, 2, [43, 85, 170], [0, 0, 90]),              # 42 tokens an item, two rows unused
    ("f16", 14, 2, [18, 19, 36, 37, 500], [0, 126, 127, 128, 3]),
    ("bf16", 128, 2, [3, 65], [130, 0]),                    # two tokens an item
    ("f16", 128, 1, [5], [124]),                            # one
    ("f16", 129, 1, [5], [124]),                            # a group wider than an item: three of 43
    ("bf16", 32, 8, [64] * 75, [0] * 75),                   # units of one key tile, eight a cluster, list in memory
    ("f16", 32, 8, [64] * 37, [64] * 37),                   # four a cluster, list as a parameter
    ("f16", 16, 2, [100], [2000]),                          # few units, cut along the keys
])
def test_units(native_libs, dtype, q_heads, kv_heads, lens, starts):
    import torch
    from orinmllm_b200 import capi
    q, kp, vp, table, cu, out = _call(capi, torch, dtype, q_heads, kv_heads, lens, starts, seed=sum(lens) + q_heads)
    ref = _reference(torch, dtype, q_heads, kv_heads, q, kp, vp, table, cu, lens, starts)
    got = kvtest.storage_to_f32(kvtest.from_device(out, dtype), dtype)
    kvtest.assert_attention_close(got, ref, f"{dtype} {q_heads}/{kv_heads} {lens} {starts}", dtype)


def test_first_item_is_left_alone_by_later_tiles(native_libs):
    """One head a group: the unit's second item sees a key tile that is all newer than the first item's
    rows.  An infinity and a NaN in V there reach no row of the first item."""
    import torch
    from orinmllm_b200 import capi

    def edit(vp, table):
        vp[table[0, 160 // BS], 0, 160 % BS, :] = kvtest.to_storage(np.full(D, np.inf, np.float32), "f16")
        vp[table[0, 200 // BS], 0, 200 % BS, :] = kvtest.to_storage(np.full(D, np.nan, np.float32), "f16")
    q, kp, vp, table, cu, out = _call(capi, torch, "f16", 2, 2, [256], [0], seed=9, v_edit=edit)
    got = out.float().view(256, 2, D)
    assert torch.isfinite(got[:128]).all() and torch.isfinite(got[:, 1]).all()
    assert torch.isnan(got[201:, 0]).all()
