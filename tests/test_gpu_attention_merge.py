"""Merge of key shares: numbers of shares on both sides of what a warp asks for at once, rows that do not fill the last block, more room
than live tokens, shares without a key.  Against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HD = 128


@pytest.mark.parametrize("nh,nkv", [(1, 1), (6, 3)])
@pytest.mark.parametrize("shares", [2, 4, 5, 9, 16])
def test_shares_of_causal_tokens(nh, nkv, shares):
    from recurrent_drafting import _lib

    lengths, new = [700, 65, 1], [3, 1, 1]  # keys with the new tokens'; the short rows leave most shares without a tile
    B, M, room, slots = 3, 5, 7, 720
    g = torch.Generator(device="cuda").manual_seed(shares + nh)
    q = torch.randn(room, nh * HD, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, nkv, slots, HD, generator=g, device="cuda").bfloat16() for _ in "kv")
    i32 = dict(dtype=torch.int32, device="cuda")
    row_start, zero = torch.tensor([0, 3, 4, 5], **i32), torch.zeros(B, **i32)
    base = torch.tensor([n - m for n, m in zip(lengths, new)], **i32)
    out = torch.full_like(q, 9.0)
    status = torch.zeros(1, **i32)
    plan = _lib.load().rd_attention_plan_create(_lib.ptr(q), room, _lib.ptr(k), _lib.ptr(v), B, nh, nkv, HD, slots)
    need = _lib.load().rd_attention_split_workspace_bytes(room, nh, shares)
    ws = torch.full((need // 4,), float("nan"), device="cuda")
    _lib.call("rd_attention_tc_split", plan, _lib.ptr(out), _lib.ptr(row_start), _lib.ptr(zero), _lib.ptr(base), 3, _lib.ATTN_CAUSAL, None, 0,
              shares, _lib.ptr(ws), need, _lib.ptr(status), _lib.stream())
    torch.cuda.synchronize()
    _lib.load().rd_attention_plan_destroy(plan)
    assert int(status.item()) == 0
    assert (out[M:] == 9.0).all()
    for b in range(B):
        for i in range(new[b]):
            t, n = int(row_start[b]) + i, lengths[b] - new[b] + i + 1
            qd = q[t].double().view(nh, HD)
            kd, vd = (x[b, :, :n].double().repeat_interleave(nh // nkv, dim=0) for x in (k, v))
            p = torch.softmax((qd[:, None] * kd).sum(-1) * HD ** -0.5, dim=-1)
            want, size = (p[:, :, None] * vd).sum(1), (p[:, :, None] * vd.abs()).sum(1)
            # the probabilities and the result are rounded to bf16: half a unit in the last place, 2^-8 of the value, each
            assert ((out[t].double().view(nh, HD) - want).abs() <= 2.0 ** -8 * want.abs() + 1.05 * 2.0 ** -8 * size).all()
