"""One new token per row and several query heads to a key/value head: the heads of a group are the rows of a tile.  Against float64
at tile edges, group sizes, rows that start late in their slots, an absent row, alone and with the keys cut into shares."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HD = 128


@pytest.mark.parametrize("nh,nkv", [(4, 2), (32, 8), (7, 1), (128, 1), (6, 2)])
@pytest.mark.parametrize("lengths,shares", [((1,), 1), ((64, 65, 1), 1), ((333, 0, 128, 700), 1), ((700, 63), 3), ((1, 2000), 16)])
def test_heads_of_a_group_as_rows(nh, nkv, lengths, shares):
    from recurrent_drafting import _lib

    B, slots = len(lengths), max(lengths) + 9
    g = torch.Generator(device="cuda").manual_seed(nh + sum(lengths))
    new = [1 if n else 0 for n in lengths]
    M = sum(new)
    q = torch.randn(M, nh * HD, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, nkv, slots, HD, generator=g, device="cuda").bfloat16() for _ in "kv")
    begin = [b % 3 for b in range(B)]
    i32 = dict(dtype=torch.int32, device="cuda")
    row_start = torch.tensor([sum(new[:b]) for b in range(B + 1)], **i32)
    out = torch.full_like(q, 9.0)
    status = torch.zeros(1, **i32)
    plan = _lib.load().rd_attention_plan_create(_lib.ptr(q), M, _lib.ptr(k), _lib.ptr(v), B, nh, nkv, HD, slots)
    need = _lib.load().rd_attention_split_workspace_bytes(M, nh, shares)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    kv_begin, base = torch.tensor(begin, **i32), torch.tensor([max(n - 1, 0) for n in lengths], **i32)
    args = (_lib.ptr(row_start), _lib.ptr(kv_begin), _lib.ptr(base), 1, _lib.ATTN_CAUSAL, None, 0)
    if shares > 1:
        _lib.call("rd_attention_tc_split", plan, _lib.ptr(out), *args, shares, _lib.ptr(ws), need, _lib.ptr(status), _lib.stream())
    else:
        _lib.call("rd_attention_tc", plan, _lib.ptr(out), *args, _lib.ptr(status), _lib.stream())
    torch.cuda.synchronize()
    _lib.load().rd_attention_plan_destroy(plan)
    assert int(status.item()) == 0
    for b, n in enumerate(lengths):
        if not n:
            continue
        t = int(row_start[b])
        qd = q[t].double().view(nh, HD)
        kd, vd = (x[b, :, begin[b] : begin[b] + n].double().repeat_interleave(nh // nkv, dim=0) for x in (k, v))
        p = torch.softmax((qd[:, None] * kd).sum(-1) * HD ** -0.5, dim=-1)
        want, size = (p[:, :, None] * vd).sum(1), (p[:, :, None] * vd.abs()).sum(1)
        # the probabilities and the result are rounded to bf16: half a unit in the last place, 2^-8 of the value, each
        assert ((out[t].double().view(nh, HD) - want).abs() <= 2.0 ** -8 * want.abs() + 1.05 * 2.0 ** -8 * size).all()
