"""Single tokens of grouped heads under a window or a chunk: what lies in the cache outside a row's keys, NaN and infinities among it, does not
show, alone and in shares: slots past the row's end, and the first slots of the next head where the row fills its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HD = 128


@pytest.mark.parametrize("fill", [float("nan"), float("inf")])
@pytest.mark.parametrize("nh,nkv", [(4, 2), (32, 8)])
@pytest.mark.parametrize("kind,window,keep", [("window", 100, 4), ("chunk", 128, 0)])
@pytest.mark.parametrize("lengths,spare,shares", [((1,), 9, 1), ((63, 64, 65, 127), 2, 1), ((200, 333, 1, 384), 2, 1), ((700, 63, 385), 70, 3),
                                                  ((1, 900), 2, 16)])
def test_outside_of_a_rows_keys(nh, nkv, kind, window, keep, lengths, spare, shares, fill):
    from recurrent_drafting import _lib

    B, slots = len(lengths), max(lengths) + spare
    g = torch.Generator(device="cuda").manual_seed(nh + sum(lengths))
    q = torch.randn(B, nh * HD, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, nkv, slots, HD, generator=g, device="cuda").bfloat16() for _ in "kv")
    begin = [min(2, slots - n) for n in lengths]  # the longest row may reach its head's last slot
    i32 = dict(dtype=torch.int32, device="cuda")
    row_start, status = torch.arange(B + 1, **i32), torch.zeros(1, **i32)
    kv_begin, base = torch.tensor(begin, **i32), torch.tensor([n - 1 for n in lengths], **i32)
    code = _lib.MASK_WINDOW if kind == "window" else _lib.MASK_CHUNK
    ws = torch.zeros(_lib.load().rd_attention_split_workspace_bytes(B, nh, 16), dtype=torch.uint8, device="cuda")
    outs = []
    for special in (0.0, fill):
        for b, n in enumerate(lengths):
            for x in (k, v):
                x[b, :, : begin[b]] = special
                x[b, :, begin[b] + n :] = special
        out = torch.empty_like(q)
        plan = _lib.load().rd_attention_plan_create(_lib.ptr(q), B, _lib.ptr(k), _lib.ptr(v), B, nh, nkv, HD, slots)
        args = (plan, _lib.ptr(out), _lib.ptr(row_start), _lib.ptr(kv_begin), _lib.ptr(base), 1)
        tail = (HD ** -0.5, code, window, keep, None, 0, None)
        if shares > 1:
            _lib.call("rd_attention_tc_masked_split", *args, *tail, shares, _lib.ptr(ws), ws.numel(), _lib.ptr(status), _lib.stream())
        else:
            _lib.call("rd_attention_tc_masked", *args, _lib.ATTN_CAUSAL, None, None, 0, *tail, _lib.ptr(status), _lib.stream())
        torch.cuda.synchronize()
        _lib.load().rd_attention_plan_destroy(plan)
        outs.append(out)
    assert int(status.item()) == 0
    assert outs[0].isfinite().all() and torch.equal(*outs)
