"""Single tokens of grouped heads under a window or a chunk, with kept first tokens, gate and sink, alone and with the keys cut into
shares: against float64 at tile edges, rows that start late in their slots, an absent row, more shares than tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HD = 128


@pytest.mark.parametrize("nh,nkv", [(4, 2), (32, 8), (5, 1)])
@pytest.mark.parametrize("kind,window,keep", [("window", 100, 0), ("window", 64, 70), ("window", 2000, 4), ("chunk", 128, 0), ("chunk", 300, 3)])
@pytest.mark.parametrize("lengths,shares", [((1,), 1), ((64, 65, 128, 129), 1), ((333, 0, 700), 1), ((700, 63, 384), 3), ((1, 900), 16)])
def test_against_float64(nh, nkv, kind, window, keep, lengths, shares):
    from recurrent_drafting import _lib

    B, slots = len(lengths), max(lengths) + 9
    g = torch.Generator(device="cuda").manual_seed(nh + sum(lengths) + window)
    new = [1 if n else 0 for n in lengths]
    M = sum(new)
    q = torch.randn(M, nh * HD, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(B, nkv, slots, HD, generator=g, device="cuda").bfloat16() for _ in "kv")
    gated, sunk = nh != 4, nh != 32
    gate = torch.randn(M, nh + 3, generator=g, device="cuda").bfloat16() if gated else None
    sink = torch.randn(nh, generator=g, device="cuda") if sunk else None
    begin = [b % 3 for b in range(B)]
    i32 = dict(dtype=torch.int32, device="cuda")
    row_start = torch.tensor([sum(new[:b]) for b in range(B + 1)], **i32)
    out = torch.full_like(q, 9.0)
    status = torch.zeros(1, **i32)
    plan = _lib.load().rd_attention_plan_create(_lib.ptr(q), M, _lib.ptr(k), _lib.ptr(v), B, nh, nkv, HD, slots)
    kv_begin, base = torch.tensor(begin, **i32), torch.tensor([max(n - 1, 0) for n in lengths], **i32)
    code = _lib.MASK_WINDOW if kind == "window" else _lib.MASK_CHUNK
    where, tail = (_lib.ptr(out), _lib.ptr(row_start), _lib.ptr(kv_begin), _lib.ptr(base), 1), (HD ** -0.5, code, window, keep, _lib.ptr(gate), nh + 3, _lib.ptr(sink))
    if shares > 1:
        need = _lib.load().rd_attention_split_workspace_bytes(M, nh, shares)
        ws = torch.full((need // 4,), float("nan"), device="cuda")
        with pytest.raises(_lib.RedrafterError):
            _lib.call("rd_attention_tc_masked_split", plan, *where, *tail, shares, _lib.ptr(ws), need - 1, _lib.ptr(status), _lib.stream())
        _lib.call("rd_attention_tc_masked_split", plan, *where, *tail, shares, _lib.ptr(ws), need, _lib.ptr(status), _lib.stream())
    else:
        _lib.call("rd_attention_tc_masked", plan, *where, _lib.ATTN_CAUSAL, None, None, 0, *tail, _lib.ptr(status), _lib.stream())
    torch.cuda.synchronize()
    _lib.load().rd_attention_plan_destroy(plan)
    assert int(status.item()) == 0
    for b, n in enumerate(lengths):
        if not n:
            continue
        t = int(row_start[b])
        pos = torch.arange(n, device="cuda")
        first = n - window if kind == "window" else (n - 1) // window * window
        seen = (pos >= first) | (pos < keep)
        qd = q[t].double().view(nh, HD)
        kd, vd = (x[b, :, begin[b] : begin[b] + n].double()[:, seen].repeat_interleave(nh // nkv, dim=0) for x in (k, v))
        score = (qd[:, None] * kd).sum(-1) * HD ** -0.5
        if sunk:
            score = torch.cat([score, sink.double()[:, None]], dim=1)
        p = torch.softmax(score, dim=-1)[:, : vd.shape[1]]
        f = torch.sigmoid(gate[t, :nh].double())[:, None] if gated else 1.0
        want, size = (p[:, :, None] * vd).sum(1) * f, (p[:, :, None] * vd.abs()).sum(1) * f
        # the result is rounded to bf16: 2^-8 of it.  Ahead of that: probabilities of 16 bits, and scores of 128 fp32 products, whose
        # absolute values add up to some 10: 128 x 2^-24 x 10 of a probability
        assert ((out[t].double().view(nh, HD) - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -13 * size).all()


@pytest.mark.parametrize("shares", [1, 2])
def test_an_infinite_value_that_is_seen(shares):
    from recurrent_drafting import _lib

    nh, nkv, n = 4, 2, 200
    g = torch.Generator(device="cuda").manual_seed(3)
    q = torch.randn(1, nh * HD, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(1, nkv, n, HD, generator=g, device="cuda").bfloat16() for _ in "kv")
    i32 = dict(dtype=torch.int32, device="cuda")
    row_start, zero, base, status = torch.tensor([0, 1], **i32), torch.zeros(1, **i32), torch.tensor([n - 1], **i32), torch.zeros(1, **i32)
    ws = torch.empty(_lib.load().rd_attention_split_workspace_bytes(1, nh, 2), dtype=torch.uint8, device="cuda")
    outs = []
    for special in (0.0, float("inf")):
        v[0, 0, 120:136, 5] = special  # some of these probabilities have no bits past the first part's
        v[0, 1, 64, 7] = -special
        out = torch.empty_like(q)
        plan = _lib.load().rd_attention_plan_create(_lib.ptr(q), 1, _lib.ptr(k), _lib.ptr(v), 1, nh, nkv, HD, n)
        args = (plan, _lib.ptr(out), _lib.ptr(row_start), _lib.ptr(zero), _lib.ptr(base), 1)
        tail = (HD ** -0.5, _lib.MASK_WINDOW, n, 0, None, 0, None)
        if shares > 1:
            _lib.call("rd_attention_tc_masked_split", *args, *tail, shares, _lib.ptr(ws), ws.numel(), _lib.ptr(status), _lib.stream())
        else:
            _lib.call("rd_attention_tc_masked", *args, _lib.ATTN_CAUSAL, None, None, 0, *tail, _lib.ptr(status), _lib.stream())
        torch.cuda.synchronize()
        _lib.load().rd_attention_plan_destroy(plan)
        outs.append(out.view(nh, HD))
    assert int(status.item()) == 0
    want = outs[0].clone()
    want[:2, 5], want[2:, 7] = float("inf"), -float("inf")
    assert torch.equal(outs[1], want)


@pytest.mark.parametrize("nh,nkv", [(3, 3), (6, 2)])
def test_shares_of_several_causal_tokens(nh, nkv):
    """Cut and whole differ by the rounding of the probabilities to bf16 and of the results, 2^-8 of a value each on both sides."""
    from recurrent_drafting import _lib

    lengths, new, slots, shares = [333, 90], [3, 2], 340, 4
    g = torch.Generator(device="cuda").manual_seed(nh)
    q = torch.randn(5, nh * HD, generator=g, device="cuda").bfloat16()
    k, v = (torch.randn(2, nkv, slots, HD, generator=g, device="cuda").bfloat16() for _ in "kv")
    gate, sink = torch.randn(5, nh, generator=g, device="cuda").bfloat16(), torch.randn(nh, generator=g, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    row_start, zero = torch.tensor([0, 3, 5], **i32), torch.zeros(2, **i32)
    base, status = torch.tensor([n - m for n, m in zip(lengths, new)], **i32), torch.zeros(1, **i32)
    plan = _lib.load().rd_attention_plan_create(_lib.ptr(q), 5, _lib.ptr(k), _lib.ptr(v), 2, nh, nkv, HD, slots)
    whole, cut, size = (torch.empty_like(q) for _ in range(3))
    ws = torch.empty(_lib.load().rd_attention_split_workspace_bytes(5, nh, shares), dtype=torch.uint8, device="cuda")
    arrays = (_lib.ptr(row_start), _lib.ptr(zero), _lib.ptr(base), 3)
    tail = (HD ** -0.5, _lib.MASK_WINDOW, 200, 4, _lib.ptr(gate), nh, _lib.ptr(sink))

    def run_whole(out):
        _lib.call("rd_attention_tc_masked", plan, _lib.ptr(out), *arrays, _lib.ATTN_CAUSAL, None, None, 0, *tail, _lib.ptr(status), _lib.stream())

    run_whole(whole)
    _lib.call("rd_attention_tc_masked_split", plan, _lib.ptr(cut), *arrays, *tail, shares, _lib.ptr(ws), ws.numel(), _lib.ptr(status), _lib.stream())
    v.abs_()
    run_whole(size)
    torch.cuda.synchronize()
    _lib.load().rd_attention_plan_destroy(plan)
    assert int(status.item()) == 0
    assert ((cut.double() - whole.double()).abs() <= 2.0 ** -7 * (whole.double().abs() + 1.1 * size.double())).all()
