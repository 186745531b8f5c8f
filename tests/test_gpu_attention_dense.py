"""Explicit-mask attention on the tensor cores against float64, at tile edges, with masks that hide whole tiles, whole rows and
single keys, alone and with the keys cut into shares.  The CUDA-core kernel that also serves such calls is held to the same
bound."""
import pytest
import torch

pytestmark = pytest.mark.gpu

HD = 128
# (batch, heads, kv heads, new tokens, cached tokens, slots, key shares)
SHAPES = [(1, 2, 2, 1, 0, 8, 1), (2, 4, 1, 63, 65, 140, 1), (3, 4, 2, 64, 64, 128, 1), (2, 4, 4, 129, 200, 400, 1), (1, 8, 2, 17, 700, 720, 3),
          (1, 4, 4, 130, 511, 700, 2)]


def _problem(shape, seed=5):
    B, nh, nkv, n, S, slots, _ = shape
    g = torch.Generator(device="cuda").manual_seed(seed + n)
    q = torch.randn(B * n, nh * HD, generator=g, device="cuda").bfloat16()
    k = torch.randn(B, nkv, slots, HD, generator=g, device="cuda").bfloat16()
    v = torch.randn(B, nkv, slots, HD, generator=g, device="cuda").bfloat16()
    mask = torch.rand(B, n, S + n, generator=g, device="cuda") < 0.6
    mask[:, ::3] |= torch.rand(S + n, generator=g, device="cuda") < 0.5
    if n > 8:
        mask[:, 3] = False  # a row that sees nothing
        mask[:, 5] = True
        mask[:, 6, : (S + n) // 2] = False  # whole tiles hidden
        mask[:, 7] = False
        mask[:, 7, -1] = True
    return q, k, v, mask


def _exact(shape, q, k, v, mask):
    B, nh, nkv, n, S, _, _ = shape
    qd = q.double().view(B, n, nh, HD).transpose(1, 2)
    kd = k.double()[:, :, : S + n].repeat_interleave(nh // nkv, dim=1)
    vd = v.double()[:, :, : S + n].repeat_interleave(nh // nkv, dim=1)
    s = (qd @ kd.transpose(2, 3) * HD ** -0.5).masked_fill(~mask[:, None], -float("inf"))
    p = torch.softmax(s, dim=-1).nan_to_num(0.0)
    size = p @ vd.abs()
    return ((t.transpose(1, 2).reshape(B * n, nh * HD)) for t in (p @ vd, size))


@pytest.mark.parametrize("kernel", ["tensor", "cuda"])
@pytest.mark.parametrize("shape", SHAPES)
def test_dense_mask(shape, kernel):
    from recurrent_drafting import _lib

    B, nh, nkv, n, S, slots, shares = shape
    q, k, v, mask = _problem(shape)
    out = torch.full_like(q, 9.0)
    i32 = dict(dtype=torch.int32, device="cuda")
    row_start, begin, base = torch.arange(B + 1, **i32) * n, torch.zeros(B, **i32), torch.full((B,), S, **i32)
    bytes_ = mask.to(torch.uint8).contiguous()
    st = _lib.stream()
    status = torch.zeros(1, **i32)
    if kernel == "cuda":
        _lib.call("rd_attention", _lib.BF16, _lib.ptr(q), _lib.ptr(k), _lib.ptr(v), _lib.ptr(out), _lib.ptr(row_start), _lib.ptr(begin),
                  _lib.ptr(base), B, nh, nkv, HD, slots, n, S + n, _lib.ATTN_DENSE, None, 0, _lib.ptr(bytes_), bytes_.stride(1),
                  bytes_.stride(0), st)
    else:
        words = (S + n + 63) // 64
        bits = torch.full((B * n, words), -1, dtype=torch.int64, device="cuda")
        _lib.call("rd_mask_bits", _lib.ptr(bytes_), S + n, B * n, S + n, _lib.ptr(bits), words, st)
        plan = _lib.load().rd_attention_plan_create(_lib.ptr(q), B * n, _lib.ptr(k), _lib.ptr(v), B, nh, nkv, HD, slots)
        need = _lib.load().rd_attention_split_workspace_bytes(B * n, nh, shares)
        ws = torch.empty(need, dtype=torch.uint8, device="cuda")
        _lib.call("rd_attention_tc_dense", plan, _lib.ptr(out), _lib.ptr(row_start), _lib.ptr(begin), _lib.ptr(base), n, _lib.ptr(bits), words,
                  shares, _lib.ptr(ws), need, _lib.ptr(status), st)
    torch.cuda.synchronize()
    if kernel == "tensor":
        _lib.load().rd_attention_plan_destroy(plan)
    assert int(status.item()) == 0
    want, size = _exact(shape, q, k, v, mask)
    # one rounding to bf16 (half a unit in the last place: 2^-8 of the value at most) and, of the probabilities' 17 bits, the scores' fp32 sums and the exponential,
    # 2^-15 of the sum of magnitudes
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -15 * size).all()
