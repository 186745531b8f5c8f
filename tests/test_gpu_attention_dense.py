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


def _attend(shape, q, k, v, mask, kernel):
    from recurrent_drafting import _lib

    B, nh, nkv, n, S, slots, shares = shape
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
    return out


@pytest.mark.parametrize("kernel", ["tensor", "cuda"])
@pytest.mark.parametrize("shape", SHAPES)
def test_dense_mask(shape, kernel):
    q, k, v, mask = _problem(shape)
    out = _attend(shape, q, k, v, mask, kernel)
    want, size = _exact(shape, q, k, v, mask)
    # one rounding to bf16 (half a unit in the last place: 2^-8 of the value at most) and, of the scores' fp32 sums and the
    # exponential, 2^-15 of the sum of magnitudes
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -15 * size).all()


# what a hidden slot holds: NaN and infinities of either sign in its value, its key, or both
@pytest.mark.parametrize("kernel", ["tensor", "cuda"])
@pytest.mark.parametrize("shape", [(2, 4, 1, 63, 65, 140, 1), (2, 4, 2, 150, 250, 410, 1), (1, 8, 2, 17, 700, 720, 3), (3, 2, 2, 1, 40, 41, 1)])
def test_values_that_are_not_numbers(shape, kernel):
    B, nh, nkv, n, S, slots, shares = shape
    T = S + n
    q, k, v, mask = _problem(shape, seed=11)
    nan, inf = float("nan"), float("inf")
    hidden = torch.zeros(B, T, dtype=torch.bool, device="cuda")
    hidden[:, 3 : T : 29] = True  # nobody sees these
    mask &= ~hidden[:, None]
    at = hidden.nonzero().tolist()
    for i, (b, j) in enumerate(at):
        v[b, :, j, i % HD] = (nan, inf, -inf)[i % 3]
        v[b, :, j, (i + 64) % HD] = (inf, -inf, nan)[i % 3]
        if i % 2:
            k[b, :, j] = (nan, inf, -inf)[i // 2 % 3]
    v[:, :, T:] = nan  # past the live slots
    k[:, :, T:] = inf
    # and one that a third of the queries see: +inf, -inf and NaN in three features, both infinities in a fourth
    seen = torch.arange(n, device="cuda") % 3 == 0
    for b in range(B):
        mask[b, :, 7] = mask[b, :, 9] = seen
        v[b, 0, 7, 100], v[b, 0, 7, 5], v[b, 0, 9, 31], v[b, 0, 9, 64] = inf, -inf, nan, inf
        v[b, 0, 7, 96], v[b, 0, 9, 96] = inf, -inf
    out = _attend(shape, q, k, v, mask, kernel)
    want, size = _exact(shape, q, k.nan_to_num(0, 0, 0), v.nan_to_num(0, 0, 0), mask)
    want, size = want.view(B, n, nh, HD), size.view(B, n, nh, HD)
    for h in range(nh // nkv):  # the query heads of key/value head 0
        for d, x in ((100, inf), (5, -inf), (31, nan), (64, inf), (96, nan)):
            want[:, seen, h, d] = x
    out = out.double().view(B, n, nh, HD)
    finite = want.isfinite()
    assert torch.equal(out[~finite].nan_to_num(1, 2, 3), want[~finite].nan_to_num(1, 2, 3))
    off = (out - want).abs()[finite]
    assert (off <= (2.0 ** -8 * want.abs() + 2.0 ** -15 * size)[finite]).all()


@pytest.mark.parametrize("kernel", ["tensor", "cuda"])
def test_probabilities_have_24_bits(kernel):
    """Two keys of probability 1 take away the first and the second 8 bits of a third's: the rest is the result."""
    heads = 32
    q = torch.zeros(1, heads, HD, device="cuda")
    q[..., 0] = 1
    k = torch.zeros(1, heads, 4, HD, device="cuda")
    k[0, :, 2, 0] = -torch.linspace(0.37, 7.1, heads, device="cuda").bfloat16().float()
    k[0, :, 3, 0] = 50  # hidden
    p = torch.exp(k[0, :, 2, 0].double() * HD ** -0.5)
    hi = p.bfloat16().double()
    mid = (p - hi).bfloat16().double()
    rest = p - hi - mid
    assert (rest.abs() > 2.0 ** -19).sum() >= 4  # with 16 bits the result is zero
    v = torch.ones(1, heads, 4, HD, device="cuda")
    v[0, :, 0], v[0, :, 1] = -hi.float()[:, None], -mid.float()[:, None]
    mask = torch.tensor([[[True, True, True, False]]], device="cuda")
    out = _attend((1, heads, heads, 1, 3, 4, 1), q.view(1, -1).bfloat16(), k.bfloat16(), v.bfloat16(), mask, kernel)
    got = out.double().view(heads, HD) * (2 + p)[:, None]
    # the exponential: 2 units in the last place of a number below 1, its argument half of one; three fp32 sums of numbers up to 1
    assert ((got - rest[:, None]).abs() <= 2.0 ** -8 * rest.abs()[:, None] + 6 * 2.0 ** -24).all()


@pytest.mark.parametrize("kernel", ["tensor", "cuda"])
@pytest.mark.parametrize("shares", [1, 3])
def test_scores_that_are_not_numbers(shares, kernel):
    """A visible key that makes NaN of a score makes NaN of the row, also of one that sees nothing else."""
    shape = (1, 4, 2, 9, 700, 720, shares)
    q, k, v, mask = _problem(shape, seed=13)
    mask[:, :, 400] = False
    k[0, :, 400] = float("nan")
    want, size = _exact(shape, q, k.nan_to_num(0), v, mask)
    mask[:, 1] = False
    mask[:, 1, 400] = mask[:, 4, 400] = True
    want.view(9, -1)[[1, 4]] = float("nan")
    out = _attend(shape, q, k, v, mask, kernel).double()
    assert torch.equal(out.isnan(), want.isnan())
    fine = ~want.isnan()
    assert ((out - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -15 * size)[fine].all()


@pytest.mark.parametrize("shares", [1, 3])
def test_mask_of_fewer_words_than_keys(shares):
    """Keys past the mask's words are hidden, and no word of another row or past the last row is read."""
    from recurrent_drafting import _lib

    shape = (2, 4, 2, 9, 700, 720, shares)
    q, k, v, mask = _problem(shape, seed=17)
    short = mask.clone()
    short[:, :, 5 * 64 :] = False
    real = _lib.call

    def call(name, *args):  # packs five words a row; the bits' buffer ends with those of the last row
        if name == "rd_mask_bits":
            rows = args[2]
            bits = call.bits = torch.empty(rows, 5, dtype=torch.int64, device="cuda")
            return real(name, args[0], args[1], rows, 5 * 64, _lib.ptr(bits), 5, args[6])
        if name == "rd_attention_tc_dense":
            args = args[:6] + (_lib.ptr(call.bits), 5) + args[8:]
        return real(name, *args)

    _lib.call = call
    try:
        out = _attend(shape, q, k, v, mask, "tensor")
    finally:
        _lib.call = real
    want, size = _exact(shape, q, k, v, short)
    assert ((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2.0 ** -15 * size).all()
