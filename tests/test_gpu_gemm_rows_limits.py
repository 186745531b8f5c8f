"""Numbers of tokens at which projections change from slabs of weight rows to pairs of CTAs: a token's values have the same bits on both
sides, whatever the epilogue, with and without a count on the device, and hold against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _linear(n, k, g):
    from recurrent_drafting.modeling_common import Linear

    return Linear((torch.randn(n, k, generator=g, device="cuda") / k ** 0.5).bfloat16())


# tokens of a call: both sides of the limit without a count, and of twice the limit with one (as far as 256 tokens reach)
@pytest.mark.parametrize("kind,n,k,limit", [
    ("plain", 12288, 128, 192), ("swiglu", 22016, 192, 192), ("plain", 37888, 64, 192), ("slice", 16384, 128, 192), ("argmax", 18944, 128, 192),
    ("slice", 18976, 4096, 96), ("argmax", 18976, 4096, 96), ("slice", 32000, 192, 64), ("argmax", 32000, 192, 64), ("heads", 6144, 256, 96),
    ("heads", 12288, 256, 192)])
def test_both_sides(kind, n, k, limit):
    from recurrent_drafting import _lib
    from recurrent_drafting.modeling_llama import rope_tables

    g = torch.Generator(device="cuda").manual_seed(n + k)
    lin = _linear(n, k, g)
    live = 61
    a = torch.randn(257, k, generator=g, device="cuda").bfloat16()
    i32 = dict(dtype=torch.int32, device="cuda")
    status, at, row = torch.zeros(1, **i32), torch.arange(257, **i32), torch.zeros(257, **i32)
    cos, sin = rope_tables(128, 300, 10000.0, "cuda")
    rooms = {(m, counted) for m in (live, limit, limit + 1, min(2 * limit, 256), min(2 * limit + 1, 257)) for counted in (False, True)}
    seen = {}
    for m, counted in rooms:
        md = torch.tensor([live], **i32) if counted else None
        f32 = torch.full((m, n), 5.0, device="cuda")
        if kind == "plain":
            lin(a[:m], f32, m_dev=md, status=status)
            out = [f32]
        elif kind == "swiglu":
            out = [torch.empty(m, n // 2, dtype=torch.bfloat16, device="cuda")]
            lin(a[:m], out[0], _lib.EPI_SWIGLU, m_dev=md, status=status)
        elif kind == "slice":
            top = torch.empty(n // 32, 288, device="cuda")
            assert lin.with_slice_max(a[:m], f32, top, m_dev=md, status=status)
            out = [f32, top.T]
        elif kind == "argmax":
            out = [torch.full((m,), -1, **i32)]
            ws = torch.empty(_lib.load().rd_gemm_argmax_workspace_bytes(m, n), dtype=torch.uint8, device="cuda")
            lin.argmax(a[:m], out[0], ws, md, m, status)
        else:
            nh, nkv = (32, 8) if n == 6144 else (32, 32)
            q = torch.empty(m, nh * 128, dtype=torch.bfloat16, device="cuda")
            kc, vc = (torch.empty(1, nkv, 300, 128, dtype=torch.bfloat16, device="cuda") for _ in "kv")
            lin.qkv_rope(a[:m], q, kc, vc, row, at, at, cos, sin, nh, nkv, 128, md, m, status)
            out = [q, kc[0].transpose(0, 1), vc[0].transpose(0, 1)]
        seen[m, counted] = [x[:live].clone() for x in out]
        if kind in ("plain", "slice"):
            exact = a[:live].double() @ lin.weight.double().T
            slack = (k + 16) * 2.0 ** -24 * (a[:live].double().abs() @ lin.weight.double().abs().T)  # any order of k fp32 additions
            assert ((f32[:live].double() - exact).abs() <= slack).all()
            assert not counted or (f32[live:] == 5.0).all()
    assert int(status.item()) == 0
    for room, out in seen.items():
        assert all(torch.equal(x, y) for x, y in zip(out, seen[live, False])), room


@pytest.mark.parametrize("n,k", [(8192, 8192), (8192, 8128)])  # at and below 2^26 weights
def test_shares_on_both_sides(n, k):
    g = torch.Generator(device="cuda").manual_seed(n + k)
    lin = _linear(n, k, g)
    a, r = torch.randn(256, k, generator=g, device="cuda").bfloat16(), torch.randn(256, n, generator=g, device="cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    status, seen = torch.zeros(1, **i32), []
    for m, md in ((50, None), (192, None), (193, None), (256, None), (256, torch.tensor([50], **i32))):
        shares = lin.shares_bytes(m) // (4 * m * n)
        assert shares == 2
        parts, c = torch.full((shares, m, n), float("nan"), device="cuda"), torch.empty(m, n, device="cuda")
        assert lin.add_residual(a[:m], c, r[:m], md, m, status, parts.view(-1)) is not None
        seen.append(parts[:, :50].clone())
    assert int(status.item()) == 0
    exact = a[:50].double() @ lin.weight.double().T
    slack = (k + 16) * 2.0 ** -24 * (a[:50].double().abs() @ lin.weight.double().abs().T)  # any order of k fp32 additions
    assert ((seen[0].double().sum(0) - exact).abs() <= slack).all()
    assert all(torch.equal(x, seen[0]) for x in seen)


# more live tokens than half of the capacity: slabs still serve where the count is on the device.  Slabs of 128, 160, 192, 224 and 256 rows
@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("m,live,n,k", [(256, 256, 18944, 128), (256, 256, 22016, 192), (225, 225, 26000, 576), (256, 241, 32000, 128), (256, 250, 37888, 64)])
def test_a_full_capacity_with_a_count(m, live, n, k, early):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(n + k)
    lin = _linear(n, k, g)
    a, r = torch.randn(m, k, generator=g, device="cuda").bfloat16(), torch.randn(m, n, generator=g, device="cuda")
    md, status = torch.tensor([live], dtype=torch.int32, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    outs = [torch.full((m, n), 5.0, device="cuda") for _ in range(3)]
    for c in outs:  # one after the other: with early weights a launch begins while the one before runs
        lin(a, c, _lib.EPI_RES, residual=r, m_dev=md, status=status, early=early)
    act = torch.empty(m, n // 2, dtype=torch.bfloat16, device="cuda")
    lin(a, act, _lib.EPI_SWIGLU, m_dev=md, status=status, early=early)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    acc = a.double() @ lin.weight.double().T
    slack = (k + 16) * 2.0 ** -24 * (r.double().abs() + a.double().abs() @ lin.weight.double().abs().T)  # any order of k fp32 additions
    for c in outs:
        assert ((c.double() - acc - r.double()).abs()[:live] <= slack[:live]).all()
        assert (c[live:] == 5.0).all()
        assert torch.equal(c, outs[0])
    want = (torch.nn.functional.silu(acc[:, 0::2]) * acc[:, 1::2])[:live]
    # one rounding to bf16 of fp32 sums and an approximate exponential
    assert ((act[:live].double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4 * want.abs().max()).all()


@pytest.mark.parametrize("m,k", [(128, 512), (192, 4096)])
@pytest.mark.parametrize("n", [20000, 32000])
def test_maxima_of_a_full_capacity_with_a_count(m, k, n):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(n + k)
    lin = _linear(n, k, g)
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    i32 = dict(dtype=torch.int32, device="cuda")
    md, status = torch.tensor([m], **i32), torch.zeros(1, **i32)
    plain, logits, top, tok = torch.empty(m, n, device="cuda"), torch.empty(m, n, device="cuda"), torch.empty(n // 32, m, device="cuda"), torch.empty(m, **i32)
    lin(a, plain, status=status)
    assert lin.with_slice_max(a, logits, top, m_dev=md, status=status, early=True)
    ws = torch.empty(_lib.load().rd_gemm_argmax_workspace_bytes(m, n), dtype=torch.uint8, device="cuda")
    lin.argmax(a, tok, ws, md, m, status)
    assert int(status.item()) == 0
    assert torch.equal(logits, plain) and torch.equal(top, plain.view(m, n // 32, 32).amax(dim=2).T)
    assert torch.equal(tok.long(), plain.argmax(dim=1))
