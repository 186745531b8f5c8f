"""What the first iteration of the beam search stages and hands to all beams of a row (rd_drafter_begin, rd_drafter_spread), where rows
take vector copies and where they do not, one beam and the most."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("B,W,H,Lb", [(1, 1, 64, 2), (3, 5, 37, 3), (2, 64, 2056, 8), (5, 2, 1030, 4)])
def test_start_and_spread(B, W, H, Lb, dtype):
    from recurrent_drafting import _lib, modeling_drafter

    g = torch.Generator(device="cuda").manual_seed(B * W + H)
    embed, ctx = (torch.randn(n, H, generator=g, device="cuda").to(dtype) for n in (50, B))
    start = torch.randint(0, 50, (B,), generator=g, device="cuda")
    a, x = (torch.full((B * W, 2 * H), 9.0, dtype=dtype, device="cuda") for _ in range(2))
    beams = torch.full((B, W, Lb), -1, dtype=torch.int64, device="cuda")
    code, st = _lib.dtype_code(dtype), _lib.stream()
    _lib.call("rd_drafter_begin", code, _lib.ptr(embed), _lib.ptr(start), _lib.ptr(beams), _lib.ptr(ctx), _lib.ptr(a), _lib.ptr(x), B, W, Lb, H,
              0, st)
    assert (beams[:, :, 0] == start[:, None]).all() and (beams[:, :, 1:] == -1).all()
    assert torch.equal(a.view(B, W, 2 * H)[..., :H], embed[start][:, None].expand(B, W, H)) and (a[:, H:] == 0).all()
    assert torch.equal(x.view(B, W, 2 * H)[..., :H], ctx[:, None].expand(B, W, H)) and (x[:, H:] == 9).all()
    x[:, H:] = torch.randn(B * W, H, generator=g, device="cuda").to(dtype)
    first, q = modeling_drafter.new_sparse(B, "cuda"), modeling_drafter.new_sparse(B * W, "cuda")
    first.val.normal_(generator=g)
    first.masked.normal_(generator=g)
    first.idx.random_(0, 50, generator=g)
    first.cnt.random_(1, 64, generator=g)
    state = x.view(B, W, 2 * H)[:, :1].clone()
    _lib.call("rd_drafter_spread", code, _lib.ptr(first.val), _lib.ptr(first.idx), _lib.ptr(first.cnt), _lib.ptr(first.masked), _lib.ptr(q.val),
              _lib.ptr(q.idx), _lib.ptr(q.cnt), _lib.ptr(q.masked), _lib.ptr(x), B, W, H, st)
    for one, all_ in ((first.val, q.val), (first.idx, q.idx), (first.cnt, q.cnt), (first.masked, q.masked)):
        assert torch.equal(all_, one.repeat_interleave(W, dim=0))
    assert torch.equal(x.view(B, W, 2 * H), state.expand(B, W, 2 * H))
