"""Gates of more heads than one slab of 128 weight rows holds, in the projection of few tokens, against float64 and against the kernel for
more tokens; the second slab's last gates lie before its end."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("m,live", [(1, None), (33, None), (256, 200)])
@pytest.mark.parametrize("nh,nkv", [(132, 4), (130, 1), (129, 3)])
def test_gates_of_a_second_slab(nh, nkv, m, live, early):
    from recurrent_drafting import _lib
    from recurrent_drafting.modeling_common import Linear
    from recurrent_drafting.modeling_llama import rope_tables

    k, max_len, n_pos, room = 256, 64, 128, 300
    g = torch.Generator(device="cuda").manual_seed(nh + m)
    w = (torch.randn((nh + 2 * nkv) * 128 + nh, k, generator=g, device="cuda") / k ** 0.5).bfloat16()
    lin = Linear(w)
    assert [_lib.load().rd_gemm_few_rows(rows, w.shape[0], k) for rows in (m, room)] == [1, 0]
    cos, sin = rope_tables(128, n_pos, 10000.0, "cuda")
    rows = m if live is None else live
    i32 = dict(dtype=torch.int32, device="cuda")
    a = torch.randn(room, k, generator=g, device="cuda").bfloat16()
    at = torch.arange(room, **i32)
    tok_row, tok_slot, status = at // max_len, at % max_len, torch.zeros(1, **i32)
    got = []
    for cap, m_dev in ((m, None if live is None else torch.tensor([live], **i32)), (room, torch.tensor([rows], **i32))):
        q = torch.full((room, nh * 128), 50.0, dtype=torch.bfloat16, device="cuda")
        kc, vc = (torch.full((5, nkv, max_len, 128), 50.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        gate = torch.full((room, nh + 5), 50.0, dtype=torch.bfloat16, device="cuda")
        lin.qkvg_rope(a[:cap], q, kc, vc, gate, tok_row, tok_slot, tok_slot, cos, sin, nh, nkv, 128, m_dev, cap, status, early=early)
        got.append((q, kc, vc, gate))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    gate = got[0][3]
    assert (gate[rows:] == 50.0).all() and (gate[:, nh:] == 50.0).all()
    exact = a[:rows].double() @ w[-nh:].double().T
    size = a[:rows].double().abs() @ w[-nh:].double().abs().T
    # any order of k fp32 additions, and one rounding to bf16
    assert ((gate[:rows, :nh].double() - exact).abs() <= 2.0 ** -8 * exact.abs() + (k + 16) * 2.0 ** -24 * size).all()
    for x, y in zip(*got):
        assert (x == 50.0).equal(y == 50.0)  # the same elements are written
        # two bf16 roundings on the way, of the product and of what it is turned into
        assert ((x.float() - y.float()).abs() <= 2.0 ** -7 * y.float().abs() + 2.0 ** -8 * 4).all()
