"""Rotary heads whose rows are shared by the CTAs of a cluster, with more blocks of 32 tokens than a cluster has CTAs (slabs of 64 rows, two
CTAs to a head, 65 to 128 tokens): every CTA finishes several blocks, through the second part of its exchange area.  Against the kernel for
more tokens, bit for bit."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("kind", ["qkv", "qkvg", "norm"])
@pytest.mark.parametrize("m,live", [(65, None), (96, None), (97, 97), (128, 100), (128, 128)])  # a count on the device: as if half as many
@pytest.mark.parametrize("nh,nkv", [(32, 8), (36, 3), (29, 9)])
def test_blocks_of_a_cluster(nh, nkv, m, live, kind, early):
    from recurrent_drafting import _lib
    from recurrent_drafting.modeling_common import Linear
    from recurrent_drafting.modeling_llama import rope_tables

    k, max_len, n_pos, room = 320, 160, 200, 300
    g = torch.Generator(device="cuda").manual_seed(nh + m)
    heads = nh + (1 if kind == "norm" else 2) * nkv
    w = (torch.randn(heads * 128 + (nh if kind == "qkvg" else 0), k, generator=g, device="cuda") / k ** 0.5).bfloat16()
    lin = Linear(w)
    assert 4736 < w.shape[0] <= 9472  # slabs of 64 rows
    assert [_lib.load().rd_gemm_few_rows(rows, w.shape[0], k) for rows in (m, room)] == [1, 0]
    cos, sin = rope_tables(128, n_pos, 10000.0, "cuda")
    i32 = dict(dtype=torch.int32, device="cuda")
    rows = m if live is None else live
    a = torch.randn(room, k, generator=g, device="cuda").bfloat16()
    at = torch.arange(room, **i32)
    toks = (at % 2, torch.randint(0, n_pos, (room,), generator=g, device="cuda", dtype=torch.int32), at // 2, cos, sin, nh, nkv)
    status, got = torch.zeros(1, **i32), []
    for cap, m_dev in ((m, None if live is None else torch.tensor([live], **i32)), (room, torch.tensor([rows], **i32))):
        q = torch.full((room, nh * 128), 50.0, dtype=torch.bfloat16, device="cuda")
        kc, vc = (torch.full((2, nkv, max_len, 128), 50.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        gate = torch.full((room, nh), 50.0, dtype=torch.bfloat16, device="cuda")
        if kind == "qkv":
            lin.qkv_rope(a[:cap], q, kc, vc, *toks, 128, m_dev, cap, status, early=early)
        elif kind == "qkvg":
            lin.qkvg_rope(a[:cap], q, kc, vc, gate, *toks, 64, m_dev, cap, status, early=early)
        else:
            lin.qk_rope_norm(a[:cap], q, kc, vc, *toks, 128, 1e-6, m_dev, cap, status, early=early)
        got.append((q, kc, vc, gate))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert (got[0][0][:rows] != 50.0).all() and (got[0][0][rows:] == 50.0).all()
    for x, y in zip(*got):
        assert torch.equal(x, y)
