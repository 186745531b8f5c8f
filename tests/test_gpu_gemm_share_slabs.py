"""Shares of K of projections with a residual for at most 256 tokens (slabs of 128 weight rows): against float64 where the token boxes, the
k-blocks of a load and the ends of slabs, shares and vectors change, in order and ahead of the dependency wait."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (rows, live rows or None, features, K): K in k-blocks of 64 that do not divide among the shares; features that end inside a slab and off a
# vector; fewer k-blocks than a ring holds and many times more
@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("m,live,n,k", [(1, None, 4096, 11008), (16, None, 256, 1024), (17, 3, 2048, 1088), (64, None, 4000, 1728), (65, 65, 4001, 2048),
                                        (128, 0, 512, 1024), (160, None, 8192, 1024), (225, 101, 4096, 5632), (256, None, 2050, 4160)])
def test_shares_add_up(m, live, n, k, early):
    from recurrent_drafting.modeling_common import Linear

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    lin = Linear((torch.randn(n, k, generator=g, device="cuda") / k ** 0.5).bfloat16())
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    r, c = torch.randn(m, n, generator=g, device="cuda"), torch.full((m, n), 5.0, device="cuda")
    shares = lin.shares_bytes(m) // (4 * m * n)
    assert shares > 1
    rows = m if live is None else live
    m_dev = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    parts = [torch.full((shares, m, n), float("nan"), device="cuda") for _ in range(2)]
    for p in parts:  # one after the other: with early weights a launch begins while the one before runs
        assert lin.add_residual(a, c, r, m_dev, m, status, p.view(-1), early=early) is not None
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert (c == 5.0).all()
    assert torch.equal(parts[0][:, :rows], parts[1][:, :rows]) and parts[0][:, rows:].isnan().all()
    exact = a.double() @ lin.weight.double().T
    slack = (k + 16) * 2.0 ** -24 * (a.double().abs() @ lin.weight.double().abs().T)  # any order of k fp32 additions
    assert ((parts[0].double().sum(0) - exact).abs()[:rows] <= slack[:rows]).all()
