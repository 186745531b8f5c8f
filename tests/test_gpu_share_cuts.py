"""Where K is cut into shares does not depend on the room for tokens: the shares of a token have the same bits on both sides of 64 tokens of
capacity (two k-blocks a load, and one) and of 256 (slabs, and pairs of CTAs), and so does their sum."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# features, K, shares: k-blocks of 64 that do not divide among the shares, shares that end inside a load of two, an odd number of k-blocks
@pytest.mark.parametrize("n,k,shares", [(4096, 11008, 4), (1024, 4800, 8), (2048, 1088, 2), (512, 1024, 2)])
def test_shares_of_a_token_at_every_capacity(n, k, shares):
    from recurrent_drafting.modeling_common import Linear

    g = torch.Generator(device="cuda").manual_seed(n + k)
    lin = Linear((torch.randn(n, k, generator=g, device="cuda") / k ** 0.5).bfloat16())
    live = 13
    a = torch.randn(1000, k, generator=g, device="cuda").bfloat16()
    r, c = torch.randn(1000, n, generator=g, device="cuda"), torch.empty(1000, n, device="cuda")
    status, m_dev = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.tensor([live], dtype=torch.int32, device="cuda")
    seen = {}
    for room in (live, 64, 65, 256, 257, 1000):
        rows = min(room, 256)
        assert lin.shares_bytes(room) == 4 * shares * rows * n
        parts = torch.full((shares, rows, n), float("nan"), device="cuda")
        assert lin.add_residual(a[:room], c[:room], r[:room], None if room == live else m_dev, room, status, parts.view(-1)) is not None
        seen[room] = parts[:, :live].clone()
    assert int(status.item()) == 0
    for room, parts in seen.items():
        assert torch.equal(parts, seen[1000]), room
