"""Arg-max over the slices of a vocabulary: both sides of what a group of threads takes at once (128 slices of 32 ids, eight times that),
of the eight tokens of a block, and equal logits in slices far apart, where the smallest id wins."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 8, 9])
@pytest.mark.parametrize("n", [32, 64, 4096, 4128, 32768, 32800, 65568])
def test_smallest_id_of_the_largest_logit(m, n):
    from recurrent_drafting import _lib
    from recurrent_drafting.modeling_common import Linear

    k = 64
    g = torch.Generator(device="cuda").manual_seed(n + m)
    w = torch.randint(-2, 3, (n, k), generator=g, device="cuda").bfloat16()
    a = torch.randint(-2, 3, (m, k), generator=g, device="cuda").bfloat16()  # whole numbers: the logits are exact
    top = a.float() @ w.float().T
    for t in range(m):  # two more rows of weights with the winner's logit, the last one of the vocabulary among them
        w[[n - 1 - 2 * t % n, n // 2 + t % 8]] = w[int(top[t].argmax())].clone()
    logits = (a.float() @ w.float().T).cpu().numpy()
    out = torch.full((m,), -1, dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    ws = torch.empty(_lib.load().rd_gemm_argmax_workspace_bytes(m, n), dtype=torch.uint8, device="cuda")
    Linear(w, None).argmax(a, out, ws, None, m, status)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    assert out.tolist() == logits.argmax(axis=1).tolist()  # numpy: the first among equals
