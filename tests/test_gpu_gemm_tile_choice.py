"""The CUDA-core GEMM at the sizes where its tiles and its kind of launch change."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# (m, n, k): 74 and 75 tiles of 32x32 (launched programmatically or not); 148 and 150; 296 and 298 (two and three on an SM); 590 and 592 of
# few rows, the last below and the first at 296 tiles of 64x64; many rows
@pytest.mark.parametrize("m,n,k", [(32, 2368, 65), (31, 2370, 65), (33, 2368, 20), (64, 2400, 20), (64, 4736, 33), (64, 4738, 33),
                                   (20, 18880, 24), (20, 18882, 24), (512, 2304, 72)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_tiles_and_launches(m, n, k, dtype):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").to(dtype)
    w = torch.randn(n, k, generator=g, device="cuda").to(dtype)
    exact = a.double() @ w.double().T
    slack = (k + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)  # any order of k fp32 additions
    outs = [torch.full((m + 1, n), 5.0, device="cuda") for _ in range(4)]
    live = torch.tensor([m - 1], dtype=torch.int32, device="cuda")
    for c in outs:  # one after the other
        _lib.call("rd_gemm", _lib.dtype_code(dtype), _lib.F32, _lib.ptr(a), k, _lib.ptr(w), k, _lib.ptr(c), n, None, None, 0, m,
                  _lib.ptr(live), n, k, _lib.EPI_NONE, _lib.stream())
    for c in outs:
        assert ((c.double()[:m - 1] - exact[:m - 1]).abs() <= slack[:m - 1] + 1e-30).all()
        assert (c[m - 1:] == 5.0).all()
