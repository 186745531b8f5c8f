"""RMS norms where the number of rows or the width changes how a row is held (registers or read again, run ahead or not), one after the
other in a stream, against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("m,live,H", [(1, None, 4096), (64, 63, 4096), (65, None, 72), (64, None, 8192), (3, None, 8200), (2048, 2047, 64),
                                      (2049, None, 64), (5, 0, 1024), (7, None, 100), (2, None, 16384)])
def test_rmsnorm(m, live, H, dtype):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(m + H)
    gain = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(dtype)
    rows = m if live is None else live
    m_dev = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    x = torch.randn(m, H, generator=g, device="cuda").to(dtype)
    steps = [x] + [torch.full_like(x, 9.0) for _ in range(3)]
    for a, b in zip(steps, steps[1:]):  # each reads what the launch before it wrote
        _lib.call("rd_rmsnorm", _lib.dtype_code(dtype), _lib.ptr(a), _lib.ptr(gain), _lib.ptr(b), m, _lib.ptr(m_dev), H, 1e-6, _lib.stream())
    for a, b in zip(steps, steps[1:]):
        want = a.double() / (a.double().square().mean(dim=1, keepdim=True) + 1e-6).sqrt() * gain.double()
        # two roundings to the type, and fp32 sums of H squares
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23 + H * 2.0 ** -24
        assert ((b.double() - want).abs()[:rows] <= 2 * eps * want.abs()[:rows] + 1e-30).all()
        assert (b[rows:] == 9.0).all()


@pytest.mark.parametrize("m,live,H,groups,n_hist", [(1, None, 4096, 1, 1), (64, 63, 4096, 8, 9), (65, None, 1024, 1, 8), (296, None, 64, 2, 17),
                                                    (297, None, 64, 2, 3), (6, None, 100, 4, 5), (3, None, 12, 3, 2), (2, None, 20000, 1, 4)])
def test_stream_norm(m, live, H, groups, n_hist):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(m + H)
    hist = torch.randn(n_hist, m, H, generator=g, device="cuda")
    coeff = torch.randn(n_hist, generator=g, device="cuda") if n_hist > 1 else None
    gain = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).bfloat16()
    rows = m if live is None else live
    m_dev = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    x, y = torch.full((m, H), 9.0, device="cuda"), torch.full((m, H), 9.0, dtype=torch.bfloat16, device="cuda")
    for _ in range(2):
        _lib.call("rd_stream_norm", _lib.BF16, None, None, 0.0, _lib.ptr(hist), hist.stride(0), _lib.ptr(coeff), n_hist, _lib.ptr(x), _lib.ptr(gain),
                  _lib.ptr(y), m, _lib.ptr(m_dev), H, groups, 1e-6, _lib.stream())
    c = coeff.double() if coeff is not None else torch.ones(1, dtype=torch.float64, device="cuda")
    terms = c[:, None, None] * hist.double()
    # a sum of n_hist fused products, each rounded once
    assert ((x.double() - terms.sum(0)).abs()[:rows] <= (n_hist + 1) * 2.0 ** -24 * terms.abs().sum(0)[:rows]).all()
    xr = x.double().view(m, groups, -1)
    want = (xr / (xr.square().mean(dim=2, keepdim=True) + 1e-6).sqrt()).view(m, H) * gain.double()
    assert ((y.double() - want).abs()[:rows] <= (2.0 ** -8 + H * 2.0 ** -23) * want.abs()[:rows] + 1e-30).all()
    assert (x[rows:] == 9.0).all() and (y[rows:] == 9.0).all()
