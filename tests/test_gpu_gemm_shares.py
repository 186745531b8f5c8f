"""Projections with a residual whose K is cut into shares for few rows, and the norms that add the shares up, against float64 at
the sizes where the cut begins, ends and changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

# (m_max, live rows or None, N, K, shares of a GPU with 74 CTA pairs): one row; the token block's edge; the last row count that is cut
# and the first that is not, also when only the device knows; features that are no multiple of a tile; a K whose k-blocks do not
# divide among the shares; a K too short to be cut
CASES = [
    (1, None, 4096, 11008, 4), (33, None, 2048, 5632, 8), (256, None, 4096, 4096, 4), (257, None, 4096, 4096, 4), (300, 256, 2048, 4104, 8),
    (300, 257, 2048, 4104, 8), (900, 45, 1064, 2048, 4), (1024, 256, 2048, 2048, 4),
    (1025, 9, 2048, 2048, 1), (31, None, 256, 1032, 2), (17, None, 512, 960, 1), (5, 0, 2048, 2048, 4),
]


def _inputs(m, n, k, dtype):
    g = torch.Generator(device="cuda").manual_seed(m * 31 + n + k)
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    w = (torch.randn(n, k, generator=g, device="cuda") / k ** 0.5).bfloat16()
    r = torch.randn(m, n, generator=g, device="cuda").to(dtype)
    gain = (1 + 0.1 * torch.randn(n, generator=g, device="cuda")).bfloat16()
    return a, w, r, gain


def _bounds(a, w, r, k):
    """float64 sums and what fp32 sums of k products in any order may be off by."""
    exact = r.double() + a.double() @ w.double().T
    size = r.double().abs() + a.double().abs() @ w.double().abs().T
    return exact, (k + 16) * 2.0 ** -24 * size


def _project(a, w, r, c, live, shares):
    from recurrent_drafting.modeling_common import Linear

    lin = Linear(w)
    m, n = a.shape[0], w.shape[0]
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    m_dev = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    room = shares * min(m, 256) * n if shares > 1 else 0
    assert lin.shares_bytes(m) == 4 * room
    # shares that are not written must not be read: NaN would show
    parts = torch.full((max(room, 4),), float("nan"), device="cuda")
    pending = lin.add_residual(a, c, r, m_dev, m, status, parts)
    assert (pending is not None) == (shares > 1)
    rows = m if live is None else live
    written = ~parts[:room].view(-1, min(m, 256), n).isnan() if room else None
    if room and rows <= 256:  # the live rows of every share, and nothing else
        assert written[:, :rows].all() and not written[:, rows:].any()
    elif room:  # C was formed whole
        assert not written.any()
    return lin, pending, m_dev, status


@pytest.mark.parametrize("m,live,n,k,shares", CASES)
def test_rmsnorm_of_shares(m, live, n, k, shares):
    from recurrent_drafting import _lib

    a, w, r, gain = _inputs(m, n, k, torch.bfloat16)
    h, y = r.clone(), torch.zeros_like(r)
    lin, pending, m_dev, status = _project(a, w, h, h, live, shares)
    if pending is None:
        _lib.call("rd_rmsnorm", _lib.BF16, _lib.ptr(h), _lib.ptr(gain), _lib.ptr(y), m, _lib.ptr(m_dev), n, 1e-6, _lib.stream())
    else:
        _lib.call("rd_rmsnorm_shares", _lib.BF16, _lib.ptr(h), _lib.ptr(pending.residual), _lib.ptr(pending.parts), pending.k,
                  _lib.ptr(gain), _lib.ptr(y), m, _lib.ptr(m_dev), n, 1e-6, _lib.stream())
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    rows = m if live is None else live
    exact, slack = _bounds(a, w, r, k)
    # one rounding to bf16: half a unit in the last place, 2^-8 of the value at most
    assert ((h.double() - exact).abs()[:rows] <= slack[:rows] + 2.0 ** -8 * exact.abs()[:rows]).all()
    assert torch.equal(h[rows:], r[rows:])
    x = h.double()
    norm = x / (x.square().mean(dim=1, keepdim=True) + 1e-6).sqrt()
    want = norm * gain.double()  # rounded to bf16 twice
    assert ((y.double() - want).abs()[:rows] <= 2.0 ** -7 * want.abs()[:rows] + 1e-6).all()


@pytest.mark.parametrize("m,live,n,k,shares", CASES)
@pytest.mark.parametrize("in_place", [True, False])
def test_stream_norm_of_shares(m, live, n, k, shares, in_place):
    from recurrent_drafting import _lib

    a, w, r, gain = _inputs(m, n, k, torch.float32)
    hist = torch.randn(3, m, n, device="cuda")
    first, coeff, x = hist.clone(), torch.tensor([0.5, -0.25, 1.25], device="cuda"), torch.zeros(m, n, device="cuda")
    if in_place:
        hist[2] = r
    residual = hist[2] if in_place else r.clone()
    y = torch.zeros(m, n, dtype=torch.bfloat16, device="cuda")
    lin, pending, m_dev, status = _project(a, w, residual, hist[2], live, shares)
    common = (_lib.ptr(x), _lib.ptr(gain), _lib.ptr(y), m, _lib.ptr(m_dev), n, 1, 1e-6, _lib.stream())
    if pending is None:
        _lib.call("rd_stream_norm", _lib.BF16, None, None, 0.0, _lib.ptr(hist), hist.stride(0), _lib.ptr(coeff), 3, *common)
    else:
        _lib.call("rd_stream_norm_shares", _lib.BF16, _lib.ptr(hist), hist.stride(0), _lib.ptr(coeff), 3, _lib.ptr(pending.residual),
                  _lib.ptr(pending.parts), pending.k, *common)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    rows = m if live is None else live
    exact, slack = _bounds(a, w, r, k)
    assert ((hist[2].double() - exact).abs()[:rows] <= slack[:rows]).all()
    assert torch.equal(hist[:2], first[:2])
    terms = [c * h.double() for c, h in zip(coeff.tolist(), hist)]
    assert ((x.double() - sum(terms)).abs()[:rows] <= 4 * 2.0 ** -24 * sum(t.abs() for t in terms)[:rows]).all()
    want = x.double() / (x.double().square().mean(dim=1, keepdim=True) + 1e-6).sqrt() * gain.double()
    assert ((y.double() - want).abs()[:rows] <= 2.0 ** -8 * want.abs()[:rows] + 1e-6).all()
