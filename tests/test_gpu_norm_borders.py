"""Numbers of rows at which norms stop running their code ahead or holding their row in registers: a row's values have the same bits on both
sides, with and without a count on the device, complete and in shares, and hold against float64."""
import pytest
import torch

pytestmark = pytest.mark.gpu

ROOMS = [(1, False), (20, False), (21, False), (128, False), (129, False), (20, True), (21, True), (256, True), (257, True)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("H,K", [(4096, 0), (1032, 0), (4096, 4096), (2048, 5632)])  # K: of a projection in shares
def test_rmsnorm_on_both_sides(H, K, dtype):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(H + K)
    code = _lib.dtype_code(dtype)
    gain = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).to(dtype)
    rows = torch.randn(257, H, generator=g, device="cuda").to(dtype)
    share = torch.randn(8, 257, H, generator=g, device="cuda")
    seen = {}
    for m, counted in ROOMS:
        live = min(m, 19)
        md = torch.tensor([live], dtype=torch.int32, device="cuda") if counted else None
        x, y = rows[:m].clone(), torch.full((m, H), 9.0, dtype=dtype, device="cuda")
        if K:
            held = min(m, 256)
            n = _lib.load().rd_gemm_shares_bytes(m, H, K) // (4 * held * H)
            assert n > 1
            parts = share[:n, :held].contiguous()
            args = (code, _lib.ptr(x), _lib.ptr(x), _lib.ptr(parts), K, _lib.ptr(gain), _lib.ptr(y), m, _lib.ptr(md), H, 1e-6, _lib.stream())
            _lib.call("rd_rmsnorm_shares", *args)
            full = rows[:live].double() + share[:n, :live].double().sum(0)
            # n + 1 fp32 additions, and one rounding to the type: half a unit in the last of its 8 or 24 significant bits, of a value that is
            # at least the power of two below it, so 2^-8 or 2^-24 of the value
            size = rows[:live].double().abs() + share[:n, :live].double().abs().sum(0)
            half = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -24
            assert ((x[:live].double() - full).abs() <= half * full.abs() + (n + 1) * 2.0 ** -24 * size).all()
        else:
            _lib.call("rd_rmsnorm", code, _lib.ptr(x), _lib.ptr(gain), _lib.ptr(y), m, _lib.ptr(md), H, 1e-6, _lib.stream())
        torch.cuda.synchronize()
        f = x[:live].double()
        want = f / (f.square().mean(dim=1, keepdim=True) + 1e-6).sqrt() * gain.double()
        # two roundings to the type, and fp32 sums of H squares
        eps = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -23 + H * 2.0 ** -24
        assert ((y[:live].double() - want).abs() <= 2 * eps * want.abs() + 1e-30).all()
        if counted:
            assert (y[live:] == 9.0).all() and torch.equal(x[live:], rows[live:m])
        seen[m, counted] = (x[:live], y[:live])
    for out in seen.values():
        for a, b in zip(out, seen[20, False]):
            assert torch.equal(a, b[: a.shape[0]])


@pytest.mark.parametrize("K", [0, 4096])  # of a projection whose shares make the last stored row
@pytest.mark.parametrize("H,groups,n_hist", [(4096, 8, 9), (4096, 1, 1), (2048, 1, 5), (1024, 1, 1), (100, 4, 5)])
def test_stream_norm_on_both_sides(H, groups, n_hist, K):
    """148 blocks of 1024 threads run at the same time; narrower rows have fewer threads."""
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(H)
    rows = torch.randn(n_hist, 297, H, generator=g, device="cuda")
    residual, share = torch.randn(297, H, generator=g, device="cuda"), torch.randn(8, 256, H, generator=g, device="cuda")
    coeff = torch.randn(n_hist, generator=g, device="cuda") if n_hist > 1 else None
    gain = (1 + 0.1 * torch.randn(H, generator=g, device="cuda")).bfloat16()
    if K and H < 256:
        pytest.skip("matrices of fewer than 256 features are not cut")
    seen = []
    for m in (19, 20, 21, 148, 149, 296, 297):
        md = torch.tensor([19], dtype=torch.int32, device="cuda") if m > 256 else None  # more live rows are not in shares
        hist = rows.clone()
        x, y = torch.empty(m, H, device="cuda"), torch.empty(m, H, dtype=torch.bfloat16, device="cuda")
        for _ in range(2):  # one after the other: the second begins while the first runs
            if K:
                held = min(m, 256)
                n = _lib.load().rd_gemm_shares_bytes(m, H, K) // (4 * held * H)
                assert n > 1
                parts = share[:n, :held].contiguous()
                _lib.call("rd_stream_norm_shares", _lib.BF16, _lib.ptr(hist), hist.stride(0), _lib.ptr(coeff), n_hist, _lib.ptr(residual),
                          _lib.ptr(parts), K, _lib.ptr(x), _lib.ptr(gain), _lib.ptr(y), m, _lib.ptr(md), H, groups, 1e-6, _lib.stream())
            else:
                _lib.call("rd_stream_norm", _lib.BF16, None, None, 0.0, _lib.ptr(hist), hist.stride(0), _lib.ptr(coeff), n_hist, _lib.ptr(x),
                          _lib.ptr(gain), _lib.ptr(y), m, _lib.ptr(md), H, groups, 1e-6, _lib.stream())
        torch.cuda.synchronize()
        if K:
            full = residual[:19].double() + share[:n, :19].double().sum(0)
            size = residual[:19].double().abs() + share[:n, :19].double().abs().sum(0)
            assert ((hist[-1, :19].double() - full).abs() <= (n + 1) * 2.0 ** -24 * size).all()  # n fp32 additions
        terms = (coeff.double()[:, None, None] if coeff is not None else 1.0) * hist[:, :19].double()
        assert ((x[:19].double() - terms.sum(0)).abs() <= (n_hist + 1) * 2.0 ** -24 * terms.abs().sum(0)).all()
        seen.append((x[:19], y[:19]))
    for x, y in seen[:-1]:
        assert torch.equal(x, seen[0][0]) and torch.equal(y, seen[0][1])
    # from 297 tokens on the sums of squares run over another number of threads: a last bit of the scale, before the rounding to bf16
    x, y = seen[-1]
    assert torch.equal(x, seen[0][0]) and ((y.float() - seen[0][1].float()).abs() <= 2.0 ** -7 * seen[0][1].float().abs()).all()
