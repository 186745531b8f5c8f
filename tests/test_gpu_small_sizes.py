"""Kernels that choose their form by how little there is to do, at the sizes where the choice changes."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# tiles of 32 with steps of 64 along K: one element, the edges, unaligned rows; and sizes on both sides of the 64x64 tiles' line
@pytest.mark.parametrize("m,n,k,pad", [(1, 2, 1, 0), (32, 32, 64, 0), (33, 34, 65, 3), (31, 30, 127, 1), (7, 256, 688, 0), (64, 1000, 256, 4),
                                       (1088, 1088, 40, 0), (1024, 1152, 33, 1), (1088, 1024, 20, 0)])
@pytest.mark.parametrize("epi", ["none", "bias_silu_res", "swiglu"])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_cuda_core_gemm(m, n, k, pad, epi, dtype):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(m + 7 * n + k)
    a = torch.randn(m, k + pad, generator=g, device="cuda").to(dtype)[:, :k]
    w = torch.randn(n, k + pad, generator=g, device="cuda").to(dtype)[:, :k]
    bias = torch.randn(n, generator=g, device="cuda").to(dtype)
    width = n // 2 if epi == "swiglu" else n
    res = torch.randn(m, width, generator=g, device="cuda")
    c = torch.full((m + 1, width), 5.0, device="cuda")
    live = max(1, m - 2)
    m_dev = torch.tensor([live], dtype=torch.int32, device="cuda")
    code = {"none": _lib.EPI_NONE, "bias_silu_res": _lib.EPI_BIAS_SILU_RES, "swiglu": _lib.EPI_SWIGLU}[epi]
    _lib.call("rd_gemm", _lib.dtype_code(dtype), _lib.F32, _lib.ptr(a), a.stride(0), _lib.ptr(w), w.stride(0), _lib.ptr(c), width,
              _lib.ptr(bias), _lib.ptr(res), width, m, _lib.ptr(m_dev), n, k, code, _lib.stream())
    acc = a.double() @ w.double().T
    slack = (k + 8) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)  # any order of k fp32 additions
    silu = torch.nn.functional.silu
    if epi == "bias_silu_res":
        want = silu(acc + bias.double()) + res.double()
        slack = 1.1 * slack + 2.0 ** -21 * (want.abs() + acc.abs() + bias.double().abs() + res.double().abs())
    elif epi == "swiglu":
        gate, up = acc[:, 0::2], acc[:, 1::2]
        want = silu(gate) * up
        slack = 1.1 * slack[:, 0::2] * up.abs() + (1.1 * slack[:, 0::2] + silu(gate).abs()) * slack[:, 1::2] + 2.0 ** -20 * (gate * up).abs()
    else:
        want = acc
    assert ((c.double()[:m] - want).abs() <= slack + 1e-30)[:live].all()
    assert (c[live:] == 5.0).all()


# rows on both sides of one 16-byte load per thread, and rows with fewer elements than are kept
@pytest.mark.parametrize("V", [3, 49, 50, 64, 250, 1000, 2047, 2048, 4095, 4096, 4104])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_vocab_topk_of_short_rows(V, dtype):
    from recurrent_drafting import modeling_drafter

    g = torch.Generator(device="cuda").manual_seed(V)
    rows = 5
    ld = (V + 7) // 8 * 8
    logits = (torch.randn(rows, ld, generator=g, device="cuda") * 3).to(dtype)[:, :V]
    if dtype == torch.float32:
        logits[2] = torch.round(logits[2])  # ties
    sp = modeling_drafter.vocab_topk(logits, modeling_drafter.new_sparse(rows, "cuda"), subtract_max=False, temperature=1.0)
    torch.cuda.synchronize()
    for r in range(rows):
        x = logits[r].double()
        order = sorted(range(V), key=lambda i: (-x[i].item(), i))
        k = min(modeling_drafter.TOP_K, V)
        kept = [i for i in order if x[i] >= x[order[k - 1]]]
        cnt = int(sp.cnt[r])
        assert cnt == min(len(kept), sp.idx.shape[1])
        assert sp.idx[r, :cnt].tolist() == kept[:cnt]
