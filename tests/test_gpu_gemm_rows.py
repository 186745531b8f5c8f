"""Projections of few tokens (rd_gemm_few_rows) against float64 where the size of a slab, the k-blocks of a load and the token boxes
change, launched in order and ahead of the dependency wait, and the forms of their epilogues against the kernel that serves more
tokens."""
import pytest
import torch


# slabs of 32, 64, 128, 160 .. 256 rows end at 148 slabs of each; narrow ones serve fewer tokens; K in whole k-blocks of 64
@pytest.mark.parametrize("m,n,k,served", [(64, 4736, 64, 1), (65, 4736, 64, 0), (128, 4737, 64, 1), (129, 9472, 64, 0), (256, 9473, 64, 1),
                                          (257, 9473, 64, 0), (1, 37888, 64, 1), (1, 37889, 64, 0), (1, 4096, 4104, 0), (1, 8, 64, 1)])
def test_what_is_served(m, n, k, served):
    from recurrent_drafting import _lib

    assert _lib.load().rd_gemm_few_rows(m, n, k) == served


def _linear(n, k, g, bias=False):
    from recurrent_drafting.modeling_common import Linear

    w = (torch.randn(n, k, generator=g, device="cuda") / k ** 0.5).bfloat16()
    return Linear(w, torch.randn(n, generator=g, device="cuda").bfloat16() if bias else None)


# (rows, live rows or None, features, K): the token boxes' edges; one slab and the last slab's ragged end; both sides of a change of
# slab; fewer steps than the ring has stages, a last step that reaches past K, many turns of the ring
SIZES = [(1, None, 32, 64), (16, None, 200, 128), (17, None, 4736, 192), (32, 5, 4736, 4096), (33, None, 4097, 704), (64, 63, 4736, 1088),
         (1, None, 4737, 64), (64, None, 9472, 320), (65, None, 6176, 1024), (128, 97, 9470, 192), (128, 0, 4738, 256),
         (16, None, 9473, 4096), (129, None, 12288, 192), (256, 241, 18944, 128), (256, 100, 18944, 1024), (225, 112, 22016, 2048),
         (1, None, 18945, 4096), (256, None, 22016, 192), (24, None, 26000, 576), (160, None, 32000, 128), (33, 32, 37888, 64)]


@pytest.mark.gpu
@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("m,live,n,k", SIZES)
def test_sums_and_residual(m, live, n, k, early):
    from recurrent_drafting import _lib

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    lin = _linear(n, k, g)
    assert _lib.load().rd_gemm_few_rows(m, n, k) == 1
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    r = torch.randn(m, n, generator=g, device="cuda")
    rows = m if live is None else live
    m_dev = None if live is None else torch.tensor([live], dtype=torch.int32, device="cuda")
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    # rows that end off a 16-byte boundary take plain stores
    outs = [torch.full((m, n + 8 - n % 4), 5.0, device="cuda")[:, :n] for _ in range(3)]
    for c in outs:  # one after the other: with early weights a launch begins while the one before runs
        lin(a, c, _lib.EPI_RES, residual=r, m_dev=m_dev, status=status, early=early)
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    exact = r.double() + a.double() @ lin.weight.double().T
    slack = (k + 16) * 2.0 ** -24 * (r.double().abs() + a.double().abs() @ lin.weight.double().abs().T)  # any order of k fp32 additions
    for c in outs:
        assert ((c.double() - exact).abs()[:rows] <= slack[:rows]).all()
        assert (c[rows:] == 5.0).all()
        assert torch.equal(c, outs[0])


@pytest.mark.gpu
@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("m,n", [(1, 4096), (40, 2048), (7, 8192), (100, 8192), (3, 12288), (130, 16512), (24, 22016), (225, 20000), (5, 32000)])
def test_epilogues(m, n, early):
    """Bias, SiLU, gated units, xIELU, split, slice maxima and arg-max: against fp32 on the same operands, rounded once."""
    from recurrent_drafting import _lib

    k = 512
    g = torch.Generator(device="cuda").manual_seed(m + n)
    lin, head = _linear(n, k, g, bias=True), _linear(n, k, g)
    assert _lib.load().rd_gemm_few_rows(m, n, k) == 1
    a = torch.randn(m, k, generator=g, device="cuda").bfloat16()
    r = torch.randn(m, n, generator=g, device="cuda").bfloat16()
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    acc, bias = a.float() @ lin.weight.float().T, lin.bias.float()
    gate, up = acc[:, 0::2], acc[:, 1::2]
    silu = torch.nn.functional.silu

    def out(width=n, dtype=torch.bfloat16):
        return torch.full((m, width), 7.0, dtype=dtype, device="cuda")

    def check(got, want):
        # one rounding to bf16 (2^-9) of fp32 sums of 512 products and approximate exponentials
        assert ((got.float() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-4 * want.abs().max()).all()

    for epi, want in ((_lib.EPI_BIAS, acc + bias), (_lib.EPI_BIAS_SILU, silu(acc + bias)), (_lib.EPI_BIAS_SILU_RES, silu(acc + bias) + r.float())):
        c = out()
        lin(a, c, epi, residual=r if epi == _lib.EPI_BIAS_SILU_RES else None, status=status, early=early)
        check(c, want)
    c = out(n // 2)
    lin(a, c, _lib.EPI_SWIGLU, status=status, early=early)
    check(c, silu(gate) * up)
    lin.clamped_glu(a, c, 0.5, 1.7, status=status, early=early)
    check(c, gate.clamp(max=0.5) * torch.sigmoid(1.7 * gate.clamp(max=0.5)) * (up.clamp(-0.5, 0.5) + 1.0))
    c = out()
    lin.xielu(a, c, 0.8, 0.6, status=status, early=early)
    low = acc.clamp(max=0.0)
    check(c, torch.where(acc > 0, 0.8 * acc * acc, 0.6 * (torch.expm1(low) - low)) + 0.5 * acc)
    at = n // 64 * 32
    lo, hi = out(at), out(n - at, torch.float32)
    lin.split(a, lo, hi, at, status=status, early=early)
    check(lo, acc[:, :at])
    assert ((hi - acc[:, at:]).abs() <= 1e-4 * acc.abs().max()).all()
    logits, plain = out(dtype=torch.float32), out(dtype=torch.float32)
    smax = torch.zeros(n // 32, (m + 31) // 32 * 32, device="cuda")
    assert head.with_slice_max(a, logits, smax, status=status, early=early)
    head(a, plain, status=status)
    assert torch.equal(logits, plain) and torch.equal(smax[:, :m], plain.view(m, n // 32, 32).amax(dim=2).T)
    tok = torch.zeros(m, dtype=torch.int32, device="cuda")
    head.argmax(a, tok, torch.empty(_lib.load().rd_gemm_argmax_workspace_bytes(m, n), dtype=torch.uint8, device="cuda"), None, m, status)
    assert torch.equal(tok.long(), plain.argmax(dim=1))
    assert int(status.item()) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("early", [False, True])
@pytest.mark.parametrize("kind", ["qkv", "qkvg", "norm"])
@pytest.mark.parametrize("m,live", [(1, None), (33, None), (64, 40)])
@pytest.mark.parametrize("nh,nkv", [(8, 2), (32, 8), (32, 32)])  # heads cut among 4 and 2 CTAs of a cluster, and whole
def test_rotary_heads(nh, nkv, m, live, kind, early):
    """Rotation, head norm, gates and cache append against the kernel for more tokens: a row's values may differ by the rounding to bf16
    where the two add up in another order."""
    from recurrent_drafting import _lib
    from recurrent_drafting.modeling_llama import rope_tables

    k, max_len, B, n_pos = 512, 90, 2, 128
    g = torch.Generator(device="cuda").manual_seed(nh + nkv + m)
    heads = nh + (1 if kind == "norm" else 2) * nkv
    lin = _linear(heads * 128 + (nh if kind == "qkvg" else 0), k, g)
    served = [_lib.load().rd_gemm_few_rows(rows, lin.weight.shape[0], k) for rows in (m, 300)]
    assert served == [1, 0]
    cos, sin = rope_tables(128, n_pos, 10000.0, "cuda")
    rows = m if live is None else live
    i32 = dict(dtype=torch.int32, device="cuda")
    a = torch.randn(300, k, generator=g, device="cuda").bfloat16()
    tok_row = torch.arange(300, **i32) % B
    tok_slot = torch.arange(300, **i32) % max_len
    tok_pos = torch.randint(0, n_pos, (300,), generator=g, device="cuda", dtype=torch.int32)
    status = torch.zeros(1, **i32)
    got = []
    for cap, m_dev in ((m, None if live is None else torch.tensor([live], **i32)), (300, torch.tensor([rows], **i32))):
        q = torch.full((300, nh * 128), 5.0, dtype=torch.bfloat16, device="cuda")
        kc, vc = (torch.full((B, nkv, max_len, 128), 5.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        gate = torch.full((300, nh), 5.0, dtype=torch.bfloat16, device="cuda")
        args = (a[:cap], q, kc, vc)
        toks = (tok_row, tok_pos, tok_slot, cos, sin, nh, nkv)
        if kind == "qkv":
            lin.qkv_rope(*args, *toks, 128, m_dev, cap, status, early=early)
        elif kind == "qkvg":
            lin.qkvg_rope(*args, gate, *toks, 64, m_dev, cap, status, early=early)
        else:
            lin.qk_rope_norm(*args, *toks, 128, 1e-6, m_dev, cap, status, early=early)
        got.append((q, kc, vc, gate))
    torch.cuda.synchronize()
    assert int(status.item()) == 0
    for x, y in zip(*got):
        assert (x == 5.0).equal(y == 5.0)  # the same elements are written
        # two bf16 roundings on the way, of the product and of what it is turned into
        assert ((x.float() - y.float()).abs() <= 2.0 ** -7 * y.float().abs() + 2.0 ** -8 * 4).all()
        assert ((x.float() - y.float()).norm() <= 2.0 ** -8 * y.float().norm())


@pytest.mark.gpu
def test_weights_written_just_before_a_step():
    """Weights that the stream's earlier work writes are those that a step reads, however early its kernels ask for them."""
    from recurrent_drafting import _lib
    from gpu_helpers import llama_config
    import recurrent_drafting as rd

    llm = rd.modeling_llama.LlamaForCausalLM(llama_config(dict(
        hidden_size=1024, num_attention_heads=8, num_key_value_heads=2, num_hidden_layers=2, intermediate_size=2816, vocab_size=1024,
        rms_norm_eps=1e-6, rope_theta=10000.0))).to(device="cuda", dtype=torch.bfloat16)
    llm.init_random(std=0.05, seed=1)
    i32 = dict(dtype=torch.int32, device="cuda")
    sets = [[p + 0.01 * (i + 1) * torch.randn_like(p) for p in llm.parameters()] for i in range(2)]
    cache, one = llm.new_cache(1, 64), torch.zeros(1, **i32)
    llm.gemm_status = torch.zeros(1, **i32)
    ids = torch.tensor([3], device="cuda")

    def step(values, wait):
        with torch.inference_mode():
            for p, v in zip(llm.parameters(), values):
                p.copy_(v)
            if wait:
                torch.cuda.synchronize()
            return llm.backbone(llm.workspace(1, 1), cache.storage, 1, None, ids, one, one, one, torch.tensor([0, 1], **i32), one, one, 1, 1, 64,
                                _lib.ATTN_CAUSAL, n_pos=128).clone()

    want = [step(v, True) for v in sets]
    assert not torch.equal(*want)
    for _ in range(20):
        for v, w in zip(sets, want):
            assert torch.equal(step(v, False), w)
