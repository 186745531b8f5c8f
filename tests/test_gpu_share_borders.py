"""bf16 models on both sides of the row counts at which projections with a residual change the order of their sums: 256 live rows and
a capacity of 1024.  The hidden states of a token must agree within the rounding of what differs, and its greedy token must be
the same where the margin is clear."""
import pytest
import torch

pytestmark = pytest.mark.gpu

H, FF, VOCAB = 512, 2048, 1024


def _model(design):
    import recurrent_drafting as rd
    from gpu_helpers import llama_config

    if design == "llama":
        llm = rd.modeling_llama.LlamaForCausalLM(llama_config(dict(
            hidden_size=H, num_attention_heads=4, num_key_value_heads=2, num_hidden_layers=2, intermediate_size=FF, vocab_size=VOCAB,
            rms_norm_eps=1e-6, rope_theta=10000.0))).to(device="cuda", dtype=torch.bfloat16)
    else:
        import nulunex_builders as nb

        cfg = nb.config([nb.attention(heads=4, kv_heads=2, dim=128, rot=128, scale=128 ** -0.5, chunk=128, ff=FF, limit=7.0),
                         nb.latent(heads=4, dim=128, rot_dim=64, vdim=128, rank=256, window=128, scale=192 ** -0.5, ff=FF, limit=7.0)],
                        vocab=VOCAB, width=H, eps=1e-6)
        llm = rd.registry.new_model(cfg, torch.bfloat16, "cuda")
    llm.init_random(std=0.05, seed=5)
    embed = llm.get_input_embeddings().weight
    g = torch.Generator(device="cuda").manual_seed(9)
    embed.copy_(torch.randn(VOCAB, H, generator=g, device="cuda") * 2)
    llm.lm_head.weight.copy_(torch.roll(embed, 1, dims=0) * 0.02)  # token t is followed by t + 1
    llm._invalidate()
    return llm


def _forward(llm, live, capacity):
    """Final hidden states and tokens of the first 200 of `live` tokens of a prompt, run with room for `capacity`."""
    from recurrent_drafting import _lib

    i32 = dict(dtype=torch.int32, device="cuda")
    ids = torch.arange(capacity, device="cuda") * 37 % (VOCAB - 1) + 1
    at = torch.arange(capacity, **i32) % live
    cache = llm.new_cache(1, 1200)
    status = llm.gemm_status = torch.zeros(1, **i32)
    ws = llm.workspace(capacity, 200)
    assert ws["parts"].numel() > 0
    m_dev = torch.tensor([live], **i32)
    with torch.inference_mode():
        hidden = llm.backbone(ws, cache.storage, capacity, m_dev, ids, torch.zeros(capacity, **i32), at, at, torch.tensor([0, live], **i32),
                              torch.zeros(1, **i32), torch.zeros(1, **i32), 1, capacity, 1100, _lib.ATTN_CAUSAL, n_pos=1300)[:200].clone()
        logits = llm.lm_logits(hidden, ws["logits"]).clone()
    assert int(status.item()) == 0
    return hidden.double(), logits.double()


@pytest.mark.parametrize("design", ["llama", "nulunex"])
def test_tokens_on_both_sides_of_a_border(design):
    llm = _model(design)
    base, want = _forward(llm, 256, 1024)
    head = llm.lm_head.weight.double()
    for live, capacity in ((255, 1024), (257, 1024), (256, 1025), (300, 300), (256, 256), (200, 200), (200, 1100)):
        hidden, logits = _forward(llm, live, capacity)
        # Llama's stream is rounded to bf16 after each of 4 projections, and so is everything that the projections read: half a unit in
        # the last place (2^-9 of the norm) for each of 4 projections and 4 of their inputs, and as much again for what layer 2 makes of it
        off = (hidden - base).norm(dim=1) / base.norm(dim=1)
        assert off.max() <= 16 * 2.0 ** -9, (live, capacity, off.max())
        slack = 2 * head.norm(dim=1).max() * (hidden - base).norm(dim=1)  # two logits may each move by this
        top = want.topk(2, dim=1).values
        clear = top[:, 0] - top[:, 1] > slack
        assert clear.sum() >= 190
        assert torch.equal(logits.argmax(1)[clear], want.argmax(1)[clear])
