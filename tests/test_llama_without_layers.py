"""A Llama without layers: embedding, norm and head."""
import pytest
import torch

from gpu_helpers import HD128_LLAMA, llama_config

CONFIG = dict(HD128_LLAMA, num_hidden_layers=0, vocab_size=320)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_workspace(dtype):
    from recurrent_drafting import modeling_llama

    ws = modeling_llama.LlamaForCausalLM(llama_config(CONFIG)).to(dtype).workspace(5, 3)
    assert ws["h"].shape == (5, 512) and ws["logits"].shape == (3, 320) and ws["parts"].numel() == 0


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_logits(dtype):
    import recurrent_drafting as rd

    llm = rd.modeling_llama.LlamaForCausalLM(llama_config(CONFIG)).to(device="cuda", dtype=dtype).init_random(std=0.05, seed=3)
    ids = torch.arange(1, 7, device="cuda").view(2, 3)
    cache = llm.new_cache(2, 3)
    view = rd.kv_cache.Cache(2, 3, 1, 4, 128, dtype, torch.device("cuda"))  # forward() finds the cache through a layer's view
    assert len(cache.sliced) == 0
    out = llm.forward(ids, torch.ones(2, 3, 3, dtype=torch.bool, device="cuda").tril(), torch.arange(3, device="cuda").expand(2, 3), view.sliced)
    x = llm.model.embed_tokens.weight[ids].double()
    x = (x * torch.rsqrt(x.square().mean(-1, keepdim=True) + 1e-6)).to(dtype).double()
    want = x @ llm.lm_head.weight.double().T
    # one rounding to the dtype of each row, sums of 512 products in fp32
    step = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -20
    assert ((out.logits.double() - want).abs() <= step * (x.abs() @ llm.lm_head.weight.double().abs().T)).all()
