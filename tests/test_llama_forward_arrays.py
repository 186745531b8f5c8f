"""The arrays that the reference-style forward hands to the kernels: whole, contiguous, one element a token, whatever the batch and however the
caller's ids and positions are laid out."""
import pytest
import torch

from gpu_helpers import HD128_LLAMA, llama_config

MODEL = dict(HD128_LLAMA, num_hidden_layers=1, vocab_size=320)


@pytest.mark.parametrize("B,q_len", [(1, 1), (1, 3), (2, 1), (3, 4)])
@pytest.mark.parametrize("expanded", [False, True])
def test_arrays_of_a_forward(B, q_len, expanded, monkeypatch):
    from recurrent_drafting import _lib, modeling_llama

    past, seen = 5, {}
    names = ("tok_ids", "tok_row", "tok_pos", "tok_slot", "row_start", "kv_begin", "base_len")

    def backbone(ws, cache_tensor, m_max, m_dev, *arrays, **kw):
        seen.update(zip(names, arrays))
        return ws["hidden"]

    class Library:  # sizes; nothing is launched
        def __getattr__(self, name):
            return lambda *args: 0

    monkeypatch.setattr(_lib, "call", lambda *args: None)
    monkeypatch.setattr(_lib, "load", lambda: Library())
    llm = modeling_llama.LlamaForCausalLM(llama_config(MODEL)).to(torch.bfloat16)
    monkeypatch.setattr(llm, "backbone", backbone)
    monkeypatch.setattr(llm, "lm_logits", lambda hidden, logits: logits)
    cache = llm.new_cache(B, past + q_len)
    cache.set_length(past)
    ids, pos = torch.arange(B * q_len).view(B, q_len), torch.arange(past, past + q_len).repeat(B, 1)
    if expanded:
        ids, pos = torch.full((1, 1), 7).expand(B, q_len), torch.full((1, 1), past).expand(B, q_len)
    llm.forward(ids, torch.ones(B, q_len, past + q_len, dtype=torch.bool), pos, cache.sliced)
    want = dict(tok_ids=ids.reshape(-1), tok_pos=pos.reshape(-1), tok_row=torch.arange(B).repeat_interleave(q_len),
                tok_slot=torch.arange(past, past + q_len).repeat(B), row_start=torch.arange(B + 1) * q_len, kv_begin=torch.zeros(B),
                base_len=torch.full((B,), past))
    for name, t in seen.items():
        assert t.is_contiguous() and t.untyped_storage().nbytes() >= t.numel() * t.element_size(), name
        assert t.tolist() == want[name].tolist(), name
