"""Explicit masks of every memory layout reach the kernels row by row: where rd_mask_bits would read is followed on the CPU, and on
the GPU the forward is compared with that of a plainly laid out mask."""
import ctypes

import pytest
import torch

from gpu_helpers import HD128_LLAMA, llama_config

LAYERS_1 = dict(HD128_LLAMA, num_hidden_layers=1, vocab_size=320)


def _masks(B, q_len, keys):
    """The same bool mask [B, q_len, keys] in several layouts."""
    g = torch.Generator().manual_seed(B + keys)
    m = torch.rand(B, q_len, keys, generator=g) < 0.5
    m[:, :, 0] = True
    wide = torch.zeros(B, q_len + 2, keys + 3, dtype=torch.bool)
    wide[:, 1 : 1 + q_len, 2 : 2 + keys] = m

    def laid_out(*order):
        """m in memory that is filled in this order of its dimensions (a fresh tensor: its strides are those of that order)."""
        t = torch.empty([m.shape[d] for d in order], dtype=torch.bool).copy_(m.permute(order))
        return t.permute([order.index(d) for d in range(3)])

    return m, {"plain": m.clone(), "queries first": laid_out(1, 0, 2), "keys before queries": laid_out(0, 2, 1), "keys first": laid_out(2, 0, 1),
               "part of a wider one": wide[:, 1 : 1 + q_len, 2 : 2 + keys], "bytes": m.to(torch.uint8) * 2}


LAYOUTS = ["plain", "queries first", "keys before queries", "keys first", "part of a wider one", "bytes"]
SIZES = [(3, 1, 70), (2, 5, 64), (1, 1, 9), (4, 1, 1), (1, 3, 130)]


@pytest.mark.parametrize("layout", LAYOUTS)
@pytest.mark.parametrize("B,q_len,keys", SIZES)
def test_rows_that_the_mask_kernel_reads(B, q_len, keys, layout, monkeypatch):
    from recurrent_drafting import _lib, modeling_llama

    keys = max(keys, q_len)
    want, masks = _masks(B, q_len, keys)
    seen = []

    def call(name, *args):
        if name == "rd_mask_bits":
            mask, ld, rows, cols = args[:4]
            assert (rows, cols) == (B * q_len, keys) and ld >= cols
            assert (rows - 1) * ld + cols <= B * q_len * keys  # inside the mask's bytes
            raw = ctypes.string_at(mask, (rows - 1) * ld + cols)
            seen.append(torch.tensor([[raw[r * ld + c] != 0 for c in range(cols)] for r in range(rows)]))

    class Library:  # plans and sizes; nothing is launched
        def __getattr__(self, name):
            return lambda *args: 1

    monkeypatch.setattr(_lib, "call", call)
    monkeypatch.setattr(_lib, "ptr", lambda t: None if t is None else t.data_ptr())
    monkeypatch.setattr(_lib, "stream", lambda: None)
    monkeypatch.setattr(_lib, "load", lambda: Library())
    llm = modeling_llama.LlamaForCausalLM(llama_config(LAYERS_1)).to(torch.bfloat16)
    cache = llm.new_cache(B, keys)
    cache.set_length(keys - q_len)
    llm.forward(torch.ones(B, q_len, dtype=torch.int64), masks[layout], torch.zeros(B, q_len, dtype=torch.int64), cache.sliced)
    assert len(seen) == 1 and torch.equal(seen[0], want.reshape(B * q_len, keys))


@pytest.mark.gpu
@pytest.mark.parametrize("layout", LAYOUTS[1:])
@pytest.mark.parametrize("B,q_len,keys", SIZES)
def test_forward_of_every_layout(B, q_len, keys, layout):
    import recurrent_drafting as rd

    keys = max(keys, q_len)
    _, masks = _masks(B, q_len, keys)
    llm = rd.modeling_llama.LlamaForCausalLM(llama_config(LAYERS_1)).to(device="cuda", dtype=torch.bfloat16).init_random(std=0.05, seed=3)
    ids = (torch.arange(B * q_len, device="cuda") % 300 + 1).view(B, q_len)
    pos = torch.arange(keys - q_len, keys, device="cuda").expand(B, q_len)
    out = []
    for name in ("plain", layout):
        cache = llm.new_cache(B, keys)
        g = torch.Generator(device="cuda").manual_seed(7)
        cache._cache.copy_(torch.randn(cache._cache.shape, generator=g, device="cuda"))
        cache.set_length(keys - q_len)
        mask = masks[name].cuda()
        # the copy to the device may lay the mask out anew: give it the strides that it had
        mask = torch.empty_strided(masks[name].shape, masks[name].stride(), dtype=mask.dtype, device="cuda").copy_(mask)
        out.append(llm.forward(ids, mask, pos, cache.sliced))
    assert torch.equal(out[0].logits, out[1].logits) and torch.equal(out[0].hidden_states, out[1].hidden_states)
