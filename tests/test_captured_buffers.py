"""Captured decode steps keep the device memory that they address: a request whose steps are replayed from graphs goes on with the
same tokens after other requests have made the models replace their scratch memory and rotary tables."""
import pytest
import torch

from gpu_helpers import build_models, llama_config

# grouped heads and few of them: one-token steps and drafts of a small batch cut the keys into shares
LLAMA = dict(hidden_size=512, num_attention_heads=4, num_key_value_heads=2, num_hidden_layers=2, intermediate_size=704, vocab_size=1024,
             rms_norm_eps=1e-6, rope_theta=10000.0)
DRAFTER = dict(vocab_size=1024, hidden_size=512, exit_dim=1024, num_draft_layers=1, rnn=True)


def test_llama_names_the_memory_that_it_may_replace():
    from recurrent_drafting import modeling_llama

    llm = modeling_llama.LlamaForCausalLM(llama_config(LLAMA)).to(torch.bfloat16)
    assert llm.held_buffers() == []
    cos, sin = llm._rope_tables(64)
    llm._attn_split_ws, llm._head_ws = torch.zeros(8, dtype=torch.uint8), torch.zeros(4)
    held = llm.held_buffers()
    for t in (cos, sin, llm._attn_split_ws, llm._head_ws):
        assert any(t is h for h in held)


def _disturb(llm, drafter):
    """Requests that need more of everything; then what they freed is given to others and overwritten."""
    import recurrent_drafting as rd

    before = [t.data_ptr() for t in llm.held_buffers()]
    ids = torch.arange(24 * 40, device="cuda").view(24, 40) % 1000 + 1
    cache = llm.new_cache(4, 5000)
    cache.set_length(4400)
    mask = torch.ones(4, 60, 4460, dtype=torch.bool, device="cuda")
    llm.forward(ids.view(-1)[:240].view(4, 60), mask, torch.arange(4400, 4460, device="cuda").expand(4, 60), cache.sliced)
    model = rd.RecurrentDrafting(llm, drafter, cuda_graphs=False)
    for width in range(4, 10):  # more shapes than the drafter keeps
        next(iter(model.generate(rd.stats.Ledger(), ids, 60, rd.modeling_drafter.BeamShape(width, 4), rd.SamplingArgs(1.0, True),
                                 rd.SpecialTokens(0, None))))
    assert not set(before) & {t.data_ptr() for t in llm.held_buffers()}  # all of it was replaced
    torch.cuda.synchronize()
    return [torch.full((n,), 0xFF, dtype=torch.uint8, device="cuda") for n in [1 << k for k in range(9, 24)] * 4]


def _steps(kind, llm, drafter, greedy):
    import recurrent_drafting as rd

    ids = (torch.arange(2 * 30, device="cuda") * 7 % 1000 + 1).view(2, 30)
    args = rd.SamplingArgs(1.0, True) if greedy else rd.SamplingArgs(0.8, False)
    if kind == "autoregressive":
        return rd.autoregressive.generate(llm, ids, 700, rd.SpecialTokens(0, None), args, cuda_graphs=True)
    return rd.RecurrentDrafting(llm, drafter, cuda_graphs=True).generate(
        rd.stats.Ledger(), ids, 700, rd.modeling_drafter.BeamShape(6, 4), args, rd.SpecialTokens(0, None))


@pytest.mark.gpu
@pytest.mark.parametrize("greedy", [True, False])
@pytest.mark.parametrize("kind", ["autoregressive", "speculative"])
def test_replayed_steps_after_other_requests(kind, greedy, monkeypatch):
    import recurrent_drafting as rd

    captured = []
    name = "DecodeGraphs" if kind == "autoregressive" else "_StepGraphs"
    home = rd.autoregressive if kind == "autoregressive" else rd.recurrent_drafting
    graphs = getattr(home, name)
    monkeypatch.setattr(home, name, lambda *a: captured.append(graphs(*a)) or captured[-1])
    runs = []
    for disturbed in (False, True):
        # models of their own for each run, so that both start with nothing held
        llm, drafter, _, _ = build_models(LLAMA, DRAFTER, 41, dtype=torch.bfloat16)
        outs, keep = [], []
        steps = _steps(kind, llm, drafter, greedy)
        for n in range(12):
            torch.manual_seed(n)  # of the step's own uniforms, whatever was drawn in between
            outs.append(next(steps).clone())
            if disturbed and n == 5:
                assert len(captured) == 2 and captured[-1].buffers is not None
                held = {t.data_ptr() for t in llm.held_buffers()}
                assert llm._attn_split_ws is not None  # the keys were in shares
                keep = _disturb(llm, drafter)
                flat = [b for part in captured[-1].buffers if isinstance(part, list) for b in part]
                assert held <= {t.data_ptr() for t in flat}  # and is still held
        runs.append(outs)
        del keep
    for a, b in zip(*runs):
        assert torch.equal(a, b)
