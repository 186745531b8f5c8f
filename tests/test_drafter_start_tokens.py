"""The start tokens that a beam search hands to its kernels, which read one for each row of the batch: from the caller's one or many, whole;
any other number is refused before a launch reads them."""
import pytest
import torch

import model_builders as mb


@pytest.fixture
def start_of(monkeypatch):
    from recurrent_drafting import _lib, configuration_drafter, modeling_drafter

    calls = []
    monkeypatch.setattr(_lib, "call", lambda name, *args: calls.append((name, args)))
    monkeypatch.setattr(_lib, "stream", lambda: 0)
    monkeypatch.setattr(_lib, "ptr", lambda t: t)  # the tensor itself: nothing is launched
    drafter = modeling_drafter.Drafter(configuration_drafter.DrafterConfig(**mb.NANO_DRAFTER))
    embed = torch.nn.Embedding(drafter.config.vocab_size, drafter.config.hidden_size)

    def run(tokens, batch):
        calls.clear()
        drafter.beam_search_sparse(torch.zeros(batch, drafter.config.hidden_size), tokens, embed, modeling_drafter.BeamShape(4, 3))
        (args,) = [args for name, args in calls if name == "rd_drafter_begin"]
        return args[2]

    run.calls = calls
    return run


@pytest.mark.parametrize("tokens,batch,want", [
    (torch.tensor([7]), 1, [7]), (torch.tensor([7]), 3, [7, 7, 7]), (torch.tensor([4, 9, 2]), 3, [4, 9, 2]),
    (torch.arange(6)[::2], 3, [0, 2, 4]), (torch.tensor([5]).expand(3), 3, [5, 5, 5])])
def test_one_token_for_each_row(start_of, tokens, batch, want):
    got = start_of(tokens, batch)
    assert got.is_contiguous() and got.untyped_storage().nbytes() >= 8 * batch
    assert got.tolist() == want


@pytest.mark.parametrize("n,batch", [(2, 3), (4, 3), (2, 1), (0, 2)])
def test_another_number_is_refused(start_of, n, batch):
    with pytest.raises(RuntimeError):
        start_of(torch.arange(n), batch)
    assert not start_of.calls
