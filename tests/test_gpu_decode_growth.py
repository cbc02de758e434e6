"""Decode steps whose sequences grow past the length from which their attention runs other kernels: a graph holds for one choice."""
import pytest
import torch

from helpers import model_folder, random_tokens

pytestmark = pytest.mark.gpu


def logits_of(engine, length, steps, graphs, single):
    """The logits of ``steps`` single tokens behind four prompts of about ``length`` tokens, room for 600 reserved."""
    from gguf2bin_b200.engine import DecodeSession
    from gguf2bin_b200.engine.step import StepEntry
    from gguf2bin_b200.sampling import Sampler, SamplingParams
    seqs, out = [engine.open_sequence() for _ in range(4)], []
    try:
        for s in seqs:
            engine.cache.reserve(s, 600)
        engine.step([StepEntry(s, random_tokens("c", length - less, less), ()) for s, less in zip(seqs, (0, 10, 20, 34))])      # a multiple of 64 rows: no padding
        sampler = Sampler(engine.cache.seq_state, engine.device)
        sampler.seed([s.slot for s in seqs], range(4), 0)
        session = None if single else DecodeSession(engine, seqs, sampler, SamplingParams.plain(0.0), use_graph=graphs)
        for t in range(steps):
            tokens = random_tokens("c", 4, 100 + t)
            if single:
                out.append(engine.step([StepEntry(s, [x], (0,)) for s, x in zip(seqs, tokens)]).clone())
            else:
                session.set_tokens(tokens)
                session.run()
                out.append(session.logits.clone())
        engine.check()
    finally:
        for s in seqs:
            engine.close_sequence(s)
    return torch.stack(out)


@pytest.mark.parametrize("single", [False, True], ids=["session", "steps"])
def test_the_choice_goes_by_the_length_and_not_by_the_first_step_of_a_shape(single, monkeypatch):
    from gguf2bin_b200 import kernels_bf16
    from gguf2bin_b200.engine import Engine, Model
    monkeypatch.setattr(kernels_bf16, "DECODE_FINE_BELOW", 9)         # eight units: short chunks up to 256 keys
    model = Model.from_folder(model_folder("c", "bfloat16"), dtype="bfloat16")
    graphs, plain = Engine(model, 4096), Engine(model, 4096, step_graphs=False)
    lengths = [(240, 40), (304, 12), (96, 12), (224, 40)]             # across the border, behind it, before it, across it again
    for length, steps in lengths:
        got, ref = logits_of(graphs, length, steps, True, single), logits_of(plain, length, steps, False, single)
        assert torch.equal(got, ref), (length, (got - ref).abs().amax(dim=(1, 2)).tolist())
    captured = graphs.graph_captures
    assert captured >= 2 and plain.graph_captures == 0
    for length, steps in lengths[1:]:
        logits_of(graphs, length, steps, True, single)
    assert graphs.graph_captures - captured <= 3, "a choice that came back was captured again"      # prompts of a length that comes for the third time
