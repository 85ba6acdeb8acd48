"""What a step hands out is the caller's tensor: reshaping it in place does not reach later steps."""

import pytest
import torch

import tiny

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_reshaped_logits_do_not_reach_the_next_step(tmp_path, dtype):
    from freetoken_b200.engine import Engine, EngineArgs, StepEntry
    tiny.write_tiny(str(tmp_path), "A")
    vocab = tiny.TINY["A"]["vocab_size"]
    tokens = tiny.tokens(3, 12, vocab)
    runs = []
    for reshape in (False, True):
        engine = Engine.from_folder(str(tmp_path), EngineArgs(dtype=dtype, page_size=4, num_pages=16, max_running_requests=2))
        rows = []
        for i in range(0, 12, 1):                        # one key, run eagerly, captured and replayed
            logits = engine.step([StepEntry("r", [tokens[i]], [0])])
            assert logits.shape == (1, vocab)
            rows.append(logits.clone())
            if reshape:
                logits.unsqueeze_(0).transpose_(0, 2)
        runs.append(torch.cat(rows))
    assert torch.equal(*runs)
