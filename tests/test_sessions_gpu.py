"""Sessions past their first tokens, where the decode step is a captured graph: the same logits as the plain
implementation before and after the capture."""
import random

import numpy as np
import pytest
import torch

from helpers import check_logits, random_tokens

pytestmark = pytest.mark.gpu


def session_rows(llm, tokens, prompt):
    """The logits of positions prompt - 1 .. of ``tokens``: a prompt, then token by token."""
    session = llm.new_session()
    rows = [session.prefill(tokens[:prompt])]
    rows += [session.decode_one(t) for t in tokens[prompt:]]
    session.close()
    return np.stack(rows)


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_a_model_with_one_sublayer(dtype, tmp_path):
    """One layer without a feed-forward: its block takes its two stream buffers in turn, an odd number of times a step,
    and the recording of a step is a second run of the same step."""
    import plain_tazadra as P
    from nnis_b200 import LLM
    from nnis_b200.engine import SequenceStep
    from tazadra_models import ONLY_MAMBA, load_weights, make_model
    d = make_model(str(tmp_path), ONLY_MAMBA, seed=61)
    llm = LLM(d, dtype=dtype, max_tokens=64 * 32, max_batch=2)
    w, bf = load_weights(d, dtype == "bfloat16"), dtype == "bfloat16"
    tokens = random_tokens(random.Random(3), 300, ONLY_MAMBA["vocab"])
    want = P.forward(ONLY_MAMBA, w, tokens, emulate_bf16=bf)
    check_logits(session_rows(llm, tokens[:30], 9), want[8:30], dtype, "session")
    engine = llm.engine
    for _ in range(3):  # a prompt of one shape: launched one by one, recorded, replayed
        slot = engine.acquire_slot()
        got = engine.step([SequenceStep(slot, tokens, [0, 150, 299])]).cpu().numpy()
        engine.release_slot(slot)
        check_logits(got, want[[0, 150, 299]], dtype, "prompt")
