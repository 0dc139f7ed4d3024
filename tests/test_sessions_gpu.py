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


def design(name, kind, folder, dtype="float32"):
    """(model folder, vocabulary, plain logits of a token list) of one of a design's test models."""
    import importlib
    models, P = importlib.import_module(f"{name}_models"), importlib.import_module(f"plain_{name}")
    cfg = models.CONFIGS[kind]
    d = models.make_model(str(folder), cfg, seed=71)
    w, bf = models.load_weights(d, dtype == "bfloat16"), dtype == "bfloat16"
    if name in ("selovik", "setenex", "zadurax"):
        return d, cfg["vocab"], lambda tokens: P.forward(tokens, w, cfg, emulate_bf16=bf)
    return d, cfg["vocab"], lambda tokens: P.forward(cfg, w, tokens, emulate_bf16=bf)


def test_a_step_that_cannot_be_captured_runs_as_before(tmp_path, monkeypatch):
    """A recording that fails (no memory for the graph, say) leaves the session with steps launched one by one."""
    from nnis_b200 import LLM
    from nnis_b200.engine.decode import GraphDecoder
    d, vocab, plain = design("nafezen", "mixed", tmp_path)
    llm = LLM(d, dtype="float32", max_tokens=64 * 32, max_batch=2)
    tokens, calls = random_tokens(random.Random(5), 40, vocab), []

    def fails(self):
        calls.append(1)
        raise RuntimeError("planted")

    monkeypatch.setattr(GraphDecoder, "capture", fails)
    with pytest.warns(RuntimeWarning, match="planted"):
        rows = session_rows(llm, tokens, 9)
    check_logits(rows, plain(tokens)[8:], "float32", "session")
    assert len(calls) == 1  # (not tried again for every token)


def test_a_session_captures_its_step_once_that_pays(tmp_path):
    """The first five tokens are launched one by one; another session takes the graph that is there from its first on."""
    from nnis_b200 import LLM
    d, vocab, plain = design("tazadra", "wkv", tmp_path)
    llm = LLM(d, dtype="float32", max_tokens=64 * 32, max_batch=2)
    session, graphs = llm.new_session(), []
    tokens = random_tokens(random.Random(2), 20, vocab)
    rows = [session.prefill(tokens[:9])]
    for t in tokens[9:]:
        rows.append(session.decode_one(t))
        graphs.append(sum(dec.graph is not None for dec in llm.backend._decoders.values()))
    assert graphs == [0] * 5 + [1] * 6
    check_logits(np.stack(rows), plain(tokens)[8:], "float32", "session")
    other = llm.new_session()
    other.prefill(tokens[:9])
    replayed = []
    llm.backend._decoders[next(iter(llm.backend._decoders))].launch = lambda: replayed.append(1)
    other.decode_one(tokens[9])
    assert replayed == [1]


@pytest.mark.parametrize("name", ["nafezen", "sedopel", "selovik", "setenex", "tazadra", "zadurax"])
def test_long_sessions_of_every_design(name, tmp_path):
    """Two sessions that take turns, over the context where the next larger graph takes over: the states, caches and
    page tables that a replay reads are those of its own session."""
    from nnis_b200 import LLM
    d, vocab, plain = design(name, "mixed", tmp_path)
    llm = LLM(d, dtype="float32", max_tokens=64 * 32, max_batch=2)
    rng = random.Random(9)
    a, b = random_tokens(rng, 275, vocab), random_tokens(rng, 60, vocab)
    one, two = llm.new_session(), llm.new_session()
    rows = {0: [one.prefill(a[:240])], 1: [two.prefill(b[:30])]}
    for i in range(35):
        rows[0].append(one.decode_one(a[240 + i]))
        if i < 30:
            rows[1].append(two.decode_one(b[30 + i]))
    assert len(llm.backend._decoders) >= 2  # (contexts of up to 256 and of up to 512)
    check_logits(np.stack(rows[0]), plain(a)[239:], "float32", f"{name}: long session")
    check_logits(np.stack(rows[1]), plain(b)[29:], "float32", f"{name}: short session")
    one.close()
    two.close()
