"""Captured steps of a hybrid of gated delta nets and gated attention: batches that fill neither their decode nor their prompt bucket
and graphs replayed with other state slots and lengths, against the same steps run eagerly.  States of sequences outside a batch
keep their bits."""
import numpy as np
import pytest
import torch

from xllm_b200.engine.llm_engine import EngineConfig, LLMEngine
from xllm_b200.models import ModelArgs

pytestmark = pytest.mark.gpu

# per step: (sequence, new tokens); a sequence's first appearance is the beginning of its prompt
STEPS = [
    [("a", 5), ("b", 1), ("c", 17)],                   # prompts, one of them a single token: it goes with the decode rows
    [("a", 1), ("b", 1), ("c", 1)],                    # three rows in a bucket of four
    [("c", 1), ("a", 1), ("b", 1)],                    # the same graph, other slots in its rows
    [("a", 1), ("d", 40), ("e", 1)],                   # decode rows, a portion and a fresh row
    [("d", 33), ("f", 50), ("b", 1)],                  # a portion that goes on beside one that begins
    [("f", 70), ("c", 1), ("d", 1), ("e", 1)],         # the same prompt bucket, other lengths, one portion instead of two
    [("f", 1)],
    [("e", 1), ("d", 1)],
]


def _engine(graph, dk, dv):
    args = ModelArgs(model_type="qwen3_next", vocab_size=1000, hidden_size=256, num_hidden_layers=4, num_attention_heads=4,
                     num_key_value_heads=2, head_dim=64, intermediate_size=512, qk_norm=True, partial_rotary_factor=0.25,
                     rope_theta=10000.0, max_position_embeddings=512, tie_word_embeddings=False,
                     extra=dict(linear_num_value_heads=4, linear_num_key_heads=2, linear_key_head_dim=dk,
                                linear_value_head_dim=dv, linear_conv_kernel_dim=4, full_attention_interval=4))
    engine = LLMEngine(EngineConfig(model="n", device="cuda:0", dtype="bfloat16", block_size=16, num_blocks=64, enable_graph=graph,
                                    max_seqs_per_batch=8, max_tokens_per_batch=256, max_model_len=512, max_running_seqs=8,
                                    enable_prefix_cache=False, random_weights=True), model_args=args)
    engine.model.init_random(std=0.05, seed=5)
    return engine


def _run(engine, tokens):
    """Per step: the logits by sequence and the states of all slots."""
    sched, runner, state, at, out = engine.scheduler, engine.runner, engine.model.state, {}, []
    for step in STEPS:
        new = [tokens[s][at.get(s, 0):at.get(s, 0) + n].tolist() for s, n in step]
        before = state.rec.clone(), state.conv.clone()
        batch = sched.schedule_replay([s for s, _ in step], new, [[n - 1] for _, n in step])
        order = [batch.request_id(i) for i in range(batch.n_seqs)]
        logits = runner.execute(batch, want_host=False, want_logits=True)
        slots = engine._slots_of(batch).tolist()
        sched.process_output(batch.batch_id, np.empty(0, dtype=np.int64), None)
        for s, n in step:
            at[s] = at.get(s, 0) + n
        others = [i for i in range(state.rec.shape[1]) if i not in slots]
        assert torch.equal(state.rec[:, others], before[0][:, others]) and torch.equal(state.conv[:, others], before[1][:, others])
        out.append(({s: logits[i].float().clone() for i, s in enumerate(order)},
                    {s: (state.rec[:, slots[i]].clone(), state.conv[:, slots[i]].float()) for i, s in enumerate(order)}))
    return out


@pytest.mark.parametrize("dk,dv", [(32, 32), (128, 64)])
def test_captured_steps_match_eager_ones(dk, dv):
    g = torch.Generator().manual_seed(dk)
    tokens = {s: torch.randint(0, 1000, (200,), generator=g) for s in "abcdef"}
    eager = _engine(False, dk, dv)
    want = _run(eager, tokens)
    engine = _engine(True, dk, dv)
    engine.model.copy_params_from(dict(eager.model.named_params()))
    got = _run(engine, tokens)
    assert engine.runner.graph_replays == len(STEPS) > len(engine.runner.graphs)       # all of them, some more than once
    for step, (a, b) in enumerate(zip(want, got)):
        for s in a[0]:
            # bf16: products of other numbers of rows add in another order
            assert (b[0][s] - a[0][s]).norm() <= 0.03 * a[0][s].norm(), (step, s)
            for x, y in zip(a[1][s], b[1][s]):
                assert (y - x).norm() <= 0.03 * x.norm(), (step, s)
