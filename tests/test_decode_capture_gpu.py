"""Decode steps replayed from a CUDA graph against eager ones, with what a step keeps besides its tokens: seen tokens, recorded routing."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"
PROMPTS = [[5, 6, 7, 8, 9], [10, 11, 12], [20, 21, 22, 23, 24, 25, 26], [3, 4], [7, 7, 7, 7]]


def _generate(moe: bool, graph: bool, params, **kw):
    from verl_b200.models import FlatParams, ModelConfig
    from verl_b200.workers.rollout.native.engine import RolloutEngine

    cfg = ModelConfig(model_type="qwen3_moe" if moe else "qwen2", vocab_size=2048, hidden_size=512, intermediate_size=1024, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, head_dim=128, eos_token_id=-1, pad_token_id=0,
                      **(dict(num_experts=16, num_experts_per_tok=4, moe_intermediate_size=256, qk_norm=True) if moe else {}))
    P = FlatParams(cfg, dtype=torch.bfloat16, device=DEV)
    P.init_weights(seed=0, std=0.05)
    eng = RolloutEngine(cfg, P, max_num_seqs=3, max_model_len=64, block_size=16, num_blocks=32, sync_interval=3, use_cuda_graph=graph,
                        eos_token_id=-1, **kw)
    return [eng.generate(PROMPTS, params) for _ in range(2)]


@pytest.mark.parametrize("moe", [False, True])
def test_step_before_the_capture_marks_no_token_as_seen(moe):
    """A strong penalty makes a greedy sequence leave every token that it has seen: one marked by the warm-up step would be left at once."""
    from verl_b200.workers.rollout.native.engine import SamplingParams

    params = SamplingParams(temperature=0.0, max_tokens=9, repetition_penalty=50.0)
    captured, eager = _generate(moe, True, params), _generate(moe, False, params)
    for a, b in zip(captured, eager):
        assert [o.token_ids for o in a] == [o.token_ids for o in b]
        for x, y in zip(a, b):
            torch.testing.assert_close(torch.tensor(x.log_probs), torch.tensor(y.log_probs), rtol=0, atol=1e-4)


def test_recorded_routing_of_captured_steps():
    from verl_b200.workers.rollout.native.engine import SamplingParams

    params = SamplingParams(temperature=0.0, max_tokens=9)
    captured, eager = (_generate(True, graph, params, record_routing=True) for graph in (True, False))
    for a, b in zip(captured, eager):
        for x, y in zip(a, b):
            assert x.token_ids == y.token_ids
            assert torch.equal(x.extra_fields["routed_experts"], y.extra_fields["routed_experts"])
            assert x.extra_fields["routed_experts"].shape[0] == len(x.prompt_ids) + len(x.token_ids) - 1
