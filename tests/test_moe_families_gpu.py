"""Scoring and updates of a mixture-of-experts model agree to the bit, although passes that keep nothing run the expert products on the tile
that their rows fill: a last bit in front of a router would turn into another choice of experts."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _model(recompute="none"):
    from verl_b200.models import DecoderModel, FlatParams, ModelConfig

    cfg = ModelConfig(model_type="qwen3_moe", vocab_size=2048, hidden_size=512, intermediate_size=1024, num_hidden_layers=2, num_attention_heads=4,
                      num_key_value_heads=2, head_dim=128, num_experts=16, num_experts_per_tok=4, moe_intermediate_size=320, qk_norm=True)
    params = FlatParams(cfg, dtype=torch.bfloat16, device=DEV, with_main_grad=True)
    params.init_weights(seed=0, std=0.05)
    return DecoderModel(cfg, params, recompute=recompute)


@pytest.mark.parametrize("lens", [[9], [30, 20], [60, 41, 7], [300, 200]])
@pytest.mark.parametrize("recompute", ["none", "full"])
def test_scores_are_the_log_probs_of_the_update(lens, recompute):
    from verl_b200.models import PackedBatch

    model = _model(recompute)
    ids = torch.randint(3, 2048, (sum(lens) + 1,), device=DEV, generator=torch.Generator(device=DEV).manual_seed(sum(lens)))
    batch = PackedBatch.from_lengths(ids[:-1], lens, device=DEV)
    with torch.no_grad():
        scored, _ = model.forward_logprobs(batch, ids[1:], 1.0, need_grad=False)
    updated, _ = model.forward_logprobs(batch, ids[1:], 1.0)
    assert torch.equal(scored, updated.detach())


@pytest.mark.parametrize("T,k,E,N,K", [(1, 1, 1, 8, 64), (33, 3, 7, 136, 256), (70, 4, 9, 384, 1152), (300, 2, 4, 1536, 2048), (64, 8, 128, 2048, 768)])
def test_tiles_of_few_tokens_give_the_bits_of_the_training_product(T, k, E, N, K):
    from verl_b200.ops import native

    ops = native.ops()
    g = torch.Generator(device=DEV).manual_seed(T)
    idx = torch.rand(T, E, device=DEV, generator=g).topk(k, -1).indices
    counts = torch.bincount(idx.reshape(-1), minlength=E).int()
    x, w = torch.randn(T, K, device=DEV, generator=g).bfloat16(), (torch.randn(E, N, K, device=DEV, generator=g) * 0.05).bfloat16()
    got = []
    for tile in (128, 16, 32, 64):
        slot, src, _, te, num = ops.moe_plan(idx, counts, tile)
        xp = ops.moe_gather_tiles(x, src, None, num, tile)
        rows = slot.reshape(-1).long()
        if tile == 128:
            want = ops.gemm_grouped_rows(xp, w, False, te, num)[rows]
        got.append(ops.gemm_grouped_tiles(xp, w, te, num, tile)[rows])
    assert all(torch.equal(y, want) for y in got)
    assert int(ops.gemm_status()) == 0
