"""Kernels at the sizes where their tiling can go wrong: edges of tiles, remainders, the smallest and largest of a rule's range."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.fixture(scope="module")
def ops():
    from verl_b200.ops import native

    return native.ops()


def rel(a, b):
    return float((a.double() - b.double()).norm() / b.double().norm().clamp_min(1e-30))


# ------------------------------------------------------------------------------------------------ advantages
@pytest.mark.parametrize("B,L", [(1, 1), (3, 17), (5, 128), (2, 1024), (2, 1025), (1300, 33), (7, 4099)])
@pytest.mark.parametrize("gamma,lam", [(1.0, 0.95), (0.9, 0.0)])
def test_gae_tiles(ops, B, L, gamma, lam):
    from verl_b200.ops import functional as F

    g = torch.Generator().manual_seed(B * 31 + L)
    r, v = torch.randn(B, L, generator=g) * 0.1, torch.randn(B, L, generator=g)
    m = (torch.rand(B, L, generator=g) > 0.3).float()
    m[:, 0] = 1
    adv, ret = F.gae_advantage(r.to(DEV), v.to(DEV), m.to(DEV), gamma, lam, whiten=False)
    want, nextv, last = torch.zeros(B, L, dtype=torch.float64), torch.zeros(B, dtype=torch.float64), torch.zeros(B, dtype=torch.float64)
    rd, vd = r.double(), v.double()
    for t in reversed(range(L)):
        step = rd[:, t] + gamma * nextv - vd[:, t] + gamma * lam * last
        nextv = torch.where(m[:, t] > 0, vd[:, t], nextv)
        last = torch.where(m[:, t] > 0, step, last)
        want[:, t] = last
    # 24 significant bits per step of a chain that forgets with gamma * lam: 1e-5 leaves room for some tens of roundings
    assert rel(adv.cpu(), want) < 1e-5 and rel(ret.cpu(), want + vd) < 1e-5
    white, _ = F.gae_advantage(r.to(DEV), v.to(DEV), m.to(DEV), gamma, lam, whiten=True)
    md, n = m.double(), m.double().sum()
    mean = (want * md).sum() / n
    var = ((want - mean).square() * md).sum() / (n - 1).clamp(min=1)
    if n > 1:
        assert rel(white.cpu(), (want - mean) * torch.rsqrt(var + 1e-8)) < 2e-5
    again, _ = F.gae_advantage(r.to(DEV), v.to(DEV), m.to(DEV), gamma, lam, whiten=True)
    assert torch.equal(again, white)


@pytest.mark.parametrize("B,L,dtype", [(1, 1, torch.int64), (6, 129, torch.int32), (1024, 7, torch.int64), (1025, 7, torch.int32), (1025, 7, torch.int64)])
def test_group_advantage_rows(ops, B, L, dtype):
    from verl_b200.ops import functional as F

    g = torch.Generator().manual_seed(B)
    groups = max(1, B // 5)
    ids = torch.randint(groups, (B,), generator=g)
    r, m = torch.rand(B, L, generator=g), (torch.rand(B, L, generator=g) > 0.2).float()
    for by_std in (True, False):
        adv, score = F.grpo_advantage(r.to(DEV), m.to(DEV), ids.to(DEV).to(dtype), groups, 1e-6, by_std)
        s = r.double().sum(-1)
        want = torch.zeros(B, dtype=torch.float64)
        for k in range(groups):
            sel = ids == k
            if sel.sum() == 1:
                want[sel] = s[sel] / (1 + 1e-6) if by_std else s[sel]
            elif sel.any():
                want[sel] = s[sel] - s[sel].mean()
                if by_std:
                    want[sel] /= s[sel].std() + 1e-6
        # the sums of squares of the atomic form cancel about two digits of the 7 that fp32 has
        assert rel(score.cpu(), s) < 1e-6 and rel(adv.cpu(), want[:, None] * m.double()) < (1e-5 if B <= 1024 else 2e-4)


@pytest.mark.parametrize("B", [2, 1024, 1025, 4000])
@pytest.mark.parametrize("offset,spread", [(0.5, 0.3), (50.0, 0.01), (-1000.0, 0.01)])
def test_group_advantage_of_close_scores(ops, B, offset, spread):
    """One reward per row, so that the scores are exact: mean and deviation then leave only the rounding of the result (2^-24)."""
    from verl_b200.ops import functional as F

    g = torch.Generator().manual_seed(B)
    ids = torch.randint((B + 4) // 5, (B,), generator=g)
    r = torch.zeros(B, 5)
    r[:, 3] = offset + spread * torch.randn(B, generator=g)
    s = r.double().sum(-1)
    n = torch.bincount(ids)[ids]
    mean = (torch.zeros(B, dtype=torch.float64).index_add(0, ids, s)[ids] / n) * (n > 1)
    var = torch.zeros(B, dtype=torch.float64).index_add(0, ids, (s - mean) ** 2)[ids] / (n - 1).clamp(min=1)
    for by_std in (True, False):
        adv, score = F.grpo_advantage(r.to(DEV), torch.ones(B, 5, device=DEV), ids.to(DEV), (B + 4) // 5, 1e-6, by_std)
        want = (s - mean) / (torch.where(n > 1, var.sqrt(), 1.0) + 1e-6) if by_std else s - mean
        assert torch.equal(score.cpu().double(), s)
        # (the double sums of squares of more than 1024 rows: 2^-53 n offset^2 / spread^2 below 1e-4 of a variance at the widest ratio)
        bound = 1e-6 + (1e-14 * (offset / spread) ** 2 if B > 1024 else 0)
        assert rel(adv.cpu(), want[:, None].expand(B, 5)) < bound


# ------------------------------------------------------------------------------------------------ sampler
def _uniforms(seeds, V, step):
    """The sampler's stream of uniforms: splitmix64's finaliser on uint64, the upper 24 bits, halfway between the grid points."""
    def mix(z):
        z = z + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))

    with np.errstate(over="ignore"):
        key = mix(seeds.astype(np.uint64) ^ (np.uint64(step) * np.uint64(0xD1342543DE82EF95)))
        h = (mix(key[:, None] + np.arange(V, dtype=np.uint64)[None]) >> np.uint64(40)).astype(np.int64)
    return h, (h.astype(np.float32) + np.float32(0.5)).astype(np.float64) / 2.0**24


@pytest.mark.parametrize("B,V,ld,valid", [(1, 8, 8, 8), (3, 4096, 4096, 4095), (5, 4104, 4104, 4104), (2, 16392, 16400, 0), (2, 33001, 33003, 0),
                                          (170, 9000, 9000, 8999), (1200, 1000, 1000, 0)])
@pytest.mark.parametrize("scale", [0.3, 2.5, 40.0])
def test_sampler_takes_the_token_of_the_whole_row(ops, B, V, ld, valid, scale):
    from verl_b200.ops import functional as F

    g = torch.Generator().manual_seed(V + B)
    lg = (torch.randn(B, ld, generator=g) * scale).bfloat16()
    lg[:, ::97] = -math.inf  # masked logits
    if B > 1:
        lg[0] = -math.inf  # a row with one token left
        lg[0, (valid or V) // 2] = -300.0
    seeds = torch.randint(1 << 40, (B,), generator=g)
    row = lg.to(DEV)[:, :V]
    n = valid or V
    x = lg[:, :n].double()
    for T in (1.0, 0.7, 0.0):
        tok, lp = F.sample_tokens(row, T, seeds.to(DEV), 3, valid)
        tok, lp = tok.cpu(), lp.cpu()
        xt = (lg[:, :n].float() * torch.tensor(1.0 / T if T else 1.0, dtype=torch.float32)).double()
        if T:
            h, u = _uniforms(seeds.numpy(), n, 3)
            score = xt - torch.log(-torch.log(torch.from_numpy(u)))
            plain = torch.from_numpy((h < 2**24 - 512).all(-1))  # near u = 1 the device's logarithm is coarser than the spacing of u
        else:
            score, plain = x, torch.ones(B, dtype=torch.bool)
            assert torch.equal(tok, x.argmax(-1))
        got = score.gather(1, tok[:, None])[:, 0]
        assert ((score.max(-1).values - got)[plain] <= 1e-4 * (1 + score.max(-1).values.abs()[plain])).all()
        want = xt.gather(1, tok[:, None])[:, 0] - xt.logsumexp(-1)
        assert (lp.double() - want).abs().max() < 1e-4 * (1 + xt[xt > -math.inf].abs().max())


@pytest.mark.parametrize("scale", [2.5, 20.0, 200.0])
@pytest.mark.parametrize("T", [1.0, 0.7, 0.1, 0.01, 0.0])
def test_sampler_log_probs_of_sharp_rows(ops, scale, T):
    """The largest logit's term of the sum is 1, so that no log-prob is positive. Error: half a unit in the last place of m + log l and of the
    two scaled logits (2^-24 of the next power of two each), the sum's and the fast logarithm's 4e-6."""
    from verl_b200.ops import functional as F

    g = torch.Generator(device=DEV).manual_seed(int(scale))
    lg = (torch.randn(512, 20011, device=DEV, generator=g) * scale).bfloat16()
    tok, lp = F.sample_tokens(lg, T, torch.arange(512, device=DEV), 3, 0)
    x = lg.double() * (torch.tensor(1.0 / T if T else 1.0, dtype=torch.float32)).double()
    want = x.gather(1, tok[:, None])[:, 0] - x.logsumexp(-1)
    unit = 2.0 ** (x.max(-1).values.abs().log2().ceil() - 24)
    assert ((lp.double() - want).abs() <= (1 if T in (1.0, 0.0) else 3) * unit + 4e-6).all()
    assert float(lp.max()) <= 2.0**-22


@pytest.mark.parametrize("V,ld,valid", [(8, 8, 0), (1000, 1000, 0), (2049, 2056, 0), (33001, 33003, 32999)])
def test_sampler_of_rows_without_numbers(ops, V, ld, valid):
    """NaN and masked logits: a token of the vocabulary all the same (the first where there is none to take), and a log-prob that is NaN."""
    from verl_b200.ops import functional as F

    n = valid or V
    lg = torch.full((5, ld), math.nan)
    lg[1] = -math.inf
    lg[2, : n // 2] = -math.inf
    lg[3, n - 1] = 1.5
    lg[4] = -math.inf
    lg[4, n - 1] = 1.5
    seeds = torch.arange(5, device=DEV)
    for T in (1.0, 0.3, 0.0):
        tok, lp = F.sample_tokens(lg.bfloat16().to(DEV)[:, :V], T, seeds, 3, valid)
        assert tok.tolist() == [0, 0, 0, n - 1, n - 1]
        assert lp[:4].isnan().all() and float(lp[4]) == 0.0


# ------------------------------------------------------------------------------------------------ head and optimizer
@pytest.mark.parametrize("T,V", [(1, 8), (31, 4096), (33, 4360), (130, 264)])
def test_head_merges_its_tiles(ops, T, V):
    from verl_b200.ops import functional as F

    g = torch.Generator(device=DEV).manual_seed(T)
    h = torch.randn(T, 64, device=DEV, generator=g).bfloat16()
    w = (torch.randn(V, 64, device=DEV, generator=g) * 0.5).bfloat16()
    lab = torch.randint(V, (T,), device=DEV, generator=g)
    lp, ent, lse = F.lmhead_logprob_entropy(h, w, lab, 0.8)
    logp = (h.double() @ w.double().T / 0.8).log_softmax(-1)
    # fp32 logits of magnitude up to about 20: 1e-5 absolute; the kernel's exponentials are the fast ones
    assert (lp - logp.gather(1, lab[:, None])[:, 0]).abs().max() < 1e-4
    assert (ent + (logp.exp() * logp).sum(-1)).abs().max() < 2e-4


@pytest.mark.parametrize("n,shift", [(1, 0), (3, 0), (4, 0), (1027, 0), (1030, 1)])
def test_adamw_remainders_and_alignment(ops, n, shift):
    g = torch.Generator(device=DEV).manual_seed(n)
    rnd = lambda: torch.randn(n + shift, device=DEV, generator=g)[shift:]
    p, gr, m, v = rnd(), rnd(), rnd() * 0.1, rnd().square()
    out = torch.zeros(n + shift, device=DEV, dtype=torch.bfloat16)[shift:]
    ctrl = torch.tensor([0.0, 0.5, 0.0, 0.0], device=DEV)
    pd, gd, md, vd = (t.double() for t in (p, gr, m, v))
    gd = gd * 0.5
    md, vd = 0.9 * md + 0.1 * gd, 0.999 * vd + 0.001 * gd.square()
    pd = pd * (1 - 1e-3 * 0.01) - 1e-3 * (md / (1 - 0.9**3)) / ((vd / (1 - 0.999**3)).sqrt() + 1e-8)
    ops.adamw_(p, gr, m, v, out, ctrl, 1e-3, 0.9, 0.999, 1e-8, 0.01, 3, 1.0, True)
    assert rel(p, pd) < 1e-6 and rel(m, md) < 1e-6 and rel(v, vd) < 1e-6 and torch.equal(out, p.bfloat16()) and not gr.any()


# ------------------------------------------------------------------------------------------------ attention
def _attention64(q, k, v, keys_of, scale):
    """fp64 attention of a packed stream; ``keys_of(t)`` = stream rows that query row t sees."""
    T, nh, hd = q.shape
    per = nh // k.shape[1]
    see = torch.zeros(T, T, dtype=torch.bool, device=q.device)
    for t in range(T):
        see[t, keys_of[t]] = True
    out = []
    for h in range(nh):
        s = (q[:, h] @ k[:, h // per].T * scale).masked_fill(~see, -math.inf)
        out.append(s.softmax(-1) @ v[:, h // per])
    return torch.stack(out, 1)


@pytest.mark.parametrize("hd,nh,nkv", [(64, 14, 2), (128, 4, 4), (128, 7, 1)])
@pytest.mark.parametrize("groups", [[(0, [1])], [(0, [63, 64, 65, 1, 200])], [(1, [1, 129]), (130, [128, 5, 64]), (0, [33])],
                                    [(64, [1, 127]), (65, [2, 2]), (128, [130])]])
def test_attention_of_prompts_and_their_continuations(ops, hd, nh, nkv, groups):
    """(prompt length, response lengths) per group; a prompt of 0 stands for separate sequences. Both directions, rotary tables folded
    into the backward pass, against fp64 over the same stream."""
    from verl_b200.ops import functional as F

    cu, parent, keys, pos = [0], [], [], []
    for p, rs in groups:
        if p:
            base, prompt_seg = cu[-1], len(parent)
            cu.append(base + p)
            parent.append(-1)
            keys += [list(range(base, base + i + 1)) for i in range(p)]
            pos += list(range(p))
        for r in rs:
            a = cu[-1]
            cu.append(a + r)
            parent.append(prompt_seg if p else -1)
            pre = list(range(base, base + p)) if p else []
            keys += [pre + list(range(a, a + i + 1)) for i in range(r)]
            pos += list(range(p, p + r))
    T = cu[-1]
    g = torch.Generator(device=DEV).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    qkv, dout = rnd(T, (nh + 2 * nkv) * hd), rnd(T, nh, hd)
    heads = lambda x: (x[:, : nh * hd].view(T, nh, hd), x[:, nh * hd : (nh + nkv) * hd].view(T, nkv, hd), x[:, (nh + nkv) * hd :].view(T, nkv, hd))
    q, k, v = heads(qkv)
    cu_t, par_t = torch.tensor(cu, dtype=torch.int32, device=DEV), torch.tensor(parent, dtype=torch.int32, device=DEV)
    scale = hd**-0.5
    longest = max(b - a for a, b in zip(cu, cu[1:]))
    cos, sin = F.rope_table(512, hd, 1e4, DEV)
    pos_t = torch.tensor(pos, dtype=torch.int32, device=DEV)
    out, lse = F.attention_shared_prefix(q, k, v, cu_t, par_t)
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    want = _attention64(*ref, keys, scale)
    # bf16 inputs, bf16 probabilities (2^-9 each) and a bf16 result
    assert rel(out, want.detach()) < 6e-3
    want.backward(dout.double())
    c, s = cos[pos_t.long()].double()[:, None], sin[pos_t.long()].double()[:, None]

    def back(x):  # inverse rotation
        a, b = x.chunk(2, -1)
        return torch.cat([a * c + b * s, b * c - a * s], -1)

    grads = torch.full_like(qkv, float("nan"))
    dq, dk, dv = heads(grads)
    F.attention_bwd_into_(dout, q, k, v, out, lse, cu_t, longest, dq, dk, dv, parent=par_t, rope=(pos_t, cos, sin))
    # dS is rounded to bf16 and its terms cancel: about 1e-2
    small = 1e-6 * float(dout.double().norm())  # (a single key: dQ and dK are zero)
    for got, w in ((dq, back(ref[0].grad)), (dk, back(ref[1].grad)), (dv, ref[2].grad)):
        assert float((got.double() - w).norm()) < 1.5e-2 * float(w.norm()) + small
    if max(parent) < 0:
        plain, plain_lse = F.attention_varlen(q, k, v, cu_t, longest)
        assert torch.equal(plain, out) and torch.equal(plain_lse, lse)
        for got, w in zip(F.attention_varlen_bwd(dout, q, k, v, out, lse, cu_t, longest), (r.grad for r in ref)):
            assert float((got.double() - w).norm()) < 1.5e-2 * float(w.norm()) + small


@pytest.mark.parametrize("hd,nh,nkv", [(128, 4, 4), (64, 4, 2)])
@pytest.mark.parametrize("lens,parent", [([70, 40, 33, 130, 5], [-1, -1, 0, 1, 0]), ([9, 200, 130], [1, -1, 1]), ([40, 129, 64, 1], [3, -1, 3, -1]),
                                         ([100, 50, 60], [-1, 0, 1])])
def test_continuations_anywhere_in_the_stream(ops, hd, nh, nkv, lens, parent):
    """Sequences that continue an earlier or a later one with others between, and one that continues a continuation (of which it sees only the
    keys of its own parent). One head per KV head: the prompt's own CTA would store what others add."""
    from verl_b200.ops import functional as F

    cu = np.cumsum([0] + lens).tolist()
    keys = [(list(range(cu[p], cu[p + 1])) if p >= 0 else []) + list(range(a, a + i + 1)) for a, n, p in zip(cu, lens, parent) for i in range(n)]
    T = cu[-1]
    g = torch.Generator(device=DEV).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    q, k, v, dout = rnd(T, nh, hd), rnd(T, nkv, hd), rnd(T, nkv, hd), rnd(T, nh, hd)
    cu_t, par_t = torch.tensor(cu, dtype=torch.int32, device=DEV), torch.tensor(parent, dtype=torch.int32, device=DEV)
    out, lse = F.attention_shared_prefix(q, k, v, cu_t, par_t)
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    want = _attention64(*ref, keys, hd**-0.5)
    assert rel(out, want.detach()) < 6e-3
    want.backward(dout.double())
    got = [torch.empty_like(t) for t in (q, k, v)]
    for _ in range(3):
        F.attention_bwd_into_(dout, q, k, v, out, lse, cu_t, max(lens), *got, parent=par_t)
        for x, w in zip(got, ref):
            assert rel(x, w.grad) < 1.5e-2  # dS is rounded to bf16 and its terms cancel


@pytest.mark.parametrize("where,dtype", [("cpu", torch.int32), ("cpu", torch.int64), (DEV, torch.int64)])
def test_lengths_from_the_host(where, dtype):
    """An update over a batch whose lengths lie on the host, as the plain attention ops take them, and both ops on a shared prompt."""
    from verl_b200.models import DecoderModel, FlatParams, PackedBatch
    from verl_b200.models.config import get_preset
    from verl_b200.ops import functional as F

    cfg = get_preset("qwen2.5-0.5b")
    cfg.num_hidden_layers = 1
    got = []
    for kind in ("as packed", "moved"):
        params = FlatParams(cfg, dtype=torch.bfloat16, device=DEV, with_main_grad=True)
        params.init_weights(seed=3, std=0.05)
        batch = PackedBatch.from_lengths(torch.arange(3, 53, device=DEV), [20, 30], device=DEV)
        if kind == "moved":
            batch.cu_seqlens = batch.cu_seqlens.to(where, dtype)
        lp, _ = DecoderModel(cfg, params).forward_logprobs(batch, torch.arange(4, 54, device=DEV), 1.0)
        lp.sum().backward()
        got.append((lp.detach(), params.main_grad))
    assert torch.equal(got[0][0], got[1][0]) and rel(got[1][1], got[0][1]) < 1e-3
    x = torch.randn(50, 2, 64, device=DEV).bfloat16()
    cu, parent = torch.tensor([0, 20, 50], dtype=torch.int32, device=DEV), torch.tensor([-1, 0], dtype=torch.int32, device=DEV)
    res = []
    for c, p in ((cu, parent), (cu.to(where, dtype), parent.to(where, dtype))):
        out, lse = F.attention_shared_prefix(x, x, x, c, p)
        grads = [torch.empty_like(x) for _ in range(3)]
        F.attention_bwd_into_(x, x, x, x, out, lse, c, 30, *grads, parent=p)
        res.append([out, *grads])
    assert torch.equal(res[0][0], res[1][0]) and all(rel(a, b) < 1e-3 for a, b in zip(res[1], res[0]))


def test_audit_names_a_parent_out_of_range():
    from verl_b200.ops import audit
    from verl_b200.ops import functional as F

    x, cu = torch.zeros(4, 2, 64, device=DEV, dtype=torch.bfloat16), torch.tensor([0, 2, 4], dtype=torch.int32, device=DEV)
    with audit.scope(), pytest.raises(audit.AuditError, match="parent"):
        F.attention_shared_prefix(x, x, x, cu, torch.tensor([-1, 2], dtype=torch.int32, device=DEV))


@pytest.mark.parametrize("preset,layers", [("qwen2.5-0.5b", 2), ("tiny-shared", 2)])
def test_update_with_shared_prompts_equals_separate_rows(ops, preset, layers):
    from verl_b200.models import DecoderModel, FlatParams
    from verl_b200.models.config import ModelConfig, get_preset
    from verl_b200.trainer.ppo.prefix_grouper_utils import pack_shared_prefix_batch
    from verl_b200.workers.engine.native.engine import pack_padded_batch

    cfg = get_preset(preset) if preset != "tiny-shared" else ModelConfig(
        model_type="qwen3", vocab_size=512, hidden_size=256, intermediate_size=512, num_attention_heads=4, num_key_value_heads=2, head_dim=128)
    cfg.num_hidden_layers = layers
    plen, rlen, P, R = [70, 70, 70, 33, 5, 5], [1, 130, 64, 9, 77, 40], 80, 130
    gids = [0, 0, 0, 1, 2, 2]
    g = torch.Generator().manual_seed(1)
    ids = torch.randint(3, 500, (6, P + R), generator=g)
    for i in range(1, 6):
        if gids[i] == gids[i - 1]:
            ids[i, :P] = ids[i - 1, :P]
    at = torch.arange(P + R)[None]
    mask = ((at >= P - torch.tensor(plen)[:, None]) & (at < P + torch.tensor(rlen)[:, None])).long()
    ids, mask = (ids * mask).to(DEV), mask.to(DEV)
    w = torch.randn(sum(rlen), generator=g).to(DEV)
    got = []
    for shared in (True, False):
        params = FlatParams(cfg, dtype=torch.bfloat16, device=DEV, with_main_grad=True)
        params.init_weights(seed=3, std=0.05)
        model = DecoderModel(cfg, params)
        if shared:
            batch, pos, lab, _ = pack_shared_prefix_batch(ids, mask, None, R, gids, plen, rlen)
            lp, _ = model.forward_logprobs(batch, None, 1.0, positions=pos, position_labels=lab)
        else:
            batch, lab, index, valid = pack_padded_batch(ids, mask, None, R)
            lp, _ = model.forward_logprobs(batch, lab, 1.0, positions=index[valid])
        (lp * w).sum().backward()
        got.append((lp.detach(), params.main_grad))
    # the same numbers in another order of summation, rounded to bf16 in between; std 0.05 weights magnify it a little
    assert (got[0][0] - got[1][0]).abs().max() < 0.1 and rel(got[0][1], got[1][1]) < 3e-2


@pytest.mark.parametrize("T,N,ld", [(1, 1, 1), (63, 511, 511), (65, 513, 520), (130, 1026, 1031), (1000, 4608, 4608)])
def test_column_sums(ops, T, N, ld):
    from verl_b200.ops import functional as F

    g = torch.Generator(device=DEV).manual_seed(N)
    x = torch.randn(T, ld, device=DEV, generator=g).bfloat16()[:, :N]
    out = torch.randn(N, device=DEV, generator=g)
    want = out.double() + x.double().sum(0)
    F.colsum_add_(x, out)
    assert (out - want).abs().max() < 1e-6 * (10 + T)


@pytest.mark.parametrize("T,N", [(7900, 4608), (12000, 1152), (40000, 130)])
def test_column_sums_lose_no_digits_over_many_rows(ops, T, N):
    """Terms of one sign mostly, as a mean that does not cancel: eight chains of eight and three pairs in fp32 (averaged over the chunks of 64
    rows), then one rounding (at most 2^-24, its root mean square below half of that)."""
    from verl_b200.ops import functional as F

    g = torch.Generator(device=DEV).manual_seed(N)
    x = (torch.randn(T, N, device=DEV, generator=g) * 0.01 + 0.02).bfloat16()
    out = torch.zeros(N, device=DEV)
    F.colsum_add_(x, out)
    want = x.double().sum(0)
    assert float(((out.double() - want) / want).square().mean().sqrt()) < 2.0**-25


# ------------------------------------------------------------------------------------------------ expert products on tiles of tokens
def _choices(T, k, E, seed, skew=False):
    """Distinct experts per token; with ``skew`` most tokens meet the first ones and some experts stay empty."""
    g = torch.Generator().manual_seed(seed)
    score = torch.rand(T, E, generator=g)
    if skew:
        score[:, :k] += 0.9
        score[:, E // 2 + 1 :] -= 2.0
    return score.topk(k, dim=-1).indices.cuda()


@pytest.mark.parametrize("tile", [16, 32, 64, 128])
@pytest.mark.parametrize("T,k,E,skew", [(1, 1, 1, False), (3, 2, 5, True), (32, 8, 128, False), (257, 4, 60, True), (2049, 8, 128, False),
                                        (40, 2, 1024, False), (8192, 1, 3, False), (8193, 1, 1, False), (1025, 8, 1024, False), (1366, 6, 64, True),
                                        (40000, 4, 1023, False), (30000, 8, 128, True)])
def test_expert_plan_is_the_stable_sort_by_expert(ops, tile, T, k, E, skew):
    idx = _choices(T, k, E, T + E, skew)
    counts = torch.bincount(idx.reshape(-1), minlength=E).int()
    for choice in (idx, idx.int()):
        slot, src, seg, te, num = ops.moe_plan(choice.contiguous(), counts, tile)
        pad = (counts.long() + tile - 1) // tile * tile
        first = pad.cumsum(0) - pad
        assert seg.tolist() == [0] + pad.cumsum(0).tolist() and int(num) == int(pad.sum()) // tile
        flat = idx.reshape(-1)
        order = torch.argsort(flat, stable=True)
        rank = torch.arange(T * k, device=DEV) - (counts.long().cumsum(0) - counts.long())[flat[order]]
        want = torch.empty_like(flat)
        want[order] = first[flat[order]] + rank
        assert torch.equal(slot.reshape(-1).long(), want)
        rows = torch.full_like(src, -1)
        rows[want] = (torch.arange(T * k, device=DEV) // k).int()
        assert torch.equal(src, rows)
        used = int(num)
        assert torch.equal(te[:used].long(), torch.repeat_interleave(torch.arange(E, device=DEV), pad // tile))
        assert src.numel() % tile == 0 and used <= te.numel()


@pytest.mark.parametrize("n", [64, 20000])
def test_expert_plan_of_foreign_counts_stays_in_range(ops, n):
    """Choices without an expert, and counts that are not the list's: every row and every slot is one of the buffers' own."""
    g = torch.Generator().manual_seed(n)
    idx = torch.randint(-2, 11, (n // 2, 2), generator=g).to(DEV)
    for counts in (torch.zeros(9), torch.full((9,), n // 9), torch.arange(9) * n):
        slot, src, seg, te, num = ops.moe_plan(idx, counts.int().to(DEV), 16)
        assert int(slot.min()) >= 0 and int(slot.max()) < src.numel() and int(src.min()) >= -1 and int(src.max()) < n // 2
        assert int(te.min()) >= 0 and int(te.max()) < 9 and 0 <= int(num) <= te.numel()


@pytest.mark.parametrize("tile", [16, 32, 64, 128])
@pytest.mark.parametrize("T,k,E,N,K", [(1, 1, 1, 8, 128), (33, 3, 7, 136, 256), (70, 4, 9, 384, 1152), (300, 2, 4, 128, 384)])
def test_grouped_tiles_match_the_product_per_expert(ops, tile, T, k, E, N, K):
    """bf16 operands: products are exact in fp32, so the bound is the rounding of the result (2^-9) and of fp32 sums of K terms.
    fp8: the same for the dequantised operands."""
    from verl_b200.ops import functional as F

    idx = _choices(T, k, E, N + K)
    counts = torch.bincount(idx.reshape(-1), minlength=E).int()
    slot, src, seg, te, num = ops.moe_plan(idx.contiguous(), counts, tile)
    g = torch.Generator().manual_seed(T)
    x = torch.randn(T, K, generator=g).cuda().bfloat16()
    w = (torch.randn(E, N, K, generator=g) * 0.05).cuda().bfloat16()
    xp = ops.moe_gather_tiles(x, src, None, num, tile)
    rows = slot.reshape(-1).long()
    tok, exp = torch.arange(T * k, device=DEV) // k, idx.reshape(-1)
    assert torch.equal(xp[rows], x[tok])
    y = ops.gemm_grouped_tiles(xp, w, te, num, tile)[rows].double()
    want = torch.einsum("rk,rnk->rn", x[tok].double(), w[exp].double())
    size = torch.einsum("rk,rnk->rn", x[tok].double().abs(), w[exp].double().abs())
    assert ((y - want).abs() <= want.abs() * 2.0**-8 + size * K * 2.0**-24).all()
    xq, xs = F.fp8_quantize_1x128(xp)
    xd = F.fp8_dequantize_1x128(xq, xs).double()[rows]
    wq, ws = F.fp8_quantize_1x128(w.reshape(E * N, K))
    wd = F.fp8_dequantize_1x128(wq, ws).view(E, N, K).double()
    want, size = torch.einsum("rk,rnk->rn", xd, wd[exp]), torch.einsum("rk,rnk->rn", xd.abs(), wd[exp].abs())
    if tile == 128:
        y = ops.gemm_fp8_blockscale_grouped(xq, xs, wq, ws, N, te, num)[rows].double()
        assert ((y - want).abs() <= want.abs() * 2.0**-8 + size * K * 2.0**-24).all()
    if N % 128 == 0 and K % 128 == 0:  # the whole expert: gate, up of width N / 2 and back
        I = N // 2 if (N // 2) % 128 == 0 else N
        wgu = (torch.randn(E, 2 * I, K, generator=g) * 0.05).cuda().bfloat16()
        wdn = (torch.randn(E, K, I, generator=g) * 0.05).cuda().bfloat16()
        a, b = F.fp8_quantize_1x128(wgu.reshape(-1, K)), F.fp8_quantize_1x128(wdn.reshape(-1, I))
        y = ops.moe_experts_fp8(x, src, a[0], a[1], b[0], b[1], I, te, num, tile)[rows]
        gu = torch.einsum("rk,rnk->rn", xd, F.fp8_dequantize_1x128(*a).view(E, 2 * I, K).double()[exp]).bfloat16()
        act = F.swiglu(gu.contiguous())
        ad = F.fp8_dequantize_1x128(*F.fp8_quantize_1x128(act)).double()
        want = torch.einsum("rk,rnk->rn", ad, F.fp8_dequantize_1x128(*b).view(E, K, I).double()[exp])
        # a gate or up value rounded the other way moves an e4m3 activation by up to 2^-3 of itself: a few per row
        assert float((y.double() - want).norm() / want.norm()) < 0.02
    assert int(ops.gemm_status()) == 0


@pytest.mark.parametrize("M", [1, 16, 17, 32, 33, 64, 65, 129, 300])
def test_fp8_block_scaled_product_over_token_tiles(ops, M):
    from verl_b200.ops import functional as F

    N, K = 200, 384
    g = torch.Generator().manual_seed(M)
    x, w = torch.randn(M, K, generator=g).cuda().bfloat16(), torch.randn(N, K, generator=g).cuda().bfloat16()
    bias = torch.randn(N, generator=g).cuda().bfloat16()
    xq, xs = F.fp8_quantize_1x128(x)
    wq, ws = F.fp8_quantize_1x128(w)
    y = ops.gemm_fp8_blockscale(xq, xs, wq, ws, bias).double()
    xd, wd = F.fp8_dequantize_1x128(xq, xs).double(), F.fp8_dequantize_1x128(wq, ws).double()
    want = xd @ wd.T + bias.double()
    assert ((y - want).abs() <= want.abs() * 2.0**-8 + (xd.abs() @ wd.abs().T) * K * 2.0**-24).all()


@pytest.mark.parametrize("T,nh,nkv,hd", [(1, 1, 1, 64), (5, 4, 2, 128), (33, 3, 1, 256), (70, 8, 8, 96), (2000, 8, 2, 128)])
def test_qk_norm_rotation_and_append_in_one(ops, T, nh, nkv, hd):
    """The bits of the separate kernels."""
    from verl_b200.ops import functional as F

    g = torch.Generator().manual_seed(T + hd)
    qkv = torch.randn(T, (nh + 2 * nkv) * hd, generator=g).cuda().bfloat16()
    wq, wk = (1 + 0.1 * torch.randn(2, hd, generator=g)).cuda().bfloat16()
    cos, sin = F.rope_table(128, hd, 1e4, DEV)
    pos = torch.randint(0, 128, (T,), generator=g).int().cuda()
    slots = torch.randperm(3 * T + 4, generator=g)[:T].cuda()
    slots[0] = -1 if T > 1 else slots[0]
    kc, vc = torch.zeros(2, (3 * T + 5) // 2 + 1, 2, nkv, hd, device=DEV, dtype=torch.bfloat16)
    kr, vr = kc.clone(), vc.clone()
    ref = qkv.clone()
    q, k, v = (t.view(T, -1, hd) for t in ref.split([nh * hd, nkv * hd, nkv * hd], -1))
    qp, kp = q.reshape(-1, hd).clone(), k.reshape(-1, hd).clone()
    qn, _, rq = F.rms_norm(qp, wq, 1e-6)
    kn, _, rk = F.rms_norm(kp, wk, 1e-6)
    q.copy_(qn.view_as(q))
    k.copy_(kn.view_as(k))
    F.apply_rope_(q, pos, cos, sin)
    F.apply_rope_(k, pos, cos, sin)
    F.kv_append_(k, v, slots, kr, vr)
    saved = F.qk_norm_rope_(qkv, pos, cos, sin, wq, wk, 1e-6, nh, nkv, hd, slots, kc, vc, save=True)
    assert torch.equal(saved[0], qp) and torch.equal(saved[1], kp)
    assert torch.equal(saved[2], rq) and torch.equal(saved[3], rk)
    assert int((qkv != ref).sum()) == 0 and torch.equal(kc, kr) and torch.equal(vc, vr)


# ------------------------------------------------------------------------------------------------ products of at most 64 tokens
@pytest.mark.parametrize("M", [1, 7, 8, 9, 16, 17, 32, 33, 64])
@pytest.mark.parametrize("N,K", [(2, 8), (24, 64), (130, 72), (896, 4864), (1152, 896), (9600, 136)])
def test_few_tokens(ops, M, N, K):
    """bf16 products are exact in fp32: the bound is the rounding of the result (2^-9, twice with the activation's inputs) and of the sums."""
    g = torch.Generator().manual_seed(M + N + K)
    x = torch.randn(M, K + 8, generator=g).to(DEV).bfloat16()[:, :K]
    w = (torch.randn(2 * N, K, generator=g) * 0.1).to(DEV).bfloat16()
    bias = torch.randn(N, generator=g).to(DEV).bfloat16()
    full, size = x.double() @ w.double().T, x.double().abs() @ w.double().abs().T
    for b in (None, bias):
        want = full[:, :N] + (b.double() if b is not None else 0)
        y = ops.gemm_few_tokens(x, w[:N], b, False).double()
        assert ((y - want).abs() <= want.abs() * 2.0**-8 + size[:, :N] * K * 2.0**-24 + 1e-30).all()
    gu = ops.gemm_few_tokens(x, w, None, False)
    if M > 16:  # the gated form ends here
        with pytest.raises(RuntimeError):
            ops.gemm_few_tokens(x, w, None, True)
        return
    act = ops.gemm_few_tokens(x, w, None, True)
    want = torch.nn.functional.silu(gu[:, :N].double()) * gu[:, N:].double()
    assert rel(act, want) < 4e-3  # 2^-9 for the result, 2^-9 where another order of the sums rounds a gate or an up value differently


# ------------------------------------------------------------------------------------------------ weight gradients added in L2
@pytest.mark.parametrize("M,N,K", [(32, 136, 64), (96, 264, 72), (128, 256, 64), (160, 776, 200), (2048, 768, 640), (40, 264, 128)])
def test_weight_gradient_accumulates(ops, M, N, K):
    g = torch.Generator().manual_seed(M + N + K)
    dy, x = torch.randn(K, M, generator=g).to(DEV).bfloat16(), torch.randn(K, N, generator=g).to(DEV).bfloat16()
    out = torch.randn(M, N + 8, generator=g).to(DEV)
    before = out.clone()
    for _ in range(2):
        ops.gemm(dy, x, None, out[:, :N], True, True, True, True, 0)
    want = before[:, :N].double() + 2 * (dy.double().T @ x.double())
    size = dy.double().abs().T @ x.double().abs()
    assert ((out[:, :N].double() - want).abs() <= (2 * size * K + before[:, :N].double().abs() + want.abs()) * 2.0**-23).all()
    assert torch.equal(out[:, N:], before[:, N:])
    assert int(ops.gemm_status()) == 0


@pytest.mark.parametrize("ctas", [1, 2, 0])
@pytest.mark.parametrize("M,N,K", [(160, 2056, 16), (96, 2056, 64), (224, 1288, 8), (32, 4104, 24)])
def test_weight_gradient_of_slabs_behind_the_last_row(ops, ctas, M, N, K):
    """Many short tiles per CTA, every second one with slabs of 32 rows behind the last row. Small integers: every sum is exact."""
    g = torch.Generator().manual_seed(M + N + K)
    dy, x = torch.randint(-4, 5, (K, M), generator=g).to(DEV).bfloat16(), torch.randint(-4, 5, (K, N), generator=g).to(DEV).bfloat16()
    out = torch.randint(-99, 100, (M, N), generator=g).to(DEV).float()
    want = out + 8 * (dy.float().T @ x.float())
    for _ in range(8):
        ops.gemm(dy, x, None, out, True, True, True, True, ctas)
    assert torch.equal(out, want)
    assert int(ops.gemm_status()) == 0


@pytest.mark.parametrize("M,N", [(128, 256), (160, 264), (96, 768), (72, 264)])
def test_weight_gradient_per_expert_accumulates(ops, M, N):
    counts = [130, 0, 128, 5, 0]
    seg = torch.tensor([0] + np.cumsum([(c + 127) // 128 * 128 for c in counts]).tolist(), dtype=torch.int32, device=DEV)
    rows = int(seg[-1]) + 128
    g = torch.Generator().manual_seed(M + N)
    dy, x = torch.zeros(rows, M, device=DEV, dtype=torch.bfloat16), torch.zeros(rows, N, device=DEV, dtype=torch.bfloat16)
    for e, c in enumerate(counts):
        dy[seg[e] : seg[e] + c] = torch.randn(c, M, generator=g).to(DEV).bfloat16()
        x[seg[e] : seg[e] + c] = torch.randn(c, N, generator=g).to(DEV).bfloat16()
    out = torch.randn(len(counts), M, N, generator=g).to(DEV)
    want = out.double()
    for e, c in enumerate(counts):
        want[e] += dy[seg[e] : seg[e] + c].double().T @ x[seg[e] : seg[e] + c].double()
    ops.gemm_grouped_wgrad_(dy, x, out, seg, True)
    assert float((out.double() - want).abs().max()) < 1e-3  # sums of at most 130 products of size 1..10 in fp32
    assert int(ops.gemm_status()) == 0


def test_grouped_products_on_every_device_of_the_process(ops):
    for d in range(torch.cuda.device_count()):
        g = torch.Generator().manual_seed(1)
        seg = torch.tensor([0, 128, 256], dtype=torch.int32, device=f"cuda:{d}")
        dy, x = torch.randint(-3, 4, (256, 96), generator=g).to(seg.device).bfloat16(), torch.randint(-3, 4, (256, 264), generator=g).to(seg.device).bfloat16()
        out = torch.ones(2, 96, 264, device=seg.device)
        ops.gemm_grouped_wgrad_(dy, x, out, seg, True)
        for e in range(2):
            part = slice(128 * e, 128 * e + 128)
            assert torch.equal(out[e].cpu(), 1 + dy[part].float().cpu().T @ x[part].float().cpu())
        w = torch.randint(-3, 4, (2, 24, 264), generator=g).to(seg.device).bfloat16()
        te, num = torch.arange(16, dtype=torch.int32, device=seg.device) // 8, torch.tensor([16], dtype=torch.int32, device=seg.device)
        y = ops.gemm_grouped_tiles(x, w, te, num, 16)
        for e in range(2):
            part = slice(128 * e, 128 * e + 128)
            assert torch.equal(y[part].float().cpu(), (x[part].float().cpu() @ w[e].float().cpu().T).bfloat16().float())


# ------------------------------------------------------------------------------------------------ norms
@pytest.mark.parametrize("T,H", [(1, 8), (3, 248), (5, 264), (639, 264), (1183, 896), (1184, 1024), (640, 1032), (700, 2040), (1185, 2048),
                                 (641, 2056), (9, 3584), (700, 3584), (640, 4096), (640, 4104), (2, 8192), (1300, 3592)])
def test_rmsnorm_rows(ops, T, H):
    g = torch.Generator().manual_seed(T + H)
    x, res, dy, dres = (torch.randn(T, H, generator=g).to(DEV).bfloat16() for _ in range(4))
    w = (1 + 0.1 * torch.randn(H, generator=g)).to(DEV).bfloat16()
    for r in (None, res):
        y, xe, rstd = ops.rmsnorm_fwd(x, r, w, 1e-6)
        if r is not None:
            assert torch.equal(xe, (x.float() + r.float()).bfloat16())
        xd = xe.double()
        want = torch.rsqrt(xd.square().mean(-1) + 1e-6)
        torch.testing.assert_close(rstd.double(), want, rtol=2e-6, atol=0)  # fp32 sums of squares and the approximate root
        full = xd * want[:, None] * w.double()
        assert ((y.double() - full).abs() <= 2.0**-8 * full.abs() + 1e-30).all()
        few = ops.rmsnorm_fwd(x[:3].contiguous(), None if r is None else r[:3].contiguous(), w, 1e-6)
        assert torch.equal(few[0], y[:3]) and torch.equal(few[2], rstd[:3])  # a row's bits do not depend on the number of rows
    dw = torch.randn(H, generator=g).to(DEV)
    dw0 = dw.clone()
    dx = ops.rmsnorm_bwd(dy, x, w, ops.rmsnorm_fwd(x, None, w, 1e-6)[2], dres, dw, True)
    xd = x.double().requires_grad_()
    wd = w.double().requires_grad_()
    (xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * wd).backward(dy.double())
    assert rel(dx, xd.grad + dres.double()) < 4e-3  # rounding of the result
    assert rel(dw - dw0, wd.grad) < 1e-5


@pytest.mark.parametrize("T,nh,nkv,hd", [(1, 1, 1, 64), (5, 4, 2, 128), (33, 3, 1, 256), (70, 8, 8, 96), (1000, 32, 4, 128)])
def test_qk_norm_backward_in_place(ops, T, nh, nkv, hd):
    from verl_b200.ops import functional as F

    g = torch.Generator().manual_seed(T + hd)
    gq = torch.randn(T, (nh + 2 * nkv) * hd, generator=g).to(DEV).bfloat16()
    pre = [torch.randn(T * n, hd, generator=g).to(DEV).bfloat16() for n in (nh, nkv)]
    w = [(1 + 0.1 * torch.randn(hd, generator=g)).to(DEV).bfloat16() for _ in range(2)]
    rstd = [torch.rsqrt(p.float().square().mean(-1) + 1e-6) for p in pre]
    dw = [torch.ones(hd, device=DEV) for _ in range(2)]
    out = gq.clone()
    F.qk_norm_bwd_(out, *pre, *rstd, *w, *dw, nh, nkv, hd)
    assert torch.equal(out[:, (nh + nkv) * hd :], gq[:, (nh + nkv) * hd :])
    for i, sl in enumerate((slice(0, nh * hd), slice(nh * hd, (nh + nkv) * hd))):
        xd, wd = pre[i].double().requires_grad_(), w[i].double().requires_grad_()
        (xd * torch.rsqrt(xd.square().mean(-1, keepdim=True) + 1e-6) * wd).backward(gq[:, sl].reshape(-1, hd).double())
        assert rel(out[:, sl].reshape(-1, hd), xd.grad) < 4e-3
        assert rel(dw[i] - 1, wd.grad) < 1e-5


# ------------------------------------------------------------------------------------------------ a group's heads over several CTAs
@pytest.mark.parametrize("nh,nkv,hd,lens", [(64, 32, 64, [700, 600]), (7, 1, 64, [1, 64, 65, 300]), (48, 16, 128, [513, 97, 700, 640]),
                                            (14, 2, 128, [31, 33, 129]), (32, 8, 64, [1500, 700]), (14, 2, 128, [400] * 6)])
def test_attention_backward_over_shares_of_heads(ops, nh, nkv, hd, lens):
    """One CTA for all heads of a group, two, four (the last with fewer heads), and one per head; without parents, so that a single CTA stores
    dK and dV."""
    from verl_b200.ops import functional as F

    T = sum(lens)
    cu = np.cumsum([0] + lens).tolist()
    g = torch.Generator(device=DEV).manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    q, k, v, dout = rnd(T, nh, hd), rnd(T, nkv, hd), rnd(T, nkv, hd), rnd(T, nh, hd)
    cu_t = torch.tensor(cu, dtype=torch.int32, device=DEV)
    out, lse = F.attention_varlen(q, k, v, cu_t, max(lens))
    got = F.attention_varlen_bwd(dout, q, k, v, out, lse, cu_t, max(lens))
    ref = [t.double().requires_grad_(True) for t in (q, k, v)]
    want = _attention64(*ref, [list(range(a, a + i + 1)) for a, n in zip(cu, lens) for i in range(n)], hd**-0.5)
    assert rel(out, want.detach()) < 6e-3
    want.backward(dout.double())
    for x, w in zip(got, ref):
        assert rel(x, w.grad) < 1.5e-2  # dS is rounded to bf16 and its terms cancel
    assert int(ops.gemm_status()) == 0


@pytest.mark.parametrize("hd", [64, 128])
@pytest.mark.parametrize("scale", [0.125, 0.0, -0.05])
def test_attention_scales_and_growing_scores(ops, hd, scale):
    """Scores that grow along the keys (the maximum moves in every block, in small and large steps), 33 sequences, any sign of the scale."""
    nh, nkv = 4, 2
    lens = [1, 3] * 16 + [700]
    T, cu = sum(lens), np.cumsum([0] + lens).tolist()
    g = torch.Generator(device=DEV).manual_seed(hd)
    rnd = lambda *s: torch.randn(*s, device=DEV, generator=g).bfloat16()
    q, k, v = rnd(T, nh, hd), rnd(T, nkv, hd), rnd(T, nkv, hd)
    q[:, 0] = q[:, 0].abs()
    k[:, 0] = (k[:, 0].abs() * torch.linspace(0.01, 4, T, device=DEV)[:, None]).bfloat16()
    out, lse = ops.attn_fwd(q, k, v, torch.tensor(cu, dtype=torch.int32, device=DEV), scale, None)
    keys = [list(range(a, a + i + 1)) for a, n in zip(cu, lens) for i in range(n)]
    want = _attention64(q.double(), k.double(), v.double(), keys, scale)
    assert rel(out, want) < 6e-3
    for h in range(nh):
        s = (q[:, h].double() @ k[:, h // 2].double().T * scale)
        see = torch.full((T, T), -math.inf, dtype=torch.float64, device=DEV)
        for t in range(T):
            see[t, keys[t]] = 0
        torch.testing.assert_close(lse[h].double(), (s + see).logsumexp(-1), rtol=1e-5, atol=1e-4)
