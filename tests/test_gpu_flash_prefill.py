"""Prompt flash attention on tcgen05 / tensor memory against a plain fp32 PyTorch attention."""
import math

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _ref(q, k, v, pos0):
    """q [n_q, T, d] (pre-scaled), k / v [n_kv, n_keys, d]; causal: query t sees keys 0 .. pos0 + t."""
    n_q, T, d = q.shape
    n_kv, n_keys, _ = k.shape
    g = n_q // n_kv
    kk = k.repeat_interleave(g, 0).float()
    vv = v.repeat_interleave(g, 0).float()
    s = torch.einsum("htd,hkd->htk", q.float(), kk)
    t_idx = torch.arange(T, device=q.device)[:, None] + pos0
    k_idx = torch.arange(n_keys, device=q.device)[None, :]
    s = s.masked_fill((k_idx > t_idx)[None], float("-inf"))
    return torch.einsum("htk,hkd->htd", torch.softmax(s, -1), vv)          # [n_q, T, d]


@pytest.mark.parametrize("n_q,n_kv,T,pos0", [(8, 2, 300, 0), (4, 4, 257, 77), (32, 4, 1024, 0), (2, 1, 128, 4000), (8, 1, 64, 0)])
def test_flash_prefill_matches_fp32_attention(n_q, n_kv, T, pos0):
    from bloomery_b200.ops import gemm as G
    torch.manual_seed(0)
    d = 128
    n_keys = pos0 + T
    t_pad = (n_keys + 127) // 128 * 128
    q = (torch.randn(n_q, T, d, device=DEV) / math.sqrt(d)).bfloat16()
    k = torch.randn(n_kv, n_keys, d, device=DEV).bfloat16()
    v = torch.randn(n_kv, n_keys, d, device=DEV).bfloat16()
    Kb = torch.zeros(n_kv, t_pad, d, device=DEV, dtype=torch.bfloat16)
    Vt = torch.zeros(n_kv, d, t_pad, device=DEV, dtype=torch.bfloat16)
    Kb[:, :n_keys] = k
    Vt[:, :, :n_keys] = v.transpose(1, 2)
    out = torch.full((T, n_q * d), float("nan"), device=DEV, dtype=torch.bfloat16)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    G.flash_prefill(q, Kb, Vt, out, pos0, status)
    torch.cuda.synchronize()
    assert int(status) == 0
    ref = _ref(q, k, v, pos0).permute(1, 0, 2).reshape(T, n_q * d)
    err = (out.float() - ref).abs().max().item()
    assert torch.isfinite(out.float()).all()
    assert err < 2e-2 * max(1.0, ref.abs().max().item()), err      # bf16 probabilities and outputs
    out2 = torch.zeros_like(out)
    G.flash_prefill(q, Kb, Vt, out2, pos0, status)
    assert torch.equal(out, out2)                                   # bit-identical rerun


@pytest.mark.parametrize("T", [200, 300, 511])
def test_flash_prefill_repeats_itself_with_cold_caches(T):
    """Values that arrive late hold a value product back; the next tile's probabilities must wait for it whether or not a
    row rescales its output (scores this small never do), and so must the output.  Every launch reads from memory."""
    from bloomery_b200.ops import gemm as G
    g = torch.Generator(device=DEV).manual_seed(T)
    n_q, n_kv, d = 32, 4, 128
    t_pad = (T + 127) // 128 * 128
    q = (torch.randn(n_q, T, d, device=DEV, generator=g) / d).bfloat16()
    k, v = (torch.randn(n_kv, T, d, device=DEV, generator=g).bfloat16() for _ in range(2))
    Kb, Vt = torch.zeros(n_kv, t_pad, d, device=DEV, dtype=torch.bfloat16), torch.zeros(n_kv, d, t_pad, device=DEV, dtype=torch.bfloat16)
    Kb[:, :T], Vt[:, :, :T] = k, v.transpose(1, 2)
    ref = _ref(q, k, v, 0).permute(1, 0, 2).reshape(T, n_q * d)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    outs = torch.zeros(150, T, n_q * d, device=DEV, dtype=torch.bfloat16)
    for out in outs:
        flush.fill_(1)
        G.flash_prefill(q, Kb, Vt, out, 0, status)
    torch.cuda.synchronize()
    assert int(status) == 0
    # probabilities (near 1 before the division) and outputs in bf16: 2^-9 of a mean of unit values each, and fp32 below it
    assert float((outs[0].float() - ref).norm() / ref.norm()) < 2 ** -7
    assert [i for i, out in enumerate(outs) if not torch.equal(out, outs[0])] == []


def test_engine_prompt_through_flash_matches_the_three_launch_path():
    """A prompt through the GEMM path with and without the fused attention: same greedy token, logits in band."""
    from bloomery_b200.models.spec import ModelSpec
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.runtime.engine import DecodeEngine
    spec = ModelSpec(arch="qwen3moe", name="flash-test", n_layer=2, hidden=512, n_q=8, n_kv=2, head_dim=128, vocab=4096,
                     ctx_train=4096, rms_eps=1e-6, rope_theta=1e6, qk_norm=True, n_expert=16, n_used=4, moe_inter=256)
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=3), "cpu").to(DEV)
    g = torch.Generator().manual_seed(2)
    prompt = torch.randint(0, spec.vocab, (333,), generator=g).tolist()
    outs = []
    for flash in (True, False):
        eng = DecodeEngine(w, n_slots=1, slot_ctx=512)
        eng._gemm_prefill = eng._new_gemm_prefill()
        eng._gemm_prefill.flash = flash
        tok = eng.prefill(0, prompt, gemm=True)
        outs.append((tok, eng.logits[0].clone()))
    scale = outs[1][1].abs().max().item()
    assert (outs[0][1] - outs[1][1]).abs().max().item() < 3e-2 * scale
    assert outs[0][0] == outs[1][0]


@pytest.mark.parametrize("n_q,n_kv,T,pos0", [(3, 1, 129, 0), (3, 1, 300, 65), (5, 1, 1, 0), (7, 7, 128, 1), (6, 2, 385, 1000), (1, 1, 640, 0)])
def test_query_tiles_that_pair_across_positions(n_q, n_kv, T, pos0):
    """An odd number of heads a KV head pairs the last tile of one position with the first of the one before it, whose keys end
    earlier, and may leave a tile alone."""
    test_flash_prefill_matches_fp32_attention(n_q, n_kv, T, pos0)


@pytest.mark.parametrize("splits", [2, 3, 4])
@pytest.mark.parametrize("n_q,n_kv,T,pos0", [(8, 2, 130, 512), (3, 1, 129, 1000), (5, 1, 1, 2048), (32, 4, 300, 3001)])
def test_query_tiles_whose_keys_are_shared(n_q, n_kv, T, pos0, splits, monkeypatch):
    """Shares of unequal length, a last share that some rows only see masked keys of, an odd tile that stays alone: the same
    rows as without shares to the rounding of one bf16 output, and the same bits on every run whoever arrives last."""
    from bloomery_b200.ops import gemm as G
    g = torch.Generator(device=DEV).manual_seed(T + splits)
    n_keys = pos0 + T
    t_pad = (n_keys + 127) // 128 * 128
    q = (torch.randn(n_q, T, 128, device=DEV, generator=g) / 128 ** 0.5).bfloat16()
    k, v = (torch.randn(n_kv, n_keys, 128, device=DEV, generator=g).bfloat16() for _ in range(2))
    k[:, n_keys // 3] *= 8                                        # a maximum that only one share holds
    Kb, Vt = torch.zeros(n_kv, t_pad, 128, device=DEV, dtype=torch.bfloat16), torch.zeros(n_kv, 128, t_pad, device=DEV, dtype=torch.bfloat16)
    Kb[:, :n_keys], Vt[:, :, :n_keys] = k, v.transpose(1, 2)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    work = G.FlashWork(DEV)
    monkeypatch.setattr(G, "flash_splits", lambda *a: splits)
    outs = torch.full((30, T, n_q * 128), float("nan"), device=DEV, dtype=torch.bfloat16)
    for out in outs:
        G.flash_prefill(q, Kb, Vt, out, pos0, status, work)
    torch.cuda.synchronize()
    assert int(status) == 0 and int(work.tickets.abs().sum()) == 0
    assert [i for i, out in enumerate(outs) if not torch.equal(out, outs[0])] == []
    ref = _ref(q, k, v, pos0).permute(1, 0, 2).reshape(T, n_q * 128)
    assert float((outs[0].float() - ref).norm() / ref.norm()) < 2 ** -7          # as without shares


@pytest.mark.parametrize("n_q,n_kv,T,pos0,splits", [(1, 1, 300, 0, 1), (3, 1, 300, 0, 1), (10, 2, 513, 70, 1), (8, 2, 300, 0, 1), (3, 1, 300, 1000, 3),
                                                    (1, 1, 129, 512, 4)])
def test_values_behind_a_row_reach_no_tile_in_front_of_theirs(n_q, n_kv, T, pos0, splits, monkeypatch):
    """An infinite value weighs zero for earlier queries, and zero times infinity is NaN: rows whose key tiles end in front of its
    tile must not meet it, whichever tile shares their CTA."""
    from bloomery_b200.ops import gemm as G
    g = torch.Generator(device=DEV).manual_seed(T)
    n_keys = pos0 + T
    t_pad = (n_keys + 127) // 128 * 128
    q = (torch.randn(n_q, T, 128, device=DEV, generator=g) / 128 ** 0.5).bfloat16()
    Kb, Vt = torch.zeros(n_kv, t_pad, 128, device=DEV, dtype=torch.bfloat16), torch.zeros(n_kv, 128, t_pad, device=DEV, dtype=torch.bfloat16)
    Kb[:, :n_keys] = torch.randn(n_kv, n_keys, 128, device=DEV, generator=g).bfloat16()
    Vt[:, :, :n_keys] = torch.randn(n_kv, 128, n_keys, device=DEV, generator=g).bfloat16()
    monkeypatch.setattr(G, "flash_splits", lambda *a: splits)
    status, outs = torch.zeros(1, dtype=torch.int32, device=DEV), []
    for bad in (False, True):
        if bad:
            Vt[:, 5, n_keys - 1] = float("inf")
        out = torch.zeros(T, n_q * 128, device=DEV, dtype=torch.bfloat16)
        G.flash_prefill(q, Kb, Vt, out, pos0, status, G.FlashWork(DEV))
        outs.append(out)
    assert int(status) == 0
    # rows of query tiles whose last key tile lies in front of the one that holds the value
    clear = [t for t in range(T) if (pos0 + min(t // 128 * 128 + 128, T) - 1) // 128 < (n_keys - 1) // 128]
    assert clear and torch.equal(outs[0][clear], outs[1][clear])
    assert bool(torch.isinf(outs[1][T - 1].view(n_q, 128)[:, 5]).all())
