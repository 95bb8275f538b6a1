"""Kernels of decode rounds and short prompts at the sizes where their tiles and splits end: the tensor-core segment pass
of decode attention, the expert plan shared by a cluster, the router of many rows, the combine with its norm."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def _fault():
    return torch.full((1,), -1, dtype=torch.int32, device=DEV)


@pytest.mark.parametrize("head,n_q,n_kv", [(128, 32, 4), (128, 8, 8), (64, 14, 2), (64, 16, 2), (128, 24, 2)])
@pytest.mark.parametrize("lengths,n_seg", [([1, 15, 16, 17, 31, 33], 3), ([64, 65, 500, 1021], 5), ([3000], 37), ([200, 7], 1)])
def test_decode_attention_against_64_bits(head, n_q, n_kv, lengths, n_seg):
    """Rows whose keys end inside a step, a tile and a page; queries of very different size per head."""
    from bloomery_b200.ops import decode as K
    g = torch.Generator().manual_seed(5)
    M, mp = len(lengths), (max(lengths) + 63) // 64
    k = torch.randn(M * mp, n_kv, 64, head, generator=g).half()
    v = torch.randn(M * mp, n_kv, 64, head, generator=g).half()
    table = torch.randperm(M * mp, generator=g).int().view(M, mp)
    q = torch.randn(M, n_q, head, generator=g) * head ** -0.5 * torch.logspace(-3, 1, n_q).view(1, n_q, 1)
    ref = torch.zeros(M, n_q * head, dtype=torch.float64)
    for m, n in enumerate(lengths):
        kk, vv = (c[table[m].long()].permute(1, 0, 2, 3).reshape(n_kv, -1, head)[:, :n].double() for c in (k, v))
        s = q[m].double().view(n_kv, n_q // n_kv, head) @ kk.transpose(1, 2)
        ref[m] = (torch.softmax(s, -1) @ vv).reshape(-1)
        if n % 64 and n_q // n_kv <= 8:                  # what lies behind the last key is never part of a sum
            k[table[m, n // 64], :, n % 64:] = float("nan")
            v[table[m, n // 64], :, n % 64:] = float("nan")
    k, v, table, q = k.to(DEV), v.to(DEV), table.contiguous().to(DEV), q.to(DEV)
    pos = torch.tensor([n - 1 for n in lengths], dtype=torch.int32, device=DEV)
    seq = torch.arange(M, dtype=torch.int32, device=DEV)
    ml = torch.zeros(M * n_q * n_seg * 2, device=DEV)
    acc = torch.zeros(M * n_q * n_seg * head, device=DEV)
    out = torch.zeros(M, n_q * head, device=DEV)
    oq = torch.zeros(M, n_q * head, dtype=torch.int8, device=DEV)
    od = torch.zeros(M, n_q * head // 32, 2, device=DEV)
    ob = torch.zeros(M, n_q * head, dtype=torch.bfloat16, device=DEV)
    f = _fault()
    K.flash_decode(q, k, v, pos, seq, table, M * mp, head, n_q, n_kv, M, n_seg, mp * 64, ml, acc, out, oq, od, f, 0)
    K.flash_decode_bf16(q, k, v, pos, seq, table, M * mp, head, n_q, n_kv, M, n_seg, mp * 64, ml, acc, ob, f, 0)
    torch.cuda.synchronize()
    assert int(f) == -1
    # scores of up to about 40 in fp32 steps of 2^-18 move a probability by as much; the exponential adds 2^-22
    assert float((out.cpu().double() - ref).norm() / ref.norm()) < 1e-5
    assert torch.equal(ob, out.bfloat16())


@pytest.mark.parametrize("head,n_q,n_kv", [(128, 32, 4), (64, 8, 8)])
def test_decode_attention_over_infinite_keys_and_values(head, n_q, n_kv):
    """f16 caches hold an infinity where a key or value left the range: a score of -inf weighs nothing, an infinite value
    stays one, and neither touches the other dimensions."""
    from bloomery_b200.ops import decode as K
    g = torch.Generator().manual_seed(6)
    n, mp, n_seg = 150, 3, 2
    k, v = (torch.randn(mp, n_kv, 64, head, generator=g).half() for _ in range(2))
    q = torch.randn(1, n_q, head, generator=g) * head ** -0.5
    q[:, :, 3] = q[:, :, 3].abs() + 0.01
    k[0, :, 7, 3] = -float("inf")
    v[1, :, 20, 5] = float("inf")
    v[2, :, 1, 9] = -float("inf")
    kk, vv = (c.permute(1, 0, 2, 3).reshape(n_kv, -1, head)[:, :n].double() for c in (k, v))
    ref = (torch.softmax(q[0].double().view(n_kv, n_q // n_kv, head) @ kk.transpose(1, 2), -1) @ vv).reshape(-1)
    table = torch.arange(mp, dtype=torch.int32, device=DEV).view(1, mp)
    pos, seq = torch.tensor([n - 1], dtype=torch.int32, device=DEV), torch.zeros(1, dtype=torch.int32, device=DEV)
    ml, acc = torch.zeros(n_q * n_seg * 2, device=DEV), torch.zeros(n_q * n_seg * head, device=DEV)
    out = torch.zeros(1, n_q * head, device=DEV)
    oq, od = torch.zeros(1, n_q * head, dtype=torch.int8, device=DEV), torch.zeros(1, n_q * head // 32, 2, device=DEV)
    K.flash_decode(q.to(DEV), k.to(DEV), v.to(DEV), pos, seq, table, mp, head, n_q, n_kv, 1, n_seg, mp * 64, ml, acc, out, oq,
                   od, _fault(), 0)
    torch.cuda.synchronize()
    out, wild = out[0].cpu().double(), ref.isinf()
    assert int(wild.sum()) == 2 * n_q and torch.equal(out[wild], ref[wild])
    assert float((out[~wild] - ref[~wild]).norm() / ref[~wild].norm()) < 1e-5       # as in the test above


@pytest.mark.parametrize("n,E,tile", [(1, 4, 32), (2048, 128, 32), (2049, 128, 128), (4100, 40, 128), (32768, 512, 128), (8192, 1, 64)])
def test_expert_plan_of_one_block_and_of_a_cluster(n, E, tile):
    from bloomery_b200.ops import gemm as G
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(-1, E, (n,), generator=g, dtype=torch.int32)
    wts = torch.rand(n, generator=g)
    tiles = G.TileTable(n, E, DEV, tile)
    cap = n + 128
    pos = torch.full((n,), -7, dtype=torch.int32, device=DEV)
    dst = torch.full((cap,), -7, dtype=torch.int32, device=DEV)
    sc = torch.zeros(cap, device=DEV)
    G.moe_plan(ids.to(DEV), wts.to(DEV), E, tiles, pos, dst, sc)
    torch.cuda.synchronize()
    counts = torch.bincount(ids[ids >= 0].long(), minlength=E)
    off = torch.cat([torch.zeros(1, dtype=torch.long), counts.cumsum(0)])
    assert torch.equal(tiles.offsets.cpu().long(), off)
    want = [(e, r, int(off[e + 1])) for e in range(E) for r in range(int(off[e]), int(off[e + 1]), tile)]
    assert int(tiles.n_mtiles) == len(want) and [tuple(r[:3]) for r in tiles.mtiles[:len(want)].tolist()] == want
    pos, dst, sc = pos.cpu().long(), dst.cpu().long(), sc.cpu()
    assert bool((pos[ids < 0] == -1).all()) and bool((dst[int(off[E]):] == -1).all())
    used = (ids >= 0).nonzero().flatten()
    assert torch.equal(dst[pos[used]], used) and torch.equal(sc[pos[used]], wts[used])
    assert bool((pos[used] >= off[ids[used].long()]).all()) and bool((pos[used] < off[ids[used].long() + 1]).all())


@pytest.mark.parametrize("t", ["F32", "F16", "BF16"])
@pytest.mark.parametrize("M,E,K", [(9, 128, 2048), (64, 128, 2048), (17, 6, 256), (127, 30, 4096)])
def test_router_of_many_rows_agrees_with_the_router(t, M, E, K):
    from bloomery_b200.ops import decode as D
    torch.manual_seed(7)
    dt = {"F32": torch.float32, "F16": torch.float16, "BF16": torch.bfloat16}[t]
    w = D.QWeight((torch.randn(E, K, device=DEV) * 0.05).to(dt).view(torch.uint8), t, K)
    x, gain = torch.randn(M, K, device=DEV) * 3, torch.rand(K, device=DEV) + 0.5
    a, b = torch.zeros(M, E, device=DEV), torch.zeros(M, E, device=DEV)
    xn = torch.zeros(M, K, dtype=torch.bfloat16, device=DEV)
    D.router(x, gain, 1e-6, w, M, a, None, None, None, _fault(), 0)
    D.router_rows(x, gain, 1e-6, w, M, b, xn)
    torch.cuda.synchronize()
    # the same sums in the same order; the compiler may contract the squares of the norm differently
    assert torch.allclose(a, b, rtol=1e-6, atol=1e-6)
    ref = x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-6) * gain
    assert torch.allclose(xn.float(), ref, rtol=2 ** -8, atol=1e-6)      # one rounding to bf16 and a few fp32 ones


@pytest.mark.parametrize("seqs", [[0, -1], [3, 1, 2, 0, 4, -1, -1, -1], [-1, 5, -1, 6], [0, 1, 2, 3]])
def test_rows_that_fill_a_bucket_route_nowhere(seqs):
    """Both calls that route: a dead row's ids are -1 and its weights 0 whatever its logits hold, it counts nowhere, the
    launch behind leaves its residual as it is, and the rows beside it keep their bits."""
    from bloomery_b200.formats.resident import quantize_resident
    from bloomery_b200.ops import decode as D
    torch.manual_seed(12)
    M, E, n, H, I_ = len(seqs), 16, 4, 512, 256
    q = [D.QWeight(quantize_resident(torch.randn(E * r, k) * 0.05, "Q4_K", values=False)[0].to(DEV).reshape(E, r, -1).contiguous(), "Q4_K", k)
         for r, k in ((I_, H), (I_, H), (H, I_))]
    wr = D.QWeight((torch.randn(E, H, device=DEV) * 0.05).view(torch.uint8), "F32", H)
    x, gain = torch.randn(M, H, device=DEV), torch.ones(H, device=DEV)
    xq, xds = torch.zeros(M, H, dtype=torch.int8, device=DEV), torch.zeros(M, H // 32, 2, device=DEV)
    logits, rule = torch.zeros(M, E, device=DEV), D.RouteRule(n)
    D.router(x, gain, 1e-6, wr, M, logits, xq, xds, None, _fault(), 0)
    seq = torch.tensor(seqs, dtype=torch.int32, device=DEV)
    dead, poison = seq < 0, logits.clone()
    poison[dead] = float("nan")

    def run(lg, row_seq, rows):
        ids, wts = torch.full((M, n), 7, dtype=torch.int32, device=DEV), torch.full((M, n), float("nan"), device=DEV)
        heat, f = torch.zeros(E, dtype=torch.int32, device=DEV), _fault()
        actq = torch.full((M, n, I_), 99, dtype=torch.int8, device=DEV)
        actds = torch.full((M, n, I_ // 32, 2), float("nan"), device=DEV)
        y = torch.full((M, H), float("nan"), device=DEV)
        if rows:
            D.route_rows(lg, rule, M, ids, wts, heat, f, 0, row_seq)
        else:
            D.gate_up_sel(xq, xds, ids, None, q[0], q[1], E, n, M, actq, actds, None, f, 0, route_logits=lg, rule=rule, wts=wts,
                          heat=heat, row_seq=row_seq)
            D.down_combine(actq, actds, ids, wts, None, q[2], E, n, M, x, None, y, f, 0)
        torch.cuda.synchronize()
        assert int(f) == -1
        return ids, wts, heat, y

    for rows in (True, False):
        ids, wts, heat, y = run(logits, None, rows)              # every row alive
        got = run(poison, seq, rows)
        assert bool((got[0][dead] == -1).all()) and bool((got[1][dead] == 0).all())
        assert torch.equal(got[0][~dead], ids[~dead]) and torch.equal(got[1][~dead], wts[~dead])
        assert torch.equal(got[2].long(), torch.bincount(ids[~dead].flatten().long(), minlength=E))
        if not rows:
            assert torch.equal(got[3][dead], x[dead]) and torch.equal(got[3][~dead], y[~dead])


@pytest.mark.parametrize("T,k,H", [(1, 8, 2048), (33, 2, 4), (5, 3, 8192), (7, 8, 1028)])
def test_combine_with_the_next_norm(T, k, H):
    from bloomery_b200.ops import gemm as G
    torch.manual_seed(8)
    slot, x, gain = torch.randn(T * k, H, device=DEV), torch.randn(T, H, device=DEV), torch.rand(H, device=DEV) + 0.5
    pos = torch.arange(T * k, dtype=torch.int32, device=DEV)
    pos[::5] = -1
    slot[::5] = float("nan")                                             # dropped slots are not read
    y, z = torch.zeros(T, H, device=DEV), x.clone()
    xn = torch.zeros(T, H, dtype=torch.bfloat16, device=DEV)
    G.moe_combine(slot, pos, T, k, x, y)
    G.moe_combine_norm(slot, pos, T, k, z, z, gain, 1e-6, xn)            # in place, as the layers use it
    torch.cuda.synchronize()
    assert torch.equal(y, z)
    ref = y * torch.rsqrt(y.pow(2).mean(-1, keepdim=True) + 1e-6) * gain
    assert torch.allclose(xn.float(), ref, rtol=2 ** -8, atol=1e-6)


@pytest.mark.parametrize("n,start", [(12, 0), (33, 0), (64, 40), (100, 3), (128, 0), (129, 0)])
def test_short_prompts_over_quantised_blocks_agree_with_the_bf16_copies(n, start):
    from bloomery_b200.models.spec import tiny_qwen3moe
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.runtime.engine import DecodeEngine
    spec = tiny_qwen3moe()
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=0), "cpu").to(DEV)
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(0, spec.vocab, (start + n,), generator=g).tolist()
    out = []
    for rows in (128, 0):
        eng = DecodeEngine(w, n_slots=1, slot_ctx=512)
        eng._gemm_prefill = eng._new_gemm_prefill()
        eng._gemm_prefill.direct_rows = rows
        eng._gemm_prefill.resident_bf16 = rows == 0              # the blocks are for prompts without kept copies, or short ones
        assert eng._gemm_prefill._direct(n, short=n < 64) == (n <= rows)
        if start:
            eng.prefill(0, ids[:start], gemm=False)
        eng.prefill(0, ids[start:], start, gemm=True)
        out.append(eng.logits[0].double().cpu())
    # the same bf16 operands, their fp32 sums in another order: a layer's roundings to bf16 differ in places, four layers deep
    assert float((out[0] - out[1]).norm() / out[1].norm()) < 2e-2


@pytest.mark.parametrize("kept", [False, True])
@pytest.mark.parametrize("n", [129, 256, 257, 600])
def test_experts_over_blocks_beside_bf16_projections_agree_with_the_copies(n, kept):
    """Prompts on either side of the last one whose experts take their blocks (16 experts, 4 of them a row, 64 rows each: 256),
    with copies that are kept and without, and a longer prompt behind a shorter one, which completes the copies; 600 ids
    are products of CTA pairs."""
    from bloomery_b200.models.spec import tiny_qwen3moe
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.runtime.engine import DecodeEngine
    spec = tiny_qwen3moe()
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=0), "cpu").to(DEV)
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(0, spec.vocab, (n,), generator=g).tolist()
    out = []
    for rows in (128, 0):
        eng = DecodeEngine(w, n_slots=2, slot_ctx=768)
        pre = eng._gemm_prefill = eng._new_gemm_prefill()
        pre.direct_rows, pre.resident_bf16 = rows, kept
        pre.pair_rows = 128 if rows else 1 << 20
        assert pre._expert_blocks(n) == (rows > 0 and n <= 256)
        eng.prefill(1, ids[:140], gemm=True)
        eng.prefill(0, ids, gemm=True)
        out.append(eng.logits[0].double().cpu())
    # the same bf16 operands, their fp32 sums in another order, four layers deep (as above)
    assert float((out[0] - out[1]).norm() / out[1].norm()) < 2e-2


@pytest.mark.parametrize("rows", [1 << 30, 200, 1])
def test_a_prompt_has_a_table_for_pairs_where_a_projection_goes_to_them(monkeypatch, rows):
    """The 256-row table is written by the host, two blocking copies in front of the first layer: prompts below the products that
    pairs pay for do without it."""
    from bloomery_b200.models.spec import tiny_qwen3moe
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.ops import gemm as G
    from bloomery_b200.runtime.engine import DecodeEngine
    spec = tiny_qwen3moe()
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=0), "cpu").to(DEV)
    made, dense = [], G.TileTable.dense
    monkeypatch.setattr(G.TileTable, "dense", lambda n, dev, tile_rows=128, host=False: made.append(tile_rows) or dense(n, dev, tile_rows, host))
    monkeypatch.setattr(G, "pairs_pay", lambda n, width: n >= rows)
    eng = DecodeEngine(w, n_slots=1, slot_ctx=512)
    for n in (140, 300):
        made.clear()
        eng.prefill(0, list(range(n)), gemm=True)
        assert (G.PAIR_ROWS in made) == (n >= rows), (n, rows, made)


@pytest.mark.parametrize("n", [257, 600])
def test_projections_on_pairs_of_ctas_agree_with_single_ones(monkeypatch, n):
    """QKV and the output projection, which adds to the residual rows in place, of a prompt of two and of three tiles of 256 rows."""
    from bloomery_b200.models.spec import tiny_qwen3moe
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.ops import gemm as G
    from bloomery_b200.runtime.engine import DecodeEngine
    spec = tiny_qwen3moe()
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=0), "cpu").to(DEV)
    ids = torch.randint(0, spec.vocab, (n,), generator=torch.Generator().manual_seed(n)).tolist()
    calls, pair = [], G.gemm_pair
    monkeypatch.setattr(G, "gemm_pair", lambda X, W, tiles, **kw: calls.append((W.shape[0], kw.get("resid") is not None)) or pair(X, W, tiles, **kw))
    out = []
    for pays in (True, False):
        monkeypatch.setattr(G, "pairs_pay", lambda rows, width: pays)
        eng = DecodeEngine(w, n_slots=1, slot_ctx=768)
        pre = eng._gemm_prefill = eng._new_gemm_prefill()
        pre.pair_rows = 1 << 20                                  # experts on single CTAs in both
        calls.clear()
        eng.prefill(0, ids, gemm=True)
        widths = [(spec.q_rows + 2 * spec.kv_rows, False), (spec.hidden, True)]
        assert calls == (widths * spec.n_layer if pays else [])
        out.append(eng.logits[0].double().cpu())
    # the same bf16 operands, their fp32 sums in another order, four layers deep (as above)
    assert float((out[0] - out[1]).norm() / out[1].norm()) < 2e-2


def test_prompts_run_where_only_the_projections_copies_found_room():
    """A prompt over the experts' blocks that keeps the projections' copies, then one that needs the experts' and is refused them: the
    bits of prompts that keep nothing."""
    from bloomery_b200.models.spec import tiny_qwen3moe
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.runtime.engine import DecodeEngine
    spec = tiny_qwen3moe()
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=0), "cpu").to(DEV)
    ids = torch.randint(0, spec.vocab, (600,), generator=torch.Generator().manual_seed(7)).tolist()
    out = []
    for room in (True, False):
        eng = DecodeEngine(w, n_slots=2, slot_ctx=768)
        pre = eng._gemm_prefill = eng._new_gemm_prefill()
        pre._resident_ok, pre._resident_experts_ok = room, False
        for slot, n in ((0, 140), (1, 600), (0, 200)):
            eng.prefill(slot, ids[:n], gemm=True)
            out.append(eng.logits[0].clone())
        assert ("wqkv" in pre._resident.get(0, {})) == room and "wg" not in pre._resident.get(0, {})
    assert all(torch.equal(a, b) for a, b in zip(out[:3], out[3:]))


@pytest.mark.parametrize("n", [32, 33, 63])
@pytest.mark.parametrize("mix", ["Q4_K_M", "NVFP4"])
def test_prompts_below_the_gemm_threshold_round_activations_and_nothing_else(n, mix):
    """Keys and values behind the first layer against the fp32 oracle.  The bf16 copies round weights, queries,
    probabilities, keys and values as well, the chain rounds activations to eight bits."""
    from bloomery_b200.models.cpu_ref import CpuModel
    from bloomery_b200.models.spec import tiny_qwen3moe
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.runtime.engine import DecodeEngine
    spec = tiny_qwen3moe()
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=0, mix=mix), "cpu")
    g = torch.Generator().manual_seed(n)
    ids = torch.randint(0, spec.vocab, (n,), generator=g)
    oracle = CpuModel(w, quantize_acts=False)
    oracle.forward(ids)
    w = w.to(DEV)
    err = {}
    for route in ("chain", "blocks", "copies"):
        eng = DecodeEngine(w, n_slots=1, slot_ctx=512)
        eng._gemm_prefill = eng._new_gemm_prefill()
        eng._gemm_prefill.direct_rows = 128 if route == "blocks" else 0
        assert eng._gemm_prefill._direct(n, short=True) == (route == "blocks")
        eng.prefill(0, ids.tolist(), gemm=route != "chain")
        pages = torch.tensor(eng.kv.pages[0], device=DEV)
        new = [c[1, pages].permute(0, 2, 1, 3).reshape(-1, spec.n_kv, spec.head_dim)[:n].float().cpu()
               for c in (eng.kv.k, eng.kv.v)]
        want = [oracle.k[1], oracle.v[1]]
        # a median over the rows: where two experts are all but equal, one rounding chooses another
        err[route] = float(torch.stack([((a - b).flatten(1).norm(dim=1) / b.flatten(1).norm(dim=1)).median()
                                        for a, b in zip(new, want)]).mean())
    # rounding weights and activations alike adds 1.41 times what activations alone add
    assert err["blocks"] < 0.85 * err["copies"] and err["blocks"] < 0.5 * err["chain"], err


def test_a_short_prompt_leaves_the_logits_of_its_last_rows_unless_the_server_feeds_it():
    from bloomery_b200.models.spec import tiny_qwen3moe
    from bloomery_b200.models.weights import Weights, synth_tensors
    from bloomery_b200.runtime.engine import DecodeEngine
    from bloomery_b200.serve.engine import GpuEngine
    from bloomery_b200.serve.tokenizer import ByteTokenizer
    spec = tiny_qwen3moe()
    w = Weights.from_items(spec, synth_tensors(spec, "cpu", seed=0), "cpu").to(DEV)
    g = torch.Generator().manual_seed(9)
    ids = torch.randint(0, spec.vocab, (45,), generator=g).tolist()
    eng = [DecodeEngine(w, n_slots=2, slot_ctx=256) for _ in range(2)]
    first = eng[0].prefill(0, ids), eng[1].prefill(0, ids, gemm=False)
    assert first[0] == first[1] and torch.equal(eng[0].logits[:5], eng[1].logits[:5])
    GpuEngine(eng[0], ByteTokenizer(), "m").prefill(1, ids, 0)
    eng[1].prefill(1, ids, gemm=True)
    rows = [e.kv.k[:, e.kv.pages[1][0], :, :45] for e in eng]
    assert torch.equal(*rows)
    assert not torch.equal(rows[0], eng[0].kv.k[:, eng[0].kv.pages[0][0], :, :45])


@pytest.mark.parametrize("E,k", [(32, 8), (64, 1), (128, 8), (256, 16), (96, 4)])
def test_routing_by_a_warp_a_row(E, k):
    """Rows of many ties, of zeros of both signs, of one finite huge value, and one row that is not finite, against a stable
    sort of the same logits (96 experts take the block's counting)."""
    from bloomery_b200.ops import decode as D
    g = torch.Generator().manual_seed(E)
    M = 19
    lg = torch.randn(M, E, generator=g)
    lg[1] = 0.0
    lg[2] = torch.where(torch.rand(E, generator=g) < 0.5, 0.0, -0.0)
    lg[3] = torch.randint(-2, 3, (E,), generator=g).float()
    lg[4] = -torch.arange(E).float() - 1e30
    lg[5, E - 1] = 3e38
    lg[6] = -3.4028234663852886e38
    lg[17, E // 2] = float("nan")
    ids = torch.full((M, k), 7, dtype=torch.int32, device=DEV)
    wts, heat, f = torch.full((M, k), 9.0, device=DEV), torch.zeros(E, dtype=torch.int32, device=DEV), _fault()
    seq = torch.zeros(M, dtype=torch.int32, device=DEV)
    seq[18] = -1
    D.route_rows(lg.to(DEV), D.RouteRule(k), M, ids, wts, heat, f, 3, seq)
    torch.cuda.synchronize()
    assert int(f) != -1 and (int(f) >> 8) == 3                   # the row that is not finite
    live = [m for m in range(M) if m not in (17, 18)]
    order = torch.sort(lg[live], dim=1, descending=True, stable=True)
    assert torch.equal(ids.cpu()[live].long(), order.indices[:, :k])
    want = torch.softmax(order.values[:, :k].double(), 1)
    assert torch.allclose(wts.cpu()[live].double(), want, rtol=1e-5, atol=1e-7)
    assert bool(wts[17].isnan().all()) and bool((ids[17] == 0).all())
    assert bool((ids[18] == -1).all()) and bool((wts[18] == 0).all())
    assert torch.equal(heat.cpu().long(), torch.bincount(order.indices[:, :k].flatten(), minlength=E))


@pytest.mark.parametrize("head,n_q,n_kv", [(128, 32, 4), (128, 1, 1), (64, 14, 2), (128, 40, 8), (64, 37, 1)])
def test_prompt_rows_are_normed_and_rotated_as_decode_rows_are(head, n_q, n_kv):
    """Cached keys and values bit for bit those of the decode launch, queries its fp32 rows rounded to bf16, for numbers of
    heads that the warps' groups divide and do not."""
    from bloomery_b200.ops import decode as D
    from bloomery_b200.ops import gemm as G
    g = torch.Generator(device=DEV).manual_seed(head + n_q)
    T, n_pages = 9, 4
    qkv = torch.randn(T, (n_q + 2 * n_kv) * head, device=DEV, generator=g)
    qg, kg = (1 + 0.1 * torch.randn(head, device=DEV, generator=g) for _ in range(2))
    inv = (1.0 / (1e6 ** (torch.arange(0, head, 2, dtype=torch.float64) / head))).float().to(DEV)
    pos = torch.tensor([0, 1, 63, 64, 65, 127, 128, 190, 200], dtype=torch.int32, device=DEV)
    seq = torch.zeros(T, dtype=torch.int32, device=DEV)
    table = torch.tensor([[2, 0, 3, 1]], dtype=torch.int32, device=DEV)
    caches = [[torch.zeros(n_pages, n_kv, 64, head, dtype=torch.float16, device=DEV) for _ in range(2)] for _ in range(2)]
    q32 = torch.zeros(T, n_q, head, device=DEV)
    qbf = torch.zeros(n_q, T, head, device=DEV, dtype=torch.bfloat16)
    f = _fault()
    D.qk_norm_rope_append(qkv, qg, kg, inv, 1e-6, 0.125, head, n_q, n_kv, T, pos, seq, table, n_pages, *caches[0], q32, f, 0)
    G.qk_norm_rope_append_prefill(qkv, qg, kg, inv, 1e-6, 0.125, head, n_q, n_kv, T, pos, seq, table, n_pages, *caches[1], qbf, f, 0)
    torch.cuda.synchronize()
    assert int(f) == -1
    assert torch.equal(caches[0][0], caches[1][0]) and torch.equal(caches[0][1], caches[1][1])
    assert torch.equal(q32.bfloat16().transpose(0, 1), qbf)
