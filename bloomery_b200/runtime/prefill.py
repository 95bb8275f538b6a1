"""Prompt (prefill) path on the tcgen05 GEMM: whole micro-batches of prompt rows per layer
instead of 8-row passes.

Counterpart of the reference's GEMM ubatches (``crates/gpu/src/arch/qwen3moe/ubatch.rs:1-40``:
per layer norm -> QKV GEMM -> norm/RoPE/append -> prefill flash -> o GEMM -> router logits +
route -> grouped gate/up GEMM with SwiGLU -> grouped down GEMM -> combine).  Here:

  * short micro-batches multiply the quantised blocks as they are, the routed experts of longer ones too up to some rows an
    expert (``direct_rows``, ``block_rows``); other products read bf16 copies of the weights, which are kept between prompts
    where memory allows, else expanded a layer ahead on a side stream (one expander kernel per matrix);
  * products over copies are persistent TMA + tcgen05 kernels, on single CTAs or pairs of them; gate and up run in one main
    loop with SwiGLU in the epilogue; the down GEMM's epilogue scatters router-weighted rows to
    their (token, slot) cell and a fixed-order combine adds slots in ascending order;
  * attention is one launch (``csrc/flash_tcgen05.cu``) for heads of 128; other head sizes take three per query chunk: Q K^T
    (grouped over heads, KV head shared by its query heads), causal softmax, P V (epilogue writes token-major rows).

Token bits are not equal to the 8-row pass path (bf16 operands, different sum order); a
band test covers it, as the reference does (``ubatch.rs:19-30``).
"""
from __future__ import annotations

import math
from typing import List, Optional, Sequence

import os

import torch

from ..ops import decode as K
from ..ops import gemm as G
from .engine import GEMM_THRESHOLD
from .kv import PAGE

PROCESSORS = 148       # of a B200

POISON = None          # None: follow the BLOOMERY_POISON lever; tests set True / False


def _poison() -> bool:
    if POISON is not None:
        return bool(POISON)
    from ..utils import levers
    return bool(levers.get("BLOOMERY_POISON"))


class GemmPrefill:
    def __init__(self, engine, ubatch: int = 2048, score_bytes: int = 1 << 30):
        self.e = engine
        self.ubatch = ubatch
        self.score_bytes = score_bytes
        self._buf = {}
        self._router_w = {}
        self.status = torch.zeros(1, dtype=torch.int32, device=engine.device)
        self.launches = 0
        # where a layer's expert stacks come from: the resident weights, or a streamer that brings them from the host
        self.expert_source = None
        self.expand_ahead = True                # bf16 expansion of layer l + 1's weights on a side stream during layer l
        self._side = None
        self.flash = True                       # head size 128: fused attention on tensor memory (csrc/flash_tcgen05.cu)
        # Resident bf16 copy of every layer's matrices, built by the first prompt that multiplies them (58 GB for a 30 B-parameter
        # mixture beside its 17 GB of Q4_K_M blocks, 56 of them the routed experts'): later prompts skip the expansion launches
        # altogether.  None = only when the copy leaves a quarter of the card free; True / False force it.
        from ..utils import levers
        self.resident_bf16 = {"1": True, "0": False}.get(str(levers.get("BLOOMERY_PREFILL_BF16")), None)
        self._resident = {}
        self._resident_ok = self._resident_experts_ok = None
        from .timing import PromptTiming
        self.timing = PromptTiming()            # arm() it to get per-unit milliseconds of the next micro-batch
        # Micro-batches of at most this many tokens multiply the block-quantised weights as they are (csrc/qgemm_tcgen05.cu)
        # where every prompt would have to expand them to bf16 first: a layer of the 30 B shape is 0.35 GB of blocks and 1.2 GB
        # of copies that are written and read.  Eight layers, 64 / 128 tokens, milliseconds: Q4_K_M 3.1 / 4.1 over the blocks,
        # 6.0 / 5.8 with the expansion; FP8 3.3 / 4.3 and 9.9 / 10.1; NVFP4 3.6 / 4.6 and 6.2 / 6.5.  With copies that
        # are kept, the blocks serve every product of the prompts below GEMM_THRESHOLD, which need their bits (run); above it only
        # the experts' (block_rows), the projections read their copies (3.2 to 3.6 / 3.5 with copies alone in all three).
        # (0: no micro-batch multiplies blocks.)
        self.direct_rows = 128
        # Experts alone take their blocks further, copies or not, up to this many rows an expert on average: the products are then
        # bound by what they read, and the blocks are a quarter of the copies, or half.  Types of gate and up whose expander
        # keeps up with that; NVFP4 and Q8_0 do not.  Gate+up and down of the 30 B shape, us a layer:
        #            copies     Q4_K       Q5_K       Q6_K       FP8        Q8_0       NVFP4
        #   160 ids  154 + 66   109 + 57   122 + 61   128 + 61   129 + 65   177 + 76   151 + 83
        #   700      157 + 73   117 + 61   130 + 65   136 + 66   136 + 71   185 + 79   158 + 87
        #   832      159 + 75   117 + 65   131 + 70   136 + 69   136 + 75   186 + 83   158 + 92
        #   1,000    159 + 77   149 + 83   168 + 90   174 + 89   173 + 93   235 + 104  201 + 116
        # (whole prompts in Q4_K_M, blocks / copies: 900 ids 20.3 / 21.3 ms, 960 21.2 / 21.5, 1,000 22.3 / 21.6).  A down stack of any
        # type costs less than gate and up save up to 52 rows an expert, beyond them only one that is in the table.  What ends
        # the blocks' lead is a second 64-row tile of many experts, for which their weights are expanded again.  Where two tiles of every
        # expert find a processor at once that takes no longer, so stacks that small go up to 64 rows in every type of the table
        # (16 experts of 256 x 512, 256 ids, whole prompts, us, blocks / copies: Q4_K 1,565 / 1,671, kept copies 1,265 / 1,252; FP8 1,557 /
        # 1,677 and 1,262 / 1,261).
        self.block_rows = {"Q4_K": 60, "Q5_K": 52, "Q6_K": 52, "FP8_B128": 52}
        self.block_rows_any_down = 52
        # From this many rows an expert on, products over the copies go to pairs of CTAs with 256-row tiles (gate+up and down, us a
        # layer, pairs / single CTAs: 1,000 ids 263 / 246, 2,048 ids 287 / 288, 4,096 ids 433 / 440; whole prompts with the projections on
        # single CTAs in both, ms: 2,000 ids 27.6 / 27.6, 2,700 33.9 / 34.9, 4,096 47.0 / 47.5, and with them on pairs too 27.4,
        # 33.5, 46.4).
        self.pair_rows = 128
        self._direct_ok = None
        self._block_limit = None
        self._work = None
        self._flash_work = G.FlashWork(engine.device)

    def _get(self, name: str, shape, dtype) -> torch.Tensor:
        n = 1
        for d in shape:
            n *= d
        b = self._buf.get(name)
        if b is None or b.numel() < n or b.dtype != dtype:
            b = torch.empty(n, dtype=dtype, device=self.e.device)
            if _poison():                   # scratch starts as NaN / -1: a read of something never written shows at once
                b.fill_(float("nan") if dtype.is_floating_point else -1)
            self._buf[name] = b
        return b[:n].view(*shape)

    def run(self, slot: int, tokens: Sequence[int], start: int = 0) -> None:
        """Append ``tokens`` at positions start.. of ``slot``; leaves the last row's hidden
        state in ``engine.x[0]`` (the caller runs the head)."""
        e = self.e
        n = len(tokens)
        e.kv.ensure(slot, start + n)
        for p in range(start, start + n, PAGE):
            e.kv.own(slot, p)
        e.kv.sync_table()
        # A prompt that would run on the 8-row chain if it were not here keeps what the chain gives it: weights that are not
        # rounded to bf16 (value and remainder) and queries, probabilities, keys and values as decode attention has them.
        fine = n < GEMM_THRESHOLD and self._direct(n, short=True)
        i = 0
        while i < n:
            chunk = tokens[i:i + self.ubatch]
            self._ubatch(slot, chunk, start + i, fine)
            i += len(chunk)
        e.slot_len[slot] = max(e.slot_len[slot], start + n)

    def _ubatch(self, slot: int, tokens: Sequence[int], p0: int, fine: bool = False) -> None:
        e = self.e
        s, w, dev = e.spec, e.w, e.device
        T = len(tokens)
        H, V = s.hidden, s.vocab
        bf, f32, i32 = torch.bfloat16, torch.float32, torch.int32
        tok = torch.tensor(list(tokens), dtype=i32, device=dev)
        row_pos = torch.arange(p0, p0 + T, dtype=i32, device=dev)
        row_seq = torch.full((T,), slot, dtype=i32, device=dev)
        x = self._get("x", (T, H), f32)
        xn = self._get("xn", (T, H), bf)
        K.embed_rows(tok, T, w.q["token_embd.weight"], V, x, e.fault)
        qkv_w = s.q_rows + 2 * s.kv_rows
        qkv = self._get("qkv", (T, qkv_w), f32)
        # Quantised weights are expanded to bf16 one layer AHEAD of their use, on a side stream: the expansion is bound
        # by HBM traffic, the products by the tensor cores, so the two overlap.  Two sets of bf16 buffers alternate.
        direct = fine or self._direct(T)
        blocks = direct or self._expert_blocks(T)           # the routed experts' weights are multiplied as they are
        resident = not direct and self._use_resident(experts=not blocks)
        ahead = self.expert_source is None and self.expand_ahead and not resident and not direct
        nset = 2 if ahead else 1
        wqkv_s = [None if direct else self._get(f"wqkv{i}", (qkv_w, H), bf) for i in range(nset)]
        wo_s = [None if direct else self._get(f"wo{i}", (H, s.q_rows), bf) for i in range(nset)]
        form = dict(fine=True) if fine else dict(exact=True)
        if fine:
            # key segments as in a decode round: about eight blocks a processor
            n_seg = max(1, min(e.n_seg, 8 * K.sm_count(dev) // (s.n_kv * T)))
            q_rows = self._get("q_rows", (T, s.n_q, s.head_dim), f32)
            part_ml = self._get("part_ml", (T * s.n_q * n_seg * 2,), f32)
            part_acc = self._get("part_acc", (T * s.n_q * n_seg * s.head_dim,), f32)
        else:
            q_bf = self._get("q_bf", (s.n_q, T, s.head_dim), bf)
        attn = self._get("attn", (T, s.q_rows), bf)
        if direct:
            dense_tiles = G.TileTable.dense(T, dev, 32 if T <= 32 else 64 if T <= 64 else 128, host=True)
            if self._work is None:
                self._work = G.QgemmWork(dev, 128)
        else:
            dense_tiles = G.TileTable.dense(T, dev, host=True)
            on_pairs = {n for n in (qkv_w, H) if G.pairs_pay(T, n)}       # widths of the projections that go to pairs of CTAs
            pair_tiles = G.TileTable.dense(T, dev, G.PAIR_ROWS, host=True) if on_pairs else None

        def project(X, W, **out):
            """A dense product over a bf16 copy."""
            if W.shape[0] in on_pairs:
                G.gemm_pair(X, W, pair_tiles, status=self.status, **out)
            else:
                G.gemm_bf16(X, W, dense_tiles, status=self.status, **out)
        n_keys = p0 + T
        T_pad = (n_keys + 127) // 128 * 128
        if not fine:
            Kb = self._get("Kb", (s.n_kv, T_pad, s.head_dim), bf)
            Vt = self._get("Vt", (s.n_kv, s.head_dim, T_pad), bf)
        Tq_max = max(128, min(T, self.score_bytes // (s.n_q * T_pad * 4) // 128 * 128))
        Gq = s.n_q // s.n_kv
        if s.is_moe:
            E, I_, k = s.n_expert, s.moe_inter, s.n_used
            nslot = T * k
            cap = nslot + 128
            wg_s = [None if blocks else self._get(f"wg{i}", (E, I_, H), bf) for i in range(nset)]
            wu_s = [None if blocks else self._get(f"wu{i}", (E, I_, H), bf) for i in range(nset)]
            wd_s = [None if blocks else self._get(f"wd{i}", (E, H, I_), bf) for i in range(nset)]
            logits = self._get("rl", (T, E), f32)
            xn3 = self._get("xn3", (T, 3 * H), bf)
            ids = self._get("ids", (T, k), i32)
            wts = self._get("wts", (T, k), f32)
            counts = self._get("counts", (E,), i32)
            cursor = self._get("cursor", (E,), i32)
            pos_of = self._get("pos_of", (nslot,), i32)
            dst_row = self._get("dst_row", (cap,), i32)
            row_scale = self._get("row_scale", (cap,), f32)
            Ap = self._get("Ap", (cap, H), bf)
            act = self._get("act", (cap, I_), bf)
            slot_out = self._get("slot_out", (nslot, H), f32)
            pairs = not blocks and nslot >= self.pair_rows * E
            moe_tiles = G.TileTable(nslot, E, dev, (32 if direct or nslot <= 8 * E else 64) if blocks else G.PAIR_ROWS if pairs else G.BM)
        if s.dense_inter and (s.first_dense > 0 or not s.is_moe):
            Id = s.dense_inter
            dg_s = [self._get(f"dg{i}", (Id, H), bf) for i in range(nset)]
            du_s = [self._get(f"du{i}", (Id, H), bf) for i in range(nset)]
            dd_s = [self._get(f"dd{i}", (H, Id), bf) for i in range(nset)]
            dact = self._get("dact", (T, Id), bf)
        st = self.status

        def expand(il: int, which: str) -> None:
            """bf16 copies of layer il's weights into buffer set il % nset: 'attn', 'gate_up', 'down', 'experts' (both) or 'all'.
            Routed experts whose blocks are multiplied as they are have none."""
            b = f"blk.{il}."
            i = il % nset
            if which in ("attn", "all"):
                G.dequant_bf16(w.q[b + "attn_q.weight"], wqkv_s[i][:s.q_rows])
                G.dequant_bf16(w.q[b + "attn_k.weight"], wqkv_s[i][s.q_rows:s.q_rows + s.kv_rows])
                G.dequant_bf16(w.q[b + "attn_v.weight"], wqkv_s[i][s.q_rows + s.kv_rows:])
                G.dequant_bf16(w.q[b + "attn_output.weight"], wo_s[i])
            if s.layer_is_moe(il):
                if blocks:
                    return
                if self.expert_source is not None:
                    qg, qu, qd = self.expert_source(il)
                else:
                    qg, qu, qd = (w.q[b + f"ffn_{n}_exps.weight"] for n in ("gate", "up", "down"))
                if which in ("gate_up", "experts", "all"):
                    G.dequant_bf16(qg, wg_s[i])
                    G.dequant_bf16(qu, wu_s[i])
                if which in ("down", "experts", "all"):
                    G.dequant_bf16(qd, wd_s[i])
            else:
                if which in ("gate_up", "all"):
                    G.dequant_bf16(w.q[b + "ffn_gate.weight"], dg_s[i])
                    G.dequant_bf16(w.q[b + "ffn_up.weight"], du_s[i])
                if which in ("down", "all"):
                    G.dequant_bf16(w.q[b + "ffn_down.weight"], dd_s[i])

        main = torch.cuda.current_stream(dev)
        if ahead:
            if self._side is None:
                self._side = torch.cuda.Stream(device=dev)
            side = self._side
            ready = [torch.cuda.Event() for _ in range(s.n_layer)]
            freed = [torch.cuda.Event() for _ in range(s.n_layer)]
            side.wait_stream(main)
            with torch.cuda.stream(side):
                expand(0, "all")
                ready[0].record(side)
        normed = False                          # xn holds the layer's normed rows already
        for il in range(s.n_layer):
            b = f"blk.{il}."
            self.timing.mark(il, "ffn")
            i = il % nset
            wqkv, wo = wqkv_s[i], wo_s[i]
            if s.is_moe:
                wg, wu, wd = wg_s[i], wu_s[i], wd_s[i]
            if s.dense_inter and (s.first_dense > 0 or not s.is_moe):
                dg, du, dd = dg_s[i], du_s[i], dd_s[i]
            if resident:
                hit = self._resident.setdefault(il, {})
                moe = s.layer_is_moe(il)
                if "wqkv" not in hit or (moe and not blocks and "wg" not in hit):
                    # first use of this layer (of its experts): expand into the shared scratch as always, then keep a copy
                    expand(il, "all" if "wqkv" not in hit else "experts")
                    if "wqkv" not in hit:
                        hit.update(wqkv=wqkv.clone(), wo=wo.clone())
                    if not moe:
                        hit.update(dg=dg.clone(), du=du.clone(), dd=dd.clone())
                    elif not blocks:
                        hit.update(wg=wg.clone(), wu=wu.clone(), wd=wd.clone())
                wqkv, wo = hit["wqkv"], hit["wo"]
                if moe:
                    wg, wu, wd = hit.get("wg"), hit.get("wu"), hit.get("wd")
                else:
                    dg, du, dd = hit["dg"], hit["du"], hit["dd"]
            if ahead:
                if il + 1 < s.n_layer:
                    with torch.cuda.stream(side):
                        if il >= 1:
                            side.wait_event(freed[il - 1])          # the set's previous user (layer il - 1) is done with it
                        expand(il + 1, "all")
                        ready[il + 1].record(side)
                main.wait_event(ready[il])
            if not normed:
                G.rmsnorm_bf16(x, w.f[b + "attn_norm.weight"], s.rms_eps, xn)
            normed = False
            if direct:
                lo = 0
                for nm in ("attn_q", "attn_k", "attn_v"):
                    wq = w.q[b + nm + ".weight"]
                    G.qgemm(xn, wq, dense_tiles, out_f32=qkv[:, lo:lo + wq.rows], status=st, work=self._work, **form)
                    lo += wq.rows
            else:
                if not ahead and not resident:
                    expand(il, "attn")
                project(xn, wqkv, out_f32=qkv)
            self.timing.mark(il, "qkv_gemm")
            if fine:
                K.qk_norm_rope_append(qkv, w.f.get(b + "attn_q_norm.weight"), w.f.get(b + "attn_k_norm.weight"), e.inv_freq,
                                      s.rms_eps, e.attn_scale, s.head_dim, s.n_q, s.n_kv, T, row_pos, row_seq, e.kv.table,
                                      e.kv.n_pages, e.kv.k[il], e.kv.v[il], q_rows, e.fault, il)
                self.timing.mark(il, "rope_append")
                K.flash_decode_bf16(q_rows, e.kv.k[il], e.kv.v[il], row_pos, row_seq, e.kv.table, e.kv.n_pages, s.head_dim,
                                    s.n_q, s.n_kv, T, n_seg, e.slot_ctx, part_ml, part_acc, attn, e.fault, il)
                self.timing.mark(il, "flash")
            else:
                G.qk_norm_rope_append_prefill(qkv, w.f.get(b + "attn_q_norm.weight"), w.f.get(b + "attn_k_norm.weight"),
                                              e.inv_freq, s.rms_eps, 1.0 / math.sqrt(s.head_dim), s.head_dim, s.n_q, s.n_kv,
                                              T, row_pos, row_seq, e.kv.table, e.kv.n_pages, e.kv.k[il], e.kv.v[il], q_bf,
                                              e.fault, il)
                self.timing.mark(il, "rope_append")
                G.kv_gather_bf16(e.kv.k[il], e.kv.v[il], e.kv.table[slot], e.kv.n_pages, s.n_kv, s.head_dim, n_keys, T_pad,
                                 Kb, Vt)
                self.timing.mark(il, "qkv")
                if s.head_dim == 128 and self.flash:
                    # scores, softmax and values in one tcgen05 launch: the score matrix stays in tensor memory
                    G.flash_prefill(q_bf, Kb, Vt, attn, p0, st, self._flash_work)
                    self.timing.mark(il, "flash")
                for c0 in range(0, T if not (s.head_dim == 128 and self.flash) else 0, Tq_max):
                    Tq = min(Tq_max, T - c0)
                    rows = s.n_q * Tq
                    S = self._get("S", (rows, T_pad), f32)
                    P = self._get("P", (rows, T_pad), bf)
                    qk_tiles, pv_tiles, map_s, map_o = self._attn_tables(T, Tq, c0, s.n_q, Gq, p0)
                    G.gemm_bf16(q_bf.view(s.n_q * T, s.head_dim), Kb, qk_tiles, out_f32=S, dst_row=map_s, status=st)
                    self.timing.mark(il, "scores")
                    G.softmax_causal(S, rows, Tq, p0 + c0, T_pad, P)
                    self.timing.mark(il, "softmax")
                    G.gemm_bf16(P, Vt, pv_tiles, out_bf16=attn.view(T * s.n_q, s.head_dim), dst_row=map_o, status=st)
                    self.timing.mark(il, "values")
            self.timing.mark(il, "attention")
            if direct:
                G.qgemm(attn, w.q[b + "attn_output.weight"], dense_tiles, out_f32=x, resid=x, status=st, work=self._work,
                        **form)
            else:
                project(attn, wo, out_f32=x, resid=x)
            self.timing.mark(il, "o_proj")
            if s.layer_is_moe(il):
                rw = w.q[b + "ffn_gate_inp.weight"]
                if rw.qtype == "F32" and T >= 128 and E % 32 == 0:
                    # split-precision tensor-core router: fp32-grade logits from one bf16 GEMM of depth 3K
                    wr = self._router_w.get(il)
                    if wr is None:
                        wr = G.hilo_weights(rw.data.view(torch.float32).view(E, H))
                        self._router_w[il] = wr
                    G.rmsnorm_hilo(x, w.f[b + "ffn_norm.weight"], s.rms_eps, xn3)
                    G.gemm_bf16(xn3, wr, dense_tiles, out_f32=logits, status=st)
                    rows_in = xn3[:, :H]                # the high halves are the bf16 rows that the experts take
                else:
                    K.router_rows(x, w.f[b + "ffn_norm.weight"], s.rms_eps, rw, T, logits, xn)
                    rows_in = xn
                self.timing.mark(il, "router_logits")
                K.route_rows(logits, e._rule(il), T, ids, wts, e.heat[il], e.fault, il)
                self.timing.mark(il, "route")
                G.moe_plan(ids, wts, E, moe_tiles, pos_of, dst_row, row_scale)
                self.timing.mark(il, "count_scatter")
                G.gather_rows_bf16(rows_in, dst_row, moe_tiles.offsets[E:E + 1], cap, k, Ap)
                self.timing.mark(il, "dispatch")
                if blocks:
                    qg, qu, qd = (w.q[b + f"ffn_{n}_exps.weight"] for n in ("gate", "up", "down"))
                    G.qgemm(Ap, qg, moe_tiles, out_bf16=act, W2=qu, status=st, **form)
                    self.timing.mark(il, "gemm_gate_up")
                    G.qgemm(act, qd, moe_tiles, out_f32=slot_out, dst_row=dst_row, row_scale=row_scale, status=st, **form)
                else:
                    if not ahead and not resident:
                        expand(il, "gate_up")
                    self.timing.mark(il, "expand_gate_up")
                    if pairs:
                        G.gemm_pair(Ap, wg, moe_tiles, out_bf16=act, W2=wu, status=st)
                    else:
                        G.gemm_bf16(Ap, wg, moe_tiles, out_bf16=act, B2=wu, status=st)
                    self.timing.mark(il, "gemm_gate_up")
                    if not ahead and not resident:
                        expand(il, "down")
                    self.timing.mark(il, "expand_down")
                    (G.gemm_pair if pairs else G.gemm_bf16)(act, wd, moe_tiles, out_f32=slot_out, dst_row=dst_row,
                                                            row_scale=row_scale, status=st)
                self.timing.mark(il, "gemm_down")
                if il + 1 < s.n_layer and H <= 8192:
                    G.moe_combine_norm(slot_out, pos_of, T, k, x, x, w.f[f"blk.{il + 1}.attn_norm.weight"], s.rms_eps, xn)
                    normed = True
                else:
                    G.moe_combine(slot_out, pos_of, T, k, x, x)
                self.timing.mark(il, "combine")
            else:
                G.rmsnorm_bf16(x, w.f[b + "ffn_norm.weight"], s.rms_eps, xn)
                if not ahead and not resident:
                    expand(il, "gate_up")
                G.gemm_bf16(xn, dg, dense_tiles, out_bf16=dact, B2=du, status=st)
                if not ahead and not resident:
                    expand(il, "down")
                G.gemm_bf16(dact, dd, dense_tiles, out_f32=x, resid=x, status=st)
            if ahead:
                freed[il].record(main)
        if ahead:
            main.wait_stream(side)
        e.x[0].copy_(x[T - 1])
        if int(st.item()) != 0:
            self._flash_work = G.FlashWork(dev)             # its tickets may not be back at zero
            raise RuntimeError("a bounded wait inside the GEMM kernel ran out (status word set)")

    def _direct(self, T: int, short: bool = False) -> bool:
        """Whether a micro-batch of T tokens multiplies the quantised blocks themselves: a small one of a model whose layers
        are all routed and whose matrices all have a kernel for that (and whose experts are on the card), where no bf16
        copies are kept; ``short``: a whole prompt below the GEMM threshold, whatever is kept."""
        if T > self.direct_rows or self.expert_source is not None:
            return False
        if self._direct_ok is None:
            s, w = self.e.spec, self.e.w
            self._direct_ok = all(s.layer_is_moe(il) for il in range(s.n_layer)) and self._blocks_ok() and all(
                G.qgemm_supports(w.q[f"blk.{il}.{n}.weight"]) for n in ("attn_q", "attn_k", "attn_v", "attn_output")
                for il in range(s.n_layer))
        return self._direct_ok and (short or not self._use_resident())

    def _blocks_ok(self) -> bool:
        """Whether every routed layer's stacks have a kernel that multiplies their blocks."""
        s, w = self.e.spec, self.e.w
        return all(all(G.qgemm_supports(w.q[f"blk.{il}.{n}.weight"]) for n in ("ffn_gate_exps", "ffn_up_exps", "ffn_down_exps"))
                   and w.q[f"blk.{il}.ffn_gate_exps.weight"].qtype == w.q[f"blk.{il}.ffn_up_exps.weight"].qtype
                   for il in range(s.n_layer) if s.layer_is_moe(il))

    def _expert_blocks(self, T: int) -> bool:
        """Whether a micro-batch of T tokens multiplies the routed experts' blocks as they are (block_rows)."""
        s = self.e.spec
        if not s.is_moe or self.expert_source is not None or not self.direct_rows:
            return False
        if self._block_limit is None:
            q = self.e.w.q
            kinds = {n: {q[k].qtype for k in (f"blk.{il}.ffn_{n}_exps.weight" for il in range(s.n_layer) if s.layer_is_moe(il)) if k in q}
                     for n in ("gate", "up", "down")}
            limits = [self.block_rows.get(t, 0) for t in kinds["gate"] | kinds["up"]]
            listed = kinds["down"] <= self.block_rows.keys()
            if not listed:
                limits.append(self.block_rows_any_down)
            self._block_limit = min(limits, default=0) if self._blocks_ok() else 0
            tiles = 2 * s.n_expert
            if self._block_limit and listed and tiles <= PROCESSORS and tiles * -(-max(s.hidden, s.moe_inter) // 128) <= PROCESSORS:
                self._block_limit = max(self._block_limit, 64)
        return T * s.n_used <= self._block_limit * s.n_expert

    def _use_resident(self, experts: bool = False) -> bool:
        """Whether the layers' bf16 copies stay in HBM between prompts; ``experts``: whether those of the routed experts do, which
        the first prompt that needs them makes.  Each is decided once, by the memory that is free right before its first copy."""
        if self.expert_source is not None or self.resident_bf16 is False:
            return False
        if any(q.qtype == "BF16" and q.data.dim() == 3 for q in self.e.w.q.values()):     # bf16 stacks: a copy would only double them
            return False
        s = self.e.spec
        of_experts = 2 * 3 * s.n_expert * s.moe_inter * s.hidden * s.n_layer if s.is_moe else 0
        if self._resident_ok is None:
            per_layer = (s.q_rows + 2 * s.kv_rows) * s.hidden + s.hidden * s.q_rows
            per_layer += 0 if s.is_moe else 3 * (s.dense_inter or 0) * s.hidden
            self._resident_ok = bool(self.resident_bf16) or self._room_for(2 * per_layer * s.n_layer + of_experts)
        if not experts or not of_experts or not self._resident_ok:
            return self._resident_ok
        if self._resident_experts_ok is None:
            self._resident_experts_ok = bool(self.resident_bf16) or self._room_for(of_experts)
        return self._resident_experts_ok

    def _room_for(self, need: int) -> bool:
        """Whether ``need`` more bytes leave a quarter of the card free."""
        free, total = torch.cuda.mem_get_info(self.e.device)
        return free - need >= total // 4

    def _attn_tables(self, T: int, Tq: int, c0: int, n_q: int, Gq: int, pos0: int = 0):
        key = ("attn", T, Tq, c0, n_q, pos0)
        hit = self._buf.get(key)
        if hit is not None:
            return hit
        dev = self.e.device
        i32 = torch.int32
        rows = torch.full((n_q,), Tq, dtype=i32, device=dev)
        qk = G.TileTable(n_q * Tq, n_q, dev)
        qk.build(rows, group_div=Gq, group_stride=T, base=c0, causal_pos0=pos0 + c0, causal_kind=1)
        pv = G.TileTable(n_q * Tq, n_q, dev)
        pv.build(rows, group_div=Gq, causal_pos0=pos0 + c0, causal_kind=2)
        h = torch.arange(n_q, device=dev).view(n_q, 1)
        i = torch.arange(Tq, device=dev).view(1, Tq)
        map_s = torch.full((n_q * T,), -1, dtype=i32, device=dev)
        map_s.view(n_q, T)[:, c0:c0 + Tq] = (h * Tq + i).to(i32)
        map_o = ((c0 + i) * n_q + h).to(i32).reshape(-1).contiguous()   # index h*Tq + i -> token-major row
        out = (qk, pv, map_s, map_o)
        self._buf[key] = out
        return out
