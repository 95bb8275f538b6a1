"""The calls by which the framework's speed is measured: what a server asks of one GPU.

A server loads its model once and then takes two kinds of call for as long as it runs: it feeds prompts
(``GpuEngine.prefill``, from an empty cache or as the next turn of a conversation that the cache holds) and it decodes rounds
(``GpuEngine.step``, one token for every sequence that is active, greedy or with the sampling chain).  Both run here at
full depth on the Qwen3-30B-A3B shape in Q4_K_M, rounds also in the FP8 and NVFP4 block formats and on the tiny shape,
whose calls are as short as calls get.

The model is one per shape and format and does not depend on a case's seed; a seed gives a request: prompt ids, cache
contents, tokens, sampling parameters.  Weights are random, with the proportions that keep a deep network tame as
training does: embeddings of order one, projections that add to the residual stream scaled down by sqrt(2 x layers), and
a router that prefers some experts clearly.  (With equal scales everywhere the last bit of a sum decides which experts
the later layers choose, and no two correct implementations agree after a few layers.)
"""
from __future__ import annotations

import gc
import math
import random

import torch

from bloomery_b200.formats import quant
from bloomery_b200.formats.resident import PLANE_TYPES, quantize_resident
from bloomery_b200.models.spec import NAMED
from bloomery_b200.models.weights import Weights, q4_k_m_type
from bloomery_b200.runtime.engine import DecodeEngine
from bloomery_b200.runtime.kv import PAGE
from bloomery_b200.serve.engine import GpuEngine
from bloomery_b200.serve.sampler import SamplingParams
from bloomery_b200.serve.tokenizer import ByteTokenizer

BITS = {"F32": 32, "Q4_K": 4.5, "Q6_K": 6.5625, "FP8_B128": 8 + 32 / 128 ** 2, "NVFP4": 4.5}
CTX = 16384                     # positions a slot can hold
MAX_ROWS = 64                   # sequences in the largest round
# KV pages of a server: three of the largest round (64 sequences, 2,000 positions each on average)
PAGES = 6600


def listed():
    big = "qwen3-30b-a3b"
    return [
        # the smallest call: one token of one sequence on a model of four layers; launches and the host are all it costs
        step("tiny round of 1", "tiny-qwen3moe", "Q4_K_M", 1, 64),
        # one person's chat, early in it: the headline decode (512 ids in the cache)
        step("round of 1, short", big, "Q4_K_M", 1, 512),
        # the same with a long document in the cache
        step("round of 1, long", big, "Q4_K_M", 1, 12000),
        # a small office: five chats of unequal length, each with its own sampling parameters
        step("round of 5, sampled", big, "Q4_K_M", 5, 1500, sampled=True),
        # a busy server, and a full one: ragged contexts around 1,000 and 2,000 positions
        step("round of 24", big, "Q4_K_M", 24, 1000),
        step("round of 64, sampled", big, "Q4_K_M", 64, 2000, sampled=True),
        # checkpoints in block-scaled float formats, decoded as they are
        step("fp8 round of 32", big, "FP8_B128", 32, 700),
        step("nvfp4 round of 1", big, "NVFP4", 1, 900),
        # prompts: a short question, the headline prompt, the headline long prompt
        prompt("prompt of 37", big, "Q4_K_M", 37, 0),
        prompt("prompt of 512", big, "Q4_K_M", 512, 0),
        prompt("prompt of 4096", big, "Q4_K_M", 4096, 0),
        # the next turn of a long conversation: new ids behind a cached prefix
        prompt("turn of 700 behind 9000", big, "Q4_K_M", 700, 9000),
    ]


def step(name, model, mix, rows, ctx, sampled=False):
    return {"name": name, "kind": "step", "model": model, "mix": mix, "rows": rows, "ctx": ctx, "sampled": sampled}


def prompt(name, model, mix, n, start):
    return {"name": name, "kind": "prompt", "model": model, "mix": mix, "n": n, "start": start}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Rounds of 1 to 64 sequences with 32 to 12,000 positions each, prompts of 2 to 4,096 ids, turns of up to 1,000 ids
    behind up to 12,000."""
    r = rng.random()
    if r < 0.4:                                                  # prompts
        start = _log(rng, 64, 12000) if rng.random() < 0.4 else 0
        case = prompt("", "qwen3-30b-a3b", "Q4_K_M", _log(rng, 2, 1000 if start else 4096), start)
    else:
        model, mix = "qwen3-30b-a3b", "Q4_K_M"
        if r > 0.92:
            model = "tiny-qwen3moe"
        elif r > 0.8:
            mix = rng.choice(["FP8_B128", "NVFP4"])
        rows = _log(rng, 1, MAX_ROWS)
        ctx = _log(rng, 32, 3000 if model == "tiny-qwen3moe" else min(12000, 128000 // rows))
        case = step("", model, mix, rows, min(ctx, CTX * 2 // 3), rng.random() < 0.4)
    del case["name"]
    return case


# ---- the model and its server -------------------------------------------------------------------------------------
def _matrices(spec, il):
    """Name, shape and standard deviation of the matrices of layer ``il``."""
    H, E, I = spec.hidden, spec.n_expert, spec.moe_inter
    into = 0.02 / math.sqrt(2 * spec.n_layer)                    # what adds to the residual stream
    return [("attn_q", (spec.q_rows, H), 0.02), ("attn_k", (spec.kv_rows, H), 0.02), ("attn_v", (spec.kv_rows, H), 0.02),
            ("attn_output", (H, spec.q_rows), into), ("ffn_gate_inp", (E, H), 0.1), ("ffn_gate_exps", (E, I, H), 0.02),
            ("ffn_up_exps", (E, I, H), 0.02), ("ffn_down_exps", (E, H, I), into)]


def _types(spec, mix, name, il):
    t = q4_k_m_type(name, il, spec.n_layer)
    return t if mix == "Q4_K_M" or t == "F32" else mix


def _tensors(spec, mix, device):
    """Every tensor of the model as a checkpoint's reader would hand it over."""
    gen = torch.Generator(device=device)
    gen.manual_seed(20240611)

    def matrix(name, shape, std, il=0):
        w = torch.randn(math.prod(shape[:-1]), shape[-1], generator=gen, device=device) * std
        t = _types(spec, mix, name, il)
        return name, shape, t, (quantize_resident(w, t, values=False)[0] if t in PLANE_TYPES else quant.quantize(w, t))

    def gain(name, n):
        w = 1 + 0.02 * torch.randn(1, n, generator=gen, device=device)
        return name, (n,), "F32", quant.quantize(w, "F32")

    yield matrix("token_embd.weight", (spec.vocab, spec.hidden), 1.0)
    for il in range(spec.n_layer):
        b = f"blk.{il}."
        for name, n in (("attn_norm", spec.hidden), ("attn_q_norm", spec.head_dim), ("attn_k_norm", spec.head_dim),
                        ("ffn_norm", spec.hidden)):
            yield gain(b + name + ".weight", n)
        for name, shape, std in _matrices(spec, il):
            yield matrix(b + name + ".weight", shape, std, il)
    yield gain("output_norm.weight", spec.hidden)
    yield matrix("output.weight", (spec.vocab, spec.hidden), 0.02)


class _Server:
    """A loaded model with its engine, and the slots that no request holds."""

    def __init__(self, model, mix):
        spec = NAMED[model]()
        weights = Weights.from_items(spec, _tensors(spec, mix, "cuda"), "cuda")
        dec = DecodeEngine(weights, n_slots=3 * MAX_ROWS + 8, slot_ctx=CTX, kv_pages=PAGES)
        self.engine = GpuEngine(dec, ByteTokenizer(), model)
        self.free = list(range(dec.n_slots))


_loaded = {}


def _server(model, mix):
    """The server of a model: loaded once, and given back when another model's is asked for."""
    if (model, mix) not in _loaded:
        _loaded.clear()
        gc.collect()
        torch.cuda.empty_cache()
        _loaded[model, mix] = _Server(model, mix)
    return _loaded[model, mix]


# ---- requests -----------------------------------------------------------------------------------------------------
def _lengths(case):
    """Positions that each sequence of a round has in the cache: from half of the average to one and a half times it."""
    if case["rows"] == 1:
        return [case["ctx"]]
    r = random.Random(case["rows"] * 100003 + case["ctx"])
    return [max(1, int(case["ctx"] * r.uniform(0.5, 1.5))) for _ in range(case["rows"])]


class _Request:
    """Some slots of a server and what is asked of them next; the slots go back with it."""

    def __init__(self, server, n):
        self.server, self.engine = server, server.engine
        self.slots = [server.free.pop(0) for _ in range(n)]

    def __del__(self):
        for s in self.slots:
            self.engine.reset(s)
        self.server.free[:0] = self.slots


def _fill(engine, slot, n, gen):
    """Cached keys and values of ``n`` positions, through the engine's own way of bringing a saved sequence back.  Keys
    are normalised per head, values are the projection of normalised rows: both have about unit variance."""
    kv = engine.dec.kv
    shape = (kv.n_layer, (n + PAGE - 1) // PAGE, kv.n_kv, PAGE, kv.head_dim)
    rows = [torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float16) for _ in range(2)]
    kv.restore(slot, {"k": rows[0], "v": rows[1], "n": n}, n)
    engine.dec.slot_len[slot] = n


def prepare(case, seed):
    server = _server(case["model"], case["mix"])
    engine, vocab = server.engine, server.engine.n_vocab
    rng = random.Random(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["kind"] == "prompt":
        req = _Request(server, 1)
        req.slot, req.start = req.slots[0], case["start"]
        req.ids = [rng.randrange(vocab) for _ in range(case["n"])]
        if req.start:
            _fill(engine, req.slot, req.start, gen)
        return req
    lengths = _lengths(case)
    req = _Request(server, len(lengths))
    for slot, n in zip(req.slots, lengths):
        _fill(engine, slot, n, gen)
    req.rows = [(slot, rng.randrange(vocab), n) for slot, n in zip(req.slots, lengths)]
    req.sampling = None
    if case["sampled"]:
        req.sampling = [[SamplingParams(temperature=rng.uniform(0.3, 1.1), top_k=rng.choice([20, 40, 64]),
                                        top_p=rng.choice([0.8, 0.9, 0.95]), min_p=rng.choice([0.0, 0.05]),
                                        repeat_penalty=rng.choice([1.0, 1.0, 1.1]), seed=rng.randrange(1 << 40)),
                         rng.randrange(500), [rng.randrange(vocab) for _ in range(min(64, n))]] for n in lengths]
    # where the round's own keys and values land
    kv = engine.dec.kv
    for slot, n in zip(req.slots, lengths):
        kv.ensure(slot, n + 1)
    kv.sync_table()
    req.page = torch.tensor([kv.pages[s][n // PAGE] for s, n in zip(req.slots, lengths)], device="cuda")
    req.at = torch.tensor([n % PAGE for n in lengths], device="cuda")
    return req


def run(req):
    """One call of the server, and what it leaves: logits of the rows that are asked for, keys and values of the new
    positions.  (The ids are picked from the logits inside the call.  They stay out of the outputs: the two best of
    150,000 logits are often closer to each other than two correct sums of their terms.)"""
    engine, kv = req.engine, req.engine.dec.kv
    if hasattr(req, "rows"):
        engine.step(req.rows, want_logits=False, sampling=req.sampling)
        n = len(req.rows)
        logits = engine.dec.logits if n <= engine.max_rows else engine._batch().logits
        if n == 1:
            page, at = kv.pages[req.rows[0][0]][req.rows[0][2] // PAGE], req.rows[0][2] % PAGE
            return {"logits": logits[:1], "k": kv.k[:, page, :, at], "v": kv.v[:, page, :, at]}
        return {"logits": logits[:n], "k": kv.k[:, req.page, :, req.at], "v": kv.v[:, req.page, :, req.at]}
    last = req.start + len(req.ids) - 1
    engine.cut(req.slot, req.start)
    engine.prefill(req.slot, req.ids[:-1], req.start)            # a prompt's last id opens its first round
    engine.step([(req.slot, req.ids[-1], last)], want_logits=False)
    return {"logits": engine.dec.logits[:1], **_new_rows(kv, req.slot, req.start, len(req.ids))}


def _new_rows(kv, slot, start, n):
    """Views of the whole pages that hold positions start .. start + n (a copy where the pages do not follow each other)."""
    pages = kv.pages[slot][start // PAGE:(start + n + PAGE - 1) // PAGE]
    first = pages[0]
    if pages == list(range(first, first + len(pages))):
        k, v = kv.k[:, first:first + len(pages)], kv.v[:, first:first + len(pages)]
    else:
        at = torch.tensor(pages, device=kv.k.device)
        k, v = kv.k.index_select(1, at), kv.v.index_select(1, at)
    if len(pages) == 1:                                          # leave out what the page holds behind the last position
        a = start % PAGE
        return {"k": k[:, 0, :, a:a + n], "v": v[:, 0, :, a:a + n]}
    end = (start + n - 1) % PAGE + 1
    return {"k": k[:, :-1], "v": v[:, :-1], "k_last": k[:, -1, :, :end], "v_last": v[:, -1, :, :end]}


def work(case):
    """Every weight that some row needs read once (of the routed experts the number that as many independent choices
    reach), cached keys and values of the attended positions read once, new ones and the logits written once."""
    spec, mix = NAMED[case["model"]](), case["mix"]
    if case["kind"] == "step":
        rows, heads = case["rows"], case["rows"]
        cached = sum(_lengths(case))
        pairs = cached + rows                                    # (query, key) pairs
    else:
        rows, heads, cached = case["n"], 1, case["start"]
        pairs = rows * cached + rows * (rows + 1) // 2
    reached = 1 - (1 - spec.n_used / spec.n_expert) ** rows
    bits = flops = 0.0
    for il in range(spec.n_layer):
        for name, shape, _ in _matrices(spec, il):
            n = math.prod(shape)
            routed = name.endswith("_exps")
            bits += n * BITS[_types(spec, mix, f"blk.{il}.{name}.weight", il)] * (reached if routed else 1)
            flops += 2.0 * n * rows * (spec.n_used / spec.n_expert if routed else 1)
    head = spec.vocab * spec.hidden
    bits += head * BITS[_types(spec, mix, "output.weight", 0)]
    flops += 2.0 * head * heads + 4.0 * pairs * spec.q_rows * spec.n_layer
    row = spec.n_layer * 2 * spec.kv_rows * 2                    # bytes that a position has in the cache
    return {"bytes": bits / 8 + row * (cached + rows) + 4.0 * heads * spec.vocab, "flops": flops}


def tolerance(case):
    """Activations are rounded in front of every product, to bf16 or to 8-bit integers with a scale for 32 values, with
    FP8 weights to E4M3, which keeps three bits behind the leading one: two correct orders of summation round
    differently, and what differs passes through all layers."""
    return {"rel": 3e-2 if case["mix"] == "FP8_B128" and case["rows"] > 8 else 1e-2, "max": 0.3}
