"""Performance cases of the engine: speculative decode steps, prefills and image encodings, each through
the entry point a serving process calls (``SpecDecoder.step``, ``run_prefill``, ``VisionTower.encode``).

Two model geometries, with their full widths and a few of their layers (a layer's cost does not depend
on how many there are): ``flash`` is ``flash_b200_config`` with four layers, the first of which owns the
compressed stream and the indexer (``bench.py --layers`` builds the same model), ``ref`` is
``reference_1017_config`` with two layers (low-rank query, grouped output projection, 512-wide latent
heads, four residual copies, 384 experts).  Both carry a one-layer draft head.

Weights are random with the structure a trained model has where the path takes discrete decisions: a token
belongs to one of 256 classes, each class has its own top-k experts in every layer, and the head knows
each token's successor, so that neither the routing nor the sampling hangs on the last bit of a sum.
Experts stay evenly loaded and a block of rows meets as many different experts as random routing gives.
The embeddings are ten times as large as what one sublayer adds, as the residual stream of a deep model is:
the FP8 and MXFP8 roundings of a layer then move the logits by about a hundredth.
"""
from __future__ import annotations

import gc
import math

import torch

from titanic_flash_41_b200.config import DraftConfig, EngineConfig, VisionConfig, flash_b200_config, reference_1017_config
from titanic_flash_41_b200.formats import codecs
from titanic_flash_41_b200.models.engine import Engine, quant_fp8_device
from titanic_flash_41_b200.models.vision import VisionTower, init_vision_weights
from titanic_flash_41_b200.ops import bigpath
from titanic_flash_41_b200.serve.prefill import run_prefill
from titanic_flash_41_b200.spec.decoder import DecodeSlot, SpecDecoder

CONTEXT = 131072            # the default context limit of the engine configuration
CHUNK = 16384               # the default prefill chunk
CLASSES = 256
DEV = "cuda"


def listed():
    return [
        # one chat turn answered shortly after its start: a step is bound by latency and launches
        dict(name="decode 1x300", kind="decode", model="flash", sessions=1, context=300, ragged=False),
        # one agent deep in a long document
        dict(name="decode 1x131K", kind="decode", model="flash", sessions=1, context=131000, ragged=False),
        # three conversations of very different lengths in one step
        dict(name="decode 3 ragged", kind="decode", model="flash", sessions=3, context=65537, ragged=True),
        # all four admitted conversations near the context limit: the headline decode workload
        dict(name="decode 4x131K", kind="decode", model="flash", sessions=4, context=130560, ragged=False),
        # a short request, cold
        dict(name="prefill 197", kind="prefill", model="flash", tokens=197, start=0),
        # the next turn of a long conversation: a follow-up behind a restored prefix, inside a pooling group
        dict(name="prefill 2049 at 127K", kind="prefill", model="flash", tokens=2049, start=127003),
        # a document of one full chunk
        dict(name="prefill 16384", kind="prefill", model="flash", tokens=16384, start=0),
        # the headline cold prompt
        dict(name="prefill 129553", kind="prefill", model="flash", tokens=129553, start=0),
        # the reference geometry: a full batch of deep drafts (24 rows), and a prompt
        dict(name="ref decode 4x16K", kind="decode", model="ref", sessions=4, context=16411, ragged=True),
        dict(name="ref prefill 4001", kind="prefill", model="ref", tokens=4001, start=0),
        # images: the smallest patch grid the input planner makes, and a page at the token limit
        dict(name="image 39x39", kind="image", rows=39, cols=39),
        dict(name="image 110x78", kind="image", rows=110, cols=78),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("decode", "decode", "prefill", "prefill", "image"))
    if kind == "image":
        rows = rng.randint(39, 110)
        cols = rng.randint(39, max(39, min(110, 8580 // rows)))
        return dict(kind=kind, rows=rows, cols=cols)
    model = rng.choice(("flash", "flash", "ref"))
    if kind == "decode":
        s = rng.randint(1, 4)
        top = CONTEXT - 512 if model == "flash" else 32000
        return dict(kind=kind, model=model, sessions=s, context=_log_int(rng, 130, top), ragged=s > 1 and rng.random() < 0.5)
    n = _log_int(rng, 5, 100000 if model == "flash" else 4000)
    start = 0
    if rng.random() < 0.5 and n < 8192:
        start = _log_int(rng, 130, CONTEXT - 8192 if model == "flash" else 32000)
    return dict(kind=kind, model=model, tokens=n, start=start)


# ------------------------------------------------------------------------------------------ models
def _config(model):
    if model == "flash":
        return flash_b200_config(n_layers=4, kv_source_layers=(0,), index_source_layers=(0,), late_start=-1)
    return reference_1017_config(n_layers=2, kv_source_layers=(0,), compress_ratio=2, compress_ratios=(2,),
                                 index_source_layers=(0,), late_start=-1, dense_quant="fp8_block128", vision=None, engram=None,
                                 draft=DraftConfig(layers=1, depth=5))


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _structure(eng, seed):
    """Class structure of the embeddings and the routers, successor structure of the head (see above)."""
    cfg, g = eng.cfg, _generator(seed + 101)
    V, d = cfg.vocab, cfg.hidden

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV, dtype=torch.bfloat16)
    centre = randn(CLASSES, d)
    member = torch.randint(0, CLASSES, (V,), generator=g, device=DEV)
    eng.embed_w.copy_(randn(V, d) * 6.0 + centre[member] * 8.0)
    for L in eng.layers + eng.draft_layers:
        experts = torch.rand(CLASSES, cfg.n_experts, generator=g, device=DEV).argsort(1)[:, :cfg.topk]
        hit = torch.zeros(CLASSES, cfg.n_experts, device=DEV).scatter_(1, experts, 1.0)
        gate = torch.randn(cfg.n_experts, d, generator=g, device=DEV) * (0.5 / math.sqrt(d)) + hit.t() @ centre.float() * (8.0 / d)
        L.gate.copy_(gate)
    following = torch.randperm(V, generator=g, device=DEV)
    eng.head_w[following] = eng.embed_w * 0.002
    mix = torch.randn(d, 2 * d, generator=g, device=DEV) * 0.002
    mix[:, :d] += torch.eye(d, device=DEV)
    eng.draft_extra["main_proj"] = quant_fp8_device(mix)
    eng.draft_extra["head"] = quant_fp8_device(eng.head_w)


def _engine(model, widest, seed):
    cfg = _config(model)
    ecfg = EngineConfig(regions=4, max_context=CONTEXT, prefill_widths=(widest,))
    eng = Engine.random_init(cfg, ecfg, device=DEV, seed=seed, max_chunk=widest)
    bigpath.attach(eng)
    _structure(eng, seed)
    return eng


def _history(eng, region, length, seed):
    """The KV state of a conversation of ``length`` tokens: normalised latents in the stored formats."""
    cfg, g = eng.cfg, _generator(seed + 211)

    def randn(*shape):
        return torch.randn(*shape, generator=g, device=DEV)
    D, n = cfg.head_dim, length // cfg.compress_ratio
    w = codecs.kv_v41_encode(randn(eng.win.shape[0], min(length, eng.ring), D))
    slots = torch.arange(length - w.shape[1], length, device=DEV) % eng.ring
    eng.win[:, region, slots, :w.shape[-1]] = w
    for lo in range(0, n, 8192):
        m = min(8192, n - lo)
        e = codecs.kv_v41fp4_encode(randn(m, D))
        eng.comp[0, region, lo:lo + m, :e.shape[-1]] = e
        eng.keys[0, region, lo:lo + m] = codecs.index_key_encode(randn(m, cfg.index_dim))
    eng.carry[:, region] = randn(*eng.carry[:, region].shape)


def _lengths(case):
    """Contexts of the conversations; ragged ones fall off from the longest by factors of about five."""
    s, n = case["sessions"], case["context"]
    return [n - r if not case["ragged"] else max(131, n // 5 ** r - r) for r in range(s)]


def prepare(case, seed):
    gc.collect()            # engines of earlier cases hold reference cycles
    if case["kind"] == "image":
        vc = VisionConfig(layers=8)
        tower = VisionTower(vc, 5120, init_vision_weights(vc, 5120, seed), device=DEV)
        patches = (torch.rand(case["rows"] * case["cols"], 588, generator=_generator(seed + 307), device=DEV) * 2 - 1).bfloat16()
        return dict(kind="image", tower=tower, patches=patches, rows=case["rows"], cols=case["cols"])
    cpu = torch.Generator().manual_seed(seed + 401)
    if case["kind"] == "prefill":
        widest = min(CHUNK, max(256, case["tokens"]))
        eng = _engine(case["model"], widest, seed)
        vocab = eng.cfg.vocab
        run_prefill(eng, 1, torch.randint(0, vocab, (128,), generator=cpu, dtype=torch.int32), widest)     # a server's self-check
        if case["start"]:
            _history(eng, 0, case["start"], seed)
        tokens = torch.randint(0, vocab, (case["tokens"],), generator=cpu, dtype=torch.int32)
        return dict(kind="prefill", eng=eng, tokens=tokens, start=case["start"], chunk=widest, carry=eng.carry[:, 0].clone())
    eng = _engine(case["model"], 256, seed)
    lengths = _lengths(case)
    for r, n in enumerate(lengths):
        _history(eng, r, n, seed + 7 * r)
    anchors = torch.randint(0, eng.cfg.vocab, (len(lengths),), generator=cpu).tolist()
    slots = [dict(region=r, length=n, anchor=anchors[r], seed=seed + r) for r, n in enumerate(lengths)]
    dec = SpecDecoder(eng, len(lengths))
    hidden = torch.randn(len(lengths), eng.cfg.hidden, generator=_generator(seed + 503), device=DEV).bfloat16()
    dec.step([DecodeSlot(**s) for s in slots])                  # a server's self-check captures the step
    return dict(kind="decode", eng=eng, dec=dec, slots=slots, hidden=hidden)


# ------------------------------------------------------------------------------------------ one pass
def run(state):
    if state["kind"] == "image":
        return state["tower"].encode(state["patches"], state["rows"], state["cols"])
    eng = state["eng"]
    if state["kind"] == "prefill":
        # state is addressed by position: the pass writes the same rows again; the open pooling group of a
        # continued conversation is put back as restoring its state does
        start, n = state["start"], state["tokens"].shape[0]
        eng.carry[:, 0].copy_(state["carry"])
        logits = run_prefill(eng, 0, state["tokens"], state["chunk"], start)
        r = eng.cfg.compress_ratio
        lo, hi = start // r, (start + n) // r
        return dict(logits=logits, hidden=eng.last_hidden[-1:], window=eng.win[0, 0], compressed=eng.comp[0, 0, lo:hi],
                    keys=eng.keys[0, 0, lo:hi], carry=eng.carry[:, 0])
    dec = state["dec"]
    dec.hidden.copy_(state["hidden"])
    slots = [DecodeSlot(**s) for s in state["slots"]]
    tokens = dec.step(slots)
    return dict(tokens=tokens, following=[s.anchor for s in slots], draft_logits=dec.dlogits, hidden=dec.hidden)


# ------------------------------------------------------------------------------------------ what it takes
def _layer_cost(cfg, T, keys, draft=False, source=False):
    """(weight and KV bytes, operations) of one layer over T rows that attend to ``keys`` keys each."""
    d, D, H, I, k, E = cfg.hidden, cfg.head_dim, cfg.n_heads, cfg.moe_inter, cfg.topk, cfg.n_experts
    q = d * cfg.q_lora_rank + cfg.q_lora_rank * H * D if cfg.q_lora_rank else d * H * D
    o = H * D * cfg.o_lora_rank + cfg.o_groups * cfg.o_lora_rank * d if cfg.o_groups else d * H * D
    dense = q + o + d * D + 3 * d * cfg.shared_inter * cfg.n_shared
    if source:
        dense += d * (2 * (D + cfg.index_dim) + cfg.index_heads * (cfg.index_dim + 1))
    expert = 3 * d * I
    distinct = E * (1.0 - (1.0 - k / E) ** T)
    nbytes = dense + distinct * expert * (0.5 + 1 / 32) + E * d * 2
    flops = 2.0 * T * (dense + k * expert + E * d) + 4.0 * T * H * D * keys
    return nbytes, flops


def work(case):
    if case["kind"] == "image":
        vc, n = VisionConfig(layers=8), case["rows"] * case["cols"]
        w, m, dm = vc.hidden, vc.intermediate, 5120
        cells = -(-case["rows"] // 3) * -(-case["cols"] // 3)
        params = vc.layers * (4 * w * w + 3 * w * m) + 588 * w
        align = 9 * w * dm + dm * dm
        return dict(bytes=2.0 * (params + align + n * 588 + cells * dm),
                    flops=2.0 * n * params + 2.0 * cells * align + 4.0 * vc.layers * n * n * w)
    cfg = _config(case["model"])
    r, head = cfg.compress_ratio, cfg.vocab * cfg.hidden
    key_row, comp_row, win_row = cfg.index_key_bytes, cfg.head_dim // 2 + cfg.head_dim // 16, cfg.head_dim + cfg.head_dim // 32
    nbytes = flops = 0.0
    if case["kind"] == "prefill":
        n, start = case["tokens"], case["start"]
        mean = sum(min((start + n * (i + 0.5) / 64) / r, cfg.index_topk) for i in range(64)) / 64
        for l in range(cfg.n_layers):
            b, f = _layer_cost(cfg, n, min(cfg.window, start + n / 2) + mean, source=l == 0)
            nbytes, flops = nbytes + b + n * win_row, flops + f
        flops += 2.0 * n * (start + n / 2) / r * cfg.index_heads * cfg.index_dim + 2.0 * head
        nbytes += n * cfg.hidden * 2 + (start + n) / r * (comp_row + key_row) + 2 * head
        return dict(bytes=nbytes, flops=flops)
    lengths, g = _lengths(case), cfg.draft.depth
    rows = len(lengths) * (g + 1)
    entries = [x // r for x in lengths]
    picked = [min(e, cfg.index_topk) for e in entries]
    keys = sum(picked) / len(lengths) + cfg.window
    for l in range(cfg.n_layers):
        b, f = _layer_cost(cfg, rows, keys, source=l == 0)
        nbytes, flops = nbytes + b + sum(picked) * comp_row + len(lengths) * cfg.window * win_row, flops + f
    nbytes += sum(entries) * key_row + 2 * head
    flops += 2.0 * (g + 1) * sum(entries) * cfg.index_heads * cfg.index_dim + 2.0 * rows * head
    b, f = _layer_cost(cfg, len(lengths), cfg.window)
    mix = 2 * cfg.hidden ** 2
    nbytes += g * (b + mix + head)
    flops += g * (f + 2.0 * len(lengths) * (mix + head))
    return dict(bytes=nbytes, flops=flops)


def tolerance(case):
    # Four times what a permutation of the hidden inputs inside their quantisation groups (the same model, its
    # sums in another order) does to the outputs: 0.8 % of the logits and hidden rows, because a last-bit
    # difference decides some FP8 and MXFP8 roundings; 4e-5 of the stored bytes.
    if case["kind"] == "image":
        return {"rel": 0.03, "max": 0.4}        # bf16 rows between the operators: 1.7 % from an fp32 evaluation
    return {"rel": 0.03, "max": 0.2, "differ": 0.0005}
