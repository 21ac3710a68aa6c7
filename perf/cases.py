"""The work that programs have this library do, as timed cases.

A case is one pass through the public entry points of `fastar_b200.mla`:

  layer      the layer calls of one model step for a batch of sequences: decode (one new row per
             sequence), verify blocks (a few causal rows over a long cache) and prefill chunks (many
             causal rows over a short one).  io "device": plan once, `run_device` per layer;
             "pinned" and "pageable": `forward` with host buffers, as the engine calls it.  The
             positions move on by one row from pass to pass, so every pass is a new step with a plan
             of its own, and go back after STEPS passes.
  speculate  a verify block on layers with a KV compressor: snapshot, the layer calls, roll back
  draft      the draft model's layer: main row appended, candidate block, block dropped again
  noalloc    decode attention alone over a contiguous cache, nothing allocated

Weights N(0, 0.02^2), norm weights about 1, activations, cached rows and sink logits N(0, 1), as in
the rest of the repository.  Pages of the sequences are interleaved, as sequences that grow side by
side leave them.
"""
import math
import random

import numpy as np
import torch

from fastar_b200 import mla

STEPS = 64  # passes until the positions start again


def _case(name, path="layer", preset="baseline", io="device", layers=1, batch=1, q=(1, 1), ctx=(1, 1), causal=False,
          window=0):
    return {"name": name, "path": path, "preset": preset, "io": io, "layers": layers, "batch": batch, "q_lo": q[0],
            "q_hi": q[1], "ctx_lo": ctx[0], "ctx_hi": ctx[1], "causal": causal, "window": window}


def listed():
    return [
        # one chat at its start, the engine's own loop: four layers, plain vectors for the activations
        _case("decode_1x128_pageable", io="pageable", layers=4, ctx=(128, 128)),
        # one chat over 4096 cached rows, activations on the device
        _case("decode_1x4096", layers=2, ctx=(4096, 4096)),
        # a few users of the live engine's form, page-locked activations
        _case("decode_v4_5_pinned", preset="v4", io="pinned", layers=2, batch=5, ctx=(700, 3000)),
        # the batched-decode workload of the benchmark: 64 users, 1024 to 8192 cached rows
        _case("decode_64", layers=2, batch=64, ctx=(1024, 8192)),
        # many users with short contexts, the live engine's form
        _case("decode_v4_192", preset="v4", batch=192, ctx=(250, 2000)),
        # one very long document
        _case("decode_1x131072", ctx=(131072, 131072)),
        # speculative verify: 16 causal rows of each of 32 sequences over 16384 cached rows
        _case("verify_32x16x16384", batch=32, q=(16, 16), ctx=(16384, 16384), causal=True),
        # a prompt of 2048 rows from an empty cache
        _case("prefill_2048", q=(2048, 2048), ctx=(0, 0), causal=True),
        # chunks of three prompts of uneven length behind what is cached already
        _case("prefill_v4_3_pinned", preset="v4", io="pinned", batch=3, q=(100, 700), ctx=(64, 3000), causal=True),
        # a verify block of six rows on a ratio-4 and a ratio-128 layer, rejected again
        _case("speculate_v4_4x6", path="speculate", preset="v4", io="pinned", layers=2, batch=4, q=(6, 6),
              ctx=(1500, 1500), causal=True),
        # the draft model's layer: five candidate rows over a window of 128
        _case("draft_v4_5", path="draft", preset="v4", io="pageable", q=(5, 5), ctx=(1000, 1000), window=128),
        # decode attention for a host that cannot allocate
        _case("noalloc_20000", path="noalloc", ctx=(20000, 20000)),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["decode", "decode", "decode", "long", "verify", "prefill", "speculate", "draft", "noalloc"])
    preset = rng.choice(["baseline", "v4"])
    io = rng.choice(["device", "device", "pinned", "pageable"])
    if kind == "decode":
        batch = _log(rng, 1, 256)
        hi = _log(rng, 64, min(16384, 400000 // batch))
        lo = rng.randint(max(1, hi // 8), hi)
        c = _case("", preset=preset, io=io, layers=1 if batch * hi > 100000 else rng.choice([1, 2, 4]), batch=batch,
                  ctx=(lo, hi))
    elif kind == "long":
        n = _log(rng, 16384, 131072)
        c = _case("", preset=preset, io=io, ctx=(n, n))
    elif kind == "verify":
        batch, q = _log(rng, 1, 32), rng.randint(2, 16)
        hi = _log(rng, 256, 16384)
        c = _case("", preset=preset, io=io, batch=batch, q=(q, q), ctx=(rng.randint(hi // 2, hi), hi), causal=True)
    elif kind == "prefill":
        batch = rng.choice([1, 1, 2, 3, 5])
        hi = _log(rng, 33, 2048 // batch)
        lo = hi if batch == 1 else rng.randint(max(1, hi // 4), hi)
        ctx = rng.choice([0, _log(rng, 64, 4096 // batch)])
        c = _case("", preset=preset, io=io, batch=batch, q=(lo, hi), ctx=(ctx // 2, ctx), causal=True)
    elif kind == "speculate":
        n = _log(rng, 130, 2048)
        q = rng.randint(1, 8)
        c = _case("", path="speculate", preset="v4", io="pinned", layers=2, batch=_log(rng, 1, 8), q=(q, q), ctx=(n, n),
                  causal=True)
    elif kind == "draft":
        q = rng.randint(1, 8)
        n = _log(rng, 20, 8192)
        c = _case("", path="draft", preset="v4", io="pageable", q=(q, q), ctx=(n, n), window=128)
    else:
        n = _log(rng, 64, 65536)
        c = _case("", path="noalloc", preset=preset, ctx=(n, n))
    del c["name"]
    return c


def _spread(lo, hi, n, phase):
    """n whole numbers spread over [lo, hi], not in order."""
    if n == 1:
        return [hi]
    return [lo + int((hi - lo) * ((phase + i * 0.6180339887498949) % 1.0)) for i in range(n)]


def _sizes(case):
    return (_spread(case["q_lo"], case["q_hi"], case["batch"], 0.5),
            _spread(case["ctx_lo"], case["ctx_hi"], case["batch"], 0.0))


def _ratio(case, lid):
    return (4, 128)[lid % 2] if case["path"] == "speculate" else 0


def _preset(case):
    return mla.PRESET_FASTAR_V4 if case["preset"] == "v4" else mla.PRESET_BASELINE


def _bits(t):
    """A bf16 tensor's values as the 16-bit patterns the library takes, on the host."""
    return t.view(torch.int16).cpu().numpy().view(np.uint16)


def _normal(gen, *shape, std=1.0, mean=0.0):
    t = torch.randn(*shape, generator=gen, device="cuda", dtype=torch.float32)
    return t.mul_(std).add_(mean).to(torch.bfloat16)


def _layer_weights(cfg, gen):
    w = {}
    for name, shape in mla.weight_shapes(cfg).items():
        if name == "attn_sinks":
            w[name] = torch.randn(*shape, generator=gen, device="cuda").cpu().numpy()
        elif name in ("q_norm", "kv_norm"):
            w[name] = _bits(_normal(gen, *shape, std=0.1, mean=1.0))
        else:
            w[name] = _bits(_normal(gen, *shape, std=0.02))
    if cfg.preset == mla.PRESET_FASTAR_V4:  # the live engine's layer call takes the rows before attn_norm
        w["attn_norm"] = _bits(_normal(gen, cfg.hidden, std=0.1, mean=1.0))
    return w


def _prepare_noalloc(case, gen):
    d_qk = 512 if case["preset"] == "v4" else 576
    n = case["ctx_hi"]
    return {"case": case, "q": _normal(gen, 64, d_qk), "cache": _normal(gen, n, d_qk), "n": n, "d_qk": d_qk,
            "out": torch.zeros(64, 512, dtype=torch.bfloat16, device="cuda"), "scale": 1.0 / math.sqrt(192.0)}


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if case["path"] == "noalloc":
        return _prepare_noalloc(case, gen)
    q_lens, ctx_lens = _sizes(case)
    T, B, L = sum(q_lens), case["batch"], case["layers"]
    ends = [c + STEPS + q + 1 for c, q in zip(ctx_lens, q_lens)]
    n_pages = sum((e + 63) // 64 + (e // 4 + 63) // 64 + 1 for e in ends) + 8
    speculate = case["path"] == "speculate"
    cfg = mla.make_config(_preset(case), n_layers=L, n_pages=n_pages, max_seqs=B, max_tokens=max(T, 256 if speculate else 1))
    ctx = mla.MlaContext(cfg)
    row = ctx.dims["row"]
    for lid in range(L):
        ctx.set_layer_weights(lid, _layer_weights(cfg, gen))
        ratio = _ratio(case, lid)
        if ratio:
            width = 2 * cfg.kv_lora if ratio == 4 else cfg.kv_lora
            ctx.set_layer_rope(lid, True)
            ctx.set_layer_compressor(lid, ratio, _bits(_normal(gen, width, cfg.hidden, std=0.02)),
                                     _bits(_normal(gen, width, cfg.hidden, std=0.02)),
                                     torch.randn(ratio, width, generator=gen, device="cuda").cpu().numpy(),
                                     _bits(_normal(gen, cfg.kv_lora, std=0.1, mean=1.0)))
        if case["path"] == "draft":
            ctx.set_layer_draft_form(lid, True)
    seqs = [ctx.seq_alloc() for _ in range(B)]
    if speculate:
        # rows of a layer with a compressor come through layer calls only: prefill in chunks
        for b, s in enumerate(seqs):
            for p in range(0, ctx_lens[b], 256):
                n = min(256, ctx_lens[b] - p)
                h = _bits(_normal(gen, n, cfg.hidden))
                for lid in range(L):
                    ctx.forward(lid, h, [s], [p], [n], causal=True)
    else:
        have = [c + STEPS for c in ctx_lens]
        grow = [b for b in range(B) for _ in range((have[b] + 63) // 64)]
        random.Random(seed).shuffle(grow)
        taken = [0] * B
        for b in grow:
            taken[b] += 1
            ctx.seq_reserve(seqs[b], min(64 * taken[b], have[b]))
        for b, s in enumerate(seqs):
            for lid in range(L):
                ctx.cache_write(lid, s, 0, _bits(_normal(gen, have[b], row)))
    st = {"case": case, "ctx": ctx, "seqs": seqs, "q": q_lens, "pos": ctx_lens, "pass": 0, "layers": L}
    h = _normal(gen, T, cfg.hidden)
    if case["io"] == "device":
        st["h"] = h
        st["outs"] = [torch.zeros_like(h) for _ in range(L)]
    elif case["io"] == "pinned":
        hh = torch.empty(T, cfg.hidden, dtype=torch.int16, pin_memory=True)
        hh.copy_(h.view(torch.int16))
        outs = [torch.zeros(T, cfg.hidden, dtype=torch.int16, pin_memory=True) for _ in range(L)]
        st["p"] = np.array(ctx_lens, np.int32)
        s, q = np.array(seqs, np.int32), np.array(q_lens, np.int32)
        st["calls"] = [ctx.bind_forward(lid, hh.numpy().view(np.uint16), outs[lid].numpy().view(np.uint16), s, st["p"], q,
                                        case["causal"]) for lid in range(L)]
        st["outs"] = [o.view(torch.bfloat16) for o in outs]
    else:
        st["h"] = _bits(h)
    if case["path"] == "draft":
        st["main"] = _bits(_normal(gen, 1, cfg.hidden))
    torch.cuda.synchronize()
    return st


def _values(a):
    return torch.from_numpy(a).view(torch.bfloat16)


def run(st):
    case = st["case"]
    if case["path"] == "noalloc":
        rc = mla.attention_noalloc(st["q"].data_ptr(), st["cache"].data_ptr(), st["n"], 64, st["d_qk"], 512, st["scale"],
                                   st["out"].data_ptr())
        if rc:
            raise RuntimeError("attention_noalloc: %d" % rc)
        return st["out"]
    ctx, seqs, q, L = st["ctx"], st["seqs"], st["q"], st["layers"]
    if case["path"] == "draft":
        anchor, window = st["pos"][0], case["window"]
        ctx.append_rows(0, st["main"], seqs, [anchor], [1])
        ctx.set_window(window + q[0] if anchor + 1 > window else 0)
        out = ctx.forward(0, st["h"], seqs, [anchor + 1], q)
        ctx.set_window(0)
        ctx.seq_truncate(seqs[0], anchor + 1)
        return _values(out)
    if case["path"] == "speculate":
        for s in seqs:
            ctx.seq_snapshot(s)
        for call in st["calls"]:
            call()
        for s, p in zip(seqs, st["pos"]):
            ctx.seq_truncate(s, p)
        return st["outs"]
    k = st["pass"] % STEPS
    st["pass"] += 1
    pos = [p + k for p in st["pos"]]
    if case["io"] == "device":
        ctx.plan([(s, p, n) for s, p, n in zip(seqs, pos, q)], causal=case["causal"])
        for lid in range(L):
            ctx.run_device(lid, st["h"].data_ptr(), st["outs"][lid].data_ptr())
        return st["outs"]
    if case["io"] == "pinned":
        st["p"][:] = pos
        for call in st["calls"]:
            call()
        return st["outs"]
    return [_values(ctx.forward(lid, st["h"], seqs, pos, q, causal=case["causal"])) for lid in range(L)]


def work(case):
    """Weights, the cached rows that are attended to, and the rows in and out, each once."""
    v4 = case["preset"] == "v4"
    row = 512 if v4 else 576
    if case["path"] == "noalloc":
        n = case["ctx_hi"]
        return {"bytes": 2 * (n * row + 64 * (row + 512)), "flops": 2 * 64 * (row + 512) * n}
    cfg = mla.make_config(_preset(case))
    weights = sum(math.prod(s) for s in mla.weight_shapes(cfg).values())
    q_lens, ctx_lens = _sizes(case)
    n_bytes = flops = 0
    T = sum(q_lens)
    for lid in range(case["layers"]):
        ratio = _ratio(case, lid)
        w = weights + (2 * 4096 * (1024 if ratio == 4 else 512) if ratio else 0)
        rows = pairs = 0  # cached rows, (new row, cached row) pairs
        for q, c in zip(q_lens, ctx_lens):
            if case["window"]:
                c = min(c, case["window"])
            cmp_rows = c // ratio if ratio else 0
            rows += c + cmp_rows
            pairs += q * (c + cmp_rows) + (q * (q + 1) // 2 if case["causal"] else q * q)
        n_bytes += 2 * (w + rows * row + 2 * T * 4096 + T * row)
        flops += 2 * T * w + 2 * 64 * (row + 512) * pairs
    return {"bytes": n_bytes, "flops": flops}


def tolerance(case):
    # bf16 operands and a chain of bf16 intermediates with fp32 accumulation; the compressed rows of
    # a ratio-4 or ratio-128 layer are E4M3 values, where a neighbouring value may appear
    return {"rel": 1e-2}
