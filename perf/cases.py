"""Performance cases of the FP4 MLA decode engine, each one pass of a program that uses it through its public entry points.

Three kinds of pass, told apart by ``kind``:

* ``decode``  ``BatchMLADecodeCuteDSLFP4Wrapper.run`` on a paged cache: one attention call of one layer and decode step;
* ``write``   ``kvcache.write_tokens``: new tokens quantised and scattered into the paged cache;
* ``step``    ``FP4MLADecodeBackend``: a scheduler's metadata refreshed, the step's tokens appended, attention over them,
  launched call by call or replayed from a CUDA graph.

``draw`` gives further cases of the same ranges: 1 to 128 requests of up to 131072 tokens, 1 to 128 heads, every page size,
every output and input type, the attention variants, 1 to 262144 written tokens.
"""
import math
import random

import torch

from flashinfer_mla_fp4_b200 import (AttentionWithSink, BatchMLADecodeCuteDSLFP4Wrapper, FP4MLADecodeBackend, FP4MLAPagedCache,
                                     SoftCappingAttention, synth)
from flashinfer_mla_fp4_b200.kvcache import write_tokens

_OUT = {"bf16": torch.bfloat16, "f32": torch.float32, "e4m3": torch.float8_e4m3fn}
_IN = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def _decode(name, batch, heads, lo, hi, page=64, q_len=1, out="bf16", variant="none", lse=False, latent="normal", lens=0):
    c = {"kind": "decode", "batch": batch, "heads": heads, "lo": lo, "hi": hi, "page": page, "q_len": q_len, "out": out,
         "variant": variant, "lse": lse, "latent": latent, "lens": lens}
    return dict(c, name=name) if name else c


def _write(name, tokens, dtype, page=64, scaled=False):
    c = {"kind": "write", "tokens": tokens, "dtype": dtype, "page": page, "scaled": scaled}
    return dict(c, name=name) if name else c


def _step(name, batch, max_batch, heads, lo, hi, page=64, q_len=1, graph=False, host=False, lens=0):
    c = {"kind": "step", "batch": batch, "max_batch": max_batch, "heads": heads, "lo": lo, "hi": hi, "page": page, "q_len": q_len,
         "graph": graph, "host": host, "lens": lens}
    return dict(c, name=name) if name else c


def listed():
    return [
        # the smallest call: two short chats on a tensor-parallel shard of 16 heads; latency and host work are all there is
        _decode("decode_small", 2, 16, 256, 256),
        # a few interactive requests of ordinary length
        _decode("decode_uniform", 4, 64, 4096, 4096),
        # long documents at a small batch: the headline configuration
        _decode("decode_long", 8, 64, 32768, 32768),
        # a full serving batch, lengths spread over two orders of magnitude, latents with outliers
        _decode("decode_varlen", 128, 64, 128, 32768, latent="student_t3", lens=1002),
        # very long context, two query positions per request, 128 heads
        _decode("decode_spec", 2, 128, 131072, 131072, q_len=2),
        # data-parallel attention: the rank keeps all 128 heads of its own requests; E4M3 output for an FP8 projection
        _decode("decode_dp_heads128", 32, 128, 1024, 16384, out="e4m3", lens=1004),
        # odd everything: heads that fill no group, short ragged requests on small pages, soft cap and sink, FP32 partials with LSE
        _decode("decode_ragged", 7, 40, 1, 3000, page=16, out="f32", variant="soft_cap_sink", lse=True, lens=7),
        # the new tokens of one decode step of 61 requests
        _write("write_append", 61, "bf16"),
        # one prefill chunk from a model that keeps its activations in FP32, scales given by the caller
        _write("write_chunk", 8191, "f32", page=32, scaled=True),
        # a bulk load: long prompts written at once
        _write("write_bulk", 262144, "bf16"),
        # a serving step launched call by call, metadata on the device, batch smaller than the buffers
        _step("step_eager", 37, 64, 64, 500, 8000, lens=37),
        # the same from a captured graph, metadata from the scheduler's pinned host tensors
        _step("step_graph", 16, 16, 128, 200, 4000, graph=True, host=True, lens=16),
    ]


def _log_uniform(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1)))))))


def draw(rng):
    kind = rng.choices(("decode", "write", "step"), (6, 3, 3))[0]
    if kind == "write":
        return _write(None, _log_uniform(rng, 1, 262144), rng.choice(("bf16", "bf16", "f16", "f32")), rng.choice((16, 32, 64, 128)),
                      rng.random() < 0.25)
    heads = rng.choice((8, 16, 32, 64, 64, 128, 128, rng.randint(1, 128)))
    page = rng.choice((8, 16, 32, 64, 64, 64, 128))
    q_len = rng.choice((1, 1, 1, 1, 2, 3))
    lens = rng.randrange(1 << 30)
    # as many tokens as the largest listed decode reads: 750 000 for one group of 64 heads, fewer for more groups
    budget = 750000 // (q_len * -(-heads // 64))
    hi = min(budget, _log_uniform(rng, 16, 131072))
    lo = hi if rng.random() < 0.25 else max(1, int(hi / math.exp(rng.uniform(0.0, 5.0))))
    if kind == "step":
        hi, lo = min(hi, 16384), min(lo, 16384)
    batch = _log_uniform(rng, 1, max(1, min(128, budget // hi)))
    if kind == "step":
        lo, hi = max(lo, q_len), max(hi, q_len)
        return _step(None, batch, batch + rng.choice((0, 0, rng.randint(1, 32))), heads, lo, hi, page, q_len, rng.random() < 0.5,
                     rng.random() < 0.5, lens)
    return _decode(None, batch, heads, lo, hi, page, q_len, rng.choice(("bf16", "bf16", "bf16", "f32", "e4m3")),
                   rng.choice(("none", "none", "none", "sink", "soft_cap")), rng.random() < 0.3,
                   rng.choice(("normal", "normal", "student_t3")), lens)


def _lengths(case):
    """The requests' lengths: part of the case, the same whatever the inputs."""
    rng = random.Random(case["lens"])
    return [_log_uniform(rng, case["lo"], case["hi"]) for _ in range(case["batch"])]


def _tokens(n, dtype, gen, dev):
    """Compressed KV and RoPE keys of n tokens; the magnitude differs from token to token as activations do."""
    size = torch.rand(n, 1, generator=gen, device=dev) * 3 + 0.25
    latent = (torch.randn(n, 512, generator=gen, device=dev) * size).to(dtype)
    return latent, torch.randn(n, 64, generator=gen, device=dev).to(dtype)


def _prepare_decode(case, seed, dev):
    c = synth.build_case("decode", _lengths(case), case["heads"], case["page"], case["q_len"], seed, dev, latent_dist=case["latent"])
    sink = torch.randn(case["heads"], generator=torch.Generator().manual_seed(seed)).to(dev) if "sink" in case["variant"] else None
    variant = SoftCappingAttention(30.0, sink) if "soft_cap" in case["variant"] else (AttentionWithSink(sink) if sink is not None else None)
    w = BatchMLADecodeCuteDSLFP4Wrapper(torch.empty(32 << 20, dtype=torch.int8, device=dev))
    w.plan(num_heads=case["heads"], page_size=case["page"], out_dtype=_OUT[case["out"]], variant=variant)
    # the attention output shrinks with the root of the length: an E4M3 result is brought into that type's range
    scale = 16.0 if case["out"] == "e4m3" else 1.0
    return {"kind": "decode", "w": w, "c": c, "max_len": c.max_seq_len, "lse": case["lse"], "out_scale": scale}


def _prepare_write(case, seed, dev):
    gen = torch.Generator(device=dev).manual_seed(seed)
    n, page = case["tokens"], case["page"]
    latent, rope = _tokens(n, _IN[case["dtype"]], gen, dev)
    pages = 2 * -(-n // page)
    order = torch.randperm(pages, generator=gen, device=dev)
    at = torch.arange(n, device=dev)
    if n <= 256:  # one token per request, each at the end of its own sequence
        pages = max(pages, 2 * n)
        slots = torch.randperm(pages, generator=gen, device=dev)[:n] * page + torch.randint(0, page, (n,), generator=gen, device=dev)
    else:  # consecutive tokens of scattered pages
        slots = order[at // page] * page + at % page
    cache = FP4MLAPagedCache(pages, page, dev)
    scale = latent.float().abs().amax(1) / 5.5 if case["scaled"] else None
    return {"kind": "write", "latent": latent, "rope": rope, "slots": slots, "cache": cache, "scale": scale}


def _prepare_step(case, seed, dev):
    gen = torch.Generator(device=dev).manual_seed(seed)
    batch, page, q_len, lens = case["batch"], case["page"], case["q_len"], _lengths(case)
    c = synth.build_case("step", lens, case["heads"], page, q_len, seed, dev)
    cache = FP4MLAPagedCache(c.kv_cache.shape[0], page, dev)
    cache.kv_cache.copy_(c.kv_cache)
    cache.kv_cache_sf.copy_(c.kv_cache_sf)
    backend = FP4MLADecodeBackend(case["heads"], page, case["max_batch"], case["hi"], c.softmax_scale, dev, q_len=q_len)
    latent, rope = _tokens(batch * q_len, torch.bfloat16, gen, dev)
    bt, sl = c.block_tables, c.seq_lens
    if case["host"]:
        bt, sl = bt.cpu().pin_memory(), sl.cpu().pin_memory()
    return {"kind": "step", "backend": backend, "cache": cache, "bt": bt, "sl": sl, "q": c.q, "latent": latent, "rope": rope,
            "step": backend.capture(cache) if case["graph"] else None}


def prepare(case, seed):
    return {"decode": _prepare_decode, "write": _prepare_write, "step": _prepare_step}[case["kind"]](case, seed, torch.device("cuda:0"))


def run(state):
    if state["kind"] == "decode":
        c = state["c"]
        return state["w"].run(c.q, c.kv_cache, c.block_tables, c.seq_lens, state["max_len"], c.softmax_scale,
                              output_scale=state["out_scale"], kv_cache_sf=c.kv_cache_sf, return_lse=state["lse"])
    cache = state["cache"]
    if state["kind"] == "write":
        write_tokens(state["latent"], state["rope"], state["slots"], cache.kv_cache, cache.kv_cache_sf, state["scale"])
        return cache.kv_cache, cache.kv_cache_sf
    backend, step = state["backend"], state["step"]
    n = backend.prepare(state["bt"], state["sl"])
    if step is None:
        out = backend.forward(state["q"], state["latent"], state["rope"], cache)
    else:
        step.q[:n].copy_(state["q"])
        step.latent[: state["latent"].shape[0]].copy_(state["latent"])
        step.rope[: state["rope"].shape[0]].copy_(state["rope"])
        out = step.replay()[:n]
    return out, cache.kv_cache, cache.kv_cache_sf


def work(case):
    if case["kind"] == "write":
        per = 576 * (4 if case["dtype"] == "f32" else 2) + 324 + 8 + (4 if case["scaled"] else 0)
        return {"bytes": per * case["tokens"], "flops": 0}
    lens = _lengths(case)
    rows = case["batch"] * case["q_len"] * case["heads"]
    pages = sum(-(-n // case["page"]) for n in lens)
    out = {"bf16": 2, "f32": 4, "e4m3": 1}[case.get("out", "bf16")]
    total = 324 * sum(lens) + rows * (576 + 512 * out + (4 if case.get("lse") else 0)) + 4 * pages + 4 * case["batch"]
    if case["kind"] == "step":
        total += case["batch"] * case["q_len"] * (576 * 2 + 324)
    return {"bytes": total, "flops": 2176 * sum(lens) * case["heads"] * case["q_len"]}


def tolerance(case):
    if case["kind"] == "write":
        return "exact"  # the format fixes every byte
    if case.get("out") == "e4m3":
        return {"rel": 3e-2, "max": 0.15}  # neighbouring E4M3 values are an eighth apart
    # the probabilities enter the second product with about eight bits: 1e-2 of the output's RMS at worst, on either side
    return {"rel": 5e-3, "max": 5e-2}
