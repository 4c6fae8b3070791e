"""The work users of this library have it do, as cases that can be timed and compared: whole requests through the decoder's public calls.

A case names a model shape, how its weights are stored, and a kind of request with its sizes:
  chat        a prompt in one call, then greedy generation with steps queued ahead (eval_tokens, logits, generate)
  sample      one token per call, the logits read after each: what a caller that samples on the host does (eval_tokens, logits)
  image       the rows of an image between two pieces of text (embed_tokens, eval_embeddings), then greedy generation
  batch       many sequences in one batch: every prompt into its slot, then batched steps (serving.run_batched)
  continuous  more sequences than slots (serving.run_continuous)

The models are the benchmark configurations' architectures (dooms_b200/synth.py) with seeded normal weights, quantized like theirs. So that greedy tokens
are decided by a clear margin, as a trained model's mostly are, and not by rounding, the output row of a token is the (scaled) embedding row of the token
before it in a fixed walk through the vocabulary, embedding rows have unit variance and the projections that write to the residual row are scaled by
1 / sqrt(2 n_layer). A decoder keeps one set of weights, as a user's does; prompts, images and sequence lengths come from the seed.
"""
from __future__ import annotations

import dataclasses
import json
import math
import weakref

import numpy as np
import torch

from dooms_b200 import CudaLlamaDecoder, LlamaDecoderConfig, serving, synth
from dooms_b200 import _lib as L
from dooms_b200.decoder import weight_ref
from dooms_b200.quantize import quantize

WALK_STEP = 7919        # token t is followed by (WALK_STEP t + 1) mod n_vocab
QUEUE_DEPTH = 4


def listed():
    return [
        # the smallest calls: a short context on the small model, the caller samples on the host after every token
        {"name": "sample_small_q4_0", "model": "small", "weights": "q4_0", "kind": "sample", "prompt": 23, "tokens": 16, "n_batch": 512, "rows": 1},
        # the small model's benchmark request, in its two quantizations
        {"name": "chat_small_q4_0", "model": "small", "weights": "q4_0", "kind": "chat", "prompt": 512, "tokens": 128, "n_batch": 512, "rows": 1},
        {"name": "chat_small_mix", "model": "small", "weights": "mix", "kind": "chat", "prompt": 512, "tokens": 128, "n_batch": 512, "rows": 1},
        # unquantized weights, the form published models come in; a prompt of no round length
        {"name": "chat_small_f16", "model": "small", "weights": "f16", "kind": "chat", "prompt": 181, "tokens": 64, "n_batch": 512, "rows": 1},
        # a long document in chunks of the default size, then a short answer over a long cache
        {"name": "document_small_q4_0", "model": "small", "weights": "q4_0", "kind": "chat", "prompt": 6007, "tokens": 48, "n_batch": 512, "rows": 1},
        # the text side of a vision-language request
        {"name": "image_small_mix", "model": "small", "weights": "mix", "kind": "image", "prompt": 43, "tokens": 32, "n_batch": 512, "rows": 729},
        # the 8B shape: the benchmark's prompt with an answer, and a short question whose prompt is less than one token tile
        {"name": "chat_8b_q4_0", "model": "8b", "weights": "q4_0", "kind": "chat", "prompt": 2048, "tokens": 128, "n_batch": 2048, "rows": 1},
        {"name": "question_8b_q4_0", "model": "8b", "weights": "q4_0", "kind": "chat", "prompt": 37, "tokens": 48, "n_batch": 512, "rows": 1},
        # the 32B shape, four of its layers: a document of 8192 tokens
        {"name": "document_32b_mix", "model": "32b", "weights": "mix", "kind": "chat", "prompt": 8192, "tokens": 32, "n_batch": 2048, "rows": 1},
        # serving: one batch of many sequences; and more sequences than slots
        {"name": "batch_small_q4_0", "model": "small", "weights": "q4_0", "kind": "batch", "prompt": 512, "tokens": 96, "n_batch": 2048, "rows": 128},
        {"name": "continuous_small_q4_0", "model": "small", "weights": "q4_0", "kind": "continuous", "prompt": 300, "tokens": 64, "n_batch": 512, "rows": 16},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    model = rng.choice(["small", "small", "small", "8b", "32b"])
    if model == "8b":
        kind, weights = rng.choice(["chat", "chat", "sample"]), "q4_0"
        prompt, tokens = (size(16, 2048), size(8, 96)) if kind == "chat" else (size(8, 512), size(4, 32))
        n_batch, rows = rng.choice([512, 2048]), 1
    elif model == "32b":
        kind, weights = "chat", "mix"
        prompt, tokens, n_batch, rows = size(64, 8000), size(4, 64), rng.choice([512, 2048]), 1
    else:
        kind = rng.choice(["chat", "chat", "sample", "image", "batch", "continuous"])
        weights = "q4_0" if kind in ("batch", "continuous") else rng.choice(["q4_0", "mix", "f16"])
        n_batch = rng.choice([512, 2048])
        if kind == "chat":
            prompt, tokens, rows = size(8, 8000), size(8, 128), 1
        elif kind == "sample":
            prompt, tokens, rows = size(4, 512), size(4, 48), 1
        elif kind == "image":
            prompt, tokens, rows = size(8, 200), size(8, 64), size(49, 1500)
        else:
            prompt, tokens, rows = size(64, 512), size(16, 96), size(4, 96 if kind == "batch" else 24)
    return {"model": model, "weights": weights, "kind": kind, "prompt": prompt, "tokens": tokens, "n_batch": n_batch, "rows": rows}


# ---------------------------------------------------------------- models

def _spec(case) -> synth.ModelSpec:
    spec = synth.config_spec({"small": 0, "8b": 2, "32b": 3}[case["model"]])
    if case["model"] == "32b":
        spec = dataclasses.replace(spec, n_layer=4)      # four layers of the 64: a layer costs what it costs in the whole model
    plans = {"q4_0": synth.pure(L.Q4_0), "f16": synth.pure(L.F16), "mix": synth.q4_k_m_small if case["model"] == "small" else synth.q4_k_m_large}
    return dataclasses.replace(spec, plan=plans[case["weights"]], tied=False)


def _sequences(case, seed):
    """(prompt, tokens to generate) of every sequence of a batch or continuous case: the lengths, uniform up to the case's, belong to the case, the ids to the
    seed."""
    n = case["rows"] if case["kind"] == "batch" else 3 * case["rows"]
    V = _spec(case).n_vocab
    lengths = serving.workload(n, V, 3000, (min(32, case["prompt"]), case["prompt"]), (min(8, case["tokens"]), case["tokens"]))
    g = np.random.Generator(np.random.PCG64(seed))
    return [(g.integers(0, V, len(p), dtype=np.int32), n_decode) for p, n_decode in lengths]


def _build(case) -> CudaLlamaDecoder:
    spec = _spec(case)
    E, F, V, hd = spec.n_embd, spec.n_ff, spec.n_vocab, spec.head_dim
    kv = spec.n_head_kv * hd
    gen = torch.Generator(device="cuda")
    gen.manual_seed(1000)
    keep = []

    def ref(kind, layer, values):
        dt = spec.plan(kind, layer)
        rows = max(1, (1 << 26) // values.shape[1])
        blocks = torch.cat([quantize(dt, values[r:r + rows]) for r in range(0, values.shape[0], rows)])
        keep.append(blocks.cpu().numpy())
        return weight_ref(keep[-1], dt, values.shape[0], values.shape[1])

    def normal(rows, cols, std):
        return torch.randn((rows, cols), generator=gen, device="cuda", dtype=torch.float32).mul_(std)

    def vector(n, lo, hi):
        keep.append((torch.rand(n, generator=gen, device="cuda") * (hi - lo) + lo).cpu().numpy())
        return weight_ref(keep[-1], L.F32, 1, n)

    table = normal(V, E, 1.0)
    embd = ref("token_embd", -1, table)
    nxt = (torch.arange(V, device="cuda") * WALK_STEP + 1) % V
    out_rows = torch.empty_like(table)
    out_rows[nxt] = table
    output = ref("output", -1, out_rows.mul_(0.02))
    del table, out_rows
    into_x = 0.02 / math.sqrt(2 * spec.n_layer)
    pattern = []                       # the weights of an even and of an odd layer, shared by all layers of that parity
    for l in range(min(2, spec.n_layer)):
        w = {"attn_norm": vector(E, 0.7, 1.3), "ffn_norm": vector(E, 0.7, 1.3)}
        for kind, rows, cols, std in (("attn_q", E, E, 0.02), ("attn_k", kv, E, 0.02), ("attn_v", kv, E, 0.02), ("attn_output", E, E, into_x), ("ffn_gate", F, E, 0.02),
                                      ("ffn_up", F, E, 0.02), ("ffn_down", E, F, into_x)):
            w[kind] = ref(kind, l, normal(rows, cols, std))
        if spec.bias:
            for kind, n in (("attn_q", E), ("attn_k", kv), ("attn_v", kv)):
                w[kind + "_bias"] = vector(n, -0.03, 0.03)
        pattern.append(w)
    norm = vector(E, 0.7, 1.3)
    torch.cuda.empty_cache()
    many = case["kind"] in ("batch", "continuous")
    need = case["prompt"] + case["tokens"] + 8 + (case["rows"] if case["kind"] == "image" else 0)
    n_ctx = need if many else max(2048, -(-need // 1024) * 1024)
    config = LlamaDecoderConfig(n_layer=spec.n_layer, n_embd=E, n_head=spec.n_head, n_head_kv=spec.n_head_kv, head_dim=hd, n_ff=F, n_vocab=V, rope_base=spec.rope_base,
                                rope_neox=spec.arch == "qwen2", rms_eps=spec.rms_eps, n_ctx=n_ctx, n_batch=min(case["n_batch"], n_ctx))
    return CudaLlamaDecoder.create(config, embd, norm, output, [pattern[l % 2] for l in range(spec.n_layer)], max_sequences=max(2, case["rows"]) if many else 1)


_decoders: "weakref.WeakValueDictionary[str, CudaLlamaDecoder]" = weakref.WeakValueDictionary()


def _decoder(case) -> CudaLlamaDecoder:
    """The case's decoder; requests that are alive together share one, as a program's requests do. It goes when the last of them goes."""
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    dec = _decoders.get(key)
    if dec is None:
        dec = _decoders[key] = _build(case)
    return dec


# ---------------------------------------------------------------- requests

def prepare(case, seed):
    dec, spec, g = _decoder(case), _spec(case), np.random.Generator(np.random.PCG64(seed))
    state = {"case": case, "dec": dec}
    if case["kind"] in ("batch", "continuous"):
        state["sequences"] = _sequences(case, seed)
        return state
    state["prompt"] = g.integers(0, spec.n_vocab, case["prompt"], dtype=np.int32)
    if case["kind"] == "sample":
        state["sampled"] = g.integers(0, spec.n_vocab, case["tokens"], dtype=np.int32)      # what the caller's sampler picks
    if case["kind"] == "image":
        state["image"] = g.standard_normal((case["rows"], spec.n_embd), dtype=np.float32)
    return state


def _answer(dec, n):
    """Greedy tokens; then the last one is evaluated too, so that the next turn can go on from it, and its logits come back."""
    tokens: list[int] = []
    dec.generate(n, QUEUE_DEPTH, lambda t: tokens.append(t) or True)
    dec.eval_tokens(tokens[-1:])
    return {"tokens": np.array(tokens, dtype=np.int32), "last": dec.logits()}


def run(state):
    case, dec = state["case"], state["dec"]
    kind = case["kind"]
    if kind == "chat":
        dec.reset()
        dec.eval_tokens(state["prompt"])
        first = dec.logits()
        return {"first": first, **_answer(dec, case["tokens"])}
    if kind == "sample":
        dec.reset()
        dec.eval_tokens(state["prompt"])
        rows = [dec.logits()]
        for t in state["sampled"]:
            dec.eval_tokens([t])
            rows.append(dec.logits())
        return {"logits": rows}
    if kind == "image":
        dec.reset()
        half = case["prompt"] // 2
        rows = np.concatenate([dec.embed_tokens(state["prompt"][:half]), state["image"], dec.embed_tokens(state["prompt"][half:])])
        dec.eval_embeddings(rows)
        first = dec.logits()
        return {"first": first, **_answer(dec, case["tokens"])}
    if kind == "batch":
        tokens, _ = serving.run_batched(dec, state["sequences"])
        dec.select_sequence(0)                          # one of them goes on alone
        dec.eval_tokens(tokens[0][-1:])
        return {"tokens": np.array(sum(tokens, []), dtype=np.int32), "last": dec.logits()}
    tokens, _ = serving.run_continuous(dec, state["sequences"], case["rows"])
    return {"tokens": np.array(sum(tokens, []), dtype=np.int32)}


def work(case):
    spec = _spec(case)
    E, F, V, hd = spec.n_embd, spec.n_ff, spec.n_vocab, spec.head_dim
    kv = spec.n_head_kv * hd
    layer_weights = spec.n_layer * (2 * E * E + 2 * E * kv + 3 * E * F)
    matrix_bytes = spec.matrix_bytes()
    kv_row = spec.n_layer * 2 * kv * 2                   # bytes of one position's keys and values

    def request(n_prompt, n_steps):
        """(flops, bytes of keys and values read and written) of a prompt and n_steps single positions after it."""
        total = n_prompt + n_steps
        flops = 2.0 * layer_weights * total + 2.0 * V * E * (1 + n_steps) + 4.0 * E * spec.n_layer * total * (total + 1) / 2
        return flops, kv_row * (total + sum(range(n_prompt, total)))
    if case["kind"] in ("batch", "continuous"):
        sequences = _sequences(case, 1)
        parts = [request(len(p), n - 1) for p, n in sequences]
        steps = max(n for _, n in sequences) if case["kind"] == "batch" else -(-sum(n for _, n in sequences) // case["rows"])
        return {"flops": sum(p[0] for p in parts), "bytes": matrix_bytes * steps + sum(p[1] for p in parts)}
    rows = case["prompt"] + (case["rows"] if case["kind"] == "image" else 0)
    flops, cache = request(rows, case["tokens"])
    logits = 4 * V * (case["tokens"] + 1 if case["kind"] == "sample" else 2)
    return {"flops": flops, "bytes": matrix_bytes * (1 + case["tokens"]) + cache + logits}


def tolerance(case):
    # A prompt's projections multiply operands rounded to f16 and add in f32. The same requests with every projection in f32 (prefill_tile = 1) differ by up to
    # 2.2e-4 (2-norm) and 1.0e-3 (largest) in the logits on the small shape and by 1.0e-3 and 4.4e-3 on the two deeper / wider ones: four times that. Greedy
    # tokens are decided by margins far above it.
    return {"rel": 1e-3, "max": 5e-3} if case["model"] == "small" else {"rel": 4e-3, "max": 2e-2}
