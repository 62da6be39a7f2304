"""The work that a user of this library has it do, as cases that can be timed and compared.

Three kinds of calls, all through the public binding (``litenn_b200.capi``, ``litenn_b200.llama``):

  matvec    ``Weight.gemv_f32``: 1..16 fp32 activation rows times a block-quantized weight, the linear layers of
            decoding.  A pass walks ``copies`` different weights, as a model walks its layers.
  gemm      ``Weight.gemm_bf16`` / ``Weight.gemm_f32``: many activation rows, the linear layers of a prompt.
  generate  ``LlamaModel``: a prompt through the prefill and tokens after it, for one sequence (``prefill`` and
            ``decode``, or ``step_host`` and ``last_logits`` where the host chooses the tokens) or for a batch of
            them (``batch_prefill``, ``batch_decode``).

Inputs are synthetic: payloads with the distributions of ``litenn_b200/synth.py``, activations ~ N(0, 1), random
token ids.
"""
from __future__ import annotations

import numpy as np
import torch

from litenn_b200 import capi, synth
from litenn_b200 import llama as ll

FORMATS = {"q4_0": synth.Q4_0, "q8_0": synth.Q8_0, "q4_k": synth.Q4_K, "q6_k": synth.Q6_K}
COPIED_BYTES = 640_000_000      # most bytes of weights that a matvec case keeps
DRAWN_WEIGHT_BYTES = 400_000_000  # most bytes of linear weights of a drawn model


def _matvec(name, fmt, n, k, m, copies):
    return {"name": name, "kind": "matvec", "fmt": fmt, "n": n, "k": k, "m": m, "copies": copies}


def _gemm(name, fmt, n, k, m, x, y):
    return {"name": name, "kind": "gemm", "fmt": fmt, "n": n, "k": k, "m": m, "x": x, "y": y}


def _generate(name, layers, d, heads, kv_heads, head_dim, ffn, vocab, fmt, down_fmt, embd_fmt, prompt, steps,
              batch=0, drive="device", tied=False):
    """``batch`` 0: one sequence.  ``drive``: who chooses the next token, the "device" (greedy) or the "host", which
    reads the logits after each step; here it goes on with a given text, as a scorer does."""
    return {"name": name, "kind": "generate", "layers": layers, "d": d, "heads": heads, "kv_heads": kv_heads,
            "head_dim": head_dim, "ffn": ffn, "vocab": vocab, "fmt": fmt, "down_fmt": down_fmt, "embd_fmt": embd_fmt,
            "prompt": prompt, "steps": steps, "batch": batch, "drive": drive, "tied": tied}


def listed():
    return [
        # one small matvec on its own: what a single MatMul node of a graph runner costs
        _matvec("matvec_q8_0_4096_b1", "q8_0", 4096, 4096, 1, 1),
        # the FFN projections of a 7B-shape decoder's layers, one token
        _matvec("matvec_q4_0_ffn_b1", "q4_0", 11008, 4096, 1, 12),
        # the way down of the same FFN for a handful of sequences, and for an odd number of rows of a K-quant model
        _matvec("matvec_q4_0_down_b8", "q4_0", 4096, 11008, 8, 12),
        # the widest projection of a 70B-shape layer for a full decoding batch
        _matvec("matvec_q4_k_wide_b16", "q4_k", 28672, 8192, 16, 4),
        # a prompt of 512 tokens through one FFN projection, bf16 activations
        _gemm("gemm_q4_k_512", "q4_k", 14336, 4096, 512, "bf16", "f32"),
        # a short odd prompt from an fp32 graph: padding counts here
        _gemm("gemm_q6_k_77_f32", "q6_k", 4096, 11008, 77, "f32", "f32"),
        # several prompts of a server in one product, results passed on as bf16
        _gemm("gemm_q8_0_2048_bf16", "q8_0", 4096, 4096, 2048, "bf16", "bf16"),
        # a chat answer of a 7B-shape model: 512-token prompt, 128 greedy tokens
        _generate("generate_7b", 32, 4096, 32, 32, 128, 11008, 32000, "q4_0", "q4_0", "q6_k", 512, 128),
        # a long document and one token: what the first answer waits for (the blocks repeat, four stand for all)
        _generate("prompt_7b_1999", 4, 4096, 32, 32, 128, 11008, 32000, "q4_0", "q4_0", "q6_k", 1999, 0),
        # 70B-shape layers (grouped heads, mixed K-quants), long prompt and an answer
        _generate("generate_70b_layers", 4, 8192, 64, 8, 128, 28672, 32000, "q4_k", "q6_k", "q6_k", 1024, 64),
        # sixteen sequences of a server at once
        _generate("batch16_7b_layers", 8, 4096, 32, 32, 128, 11008, 32000, "q4_k", "q6_k", "q6_k", 64, 64, 16),
        # a small model whose host reads the logits and feeds every token: launches and latency
        _generate("small_host_loop", 2, 512, 8, 2, 64, 1536, 1024, "q8_0", "q8_0", "q8_0", 20, 32, 0, "host", True),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["matvec", "gemm", "generate"])
    fmt = rng.choice(list(FORMATS))
    unit = synth.BLOCK_ELEMS[FORMATS[fmt]]
    if kind == "matvec":
        k = max(1, _log(rng, 256, 28672) // unit) * unit
        n = _log(rng, 48, 28672)
        m = rng.choice([1, 1, 1, rng.randint(2, 16)])
        most = COPIED_BYTES // synth.payload_nbytes(FORMATS[fmt], n, k)
        case = _matvec("", fmt, n, k, m, max(1, min(most, rng.choice([1, 6, 12]))))
    elif kind == "gemm":
        k = max(1, _log(rng, 512, 16384) // unit) * unit
        x = rng.choice(["bf16", "bf16", "f32"])
        y = "f32" if x == "f32" else rng.choice(["f32", "bf16"])
        case = _gemm("", fmt, _log(rng, 512, 16384), k, _log(rng, 17, 2048), x, y)
    else:
        batch = rng.choice([0, 0, rng.randint(2, 16)])
        # Random blocks of 32 make shallow models whose greedy text is chaotic: one near-tie and all that follows
        # is another text.  Those models score a given text; K-quant models settle and may choose greedily.
        fmt = "q4_k" if batch else rng.choice(["q4_0", "q4_0", "q4_k", "q8_0"])
        down = "q6_k" if fmt == "q4_k" else fmt
        head_dim = rng.choice([64, 128])
        d = max(1, _log(rng, 256, 8192) // 256) * 256
        heads = d // head_dim
        kv = rng.choice([v for v in range(1, heads + 1) if heads % v == 0 and heads // v in (1, 2, 4, 8)])
        ffn = max(1, int(d * rng.uniform(2.0, 3.5)) // 256) * 256
        vocab = _log(rng, 1024, 32000) // 8 * 8
        per_layer = sum(synth.payload_nbytes(FORMATS[f], n, k) for f, n, k in (
            (fmt, d + 2 * kv * head_dim, d), (fmt, d, d), (fmt, 2 * ffn, d), (down, d, ffn)))
        layers = max(1, min(4, rng.randint(1, 4), DRAWN_WEIGHT_BYTES // per_layer))
        prompt = _log(rng, 8, 1999) if batch == 0 else _log(rng, 8, 128)
        steps = rng.choice([1, 16, rng.randint(1, 64)])
        case = _generate("", layers, d, heads, kv, head_dim, ffn, vocab, fmt, down, rng.choice(["q6_k", "q8_0"]), prompt,
                         steps, batch, "device" if fmt == "q4_k" else "host", rng.random() < 0.3)
    del case["name"]
    return case


# ---- inputs ----------------------------------------------------------------------------------------------

def _payload_on_gpu(fmt, n, k, gen):
    """Raw ggml blocks of an [n, k] weight, made on the GPU with the distributions of synth.make_weight."""
    nblk = n * (k // synth.BLOCK_ELEMS[fmt])
    out = torch.randint(0, 256, (nblk, synth.BLOCK_BYTES[fmt]), dtype=torch.uint8, device="cuda", generator=gen)

    def scale(col, sigma, div):
        v = torch.randn(nblk, device="cuda", generator=gen).abs_() * (sigma / div)
        out[:, col:col + 2] = v.half().view(torch.uint8).view(nblk, 2)

    if fmt == synth.Q8_0:
        out[:, 2:][out[:, 2:] == 128] = 127  # quants are -127..127
        scale(0, 0.02, 127.0)
    elif fmt == synth.Q4_0:
        scale(0, 0.02, 8.0)
    elif fmt == synth.Q4_K:
        scale(0, 0.01, 1.0)
        scale(2, 0.01, 1.0)
    else:
        scale(208, 0.01, 1.0)
    return out


def _weight(fmt, n, k, gen):
    raw = _payload_on_gpu(fmt, n, k, gen)
    torch.cuda.synchronize()  # the payload is complete before the library reads it on its own stream
    return capi.Weight.from_device(fmt, raw.data_ptr(), raw.numel(), n, k)


def prepare(case, seed):
    if case["kind"] == "generate":
        return _prepare_generate(case, seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    fmt, n, k, m = FORMATS[case["fmt"]], case["n"], case["k"], case["m"]
    state = {"case": case}
    if case["kind"] == "matvec":
        state["w"] = [_weight(fmt, n, k, gen) for _ in range(case["copies"])]
        state["x"] = torch.randn(case["copies"], m, k, device="cuda", generator=gen)
        state["y"] = torch.empty(case["copies"], m, n, device="cuda")
    else:
        state["w"] = _weight(fmt, n, k, gen)
        x = torch.randn(m, k, device="cuda", generator=gen)
        state["x"] = x.bfloat16() if case["x"] == "bf16" else x
        state["y"] = torch.empty(m, n, device="cuda", dtype=torch.bfloat16 if case["y"] == "bf16" else torch.float32)
    return state


def _prepare_generate(case, seed):
    prompts = max(1, case["batch"])
    spec = ll.LlamaSpec(case["layers"], case["d"], case["heads"], case["kv_heads"], case["head_dim"], case["ffn"],
                        case["vocab"], FORMATS[case["fmt"]], FORMATS[case["down_fmt"]], FORMATS[case["embd_fmt"]],
                        max_seq=case["prompt"] + case["steps"] + 1, max_prefill=case["prompt"],
                        unit_norms=False, tied_output=case["tied"])
    stream = torch.cuda.Stream()
    model = ll.LlamaModel(spec, stream=stream.cuda_stream, seed=seed, share_layer_payloads=True)
    if case["batch"]:
        model.batch_create(case["batch"], max(1, case["steps"]))
    tokens = [synth.make_token_ids(case["prompt"], case["vocab"], seed=seed, name=f"prompt{i}") for i in range(prompts)]
    return {"case": case, "stream": stream, "model": model, "prompts": tokens,
            "text": synth.make_token_ids(max(1, case["steps"]), case["vocab"], seed=seed, name="text").tolist()}


# ---- one pass --------------------------------------------------------------------------------------------

def run(state):
    case = state["case"]
    if case["kind"] == "matvec":
        stream = torch.cuda.current_stream().cuda_stream
        for w, x, y in zip(state["w"], state["x"], state["y"]):
            w.gemv_f32(x.data_ptr(), y.data_ptr(), case["m"], stream)
        return state["y"]
    if case["kind"] == "gemm":
        stream = torch.cuda.current_stream().cuda_stream
        w, x, y = state["w"], state["x"], state["y"]
        if case["x"] == "f32":
            w.gemm_f32(x.data_ptr(), y.data_ptr(), case["m"], stream)
        else:
            w.gemm_bf16(x.data_ptr(), y.data_ptr(), case["m"],
                        capi.OUT_BF16 if case["y"] == "bf16" else capi.OUT_F32, stream)
        return y
    model, steps = state["model"], case["steps"]
    model.reset()
    if case["batch"]:
        first = np.array([model.batch_prefill(i, p) for i, p in enumerate(state["prompts"])], dtype=np.int32)
        logits = model.last_logits()  # of the last prompt: the batch's own are not handed out
        return {"first": first, "tokens": model.batch_decode(steps), "logits": logits}
    first = model.prefill(state["prompts"][0])
    out = {"first": first, "prompt_logits": model.last_logits()}
    if steps == 0:
        return out
    if case["drive"] == "host":
        out["logits"] = []
        for token in state["text"]:
            model.step_host(token)
            out["logits"].append(model.last_logits())
        out["logits"] = np.stack(out["logits"])
    else:
        out["tokens"] = model.decode(steps)
        out["logits"] = model.last_logits()
    return out


# ---- what a pass cannot do without, and how far apart correct results lie ----------------------------------

def work(case):
    if case["kind"] != "generate":
        fmt, n, k, m = FORMATS[case["fmt"]], case["n"], case["k"], case["m"]
        copies = case.get("copies", 1)
        x_item = 2 if case.get("x") == "bf16" else 4
        y_item = 2 if case.get("y") == "bf16" else 4
        return {"bytes": copies * (synth.payload_nbytes(fmt, n, k) + m * k * x_item + m * n * y_item),
                "flops": copies * 2 * m * n * k}
    d, ffn, layers, prompt, steps = case["d"], case["ffn"], case["layers"], case["prompt"], case["steps"]
    q_w, kv_w = case["heads"] * case["head_dim"], case["kv_heads"] * case["head_dim"]
    fmt, down = FORMATS[case["fmt"]], FORMATS[case["down_fmt"]]
    block = (synth.payload_nbytes(fmt, q_w + 2 * kv_w, d) + synth.payload_nbytes(fmt, d, q_w) +
             synth.payload_nbytes(fmt, 2 * ffn, d) + synth.payload_nbytes(down, d, ffn))
    head = synth.payload_nbytes(FORMATS[case["embd_fmt"]], case["vocab"], d)
    weights = layers * block + head
    mults = layers * (d * (q_w + 2 * kv_w) + q_w * d + 3 * d * ffn)
    seqs = max(1, case["batch"])
    # prompts: every weight once per prompt, keys and values written once; causal attention
    nbytes = seqs * (weights + layers * prompt * 2 * kv_w * 2)
    flops = seqs * (2 * prompt * mults + 2 * case["vocab"] * d + layers * 2 * q_w * prompt * (prompt + 1))
    # steps: every weight once per step for the whole batch, each sequence's cached keys and values once
    cached = sum(prompt + s + 1 for s in range(steps))
    nbytes += steps * weights + seqs * layers * cached * 2 * kv_w * 2
    flops += seqs * (steps * 2 * (mults + case["vocab"] * d) + layers * 4 * q_w * cached)
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """About four times what the same path shows against itself in 64 bits or with its sums in another order."""
    if case["kind"] == "matvec":
        return {"rel": 8e-5, "max": 4e-4}       # 2.1e-5 and 1.1e-4: activations quantized to 16 bits
    if case["kind"] == "gemm" and case["y"] == "f32":
        return {"rel": 5e-5, "max": 2e-4}       # 1.5e-5 and 5e-5 at k = 15072: the tensor core's accumulation
    if case["kind"] == "gemm":
        return {"rel": 6e-4, "max": 1.6e-2}     # 1.5e-4: bf16 results, some of them one unit off
    # 1.0e-4 and 4.5e-4 for a prompt taken in two pieces: sums that differ in the last bit flip bf16 roundings of the
    # activations between the layers, and another kernel flips more of them than a cut does
    return {"rel": 1e-3, "max": 5e-3, "differ": 0.01}
