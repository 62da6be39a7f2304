#!/usr/bin/env python
"""Benchmark of the block-quantized matmul hot path.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Headline workload (config.workload = "llama7b_q4_0_decode_b1"): the random-init 7B-shape
LLaMA decoder of the benchmark configurations (32 layers, d 4096, 32 heads, FFN 11008,
vocab 32000; Q4_0 linears, Q6_K embeddings/output, fp16 KV cache), a 512-token prompt
through the tcgen05 prefill path, then greedy decode at batch 1.  One *step* is one
decoded token; ``value`` is tokens per second over K steps after W warm-up steps, with
N > 1 as tensor parallelism over N GPUs (weights sharded; the two per-block sums after
attention-out and FFN-down and the arg-max candidates travel as packets over peer memory, NCCL
only for set-up and prefill), so scaling is "strong".  The 3.75 GB of weights
read per token are far larger than L2.  ``e2e`` drives every token from the host (token
H2D, step, token D2H, synchronize).

The same line carries the first half of the metric, the Q4_0 FFN GEMV W[11008,4096] at
batch 1 ("gemv"), and ``roofline`` for the kernel that dominates both: the batch-1 Q4_0
matvec, timed alone over 12 weight copies (304 MB > 2 x L2) visited round-robin.

``--impl reference`` times the CPU restatement of LiteNN's own path on the host cores
(dequantize once, then the fp32 i-k-j MatMul loop).  A step executes one block's seven linears
plus the output head on samples of their output rows (weights dequantized from real Q4_0 / Q6_K
payloads) and extrapolates to the whole token; the thread count is every core this process may
run on, whatever OMP_NUM_THREADS says.
"""
from __future__ import annotations

import argparse
import contextlib
import io
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from litenn_b200 import synth  # noqa: E402

N_OUT, K_IN = 11008, 4096          # W[11008, 4096]: the "4096x11008" FFN projection
BATCH = 1
WEIGHT_BYTES = N_OUT * (K_IN // 32) * 18
ALGO_BYTES = WEIGHT_BYTES + 4 * BATCH * (K_IN + N_OUT)   # 25,422,848 B
COPIES = 12                        # 12 x 25.4 MB = 304 MB > 2 x L2
FALLBACK_HBM_GBS = 6650.0
# dram__bytes_read.sum + dram__bytes_write.sum of one gemv_kernel launch (ncu
# capture summarised under profiles/); None until measured.
NCU_TRAFFIC_BYTES = 25395200


def measured_tensor_peak():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            return float(json.load(f)["bf16_tflops"]), "measured"
    except Exception:
        return 1590.0, "fallback"


def measured_peak():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            return float(json.load(f)["hbm_gbs"]), "measured"
    except Exception:
        return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """Samples SM clocks and throttle reasons with nvidia-smi while the timed region runs."""

    QUERY = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu_index = gpu_index
        self.proc = None
        self.lines = []
        self.thread = None

    def start(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={self.gpu_index}", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits",
                 "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
        except OSError:
            self.proc = None
            return
        self.thread = threading.Thread(target=self._pump, daemon=True)
        self.thread.start()

    def _pump(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        if self.thread:
            self.thread.join(timeout=2)
        sm, smax, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in self.lines:
            parts = [p.strip() for p in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                sm.append(float(parts[1]))
                smax.append(float(parts[2]))
            except ValueError:
                continue
            for name, val in zip(names, parts[5:9]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        return {
            "sm_mhz": float(np.median(sm)) if sm else None,
            "sm_max_mhz": float(max(smax)) if smax else None,
            "reasons": sorted(reasons),
            "samples": len(sm),
        }


def dist_env():
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    return rank, world, local


DECODE_WEIGHT_BYTES = 32 * 202375168 * 18 // 32 + 131072000 * 210 // 256   # 3,750,273,024 B per token
PROMPT_LEN = 512


def host_cores():
    try:
        return len(os.sched_getaffinity(0))
    except AttributeError:
        return os.cpu_count() or 1


class CpuDecodeSample:
    """One block's seven linears and the output head of the 7B shape on samples of their output
    rows: dequantized from real block payloads, transposed as LiteNN stores them, multiplied by
    the reference's fp32 i-k-j loop (Device.h:645-658), which is linear in the number of output
    columns, so each sample's time scales to the full matrix."""

    D, FFN, VOCAB, LAYERS = 4096, 11008, 32000, 32

    def __init__(self):
        import oracle
        self.oracle = oracle
        d, ffn = self.D, self.FFN
        # (name, full rows, k, format, sampled rows, how many such linears per block)
        plan = [("attn_qkvo", d, d, synth.Q4_0, 2048, 4), ("ffn_gate_up", ffn, d, synth.Q4_0, 2752, 2),
                ("ffn_down", d, ffn, synth.Q4_0, 2048, 1)]
        self.block = []
        for name, n, k, fmt, rows, count in plan:
            payload = synth.make_weight(fmt, rows, k, seed=0, name="cpu." + name)
            wt = oracle.transpose(oracle.dequant(fmt, payload, rows, k))       # [k, rows]
            x = synth.make_activation(1, k, seed=0, name="cpu.x." + name)
            self.block.append((x, wt, count * n / rows))
        payload = synth.make_weight(synth.Q6_K, 8000, d, seed=0, name="cpu.head")
        self.head = (synth.make_activation(1, d, seed=0, name="cpu.x.head"),
                     oracle.transpose(oracle.dequant(synth.Q6_K, payload, 8000, d)), self.VOCAB / 8000)
        payload = synth.make_weight(synth.Q4_0, 2752, K_IN, seed=0, name="cpu.gemv")
        self.gemv = (synth.make_activation(1, K_IN, seed=0, name="cpu.x.gemv"),
                     oracle.transpose(oracle.dequant(synth.Q4_0, payload, 2752, K_IN)), N_OUT / 2752)

    def _timed(self, item, threads):
        x, wt, scale = item
        t0 = time.perf_counter()
        self.oracle.matmul_ikj(x, wt, threads=threads)
        return (time.perf_counter() - t0) * scale

    def step(self, threads):
        """Runs the sample once; returns (seconds actually spent, seconds of a whole token extrapolated)."""
        t0 = time.perf_counter()
        t_block = sum(self._timed(it, threads) for it in self.block)
        t_head = self._timed(self.head, threads)
        return time.perf_counter() - t0, self.LAYERS * t_block + t_head

    def gemv_seconds(self, threads):
        return min(self._timed(self.gemv, threads) for _ in range(3))

    SAMPLE = ("fp32 i-k-j MatMul loop (Device.h:645-658) on weights dequantized from seeded Q4_0 / Q6_K payloads: per "
              "step one block's seven linears on 2048-2752 of their output rows each (scaled linearly) x 32 blocks + the "
              "output head on 8000 of 32000 rows; one-off dequantization, attention, norms and the interpreter's "
              "per-run weight copy excluded")


def cpu_decode_baseline(threads, steps=3, warmup=1, sample=None):
    sample = sample or CpuDecodeSample()
    for _ in range(warmup):
        sample.step(threads)
    spent, tokens = [], []
    for _ in range(steps):
        a, b = sample.step(threads)
        spent.append(a)
        tokens.append(b)
    t_token = float(np.mean(tokens))
    return {
        "value": 1.0 / t_token, "unit": "tok/s", "cores": threads, "kind": "port", "sample": CpuDecodeSample.SAMPLE,
        "seconds_per_token": t_token, "sample_seconds_per_step": float(np.mean(spent)),
        "gemv_gbs": ALGO_BYTES / sample.gemv_seconds(threads) / 1e9,
    }


def run_reference(args):
    rank, world, _ = dist_env()
    if rank != 0:
        return 0
    threads = host_cores()
    t0 = time.perf_counter()
    sample = CpuDecodeSample()
    res = cpu_decode_baseline(threads, steps=max(1, args.steps), warmup=max(1, args.warmup), sample=sample)
    one = cpu_decode_baseline(1, steps=3, warmup=1, sample=sample)
    line = {
        "impl": "reference",
        "metric": "7B-shape Q4_0 batch-1 decode tok/s",
        "value": res["value"],
        "unit": "tok/s",
        "n_gpus": args.gpus,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": res["seconds_per_token"] * 1e3,
        "higher_is_better": True,
        "scaling": "strong",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": {"workload": "llama7b_q4_0_decode_b1", "prompt": PROMPT_LEN, "batch": 1,
                   "l2": "CPU run", "extrapolated": True,
                   "sample_ms_per_step": res["sample_seconds_per_step"] * 1e3,
                   "note": "every step executes the sample; ms_per_step is the whole token extrapolated from it",
                   "single_core_tok_s": one["value"]},
        "cpu_baseline": {k: res[k] for k in ("value", "unit", "cores", "kind", "sample")},
        "gemv": {"value": res["gemv_gbs"], "unit": "GB/s", "workload": "q4_0_gemv_4096x11008_b1"},
        "e2e": {"value": res["value"], "unit": "tok/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
        "wall_s": time.perf_counter() - t0,
    }
    print(json.dumps(line))
    return 0


def gemv_micro(torch, capi, local, side, stream, steps, warmup):
    """The Q4_0 FFN GEMV at batch 1 over 12 weight copies, in us per call: the public call (one launch that packs and multiplies),
    the matvec kernel alone back to back (consecutive launches overlap through programmatic dependent
    launch), and the matvec kernel isolated (an ordinary one-element fill kernel between launches
    serializes them; its own time is measured separately and subtracted)."""
    weights = []
    for i in range(COPIES):
        payload = synth.make_weight(synth.Q4_0, N_OUT, K_IN, seed=0, name=f"bench.w{i % 2}")
        weights.append(capi.Weight.from_host(synth.Q4_0, payload, N_OUT, K_IN, device=local, stream=stream))
    x = torch.from_numpy(synth.make_activation(BATCH, K_IN, seed=0, name="bench.x")).cuda()
    ys = [torch.empty((BATCH, N_OUT), dtype=torch.float32, device="cuda") for _ in range(COPIES)]
    packed = torch.empty(capi.packed_activation_bytes(K_IN, BATCH), dtype=torch.uint8, device="cuda")
    capi.pack_activations(x.data_ptr(), BATCH, K_IN, packed.data_ptr(), device=local, stream=stream)
    dummy = torch.zeros(1, dtype=torch.float32, device="cuda")

    def step_full():
        for w, y in zip(weights, ys):
            w.gemv_f32(x.data_ptr(), y.data_ptr(), BATCH, stream)

    def step_kernel():
        for w, y in zip(weights, ys):
            w.gemv_packed(packed.data_ptr(), y.data_ptr(), BATCH, stream)

    def step_isolated():
        for w, y in zip(weights, ys):
            dummy.fill_(1.0)
            w.gemv_packed(packed.data_ptr(), y.data_ptr(), BATCH, stream)

    def step_fill_only():
        for _ in weights:
            dummy.fill_(1.0)

    out = []
    for fn in (step_full, step_kernel, step_isolated, step_fill_only):
        fn()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            fn()
        for _ in range(max(3, warmup)):
            g.replay()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(steps):
            g.replay()
        b.record()
        torch.cuda.synchronize()
        out.append(a.elapsed_time(b) * 1e3 / (steps * COPIES))
    capi.kernel_status(local)
    y0 = ys[0].cpu().numpy()
    if not np.isfinite(y0).all() or not np.abs(y0).max() > 0:
        raise SystemExit("bench.py: GEMV produced non-finite or all-zero output")
    for w in weights:
        w.destroy()
    return {"full_us": out[0], "kernel_us": out[1], "isolated_us": max(out[2] - out[3], 0.0), "fill_us": out[3],
            "y0": y0, "x": x.cpu().numpy()}


def gemv_error_vs_cpu(y0, x, rows=2752):
    """Part of the cpu_baseline leg: the GPU's result for the first `rows` outputs of weight copy 0 against the
    CPU restatement on the same payload and activation (max |a - e| / max |e|)."""
    import oracle
    payload = synth.make_weight(synth.Q4_0, N_OUT, K_IN, seed=0, name="bench.w0")[:rows * (K_IN // 32) * 18]
    ref = oracle.matmul_ikj(x, oracle.transpose(oracle.dequant(synth.Q4_0, payload, rows, K_IN)))
    return float(np.abs(y0[:, :rows] - ref).max() / np.abs(ref).max())


def gemm_micro(torch, capi, local, stream, steps, warmup):
    """Prefill GEMM of configs[2]: M=512 bf16 tokens x K=4096 x N=14336 in Q4_K and Q6_K.
    Four weight copies per format are visited round-robin (4 x 33-48 MB > L2)."""
    m, k, n = 512, 4096, 14336
    out = {}
    x = torch.from_numpy(synth.make_activation(m, k, seed=0, name="bench.gemm.x")).cuda().to(torch.bfloat16)
    y = torch.empty((m, n), dtype=torch.float32, device="cuda")
    for fmt, name in ((synth.Q4_K, "q4_k"), (synth.Q6_K, "q6_k")):
        payload = synth.make_weight(fmt, n, k, seed=0, name="bench.gemm.w")
        ws = [capi.Weight.from_host(fmt, payload, n, k, device=local, stream=stream) for _ in range(4)]
        for i in range(max(3, warmup)):
            ws[i % 4].gemm_bf16(x.data_ptr(), y.data_ptr(), m, capi.OUT_F32, stream)
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for i in range(steps):
            ws[i % 4].gemm_bf16(x.data_ptr(), y.data_ptr(), m, capi.OUT_F32, stream)
        b.record()
        torch.cuda.synchronize()
        us = a.elapsed_time(b) * 1e3 / steps
        out[name] = {"us": us, "tflops": 2.0 * m * n * k / (us * 1e-6) / 1e12}
        for w in ws:
            w.destroy()
    capi.kernel_status(local)
    if not torch.isfinite(y).all():
        raise SystemExit("bench.py: GEMM produced non-finite output")
    return out


def batch_decode_bench(torch, dist, model, spec, prompt_len, batch, steps, warm, world, barrier):
    """configs[4]'s second form, "decode steps at batch 16": `batch` sequences with their own prompts, caches and
    positions decode greedily together; the linears see them as the rows of one skinny product.  Device time of
    `steps` steps after `warm` warm-up steps (CUDA events, max over ranks); tokens = steps x batch."""
    import zlib
    model.batch_create(batch, warm + steps)
    for b in range(batch):
        model.batch_prefill(b, synth.make_token_ids(prompt_len, spec.vocab, seed=100 + b, name="batch-prompt"))
    model.batch_decode_enqueue(warm)
    torch.cuda.synchronize()
    barrier()
    a, z = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record()
    model.batch_decode_enqueue(steps)
    z.record()
    barrier()
    t = torch.tensor([a.elapsed_time(z)], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms = float(t.cpu()[0])
    toks = model.batch_generated(warm, steps)
    if toks.min() < 0 or toks.max() >= spec.vocab:
        raise SystemExit("bench.py: batched decode produced an out-of-range token")
    return {"batch": batch, "steps": steps, "warmup": warm, "tok_s": steps * batch / (ms * 1e-3),
            "us_per_step": ms * 1e3 / steps, "us_per_block": ms * 1e3 / steps / spec.n_layers,
            "tokens_crc32": zlib.crc32(toks.tobytes()), "first_step_tokens": [int(t) for t in toks[0]],
            "distinct_tokens": int(len(np.unique(toks))),
            "sums": "NCCL all-reduce of [batch, d_model] rows" if world > 1 else "single GPU"}


def run_ours(args):
    import torch
    import torch.distributed as dist
    from litenn_b200 import capi
    from litenn_b200 import llama as ll

    rank, world, local = dist_env()
    if not torch.cuda.is_available():
        raise SystemExit("bench.py: no CUDA device; this path has no CPU fallback (use --impl reference)")
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    capi.load()
    side = torch.cuda.Stream()
    torch.cuda.set_stream(side)
    stream = side.cuda_stream

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    if args.device_only == "gemm":
        res = gemm_micro(torch, capi, local, stream, max(4, args.steps), args.warmup)
        if rank == 0:
            print(json.dumps({"device_only": "gemm", "workload": "prefill_gemm_m512_k4096_n14336", **res}))
        return 0
    gemv_steps = 50
    gv = None if args.device_only in ("decode", "decode70b") else gemv_micro(torch, capi, local, side, stream, gemv_steps, 3)
    if args.device_only == "gemv":
        if rank == 0:
            print(json.dumps({"device_only": "gemv", "us_per_gemv": gv["full_us"], "us_per_gemv_kernel": gv["kernel_us"],
                              "us_per_gemv_kernel_isolated": gv["isolated_us"]}))
        return 0
    gm = gemm_micro(torch, capi, local, stream, 20, 3) if rank == 0 else None

    # ---- the decoder -----------------------------------------------------------------
    K, W = args.steps, max(3, args.warmup)
    e2e_steps = min(K, 32)
    import dataclasses
    spec, prompt_len = ll.SPEC_7B, PROMPT_LEN
    if args.device_only == "decode70b":   # configs[4]: 70B shape, GQA, Q4_K / Q6_K, 1024-token prompt
        spec, prompt_len = ll.SPEC_70B, 1024
        if args.layers:
            spec = dataclasses.replace(spec, n_layers=args.layers)
    spec = dataclasses.replace(spec, max_seq=prompt_len + W + K + e2e_steps + 16, max_prefill=prompt_len)
    model = ll.LlamaModel(spec, device=local, tp_rank=rank, tp_size=world, stream=stream, share_layer_payloads=True)
    if world > 1:
        path = ll.find_nccl_library()
        box = [ll.nccl_unique_id(path) if rank == 0 else None]
        dist.broadcast_object_list(box, src=0)
        model.tp_init(path, box[0])
        records = [None] * world
        dist.all_gather_object(records, model.tp_export())
        model.tp_import(records)                  # decode sums the per-block partials over peer memory
    if args.device_only in ("decode", "decode70b") and args.batch > 1:
        res = batch_decode_bench(torch, dist, model, spec, prompt_len, args.batch, K, W, world, barrier)
        capi.kernel_status(local)
        if rank == 0:
            print(json.dumps({"device_only": args.device_only, "n_gpus": world, "layers": spec.n_layers,
                              "d_model": spec.d_model, "prompt": prompt_len, **res}))
        model.close()
        if world > 1:
            dist.destroy_process_group()
        return 0
    prompt = synth.make_token_ids(prompt_len, spec.vocab, seed=0, name="prompt")
    torch.cuda.synchronize()
    t_prefill = time.perf_counter()
    first = model.prefill(prompt)        # returns after the first token has come back to the host
    prefill_ms = (time.perf_counter() - t_prefill) * 1e3
    model.decode(W)                      # warm-up steps (the first one also builds the CUDA graph)
    barrier()
    sampler = ClockSampler(local)
    if rank == 0:
        sampler.start()
        time.sleep(0.2)
    start, stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    first_timed = 1 + W                  # generated so far: the prefill's token and W warm-up tokens
    start.record()
    model.decode_enqueue(K)
    stop.record()
    barrier()
    ms_total = start.elapsed_time(stop)
    timed_tokens = model.generated(first_timed, K)
    if args.device_only in ("decode", "decode70b"):  # the timed region alone (ncu launch lists, 70B runs)
        t = torch.tensor([ms_total], dtype=torch.float64, device="cuda")
        if world > 1:
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
        if rank == 0:
            sampler.stop()
            import zlib
            print(json.dumps({"device_only": args.device_only, "tok_s": K / (float(t.cpu()[0]) * 1e-3), "steps": K,
                              "warmup": W, "n_gpus": world, "layers": spec.n_layers, "d_model": spec.d_model,
                              "tokens_crc32": zlib.crc32(timed_tokens.tobytes())}))
        model.close()
        if world > 1:
            dist.destroy_process_group()
        return 0

    # ---- end to end: every token crosses the host ---------------------------------------
    tok = first
    for _ in range(2):
        tok = model.step_host(tok)
    barrier()
    e_start, e_stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e_start.record()
    for _ in range(e2e_steps):
        tok = model.step_host(tok)
    e_stop.record()
    barrier()
    e2e_ms = e_start.elapsed_time(e_stop)
    clocks = sampler.stop() if rank == 0 else None
    capi.kernel_status(local)
    # the same model at batch 16 (outside both timed regions above)
    b16 = batch_decode_bench(torch, dist, model, spec, prompt_len, 16, min(K, 32), 3, world, barrier)
    capi.kernel_status(local)
    if not (0 <= tok < spec.vocab) or timed_tokens.min() < 0 or timed_tokens.max() >= spec.vocab:
        raise SystemExit("bench.py: decoder produced an out-of-range token")

    times = torch.tensor([ms_total, e2e_ms], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(times, op=dist.ReduceOp.MAX)
    ms_total, e2e_ms = (float(v) for v in times.cpu())

    if rank == 0:
        import zlib
        peak, peak_kind = measured_peak()
        tensor_peak = measured_tensor_peak()
        value = K / (ms_total * 1e-3)
        kernel_us, full_us = gv["kernel_us"], gv["full_us"]
        achieved = ALGO_BYTES / (kernel_us * 1e-6) / 1e9
        # per block: qkv matvec, attention, attn_output matvec, gate|up matvec, down matvec; per token also:
        # embedding row, output matvec, arg-max, commit
        per_block = 5  # also with tensor parallelism: the two sums over the ranks happen inside the matvecs
        kernels_per_token = 1 + spec.n_layers * per_block + 3
        line = {
            "metric": "7B-shape Q4_0 batch-1 decode tok/s",
            "value": value,
            "unit": "tok/s",
            "n_gpus": world,
            "steps": K,
            "warmup": W,
            "ms_per_step": ms_total / K,
            "higher_is_better": True,
            "scaling": "strong",
            "vs_baseline": None,
            "dtype": "int8 tensor-core products, fp32 accumulate (decode); bf16 tcgen05 (prefill)",
            "data": "synthetic",
            "config": {"workload": "llama7b_q4_0_decode_b1", "layers": 32, "d_model": 4096, "heads": 32, "ffn": 11008,
                       "vocab": 32000, "prompt": PROMPT_LEN, "batch": 1, "kv_cache": "fp16",
                       "parallelism": f"tp{world}" if world > 1 else "single",
                       "launch": "one CUDA graph per token",
                       "kernels_per_block": per_block,
                       "us_per_block": ms_total / K * 1e3 / spec.n_layers,
                       "l2": "inputs larger than L2: 3.75 GB of weights are read per token",
                       "prefill_ms_first_call": prefill_ms,
                       "weight_bytes_per_token": DECODE_WEIGHT_BYTES,
                       "frac_of_weight_stream_bound": value / (peak * 1e9 / DECODE_WEIGHT_BYTES * world),
                       "bound_tok_s_at_peak": peak * 1e9 / DECODE_WEIGHT_BYTES * world,
                       # the K timed tokens: identical at every N when tensor parallelism is correct
                       "tokens_crc32": zlib.crc32(timed_tokens.tobytes()),
                       "first_tokens": [int(t) for t in timed_tokens[:8]]},
            "gemv": {"metric": "Q4_0 GEMV achieved HBM GB/s", "workload": "q4_0_gemv_4096x11008_b1",
                     "value": ALGO_BYTES / (full_us * 1e-6) / 1e9, "unit": "GB/s", "us_per_call": full_us,
                     "copies": COPIES, "algorithmic_bytes": ALGO_BYTES,
                     "note": "public call qmm_gemv_f32 (packs and multiplies in one launch), one CUDA graph of 12 calls"},
            "batch16": {"workload": "llama7b_q4_0_decode_b16", **b16},
            "gemm": {"workload": "prefill_gemm_m512_k4096_n14336", "q4_k_us": gm["q4_k"]["us"], "q6_k_us": gm["q6_k"]["us"],
                     "q4_k_tflops": gm["q4_k"]["tflops"], "q6_k_tflops": gm["q6_k"]["tflops"],
                     "peak_tflops": tensor_peak[0], "peak_source": f"of {tensor_peak[1]} (burst)",
                     "frac_of_burst": gm["q4_k"]["tflops"] / tensor_peak[0],
                     "q6_k_frac_of_burst": gm["q6_k"]["tflops"] / tensor_peak[0]},
            "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                         "frac": achieved / peak, "traffic": NCU_TRAFFIC_BYTES, "peak_source": f"of {peak_kind}",
                         "frac_of_nominal_8tbs": achieved / 8000.0,
                         "kernel": "gemv_kernel<Q4_0, batch 1> on W[11008,4096]", "us_per_launch": kernel_us,
                         "us_per_launch_isolated": gv["isolated_us"],
                         "frac_isolated": ALGO_BYTES / (gv["isolated_us"] * 1e-6) / 1e9 / peak if gv["isolated_us"] > 0 else None,
                         "how": "CUDA events around graph replays of 12 launches of this kernel alone (12 weight copies = "
                                "304 MB > 2 x L2), activations packed once; back to back the launches overlap through "
                                "programmatic dependent launch, 'isolated' puts a one-element fill kernel between them "
                                "and subtracts its separately measured time"},
            "e2e": {"value": e2e_steps / (e2e_ms * 1e-3), "unit": "tok/s", "h2d_bytes_per_step": 4,
                    "d2h_bytes_per_step": 12, "steps": e2e_steps,
                    "how": "qmm_llama_step_host per token: the input token is copied host to device (4 B), the step's "
                           "graph runs, its last kernel stores the new token and the two status words (12 B) into "
                           "mapped pinned host memory, the host waits for the stream and reads them"},
            "gpu_launches": kernels_per_token * (K + e2e_steps) * world,
            "clocks": clocks,
        }
        if world == 1:
            cpu = cpu_decode_baseline(1, steps=150, warmup=2)
            line["cpu_baseline"] = {k: cpu[k] for k in ("value", "unit", "cores", "kind", "sample")}
            line["gemv"]["max_rel_err_vs_cpu"] = gemv_error_vs_cpu(gv["y0"], gv["x"])
        print(json.dumps(line))
    model.close()
    if world > 1:
        dist.destroy_process_group()
    return 0


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=128)
    ap.add_argument("--warmup", type=int, default=8)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--device-only", choices=["gemv", "decode", "gemm", "decode70b"], default=None,
                    help="run one device-timed part alone (used for ncu captures): the Q4_0 GEMV, the decode\n"
                         "steps, or the prefill GEMM of configs[2]")
    ap.add_argument("--layers", type=int, default=0, help="with --device-only decode70b: blocks to build (default 80)")
    ap.add_argument("--batch", type=int, default=1,
                    help="with --device-only decode / decode70b: sequences decoded together (2..16)")
    args = ap.parse_args()
    # The JSON line must be the only thing on stdout: libraries that write to file descriptor 1 themselves
    # (NCCL prints its version there) are pointed at stderr while the run lasts.
    sys.stdout.flush()
    real_stdout = os.dup(1)
    os.dup2(2, 1)
    captured = io.StringIO()
    try:
        with contextlib.redirect_stdout(captured):
            rc = run_reference(args) if args.impl == "reference" else run_ours(args)
    finally:
        sys.stdout.flush()
        os.dup2(real_stdout, 1)
        os.close(real_stdout)
    sys.stdout.write(captured.getvalue())
    sys.stdout.flush()
    return rc


if __name__ == "__main__":
    sys.exit(main())
