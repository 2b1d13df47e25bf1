#!/usr/bin/env python3
"""bench.py — resident decode throughput of the B200-native engine (decoded tokens per second).

    python bench.py [--gpus N] [--steps K] [--warmup W] [--workload NAME] [--impl ours|reference]
    python -m torch.distributed.run --nnodes=1 --nproc-per-node N ... bench.py --gpus N ...

A "step" is one decoded token (batch 1) of the named Llama-3 shape with synthetic, seeded random GGUF blocks
generated on the GPU.  N > 1 runs the same model tensor-parallel over N ranks (strong scaling).
Prints ONE JSON line on rank 0: value = tok/s with the token already handed to the
device-side step state; e2e = tok/s through the C-ABI with HOST token ids in and HOST logits out every step.

--impl reference times the UNMODIFIED reference (its own CUDA kernels and Transformer::forward, compiled for
sm_100 into oracle/_ref by oracle/Makefile) on the same synthetic model on one GPU of this box.  The reference
has no CPU path, so its own implementation of this path IS a CUDA implementation; the CPU figure
reported next to it (cpu_baseline, kind "port") is the oracle's C restatement on the host cores.
"""
from __future__ import annotations

import argparse
import ctypes as C
import json
import os
import subprocess
import sys
import tempfile
import threading
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

WORKLOADS = {
    # name: (shape, mix, prompt_len, max_seq)          the 70B decode is the metric's own workload
    "llama3-70b-q4_k_m-decode": ("70b", "Q4_K_M", 16, 4096),
    "llama3-8b-q4_k_m-decode-ctx2048": ("8b", "Q4_K_M", 2047, 4096),
    "llama3-8b-q8_0-decode": ("8b", "Q8_0", 16, 4096),
    "llama3-70b-q6_k-decode": ("70b", "Q6_K", 16, 4096),
    "llama3-8b-q4_k_m-decode": ("8b", "Q4_K_M", 16, 4096),
    "tiny-q4_k_m-decode": ("tiny", "Q4_K_M", 8, 128),
    # the step is one whole 4096-token prompt (metric prefill_tok_s); see run_prefill
    "llama3-8b-f16-prefill-4096": ("8b", "F16", 4096, 4096),
    "tiny-f16-prefill-96": ("tiny", "F16", 96, 128),
    # quantised weights on the tensor-core prefill path (dequantised to an F16 hi/lo pair per matrix, two GEMMs each)
    "llama3-8b-q4_k_m-prefill-4096": ("8b", "Q4_K_M", 4096, 4096),
    "llama3-70b-q4_k_m-prefill-4096": ("70b", "Q4_K_M", 4096, 4096),
}
DTYPE_NOTE = "quantised codes x block-scaled 24-bit activations via integer matrix instructions (s32 exact) + f32 scales/accumulate; KV f16"


def shape_cfg(shape: str, max_seq: int):
    from dataclasses import replace
    from ntransformer_b200.model_spec import LLAMA3_8B, LLAMA3_70B, TINY
    return replace({"8b": LLAMA3_8B, "70b": LLAMA3_70B, "tiny": TINY}[shape], max_seq_len=max_seq)


def token_at(i: int, vocab: int) -> int:
    return (i * 7919 + 11) % min(vocab, 128000)


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled every 100 ms while the timed region runs."""
    Q = "clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown," \
        "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap"

    def __init__(self, index: int):
        self.index, self.proc, self.path = index, None, None

    def start(self):
        try:
            self.path = tempfile.NamedTemporaryFile(prefix="clk", suffix=".csv", delete=False).name
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits", "-lms", "100",
                                          "-i", str(self.index)], stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self) -> dict:
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.12)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, mx, pw, reasons = [], [], [], set()
        for line in open(self.path):
            p = [x.strip() for x in line.split(",")]
            if len(p) < 7:
                continue
            try:
                sm.append(float(p[0])); mx.append(float(p[1])); pw.append(float(p[2]))
            except ValueError:
                continue
            for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), p[3:7]):
                if v.lower().startswith("active"):
                    reasons.add(name)
        os.unlink(self.path)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["no samples"]}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": max(mx), "power_w_max": max(pw), "samples": len(sm),
                "reasons": sorted(reasons)}


def ncu_traffic(workload: str, world: int, name: str = "gemv_mma_gateup_ncu.json"):
    """dram__bytes_read.sum + dram__bytes_write.sum per launch of the dominant kernel, from the committed ncu
    capture of the same shape (profiles/<name>); None when no capture exists for this workload."""
    p = ROOT / "profiles" / name
    if world != 1 or not p.exists():
        return None
    try:
        d = json.load(open(p))
        return d["dram_bytes_per_launch"] if workload in d.get("workloads", []) else None
    except Exception:
        return None


def measured_peak_hbm():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return float(json.load(open(p))["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs, copy read+write)"
        except Exception:
            pass
    return 6650.0, "fallback (B200_PROFILING.md 6.65 TB/s)"


def measured_peak_tensor():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        try:
            return float(json.load(open(p))["bf16_tflops"]), "measured (MEASURED_PEAKS.json bf16_tflops, cuBLAS 8192^3 burst)"
        except Exception:
            pass
    return 1750.0, "fallback (B200_PROFILING.md dense bf16)"


# ------------------------------------------------------------------------------------------------
def run_prefill(args, rank, world):
    """F16 prefill of a whole prompt through the batched tcgen05 path.  One step = one prompt;
    value = prompt tokens / s with the prompt ids already on the host side of the C-ABI call but no logits read-back,
    e2e = the same through nt_model_forward (token ids H2D + logits D2H inside the timed region)."""
    import torch
    from ntransformer_b200 import kernels as K
    from ntransformer_b200.engine import Model

    if world > 1:
        if rank == 0:
            print(json.dumps({"metric": "prefill_tok_s", "unavailable": "the batched prefill path is single-GPU in this round"}))
        return
    shape, mix, prompt_len, max_seq = WORKLOADS[args.workload]
    if args.prompt_tokens is not None:
        prompt_len = args.prompt_tokens
    cfg = shape_cfg(shape, max_seq)
    torch.cuda.set_device(0)
    model = Model.synthetic(cfg, mix, seed=1234)
    stream = torch.cuda.ExternalStream(model.stream)
    vocab = cfg.vocab_size
    steps = min(args.steps, 16)                                  # a step is a whole prompt
    prompts = [[token_at(i + 97 * j, vocab) for i in range(prompt_len)] for j in range(4)]
    for i in range(args.warmup):
        model.forward_async(prompts[i % 4], 0)
    model.sync()
    sampler = ClockSampler(0)
    launches0 = K.launch_count()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    sampler.start()
    ev0.record(stream)
    for i in range(steps):
        model.forward_async(prompts[i % 4], 0)
    ev1.record(stream)
    model.sync()
    ms = ev0.elapsed_time(ev1)
    launches = K.launch_count() - launches0
    clocks = sampler.stop()
    tok_s = steps * prompt_len / (ms / 1e3)
    # end to end
    t0 = time.perf_counter()
    for i in range(steps):
        logits = model.forward(prompts[i % 4], 0)
    e2e_ms = (time.perf_counter() - t0) * 1e3
    assert np.isfinite(logits).all(), "non-finite logits"
    # per-token replay of the decode step (what the reference's forward loop does, on our kernels) for comparison
    model.set_prefill_min_tokens(0)
    n_cmp = min(prompt_len, 64)
    model.forward_async(prompts[0][:n_cmp], 0)
    model.sync()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    a.record(stream)
    model.forward_async(prompts[1][:n_cmp], 0)
    b.record(stream)
    model.sync()
    per_token_tok_s = n_cmp / (a.elapsed_time(b) / 1e3)
    model.set_prefill_min_tokens(16)

    # ---- roofline of the dominant kernel (tcgen05 GEMM, ffn gate+up shape), measured live (F16 weights) ----
    peak, peak_src = measured_peak_tensor()
    ach = flops = dur_ms = None
    evs = []
    if mix == "F16":
        T, N, Kd = prompt_len, cfg.intermediate_size, cfg.hidden_size
        A = torch.randn(T, Kd, device="cuda")
        Wg, Wu = model._keep["blk.0.ffn_gate.weight"][0], model._keep["blk.0.ffn_up.weight"][0]
        ws = torch.empty(K.gemm_f16_tc_workspace_bytes(T, Kd), dtype=torch.uint8, device="cuda")
        ws2 = torch.empty(K.gemm_f16_tc_workspace_bytes(T, N), dtype=torch.uint8, device="cuda")
        K.split_activations(ws, A, T, Kd)
        evs = []
        for r in range(6):
            x, y = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            x.record()
            K.gemm_f16_tc_swiglu_ws(ws2, ws, Wg, Wu, T, N, Kd)
            y.record()
            if r > 0:
                evs.append((x, y))
        torch.cuda.synchronize()
        dur_ms = float(np.mean([x.elapsed_time(y) for x, y in evs]))
        flops = 2.0 * T * (2 * N) * Kd
        ach = flops / (dur_ms / 1e3) / 1e12
    n_mat = (cfg.n_heads * cfg.head_dim * cfg.hidden_size * 2 + cfg.n_kv_heads * cfg.head_dim * cfg.hidden_size * 2 +
             3 * cfg.intermediate_size * cfg.hidden_size) * cfg.n_layers                   # projection weights (elements)
    step_flops = 2.0 * prompt_len * n_mat + 4.0 * cfg.n_layers * cfg.n_heads * cfg.head_dim * prompt_len * (prompt_len + 1) / 2
    step_tf = step_flops / (ms / steps / 1e3) / 1e12
    if mix == "F16":
        roof = {"bound": "tensor", "kernel": "gemm_f16_tc_kernel<256, SWIGLU> (ffn gate+up, M=%d N=2x%d K=%d)" % (T, N, Kd),
                "achieved": round(ach, 1), "peak": peak, "unit": "TFLOP/s", "frac": round(ach / peak, 4),
                "traffic": ncu_traffic(args.workload, 1, "r01_gemm_tc_ncu.json"),
                "flops_per_launch": flops, "avg_launch_us": round(dur_ms * 1e3, 1), "launches_timed": len(evs), "peak_source": peak_src,
                "note": "algorithmic flops 2MNK; the kernel issues 2x that (F32 activations split into F16 hi+lo to keep parity <= 1e-3)",
                "step_achieved": round(step_tf, 1), "step_frac": round(step_tf / peak, 4)}
    else:
        roof = {"bound": "tensor", "kernel": "whole prefill step (gemm_blocks_kernel: blocks expanded on the way into tensor memory)",
                "achieved": round(step_tf, 1), "peak": peak, "unit": "TFLOP/s", "frac": round(step_tf / peak, 4), "traffic": None,
                "peak_source": peak_src,
                "note": "algorithmic flops; the path issues 2x that for Q4_K and Q5_K (activations as F16 hi+lo, weights as integers) and 3x for the other formats (weights as F16 hi+lo too, lo.lo left out)",
                "step_achieved": round(step_tf, 1), "step_frac": round(step_tf / peak, 4)}
    line = {
        "metric": "prefill_tok_s", "value": round(tok_s, 1), "unit": "tok/s", "n_gpus": 1, "steps": steps, "warmup": args.warmup,
        "ms_per_step": round(ms / steps, 3), "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
        "dtype": ("f16 weights" if mix == "F16" else mix + " weights dequantised to f16 hi+lo") +
                 " x f32 activations as f16 hi+lo on tcgen05 (f32 accumulate in TMEM); KV f16; attention f32",
        "data": "synthetic (seeded random weights generated on the GPU)",
        "config": {"workload": args.workload, "quant_mix": mix, "batch": 1, "prompt_tokens": prompt_len, "max_seq": max_seq,
                   "parallelism": "single", "l2_policy": "the weights read per prompt (GBs) exceed the 126 MB L2; no flush needed"},
        "clocks": clocks,
        "e2e": {"value": round(steps * prompt_len / (e2e_ms / 1e3), 1), "unit": "tok/s", "h2d_bytes_per_step": 4 * prompt_len,
                "d2h_bytes_per_step": vocab * 4, "ms_per_step": round(e2e_ms / steps, 3)},
        "gpu_launches": int(launches),
        "roofline": roof,
        "per_token_replay_tok_s": round(per_token_tok_s, 1),
    }
    print(json.dumps(line), flush=True)
    model.close()


# ------------------------------------------------------------------------------------------------
def workload_config(workload, prompt_len, ctx_first, steps, world):
    """The workload's description: the same keys and values for both arms (ours / --impl reference) of one run."""
    shape, mix, _, max_seq = WORKLOADS[workload]
    return {"workload": workload, "quant_mix": mix, "batch": 1, "prompt_tokens": prompt_len,
            "ctx_during_timing": [ctx_first, ctx_first + steps], "max_seq": max_seq,
            "l2_policy": "weights read per step exceed the 126 MB L2 on every GPU; no flush needed"}


def run_ours(args, rank, world):
    import torch
    import torch.distributed as dist

    local = int(os.environ.get("LOCAL_RANK", 0))
    torch.cuda.set_device(local)
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))
    line = measure_decode(args, rank, world, args.workload, with_cpu=not args.no_cpu_baseline)
    # 70B Q6_K, 8-way tensor parallel, rides along with the 8-GPU run of the metric's own config
    # (Q4_K_M at every N, so that the 1/2/4/8 series stays one workload): reported under "configs3".
    if world == 8 and args.workload == "llama3-70b-q4_k_m-decode" and not args.no_configs3:
        extra = measure_decode(args, rank, world, "llama3-70b-q6_k-decode", with_cpu=False)
        if rank == 0:
            line["configs3"] = {k: extra[k] for k in ("metric", "value", "unit", "ms_per_step", "config", "e2e", "gpu_launches", "roofline", "tp")}
    if rank == 0:
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()


def measure_decode(args, rank, world, workload, with_cpu):
    import torch
    import torch.distributed as dist
    from ntransformer_b200 import kernels as K
    from ntransformer_b200.dtypes import DType
    from ntransformer_b200.engine import Model

    shape, mix, prompt_len, max_seq = WORKLOADS[workload]
    if args.prompt_tokens is not None:
        prompt_len = args.prompt_tokens
    cfg = shape_cfg(shape, max_seq)
    local = int(os.environ.get("LOCAL_RANK", 0))
    model = Model.synthetic(cfg, mix, seed=1234, tp_rank=rank, tp_size=world)
    if world > 1:
        model.init_tp()
    stream = torch.cuda.ExternalStream(model.stream)
    vocab = cfg.vocab_size

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    # ---- prefill (untimed) then warm-up ----
    prompt = [token_at(i, vocab) for i in range(prompt_len)]
    model.forward(prompt, 0, want_logits=False)
    pos = prompt_len
    for i in range(args.warmup):
        model.forward_async([token_at(pos, vocab)], pos)
        pos += 1
    model.sync()

    # ---- timed: device-resident decode (value) ----
    sampler = ClockSampler(local)
    launches0 = K.launch_count()
    ev0, ev1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    if rank == 0:
        sampler.start()
    ctx_first = pos
    ev0.record(stream)
    for i in range(args.steps):
        model.forward_async([token_at(pos, vocab)], pos)
        pos += 1
    ev1.record(stream)
    model.sync()
    barrier()
    ms = ev0.elapsed_time(ev1)
    launches = K.launch_count() - launches0
    clocks = sampler.stop() if rank == 0 else None
    if world > 1:
        t = torch.tensor([ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms = float(t.item())
    tok_s = args.steps / (ms / 1e3)

    # ---- timed: end to end through the C-ABI, host token in / host logits out each step ----
    for i in range(min(3, args.warmup)):
        model.forward([token_at(pos, vocab)], pos)
        pos += 1
    barrier()
    t0 = time.perf_counter()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for i in range(args.steps):
        logits = model.forward([token_at(pos, vocab)], pos)     # sync + 513 KB D2H inside
        pos += 1
    e1.record(stream)
    model.sync()
    barrier()
    e2e_ms = e0.elapsed_time(e1)
    wall_ms = (time.perf_counter() - t0) * 1e3
    e2e_ms = max(e2e_ms, wall_ms)                                # host-visible time is what a caller sees
    if world > 1:
        t = torch.tensor([e2e_ms], device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_ms = float(t.item())
    e2e_tok_s = args.steps / (e2e_ms / 1e3)
    assert np.isfinite(logits).all(), "non-finite logits"
    tp_info = None
    if world > 1:
        # tensor-parallel lock-step: every rank must hold bit-identical logits (the replicas sample the same token)
        mine = torch.from_numpy(np.ascontiguousarray(logits)).cuda()
        ref = mine.clone()
        dist.broadcast(ref, src=0)
        same = torch.tensor([1.0 if torch.equal(mine, ref) else 0.0], device="cuda")
        dist.all_reduce(same, op=dist.ReduceOp.MIN)
        assert float(same.item()) == 1.0, "tensor-parallel ranks diverged (logits differ between ranks)"
        tp_info = {"ranks_bit_identical": True, "exchange": model.tp_exchange}

    # ---- roofline of the dominant kernel (fused gate+up K-quant GEMV), measured live ----
    peak, peak_src = measured_peak_hbm()
    ctx_mid = ctx_first + args.steps // 2
    b_tok = model.bytes_per_token(ctx_mid)                       # this rank's algorithmic bytes per token
    roof = None
    if rank == 0:
        names = [(f"blk.{i}.ffn_gate.weight", f"blk.{i}.ffn_up.weight") for i in range(cfg.n_layers)]
        g0, dt0 = model._keep[names[0][0]][:2]
        if dt0 in (DType.Q4_K_M, DType.Q5_K, DType.Q6_K):
            inter_l = cfg.intermediate_size // world
            x = torch.randn(cfg.hidden_size, device="cuda")
            xq = torch.zeros(K.xq_bytes(cfg.hidden_size), device="cuda", dtype=torch.uint8)
            act, up = torch.zeros(inter_l, device="cuda"), torch.zeros(inter_l, device="cuda")
            K.quantize_x(x, xq, cfg.hidden_size)
            reps = 3 if cfg.n_layers >= 16 else 50
            evs = []
            for r in range(reps + 1):
                for gn, un in names:
                    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                    a.record()
                    K.gemv_fused([act, up], [model._keep[gn][0], model._keep[un][0]], [inter_l, inter_l], [dt0, dt0],
                                 cfg.hidden_size, xq, epilogue=2)
                    b.record()
                    if r > 0:
                        evs.append((a, b))
            torch.cuda.synchronize()
            dur_ms = float(np.mean([a.elapsed_time(b) for a, b in evs]))
            kbytes = 2 * model._keep[names[0][0]][0].numel()
            ach = kbytes / (dur_ms / 1e3) / 1e9
            roof = {"bound": "hbm", "kernel": "gemv_mma_kernel (ffn gate+up fused, SwiGLU epilogue)", "achieved": round(ach, 1),
                    "peak": peak, "unit": "GB/s", "frac": round(ach / peak, 4), "traffic": ncu_traffic(workload, world),
                    "bytes_per_launch": kbytes, "avg_launch_us": round(dur_ms * 1e3, 2), "launches_timed": len(evs),
                    "peak_source": peak_src}
        step_ach = b_tok * tok_s / 1e9
        if model.megakernel_active:
            # one launch per token IS the step: the dominant kernel is decode_step_kernel, timed live by the step loop above
            roof = {"bound": "hbm", "kernel": "decode_step_kernel (persistent: all layers + LM head of one token)",
                    "achieved": round(step_ach, 1), "peak": peak, "unit": "GB/s", "frac": round(step_ach / peak, 4), "traffic": None,
                    "bytes_per_launch": b_tok, "avg_launch_us": round(ms / args.steps * 1e3, 2), "launches_timed": args.steps,
                    "peak_source": peak_src, "component_gate_up_gemv": roof}
        if roof is None:
            roof = {"bound": "hbm", "kernel": "whole decode step", "achieved": round(step_ach, 1), "peak": peak, "unit": "GB/s",
                    "frac": round(step_ach / peak, 4), "traffic": None, "peak_source": peak_src}
        roof["step_achieved"] = round(step_ach, 1)
        roof["step_frac"] = round(step_ach / peak, 4)
        roof["step_bytes_per_gpu"] = b_tok

    cpu = cpu_baseline(model, cfg, mix, world) if (rank == 0 and world == 1 and with_cpu) else None

    line = None
    if rank == 0:
        line = {
            "metric": "decode_tok_s", "value": round(tok_s, 2), "unit": "tok/s", "n_gpus": world, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 4), "higher_is_better": True, "scaling": "strong",
            "vs_baseline": None, "dtype": DTYPE_NOTE, "data": "synthetic (seeded random valid GGUF blocks generated on the GPU)",
            "config": workload_config(workload, prompt_len, ctx_first, args.steps, world),
            "path": {"parallelism": f"tp{world}" if world > 1 else "single", "cuda_graph": not model.megakernel_active,
                     "decode_path": "persistent kernel (NT_B200_MEGAKERNEL)" if model.megakernel_active else "cuda graph of fused launches",
                     "launches_per_step": round(launches / max(1, args.steps), 1), "weights_gb_per_gpu": round(b_tok / 1e9, 2)},
            "clocks": clocks,
            "e2e": {"value": round(e2e_tok_s, 2), "unit": "tok/s", "h2d_bytes_per_step": 8, "d2h_bytes_per_step": vocab * 4,
                    "ms_per_step": round(e2e_ms / args.steps, 4)},
            "gpu_launches": int(launches),
            "roofline": roof,
        }
        if cpu:
            line["cpu_baseline"] = cpu
        if tp_info:
            line["tp"] = tp_info
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    model.close()
    del model
    torch.cuda.empty_cache()
    return line


def cpu_baseline(model, cfg, mix, world):
    """Times the oracle's C restatement of one decoded token on a bounded sample (2 layers + LM head), host cores."""
    from oracle import oracle as O
    from ntransformer_b200.model_spec import use_more_bits

    n = cfg.n_layers
    hi = 0
    lo = next((i for i in range(n) if not use_more_bits(i, n)), 0)
    picks = [hi, lo] if n > 1 else [0]
    host = {}
    for name in ("token_embd.weight", "output.weight", "output_norm.weight"):
        t, dt = model._keep[name][:2]
        host[name] = (t.cpu().numpy(), int(dt))
    for j, li in enumerate(picks):
        for suffix in ("attn_norm", "attn_q", "attn_k", "attn_v", "attn_output", "ffn_norm", "ffn_gate", "ffn_up", "ffn_down"):
            t, dt = model._keep[f"blk.{li}.{suffix}.weight"][:2]
            host[f"blk.{j}.{suffix}.weight"] = (t.cpu().numpy(), int(dt))
    for j in range(len(picks), n):          # unused layer slots alias the first sample (never run)
        for suffix in ("attn_norm", "attn_q", "attn_k", "attn_v", "attn_output", "ffn_norm", "ffn_gate", "ffn_up", "ffn_down"):
            host[f"blk.{j}.{suffix}.weight"] = host[f"blk.0.{suffix}.weight"]
    c = cfg.dict()
    c["max_seq_len"] = 64
    om = O.Model(c, host)

    def timed(k, min_s):
        """fastest of >= 3 calls (a fixed amount of work per call): host-core contention from other tenants only ever adds time,
        so the minimum is the stable figure (the mean swung 5x between runs)"""
        om.forward([5], 0, n_layers_run=k)                       # warm page cache / thread pool
        t_all, best, reps = time.perf_counter(), float("inf"), 0
        while reps < 3 or time.perf_counter() - t_all < min_s:
            t0 = time.perf_counter()
            om.forward([6 + reps], 1 + reps, n_layers_run=k)
            best = min(best, time.perf_counter() - t0)
            reps += 1
            if reps >= 30:
                break
        return best, reps

    t_head, r0 = timed(0, 2.0)                                  # final norm + LM head only
    t_1, r1 = timed(1, 3.0)                                     # + layer picks[0]
    t_2, r2 = timed(len(picks), 4.0) if len(picks) == 2 else (t_1, r1)
    n_hi = sum(1 for i in range(n) if use_more_bits(i, n)) if len(picks) == 2 else n
    l_hi, l_lo = max(t_1 - t_head, 1e-9), max(t_2 - t_1, 1e-9)
    token_s = n_hi * l_hi + (n - n_hi) * l_lo + t_head
    om.close()
    return {"value": round(1.0 / token_s, 4), "unit": "tok/s", "cores": O.num_threads(), "kind": "port",
            "sample": f"oracle/nt_oracle.c (C + OpenMP) forward of 1 token, fastest of >= 3 calls each: LM head {t_head * 1e3:.0f} ms, layer "
                      f"{picks[0]} {l_hi * 1e3:.0f} ms, layer {picks[-1]} {l_lo * 1e3:.0f} ms ({r0 + r1 + r2} timed calls), extrapolated to "
                      f"{n} layers ({n_hi} of the first kind)"}


# ------------------------------------------------------------------------------------------------
def run_reference(args, rank, world):
    """The reference's own CUDA path (oracle/_ref, built from /root/reference for sm_100) on the same synthetic model."""
    if rank != 0:
        return
    so = ROOT / "oracle" / "_ref" / "libnt_ref.so"
    shape, mix, prompt_len, max_seq = WORKLOADS[args.workload]
    if not so.exists():
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libnt_ref.so was not built (no /root/reference at build time)"}))
        return
    import torch
    from ntransformer_b200.gguf_write import write_gguf_streaming
    from ntransformer_b200.synth import random_blocks_cuda
    from ntransformer_b200.model_spec import tensor_table

    cfg = shape_cfg(shape, max_seq)
    torch.cuda.set_device(0)
    tmpdir = "/dev/shm" if os.path.isdir("/dev/shm") else tempfile.gettempdir()
    path = os.path.join(tmpdir, f"nt_ref_{args.workload}_{os.getpid()}.gguf")
    t_gen = time.perf_counter()

    def gen():
        for idx, (name, dt, rows, cols) in enumerate(tensor_table(cfg, mix)):
            s = 1234 + idx * 16
            if name.endswith("norm.weight"):
                g = torch.Generator(device="cuda")
                g.manual_seed(s)
                t = 1.0 + 0.1 * torch.randn(cols, generator=g, device="cuda", dtype=torch.float32)
            else:
                t = random_blocks_cuda(dt, rows, cols, s)
            yield name, t.cpu().numpy(), dt, rows, cols
    write_gguf_streaming(path, cfg, gen(), tensor_table(cfg, mix))
    t_gen = time.perf_counter() - t_gen
    try:
        ref = C.CDLL(str(so))
        ref.ref_model_load.restype = C.c_void_p
        ref.ref_model_load.argtypes = [C.c_char_p, C.c_int]
        ref.ref_model_forward.restype = C.c_float
        ref.ref_model_forward.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p]
        ref.ref_model_free.argtypes = [C.c_void_p]
        devnull = os.open(os.devnull, os.O_WRONLY)
        saved = os.dup(2)
        os.dup2(devnull, 2)                                       # the reference logs every layer to stderr
        try:
            h = ref.ref_model_load(path.encode(), max_seq)
        finally:
            os.dup2(saved, 2)
            os.close(devnull)
        if not h:
            print(json.dumps({"impl": "reference", "unavailable": "reference failed to load the synthetic GGUF"}))
            return
        vocab = cfg.vocab_size
        if "prefill" in args.workload:
            # The reference prefills with one GEMV pass over every weight matrix per prompt token (transformer.cpp:604-669),
            # so its prompt rate does not depend on the prompt length apart from the attention term: a 128-token prompt per
            # step is the bounded sample of the 4096-token workload.
            n_ref = min(prompt_len, 128)
            steps = min(args.steps, 4)
            logits = np.empty(vocab, np.float32)
            toks = np.array([token_at(i, vocab) for i in range(n_ref)], np.int32)
            ref.ref_model_forward(h, toks.ctypes.data_as(C.c_void_p), min(n_ref, 8), 0, None)          # warm-up
            sampler = ClockSampler(0)
            sampler.start()
            torch.cuda.synchronize()
            t0 = time.perf_counter()
            for i in range(steps):
                ref.ref_model_forward(h, toks.ctypes.data_as(C.c_void_p), n_ref, 0, logits.ctypes.data_as(C.c_void_p))
            torch.cuda.synchronize()
            ms = (time.perf_counter() - t0) * 1e3
            clocks = sampler.stop()
            ref.ref_model_free(h)
            tok_s = steps * n_ref / (ms / 1e3)
            print(json.dumps({
                "impl": "reference", "metric": "prefill_tok_s", "value": round(tok_s, 2), "unit": "tok/s", "n_gpus": 1, "steps": steps,
                "warmup": 1, "ms_per_step": round(ms / steps, 3), "higher_is_better": True, "scaling": "strong", "vs_baseline": None,
                "dtype": "f32 activations x f16 weights (reference CUDA-core GEMV per token, sm_100 build)",
                "data": "synthetic (same seeded weights as the B200 arm, written to a GGUF in /dev/shm)",
                "config": {"workload": args.workload, "quant_mix": mix, "batch": 1, "prompt_tokens": n_ref, "max_seq": max_seq,
                           "parallelism": "single (the reference is single-GPU)",
                           "note": "bounded sample: %d-token prompts; the reference's prefill is a per-token loop" % n_ref},
                "clocks": clocks,
                "cpu_baseline": {"value": round(tok_s, 2), "unit": "tok/s", "cores": 1, "kind": "reference",
                                 "sample": f"{steps} prompts of {n_ref} tokens through nt::Transformer::forward"},
                "e2e": {"value": round(tok_s, 2), "unit": "tok/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
                "setup_s": round(t_gen, 1)}), flush=True)
            return
        # bounded prefill: the reference prefills with per-token GEMVs, so keep the prompt short
        p_len = min(prompt_len, 16)
        toks = np.array([token_at(i, vocab) for i in range(p_len)], np.int32)
        logits = np.empty(vocab, np.float32)
        ref.ref_model_forward(h, toks.ctypes.data_as(C.c_void_p), p_len, 0, None)
        pos = p_len
        for i in range(args.warmup):
            t = np.array([token_at(pos, vocab)], np.int32)
            ref.ref_model_forward(h, t.ctypes.data_as(C.c_void_p), 1, pos, None)
            pos += 1
        sampler = ClockSampler(0)
        sampler.start()
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for i in range(args.steps):
            t = np.array([token_at(pos, vocab)], np.int32)
            ref.ref_model_forward(h, t.ctypes.data_as(C.c_void_p), 1, pos, logits.ctypes.data_as(C.c_void_p))
            pos += 1
        torch.cuda.synchronize()
        ms = (time.perf_counter() - t0) * 1e3
        clocks = sampler.stop()
        ref.ref_model_free(h)
    finally:
        if os.path.exists(path):
            os.unlink(path)
    tok_s = args.steps / (ms / 1e3)
    print(json.dumps({
        "impl": "reference", "metric": "decode_tok_s", "value": round(tok_s, 2), "unit": "tok/s", "n_gpus": 1, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": round(ms / args.steps, 4), "higher_is_better": True, "scaling": "strong",
        "vs_baseline": None, "dtype": "f32 activations x dequantised codes (reference CUDA-core kernels, sm_100 build)",
        "data": "synthetic (same seeded blocks as the B200 arm, written to a GGUF in /dev/shm)",
        "config": workload_config(args.workload, p_len, p_len + args.warmup, args.steps, 1),
        "path": {"parallelism": "single (the reference is single-GPU)", "cuda_graph": False, "device": "cuda:0",
                 "decode_path": "the reference's own CUDA path rebuilt for sm_100 (oracle/Makefile ref); it has no CPU path"},
        "clocks": clocks,
        "cpu_baseline": {"value": round(tok_s, 2), "unit": "tok/s", "cores": 1, "kind": "reference",
                         "sample": f"{args.steps} decode steps through nt::Transformer::forward (1 host thread drives the GPU)"},
        "e2e": {"value": round(tok_s, 2), "unit": "tok/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "setup_s": round(t_gen, 1),
    }), flush=True)


def run_check(args, rank, world):
    """Parity at the benchmarked configuration (not a timing): the workload's seeded model is written to a GGUF once, loaded by
    the reference (oracle/_ref: its own loader + CUDA kernels, sm_100 build) and by our engine, and both decode greedily from the
    same prompt.  Asserts logits <= 1e-3 relative (max |a - b| / max |b|) at every step where the histories agree and identical
    greedy ids for --steps tokens.  One GPU (the reference is single-GPU); prints one JSON line."""
    if rank != 0:
        return
    so = ROOT / "oracle" / "_ref" / "libnt_ref.so"
    if not so.exists():
        print(json.dumps({"check": args.workload, "unavailable": "oracle/_ref/libnt_ref.so was not built"}))
        return
    import torch
    from ntransformer_b200.engine import Model
    from ntransformer_b200.gguf_write import write_gguf_streaming
    from ntransformer_b200.synth import random_blocks_cuda
    from ntransformer_b200.model_spec import tensor_table

    shape, mix, prompt_len, max_seq = WORKLOADS[args.workload]
    cfg = shape_cfg(shape, max_seq)
    if args.layers:                                   # a slice of the stack with full-width tensors (70B shapes in seconds)
        from dataclasses import replace
        cfg = replace(cfg, n_layers=args.layers)
    torch.cuda.set_device(0)
    tmpdir = "/dev/shm" if os.path.isdir("/dev/shm") else tempfile.gettempdir()
    path = os.path.join(tmpdir, f"nt_check_{args.workload}_{os.getpid()}.gguf")

    def gen():
        for idx, (name, dt, rows, cols) in enumerate(tensor_table(cfg, mix)):
            s = 1234 + idx * 16
            if name.endswith("norm.weight"):
                g = torch.Generator(device="cuda")
                g.manual_seed(s)
                t = 1.0 + 0.1 * torch.randn(cols, generator=g, device="cuda", dtype=torch.float32)
            else:
                t = random_blocks_cuda(dt, rows, cols, s)
            yield name, t.cpu().numpy(), dt, rows, cols
    write_gguf_streaming(path, cfg, gen(), tensor_table(cfg, mix))
    try:
        ref = C.CDLL(str(so))
        ref.ref_model_load.restype = C.c_void_p
        ref.ref_model_load.argtypes = [C.c_char_p, C.c_int]
        ref.ref_model_forward.restype = C.c_float
        ref.ref_model_forward.argtypes = [C.c_void_p, C.c_void_p, C.c_int, C.c_int, C.c_void_p]
        ref.ref_model_free.argtypes = [C.c_void_p]
        devnull, saved = os.open(os.devnull, os.O_WRONLY), os.dup(2)
        os.dup2(devnull, 2)
        try:
            h = ref.ref_model_load(path.encode(), max_seq)
            ours = Model.load(path, max_seq)
        finally:
            os.dup2(saved, 2)
            os.close(devnull)
        assert h, "reference failed to load the GGUF"
        vocab = cfg.vocab_size
        p_len = min(prompt_len, 16)                    # the reference prefills token by token
        toks = np.array([token_at(i, vocab) for i in range(p_len)], np.int32)
        lr = np.empty(vocab, np.float32)
        ref.ref_model_forward(h, toks.ctypes.data_as(C.c_void_p), p_len, 0, lr.ctypes.data_as(C.c_void_p))
        if args.per_token_prompt:
            ours.set_prefill_min_tokens(0)
        lo = ours.forward([int(t) for t in toks], 0).copy()          # 16 tokens: the batched tensor-core prefill, as a user gets it
        rel = lambda a, b: float(np.abs(a - b).max() / np.abs(b).max())
        errs = [rel(lo, lr)]
        # conditioning of the synthetic model: the F64-accumulating CPU oracle on the same weights tells how far two correct F32
        # implementations may drift apart (random weights make a deep stack chaotic; a trained checkpoint is far better behaved)
        cond = None
        if args.oracle_steps > 0:
            from oracle import oracle as O
            host = {name: (arr, int(dt)) for name, arr, dt, rows, cols in gen()}
            c = cfg.dict()
            c["max_seq_len"] = p_len + args.oracle_steps + 4
            om = O.Model(c, host)
            lq = om.forward([int(t) for t in toks], 0)
            cond = {"ref_vs_f64": [rel(lr, lq)], "ours_vs_f64": [rel(lo, lq)]}
        ids_o, ids_r, to, tr, pos, agree, first_bad = [], [], int(np.argmax(lo)), int(np.argmax(lr)), p_len, True, None
        for step in range(args.steps):
            ids_o.append(to)
            ids_r.append(tr)
            t = np.array([tr], np.int32)
            ref.ref_model_forward(h, t.ctypes.data_as(C.c_void_p), 1, pos, lr.ctypes.data_as(C.c_void_p))
            lo = ours.forward([to], pos).copy()
            if agree and to != tr:
                agree, first_bad = False, step
            if agree:
                errs.append(rel(lo, lr))
                if cond is not None and step < args.oracle_steps:
                    lq = om.forward([tr], pos)
                    cond["ref_vs_f64"].append(rel(lr, lq))
                    cond["ours_vs_f64"].append(rel(lo, lq))
            to, tr, pos = int(np.argmax(lo)), int(np.argmax(lr)), pos + 1
        worst = max(errs)
        ref.ref_model_free(h)
        ours.close()
    finally:
        if os.path.exists(path):
            os.unlink(path)
    # Pass: greedy ids identical and logits within 1e-3 of the reference — or, with the F64 oracle beside them (--oracle-steps), our
    # distance from the F64 result within twice the reference's own (+1e-4): deep stacks of random blocks are ill-conditioned, the
    # reference's F32 path itself drifts up to 2.9e-3 from exact arithmetic on an 8-layer 8B slice over 128 steps (profiles/r02_parity_8b.txt).
    ok = ids_o == ids_r and worst <= 1e-3
    if not ok and ids_o == ids_r and cond is not None:
        r_err, o_err = max(cond["ref_vs_f64"]), max(cond["ours_vs_f64"])
        ok = o_err <= 2.0 * r_err + 1e-4 and worst <= 2.0 * r_err + 1e-3
    if cond is not None:
        cond = {k: [float("%.3g" % v) for v in vs] for k, vs in cond.items()}
    print(json.dumps({"check": args.workload, "layers": cfg.n_layers, "steps": args.steps, "prompt_tokens": p_len,
                      "max_rel_logit_err": worst, "err_after_prompt": errs[0], "err_first_steps": [float("%.3g" % e) for e in (errs[1:] if args.all_errs else errs[1:9])],
                      "first_id_mismatch_step": first_bad, "conditioning": cond,
                      "tolerance": 1e-3, "greedy_ids_identical": ids_o == ids_r, "ok": ok,
                      "against": "oracle/_ref (the reference's loader + CUDA kernels + Transformer::forward, sm_100 build), same GGUF"}),
          flush=True)
    if not ok:
        sys.exit(1)


FAMILY_SIZES = {
    # name: (width, heads, kv_heads, head dim, ff); 4 layers of each, vocabulary 32000, random weights
    "2048x8192": (2048, 16, 4, 128, 8192),
    "4096x14336": (4096, 32, 8, 128, 14336),
}


VEBOTAR_SIZES = {
    # name: (width, heads, kv_heads, map dim, value dim, experts, top, expert ff, shared ff); the Zelunex model beside it has the same width and
    # head counts, head dim = value dim, and a gated ff with as many weights as one token's experts use: (top * ff + shared) * 2 / 3
    "2048_e8x2048": (2048, 16, 4, 64, 128, 8, 2, 2048, 2048),
    "4096_e16x2048": (4096, 32, 8, 64, 128, 16, 4, 2048, 4096),
}


def run_family_compare_vebotar(args):
    """--family-compare --family vebotar: prompt-pass and decode throughput of the Vebotar family (BF16 weights; differential attention
    inside blocks of 1024 positions, 2 residual streams, routed experts) beside the closest existing family (Zelunex: BF16 weights,
    window of 1024) at equal width, heads and active feed-forward weights.  Device-timed with CUDA events on the model's stream;
    prompts differ between steps and the weights of either model exceed L2."""
    import torch
    from ntransformer_b200 import kernels as K
    from ntransformer_b200.engine import Model
    from ntransformer_b200.model_spec import vebotar_config, vebotar_random_tensors, zelunex_config, zelunex_random_tensors

    torch.cuda.set_device(0)
    n_layers, vocab, prompt_len, max_seq, span = 4, 32000, 2048, 4096, 1024
    hbm, hbm_src = measured_peak_hbm()
    rows = []
    for name, (width, heads, kv, dim, vdim, experts, top, ff, sff) in VEBOTAR_SIZES.items():
        vc = vebotar_config(vocab=vocab, width=width, n_layers=n_layers, heads=heads, kv_heads=kv, dim=dim, vdim=vdim, chunk=span, rot_dims=dim // 2,
                            experts=experts, top=top, ff=ff, shared_ff=sff, streams=2, kv_from={n_layers - 1: n_layers - 2})
        zc = zelunex_config(vocab=vocab, width=width, n_layers=n_layers, heads=heads, kv_heads=kv, dim=vdim, vdim=vdim, ff=(top * ff + sff) * 2 // 3 // 128 * 128,
                            window=span)
        row = {"size": name, "layers": n_layers, "prompt_tokens": prompt_len, "decode_context": prompt_len, "span": span}
        for label, make in (("vebotar_bf16", lambda: Model.from_config_json(vc, vebotar_random_tensors(vc), max_context=max_seq)),
                            ("zelunex_bf16", lambda: Model.from_config_json(zc, zelunex_random_tensors(zc), max_context=max_seq))):
            model = make()
            stream = torch.cuda.ExternalStream(model.stream)
            prompts = [[token_at(i + 97 * j, vocab) for i in range(prompt_len)] for j in range(4)]
            for i in range(args.warmup):
                model.forward_async(prompts[i % 4], 0)
            model.sync()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            n0 = K.launch_count()
            psteps = max(3, min(args.steps, 8))
            a.record(stream)
            for i in range(psteps):
                model.forward_async(prompts[i % 4], 0)
            b.record(stream)
            model.sync()
            prefill = psteps * prompt_len / (a.elapsed_time(b) / 1e3)
            dsteps = max(8, min(args.steps, 256))
            for i in range(args.warmup):
                model.forward_async([token_at(i, vocab)], prompt_len + i)
            model.sync()
            a.record(stream)
            for i in range(dsteps):
                model.forward_async([token_at(i + 5, vocab)], prompt_len + args.warmup + i)
            b.record(stream)
            model.sync()
            ms = a.elapsed_time(b) / dsteps
            bpt = model.bytes_per_token(prompt_len + args.warmup + dsteps // 2)
            row[label] = {"prefill_tok_s": round(prefill, 1), "decode_tok_s": round(1e3 / ms, 1), "decode_ms": round(ms, 4),
                          "decode_bytes_per_token": bpt, "decode_frac_of_hbm_peak": round(bpt / (ms * 1e-3) / (hbm * 1e9), 3),
                          "launches": int(K.launch_count() - n0)}
            model.close()
            del model
            torch.cuda.empty_cache()
        rows.append(row)
    print(json.dumps({"metric": "family_compare", "family": "vebotar", "unit": "tok/s", "hbm_peak_gbs": hbm, "hbm_peak_source": hbm_src,
                      "dtype": "bf16 weights, f32 activations", "data": "synthetic", "rows": rows}))


TANOLORN_SIZES = {
    # name: (width, attention heads, unrotated dim, rotated dim, value dim, query rank, key/value rank, scan heads, scan head width, state, experts, top, expert ff).
    # 4 layers: scan + dense ff, latent attention + experts, scan + experts, latent attention reading layer 1's rows + experts.
    # The Vebotar model beside it has the same width, attention heads, experts and top; its experts are ungated (2 matrices), so their ff is
    # 3/2 of ours: equal weights per token.
    "2048_e8x1536": (2048, 16, 64, 32, 64, 768, 256, 32, 64, 64, 8, 2, 1536),
    "4096_e16x1536": (4096, 32, 128, 64, 128, 1536, 512, 64, 64, 128, 16, 4, 1536),
}


def run_family_compare_tanolorn(args):
    """--family-compare --family tanolorn: prompt-pass and decode throughput of the Tanolorn family (BF16 weights; latent attention and
    state-space scan layers, post-norm, gated experts with grouped sigmoid routing, per-layer token input) beside the closest existing
    family (Vebotar: BF16 weights, routed experts, shared caches) at equal width, heads and active expert weights.  Device-timed with CUDA
    events on the model's stream; prompts differ between steps and the weights of either model exceed L2."""
    import torch
    from ntransformer_b200 import kernels as K
    from ntransformer_b200.engine import Model
    from ntransformer_b200.model_spec import tanolorn_config, tanolorn_random_tensors, vebotar_config, vebotar_random_tensors

    torch.cuda.set_device(0)
    n_layers, vocab, prompt_len, max_seq = 4, 32000, 2048, 4096
    hbm, hbm_src = measured_peak_hbm()
    rows = []
    for name, (width, heads, dim, rot, vdim, qr, kvr, sh, sv, state, experts, top, eff) in TANOLORN_SIZES.items():
        tc = tanolorn_config(vocab=vocab, width=width, pattern=("mamba2", "latent_attention", "mamba2", "latent_attention"), kv_from={3: 1},
                             mlp=("dense", "moe", "moe", "moe"), heads=heads, dim=dim, rot_dim=rot, vdim=vdim, q_rank=qr, kv_rank=kvr, s_heads=sh, s_vdim=sv,
                             state=state, groups=8, norm_groups=8, ff=2 * width, experts=experts, top=top, eff=eff, route_groups=(4, 2), side=256)
        vc = vebotar_config(vocab=vocab, width=width, n_layers=n_layers, heads=heads, kv_heads=heads // 4, dim=vdim // 2, vdim=vdim, chunk=max_seq, rot_dims=vdim // 4,
                            experts=experts, top=top, ff=eff * 3 // 2 // 128 * 128, shared_ff=0, streams=0, kv_from={n_layers - 1: n_layers - 2})
        row = {"size": name, "layers": n_layers, "prompt_tokens": prompt_len, "decode_context": prompt_len}
        for label, make in (("tanolorn_bf16", lambda: Model.from_config_json(tc, tanolorn_random_tensors(tc), max_context=max_seq)),
                            ("vebotar_bf16", lambda: Model.from_config_json(vc, vebotar_random_tensors(vc), max_context=max_seq))):
            model = make()
            stream = torch.cuda.ExternalStream(model.stream)
            prompts = [[token_at(i + 97 * j, vocab) for i in range(prompt_len)] for j in range(4)]
            for i in range(args.warmup):
                model.forward_async(prompts[i % 4], 0)
            model.sync()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            n0 = K.launch_count()
            psteps = max(3, min(args.steps, 8))
            a.record(stream)
            for i in range(psteps):
                model.forward_async(prompts[i % 4], 0)
            b.record(stream)
            model.sync()
            prefill = psteps * prompt_len / (a.elapsed_time(b) / 1e3)
            dsteps = max(8, min(args.steps, 256))
            for i in range(args.warmup):
                model.forward_async([token_at(i, vocab)], prompt_len + i)
            model.sync()
            a.record(stream)
            for i in range(dsteps):
                model.forward_async([token_at(i + 5, vocab)], prompt_len + args.warmup + i)
            b.record(stream)
            model.sync()
            ms = a.elapsed_time(b) / dsteps
            bpt = model.bytes_per_token(prompt_len + args.warmup + dsteps // 2)
            row[label] = {"prefill_tok_s": round(prefill, 1), "decode_tok_s": round(1e3 / ms, 1), "decode_ms": round(ms, 4),
                          "decode_bytes_per_token": bpt, "decode_frac_of_hbm_peak": round(bpt / (ms * 1e-3) / (hbm * 1e9), 3),
                          "launches": int(K.launch_count() - n0)}
            model.close()
            del model
            torch.cuda.empty_cache()
        rows.append(row)
    print(json.dumps({"metric": "family_compare", "family": "tanolorn", "unit": "tok/s", "hbm_peak_gbs": hbm, "hbm_peak_source": hbm_src,
                      "dtype": "bf16 weights, f32 activations", "data": "synthetic", "rows": rows}))


# width -> (left attention: heads, kv heads, key width, value width), (delta rule: heads, q / k heads, key width, value width, ranks),
# (sink attention: heads, kv heads, key / value width), and the matching state-space / latent sizes of the family it stands beside
SAVIDRA_SIZES = {
    "w2048": dict(width=2048, left=dict(heads=16, kv_heads=2, dim=128, vdim=64), right=dict(heads=16, kv_heads=16, dim=64, vdim=128, decay_rank=64, gate_rank=64),
                  attn=dict(heads=16, kv_heads=4, dim=128, vdim=128), other=dict(heads=16, dim=64, rot_dim=64, vdim=128, q_rank=768, kv_rank=256, s_heads=32, s_vdim=64, state=64)),
    "w4096": dict(width=4096, left=dict(heads=32, kv_heads=2, dim=128, vdim=64), right=dict(heads=32, kv_heads=16, dim=128, vdim=128, decay_rank=128, gate_rank=128),
                  attn=dict(heads=32, kv_heads=8, dim=128, vdim=128), other=dict(heads=32, dim=64, rot_dim=64, vdim=128, q_rank=1536, kv_rank=512, s_heads=64, s_vdim=64, state=128)),
}


def run_family_compare_savidra(args):
    """--family-compare --family savidra: prompt-pass and decode throughput of the Savidra family (BF16 weights; head-mixed attention beside
    the gated delta rule, sink attention with blended values, token shift, norm on the residual sum, ReLU-gated feed-forward) beside the
    closest existing family (Tanolorn: post-norm, a recurrent mixer with a short convolution and carried state alternating with rotary
    attention, dense gated feed-forward) at equal width, layer count and feed-forward width.  Device-timed with CUDA events on the model's
    stream; prompts differ between steps and the weights of either model exceed L2."""
    import torch
    from ntransformer_b200 import kernels as K
    from ntransformer_b200.engine import Model
    from ntransformer_b200.model_spec import savidra_config, savidra_random_tensors, tanolorn_config, tanolorn_random_tensors

    torch.cuda.set_device(0)
    vocab, prompt_len, max_seq = 32000, 2048, 4096
    hbm, hbm_src = measured_peak_hbm()
    rows = []
    for name, z in SAVIDRA_SIZES.items():
        width, o = z["width"], z["other"]
        sc = savidra_config(vocab=vocab, width=width, ff=2 * width, left=z["left"], right=z["right"], attn=z["attn"])
        tc = tanolorn_config(vocab=vocab, width=width, pattern=("mamba2", "latent_attention", "mamba2", "latent_attention"), mlp=("dense",), heads=o["heads"],
                             dim=o["dim"], rot_dim=o["rot_dim"], vdim=o["vdim"], q_rank=o["q_rank"], kv_rank=o["kv_rank"], s_heads=o["s_heads"], s_vdim=o["s_vdim"],
                             state=o["state"], groups=8, norm_groups=8, ff=2 * width, side=0)
        row = {"size": name, "layers": 4, "prompt_tokens": prompt_len, "decode_context": prompt_len}
        for label, make in (("savidra_bf16", lambda: Model.from_config_json(sc, savidra_random_tensors(sc), max_context=max_seq)),
                            ("tanolorn_bf16", lambda: Model.from_config_json(tc, tanolorn_random_tensors(tc), max_context=max_seq))):
            model = make()
            stream = torch.cuda.ExternalStream(model.stream)
            prompts = [[token_at(i + 97 * j, vocab) for i in range(prompt_len)] for j in range(4)]
            for i in range(args.warmup):
                model.forward_async(prompts[i % 4], 0)
            model.sync()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            n0 = K.launch_count()
            psteps = max(3, min(args.steps, 8))
            a.record(stream)
            for i in range(psteps):
                model.forward_async(prompts[i % 4], 0)
            b.record(stream)
            model.sync()
            prefill = psteps * prompt_len / (a.elapsed_time(b) / 1e3)
            dsteps = max(8, min(args.steps, 256))
            for i in range(args.warmup):
                model.forward_async([token_at(i, vocab)], prompt_len + i)
            model.sync()
            a.record(stream)
            for i in range(dsteps):
                model.forward_async([token_at(i + 5, vocab)], prompt_len + args.warmup + i)
            b.record(stream)
            model.sync()
            ms = a.elapsed_time(b) / dsteps
            bpt = model.bytes_per_token(prompt_len + args.warmup + dsteps // 2)
            row[label] = {"prefill_tok_s": round(prefill, 1), "decode_tok_s": round(1e3 / ms, 1), "decode_ms": round(ms, 4),
                          "decode_bytes_per_token": bpt, "decode_frac_of_hbm_peak": round(bpt / (ms * 1e-3) / (hbm * 1e9), 3),
                          "launches": int(K.launch_count() - n0)}
            model.close()
            del model
            torch.cuda.empty_cache()
        rows.append(row)
    print(json.dumps({"metric": "family_compare", "family": "savidra", "unit": "tok/s", "hbm_peak_gbs": hbm, "hbm_peak_source": hbm_src,
                      "dtype": "bf16 weights, f32 activations", "data": "synthetic", "rows": rows}))


# width -> latent attention (shared by both models), recurrence (WKV heads x width against scan heads x width x state), experts
FUVOZEN_SIZES = {
    "w2048": dict(width=2048, latent=dict(heads=16, dim=64, rot_dim=64, vdim=128, kv_rank=256), q_rank=768, w_heads=32, w_dim=64, decay_rank=64, state=64, experts=16, eff=1408),
    "w4096": dict(width=4096, latent=dict(heads=32, dim=64, rot_dim=64, vdim=128, kv_rank=512), q_rank=1536, w_heads=64, w_dim=64, decay_rank=128, state=64, experts=16, eff=1536),
}


def time_family_model(model, args, prompt_len, vocab, hbm):
    """Prompt-pass and decode throughput of one model: CUDA events on the model's stream behind args.warmup steps; prompts differ between steps."""
    import torch
    from ntransformer_b200 import kernels as K

    stream = torch.cuda.ExternalStream(model.stream)
    prompts = [[token_at(i + 97 * j, vocab) for i in range(prompt_len)] for j in range(4)]
    for i in range(args.warmup):
        model.forward_async(prompts[i % 4], 0)
    model.sync()
    a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    n0 = K.launch_count()
    psteps = max(3, min(args.steps, 8))
    a.record(stream)
    for i in range(psteps):
        model.forward_async(prompts[i % 4], 0)
    b.record(stream)
    model.sync()
    prefill = psteps * prompt_len / (a.elapsed_time(b) / 1e3)
    dsteps = max(8, min(args.steps, 256))
    for i in range(args.warmup):
        model.forward_async([token_at(i, vocab)], prompt_len + i)
    model.sync()
    a.record(stream)
    for i in range(dsteps):
        model.forward_async([token_at(i + 5, vocab)], prompt_len + args.warmup + i)
    b.record(stream)
    model.sync()
    ms = a.elapsed_time(b) / dsteps
    bpt = model.bytes_per_token(prompt_len + args.warmup + dsteps // 2)
    return {"prefill_tok_s": round(prefill, 1), "decode_tok_s": round(1e3 / ms, 1), "decode_ms": round(ms, 4), "decode_bytes_per_token": bpt,
            "decode_frac_of_hbm_peak": round(bpt / (ms * 1e-3) / (hbm * 1e9), 3), "launches": int(K.launch_count() - n0)}


def fuvozen_pair(z, vocab):
    """(Fuvozen, Tanolorn) configurations of one size: recurrence + dense feed-forward, latent attention + experts, twice.  Equal feed-forward
    weights: an ungated unit of 3 x width against a gated one of 2 x width; three routed experts and a shared one against four routed ones."""
    from ntransformer_b200.model_spec import fuvozen_config, tanolorn_config

    w, A = z["width"], z["latent"]
    fc = fuvozen_config(vocab=vocab, width=w, w_heads=z["w_heads"], w_dim=z["w_dim"], decay_rank=z["decay_rank"], ff=3 * w, experts=z["experts"], top=3, eff=z["eff"],
                        shared=z["eff"], window=1024, **A)
    tc = tanolorn_config(vocab=vocab, width=w, pattern=("mamba2", "latent_attention", "mamba2", "latent_attention"), mlp=("dense", "moe", "dense", "moe"),
                         q_rank=z["q_rank"], s_heads=z["w_heads"], s_vdim=z["w_dim"], state=z["state"], groups=8, norm_groups=8, ff=2 * w, experts=z["experts"], top=4,
                         eff=z["eff"], route_groups=None, side=0, **A)
    return fc, tc


def run_family_compare_fuvozen(args):
    """--family-compare --family fuvozen: prompt-pass and decode throughput of the Fuvozen family (BF16 weights; WKV time mixers alternating
    with windowed latent attention, mixer and feed-forward in parallel, average over depth, grouped norms, experts with a shared one)
    beside the closest existing family (Tanolorn: state-space scans alternating with latent attention, gated experts) at equal width, layer
    count, heads, latent rank, recurrent state and active feed-forward weights."""
    import torch
    from ntransformer_b200.engine import Model
    from ntransformer_b200.model_spec import fuvozen_random_tensors, tanolorn_random_tensors

    torch.cuda.set_device(0)
    vocab, prompt_len, max_seq = 32000, 2048, 4096
    hbm, hbm_src = measured_peak_hbm()
    rows = []
    for name, z in FUVOZEN_SIZES.items():
        fc, tc = fuvozen_pair(z, vocab)
        row = {"size": name, "layers": 4, "prompt_tokens": prompt_len, "decode_context": prompt_len}
        for label, make in (("fuvozen_bf16", lambda: Model.from_config_json(fc, fuvozen_random_tensors(fc), max_context=max_seq)),
                            ("tanolorn_bf16", lambda: Model.from_config_json(tc, tanolorn_random_tensors(tc), max_context=max_seq))):
            model = make()
            row[label] = time_family_model(model, args, prompt_len, vocab, hbm)
            model.close()
            del model
            torch.cuda.empty_cache()
        rows.append(row)
    print(json.dumps({"metric": "family_compare", "family": "fuvozen", "unit": "tok/s", "hbm_peak_gbs": hbm, "hbm_peak_source": hbm_src,
                      "dtype": "bf16 weights, f32 activations", "data": "synthetic", "rows": rows}))


# width -> latent attention (shared by both models), matrix memory against WKV of equal state volume, grouped-query attention, experts
TIBELIX_SIZES = {
    "w2048": dict(width=2048, latent=dict(dim=64, rot_dim=64, kv_rank=256), l_heads=16, vdim=128, q_rank=768, m_heads=8, m_dim=128, w_heads=32, w_dim=64, decay_rank=64,
                  heads=16, kv_heads=4, experts=16, eff=1408),
    "w4096": dict(width=4096, latent=dict(dim=64, rot_dim=64, kv_rank=512), l_heads=32, vdim=128, q_rank=1536, m_heads=16, m_dim=128, w_heads=64, w_dim=64, decay_rank=128,
                  heads=32, kv_heads=8, experts=16, eff=1536),
}


def tibelix_pair(z, vocab, mixers=("mlstm", "latent_attention")):
    """(Tibelix, Fuvozen) configurations of one size: recurrence + dense feed-forward, attention + experts, twice.  Equal width, latent heads and
    ranks, feed-forward widths and experts; the recurrences' states hold equally many numbers (heads x 128 x 128 against 4 heads x 64 x 64)."""
    from ntransformer_b200.model_spec import fuvozen_config, tibelix_config

    w = z["width"]
    tc = tibelix_config(vocab=vocab, width=w, pattern=mixers * 2, l_heads=z["l_heads"], l_dim=z["latent"]["dim"], rot_dim=z["latent"]["rot_dim"], l_vdim=z["vdim"],
                        kv_rank=z["latent"]["kv_rank"], q_rank=z["q_rank"], m_heads=z["m_heads"], m_dim=z["m_dim"], m_vdim=z["m_dim"], heads=z["heads"], kv_heads=z["kv_heads"],
                        ff=3 * w, experts=z["experts"], top=3, eff=z["eff"], shared=z["eff"])
    fc = fuvozen_config(vocab=vocab, width=w, heads=z["l_heads"], vdim=z["vdim"], w_heads=z["w_heads"], w_dim=z["w_dim"], decay_rank=z["decay_rank"], ff=3 * w,
                        experts=z["experts"], top=3, eff=z["eff"], shared=z["eff"], window=0, **z["latent"])
    return tc, fc


def run_family_compare_tibelix(args):
    """--family-compare --family tibelix: prompt-pass and decode throughput of the Tibelix family (BF16 weights; matrix memories alternating with
    latent attention or with distance-biased attention, norms in front of and behind each sublayer, experts with a shared one) beside the closest
    existing family (Fuvozen: WKV time mixers alternating with latent attention, experts with a shared one) at equal width, layer count, heads,
    latent rank, recurrent state and feed-forward weights."""
    import torch
    from ntransformer_b200.engine import Model
    from ntransformer_b200.model_spec import fuvozen_random_tensors, tibelix_random_tensors

    torch.cuda.set_device(0)
    vocab, prompt_len, max_seq = 32000, 2048, 4096
    hbm, hbm_src = measured_peak_hbm()
    rows = []
    for name, z in TIBELIX_SIZES.items():
        tc, fc = tibelix_pair(z, vocab)
        ac, _ = tibelix_pair(z, vocab, ("mlstm", "attention"))
        row = {"size": name, "layers": 4, "prompt_tokens": prompt_len, "decode_context": prompt_len}
        for label, make in (("tibelix_bf16", lambda: Model.from_config_json(tc, tibelix_random_tensors(tc), max_context=max_seq)),
                            ("tibelix_biased_attention_bf16", lambda: Model.from_config_json(ac, tibelix_random_tensors(ac), max_context=max_seq)),
                            ("fuvozen_bf16", lambda: Model.from_config_json(fc, fuvozen_random_tensors(fc), max_context=max_seq))):
            model = make()
            row[label] = time_family_model(model, args, prompt_len, vocab, hbm)
            model.close()
            del model
            torch.cuda.empty_cache()
        rows.append(row)
    print(json.dumps({"metric": "family_compare", "family": "tibelix", "unit": "tok/s", "hbm_peak_gbs": hbm, "hbm_peak_source": hbm_src,
                      "dtype": "bf16 weights, f32 activations", "data": "synthetic", "rows": rows}))


def run_family_compare(args):
    """--family-compare: prompt-pass and decode throughput of the Zelunex family (BF16 weights, windowed attention) beside the
    closest GGUF family member (Llama block, F16 weights, full causal attention) at equal layer sizes.  Device-timed with CUDA
    events on the model's stream; prompts differ between steps and the weights of either model exceed L2."""
    import torch
    from dataclasses import replace
    from ntransformer_b200 import kernels as K
    from ntransformer_b200.engine import Model
    from ntransformer_b200.model_spec import LLAMA3_8B, zelunex_config, zelunex_random_tensors

    torch.cuda.set_device(0)
    n_layers, vocab, prompt_len, max_seq, window = 4, 32000, 2048, 4096, 1024
    hbm, hbm_src = measured_peak_hbm()
    rows = []
    for name, (width, heads, kv, dim, ff) in FAMILY_SIZES.items():
        zc = zelunex_config(vocab=vocab, width=width, n_layers=n_layers, heads=heads, kv_heads=kv, dim=dim, vdim=dim, ff=ff, window=window)
        lc = replace(LLAMA3_8B, vocab_size=vocab, hidden_size=width, intermediate_size=ff, n_layers=n_layers, n_heads=heads, n_kv_heads=kv, head_dim=dim,
                     max_seq_len=max_seq)
        row = {"size": name, "layers": n_layers, "prompt_tokens": prompt_len, "decode_context": prompt_len, "window": window}
        for label, make in (("zelunex_bf16", lambda: Model.from_config_json(zc, zelunex_random_tensors(zc), max_context=max_seq)),
                            ("llama_f16", lambda: Model.synthetic(lc, "F16", seed=1234))):
            model = make()
            stream = torch.cuda.ExternalStream(model.stream)
            prompts = [[token_at(i + 97 * j, vocab) for i in range(prompt_len)] for j in range(4)]
            for i in range(args.warmup):
                model.forward_async(prompts[i % 4], 0)
            model.sync()
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            n0 = K.launch_count()
            psteps = max(3, min(args.steps, 8))
            a.record(stream)
            for i in range(psteps):
                model.forward_async(prompts[i % 4], 0)
            b.record(stream)
            model.sync()
            prefill = psteps * prompt_len / (a.elapsed_time(b) / 1e3)
            dsteps = max(8, min(args.steps, 256))
            for i in range(args.warmup):
                model.forward_async([token_at(i, vocab)], prompt_len + i)
            model.sync()
            a.record(stream)
            for i in range(dsteps):
                model.forward_async([token_at(i + 5, vocab)], prompt_len + args.warmup + i)
            b.record(stream)
            model.sync()
            ms = a.elapsed_time(b) / dsteps
            bpt = model.bytes_per_token(prompt_len + args.warmup + dsteps // 2)
            row[label] = {"prefill_tok_s": round(prefill, 1), "decode_tok_s": round(1e3 / ms, 1), "decode_ms": round(ms, 4),
                          "decode_bytes_per_token": bpt, "decode_frac_of_hbm_peak": round(bpt / (ms * 1e-3) / (hbm * 1e9), 3),
                          "launches": int(K.launch_count() - n0)}
            model.close()
            del model
            torch.cuda.empty_cache()
        rows.append(row)
    print(json.dumps({"metric": "family_compare", "unit": "tok/s", "hbm_peak_gbs": hbm, "hbm_peak_source": hbm_src, "dtype": "bf16 / f16 weights, f32 activations",
                      "data": "synthetic", "rows": rows}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=128)
    ap.add_argument("--warmup", type=int, default=8)
    ap.add_argument("--workload", default="llama3-70b-q4_k_m-decode", choices=sorted(WORKLOADS))
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-configs3", action="store_true", help="8 GPUs: skip the extra 70B Q6_K run reported under configs3")
    ap.add_argument("--check", action="store_true",
                    help="parity instead of timing: the same seeded GGUF through the reference's CUDA path (oracle/_ref) and ours; "
                         "logits <= 1e-3 relative and --steps greedy ids identical")
    ap.add_argument("--prompt-tokens", type=int, default=None, help="override the workload's prompt length (profiling)")
    ap.add_argument("--layers", type=int, default=0, help="--check only: keep this many layers of the workload's shape (0 = all)")
    ap.add_argument("--oracle-steps", type=int, default=0, help="--check only: also run the F64-accumulating CPU oracle for the prompt and this many steps")
    ap.add_argument("--all-errs", action="store_true", help="--check only: list the error of every step, not the first 8")
    ap.add_argument("--family-compare", action="store_true",
                    help="instead of the workload: Zelunex beside the Llama block at equal layer sizes, prompt pass and decode (1 GPU)")
    ap.add_argument("--family", default="zelunex", choices=["zelunex", "vebotar", "tanolorn", "savidra", "fuvozen", "tibelix"],
                    help="--family-compare only: zelunex beside the Llama block (default), vebotar beside zelunex, tanolorn beside vebotar, savidra / fuvozen beside tanolorn, or tibelix beside fuvozen")
    ap.add_argument("--per-token-prompt", action="store_true", help="--check only: our engine replays the prompt token by token like the reference")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3)
    rank = int(os.environ.get("RANK", 0))
    world = int(os.environ.get("WORLD_SIZE", 1))
    if world != args.gpus and world == 1 and args.gpus > 1:
        sys.exit("bench.py --gpus N > 1 must be launched with torch.distributed.run (one rank per GPU)")
    if args.family_compare:
        if rank == 0:
            {"vebotar": run_family_compare_vebotar, "tanolorn": run_family_compare_tanolorn, "savidra": run_family_compare_savidra,
             "fuvozen": run_family_compare_fuvozen, "tibelix": run_family_compare_tibelix}.get(args.family, run_family_compare)(args)
    elif args.check:
        run_check(args, rank, world)
    elif args.impl == "reference":
        run_reference(args, rank, world)
    elif "prefill" in args.workload:
        run_prefill(args, rank, world)
    else:
        run_ours(args, rank, world)


if __name__ == "__main__":
    main()
