#!/usr/bin/env python
"""bench.py — greedy Jacobi decoding throughput (tokens/sec + Jacobi iterations to fixed point), Qwen2.5-7B shape,
block size n=32, synthetic 512-token prompt / 512 new tokens, random-init weights.

  python bench.py --gpus N --steps K --warmup W            this repo's B200 path (one process per GPU under torchrun)
  python bench.py --impl reference --gpus N --steps K ...  the reference's CPU path (oracle port) on the host cores

A "step" = one generation: the device-resident Jacobi loop produces `--gen` new tokens for every sequence of the batch
from an already prefilled prompt (the reference's metric excludes prefill: toks_per_sec = new_tokens / gen_only_time,
JacobiForcing/jacobi_forcing_inference_MR_humaneval.py:217-230, 250).
  value  = new tokens / device time of the generation's kernels, first to last (inputs resident in HBM), max over ranks
  e2e    = new tokens / wall time of the C-ABI call jf_jacobi_run with HOST buffers (H2D of prompts, drafts, block
           tables and D2H of the generated ids inside the timed region)
One JSON line on stdout (rank 0).
"""
from __future__ import annotations

import argparse
import json
import os
import random
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

METRIC = "tokens/sec (greedy Jacobi decode, Qwen2.5-7B random-init, n=32, 512 prompt / 512 gen, prefill excluded)"
UNIT = "tokens/s"

SHAPES = {
    "qwen2.5-coder-7b": dict(hidden_size=3584, num_hidden_layers=28, num_attention_heads=28, num_key_value_heads=4,
                             head_dim=128, intermediate_size=18944, vocab_size=152064, tie_word_embeddings=False,
                             rope_theta=1e6, max_position_embeddings=32768, rms_norm_eps=1e-6),
    "qwen2.5-math-7b": dict(hidden_size=3584, num_hidden_layers=28, num_attention_heads=28, num_key_value_heads=4,
                            head_dim=128, intermediate_size=18944, vocab_size=152064, tie_word_embeddings=False,
                            rope_theta=1e4, max_position_embeddings=4096, rms_norm_eps=1e-6),
    "qwen2-0.5b": dict(hidden_size=896, num_hidden_layers=24, num_attention_heads=14, num_key_value_heads=2,
                       head_dim=64, intermediate_size=4864, vocab_size=151936, tie_word_embeddings=True,
                       rope_theta=1e6, max_position_embeddings=32768, rms_norm_eps=1e-6),
    "tiny": dict(hidden_size=256, num_hidden_layers=2, num_attention_heads=4, num_key_value_heads=2, head_dim=64,
                 intermediate_size=512, vocab_size=1000, tie_word_embeddings=False, rope_theta=1e6,
                 max_position_embeddings=4096, rms_norm_eps=1e-6),
}


def algorithmic_bytes_per_forward(cfg: dict, rows: float, ctx: float, batch_groups: float, tp: int = 1,
                                  shard_attention: bool = False) -> float:
    """Per GPU: every layer weight + LM head once, committed KV once per group, in-flight KV
    written and read, embedding rows gathered.  Logits are never materialised.  Tensor parallelism: the MLP and the LM
    head are sharded tp ways; the attention block (weights, KV) is sharded only with shard_attention, else replicated."""
    h, L, I, V = cfg["hidden_size"], cfg["num_hidden_layers"], cfg["intermediate_size"], cfg["vocab_size"]
    q = cfg["num_attention_heads"] * cfg["head_dim"]
    kv = cfg["num_key_value_heads"] * cfg["head_dim"]
    tpa = tp if shard_attention else 1
    w_attn = 2 * (h * (q + 2 * kv) + (q + 2 * kv) + q * h) / tpa
    w_mlp = 2 * (3 * h * I) / tp
    w_head = 2 * V * h / tp
    kvb = L * 2 * kv * 2 / tpa
    return L * (w_attn + w_mlp + 2 * 2 * h) + w_head + batch_groups * ctx * kvb + rows * kvb + rows * h * 2


class ClockSampler:
    """nvidia-smi clocks / throttle reasons sampled DURING the timed region."""
    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int):
        self.gpu = gpu_index
        self.samples = []
        self._stop = threading.Event()
        self._t = None

    def _run(self):
        while not self._stop.is_set():
            try:
                out = subprocess.run(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                      "-i", str(self.gpu)], capture_output=True, text=True, timeout=5).stdout.strip()
                if out:
                    self.samples.append([x.strip() for x in out.split(",")])
            except Exception:
                pass
            self._stop.wait(0.2)

    def start(self):
        self._t = threading.Thread(target=self._run, daemon=True)
        self._t.start()

    def stop(self) -> dict:
        self._stop.set()
        if self._t:
            self._t.join(timeout=6)
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for s in self.samples:
            try:
                sm.append(float(s[1])); mx.append(float(s[2]))
                for nm, v in zip(names, s[5:9]):
                    if v.lower().startswith("active"):
                        reasons.add(nm)
            except Exception:
                continue
        sm.sort()
        return {"sm_mhz": (sm[len(sm) // 2] if sm else None), "sm_max_mhz": (max(mx) if mx else None),
                "reasons": sorted(reasons), "samples": len(sm)}


def random_weights(cfg: dict, seed: int, device: str):
    """Yields (HF parameter name, bf16 tensor on `device`): HF `_init_weights` shape of randomness (N(0, 0.02) linears
    and embeddings, unit norms, zero biases) from one seeded generator, so the GPU arm and the CPU reference arm hold
    the SAME model when both draw on the same device type."""
    import torch
    g = torch.Generator(device=device).manual_seed(seed)
    h, I, V = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"]
    q = cfg["num_attention_heads"] * cfg["head_dim"]
    kv = cfg["num_key_value_heads"] * cfg["head_dim"]

    def rnd(*shape):
        return (torch.randn(*shape, generator=g, device=device, dtype=torch.float32) * 0.02).to(torch.bfloat16)

    def ones(k):
        return torch.ones(k, device=device, dtype=torch.bfloat16)

    def zeros(k):
        return torch.zeros(k, device=device, dtype=torch.bfloat16)

    yield "model.embed_tokens.weight", rnd(V, h)
    if not cfg["tie_word_embeddings"]:
        yield "lm_head.weight", rnd(V, h)
    yield "model.norm.weight", ones(h)
    for l in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{l}."
        yield p + "self_attn.q_proj.weight", rnd(q, h)
        yield p + "self_attn.k_proj.weight", rnd(kv, h)
        yield p + "self_attn.v_proj.weight", rnd(kv, h)
        yield p + "self_attn.q_proj.bias", zeros(q)
        yield p + "self_attn.k_proj.bias", zeros(kv)
        yield p + "self_attn.v_proj.bias", zeros(kv)
        yield p + "self_attn.o_proj.weight", rnd(h, q)
        yield p + "mlp.gate_proj.weight", rnd(I, h)
        yield p + "mlp.up_proj.weight", rnd(I, h)
        yield p + "mlp.down_proj.weight", rnd(h, I)
        yield p + "input_layernorm.weight", ones(h)
        yield p + "post_attention_layernorm.weight", ones(h)


def load_random_weights(rt, cfg: dict, seed: int, device: str):
    import torch
    for name, t in random_weights(cfg, seed, device):
        rt.load_tensor(name, t)
    rt.finalize()
    torch.cuda.synchronize()


def build_cpu_reference_model(args, cfg: dict, seed: int):
    """The oracle-side HF model holding the same weights as the GPU arm (drawn on cuda:0, copied to the host); falls
    back to the recycled-pool timing model when no GPU is visible."""
    import torch
    from oracle.cpu_baseline import build_model_from_named_tensors, build_timing_model
    if torch.cuda.is_available():
        return build_model_from_named_tensors(args.model, ((n, t.cpu()) for n, t in random_weights(cfg, seed, "cuda:0"))), \
            "same seeded N(0,0.02) weights as the GPU arm"
    return build_timing_model(args.model, dtype=torch.bfloat16, seed=0), "weights recycled from one N(0,0.02) pool"


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured (MEASURED_PEAKS.json)"
    except Exception:
        return 6650.0, "fallback (an earlier copy measurement)"


# --------------------------------------------------------------------------------------------------------------------
# reference arm: the reference's CPU HF path (oracle port) on the host cores
# --------------------------------------------------------------------------------------------------------------------
def run_reference(args, rank: int):
    if rank != 0:
        return
    import torch
    from oracle.cpu_baseline import host_cores, time_reference_jacobi
    cores = host_cores()
    torch.set_num_threads(cores)
    cfg = SHAPES[args.model]
    model, wdesc = build_cpu_reference_model(args, cfg, 1234)
    g = torch.Generator().manual_seed(1)
    prompt = torch.randint(0, cfg["vocab_size"], (args.prompt,), generator=g).tolist()
    budget = args.ref_budget_s
    per_step = []
    for i in range(args.warmup + args.steps):
        res = time_reference_jacobi(model, prompt, args.n, mode=args.mode, max_new_tokens=args.gen, budget_s=budget,
                                    K=args.K, r=args.r, pool=args.pool, pad=0, draft_seed=2 + 1000 * i)
        if i >= args.warmup:
            per_step.append(res)
    toks = sum(r["tokens"] for r in per_step)
    secs = sum(r["seconds"] for r in per_step)
    iters = sum(r["iters"] for r in per_step)
    value = toks / secs if secs > 0 else 0.0
    sample = (f"per step: prefill {args.prompt}+{args.n} tokens (untimed) then n={args.n} blocks ({args.mode}) of the "
              f"reference's HF Jacobi path on CPU until {args.gen} tokens or {budget:.0f} s, bf16, {cores} threads; "
              f"{wdesc}")
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": args.gpus, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": 1e3 * secs / max(1, len(per_step)), "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": workload_config(args, 1, "cpu"),
        "iterations": iters, "tokens": toks, "iters_per_token": (iters / toks if toks else None),
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def workload_config(args, world: int, where: str) -> dict:
    return {"workload": f"{args.model} random-init, block_size n={args.n}, {args.mode} greedy Jacobi "
                        f"(K={args.K}, r={args.r}, pool={args.pool}), batch={args.batch} per GPU, "
                        f"prompt={args.prompt}, gen={args.gen}, EOS disabled",
            "baseline_config": "configs[1]: Qwen2.5-Coder-7B random-init, block_size=32, batch=1, 1xB200, greedy "
                               "single-block Jacobi",
            "parallelism": ("single GPU" if world == 1 else
                            (f"{world} independent engines, one sequence batch per GPU, no data-path collective "
                             "(--replicas)") if getattr(args, "_tp", 1) == 1 else
                            (f"tp{args._tp} x {world // args._tp} group(s): tensor-parallel column/row split of "
                             + ("every linear layer (two exchanges per block)" if args.tp_shard_attention else
                                "gate/up/down + vocabulary-parallel LM head, attention replicated (ONE exchange per "
                                "transformer block)")
                             + ", in-kernel reduce-scatter + all-gather by push over NVLink peer memory (no NCCL on the "
                               "data path), independent sequence batches across groups")),
            "l2_policy": "inputs larger than L2: every forward streams 15.2 GB of weights (L2 = 126 MB)",
            "where": where}


# --------------------------------------------------------------------------------------------------------------------
# this repo's arm
# --------------------------------------------------------------------------------------------------------------------
def run_ours(args, rank: int, local_rank: int, world: int):
    import numpy as np
    import torch
    import torch.distributed as dist
    from jacobiforcing_b200.policy import MODES, PolicyKnobs, draw_prefill_draft, mt_state_words
    from jacobiforcing_b200.runtime import JacobiRuntime

    torch.cuda.set_device(local_rank)
    device = f"cuda:{local_rank}"
    cfg = SHAPES[args.model]
    # Layout at N GPUs: ONE tensor-parallel group of N ranks - the path shards along the
    # intermediate / vocabulary dimensions (and the heads with --tp-shard-attention), strong scaling of the batch-1
    # headline.  --tp T < N: N / T groups with independent sequence batches; --replicas: N independent engines (how the
    # reference's own sweep uses several GPUs, scripts/inference/scanning_hyperparameter_jacobi_decoding_mr.sh:31-45).
    tp = 1 if args.replicas else (args.tp if args.tp > 0 else world)
    divides = cfg["num_key_value_heads"] % tp == 0 and cfg["num_attention_heads"] % tp == 0
    args.tp_shard_attention = tp > 1 and (args.tp_attn == "shard" or (args.tp_attn == "auto" and divides))
    if world % tp or tp not in (1, 2, 4, 8) or (args.tp_shard_attention and cfg["num_key_value_heads"] % tp):
        raise SystemExit(f"--tp {tp} does not fit {world} GPUs / {cfg['num_key_value_heads']} KV heads")
    groups = world // tp
    args._tp = tp
    group_id, tp_rank = rank // tp, rank % tp
    tp_group = None
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device(device))
        for gi in range(groups):
            pg = dist.new_group(list(range(gi * tp, (gi + 1) * tp)))
            if gi == group_id:
                tp_group = pg
    B, P, G, n = args.batch, args.prompt, args.gen, args.n
    rows_cap = max(P + n, B * n * (2 if args.mode == "multiblock" else 1) * max(1, args.pool if args.mode == "multiblock" else 1))
    rows_cap = min(max(rows_cap, 64), 4096)
    pages = (P + G + 3 * n + 255) // 256 + 1
    rt = JacobiRuntime(cfg, device=local_rank, max_rows=rows_cap, max_seqs=B, num_kv_pages=pages * B,
                       max_pages_per_seq=pages, attn_chunk=args.attn_chunk, gen_capacity=P + G + 4 * n + 8,
                       max_calls=G // n + 8,
                       tp_rank=tp_rank, tp_size=tp, tp_group=tp_group, tp_shard_attention=args.tp_shard_attention)
    load_random_weights(rt, cfg, seed=1234 + group_id, device=device)

    knobs = PolicyKnobs(mode=MODES[args.mode], n=n, K=args.K, r=args.r, n_gram_pool_size=args.pool, eos=None, pad=0,
                        max_iteration_count=128, max_new_tokens=G, max_calls=G // n + 4, vocab=cfg["vocab_size"])
    g = torch.Generator().manual_seed(1 + group_id)
    prompts = torch.randint(0, cfg["vocab_size"], (B, P), generator=g).tolist()

    def one_step(step_idx: int):
        seqs, fcs, fcts, chs = [], [], [], []
        t_pre = 0.0
        for b in range(B):
            rng = random.Random(2 + 1000 * step_idx + b + 100000 * group_id)
            s = rt.new_sequence()
            fc, drafted, ms = rt.prefill(s, prompts[b], draw_prefill_draft(rng, prompts[b], n))
            t_pre += ms
            seqs.append(s); fcs.append(fc); fcts.append(drafted)
            chs.append(mt_state_words(rng))
        torch.cuda.synchronize()
        launched = rt.launches
        t0 = time.perf_counter()
        results, run = rt.jacobi_run(seqs, knobs, fcs, fcts, rng_states=chs)     # host buffers in, host ids out
        wall = time.perf_counter() - t0
        by_stages = rt.launches - launched > 1
        toks = sum(len(r.tokens) for r in results)
        iters = run["forwards"]
        h2d = 4 * (B * P + B * n + B * 625 + B * pages + 3 * B) + 64 * B
        d2h = 4 * (B * (G + 3 * n + 1) + 8 * B + B * rt.max_calls) + 16
        if by_stages:
            d2h += 188 * (iters + 1)                 # the plan's header, which the host reads before every forward (struct PlanHdr)
        for s in seqs:
            rt.release(s)
        return {"tokens": toks, "forwards": iters, "device_ms": run["device_ms"], "wall_s": wall, "rows": run["rows"],
                "prefill_ms": t_pre, "h2d": h2d, "d2h": d2h,
                "iters_per_seq": [r.total_iterations for r in results],
                "stop": [r.stop_reason for r in results]}

    # Tensor-parallel self-check on the engine about to be timed (untimed): a short greedy generation decoded
    # autoregressively (n = 1) and by Jacobi iteration (n = 8, n = args.n) must give the SAME ids (exact on this engine:
    # attention chunks are aligned to absolute key positions), and every rank of the group must return the same ids,
    # iteration counts and forward counts - the ranks run the policy independently on keys merged over NVLink peer memory.
    tp_check = None
    if tp > 1:
        from jacobiforcing_b200.runtime import hf_generate
        runs = {}
        m_chk = max(4, min(16, rt.max_calls - 2))        # n = 1 needs one call per token
        for nn in (1, 8, n):
            seqs_c, res_c, run_c = hf_generate(rt, [prompts[0][:64]], n=nn, max_new_tokens=m_chk, mode="single", pad=0,
                                               rngs=[random.Random(7)])
            runs[nn] = (res_c[0].tokens[:m_chk], list(res_c[0].iters), int(run_c["forwards"]))
            for s_c in seqs_c:
                rt.release(s_c)
        gathered = [None] * tp
        dist.all_gather_object(gathered, runs, group=tp_group)
        ok_ar = runs[1][0] == runs[8][0] == runs[n][0]
        ok_ranks = all(g2 == gathered[0] for g2 in gathered)
        flags = torch.tensor([1.0 if ok_ar else 0.0, 1.0 if ok_ranks else 0.0], device=device)
        dist.all_reduce(flags, op=dist.ReduceOp.MIN)
        tp_check = {"jacobi_equals_ar": bool(flags[0] > 0), "ranks_identical": bool(flags[1] > 0), "tokens": m_chk,
                    "block_sizes": [1, 8, n], "forwards": [runs[1][2], runs[8][2], runs[n][2]],
                    "what": f"{m_chk} greedy tokens from a 64-token prompt on the timed tensor-parallel engine: AR == Jacobi(8) == "
                            f"Jacobi({n}) ids, and ids / per-call iterations / forward counts identical on all {tp} ranks of "
                            "every group (min over all ranks)"}
        if not (tp_check["jacobi_equals_ar"] and tp_check["ranks_identical"]) and rank == 0:
            # reported, not fatal: the line below still carries the measurement, with the failed flags in `tp_check`
            print(f"[bench] WARNING: tensor-parallel self-check failed: {tp_check}", file=sys.stderr, flush=True)

    for i in range(args.warmup):
        one_step(i)
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    launches0 = rt.launches
    t_begin = time.perf_counter()
    steps = [one_step(args.warmup + i) for i in range(args.steps)]
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    t_total = time.perf_counter() - t_begin
    clocks = sampler.stop() if rank == 0 else {}
    launches = rt.launches - launches0

    toks = sum(s["tokens"] for s in steps)
    dev_s = sum(s["device_ms"] for s in steps) / 1e3
    wall_s = sum(s["wall_s"] for s in steps)
    fwd = sum(s["forwards"] for s in steps)
    rows = sum(s["rows"] for s in steps)
    lead = 1.0 if tp_rank == 0 else 0.0                  # tokens / forwards are counted once per tensor-parallel group
    stats = torch.tensor([dev_s, wall_s, lead * toks, lead * fwd, lead * rows, float(launches)], device=device,
                         dtype=torch.float64)
    if world > 1:
        mx = stats.clone(); dist.all_reduce(mx, op=dist.ReduceOp.MAX)
        sm = stats.clone(); dist.all_reduce(sm, op=dist.ReduceOp.SUM)
        dev_s_max, wall_s_max = float(mx[0]), float(mx[1])
        toks_all, fwd_all, rows_all, launches_all = float(sm[2]), float(sm[3]), float(sm[4]), int(sm[5])
    else:
        dev_s_max, wall_s_max = dev_s, wall_s
        toks_all, fwd_all, rows_all, launches_all = float(toks), float(fwd), float(rows), launches
    if rank != 0:
        if world > 1:
            dist.destroy_process_group()
        return

    value = toks_all / dev_s_max
    e2e = toks_all / wall_s_max
    peak, peak_src = measured_peaks()
    # roofline of a generation's kernels on rank 0: the persistent Jacobi kernel (one launch per step), or one kernel per stage
    one_launch = launches <= len(steps)
    mean_rows = rows / max(1, fwd)
    mean_ctx = P + G / 2.0
    groups_per_fwd = mean_rows / max(1.0, float(n)) if args.mode == "single" else max(1.0, mean_rows / (2.0 * n))
    bytes_fwd = algorithmic_bytes_per_forward(cfg, mean_rows, mean_ctx, max(float(B), groups_per_fwd), tp,
                                              args.tp_shard_attention)
    bytes_launch = bytes_fwd * fwd / max(1, len(steps))
    launch_s = dev_s / max(1, len(steps))
    achieved = bytes_launch / launch_s / 1e9
    roofline = {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                "traffic": None, "kernel": "jf_persistent_kernel" if one_launch else "one kernel per stage (jf_step.cuh), a generation's together",
                "peak_source": peak_src,
                "algorithmic_bytes_per_forward": bytes_fwd, "forwards_per_launch": fwd / max(1, len(steps)),
                "ms_per_forward": 1e3 * dev_s / max(1, fwd)}
    prof = os.path.join(ROOT, "profiles", "traffic.json")
    if os.path.exists(prof) and tp == 1 and args.model == "qwen2.5-coder-7b" and B == 1:
        try:
            per_fwd = json.load(open(prof)).get("dram_bytes_per_forward" if one_launch else "dram_bytes_per_forward_by_stages")
            # bytes of one forward of this shape; a generation runs `forwards_per_launch` of them
            roofline["traffic"] = per_fwd * roofline["forwards_per_launch"] if per_fwd else None
            roofline["traffic_source"] = ("not measured in this run: dram__bytes_read+write per forward from the ncu "
                                          "capture recorded in profiles/traffic.json, times this launch's "
                                          "forward count")
            roofline["achieved_bytes_per_launch"] = bytes_launch
        except Exception:
            pass

    cpu = None
    if not args.no_cpu_baseline and world == 1:
        try:
            from oracle.cpu_baseline import host_cores, time_reference_jacobi
            cores = host_cores()
            torch.set_num_threads(cores)
            t0 = time.perf_counter()
            model, wdesc = build_cpu_reference_model(args, cfg, 1234)
            res = time_reference_jacobi(model, prompts[0], n, mode=args.mode, max_new_tokens=G,
                                        budget_s=args.ref_budget_s, K=args.K, r=args.r, pool=args.pool, pad=0,
                                        draft_seed=2 + 1000 * args.warmup)
            cpu = {"value": res["tokens"] / res["seconds"] if res["seconds"] > 0 else 0.0, "unit": UNIT,
                   "cores": cores, "kind": "port",
                   "sample": f"{res['calls']} n={n} blocks ({res['tokens']} tokens, {res['iters']} Jacobi iterations, "
                             f"{res['seconds']:.1f} s; budget {args.ref_budget_s:.0f} s) after an untimed {P}+{n}-token "
                             f"prefill: HF transformers CPU bf16 forward driven by the pinned policy restatement, "
                             f"{wdesc}; model build+prefill {time.perf_counter() - t0 - res['seconds']:.0f} s not counted",
                   "iters_per_token": res["iters"] / max(1, res["tokens"]),
                   "iters_per_s": res["iters"] / res["seconds"] if res["seconds"] > 0 else None}
            del model
        except Exception as e:  # the baseline is a reported extra; never lose the GPU line over it
            cpu = {"value": None, "unit": UNIT, "cores": None, "kind": "port", "sample": f"failed: {e!r}"}

    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * dev_s_max / max(1, args.steps), "higher_is_better": True,
        "scaling": ("strong" if (tp > 1 and groups == 1) else "weak"),
        "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": workload_config(args, world, "B200"),
        "e2e": {"value": e2e, "unit": UNIT, "h2d_bytes_per_step": steps[0]["h2d"], "d2h_bytes_per_step": steps[0]["d2h"],
                "ms_per_step": 1e3 * wall_s_max / max(1, args.steps)},
        "gpu_launches": launches_all,
        "forwards_per_s": fwd_all / dev_s_max / max(1, groups),
        "iterations": {"forwards_total": fwd_all, "tokens_total": toks_all,
                       "iters_per_token": fwd_all / max(1.0, toks_all) * (B if B > 0 else 1) / B,
                       "tokens_per_forward_per_seq": toks_all / max(1.0, fwd_all) / B / 1.0,
                       "iters_per_block_mean": (sum(sum(s["iters_per_seq"]) for s in steps) /
                                                max(1.0, toks / float(n))),
                       "rows_per_forward": mean_rows, "stop": steps[-1]["stop"][:4]},
        "prefill_ms_per_step": sum(s["prefill_ms"] for s in steps) / max(1, len(steps)),
        "roofline": roofline, "cpu_baseline": cpu, "clocks": clocks,
        "timed_region_wall_s": t_total,
    }
    if tp_check is not None:
        line["tp_check"] = tp_check
    print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def run_compare_hybrid(args):
    """Option --compare-hybrid: the layered hybrid decoder beside the closest existing model (Qwen2) at equal width, depth
    and feed-forward size; device times from CUDA events, three warm-up passes, weights + activations larger than L2."""
    import __graft_entry__ as g
    g.build()
    from jacobiforcing_b200 import hybrid_bench as hb
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            mp = json.load(f)
        peaks = {"hbm_gbs": float(mp["hbm_gbs"]), "bf16_tflops": float(mp["bf16_tflops"]), "source": "measured"}
    except Exception:
        peaks = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "source": "fallback"}
    mon = ClockSampler(0)
    mon.start()
    res = []
    for size in args.compare_hybrid.split(","):
        row = {"size": size}
        row["hybrid"] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks)
        row["qwen2"] = hb.run_qwen2(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks)
        res.append(row)
    clocks = mon.stop()
    print(json.dumps({"metric": "hybrid_vs_qwen2_throughput", "unit": "tokens/s", "dtype": "bf16", "data": "synthetic",
                      "peaks": peaks, "clocks": clocks, "results": res}))


def run_compare_famepel(args):
    """Option --compare-famepel: Famepel (recurrence / gated recurrence / latent attention layers, routed experts) beside
    the closest existing model, the Kinetar hybrid decoder, at equal width, depth and active feed-forward size; device
    times from CUDA events, three warm-up passes, weights + activations larger than L2."""
    import __graft_entry__ as g
    g.build()
    from jacobiforcing_b200 import hybrid_bench as hb
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            mp = json.load(f)
        peaks = {"hbm_gbs": float(mp["hbm_gbs"]), "bf16_tflops": float(mp["bf16_tflops"]), "source": "measured"}
    except Exception:
        peaks = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "source": "fallback"}
    mon = ClockSampler(0)
    mon.start()
    res = []
    for size in args.compare_famepel.split(","):
        row = {"size": size}
        row["famepel"] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks, design="Famepel")
        row["kinetar"] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks)
        res.append(row)
    clocks = mon.stop()
    print(json.dumps({"metric": "famepel_vs_kinetar_throughput", "unit": "tokens/s", "dtype": "bf16", "data": "synthetic",
                      "peaks": peaks, "clocks": clocks, "results": res}))


def run_compare_vosolorn(args):
    """Option --compare-vosolorn: Vosolorn (matrix memory / window attention with pooled blocks, gated dense feed-forward
    and expert mixture) beside the closest existing model, Famepel, at equal width and depth; device times from CUDA
    events, three warm-up passes, weights + activations larger than L2."""
    import __graft_entry__ as g
    g.build()
    from jacobiforcing_b200 import hybrid_bench as hb
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            mp = json.load(f)
        peaks = {"hbm_gbs": float(mp["hbm_gbs"]), "bf16_tflops": float(mp["bf16_tflops"]), "source": "measured"}
    except Exception:
        peaks = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "source": "fallback"}
    mon = ClockSampler(0)
    mon.start()
    res = []
    for size in args.compare_vosolorn.split(","):
        row = {"size": size}
        row["vosolorn"] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks, design="Vosolorn")
        row["famepel"] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks, design="Famepel")
        res.append(row)
    clocks = mon.stop()
    print(json.dumps({"metric": "vosolorn_vs_famepel_throughput", "unit": "tokens/s", "dtype": "bf16", "data": "synthetic",
                      "peaks": peaks, "clocks": clocks, "results": res}))


def run_compare_sebavik(args):
    """Option --compare-sebavik: Sebavik (pre-norm blocks with input convolutions, biased attention over a window plus kept
    first tokens, clamped gated dense feed-forward and gated experts) beside the closest existing model, Vosolorn with
    attention in every layer, at equal width, depth, heads and feed-forward size; device times from CUDA events, three
    warm-up passes, weights + activations larger than L2."""
    import __graft_entry__ as g
    g.build()
    from jacobiforcing_b200 import hybrid_bench as hb
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            mp = json.load(f)
        peaks = {"hbm_gbs": float(mp["hbm_gbs"]), "bf16_tflops": float(mp["bf16_tflops"]), "source": "measured"}
    except Exception:
        peaks = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "source": "fallback"}
    mon = ClockSampler(0)
    mon.start()
    res = []
    for size in args.compare_sebavik.split(","):
        row = {"size": size}
        row["sebavik"] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks, design="Sebavik")
        row["vosolorn_attention"] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks,
                                                  design="VosolornAttention")
        res.append(row)
    clocks = mon.stop()
    print(json.dumps({"metric": "sebavik_vs_vosolorn_throughput", "unit": "tokens/s", "dtype": "bf16", "data": "synthetic",
                      "peaks": peaks, "clocks": clocks, "results": res}))


def run_compare_kisadra(args):
    """Option --compare-kisadra: Kisadra (gated linear attention / chunk attention / latent attention beside a gated dense or an
    expert feed-forward on one norm, a repeated layer) beside the closest existing models, Famepel and Sebavik, at equal width,
    layer runs, heads and active feed-forward size; device times from CUDA events, three warm-up passes, weights + activations
    larger than L2."""
    import __graft_entry__ as g
    g.build()
    from jacobiforcing_b200 import hybrid_bench as hb
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            mp = json.load(f)
        peaks = {"hbm_gbs": float(mp["hbm_gbs"]), "bf16_tflops": float(mp["bf16_tflops"]), "source": "measured"}
    except Exception:
        peaks = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "source": "fallback"}
    mon = ClockSampler(0)
    mon.start()
    res = []
    for size in args.compare_kisadra.split(","):
        row = {"size": size}
        for design in ("Kisadra", "Famepel", "Sebavik"):
            row[design.lower()] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks, design=design)
        res.append(row)
    clocks = mon.stop()
    print(json.dumps({"metric": "kisadra_vs_famepel_and_sebavik_throughput", "unit": "tokens/s", "dtype": "bf16", "data": "synthetic",
                      "peaks": peaks, "clocks": clocks, "results": res}))


def run_compare_mafalorn(args):
    """Option --compare-mafalorn: Mafalorn (retention / attention beside a delta rule / windowed latent attention, experts in every
    layer) beside the closest existing models, Kisadra and Kinetar, at equal width, layer runs, heads and active feed-forward
    size; device times from CUDA events, three warm-up passes, weights + activations larger than L2."""
    import __graft_entry__ as g
    g.build()
    from jacobiforcing_b200 import hybrid_bench as hb
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            mp = json.load(f)
        peaks = {"hbm_gbs": float(mp["hbm_gbs"]), "bf16_tflops": float(mp["bf16_tflops"]), "source": "measured"}
    except Exception:
        peaks = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0, "source": "fallback"}
    mon = ClockSampler(0)
    mon.start()
    res = []
    for size in args.compare_mafalorn.split(","):
        row = {"size": size}
        for design in ("Mafalorn", "Kisadra", "Kinetar"):
            row[design.lower()] = hb.run_hybrid(size, args.hybrid_prompt, args.hybrid_decode_steps, [1, 8], peaks, design=design)
        res.append(row)
    clocks = mon.stop()
    print(json.dumps({"metric": "mafalorn_vs_kisadra_and_kinetar_throughput", "unit": "tokens/s", "dtype": "bf16", "data": "synthetic",
                      "peaks": peaks, "clocks": clocks, "results": res}))


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--model", default="qwen2.5-coder-7b", choices=sorted(SHAPES))
    ap.add_argument("--mode", default="single", choices=["single", "multiblock"])
    ap.add_argument("--n", "--block-size", dest="n", type=int, default=32,
                    help="Jacobi block size (under torchrun spell it --block-size: the launcher's parser claims --n)")
    ap.add_argument("--K", type=int, default=2)
    ap.add_argument("--r", type=float, default=0.85)
    ap.add_argument("--pool", type=int, default=4)
    ap.add_argument("--batch", type=int, default=1)
    ap.add_argument("--prompt", type=int, default=512)
    ap.add_argument("--gen", type=int, default=512)
    ap.add_argument("--ref-budget-s", type=float, default=12.0)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--attn-chunk", type=int, default=64, help="keys per attention work unit (multiple of 64)")
    ap.add_argument("--tp", type=int, default=0, help="tensor-parallel group size (1, 2, 4, 8); default (0) = all N GPUs in one group")
    ap.add_argument("--replicas", action="store_true", help="N independent engines instead of tensor parallelism")
    ap.add_argument("--tp-attn", default="auto", choices=["auto", "shard", "replicate"],
                    help="attention block under tensor parallelism: sharded by heads (must divide tp), replicated on "
                         "every rank (MLP-only TP, one exchange per block), or auto = shard when the heads divide")
    ap.add_argument("--compare-hybrid", default="", metavar="SIZES",
                    help="instead of the headline workload: prefill / decode throughput of the layered hybrid decoder "
                         "(Kinetar) beside Qwen2 at equal size, e.g. w1024,w2048,w4096 (one JSON line)")
    ap.add_argument("--compare-famepel", default="", metavar="SIZES",
                    help="instead of the headline workload: prefill / decode throughput of Famepel beside the Kinetar hybrid "
                         "decoder at equal size, e.g. w1024,w2048 (one JSON line)")
    ap.add_argument("--compare-vosolorn", default="", metavar="SIZES",
                    help="instead of the headline workload: prefill / decode throughput of Vosolorn beside Famepel at equal "
                         "size, e.g. w1024,w2048 (one JSON line)")
    ap.add_argument("--compare-sebavik", default="", metavar="SIZES",
                    help="instead of the headline workload: prefill / decode throughput of Sebavik beside Vosolorn (attention "
                         "in every layer) at equal size, e.g. w1024,w2048 (one JSON line)")
    ap.add_argument("--compare-kisadra", default="", metavar="SIZES",
                    help="instead of the headline workload: prefill / decode throughput of Kisadra beside Famepel and Sebavik at "
                         "equal size, e.g. w1024,w2048 (one JSON line)")
    ap.add_argument("--compare-mafalorn", default="", metavar="SIZES",
                    help="instead of the headline workload: prefill / decode throughput of Mafalorn beside Kisadra and Kinetar at "
                         "equal size, e.g. w1024,w2048 (one JSON line)")
    ap.add_argument("--hybrid-prompt", type=int, default=4096)
    ap.add_argument("--hybrid-decode-steps", type=int, default=35)
    args = ap.parse_args()
    if args.compare_hybrid:
        run_compare_hybrid(args)
        return
    if args.compare_famepel:
        run_compare_famepel(args)
        return
    if args.compare_vosolorn:
        run_compare_vosolorn(args)
        return
    if args.compare_sebavik:
        run_compare_sebavik(args)
        return
    if args.compare_kisadra:
        run_compare_kisadra(args)
        return
    if args.compare_mafalorn:
        run_compare_mafalorn(args)
        return
    if args.warmup < 3 and args.impl == "ours":
        args.warmup = 3                                  # timing rule: at least three warm-up steps
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    if args.impl == "reference":
        run_reference(args, rank)
        return
    run_ours(args, rank, local_rank, world)


if __name__ == "__main__":
    main()
