"""Benchmark of the sparse-attention decode path (one layer, one decode step per "step").

    python bench.py [--gpus N] [--steps K] [--warmup W] [--workload c3|c2|c4|radapel|timalorn] [--impl reference]

Default workload: the 128K long-context configuration (`c3`: batch 4, 32 query / 8 KV heads,
context 131072, top-k 2048 + 64 + 256).  With N > 1 GPUs its 8 KV heads are split over the ranks
(8/N KV heads and 32/N query heads per GPU, the split GPT-FAST/tp.py:124-137,143-148 makes), so
the run is strong scaling: every rank works on the same decode step and the slowest rank sets the
step time.  The 32K configuration (`c2`) is measured in the same process and reported inside the
same JSON line under "c2".

A step = append+hash one new token, soft-hash the query, score every cached key, select the
top-k plus sink/window, sparse attention over the selected rows — the body of the reference's
`Attention.sparse_forward` between the QKV projection and the output projection.  Inputs are
seeded synthetic tensors with the benchmark configuration's shapes and distributions.

Printed JSON (one line, rank 0):
  value / ms_per_step   whole-job tokens/s per layer, inputs resident in HBM, each step one CUDA
                        graph launch timed with CUDA events; L2 is flushed between steps
  e2e                   the same step through the public host-memory API
                        (`SocketAttention.host_decoder`): q/k/v/position in pinned HOST memory, one
                        copy in, the step, the output copied back to pinned host memory
  roofline              the dominant kernel: algorithmic bytes / measured launch time
  stages                every kernel's time and achieved GB/s, and the whole step's
  cpu_baseline          the CPU restatement of the reference path on this box's host cores
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import threading
import time

import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from socket_b200.config import PRESETS  # noqa: E402

METRIC = "sparse_attn_decode_tokens_per_s"
UNIT = "tokens/s/layer"
FALLBACK_HBM_GBS = 6650.0



def ncu_traffic(kernel: str, workload: str):
    """DRAM bytes per launch (dram__bytes_read.sum + dram__bytes_write.sum) of `kernel` at `workload`
    from the ncu captures summarised under profiles/ (profiles/ncu_traffic.json, written next to the
    summaries); None where no capture of that kernel/workload exists."""
    try:
        table = json.load(open(os.path.join(ROOT, "profiles", "ncu_traffic.json")))
        return table.get(workload, {}).get(kernel)
    except Exception:
        return None


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=1000)
    ap.add_argument("--warmup", type=int, default=20)
    ap.add_argument("--workload", default="c3", choices=sorted(PRESETS) + ["c4", "c4-128k", "c4-128k-b4", "c5", "radapel", "timalorn"],
                    help="c1-c3: one attention layer (op level); c4 / c5: whole-model greedy decode, "
                         "Llama-3-8B / Llama-3-70B shape with random weights; radapel: the Radapel decoder "
                         "beside the Transformer, and its kernels one by one; timalorn: the Timalorn decoder beside "
                         "Radapel, the same way")
    ap.add_argument("--model-record", default="auto", choices=["auto", "on", "off"],
                    help="also run the whole-model decode comparison (c4) and attach it to the line; "
                         "auto = on a single GPU only")
    ap.add_argument("--model-tokens", type=int, default=64, help="decode tokens timed per mode by the attached c4 record")
    ap.add_argument("--secondary", default="c2", choices=sorted(PRESETS) + ["none"],
                    help="second workload measured in the same process and reported under its own key")
    ap.add_argument("--impl", default="socket_b200", choices=["socket_b200", "reference"])
    ap.add_argument("--shard", default="strong", choices=["weak", "strong"],
                    help="N>1: strong = the workload's KV heads are split over the GPUs (the reference's "
                         "tensor-parallel split); weak = every GPU owns a full copy of the workload")
    ap.add_argument("--shard-of", type=int, default=1,
                    help="single GPU only: run ONE rank's share of an N-way KV-head split (the per-rank shape of "
                         "the N-GPU run), for kernel work without N GPUs; the line says so in config.parallelism")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-flush", action="store_true")
    ap.add_argument("--skip-stages", action="store_true", help="skip the per-kernel timing loops")
    ap.add_argument("--skip-e2e", action="store_true", help="skip the host-buffer end-to-end loop")
    ap.add_argument("--select-path", default="auto", choices=["auto", "two_launch", "filter", "filter_f32", "filter_packed", "cluster"],
                    help="pin how the step builds its list (default: the library's own choice)")
    ap.add_argument("--seed", type=int, default=1234)
    return ap.parse_args()


def peak_hbm():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        try:
            return float(json.load(open(path))["hbm_gbs"]), "measured"
        except Exception:
            pass
    return FALLBACK_HBM_GBS, "fallback"


class ClockSampler:
    """nvidia-smi clocks and throttle reasons of one GPU, sampled every 200 ms."""
    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.rows = []
        self.proc = None
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--id={index}", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                 "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([x.strip() for x in line.split(",")])

    def stop(self):
        if self.proc is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except Exception:
            self.proc.kill()
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for r in self.rows:
            try:
                sm.append(float(r[0]))
                mx = float(r[1])
                for n, v in zip(names, r[3:7]):
                    if v.lower().startswith("active"):
                        reasons.add(n)
            except Exception:
                continue
        sm.sort()
        return {"sm_mhz": sm[len(sm) // 2] if sm else None, "sm_max_mhz": mx,
                "reasons": sorted(reasons), "samples": len(sm)}


# ------------------------------------------------------------------------------------------
def cpu_reference_steps(cfg, state, n_steps_cap=50, budget_s=12.0):
    """Times the CPU restatement of the reference path (oracle/c) on the host cores: per step
    hash the new key, soft-hash the query, score, select + list, sparse attention."""
    from oracle import c_oracle
    k, v, codes, vnorm, planes, protos, q_all, k_all, v_all = state
    B, Hkv, Tcap, D = k.shape
    T0 = cfg.context
    cores = c_oracle.num_threads()
    times = []
    t_begin = time.perf_counter()
    for i in range(n_steps_cap):
        t0 = time.perf_counter()
        pos = T0 + i
        kn = k_all[i][:, 0]                    # [B,Hkv,D]
        vn_ = v_all[i][:, 0]
        k[:, :, pos] = kn
        v[:, :, pos] = vn_
        codes[:, :, pos] = c_oracle.hash_keys(kn.contiguous(), planes, exact=False).to(torch.uint8)
        vnorm[:, :, pos] = c_oracle.value_norm(vn_.contiguous())
        T = pos + 1
        qp = c_oracle.soft_hash(q_all[i], planes, protos)
        sc = c_oracle.score(qp, codes, vnorm, T)
        lst, ln = c_oracle.select_list(sc, cfg.sink, cfg.window, cfg.topk, sorted_by_score=True)
        c_oracle.sparse_attention(q_all[i], k, v, lst, ln)
        times.append(time.perf_counter() - t0)
        if time.perf_counter() - t_begin > budget_s and len(times) >= 3:
            break
    use = times[1:] if len(times) > 1 else times
    per_step = sum(use) / len(use)
    return per_step, cores, len(times)


def host_state(cfg, seed, steps):
    """Host copies of the benchmark state for the CPU leg (same generator as the GPU leg's,
    drawn on the CPU)."""
    from oracle import c_oracle
    from socket_b200.synth import make_decode_inputs, make_step_inputs
    dt = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[cfg.kv_dtype]
    B, H, Hkv, T, D = cfg.batch, cfg.n_head, cfg.n_local_heads, cfg.context, cfg.head_dim
    dev = "cuda" if torch.cuda.is_available() else None
    inp = make_decode_inputs(B, H, Hkv, T, D=D, L=cfg.L, P=cfg.P, seed=seed, dtype=dt, device=dev)
    Tcap = T + steps + 8
    k = torch.zeros(B, Hkv, Tcap, D, dtype=dt)
    v = torch.zeros(B, Hkv, Tcap, D, dtype=dt)
    k[:, :, :T] = inp.k.cpu()
    v[:, :, :T] = inp.v.cpu()
    planes = inp.planes.cpu()
    codes = torch.zeros(B, Hkv, Tcap, cfg.L, dtype=torch.uint8)
    codes[:, :, :T] = c_oracle.hash_keys(k[:, :, :T].contiguous(), planes, exact=False).to(torch.uint8)
    vnorm = torch.zeros(B, Hkv, Tcap, dtype=torch.float16)
    vnorm[:, :, :T] = c_oracle.value_norm(v[:, :, :T].contiguous())
    q_all, k_all, v_all = make_step_inputs(B, H, Hkv, D, steps, seed + 1, dt)
    return (k, v, codes, vnorm, planes, inp.protos_T.cpu(), q_all, k_all, v_all)



def run_reference(args, cfg):
    """`--impl reference`: the reference path's CPU implementation on the host cores."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    n = max(1, min(args.steps, 50))
    state = host_state(cfg, args.seed, n + args.warmup)
    from oracle import c_oracle
    # all the host threads this process may use (torchrun exports OMP_NUM_THREADS=1 to its ranks)
    try:
        c_oracle.set_num_threads(len(os.sched_getaffinity(0)))
    except AttributeError:
        c_oracle.set_num_threads(os.cpu_count() or 1)
    per_step, cores, done = cpu_reference_steps(cfg, state, n_steps_cap=n + min(args.warmup, 3))
    val = cfg.batch / per_step
    sample = (f"{done} decode steps of workload {args.workload} (full context, all heads) with the C "
              f"restatement of the reference path, OpenMP over {cores} threads")
    line = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": UNIT, "n_gpus": args.gpus,
        "steps": done, "warmup": 1, "ms_per_step": per_step * 1e3, "higher_is_better": True,
        "scaling": "strong" if args.gpus > 1 else "weak", "vs_baseline": None, "dtype": cfg.kv_dtype,
        "data": "synthetic", "config": workload_config(args, args.workload, cfg, 1),
        "cpu_baseline": {"value": val, "unit": UNIT, "cores": cores, "kind": "port", "sample": sample},
        "e2e": {"value": val, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line))


def workload_config(args, wl, cfg, world):
    if world == 1 and getattr(args, "shard_of", 1) > 1:
        par = (f"single GPU running one rank's share of a {args.shard_of}-way KV-head split "
               f"({cfg.n_local_heads // args.shard_of} KV heads, {cfg.n_head // args.shard_of} query heads)")
    elif world == 1:
        par = "single GPU"
    elif args.shard == "strong":
        par = (f"{world} GPUs, the {cfg.n_local_heads} KV heads split {cfg.n_local_heads // world} per GPU "
               f"({cfg.n_head // world} query heads per GPU); no collective on the attention path")
    else:
        par = (f"{world} GPUs, each owning a full copy of the workload's {cfg.n_local_heads} KV-head groups "
               f"(no collective on the path)")
    return {
        "workload": f"{wl}: one layer, batch {cfg.batch}, {cfg.n_head} query / "
                    f"{cfg.n_local_heads} KV heads, head_dim {cfg.head_dim}, context {cfg.context}, "
                    f"{cfg.kv_dtype} KV, L={cfg.L} P={cfg.P}, top-k {cfg.topk} + sink {cfg.sink} + "
                    f"window {cfg.window}",
        "parallelism": par,
        "l2": "flushed between timed steps (256 MiB write)" if not args.no_flush else "not flushed",
        "timing": "per-step CUDA events around one CUDA-graph launch, summed over the steps",
    }


# ------------------------------------------------------------------------------------------
def measure(args, wl, K, W, world, rank, local_rank, full):
    """One workload on this rank's GPU: the timed decode loop, the per-kernel stages, the
    end-to-end loop through the host-memory entry.  `full` adds the bulk-hashing and dense
    comparison stages.  Returns the fields of the JSON line that belong to the workload."""
    from socket_b200 import ops
    from socket_b200.attention import SocketAttention
    from socket_b200.synth import make_decode_inputs, make_step_inputs

    cfg_full = PRESETS[wl]
    split = world > 1 and args.shard == "strong"
    if split and cfg_full.n_local_heads % world != 0:
        raise SystemExit(f"{cfg_full.n_local_heads} KV heads do not split over {world} GPUs")
    cfg = cfg_full.shard_kv_heads(world) if split else cfg_full
    if world == 1 and args.shard_of > 1:
        cfg = cfg_full.shard_kv_heads(args.shard_of)
    dev = torch.device("cuda", local_rank)

    dt = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}[cfg.kv_dtype]
    B, H, Hkv, T0, D = cfg.batch, cfg.n_head, cfg.n_local_heads, cfg.context, cfg.head_dim
    total_steps = K + W
    Tcap = T0 + 2 * total_steps + 64
    inp = make_decode_inputs(B, H, Hkv, T0, D=D, L=cfg.L, P=cfg.P, seed=args.seed + rank, dtype=dt, device=dev)
    attn = SocketAttention(H, Hkv, D, L=cfg.L, P=cfg.P, heavy_const=cfg.topk, sink_size=cfg.sink,
                           window_size=cfg.window, planes=inp.planes, protos_T=inp.protos_T, dtype=dt,
                           device=dev)
    cache = attn.setup_cache(B, Tcap, dtype=dt)
    k_bshd = inp.k.permute(0, 2, 1, 3)
    v_bshd = inp.v.permute(0, 2, 1, 3)
    for s0 in range(0, T0, 8192):
        s1 = min(T0, s0 + 8192)
        cache.append(torch.arange(s0, s1, device=dev), k_bshd[:, s0:s1].contiguous(),
                     v_bshd[:, s0:s1].contiguous(), attn.planes)
    del inp, k_bshd, v_bshd
    q_all, k_all, v_all = make_step_inputs(B, H, Hkv, D, total_steps, args.seed + 1000 + rank, dt, device=dev)

    # staging buffers the captured step reads from
    q_s = torch.empty(B, H, D, dtype=dt, device=dev)
    k_s = torch.empty(B, 1, Hkv, D, dtype=dt, device=dev)
    v_s = torch.empty(B, 1, Hkv, D, dtype=dt, device=dev)
    pos_s = torch.zeros(1, dtype=torch.int64, device=dev)
    out = torch.empty(B, H, D, dtype=dt, device=dev)
    step = ops.DecodeStep(cache, q_s, k_s, v_s, pos_s, attn.planes, attn.protos_T, out, topk=cfg.topk,
                          sink=cfg.sink, window=cfg.window, T_max=Tcap, select_path=args.select_path)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)

    def stage(i, pos):
        q_s.copy_(q_all[i])
        k_s.copy_(k_all[i])
        v_s.copy_(v_all[i])
        pos_s.fill_(pos)

    side = torch.cuda.Stream(dev)
    with torch.cuda.stream(side):
        stage(0, T0)
        step.run()                       # also sets the kernels' shared-memory attributes
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            step.run()
    torch.cuda.synchronize()

    def timed_loop(n, first, launch):
        evs = []
        for i in range(n):
            stage(first + i, T0 + first + i)
            if not args.no_flush:
                flush.fill_(i & 0xff)
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record()
            launch()
            e1.record()
            evs.append((e0, e1))
        torch.cuda.synchronize()
        return [a.elapsed_time(b) for a, b in evs]

    timed_loop(W, 0, graph.replay)
    sampler = ClockSampler(local_rank) if rank == 0 else None
    if world > 1:
        torch.distributed.barrier()
    torch.cuda.synchronize()
    per_step_ms = timed_loop(K, W, graph.replay)
    torch.cuda.synchronize()
    if world > 1:
        torch.distributed.barrier()
    total_ms = sum(per_step_ms)
    t = torch.tensor([total_ms], dtype=torch.float64, device=dev)
    if world > 1:
        torch.distributed.all_reduce(t, op=torch.distributed.ReduceOp.MAX)
    total_ms = float(t.item())
    if sampler is not None:
        # a short timed region can end before nvidia-smi's first 200 ms tick: keep the same load
        # running (untimed) until two samples exist, so the clocks are those under this load
        t_wait = time.perf_counter()
        while len(sampler.rows) < 2 and time.perf_counter() - t_wait < 2.0:
            for _ in range(50):
                graph.replay()
            torch.cuda.synchronize()
    clocks = sampler.stop() if sampler is not None else None
    assert int(step.status) == 0, f"device status {int(step.status)}"
    # split: all ranks work on the same B tokens; replicas: every rank has its own B tokens
    tokens = B * K * (1 if (split or world == 1) else world)
    value = tokens / (total_ms * 1e-3)
    ms_per_step = total_ms / K
    res = {"value": value, "ms_per_step": ms_per_step, "us_per_layer": ms_per_step * 1e3,
           "dtype": cfg.kv_dtype, "config": workload_config(args, wl, cfg_full, world), "clocks": clocks,
           "gpu_launches": K * step.n_launches, "roofline": None, "stages": {}, "e2e": None}

    # ---- per-kernel timing (same stream, same flush discipline) --------------------------
    T_now = T0 + total_steps
    peak, peak_src = peak_hbm()
    stages = {}
    a_codes = B * Hkv * T_now * cfg.L          # this GPU's share
    a_kv = B * H * cfg.ktot * 2 * D * cfg.kv_bytes()

    REP = 8

    def time_kernel(fn, n=20):
        """Per-kernel time without launch overhead in the bracket: a CUDA graph holding REP x
        (L2 flush, kernel) is timed against a graph holding REP x (L2 flush) and the difference
        is divided by REP."""
        def build(with_fn):
            with torch.cuda.stream(side):
                fn()
                side.synchronize()
                g = torch.cuda.CUDAGraph()
                with torch.cuda.graph(g, stream=side):
                    for r in range(REP):
                        if not args.no_flush:
                            flush.fill_(r)
                        if with_fn:
                            fn()
            torch.cuda.synchronize()
            return g

        def run(g):
            ts = []
            for i in range(n + 2):
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record()
                g.replay()
                e1.record()
                ts.append((e0, e1))
            torch.cuda.synchronize()
            v = sorted(a.elapsed_time(b) for a, b in ts[2:])
            return v[len(v) // 2] * 1e3
        return max(0.0, (run(build(True)) - run(build(False))) / REP)    # us

    us = {}
    if args.skip_stages:
        res["rescored_rows"] = step.rescored_rows()
        res["select_stats"] = step.select_stats()
        return res
    from socket_b200._lib import lib, ptr, stream_ptr
    probs, lut = ops.soft_hash(q_s, attn.planes, attn.protos_T, 1.0, n_kv_heads=Hkv, want_probs=False,
                               want_lut=True)
    fused = ops.score_select_applicable(B, H, Hkv, cfg.L, cfg.R, T_now, cfg.topk)
    us["kv_append"] = time_kernel(lambda: cache.append(pos_s, k_s, v_s, attn.planes))
    us["soft_hash"] = time_kernel(lambda: ops.soft_hash(q_s, attn.planes, attn.protos_T, 1.0, n_kv_heads=Hkv,
                                                        want_probs=False, want_lut=True))
    cluster = ops.score_select_cluster_size(B, H, Hkv, cfg.L, cfg.R, Tcap, cfg.topk)
    use_cluster = step.n_launches == 3
    extra = {}
    extra_notes = {}
    if cluster and not use_cluster and full:
        # not the step's path for this shape, timed for comparison only
        lst_c, ln_c = ops.score_select_cluster(lut, cache.k_hard, cache.v_norm, H, T_now, cfg.topk, cfg.sink,
                                               cfg.window)
        extra["score_select_cluster"] = time_kernel(lambda: lib().sk_score_select_cluster(
            ptr(lut), ptr(cache.k_hard), ptr(cache.v_norm), B, H, Hkv, cfg.L, cfg.R, T_now, None, Tcap, cfg.topk,
            cfg.sink, cfg.window, ptr(lst_c), lst_c.shape[-1], ptr(ln_c), None, stream_ptr(dev)))
    if use_cluster:
        # the step's middle launch: scorer + exact select on clusters of `cluster` CTAs
        lst, ln = ops.score_select_cluster(lut, cache.k_hard, cache.v_norm, H, T_now, cfg.topk, cfg.sink,
                                           cfg.window)
        ktot = lst.shape[-1]
        us["score_select_cluster"] = time_kernel(lambda: lib().sk_score_select_cluster(
            ptr(lut), ptr(cache.k_hard), ptr(cache.v_norm), B, H, Hkv, cfg.L, cfg.R, T_now, None, Tcap, cfg.topk,
            cfg.sink, cfg.window, ptr(lst), ktot, ptr(ln), None, stream_ptr(dev)))
        score_name = select_name = "score_select_cluster"
    elif fused and (args.select_path == "filter_packed" or (
            args.select_path in ("auto", "filter") and ops.packed_preferred(B, H, Hkv, cfg.L, cfg.R, Tcap, cfg.topk))):
        # the step's middle launches: packed-table scan, then the bracketed exact select
        lut, packed = ops.soft_hash_packed(q_s, attn.planes, attn.protos_T, 1.0, n_kv_heads=Hkv)
        us["soft_hash"] = time_kernel(lambda: ops.soft_hash_packed(q_s, attn.planes, attn.protos_T, 1.0,
                                                                   n_kv_heads=Hkv))
        lst, ln, fws = ops.score_select_packed(lut, packed, cache.k_hard, cache.v_norm, H, T_now, cfg.topk,
                                               cfg.sink, cfg.window)
        ktot = lst.shape[-1]

        def packed_stage(stages):
            return lambda: lib().sk_score_select_packed(
                ptr(lut), ptr(packed), ptr(cache.k_hard), ptr(cache.v_norm), B, H, Hkv, cfg.L, cfg.R, T_now, None,
                Tcap, cfg.topk, cfg.sink, cfg.window, ptr(lst), ktot, ptr(ln), ptr(fws), fws.numel(), None, stages,
                stream_ptr(dev))
        us["score_filter"] = time_kernel(packed_stage(1))
        us["select_candidates"] = time_kernel(packed_stage(2))
        score_name, select_name = "score_filter", "select_candidates"
        extra_notes = {"score_filter": "packed 12-bit table scan (score_packed_kernel)",
                       "select_candidates": "bracketed exact select on packed candidates"}
    elif fused:
        lst, ln, fws = ops.score_select_list(lut, cache.k_hard, cache.v_norm, H, T_now, cfg.topk, cfg.sink,
                                             cfg.window)
        ktot = lst.shape[-1]
        common = (ptr(lut), ptr(cache.k_hard), ptr(cache.v_norm), B, H, Hkv, cfg.L, cfg.R, T_now, None, Tcap,
                  cfg.topk)
        us["score_filter"] = time_kernel(lambda: lib().sk_score_filter(
            *common, ptr(fws), fws.numel(), None, stream_ptr(dev)))
        us["select_candidates"] = time_kernel(lambda: lib().sk_select_candidates(
            *common, cfg.sink, cfg.window, ptr(lst), ktot, ptr(ln), ptr(fws), fws.numel(), None, stream_ptr(dev)))
        score_name, select_name = "score_filter", "select_candidates"
    else:
        scores = ops.score(lut, cache.k_hard, cache.v_norm, H, T_now)
        lst, ln = ops.select_list(scores, T_now, cfg.topk, cfg.sink, cfg.window)
        us["score"] = time_kernel(lambda: ops.score(lut, cache.k_hard, cache.v_norm, H, T_now, out=scores))
        us["select_list"] = time_kernel(lambda: ops.select_list(scores, T_now, cfg.topk, cfg.sink, cfg.window))
        score_name, select_name = "score", "select_list"
    us["sparse_decode"] = time_kernel(lambda: ops.sparse_decode(q_s, cache.k_cache, cache.v_cache, lst, ln, T=T_now))
    alg = {"kv_append": 0, "soft_hash": 0, select_name: 0, "sparse_decode": a_kv}
    alg[score_name] = a_codes
    for name, t_us in us.items():
        gbs = alg[name] / (t_us * 1e-6) / 1e9 if alg[name] else None
        stages[name] = {"us": round(t_us, 2), "algorithmic_bytes": alg[name],
                        "achieved_gbs": None if gbs is None else round(gbs, 1),
                        "frac_of_hbm_peak": None if gbs is None else round(gbs / peak, 4)}
        if name in extra_notes:
            stages[name]["note"] = extra_notes[name]
    # prefill hashing of the whole context on the tensor cores (not part of the decode step)
    if full and dt == torch.bfloat16 and D == 128 and cfg.L == 32 and cfg.P == 8:
        n_rows = B * Hkv * T0
        keys2d = cache.k_cache[:, :, :T0].reshape(-1, D)
        for _ in range(2):
            ops.hash_keys_tc(keys2d, attn.planes)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(5):
            ops.hash_keys_tc(keys2d, attn.planes)
        e1.record()
        torch.cuda.synchronize()
        t_us = e0.elapsed_time(e1) / 5 * 1e3
        flops = 2.0 * n_rows * D * cfg.L * cfg.P
        tf_peak = tf_sus = None
        try:
            peaks = json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
            tf_peak, tf_sus = float(peaks["bf16_tflops"]), float(peaks.get("bf16_tflops_sustained", 0)) or None
        except Exception:
            pass
        stages["prefill_hash_tc"] = {
            "us": round(t_us, 1), "rows": n_rows, "tflops": round(flops / t_us / 1e6, 1),
            "frac_of_bf16_peak": None if tf_peak is None else round(flops / t_us / 1e6 / tf_peak, 4),
            "frac_of_bf16_sustained": None if tf_sus is None else round(flops / t_us / 1e6 / tf_sus, 4),
            "gbs": round(n_rows * (D * 2 + cfg.L) / t_us / 1e3, 1),
            "note": "sk_hash_keys_tc; not in the step"}
        del keys2d
        # the whole prefill cache write (copy K/V + v_norm + codes) of S tokens; the tokens are the
        # cache's own first S rows, so the cache is left unchanged
        S_pf = min(T0, 8192)
        k_pf = cache.k_cache[:, :, :S_pf].transpose(1, 2).contiguous()
        v_pf = cache.v_cache[:, :, :S_pf].transpose(1, 2).contiguous()
        pos_pf = torch.arange(S_pf, device=dev, dtype=torch.int64)

        def _append():
            ops.kv_append(cache.k_cache, cache.v_cache, cache.k_hard, cache.v_norm, cache.prefill_len,
                          pos_pf, k_pf, v_pf, attn.planes)
        for _ in range(2):
            _append()
        e0.record()
        for _ in range(5):
            _append()
        e1.record()
        torch.cuda.synchronize()
        t_us = e0.elapsed_time(e1) / 5 * 1e3
        rows_pf = B * Hkv * S_pf
        bytes_pf = rows_pf * (4 * D * 2 + cfg.L + 2)      # K and V read + written, codes, v_norm
        stages["prefill_kv_append"] = {
            "us": round(t_us, 1), "rows": rows_pf, "gbs": round(bytes_pf / t_us / 1e3, 1),
            "frac_of_hbm_peak": round(bytes_pf / t_us / 1e3 / peak, 4),
            "note": "sk_kv_append: copies, norms and tensor-core hashing in one launch; not in the step"}
        del k_pf, v_pf
    # context figure, not on the path: dense attention of the same query over the whole cache
    # (library kernels), i.e. what the sparse path replaces per layer and token
    dense_bytes = 2 * B * Hkv * T_now * D * cfg.kv_bytes()
    if full:
        try:
            import torch.nn.functional as F
            qd = q_s.view(B, Hkv, H // Hkv, D)                         # the rep query heads of a KV head as "rows"
            kd, vd = cache.k_cache[:, :, :T_now], cache.v_cache[:, :, :T_now]
            t_dense = time_kernel(lambda: F.scaled_dot_product_attention(qd, kd, vd))
            stages["dense_attention_sdpa"] = {
                "us": round(t_dense, 2), "algorithmic_bytes": dense_bytes,
                "achieved_gbs": round(dense_bytes / (t_dense * 1e-6) / 1e9, 1),
                "note": "torch SDPA over the full context, for comparison; not on the step's path"}
        except Exception as e:  # a comparison figure must never cost the line
            stages["dense_attention_sdpa"] = {"us": None, "note": f"unavailable: {e!r}"[:200]}
    try:
        from flash_attn import flash_attn_with_kvcache           # split-KV dense decode, a library kernel
        qf = q_s.view(B, 1, H, D)
        kf, vf = cache.k_cache.transpose(1, 2), cache.v_cache.transpose(1, 2)      # [B, Tcap, Hkv, D] views
        lens = torch.full((B,), T_now, dtype=torch.int32, device=dev)
        t_fa = time_kernel(lambda: flash_attn_with_kvcache(qf, kf, vf, cache_seqlens=lens))
        stages["dense_attention_flash_decode"] = {
            "us": round(t_fa, 2), "algorithmic_bytes": dense_bytes,
            "achieved_gbs": round(dense_bytes / (t_fa * 1e-6) / 1e9, 1),
            "note": "flash_attn_with_kvcache over the full context, for comparison; not on the step's path"}
    except Exception as e:
        stages["dense_attention_flash_decode"] = {"us": None, "note": f"unavailable: {e!r}"[:200]}
    A = a_codes + a_kv
    step_gbs = A / (ms_per_step * 1e-3) / 1e9
    stages["whole_step"] = {"us": round(ms_per_step * 1e3, 2), "algorithmic_bytes": A,
                            "achieved_gbs": round(step_gbs, 1), "frac_of_hbm_peak": round(step_gbs / peak, 4),
                            "frac_of_8tbs": round(step_gbs / 8000.0, 4),
                            "note": "this GPU's share of the layer-step (its KV heads' codes + gathered rows)"}
    fa_us = stages.get("dense_attention_flash_decode", {}).get("us")
    if fa_us:
        stages["whole_step"]["speedup_vs_dense_flash_decode"] = round(fa_us / (ms_per_step * 1e3), 3)
    for name, t_us in extra.items():
        stages[name] = {"us": round(t_us, 2), "algorithmic_bytes": a_codes,
                        "achieved_gbs": round(a_codes / (t_us * 1e-6) / 1e9, 1), "note": "not on the step's path"}
    if cluster and "score_select_cluster" in stages:
        stages["score_select_cluster"]["cluster_size"] = cluster
    dominant = max((score_name, "sparse_decode", select_name), key=lambda n: us[n])
    dom_alg = alg[dominant] if alg[dominant] else A
    dom_gbs = dom_alg / (us[dominant] * 1e-6) / 1e9
    res["roofline"] = {"bound": "hbm", "kernel": dominant, "achieved": round(dom_gbs, 1), "peak": peak,
                       "unit": "GB/s", "frac": round(dom_gbs / peak, 4), "peak_source": peak_src,
                       "traffic": ncu_traffic(dominant, wl) if world == 1 else None,
                       "per": "GPU" if world > 1 else "launch",
                       "whole_step_frac": round(step_gbs / peak, 4)}
    if dominant == "score_filter":
        # The scan's binding unit is not HBM but the SM's shared-memory data pipe: one table lookup per
        # (key, table) serves the 4 query heads of a KV head and moves 8 bytes per lane with the packed
        # table (2 wavefronts of 128 B per warp), 16 bytes with the fp32 table (4 wavefronts); an SM
        # passes one wavefront per cycle.  The floor below is that count at the SM clock sampled during
        # the run; it explains the HBM fraction above and is reported beside it.
        packed_scan = bool(extra_notes.get("score_filter", "").startswith("packed"))
        ht = 4 if (H // Hkv) % 4 == 0 else (2 if (H // Hkv) % 2 == 0 else 1)
        lookups = B * Hkv * ((H // Hkv) // ht) * T_now * cfg.L
        wavefronts = lookups / 32 * (2 if packed_scan else ht)
        mhz = (clocks or {}).get("sm_mhz") or (clocks or {}).get("sm_max_mhz") or 1965.0
        n_sm = torch.cuda.get_device_properties(dev).multi_processor_count
        floor_us = wavefronts / n_sm / mhz
        res["roofline"]["shared_memory_pipe"] = {
            "table": "packed 8 B per lookup" if packed_scan else f"fp32 {4 * ht} B per lookup",
            "wavefronts_per_launch": int(wavefronts), "sm_mhz": mhz, "floor_us": round(floor_us, 2),
            "frac": round(floor_us / us[dominant], 4),
            "note": "lookup wavefronts / (SMs x clock) over the kernel's time: the on-chip bound of the scan"}
    if world > 1:
        # the one collective that follows the path under tensor parallelism: the sum of the
        # row-sharded output projection, [B, 1, d_model] bf16 (d_model = all query heads x head_dim)
        from socket_b200 import tp
        y = torch.zeros(B, 1, cfg_full.n_head * D, dtype=torch.bfloat16, device=dev)
        for _ in range(5):
            tp.all_reduce_sum(y)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(50):
            tp.all_reduce_sum(y)
        e1.record()
        torch.cuda.synchronize()
        ar = torch.tensor([e0.elapsed_time(e1) / 50 * 1e3], dtype=torch.float64, device=dev)
        torch.distributed.all_reduce(ar, op=torch.distributed.ReduceOp.MAX)
        stages["tp_all_reduce"] = {"us": round(float(ar.item()), 2), "bytes": y.numel() * 2,
                                   "note": "NCCL all-reduce of the output projection's partial sums; follows "
                                           "the path under tensor parallelism, not inside the timed step"}
    res["stages"] = stages

    # ---- end to end through the public API with host buffers -----------------------------
    if args.skip_e2e:
        res["rescored_rows"] = step.rescored_rows()
        return res
    n_e2e = min(K, 200)
    # the public host-memory entry: one pinned staging block -> device, the step, the output back
    # to pinned memory, replayed as one graph.  Each step's inputs wait in pinned host memory in the
    # staging block's layout and are copied into it inside the timed region.
    hd = attn.host_decoder(B)
    packed = torch.zeros(n_e2e + 3, hd.h_in.numel(), dtype=torch.uint8).pin_memory()
    nq, nkv = hd.h_q.numel() * hd.h_q.element_size(), hd.h_k.numel() * hd.h_k.element_size()
    for i in range(n_e2e + 3):
        packed[i, :8].view(torch.int64)[0] = T_now + i
        packed[i, 16:16 + nq].view(dt).copy_(q_all[i].reshape(-1))
        packed[i, 16 + nq:16 + nq + nkv].view(dt).copy_(k_all[i].reshape(-1))
        packed[i, 16 + nq + nkv:].view(dt).copy_(v_all[i].reshape(-1))
    e2e_ms = []
    for i in range(n_e2e + 3):
        if not args.no_flush:
            flush.fill_(i & 0xff)
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        hd.stage(packed[i])
        hd.launch()
        e1.record()
        hd.wait()
        e1.synchronize()
        if i >= 3:
            e2e_ms.append(e0.elapsed_time(e1))
    e2e_t = torch.tensor([sum(e2e_ms) / len(e2e_ms)], dtype=torch.float64, device=dev)
    if world > 1:
        torch.distributed.all_reduce(e2e_t, op=torch.distributed.ReduceOp.MAX)
    e2e_ms_step = float(e2e_t.item())
    res["e2e"] = {"value": B * (1 if (split or world == 1) else world) / (e2e_ms_step * 1e-3), "unit": UNIT,
                  "h2d_bytes_per_step": hd.h2d_bytes, "d2h_bytes_per_step": hd.d2h_bytes,
                  "ms_per_step": e2e_ms_step, "steps": len(e2e_ms)}
    res["rescored_rows"] = step.rescored_rows()
    res["select_stats"] = step.select_stats()
    return res


MODEL_WORKLOADS = {
    # name: (architecture, batch, prompt tokens, new tokens of the full configuration, sparse overrides)
    "c4": ("llama-3-8b", 1, 32768, 256, {}),
    # the same model at the long-context point the 1.5x target is stated on (sparse parameters of c3)
    "c4-128k": ("llama-3-8b", 1, 131072, 256, dict(heavy_const=2048, sink_size=64, window_size=256)),
    "c4-128k-b4": ("llama-3-8b", 4, 131072, 256, dict(heavy_const=2048, sink_size=64, window_size=256)),
    "c5": ("llama-3-70b", 8, 65536, 128, {}),
}


def measure_model(args, wl, K, W, world, rank, local_rank):
    """Whole-model greedy decode (the reference's `generate.py` flow): random bf16 weights of the
    named architecture, a prompt of uniform random token ids, prefill (causal flash attention +
    bulk hashing), then W untimed and K timed decode tokens, one CUDA graph per token - once with
    the SOCKET sparse step in every layer and once with dense split-KV flash decode over the whole
    cache.  tokens/s = batch * K / decode time (generate.py:362-368).  Under N > 1 the model is
    tensor-parallel (heads split as GPT-FAST/tp.py does, explicit all-reduce after `wo` and the
    feed-forward)."""
    from socket_b200.model import ModelArgs, Transformer
    arch, B, T, _, over = MODEL_WORKLOADS[wl]
    dev = torch.device("cuda", local_rank)
    cfg = ModelArgs.from_name(arch, **over)
    old = torch.get_default_dtype()
    torch.set_default_dtype(torch.bfloat16)
    try:
        with torch.device(dev):
            model = Transformer(cfg, world=world, rank=rank)
    finally:
        torch.set_default_dtype(old)
    model.init_random(seed=args.seed)
    g = torch.Generator().manual_seed(args.seed)
    prompt = torch.randint(0, cfg.vocab_size, (B, T), generator=g).pin_memory()
    n_new = W + K + 32 + 8                               # warm-up, timed and end-to-end tokens, spare
    out = {"architecture": arch, "batch": B, "prompt_tokens": T, "decode_tokens_timed": K, "warmup_tokens": W,
           "layers": cfg.n_layer, "tensor_parallel": world,
           "sparse": {"L": cfg.L, "P": cfg.K, "topk": cfg.heavy_const, "sink": cfg.sink_size, "window": cfg.window_size}}
    host_tok = torch.empty(B, 1, dtype=torch.long).pin_memory()
    # untimed: a short prefill so that neither mode's prefill time carries the libraries' first-call set-up
    model.setup_caches(B, T + n_new + 8)
    model.prefill(prompt[:, :min(T, 2048)].to(dev))
    torch.cuda.synchronize()
    for mode in ("sparse", "dense"):
        model.max_seq_length = -1                         # fresh caches per mode
        model.setup_caches(B, T + n_new + 8)
        model.setup_decode(B, mode)
        t0 = torch.cuda.Event(enable_timing=True); t1 = torch.cuda.Event(enable_timing=True)
        t0.record()
        logits = model.prefill(prompt.to(dev, non_blocking=True))
        first = torch.argmax(logits, dim=-1, keepdim=True)
        t1.record()
        model.start_decode(first, T)
        for _ in range(W):
            model.decode_one_token()
        if world > 1:
            torch.distributed.barrier()
        torch.cuda.synchronize()
        e0 = torch.cuda.Event(enable_timing=True); e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(K):
            model.decode_one_token()
        e1.record()
        torch.cuda.synchronize()
        if world > 1:
            torch.distributed.barrier()
        ms = torch.tensor([e0.elapsed_time(e1)], dtype=torch.float64, device=dev)
        if world > 1:
            torch.distributed.all_reduce(ms, op=torch.distributed.ReduceOp.MAX)
        ms = float(ms.item())
        rec = {"tokens_per_s": B * K / (ms * 1e-3), "ms_per_token": ms / K,
               "prefill_s": t0.elapsed_time(t1) / 1e3, "gpu_launches_per_token_path": 4 * cfg.n_layer if mode == "sparse" else 0}
        if mode == "sparse":
            # end to end: every token is copied to pinned host memory and waited for before the next launch
            n_e = min(K, 32)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(n_e):
                tok = model.decode_one_token()
                host_tok.copy_(tok, non_blocking=True)
                torch.cuda.current_stream(dev).synchronize()
            e1.record()
            torch.cuda.synchronize()
            rec["e2e_tokens_per_s"] = B * n_e / (e0.elapsed_time(e1) * 1e-3)
            rec["status"] = int(sum(int(l.attention.kv_cache.status) for l in model.layers))
            rec["rescored_rows"] = sum((l.attention._step.rescored_rows() or 0) for l in model.layers)
            agg = {}
            for l in model.layers:
                for k, v in (l.attention._step.select_stats() or {}).items():
                    agg[k] = agg.get(k, 0) + v
            rec["select_stats"] = agg
        out[mode] = rec
        for l in model.layers:                            # release this mode's scratch
            l.attention._step = None
    out["sparse_over_dense"] = out["sparse"]["tokens_per_s"] / out["dense"]["tokens_per_s"]
    del model
    torch.cuda.empty_cache()
    return out


# ------------------------------------------------------------------------------- Radapel
RADAPEL_SIZES = {
    # name: (width, query heads, KV heads, head size, feed-forward, latent rank, state-space heads)
    "2k": (2048, 16, 4, 128, 5632, 512, 64),
    "4k": (4096, 32, 8, 128, 14336, 512, 128),
}
RADAPEL_CHUNK, RADAPEL_ROT, RADAPEL_STATE = 8192, 64, 128


def radapel_config(size):
    """Two attention layers, one latent, one state-space layer; the last three run twice: 7 layer runs."""
    W, H, G, D, F, K, M = RADAPEL_SIZES[size]
    mlp = {"kind": "dense", "ff": F, "limit": 7.0}
    att = {"type": "attention", "mlp": mlp, "mixer": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5,
                                                       "bias_max": 1024, "mask": {"size": RADAPEL_CHUNK}}}
    lat = {"type": "latent_attention", "mlp": mlp,
           "mixer": {"heads": H, "dim": D, "rot_dim": RADAPEL_ROT, "vdim": D, "kv_rank": K, "scale": (D + RADAPEL_ROT) ** -0.5,
                     "rot": {"base": 500000.0, "dims": RADAPEL_ROT}}}
    ssm = {"type": "mamba2", "mlp": None, "mixer": {"heads": M, "vdim": 64, "state": RADAPEL_STATE, "groups": 8, "conv": 4,
                                                     "norm_groups": 8}}
    return {"architecture": "Radapel", "vocab": 32768, "width": W, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "layers": [att, att, lat, ssm], "loop": {"start": 1, "stop": 4, "times": 2}}


def measure_throughput(model, vocab, B, T, K, W, dev, mode=None):
    """Prefill and decode of one decoder: seconds of a prompt of T tokens (second run), ms per graph-replayed
    decode token after it, and the same with every token copied to pinned host memory."""
    model.max_seq_length = -1
    model.setup_caches(B, T + 2 * K + W + 16)
    model.setup_decode(B, mode)
    prompt = torch.randint(0, vocab, (B, T), generator=torch.Generator().manual_seed(5)).pin_memory()
    ev = lambda: torch.cuda.Event(enable_timing=True)  # noqa: E731
    for _ in range(2):
        t0, t1 = ev(), ev()
        torch.cuda.synchronize()
        t0.record()
        logits = model.prefill(prompt.to(dev, non_blocking=True))
        first = torch.argmax(logits, dim=-1, keepdim=True)
        t1.record()
        torch.cuda.synchronize()
    model.start_decode(first, T)
    for _ in range(W):
        model.decode_one_token()
    torch.cuda.synchronize()
    e0, e1, e2 = ev(), ev(), ev()
    e0.record()
    for _ in range(K):
        model.decode_one_token()
    e1.record()
    torch.cuda.synchronize()
    host = torch.empty(B, 1, dtype=torch.long).pin_memory()
    e1b = ev()
    e1b.record()
    for _ in range(K):
        host.copy_(model.decode_one_token(), non_blocking=True)
        torch.cuda.current_stream(dev).synchronize()
    e2.record()
    torch.cuda.synchronize()
    pre, ms, e2e = t0.elapsed_time(t1), e0.elapsed_time(e1) / K, e1b.elapsed_time(e2) / K
    return {"prefill_ms": pre, "prefill_tokens_per_s": B * T / pre * 1e3, "decode_ms_per_token": ms,
            "decode_tokens_per_s": B / ms * 1e3, "e2e_decode_tokens_per_s": B / e2e * 1e3}


def time_op(fn, flush, n=20):
    """Device microseconds of fn(): CUDA graphs of [flush L2, fn] against [flush L2]."""
    fn()
    torch.cuda.synchronize()

    def graph(with_fn):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            for _ in range(4):
                flush.fill_(1)
                if with_fn:
                    fn()
        return g

    times = []
    for g in (graph(True), graph(False)):
        for _ in range(3):
            g.replay()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        a.record()
        for _ in range(n):
            g.replay()
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) / (4 * n) * 1e3)
    return times[0] - times[1]


def kernel_table(peaks):
    """(rows, add): add(...) appends one kernel with its share of the roofline, beside a like kernel and its share."""
    rows = []

    def add(name, us, like, like_us, flops=0.0, nbytes=0.0, like_flops=None, like_bytes=None):
        def frac(t, f, b):
            return max(f / (peaks["bf16_tflops"] * 1e12), b / (peaks["hbm_gbs"] * 1e9)) / (t * 1e-6)
        r = {"kernel": name, "us": round(us, 2), "roofline_frac": round(frac(us, flops, nbytes), 3)}
        if flops:
            r["tflops"] = round(flops / us / 1e6, 1)
        if nbytes:
            r["gbs"] = round(nbytes / us / 1e3, 1)
        if like is not None:
            lf, lb = flops if like_flops is None else like_flops, nbytes if like_bytes is None else like_bytes
            r.update(like=like, like_us=round(like_us, 2), like_roofline_frac=round(frac(like_us, lf, lb), 3))
            r["like_frac_over_frac"] = round(r["like_roofline_frac"] / max(r["roofline_frac"], 1e-9), 2)
        rows.append(r)
    return rows, add


def measure_radapel_kernels(size, S, T, B, dev):
    """Every kernel of the design beside the like kernel of the Llama-shaped model, at one size: prefill
    kernels on S tokens from position 0, decode kernels for B sequences at context T."""
    import torch.nn.functional as F
    from flash_attn import flash_attn_func, flash_attn_with_kvcache
    from socket_b200 import block_ops as ops
    from socket_b200.mixers import LatentCache, Mamba2, Portion, rotary_angles  # noqa: F401
    from socket_b200.model import apply_rotary_emb
    W, H, G, D, FF, K, M = RADAPEL_SIZES[size]
    R, N, P = RADAPEL_ROT, RADAPEL_STATE, 64
    bf = torch.bfloat16
    rn = lambda *s: torch.randn(*s, device=dev, dtype=bf)  # noqa: E731
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    peaks = measured_peaks()
    rows, add = kernel_table(peaks)

    # ---- attention of a prompt
    q, k, v = rn(1, S, H, D), rn(1, S, G, D), rn(1, S, G, D)
    fa = time_op(lambda: flash_attn_func(q, k, v, causal=True), flush)
    pairs = S * (S + 1) / 2
    bias = torch.randn(H, 1025, device=dev)
    f = pairs * H * 4 * D
    add("chunked attention, prefill", time_op(lambda: ops.attn(q, k, v, scale=D ** -0.5, chunk=RADAPEL_CHUNK, bias=bias), flush),
        "flash_attn_func", fa, flops=f)
    ql, kl, vl = rn(1, S, H, D + R), rn(1, S, H, D + R), rn(1, S, H, D)
    sink = torch.randn(H, device=dev)
    add("latent attention, prefill (expanded)", time_op(lambda: ops.attn(ql, kl, vl, scale=0.07, sink=sink), flush),
        "flash_attn_func", fa, flops=pairs * H * 2 * (2 * D + R), like_flops=f)
    # ---- attention of a decoded token
    pos = torch.tensor([T - 1], device=dev)
    lens = torch.full((B,), T - 1, dtype=torch.int32, device=dev)
    q1, k1 = rn(B, 1, H, D), rn(B, 1, G, D)
    kc, vc = rn(B, T, G, D), rn(B, T, G, D)
    fad = time_op(lambda: flash_attn_with_kvcache(q1, kc, vc, k=k1, v=k1, cache_seqlens=lens, causal=True), flush)
    fab = B * T * G * 2 * D * 2
    C = min(T, RADAPEL_CHUNK)
    kr, vr = kc[:, :C].contiguous(), vc[:, :C].contiguous()
    ringpos = torch.tensor([C - 1], device=dev)
    lens_c = torch.full((B,), C - 1, dtype=torch.int32, device=dev)
    fac = time_op(lambda: flash_attn_with_kvcache(q1, kr, vr, k=k1, v=k1, cache_seqlens=lens_c, causal=True), flush)
    ws = torch.empty(64 << 20, dtype=torch.uint8, device=dev)
    add(f"chunked attention, decode (chunk {C} full)",
        time_op(lambda: ops.attn(q1, kr, vr, scale=D ** -0.5, pos=ringpos, chunk=C, ring=True, bias=bias, workspace=ws), flush),
        "flash_attn_with_kvcache, same cache", fac, nbytes=B * C * G * 2 * D * 2)
    cache = rn(B, T, K + R)
    qa = rn(B, 1, H, K + R)
    shared = cache.unsqueeze(2)
    lat_f = B * H * T * 2 * (2 * K + R)
    add("latent attention, decode", time_op(lambda: ops.attn(qa, shared, shared[..., :K], scale=0.07, pos=pos, sink=sink, workspace=ws), flush),
        "flash_attn_with_kvcache, same context", fad, nbytes=B * T * (K + R) * 2, flops=lat_f, like_bytes=fab, like_flops=0.0)
    # ---- latent up- and down-projections of a decoded token
    uk, uv = rn(H * D, K), rn(H * D, K)
    qd, o, ho = rn(B, H * (D + R)), rn(B, H, K), rn(B, K)
    gemv = time_op(lambda: torch.mm(ho, uv.t()), flush)
    wb = H * D * K * 2
    add("latent absorb, decode", time_op(lambda: ops.latent_absorb(qd, uk, H, D, R, K + R), flush), "torch.mm, as many bytes", gemv,
        nbytes=H * D * K * 2, like_bytes=wb)
    add("latent up, decode", time_op(lambda: ops.latent_up(o, uv, D), flush), "torch.mm, as many bytes", gemv, nbytes=H * D * K * 2, like_bytes=wb)
    # ---- residual stream
    x, y, w = torch.randn(S, W, device=dev), rn(S, W), rn(W)
    xb = rn(S, W)
    norm = time_op(lambda: F.rms_norm(xb + y, (W,), w, 1e-5), flush)
    add("residual + two norms, prefill", time_op(lambda: ops.residual_norm(x, 1e-5, y=y, w_in=w, w_out=w), flush),
        "add + F.rms_norm", norm, nbytes=S * W * 12, like_bytes=S * W * 8)
    x1, y1, xb1 = torch.randn(B, W, device=dev), rn(B, W), rn(B, W)
    norm1 = time_op(lambda: F.rms_norm(xb1 + y1, (W,), w, 1e-5), flush)
    add("residual + two norms, decode", time_op(lambda: ops.residual_norm(x1, 1e-5, y=y1, w_in=w, w_out=w), flush),
        "add + F.rms_norm", norm1, nbytes=B * W * 12 + 4 * W, like_bytes=B * W * 8 + 2 * W)
    gu = rn(S, 2 * FF)
    add("clamped unit, prefill", time_op(lambda: ops.glu_clamped(gu, FF, 7.0), flush), "silu * up",
        time_op(lambda: F.silu(gu[:, :FF]) * gu[:, FF:], flush), nbytes=S * FF * 6)
    gu1 = rn(B, 2 * FF)
    add("clamped unit, decode", time_op(lambda: ops.glu_clamped(gu1, FF, 7.0), flush), "silu * up",
        time_op(lambda: F.silu(gu1[:, :FF]) * gu1[:, FF:], flush), nbytes=B * FF * 6)
    # ---- latent rows of a prompt
    ang = rotary_angles(S, R, 500000.0, dev)
    dkv, qq, lw, lc = rn(S, K + R), rn(S, H * (D + R)), rn(K), rn(1, S, K + R)
    fc = torch.randn(S, D // 2, 2, device=dev).to(bf)
    add("latent append + rotation, prefill",
        time_op(lambda: ops.latent_append(dkv, qq, lw, ang, lc, S=S, n_heads=H, dim=D, rot=R, rank=K, eps=1e-5), flush),
        "apply_rotary_emb of q", time_op(lambda: apply_rotary_emb(q, fc), flush),
        nbytes=S * (4 * (K + R) + 4 * H * R), like_bytes=S * H * D * 4)
    # ---- state space
    mix = Mamba2(W, M, P, N, 8, 4, 8, 1e-5).to(device=dev, dtype=bf)
    mix.finish_loading()
    st = mix.make_cache(B, T, bf, dev)
    proj, inner = rn(S, mix.w_in.shape[0]), mix.inner
    args = (mix.conv_w, mix.conv_b, mix.dt_bias_f32, mix.A_log_f32, mix.skip_f32)
    ssm_f = S * M * (2 * 64 * N / 2 + 2 * 64 * P / 2 + 4 * N * P)
    add("state space, prefill (convolution + scan)",
        time_op(lambda: ops.ssm(proj, inner, *args, st.conv[:1], st.state[:1], S=S, groups=8), flush), None, 0,
        flops=ssm_f, nbytes=S * (inner * 2 + mix.channels * 6))
    p1 = rn(B, mix.w_in.shape[0])
    add("state space, decode (convolution + step)",
        time_op(lambda: ops.ssm(p1, inner, *args, st.conv, st.state, S=1, groups=8, start=5), flush), None, 0, nbytes=B * M * N * P * 8)
    yy = rn(S, inner)
    add("gated group norm, prefill", time_op(lambda: ops.gated_group_norm(yy, proj, mix.norm_w, 8, 1e-5), flush),
        "add + F.rms_norm", norm, nbytes=S * inner * 6, like_bytes=S * W * 8)
    return rows


def measured_peaks():
    try:
        with open(os.path.join(ROOT, "MEASURED_PEAKS.json")) as f:
            d = json.load(f)
        return {"hbm_gbs": d["hbm_gbs"], "bf16_tflops": d["bf16_tflops"], "source": "measured"}
    except Exception:
        return {"hbm_gbs": FALLBACK_HBM_GBS, "bf16_tflops": 1590.0, "source": "fallback"}


def run_radapel(args, dev):
    """Prefill and decode throughput of Radapel at two sizes beside the Llama-shaped Transformer with as many
    layers, the same width, heads and feed-forward (sparse and dense decode), and the kernels one by one."""
    from socket_b200.model import ModelArgs, Transformer
    from socket_b200.registry import build_model
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    K, W = min(args.steps, 64), max(3, min(args.warmup, 8))
    clocks = ClockSampler(dev.index or 0)
    out = {}
    for size, (width, H, G, D, FF, *_rest) in RADAPEL_SIZES.items():
        cfg = radapel_config(size)
        model = build_model(cfg, dtype=torch.bfloat16, device=dev).init_random(args.seed)
        n_runs = len(model.runs)
        rec = {"layer_runs": n_runs, "width": width}
        shapes = [(1, 2048), (1, 8000), (1, 32000), (8, 8000)]   # decoding late in a chunk of 8192
        for B, T in shapes:
            rec[f"radapel B={B} T={T}"] = measure_throughput(model, cfg["vocab"], B, T, K, W, dev)
        flags = model.device_flags()
        del model
        torch.cuda.empty_cache()
        old = torch.get_default_dtype()
        torch.set_default_dtype(torch.bfloat16)
        with torch.device(dev):
            other = Transformer(ModelArgs(block_size=131072, vocab_size=cfg["vocab"], n_layer=n_runs, n_head=H, n_local_heads=G,
                                          dim=width, intermediate_size=FF, rope_base=500000))
        torch.set_default_dtype(old)
        other.init_random(args.seed)
        for B, T in shapes:
            for mode in ("sparse", "dense"):
                rec[f"transformer {mode} B={B} T={T}"] = measure_throughput(other, cfg["vocab"], B, T, K, W, dev, mode)
        del other
        torch.cuda.empty_cache()
        rec["kernels S=8192, decode B=1 T=32768"] = measure_radapel_kernels(size, 8192, 32768, 1, dev)
        rec["device_flags"] = flags
        torch.cuda.empty_cache()
        out[size] = rec
    main_rec = out["4k"]["radapel B=1 T=32000"]
    print(json.dumps({
        "metric": "decode_tokens_per_s", "value": main_rec["decode_tokens_per_s"], "unit": "tokens/s", "n_gpus": 1, "steps": K,
        "warmup": W, "ms_per_step": main_rec["decode_ms_per_token"], "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": {"model": "Radapel 4k, 7 layer runs, random weights", "global_batch": 1, "seq_len": 32000,
                   "parallelism": "single GPU", "timing": "CUDA events around K graph-replayed decode tokens; weights exceed L2; "
                   "kernels one by one with L2 flushed"},
        "e2e": {"value": main_rec["e2e_decode_tokens_per_s"], "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 8},
        "peaks": measured_peaks(), "clocks": clocks.stop(), "radapel": out}))


# ------------------------------------------------------------------------------- Timalorn
TIMALORN_MEMORY = {"2k": (8, 128, 256), "4k": (8, 256, 512)}     # heads, key size, value size
TIMALORN_WINDOW, TIMALORN_ROT, TIMALORN_CAP = 4096, 64, 50.0


def timalorn_config(size):
    """Attention and memory in turn, 7 layers, two of which use the tensors of earlier ones; width, heads and
    feed-forward of the Radapel size."""
    W, H, G, D, F, *_ = RADAPEL_SIZES[size]
    MH, N, P = TIMALORN_MEMORY[size]
    mlp = {"kind": "dense", "ff": F}
    att = {"type": "attention", "mlp": mlp,
           "mixer": {"heads": H, "kv_heads": G, "dim": D, "vdim": D, "scale": D ** -0.5, "softcap": TIMALORN_CAP,
                     "mask": {"size": TIMALORN_WINDOW},
                     "rot": {"base": 500000.0, "dims": TIMALORN_ROT,
                             "scaling": {"factor": 4.0, "original": 8192, "fast": 32.0, "slow": 1.0}}}}
    mem = {"type": "mlstm", "mlp": mlp, "mixer": {"heads": MH, "dim": N, "vdim": P, "gate_cap": 15.0}}
    return {"architecture": "Timalorn", "vocab": 32768, "width": W, "norm": {"eps": 1e-5}, "embedding": {"scale": 1.0},
            "layers": [att, mem, att, mem, dict(att, weights_of=0), dict(mem, weights_of=1), att]}


def weights_per_token(model):
    """Elements of the matrices a token passes through (shared ones as often as they are used)."""
    layers = sum(p.numel() for r in model.runs for p in model.layer_of(r).parameters())
    return layers + model.head.numel()


def measure_timalorn_kernels(size, S, T, B, dev):
    """Every kernel of the design beside the like kernel of Radapel, at one size: prefill kernels on S tokens from
    position 0, decode kernels for B sequences at context T."""
    from socket_b200 import block_ops as ops
    from socket_b200.mixers import Mamba2, YarnScaling, rotary_angles
    W, H, G, D, FF, K, M = RADAPEL_SIZES[size]
    MH, N, P = TIMALORN_MEMORY[size]
    R, WIN, RN, RP = TIMALORN_ROT, TIMALORN_WINDOW, RADAPEL_STATE, 64
    bf = torch.bfloat16
    rn = lambda *s: torch.randn(*s, device=dev, dtype=bf)  # noqa: E731
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    t = lambda fn: time_op(fn, flush)  # noqa: E731
    rows, add = kernel_table(measured_peaks())
    ws = torch.empty(64 << 20, dtype=torch.uint8, device=dev)
    # ---- attention of a prompt
    sink, bias = torch.randn(H, device=dev), torch.randn(H, 1025, device=dev)
    q, k, v = rn(1, S, H, D), rn(1, S, G, D), rn(1, S, G, D)
    kv = rn(1, S, G, D + R)
    kw = dict(scale=D ** -0.5, window=WIN, sink=sink)
    pairs, full = sum(min(i + 1, WIN) for i in range(S)), S * (S + 1) / 2
    like = t(lambda: ops.attn(q, k, v, scale=D ** -0.5, chunk=RADAPEL_CHUNK, bias=bias))
    lk = dict(like="chunked attention", like_us=like, like_flops=full * H * 4 * D)
    add(f"window attention, capped scores, prefill (window {WIN})",
        t(lambda: ops.attn(q, kv[..., R:], kv[..., :D], softcap=TIMALORN_CAP, **kw)), flops=pairs * H * 4 * D, **lk)
    big = q * (4 * TIMALORN_CAP)                   # scores at the cap: the form without the polynomial
    add("the same, scores at the cap", t(lambda: ops.attn(big, kv[..., R:], kv[..., :D], softcap=TIMALORN_CAP, **kw)),
        flops=pairs * H * 4 * D, **lk)
    add("the same without a cap", t(lambda: ops.attn(q, kv[..., R:], kv[..., :D], **kw)), flops=pairs * H * 4 * D, **lk)
    # ---- attention of a decoded token
    pos = torch.tensor([T - 1], device=dev)
    q1, ring = rn(B, 1, H, D), rn(B, WIN, G, D + R)
    kr, vr = rn(B, WIN, G, D), rn(B, WIN, G, D)
    ringpos = torch.tensor([WIN - 1], device=dev)
    add(f"window attention, decode (ring {WIN} full)",
        t(lambda: ops.attn(q1, ring[..., R:], ring[..., :D], pos=pos, ring=True, softcap=TIMALORN_CAP, workspace=ws, **kw)),
        "chunked attention, ring as long",
        t(lambda: ops.attn(q1, kr, vr, scale=D ** -0.5, pos=ringpos, chunk=WIN, ring=True, bias=bias, workspace=ws)),
        nbytes=B * WIN * G * (D + R) * 2, like_bytes=B * WIN * G * 2 * D * 2)
    # ---- rotation and cache rows
    ang = rotary_angles(max(S, T), R, 500000.0, dev, YarnScaling(4.0, 8192, 32.0, 1.0))
    ang_l = rotary_angles(max(S, T), RADAPEL_ROT, 500000.0, dev)
    cols = (H + G) * D

    def rotary(n, start, rows_out, **more):
        proj = rn(n, cols)
        qq, kk = proj[:, :H * D].unflatten(-1, (H, D)), proj[:, H * D:].unflatten(-1, (G, D))
        return t(lambda: ops.rotary_rows(qq, kk, ang, R, rows_out, start=start, **more))

    def latent(n, s, cache, **more):
        dkv, qq, lw = rn(n, K + RADAPEL_ROT), rn(n, H * (D + RADAPEL_ROT)), rn(K)
        return t(lambda: ops.latent_append(dkv, qq, lw, ang_l, cache, S=s, n_heads=H, dim=D, rot=RADAPEL_ROT, rank=K, eps=1e-5, **more))

    add("rotary rows, prefill", rotary(S, 0, torch.empty(1, S, G, D + R, dtype=bf, device=dev), B=1, S=S),
        "latent append + rotation", latent(S, S, rn(1, S, K + RADAPEL_ROT)),
        nbytes=S * 2 * (2 * H * D + G * (2 * D + R)), like_bytes=S * (4 * (K + RADAPEL_ROT) + 4 * H * RADAPEL_ROT))
    add("rotary rows, decode", rotary(B, 0, ring, B=B, S=1, pos=pos), "latent append + rotation",
        latent(B, 1, rn(B, T, K + RADAPEL_ROT), pos=pos),
        nbytes=B * 2 * (2 * H * D + G * (2 * D + R)), like_bytes=B * (4 * (K + RADAPEL_ROT) + 4 * H * RADAPEL_ROT))
    add("ring append of a prompt", t(lambda: ops.ring_append(kv, None, ring[:1], None, start=0, keep="window")),
        "ring append of a chunk", t(lambda: ops.ring_append(k, v, kr[:1], vr[:1], start=0)),
        nbytes=WIN * G * (D + R) * 4, like_bytes=WIN * G * 2 * D * 4)
    # ---- residual stream, gated unit
    for name, n in (("prefill", S), ("decode", B)):
        x, y, y16, w = torch.randn(n, W, device=dev), torch.randn(n, W, device=dev), rn(n, W), rn(W)
        add(f"residual + layer norm, {name}", t(lambda: ops.residual_norm(x, 1e-5, y=y, w_out=w, centred=True)),
            "residual + two norms", t(lambda: ops.residual_norm(x, 1e-5, y=y16, w_in=w, w_out=w)),
            nbytes=n * W * 14 + 2 * W, like_bytes=n * W * 12 + 4 * W)
        gu, wide = rn(n, 2 * FF), rn(n, FF + H * D)
        add(f"silu unit, {name}", t(lambda: ops.glu_silu(gu[:, :FF], gu[:, FF:], out=wide[:, H * D:])),
            "clamped unit", t(lambda: ops.glu_clamped(gu, FF, 7.0)), nbytes=n * FF * 6)
    # ---- recurrences
    mix = Mamba2(W, M, RP, RN, 8, 4, 8, 1e-5).to(device=dev, dtype=bf)
    mix.finish_loading()
    inner, chans = mix.inner, mix.channels
    sargs = (mix.conv_w, mix.conv_b, mix.dt_bias_f32, mix.A_log_f32, mix.skip_f32)
    st = mix.make_cache(B, T, bf, dev)
    Ss, ns, ms = (torch.zeros(s, device=dev) for s in ((B, MH, N, P), (B, MH, N), (B, MH)))
    ib, fb, nw = torch.zeros(MH, device=dev), torch.full((MH,), 3.0, device=dev), rn(MH * P)

    def memory(n, s, **more):
        proj, gates = rn(n, 2 * MH * (N + P)), torch.randn(n, 2 * MH, device=dev)
        a, b = MH * N, 2 * MH * N
        parts = (proj[:, :a], proj[:, a:b], proj[:, b:b + MH * P], proj[:, b + MH * P:])
        nb = n // s
        out = torch.empty(n, MH * P, dtype=bf, device=dev)
        return t(lambda: ops.mlstm(*parts, gates, ib, fb, nw, Ss[:nb], ns[:nb], ms[:nb], out, S=s, cap=15.0, q_scale=N ** -0.5,
                                   eps=1e-5, **more))

    def state_space(n, s, **more):
        proj, nb = rn(n, mix.w_in.shape[0]), n // s

        def run():
            y = ops.ssm(proj, inner, *sargs, st.conv[:nb], st.state[:nb], S=s, groups=8, **more)
            ops.gated_group_norm(y, proj, mix.norm_w, 8, 1e-5)
        return t(run)

    blk = 64                                       # causal half of a block's products, and the state's
    add("matrix memory, prefill (gates, blocks, norm and gate)", memory(S, S), "state space (convolution, blocks, gated norm)", state_space(S, S),
        flops=S * MH * (blk * N + blk * P + 4 * N * P), nbytes=S * MH * 2 * (2 * N + 3 * P),
        like_flops=S * M * (blk * RN + blk * RP + 4 * RN * RP), like_bytes=S * (inner * 6 + chans * 6))
    add("matrix memory, decode (step, norm and gate)", memory(B, 1, pos=pos), "state space (convolution, step, gated norm)",
        state_space(B, 1, pos=pos), nbytes=B * MH * N * P * 8, like_bytes=B * M * RN * RP * 8)
    h, wg = rn(S, W), rn(2 * MH, W)
    from socket_b200.mixers import matmul_f32
    add("gates' projection, prefill (library product)", t(lambda: matmul_f32(h, wg)), None, 0, nbytes=S * W * 2)
    add("gates' projection, decode (library product)", t(lambda: matmul_f32(h[:B], wg)), None, 0, nbytes=2 * MH * W * 2)
    return rows


def run_timalorn(args, dev):
    """Prefill and decode throughput of Timalorn at two sizes beside Radapel with as many layer runs, the same
    width, heads and feed-forward, and the kernels one by one."""
    from socket_b200.registry import build_model
    torch.backends.cuda.matmul.allow_bf16_reduced_precision_reduction = False
    K, W = min(args.steps, 64), max(3, min(args.warmup, 8))
    clocks = ClockSampler(dev.index or 0)
    out = {}
    for size in RADAPEL_SIZES:
        rec = {"width": RADAPEL_SIZES[size][0]}
        for name, cfg in (("timalorn", timalorn_config(size)), ("radapel", radapel_config(size))):
            model = build_model(cfg, dtype=torch.bfloat16, device=dev).init_random(args.seed)
            rec[f"{name} layer runs"], rec[f"{name} weights per token"] = len(model.runs), weights_per_token(model)
            for B, T in [(1, 2048), (1, 8000), (1, 32000), (8, 8000)]:
                rec[f"{name} B={B} T={T}"] = measure_throughput(model, cfg["vocab"], B, T, K, W, dev)
            rec[f"{name} device flags"] = model.device_flags()
            del model
            torch.cuda.empty_cache()
        rec["kernels S=8192, decode B=1 T=32768"] = measure_timalorn_kernels(size, 8192, 32768, 1, dev)
        torch.cuda.empty_cache()
        out[size] = rec
    main_rec = out["4k"]["timalorn B=1 T=32000"]
    print(json.dumps({
        "metric": "decode_tokens_per_s", "value": main_rec["decode_tokens_per_s"], "unit": "tokens/s", "n_gpus": 1, "steps": K,
        "warmup": W, "ms_per_step": main_rec["decode_ms_per_token"], "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "bf16", "data": "synthetic",
        "config": {"model": "Timalorn 4k, 7 layers, random weights", "global_batch": 1, "seq_len": 32000,
                   "parallelism": "single GPU", "timing": "CUDA events around K graph-replayed decode tokens; weights exceed L2; "
                   "kernels one by one with L2 flushed"},
        "e2e": {"value": main_rec["e2e_decode_tokens_per_s"], "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 8},
        "peaks": measured_peaks(), "clocks": clocks.stop(), "timalorn": out}))


def main():
    args = parse_args()
    if args.impl == "reference":
        if args.workload in MODEL_WORKLOADS or args.workload in ("radapel", "timalorn"):
            if int(os.environ.get("RANK", "0")) == 0:
                print(json.dumps({"impl": "reference", "unavailable": "the whole-model workloads have no CPU arm: the "
                                  "reference's CPU path is timed at the op level (c1-c3)"}))
            return
        run_reference(args, PRESETS[args.workload])
        return

    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device: the product path has no CPU fallback")

    from socket_b200 import tp

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local_rank)
    if world > 1:
        tp.maybe_init_dist("nccl")
    K, W = args.steps, args.warmup

    if args.workload == "radapel":
        run_radapel(args, torch.device("cuda", local_rank))
        return
    if args.workload == "timalorn":
        run_timalorn(args, torch.device("cuda", local_rank))
        return
    if args.workload in MODEL_WORKLOADS:
        K = min(K, MODEL_WORKLOADS[args.workload][3] - 1)
        m = measure_model(args, args.workload, K, W, world, rank, local_rank)
        if rank == 0:
            print(json.dumps({
                "metric": "decode_tokens_per_s", "value": m["sparse"]["tokens_per_s"], "unit": "tokens/s",
                "n_gpus": world, "steps": K, "warmup": W, "ms_per_step": m["sparse"]["ms_per_token"],
                "higher_is_better": True, "scaling": "weak" if world == 1 else "strong", "vs_baseline": None,
                "dtype": "bf16", "data": "synthetic",
                "config": {"workload": f"{args.workload}: greedy decode, {m['architecture']} shape, random bf16 weights, "
                                       f"batch {m['batch']}, prompt {m['prompt_tokens']} uniform random token ids",
                           "parallelism": "single GPU" if world == 1 else f"tensor parallel over {world} GPUs (heads split, "
                                          "NCCL all-reduce after wo and the feed-forward)",
                           "timing": "CUDA events around K graph-replayed decode tokens"},
                "model": m, "e2e": {"value": m["sparse"].get("e2e_tokens_per_s"), "unit": "tokens/s",
                                    "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 8 * m["batch"]},
                "gpu_launches": K * m["sparse"]["gpu_launches_per_token_path"]}))
        if world > 1:
            torch.distributed.destroy_process_group()
        return

    res = measure(args, args.workload, K, W, world, rank, local_rank, full=True)
    torch.cuda.empty_cache()
    second = None
    if args.secondary not in ("none", args.workload):
        wl2 = PRESETS[args.secondary]
        if not (world > 1 and args.shard == "strong" and wl2.n_local_heads % world):
            second = measure(args, args.secondary, K, W, world, rank, local_rank, full=False)
            torch.cuda.empty_cache()

    model_rec = None
    if args.model_record == "on" or (args.model_record == "auto" and world == 1):
        try:
            model_rec = measure_model(args, "c4", min(args.model_tokens, K), min(W, 8), world, rank, local_rank)
        except Exception as e:  # the comparison must never cost the op-level line
            model_rec = {"failed": repr(e)[:300]}
        torch.cuda.empty_cache()

    cfg_full = PRESETS[args.workload]
    cpu_baseline = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        try:
            state = host_state(cfg_full, args.seed, 64)
            per_step, cores, done = cpu_reference_steps(cfg_full, state)
            cpu_baseline = {"value": cfg_full.batch / per_step, "unit": UNIT, "cores": cores, "kind": "port",
                            "ms_per_step": per_step * 1e3,
                            "sample": f"{done} decode steps of workload {args.workload} (full context, all "
                                      f"heads) with the C restatement of the reference path"}
        except Exception as e:  # the baseline is a reported figure, never a reason to lose the line
            cpu_baseline = {"value": None, "unit": UNIT, "cores": os.cpu_count(), "kind": "port",
                            "sample": f"failed: {e!r}"}

    if rank == 0:
        line = {
            "metric": METRIC, "value": res["value"], "unit": UNIT, "n_gpus": world, "steps": K, "warmup": W,
            "ms_per_step": res["ms_per_step"], "us_per_layer": res["us_per_layer"], "higher_is_better": True,
            "scaling": "weak" if world == 1 else args.shard, "vs_baseline": None, "dtype": res["dtype"],
            "data": "synthetic", "config": res["config"], "roofline": res["roofline"], "stages": res["stages"],
            "e2e": res["e2e"], "cpu_baseline": cpu_baseline, "clocks": res["clocks"],
            "gpu_launches": res["gpu_launches"],
            # (batch, head) rows that took the select kernel's exact-but-slow rescoring path, over
            # every step this process ran on the timed workspace (warm-up, timed loop, whole-step stage)
            "rescored_rows": res.get("rescored_rows"),
            "select_stats": res.get("select_stats"),
        }
        if model_rec is not None:
            line["c4"] = model_rec
        if second is not None:
            line[args.secondary] = {k: second[k] for k in ("value", "ms_per_step", "us_per_layer", "config",
                                                            "roofline", "stages", "e2e", "clocks", "gpu_launches",
                                                            "rescored_rows", "select_stats") if k in second}
            line[args.secondary]["unit"] = UNIT
        print(json.dumps(line))
    if world > 1:
        torch.distributed.destroy_process_group()


if __name__ == "__main__":
    main()
