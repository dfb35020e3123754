#!/usr/bin/env python
"""Benchmark of the xLSTM inference hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Headline workload: the mLSTM decode step at the xLSTM-7B head shape,
B=16, NH=8, dqk=256, dv=512, bf16 activations, fp32 state.  A "step" is one decode step of the
cell for the whole batch (16 tokens).  Consecutive steps walk a ring of independent layer
states (8 layers x 2 buffers = 1 GiB), so every step streams a state that is cold in the
126 MB L2, as a 32-layer model's decode does.

``value``  tokens/s with inputs resident in HBM (kernel launched straight through the C ABI).
``e2e``    tokens/s through the public tensor API with HOST inputs: pinned host -> device copies
           of q,k,v,i,f and a device -> host read of h inside the timed region, every step.
``prefill``  chunkwise prefill (B=4, S=32768, heads sharded over the
           ranks, NCCL all-gather of h, 4096x4096 out-projection), reported beside the headline.
At N > 1 the decode batch is sharded (global batch 16*N, no collective): weak scaling.
``--impl reference`` times the reference's own torch_native recurrent cell (the unmodified class, placed
under oracle/_ref by oracle/make_ref.py) on all host cores for the same workload at the same global
batch; where that file is absent it times the C restatement (oracle/, OpenMP over batch x heads).
The JSON line stays short: the prefill / sLSTM / soft-cap figures ride inside ``roofline``; the long
per-kernel tables (glue kernels, 7B-shaped model) go to ``bench_details_n{N}.json`` in the folder that ``--details`` names.
"""
from __future__ import annotations

import argparse
import json
import os
import sys
import threading
import time
from pathlib import Path

ROOT = Path(__file__).resolve().parent
for _p in (ROOT, ROOT / "xlstm-metal_b200"):
    if str(_p) not in sys.path:
        sys.path.insert(0, str(_p))

B, NH, DQK, DV = 16, 8, 256, 512
N_LAYERS = 8          # ring of independent layer states (cold-L2 rule)
N_INPUT_SETS = 64     # distinct per-step inputs cycled through
WORKLOAD = "mlstm_decode_step B=16 NH=8 dqk=256 dv=512 bf16 act fp32 state"


def workload_config(world):
    """``config`` of the JSON line: the same dict in both arms, so that the two lines describe one workload."""
    return {"workload": WORKLOAD, "global_batch": B * world, "parallelism": f"batch-sharded x{world}",
            "l2": f"ring of {N_LAYERS} layer states x 2 buffers = {N_LAYERS * 2 * B * NH * DQK * DV * 4 >> 20} MiB > L2; "
                  "every step streams a cold state", "state_update": "out-of-place"}


def step_bytes(b=B, nh=NH, dqk=DQK, dv=DV, e=2):
    """Algorithmic HBM bytes of one decode step: C read+write, n read+write, m, q,k,v,h, i,f."""
    per_head = 2 * dqk * dv * 4 + 2 * dqk * 4 + 8 + 2 * dqk * e + dv * e + dv * e + 2 * e
    return b * nh * per_head


def peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), float(d.get("bf16_tflops_sustained", d["bf16_tflops"])), "measured"
    return 6650.0, 1400.0, "fallback"


def burst_tflops():
    """The bf16 GEMM peak for a kernel timed alone in a short burst (before the power cap pulls the clocks down)."""
    p = ROOT / "MEASURED_PEAKS.json"
    return float(json.loads(p.read_text())["bf16_tflops"]) if p.exists() else 1590.0


class ClockSampler:
    """Samples SM clock and throttle reasons of one GPU through NVML while a region runs."""

    def __init__(self, index: int):
        self.samples, self.reasons, self.max_mhz = [], set(), None
        self._stop = threading.Event()
        self._thread = None
        try:
            import pynvml
            pynvml.nvmlInit()
            self.nv = pynvml
            self.h = pynvml.nvmlDeviceGetHandleByIndex(index)
            self.max_mhz = pynvml.nvmlDeviceGetMaxClockInfo(self.h, pynvml.NVML_CLOCK_SM)
        except Exception:
            self.nv = None

    def _loop(self):
        nv = self.nv
        names = {
            getattr(nv, "nvmlClocksThrottleReasonHwSlowdown", 0x8): "hw_slowdown",
            getattr(nv, "nvmlClocksThrottleReasonHwThermalSlowdown", 0x40): "hw_thermal_slowdown",
            getattr(nv, "nvmlClocksThrottleReasonSwThermalSlowdown", 0x20): "sw_thermal_slowdown",
            getattr(nv, "nvmlClocksThrottleReasonSwPowerCap", 0x4): "sw_power_cap",
        }
        while not self._stop.is_set():
            try:
                self.samples.append(nv.nvmlDeviceGetClockInfo(self.h, nv.NVML_CLOCK_SM))
                r = nv.nvmlDeviceGetCurrentClocksThrottleReasons(self.h)
                for bit, name in names.items():
                    if r & bit:
                        self.reasons.add(name)
            except Exception:
                break
            time.sleep(0.002)

    def __enter__(self):
        if self.nv is not None:
            self._thread = threading.Thread(target=self._loop, daemon=True)
            self._thread.start()
        return self

    def __exit__(self, *exc):
        self._stop.set()
        if self._thread is not None:
            self._thread.join()

    def summary(self):
        s = sorted(self.samples)
        return {"sm_mhz": (s[len(s) // 2] if s else None), "sm_max_mhz": self.max_mhz,
                "reasons": sorted(self.reasons), "samples": len(s)}


def make_inputs(torch, device, seed):
    g = torch.Generator().manual_seed(seed)
    bf = torch.bfloat16
    cap = lambda x: 15.0 * torch.tanh(x / 15.0)
    q = torch.randn(N_INPUT_SETS, B, NH, DQK, generator=g).to(bf)
    k = torch.randn(N_INPUT_SETS, B, NH, DQK, generator=g).to(bf)
    v = torch.randn(N_INPUT_SETS, B, NH, DV, generator=g).to(bf)
    i = cap(torch.randn(N_INPUT_SETS, B, NH, generator=g)).to(bf)
    f = cap(torch.randn(N_INPUT_SETS, B, NH, generator=g) + 3.0).to(bf)
    return q, k, v, i, f


def host_threads():
    """Host threads this process may use (under torch.distributed.run OMP_NUM_THREADS is 1: ask the OS)."""
    try:
        return max(1, len(os.sched_getaffinity(0)))
    except AttributeError:
        return max(1, os.cpu_count() or 1)


class CpuDecode:
    """The decode workload on the host cores: the reference's own ``mLSTMRecurrentKernelCell`` (bf16 compute,
    fp32 state; ``kind`` "reference") when oracle/_ref holds it, else the C restatement (``kind`` "port")."""

    def __init__(self, batch, threads, force_port=False):
        import numpy as np
        from oracle import make_ref, oracle as xo
        self.np, self.xo, self.batch, self.threads = np, xo, batch, threads
        xo.set_threads(threads)
        cls = None if force_port else make_ref.load_cell_class()
        self.kind = "reference" if cls is not None else "port"
        rng = np.random.default_rng(1)
        n_sets = 8
        q, k = (xo.bf16_round(rng.standard_normal((n_sets, batch, NH, 1, DQK)).astype(np.float32)) for _ in range(2))
        v = xo.bf16_round(rng.standard_normal((n_sets, batch, NH, 1, DV)).astype(np.float32))
        i = xo.bf16_round((15 * np.tanh(rng.standard_normal((n_sets, batch, NH, 1)) / 15)).astype(np.float32))
        f = xo.bf16_round((15 * np.tanh((rng.standard_normal((n_sets, batch, NH, 1)) + 3) / 15)).astype(np.float32))
        st = ((rng.standard_normal((batch, NH, DQK, DV)) * 0.1).astype(np.float32),
              (rng.standard_normal((batch, NH, DQK)) * 0.1).astype(np.float32), np.zeros((batch, NH), np.float32))
        self.n_sets = n_sets
        if cls is not None:
            import torch
            torch.set_num_threads(threads)
            self.torch = torch
            self.cell = cls(NH, DQK, DV, compute_dtype=torch.bfloat16, state_dtype=torch.float32)
            self.inputs = [tuple(torch.from_numpy(a[s_]).to(torch.bfloat16) for a in (q, k, v, i, f)) for s_ in range(n_sets)]
            self.state = tuple(torch.from_numpy(a) for a in st)
            self.what = "reference torch_native mLSTMRecurrentKernelCell (bf16 compute, fp32 state), torch CPU"
        else:
            self.inputs = [tuple(a[s_] for a in (q, k, v, i, f)) for s_ in range(n_sets)]
            self.state = st
            self.what = "oracle C port of the torch_native recurrent cell (OpenMP over batch x heads)"

    def step(self, t):
        a = self.inputs[t % self.n_sets]
        if self.kind == "reference":
            with self.torch.no_grad():
                _, self.state = self.cell(*a, self.state)
        else:
            _, self.state = self.xo.mlstm_recurrent(*a, self.state)

    def run(self, steps, warmup, budget_s):
        """Up to ``steps`` decode steps within ``budget_s`` seconds; returns (steps done, seconds)."""
        for t in range(warmup):
            self.step(t)
        t0 = time.perf_counter()
        done = 0
        while done < steps:
            self.step(done)
            done += 1
            if time.perf_counter() - t0 > budget_s and done >= 3:
                break
        return done, time.perf_counter() - t0


def cpu_baseline(budget_s=12.0):
    """The decode workload on the host cores beside the GPU number, bounded sample (rank 0, N=1)."""
    threads = host_threads()
    ref = CpuDecode(B, threads)
    n, dt = ref.run(2000, 1, budget_s)
    out = {"value": B * n / dt, "unit": "tokens/s", "cores": threads, "kind": ref.kind,
           "sample": f"{n} decode steps of the headline workload in {dt:.1f} s, {ref.what}"}
    if ref.kind == "reference":     # the C restatement beside it, for scale
        port = CpuDecode(B, threads, force_port=True)
        n2, dt2 = port.run(2000, 1, 5.0)
        out["port_value"] = B * n2 / dt2
    return out


def run_reference(args):
    """CPU arm: the reference's cell on all host threads, same workload, metric and global batch as our arm."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    world = max(1, args.gpus)
    batch = B * world
    threads = host_threads()
    ref = CpuDecode(batch, threads)
    # a CPU step costs tens of milliseconds, so the run is bounded in time as well as in steps
    warm = min(args.warmup, 3)
    steps, dt = ref.run(min(args.steps, 2000), warm, 60.0)
    val = batch * steps / dt
    line = {"impl": "reference", "metric": "mlstm_decode_tokens_per_s", "value": val, "unit": "tokens/s",
            "n_gpus": args.gpus, "steps": steps, "warmup": warm, "ms_per_step": dt / steps * 1e3,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
            "dtype": "bf16" if ref.kind == "reference" else "f32",
            "data": "synthetic", "config": workload_config(world),
            "cpu_baseline": {"value": val, "unit": "tokens/s", "cores": threads, "kind": ref.kind,
                             "sample": f"{steps} full decode steps at global batch {batch} in {dt:.1f} s, {ref.what}"},
            "e2e": {"value": val, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def run_ours(args):
    import torch
    import torch.distributed as dist
    from xlstm_cuda import _lib, ops

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if not torch.cuda.is_available():
        raise SystemExit("bench.py needs a CUDA device: xlstm_cuda has no CPU path")
    torch.cuda.set_device(local)
    device = torch.device("cuda", local)
    if world > 1:
        dist.init_process_group("nccl", device_id=device)
    lib = _lib.load()
    K, W = args.steps, max(args.warmup, 3)

    q, k, v, i, f = make_inputs(torch, device, seed=1 + rank)
    qd, kd, vd, idv, fd = (t.to(device) for t in (q, k, v, i, f))
    g = torch.Generator().manual_seed(100 + rank)
    C = [[(torch.randn(B, NH, DQK, DV, generator=g) * 0.1).to(device), torch.empty(B, NH, DQK, DV, device=device)]
         for _ in range(N_LAYERS)]
    n = [[(torch.randn(B, NH, DQK, generator=g) * 0.1).to(device), torch.empty(B, NH, DQK, device=device)]
         for _ in range(N_LAYERS)]
    m = [[torch.zeros(B, NH, device=device), torch.empty(B, NH, device=device)] for _ in range(N_LAYERS)]
    h = torch.empty(B, NH, DV, dtype=torch.bfloat16, device=device)
    # pointer tuples for every (input set, layer, side): the timed loop is then one C call per step
    # the ring of layers guarantees that a step's state was written 8 launches earlier, so its first state rows may
    # be fetched while the preceding launch drains (XLSTM_STEP_STATE_SETTLED)
    fn = lib.xlstm_mlstm_step_ex
    ptr = {}
    for s_ in range(N_INPUT_SETS):
        for l in range(N_LAYERS):
            if (s_ - l) % N_LAYERS:
                continue  # step t uses set t % 64 and layer t % 8, so only matching residues occur
            for a in (0, 1):
                b = a ^ 1
                ptr[(s_, l, a)] = (qd[s_].data_ptr(), kd[s_].data_ptr(), vd[s_].data_ptr(), idv[s_].data_ptr(),
                                   fd[s_].data_ptr(), C[l][a].data_ptr(), n[l][a].data_ptr(), m[l][a].data_ptr(),
                                   h.data_ptr(), C[l][b].data_ptr(), n[l][b].data_ptr(), m[l][b].data_ptr(),
                                   B, NH, DQK, DV, 1e-6, 0.0, _lib.STEP_STATE_SETTLED, _lib.BF16)
    side = [0] * N_LAYERS

    def step(t, stream):
        l = t % N_LAYERS
        st = fn(*ptr[(t % N_INPUT_SETS, l, side[l])], stream)
        if st:
            _lib.check(st, "xlstm_mlstm_step_ex")
        side[l] ^= 1

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    # ---- device-resident leg: the K steps are captured in CUDA graphs (launch-bound loop) ----
    cur = torch.cuda.current_stream().cuda_stream
    for t in range(W):
        step(t, cur)
    barrier()
    G = min(K, 512)
    G -= G % (2 * N_LAYERS) if G >= 2 * N_LAYERS else 0   # whole ring periods, so replays chain correctly
    reps, rest = (K // G, K % G) if G else (0, K)
    graph = None
    if reps:
        graph = torch.cuda.CUDAGraph()
        cs = torch.cuda.Stream()
        cs.wait_stream(torch.cuda.current_stream())
        with torch.cuda.graph(graph, stream=cs):
            for t in range(G):
                step(W + t, torch.cuda.current_stream().cuda_stream)
        torch.cuda.current_stream().wait_stream(cs)
        graph.replay()  # warm the instantiated graph
    barrier()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    with ClockSampler(local) as clk:
        e0.record()
        for _ in range(reps):
            graph.replay()
        for t in range(rest):
            step(W + t, cur)
        e1.record()
        torch.cuda.synchronize()
        if len(clk.samples) < 3 and graph is not None:  # region shorter than the sampling period
            t_end = time.time() + 0.25
            while time.time() < t_end:
                graph.replay()
                torch.cuda.synchronize()
    barrier()
    ms = e0.elapsed_time(e1)
    tms = torch.tensor([ms], device=device)
    if world > 1:
        dist.all_reduce(tms, op=dist.ReduceOp.MAX)
    ms_max = float(tms.item())
    value = world * B * K / (ms_max * 1e-3)

    # ---- end-to-end leg: host buffers through the public host-fed decode API -----------------
    from xlstm_cuda.runtime import DecodePipeline
    pipe = DecodePipeline(B, NH, DQK, DV, device, group=N_LAYERS)   # the steps of one pass over the layer ring travel together
    packed = [pipe.pack(q[s_], k[s_], v[s_], i[s_], f[s_]) for s_ in range(N_INPUT_SETS)]
    h_host = [torch.empty(B, NH, DV, dtype=torch.bfloat16).pin_memory() for _ in range(2)]
    side2 = [0] * N_LAYERS

    def e2e_step(t):
        l = t % N_LAYERS
        a = side2[l]
        pipe.step(packed[t % N_INPUT_SETS], (C[l][a], n[l][a], m[l][a]), (C[l][a ^ 1], n[l][a ^ 1], m[l][a ^ 1]),
                  h_host[t % 2], state_settled=True)
        side2[l] ^= 1

    for t in range(W):
        e2e_step(t)
    pipe.synchronize()
    # the step loop (copy in, kernel, copy out per step) replayed as a CUDA graph, like the device leg
    Ge = min(K, 256)
    Ge -= Ge % (2 * N_LAYERS) if Ge >= 2 * N_LAYERS else 0
    reps_e, rest_e = (K // Ge, K % Ge) if Ge else (0, K)
    egraph = None
    if reps_e:
        side2 = [0] * N_LAYERS
        steps_e = []
        for t in range(Ge):
            l = t % N_LAYERS
            a = side2[l]
            steps_e.append((packed[t % N_INPUT_SETS], (C[l][a], n[l][a], m[l][a]),
                            (C[l][a ^ 1], n[l][a ^ 1], m[l][a ^ 1]), h_host[t % 2], True))
            side2[l] ^= 1
        egraph = pipe.capture(steps_e)
        egraph.replay()
        torch.cuda.synchronize()
    barrier()
    e0.record()
    for _ in range(reps_e):
        egraph.replay()
    if rest_e:
        for st_ in pipe.streams():
            st_.wait_event(e0)
        for t in range(rest_e):
            e2e_step(t)
        for st_ in pipe.streams():
            torch.cuda.current_stream().wait_stream(st_)
    e1.record()
    barrier()
    tms = torch.tensor([e0.elapsed_time(e1)], device=device)
    if world > 1:
        dist.all_reduce(tms, op=dist.ReduceOp.MAX)
    e2e_ms = float(tms.item())
    e2e_val = world * B * K / (e2e_ms * 1e-3)
    h2d = packed[0].numel() * packed[0].element_size()
    d2h = h_host[0].numel() * h_host[0].element_size()

    # ---- prefill beside it ---------------------------------------------------
    prefill = None
    if not args.no_prefill:
        prefill = run_prefill(torch, dist, ops, device, world, rank, args)

    hbm, tf, which = peaks()
    achieved = step_bytes() / (ms / K * 1e-3) / 1e9  # this rank's kernel
    roofline = {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s", "frac": achieved / hbm,
                "traffic": TRAFFIC_PER_LAUNCH, "kernel": "mlstm_step_kernel", "peak_source": which,
                "algorithmic_bytes_per_launch": step_bytes()}
    details = {}
    if prefill is not None:
        # the prefill half of the metric, kept inside `roofline` so that it survives in the run records
        r = prefill["roofline"]
        roofline["prefill"] = {
            "frac": r["frac"], "tflops": r["achieved"], "peak_tflops": r["peak"], "hbm_frac": r["hbm_frac"],
            "cell_ms": prefill["cell_ms"], "tokens_per_s": prefill["cell_tokens_per_s"], "clocks": prefill["clocks"],
            "cell_ms_burst": prefill["cell_ms_burst"], "frac_burst": r["frac_burst"],
            "with_allgather_outproj_ms": prefill["with_allgather_outproj_ms"],
            "nccl_variant_ms": prefill["nccl_allgather_variant_ms"], "world": world,
            "gather_check": prefill["gather_check"], "gather_gbs_per_rank": prefill["gather_gbs_per_rank"],
            "token_sharded_outproj_ms": prefill["token_sharded_outproj_ms"], "token_sharded_check": prefill["token_sharded_check"],
            "workload": f"B=4 S={args.prefill_seq} NH=8 256/512 bf16, heads x{world}",
            "kernel": "mlstm_chunkwise_tc_fast_kernel", "bound": "tensor"}
        details["prefill"] = prefill
    launches = K
    if not args.no_extras:
        sl = run_slstm(torch, dist, device, world, rank)
        details["slstm"] = sl
        roofline["slstm_ms"] = sl["ms"]
        if rank == 0:
            sc = run_softcap(torch, ops, device)
            details["softcap"] = sc
            roofline["softcap_frac"] = sc["roofline"]["frac"]
            details["glue"] = run_glue(torch, ops, device)
            roofline["glue_frac"] = {k_: round(v_["roofline"]["frac"], 3) for k_, v_ in details["glue"].items()}
            if not args.no_model:
                mo = run_model(torch, device, 2048, 256)
                details["model"] = mo
                roofline["model_7b"] = {"prefill_tokens_per_s": mo["prefill_tokens_per_s"],
                                        "decode_tokens_per_s": mo["decode_tokens_per_s"]}
    if "prefill" in roofline:
        # the prefill figures close the line (a record that keeps only the end of a long line still has them):
        # no empty entries, floats to five significant digits
        pf = {k_: (float(f"{v_:.5g}") if isinstance(v_, float) else v_) for k_, v_ in roofline.pop("prefill").items()
              if v_ is not None}
        roofline["prefill"] = pf
    line = {
        "metric": "mlstm_decode_tokens_per_s", "value": value, "unit": "tokens/s", "n_gpus": world, "steps": K,
        "warmup": W, "ms_per_step": ms_max / K, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "bf16", "data": "synthetic", "config": workload_config(world),
        "e2e": {"value": e2e_val, "unit": "tokens/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                "ms_per_step": e2e_ms / K},
        "gpu_launches": launches, "launch": "CUDA graph replay of the step loop",
        "clocks": clk.summary(),
    }
    if rank == 0:
        line["cpu_baseline"] = cpu_baseline() if world == 1 and not args.no_cpu else None
        line["roofline"] = roofline
        print(json.dumps(line), flush=True)
        if args.details:    # the long per-kernel tables: a file beside the run, not part of the line
            out = Path(args.details)
            out.mkdir(parents=True, exist_ok=True)
            (out / f"bench_details_n{world}.json").write_text(json.dumps({"line": line, "details": details}, indent=1))
    if world > 1:
        dist.destroy_process_group()


# dram__bytes_read.sum + dram__bytes_write.sum per launch of mlstm_step_kernel, from the ncu
# capture summarised under profiles/ (None until a capture exists)
TRAFFIC_PER_LAUNCH = 84_321_792   # 67.52 MB read + 16.80 MB written before the kernel ends (rest drains from L2 later)


def run_prefill(torch, dist, ops, device, world, rank, args):
    """Chunkwise prefill: B=4, S=32768, NH=8, 256/512, L=64, bf16; heads sharded over the ranks,
    all-gather of h, then the replicated 4096x4096 out-projection.  Strong scaling."""
    Bp, Sp, L = 4, args.prefill_seq, 64
    nh_local = NH // world if NH % world == 0 else NH
    g = torch.Generator().manual_seed(3 + rank)
    bf = torch.bfloat16
    q = torch.randn(Bp, nh_local, Sp, DQK, generator=g).to(bf).to(device)
    k = torch.randn(Bp, nh_local, Sp, DQK, generator=g).to(bf).to(device)
    v = torch.randn(Bp, nh_local, Sp, DV, generator=g).to(bf).to(device)
    i = (15 * torch.tanh(torch.randn(Bp, nh_local, Sp, generator=g) / 15)).to(bf).to(device)
    f = (15 * torch.tanh((torch.randn(Bp, nh_local, Sp, generator=g) + 3) / 15)).to(bf).to(device)
    w_out = (torch.randn(NH * DV, NH * DV, generator=g) * 0.02).to(bf).to(device)
    need = ops.chunkwise_workspace_bytes(Bp, nh_local, Sp, DQK, DV, L, bf)
    ws = torch.empty(max(need, 1), dtype=torch.uint8, device=device)
    from xlstm_cuda.parallel import FusedHeadGather, all_gather_heads
    fused = FusedHeadGather(Bp, Sp, nh_local * world, DV, bf, device) if (world > 1 and NH % world == 0) else None

    def one():
        if fused is not None:   # h tiles stored straight into every rank's [B,S,NH,dv] buffer by the kernel
            y, _ = fused.run(q, k, v, i, f, None, out_proj=w_out.t(), workspace=ws)
            return y
        h, st = ops.mlstm_chunkwise(q, k, v, i, f, None, L, 1e-6, ws)
        hh = h.permute(0, 2, 1, 3).reshape(Bp * Sp, NH * DV)
        return hh @ w_out.t()

    def one_nccl():             # the same with a separate NCCL all-gather, for comparison
        h, st = ops.mlstm_chunkwise(q, k, v, i, f, None, L, 1e-6, ws)
        hh = all_gather_heads(h).permute(0, 2, 1, 3).reshape(Bp * Sp, NH * DV)
        return hh @ w_out.t()

    e = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
    one()
    torch.cuda.synchronize()
    gather_check = None
    if world > 1:
        dist.barrier()
    if fused is not None:
        # the fused gather must leave, on every rank, exactly what a separate all-gather of h leaves
        h_loc, _ = ops.mlstm_chunkwise(q, k, v, i, f, None, L, 1e-6, ws)
        want = all_gather_heads(h_loc).permute(0, 2, 1, 3).reshape(Bp, Sp, NH * DV)
        same = torch.tensor([1 if torch.equal(fused.buf.view(Bp, Sp, NH * DV), want) else 0], device=device)
        dist.all_reduce(same, op=dist.ReduceOp.MIN)
        gather_check = "bit-exact" if int(same.item()) == 1 else "MISMATCH"
        del h_loc, want
        dist.barrier()
    reps = args.prefill_reps
    # a short burst first (the kernel timed alone, clocks still at their maximum) ...
    eb0, eb1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    eb0.record()
    for _ in range(reps):
        h, st = ops.mlstm_chunkwise(q, k, v, i, f, None, L, 1e-6, ws)
    eb1.record()
    torch.cuda.synchronize()
    burst_ms = eb0.elapsed_time(eb1) / reps
    # ... then the figure that counts: about half a second of back-to-back calls, long enough for the 1000 W power
    # cap to settle the SM clock (this kernel runs into it), with clock and throttle reasons sampled alongside
    sustained_calls = max(reps, min(2000, int(0.5e3 / max(burst_ms, 1e-3))))
    with ClockSampler(device.index or 0) as pclk:
        e[0].record()
        for _ in range(sustained_calls):
            h, st = ops.mlstm_chunkwise(q, k, v, i, f, None, L, 1e-6, ws)
        e[1].record()
        torch.cuda.synchronize()
    tail_s = pclk.samples[len(pclk.samples) // 2:]          # second half of the region: the settled clock
    prefill_clocks = {"sm_mhz": (sorted(tail_s)[len(tail_s) // 2] if tail_s else None), "reasons": sorted(pclk.reasons),
                      "sustained_calls": sustained_calls}
    if world > 1:
        dist.barrier()
    e[2].record()
    for _ in range(reps):
        one()
    e[3].record()
    torch.cuda.synchronize()
    nccl_ms = 0.0
    if world > 1:
        one_nccl()
        torch.cuda.synchronize()
        dist.barrier()
        nccl_ms = _time_cuda(torch, one_nccl, reps)
    # the cell with the fused gather alone (no out-projection): the stores to the peers ride inside the kernel
    gat_ms = 0.0
    if fused is not None:
        dist.barrier()
        gat_ms = _time_cuda(torch, lambda: fused.run(q, k, v, i, f, None, out_proj=None, workspace=ws), reps)
    tok_ms, tok_check = None, None
    if fused is not None and Sp % (128 * world) == 0:
        # token-sharded variant: a tile of h goes only to the rank owning its tokens; 1/world of the out-projection each
        from xlstm_cuda.parallel import FusedHeadScatter
        scat = FusedHeadScatter(Bp, Sp, nh_local * world, DV, bf, device)
        scat.run(q, k, v, i, f, None, out_proj=w_out.t(), workspace=ws)
        tok = Sp // world
        same = torch.tensor([1 if torch.equal(scat.buf, fused.buf[:, rank * tok:(rank + 1) * tok]) else 0], device=device)
        dist.all_reduce(same, op=dist.ReduceOp.MIN)
        tok_check = "bit-exact" if int(same.item()) == 1 else "MISMATCH"
        dist.barrier()
        tok_ms = _time_cuda(torch, lambda: scat.run(q, k, v, i, f, None, out_proj=w_out.t(), workspace=ws), reps)
        t_tok = torch.tensor([tok_ms], device=device)
        dist.all_reduce(t_tok, op=dist.ReduceOp.MAX)
        tok_ms = float(t_tok.item())
        del scat
    t_cell = torch.tensor([e[0].elapsed_time(e[1]) / sustained_calls, e[2].elapsed_time(e[3]) / reps, nccl_ms, gat_ms, burst_ms],
                          device=device)
    if world > 1:
        dist.all_reduce(t_cell, op=dist.ReduceOp.MAX)
    cell_ms, full_ms, nccl_ms, cell_ms_gather, burst_ms = (float(x) for x in t_cell)
    tokens = Bp * Sp
    flop = tokens * NH * (4 * DQK * DV + L * (DQK + DV))      # whole job, causal-half count
    byts = tokens * NH * ((2 * DQK + 2 * DV) * 2 + 2 * 2)
    hbm, tf, which = peaks()
    # bytes of h every rank pushes to its peers during the cell (fused gather), over the cell time
    gather_gbs = (world - 1) * Bp * Sp * nh_local * DV * 2 / (cell_ms_gather * 1e-3) / 1e9 if fused is not None else None
    return {"workload": f"mlstm_chunkwise_prefill B={Bp} S={Sp} NH={NH} dqk={DQK} dv={DV} L={L} bf16",
            "parallelism": f"heads sharded x{world}, fused all-gather of h, replicated out-proj", "scaling": "strong",
            "cell_tokens_per_s": tokens / (cell_ms * 1e-3), "cell_ms": cell_ms, "cell_ms_burst": burst_ms, "clocks": prefill_clocks,
            "with_allgather_outproj_tokens_per_s": tokens / (full_ms * 1e-3), "with_allgather_outproj_ms": full_ms,
            "gather": ("fused: kernel epilogue stores h into every rank's buffer over NVLink" if world > 1 else "single rank"),
            "gather_check": gather_check, "gather_gbs_per_rank": gather_gbs, "cell_with_gather_ms": cell_ms_gather,
            "nvlink_peak_gbs_per_direction": 900.0,
            "nccl_allgather_variant_ms": (nccl_ms if world > 1 else None),
            "token_sharded_outproj_ms": tok_ms, "token_sharded_check": tok_check,
            "roofline": {"bound": "tensor", "achieved": flop / world / (cell_ms * 1e-3) / 1e12, "peak": tf,
                         "unit": "TFLOP/s", "frac": flop / world / (cell_ms * 1e-3) / 1e12 / tf,
                         "frac_burst": flop / world / (burst_ms * 1e-3) / 1e12 / burst_tflops(), "peak_burst": burst_tflops(),
                         "hbm_achieved_gbs": byts / world / (cell_ms * 1e-3) / 1e9, "hbm_frac": byts / world / (cell_ms * 1e-3) / 1e9 / hbm,
                         "flop_count": "4*dqk*dv + L*(dqk+dv) per token per head (causal half)", "peak_source": which}}


def _time_cuda(torch, fn, reps):
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    for _ in range(reps):
        fn()
    e1.record()
    torch.cuda.synchronize()
    return e0.elapsed_time(e1) / reps


def run_softcap(torch, ops, device):
    """Logit soft-cap at a 2048-token prefill: [2048, 50304] fp32 (412 MB > L2)."""
    x = torch.randn(2048, 50304, device=device) * 20
    y = torch.empty_like(x)
    ops.softcap(x, 30.0, out=y)
    ms = _time_cuda(torch, lambda: ops.softcap(x, 30.0, out=y), 5)
    hbm, _, which = peaks()
    gbs = 2 * x.numel() * 4 / (ms * 1e-3) / 1e9
    return {"workload": "softcap [2048,50304] fp32 cap=30", "ms": ms,
            "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm, "unit": "GB/s", "frac": gbs / hbm, "peak_source": which}}


def run_glue(torch, ops, device):
    """The HBM-bound kernels either side of the cells at 7B-shaped sizes (bf16, every tensor > L2):
    algorithmic bytes = each input read once + each output written once."""
    hbm, _, which = peaks()
    bf = torch.bfloat16
    out = {}

    def leg(name, workload, nbytes, fn):
        fn()
        ms = _time_cuda(torch, fn, 5)
        gbs = nbytes / (ms * 1e-3) / 1e9
        out[name] = {"workload": workload, "ms": ms, "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm, "unit": "GB/s",
                                                                  "frac": gbs / hbm, "peak_source": which}}

    rows, d = 65536, 4096
    x = torch.randn(rows, d, device=device).to(bf)
    r = torch.randn(rows, d, device=device).to(bf)
    w = torch.ones(d, device=device, dtype=bf)
    leg("rms_norm", f"RMSNorm [{rows},{d}] bf16", 2 * rows * d * 2, lambda: ops.rms_norm(x, w, 1e-6))
    leg("add_rms_norm", f"residual add + RMSNorm [{rows},{d}] bf16", 4 * rows * d * 2, lambda: ops.add_rms_norm(x, r, w, 1e-6))
    del r
    B, NH, S, dv = 4, 8, 8192, 512
    h = torch.randn(B, NH, S, dv, device=device).to(bf)
    og = torch.randn(B, S, NH * dv, device=device).to(bf)
    wv = torch.ones(NH * dv, device=device, dtype=bf)
    leg("mlstm_output_gate", f"per-head RMS norm x sigmoid(ogate), h [{B},{NH},{S},{dv}] bf16", 3 * h.numel() * 2,
        lambda: ops.mlstm_output_gate(h, og, wv, 1e-6))
    del h, og
    rows, f = 16384, 10944
    gu = torch.randn(rows, 2 * f, device=device).to(bf)
    leg("swiglu", f"silu(gate)*up, two column blocks of [{rows},{2 * f}] bf16", 3 * rows * f * 2,
        lambda: ops.swiglu(gu[:, :f], gu[:, f:]))
    del gu
    # single-token Linear (weight streaming): a ring of weight matrices larger than L2, one call per matrix
    for name, N, K, kw in (("linear_token_qkvifo", 12304, 4096, "norm"), ("linear_token_out_proj", 4096, 4096, "res"),
                           ("linear_token_ffn_up_swiglu", 21888, 4096, "swiglu"), ("linear_token_ffn_down", 4096, 10944, "res")):
        ring = max(2, int(2.5e8 // (N * K * 2)) + 1)
        Ws = [torch.randn(N, K, device=device).to(bf) * 0.02 for _ in range(ring)]
        xv = torch.randn(1, K, device=device).to(bf)
        nw = torch.ones(K, device=device, dtype=bf)
        No = N // 2 if kw == "swiglu" else N
        res = torch.randn(1, No, device=device).to(bf)

        def call(kw=kw, Ws=Ws, xv=xv, nw=nw, res=res):
            for W in Ws:
                if kw == "norm":
                    ops.linear_token(W, xv, norm_weight=nw)
                elif kw == "res":
                    ops.linear_token(W, xv, residual=res)
                else:
                    ops.linear_token(W, xv, norm_weight=nw, swiglu_pair=True)

        call()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()      # replayed as a graph, as in the decode loop: no host launch gaps
        with torch.cuda.graph(graph):
            call()
        graph.replay()
        ms = _time_cuda(torch, graph.replay, 5) / ring
        del graph
        gbs = N * K * 2 / (ms * 1e-3) / 1e9
        out[name] = {"workload": f"one token, W [{N},{K}] bf16 ({kw}), ring of {ring} matrices > L2, CUDA graph", "ms": ms,
                     "roofline": {"bound": "hbm", "achieved": gbs, "peak": hbm, "unit": "GB/s", "frac": gbs / hbm,
                                  "peak_source": which}}
        del Ws
    Bc, Sc, C = 32, 4096, 1024
    xc = torch.randn(Bc, Sc, C, device=device).to(bf)
    wc = torch.randn(C, 4, device=device).to(bf)
    bc = torch.zeros(C, device=device, dtype=bf)
    leg("causal_conv1d", f"depthwise causal conv K=4 + SiLU, x [{Bc},{Sc},{C}] bf16", 2 * xc.numel() * 2,
        lambda: ops.causal_conv1d(xc, wc, bc, silu=True))
    return out


def run_slstm(torch, dist, device, world, rank):
    """4 sLSTM blocks with block-diagonal recurrent weights, d=1024, 4 heads x 256,
    B=32 (sharded over the ranks), S=1024, bf16 activations, fp32 state."""
    from xlstm_cuda.blocks import sLSTMBlockDiag

    class Cfg:
        inp_dim, head_dim, head_num, p_factor, norm_eps, gate_soft_cap = 1024, 256, 4, (2.0, 4 / 3), 1e-6, 15.0

    Bs, S = max(1, 32 // world), 1024
    torch.manual_seed(4 + rank)
    blocks = [sLSTMBlockDiag(Cfg()).to(device) for _ in range(4)]
    with torch.no_grad():
        for blk in blocks:
            for lin in (blk.R_i, blk.R_f, blk.R_z, blk.R_o):
                for b in lin.blocks:
                    b.weight.normal_(0.0, 0.02)
            blk.W_f.bias.copy_(torch.linspace(3.0, 6.0, 1024))
            blk.to(torch.bfloat16)
    x = torch.randn(Bs, S, 1024, device=device).to(torch.bfloat16)

    def fwd():
        with torch.inference_mode():
            y = x
            for blk in blocks:
                y, _ = blk(y)
        return y

    fwd()
    ms = _time_cuda(torch, fwd, 3)
    t = torch.tensor([ms], device=device)
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms = float(t.item())
    return {"workload": "4 sLSTM blocks (block-diagonal R), d=1024, 4x256, B=32, S=1024, bf16",
            "parallelism": f"batch-sharded x{world}", "scaling": "strong", "ms": ms,
            "tokens_per_s": Bs * world * S / (ms * 1e-3), "us_per_step_per_block": ms * 1e3 / (4 * S),
            "bound": "latency (sequential through h_{t-1}); includes the input-side GEMMs, norms and FFN of each block"}


def run_model(torch, device, prompt_len, new_tokens):
    """xLSTM-7B-shaped random-init model, prefill then greedy decode, B=1."""
    import tempfile
    from xlstm_cuda.generate import xLSTMRunner
    from xlstm_cuda.utils import XLSTM_7B_CONFIG, write_model_dir
    with tempfile.TemporaryDirectory() as tmp:
        d = write_model_dir(tmp, dict(XLSTM_7B_CONFIG))
        runner = xLSTMRunner(str(d), device=device)
    with torch.no_grad():
        for name, prm in runner.model.named_parameters():
            if prm.dim() >= 2:
                prm.normal_(0.0, 0.02)
            elif name.endswith("fgate_proj.bias"):
                prm.copy_(torch.linspace(3.0, 6.0, prm.numel()))
            elif name.endswith("bias"):
                prm.zero_()
    g = torch.Generator().manual_seed(2)
    ids = torch.randint(0, 50304, (1, prompt_len), generator=g)
    runner.forward(ids)  # warm-up at the timed shape (kernel loads, cuBLAS heuristics and workspaces)
    runner.reset_state()
    e = [torch.cuda.Event(enable_timing=True) for _ in range(4)]
    torch.cuda.synchronize()
    e[0].record()
    logits = runner.forward(ids)
    tok = int(logits[0, -1].argmax())
    e[1].record()
    out = [tok]
    tok = runner.generate_next_token(torch.tensor([[tok]]), temperature=0.0)   # eager step; the next call captures
    out.append(tok)
    tok = int(runner._decode_step_graph(tok).argmax())                          # builds the decode graph (untimed)
    out.append(tok)
    torch.cuda.synchronize()
    e[2].record()
    for _ in range(new_tokens):
        tok = int(runner._decode_step_graph(tok).argmax())
        out.append(tok)
    e[3].record()
    torch.cuda.synchronize()
    e_eager = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
    e_eager[0].record()
    for _ in range(16):
        tok = runner.generate_next_token(torch.tensor([[tok]]), temperature=0.0)
    e_eager[1].record()
    torch.cuda.synchronize()
    eager_ms = e_eager[0].elapsed_time(e_eager[1]) / 16
    pre_ms, dec_ms = e[0].elapsed_time(e[1]), e[2].elapsed_time(e[3])
    n_params = sum(p.numel() for p in runner.model.parameters())
    del runner
    torch.cuda.empty_cache()
    return {"workload": f"xLSTM-7B-shaped random init, B=1, prompt {prompt_len} + {new_tokens} greedy tokens, bf16",
            "params": n_params, "prefill_ms": pre_ms, "prefill_tokens_per_s": prompt_len / (pre_ms * 1e-3),
            "decode_ms_per_token": dec_ms / new_tokens, "decode_tokens_per_s": new_tokens / (dec_ms * 1e-3),
            "decode": "CUDA-graph replay of the single-token step", "decode_eager_ms_per_token": eager_ms,
            "note": "GEMM-bound context number (cuBLAS via torch); the mLSTM cell is ~1 % of prefill FLOPs"}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=4096)
    ap.add_argument("--warmup", type=int, default=64)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--no-prefill", action="store_true")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--prefill-seq", type=int, default=32768)
    ap.add_argument("--prefill-reps", type=int, default=10)
    ap.add_argument("--no-extras", action="store_true", help="skip the soft-cap, sLSTM and full-model sub-benchmarks")
    ap.add_argument("--no-model", action="store_true", help="skip the 7B-shaped full-model run")
    ap.add_argument("--glue-only", action="store_true",
                    help="time only the HBM-bound kernels either side of the cells (a small command to profile)")
    ap.add_argument("--details", metavar="DIR", help="write the per-kernel tables into this folder")
    ap.add_argument("--slstm-only", action="store_true", help="run only the sLSTM stack leg")
    ap.add_argument("--model-only", action="store_true",
                    help="run only the 7B-shaped full-model leg (prefill 2048 + 256 decode tokens)")
    args = ap.parse_args()
    if args.model_only:
        import torch
        sys.path.insert(0, str(ROOT / "xlstm-metal_b200"))
        print(json.dumps({"model": run_model(torch, torch.device("cuda:0"), 2048, 256)}))
        return
    if args.slstm_only:
        import torch
        sys.path.insert(0, str(ROOT / "xlstm-metal_b200"))
        print(json.dumps({"slstm": run_slstm(torch, None, torch.device("cuda:0"), 1, 0)}))
        return
    if args.glue_only:
        import torch
        sys.path.insert(0, str(ROOT / "xlstm-metal_b200"))
        from xlstm_cuda import ops
        print(json.dumps({"glue": run_glue(torch, ops, torch.device("cuda:0"))}))
        return
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
