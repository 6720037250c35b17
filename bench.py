"""Benchmark of the expert forward path (and, by flag, its other workloads) on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference] [--workload NAME]

Prints ONE JSON line.  A "step" is one call of `yamoe_b200.experts` on one batch of seeded
synthetic input.  The default workload is the GPT-OSS-20B-shaped expert layer forward: 4096
tokens, hidden 2880, 32 experts, top-4, bf16 (weights and biases N(0, 0.02), activations N(0, 1),
softmax/top-4 routing without renormalisation).

* `value`      tokens/s with all inputs resident in HBM, timed with CUDA events over K steps,
               barrier + synchronize on both sides, max over ranks.
* `e2e`        the same metric through the public op with HOST inputs: every step copies the step's
               inputs (hidden_states, router_indices, routing_weights) from pinned host memory to
               the device and reads the [T, H] result back, inside the timed region.  Expert
               weights are model state and stay resident.
* `roofline`   gate_up grouped GEMM (the dominant kernel): algorithmic 4*S*H^2 FLOP per launch
               divided by its mean device time, bracketed by CUDA events inside each timed step.
* `cpu_baseline`  the CPU implementation of the reference's PyTorch experts, timed on this box's
               host cores on a bounded sample (rank 0, N=1 only).
* `extra`      N = 1: the decode workloads (T = 1, 4, 16, 64 at the 120B shape) and the backward
               workload (T = 8192), each with its own clock samples.  N > 1: the strong-scaling
               expert-parallel workloads (forward and backward at T = 8192, the skewed 120B prefill)
               for the peer-store and the NCCL all-to-all exchange.
* `--impl reference`  times the CPU implementation with all host threads on the same workload.

With N > 1 (torchrun) the default workload runs EXPERT-PARALLEL and weak-scaled: every rank owns
4096 tokens (global T = 4096 * N), the 32 experts are sharded contiguously E/N per rank, and
token rows travel to the expert owners and back over NVLink (`yamoe_b200.ep.PeerExpertParallel`).
Before the timed loop every rank checks its expert-parallel output against the single-GPU op run
on the same tokens with all experts (`ep_check`); a failed check makes the run exit non-zero.
"""
from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

KEYS = ["hidden_states", "router_indices", "routing_weights", "gate_up_proj", "gate_up_proj_bias",
        "down_proj", "down_proj_bias"]
DEFAULT = "gptoss20b_fwd_t4096"

WORKLOADS = {
    # name: (T, H, E, K, mode)
    "gptoss20b_fwd_t4096": dict(T=4096, H=2880, E=32, K=4, mode="fwd"),
    "gptoss20b_bwd_t8192": dict(T=8192, H=2880, E=32, K=4, mode="bwd"),
    "gptoss120b_decode_t1": dict(T=1, H=2880, E=128, K=4, mode="fwd"),
    "gptoss120b_decode_t4": dict(T=4, H=2880, E=128, K=4, mode="fwd"),
    "gptoss120b_decode_t16": dict(T=16, H=2880, E=128, K=4, mode="fwd"),
    "gptoss120b_decode_t64": dict(T=64, H=2880, E=128, K=4, mode="fwd"),
    # expert-parallel when launched on N > 1 GPUs: tokens sharded by rows, experts contiguously
    "gptoss120b_prefill_t16384": dict(T=16384, H=2880, E=128, K=4, mode="fwd", skew=True, ep=True),
    "gptoss20b_fwd_t8192_ep": dict(T=8192, H=2880, E=32, K=4, mode="fwd", ep=True),
    "gptoss20b_bwd_t8192_ep": dict(T=8192, H=2880, E=32, K=4, mode="bwd", ep=True),
    # forward + backward through autograd: recomputing the forward (as the reference does) / keeping activations
    "gptoss20b_train_t8192": dict(T=8192, H=2880, E=32, K=4, mode="train"),
    "gptoss20b_train_saved_t8192": dict(T=8192, H=2880, E=32, K=4, mode="train", saved=True),
    "readme_fp32_t512": dict(T=512, H=2880, E=8, K=2, mode="fwd", fp32=True),
}

# DRAM bytes (read + write) of one launch of the dominant kernel, from ncu captures of that kernel;
# keyed by workload and output-tile width.  The source names the summary that holds the capture.
TRAFFIC = {
    ("gptoss20b_fwd_t4096", 256): (1.256e9, "ncu dram__bytes_read.sum + dram__bytes_write.sum of one gate_up launch, "
                                            "profiles/umma_pair_gptoss20b_fwd_t4096.md"),
}

# kernels of this library launched by one call (memsets not counted):
#   fwd     routing + row gather + gate_up GEMM + down GEMM + combine
#   bwd     routing + 2 gathers + 5 GEMMs (bias gradients ride along) + cast and routing gradients
#           (one more in either where more than 32768 assignments take the two-launch routing)
#   decode  2 GEMV kernels, or the kernels of fwd where the grouped GEMM takes the call
#   ep_fwd  2 routing + publish + dispatch + 2 GEMMs + signal + combine
#   ep_bwd  2 routing + publish + dispatch + weights + gather + 5 GEMMs + 2 column sums +
#           scalar return + signal + combine + routing gradient
LAUNCHES = {"fwd": 5, "fwd_fp32": 5, "bwd": 9, "train": 14, "decode": 2, "ep_fwd": 8, "ep_bwd": 17}


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            d = json.load(f)
        return dict(bf16_tflops=d["bf16_tflops"], hbm_gbs=d["hbm_gbs"], source="measured")
    return dict(bf16_tflops=1590.0, hbm_gbs=6650.0, source="fallback")


class ClockSampler:
    """nvidia-smi clock / throttle-reason samples taken while the timed region runs."""
    QUERY = ("timestamp,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
             "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
             "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, index: int):
        self.index, self.proc, self.lines, self.reader = index, None, [], None

    def start(self, ready_timeout: float = 20.0):
        """Starts nvidia-smi and waits for its first line: on a box with eight GPUs that takes
        seconds, and a region timed before it would get no samples."""
        import threading
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.QUERY}", "--format=csv,noheader,nounits", "-lms", "50",
                 "-i", str(self.index)], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True, bufsize=1)
        except OSError:
            self.proc = None
            return self

        def pump():
            for line in self.proc.stdout:
                self.lines.append(line)

        self.reader = threading.Thread(target=pump, daemon=True)
        self.reader.start()
        deadline = time.time() + ready_timeout
        while not self.lines and time.time() < deadline and self.proc.poll() is None:
            time.sleep(0.02)
        return self

    def stop(self, window=None):
        """Ends the sampling.  `window` = (t0, t1) in time.time() seconds keeps only the samples whose
        own timestamp lies inside it (the sampler runs from before the warm-up on)."""
        if self.proc is None:
            return dict(sm_mhz=None, sm_max_mhz=None, reasons=["nvidia-smi unavailable"])
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
            self.proc.wait()
        self.reader.join(timeout=5)
        out = "".join(self.lines)
        sm, mx, reasons = [], [], set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        import datetime
        for line in out.strip().splitlines():
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9:
                continue
            if window is not None:
                try:
                    ts = datetime.datetime.strptime(f[0], "%Y/%m/%d %H:%M:%S.%f").timestamp()
                except ValueError:
                    continue
                if not (window[0] - 0.025 <= ts <= window[1] + 0.025):
                    continue
            try:
                sm.append(float(f[1]))
                mx.append(float(f[2]))
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower().startswith("active"):
                    reasons.add(n)
        if not sm:
            return dict(sm_mhz=None, sm_max_mhz=None, reasons=["no samples"])
        return dict(sm_mhz=statistics.median(sm), sm_max_mhz=max(mx), reasons=sorted(reasons), samples=len(sm))


def make_workload(name, weights_on=None, token_seed=None, weights=None):
    """Inputs of a workload.  `token_seed` redraws the routing and the activations (not the
    weights) from another seed: the ranks of a weak-scaled run own different tokens.  `weights`
    (the four weight tensors of an earlier workload of the same shape) skips drawing them again;
    routing and activations are what `make_inputs` draws first from the same seed."""
    import torch
    from oracle.experts_oracle import workloads      # without the package and its libraries
    w = WORKLOADS[name]
    dtype = torch.float32 if w.get("fp32") else torch.bfloat16
    if weights is not None:
        gen = torch.Generator().manual_seed(42)
        idx, dense = workloads.make_routing(w["T"], w["E"], w["K"], gen)
        inp = dict(hidden_states=torch.randn(w["T"], w["H"], generator=gen).to(dtype), router_indices=idx,
                   routing_weights=dense.to(dtype))
        inp.update(zip(KEYS[3:], weights))
    elif name == "readme_fp32_t512":
        inp = workloads.make_readme_inputs(batch=2)
    else:
        big = w["E"] * w["H"] * w["H"] * 3 > 2 ** 31          # 120B-shaped: draw the weights on the device
        inp = workloads.make_inputs(w["T"], w["H"], w["E"], w["K"], seed=42, dtype=dtype,
                                    skew=w.get("skew", False), with_grad=(w["mode"] in ("bwd", "train")),
                                    weights_on=weights_on if big else None)
        if token_seed is not None:
            gen = torch.Generator().manual_seed(token_seed)
            idx, dense = workloads.make_routing(w["T"], w["E"], w["K"], gen)
            inp["router_indices"], inp["routing_weights"] = idx, dense.to(dtype)
            inp["hidden_states"] = torch.randn(w["T"], w["H"], generator=gen).to(dtype)
    return w, inp, dtype


# ---- CPU side: the reference's own PyTorch implementation when a copy travelled with the tree ------
def cpu_impl():
    """(kind, forward_fn, backward_fn).  `oracle/_ref/reference.py` is the reference project's
    own file (placed there by oracle/make_ref.py where the reference tree is present); otherwise the
    CPU restatement in oracle/experts_oracle.py is timed."""
    from oracle import experts_oracle as orc
    path = os.path.join(ROOT, "oracle", "_ref", "reference.py")
    if os.path.exists(path):
        try:
            return "reference", orc.reference_forward_from(path), orc.experts_backward_oracle
        except Exception:      # unusable copy: time the restatement
            pass
    return "port", orc.experts_forward_oracle, orc.experts_backward_oracle


def cpu_reference_time(w, inp, dtype, limit_s=20.0, threads=None):
    """Times the CPU forward (sparse per-expert loop) in the workload's dtype.
    Returns (tokens_per_s, cores, sample description, kind)."""
    import torch
    if threads:
        torch.set_num_threads(threads)
    cores = torch.get_num_threads()
    kind, fwd, bwd = cpu_impl()
    T, E, K = w["T"], w["E"], w["K"]
    args = [inp[k] for k in KEYS]
    cap = 256 if w.get("fp32") else T

    def run():
        t0 = time.perf_counter()
        with torch.no_grad():
            if w["mode"] in ("bwd", "train"):
                bwd(inp["grad_out"], *args, cap, E, K, compute_dtype=dtype)
            if w["mode"] in ("fwd", "train"):
                fwd(*args, cap, E, K, compute_dtype=dtype)
        return time.perf_counter() - t0

    first = run()                               # warm-up, also sizes the sample
    reps = max(1, min(3, int(limit_s / max(first, 1e-3)) - 1))
    best = min([run() for _ in range(reps)] + ([first] if reps == 1 and first > limit_s / 2 else []))
    return (T / best, cores,
            f"full workload ({T} tokens), best of {reps} after 1 warm-up, {dtype}, {cores} threads", kind)


def run_reference(args):
    import torch
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    w, inp, dtype = make_workload(args.workload, weights_on="cuda" if torch.cuda.is_available() else "cpu")
    inp = {k: v.cpu() for k, v in inp.items()}
    torch.set_num_threads(os.cpu_count() or 1)
    T = w["T"]
    args_list = [inp[k] for k in KEYS]
    kind, fwd, bwd = cpu_impl()
    cap = 256 if w.get("fp32") else T

    def step():
        with torch.no_grad():
            if w["mode"] in ("bwd", "train"):
                bwd(inp["grad_out"], *args_list, cap, w["E"], w["K"], compute_dtype=dtype)
            if w["mode"] in ("fwd", "train"):
                fwd(*args_list, cap, w["E"], w["K"], compute_dtype=dtype)

    steps, warm = max(1, args.steps), max(0, args.warmup)     # a forward step is about 0.2 s of CPU time
    for _ in range(warm):
        step()
    t0 = time.perf_counter()
    for _ in range(steps):
        step()
    dt = (time.perf_counter() - t0) / steps
    cores = torch.get_num_threads()
    val = T / dt
    what = ("the reference's own reference.py (GptOssExperts, sparse branch)" if kind == "reference"
            else "CPU port of the reference's PyTorch experts (sparse branch)")
    line = {
        "impl": "reference", "metric": "moe_layer_tokens_per_s", "value": val, "unit": "tokens/s",
        "n_gpus": args.gpus, "steps": steps, "warmup": warm, "ms_per_step": dt * 1e3, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "bf16" if dtype == torch.bfloat16 else "f32",
        "data": "synthetic (seeded, shapes of the reference's own benchmarks)",
        "config": {"workload": args.workload, "tokens": T, "hidden": w["H"], "experts": w["E"], "top_k": w["K"],
                   "pass": w["mode"]},
        "cpu_baseline": {"value": val, "unit": "tokens/s", "cores": cores, "kind": kind,
                         "sample": f"full workload ({T} tokens) per step, {steps} steps, {what}, {cores} threads"},
        "e2e": {"value": val, "unit": "tokens/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def place_near_gpu(local_rank):
    """Pins this process to the CPUs of the GPU's NUMA node (when the allowed CPU set holds any), so
    that the pinned host buffers allocated afterwards are local to the GPU's PCIe root.  Returns a
    small record for the JSON line.  Host-to-device copies from the far socket run at about half
    the rate."""
    info = {"numa_node": None, "cpus_before": len(os.sched_getaffinity(0)), "cpus_after": None}
    info["_allowed"] = os.sched_getaffinity(0)
    try:
        import torch
        props = torch.cuda.get_device_properties(local_rank)
        if hasattr(props, "pci_bus_id"):
            bus = f"{props.pci_domain_id:04x}:{props.pci_bus_id:02x}:{props.pci_device_id:02x}.0"
        else:
            import pynvml
            pynvml.nvmlInit()
            bus = pynvml.nvmlDeviceGetPciInfo(pynvml.nvmlDeviceGetHandleByIndex(local_rank)).busId
            bus = (bus.decode() if isinstance(bus, bytes) else bus).lower()
            if len(bus.split(":")[0]) == 8:
                bus = bus[4:]
        base = f"/sys/bus/pci/devices/{bus}/"
        info["numa_node"] = int(open(base + "numa_node").read())
        local = set()
        for part in open(base + "local_cpulist").read().strip().split(","):
            lo, _, hi = part.partition("-")
            local.update(range(int(lo), int(hi or lo) + 1))
        want = local & os.sched_getaffinity(0)
        if want:
            os.sched_setaffinity(0, want)
    except Exception as exc:   # no NVML, no sysfs, odd bus id: leave the placement alone
        info["note"] = type(exc).__name__
    info["cpus_after"] = len(os.sched_getaffinity(0))
    return info


def copy_bandwidth(torch, nbytes=64 << 20):
    """Pinned host <-> device copy rates (GB/s), each direction alone: context for `e2e`."""
    h = torch.empty(nbytes, dtype=torch.uint8).pin_memory()
    d = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    out = {}
    for name, fn in (("h2d_gbs", lambda: d.copy_(h, non_blocking=True)), ("d2h_gbs", lambda: h.copy_(d, non_blocking=True))):
        fn()
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(5):
            fn()
        b.record()
        torch.cuda.synchronize()
        out[name] = round(5 * nbytes / (a.elapsed_time(b) * 1e-3) / 1e9, 1)
    return out


class Env:
    """Process-wide facts of a run."""

    def __init__(self):
        import torch
        import torch.distributed as dist
        self.torch, self.dist = torch, dist
        self.world = int(os.environ.get("WORLD_SIZE", "1"))
        self.rank = int(os.environ.get("RANK", "0"))
        self.local_rank = int(os.environ.get("LOCAL_RANK", "0"))

    def sync_all(self):
        self.torch.cuda.synchronize()
        if self.world > 1:
            self.dist.barrier()
            self.torch.cuda.synchronize()

    def max_over_ranks(self, x: float) -> float:
        t = self.torch.tensor([x], dtype=self.torch.float64, device="cuda")
        if self.world > 1:
            self.dist.all_reduce(t, op=self.dist.ReduceOp.MAX)
        return t.item()


class Case:
    """One workload set up on this rank: device tensors and the function that runs one step."""

    def __init__(self, env: Env, name: str, ep_mode: str = "peer", weak: bool = False, weights=None):
        import yamoe_b200
        torch = env.torch
        self.env, self.name, self.ep_mode, self.weak = env, name, ep_mode, weak
        world, rank = env.world, env.rank
        self.use_ep = world > 1 and (weak or bool(WORKLOADS[name].get("ep")))
        w, inp, dtype = make_workload(name, weights_on="cuda", weights=weights,
                                      token_seed=(42 + 1000 * rank) if (weak and rank > 0) else None)
        self.w, self.dtype = w, dtype
        T, H, E, K = w["T"], w["H"], w["E"], w["K"]
        self.H, self.E, self.K, self.mode = H, E, K, w["mode"]
        self.cap = 256 if w.get("fp32") else (T * world if weak else T)
        self.decode = T * K <= 256
        self.distinct = int(torch.unique(inp["router_indices"]).numel())
        dev = [inp[k].cuda() for k in KEYS]
        self.weight_bytes = float(sum(dev[i].numel() * dev[i].element_size() for i in (3, 4, 5, 6)))
        self.grad_out = inp["grad_out"].cuda() if w["mode"] in ("bwd", "train") else None
        self.peer_ctx, self.ep_stats, self.ep_check = None, {}, None
        if self.use_ep:
            from yamoe_b200 import ep
            self.ep = ep
            if weak:
                T_total, lo, hi = T * world, 0, T
            else:
                T_total, lo, hi = T, rank * (T // world), (rank + 1) * (T // world)
            local_w = ep.shard_expert_weights(*dev[3:], rank, world)
            inp = {k: (v[lo:hi] if k in KEYS[:3] + ["grad_out"] else v) for k, v in inp.items()}
            if self.grad_out is not None:
                self.grad_out = self.grad_out[lo:hi].contiguous()
            tok = [dev[i][lo:hi].contiguous() for i in range(3)]
            if ep_mode == "peer" and w["mode"] in ("fwd", "bwd"):
                self.peer_ctx = ep.PeerExpertParallel(H, E, K, max_tokens_total=T_total, max_tokens_local=hi - lo,
                                                      dtype=dtype, backward=(w["mode"] == "bwd"))
            if weak:
                self.ep_check = self._check_against_single_gpu(tok, dev[3:], local_w)
            dev = tok + list(local_w)
            torch.cuda.empty_cache()
            T = hi - lo
        self.inp, self.dev, self.T = inp, dev, T
        if w["mode"] == "train":
            for i in (0, 2, 3, 4, 5, 6):
                dev[i].requires_grad_(True)
        self.yamoe = yamoe_b200

    def _check_against_single_gpu(self, tok, full_w, local_w):
        """Expert-parallel output of this rank's tokens against the single-GPU op run on the same
        tokens with all experts; worst rank wins.  bf16 rule of the parity tests."""
        torch, env = self.env.torch, self.env
        import yamoe_b200
        got = self._ep_forward(tok, local_w).float()
        ref = yamoe_b200.experts(*tok, *full_w, self.cap, self.E, self.K).float()
        torch.cuda.synchronize()
        status = self.peer_ctx.status() if self.peer_ctx is not None else 0
        diff = (got - ref).abs()
        rel_l2 = float(diff.norm() / ref.norm().clamp_min(1e-30))
        ratio = float((diff / (2e-2 * ref.abs() + 2e-2 * ref.abs().max())).max())
        rel_l2, ratio, status = env.max_over_ranks(rel_l2), env.max_over_ranks(ratio), int(env.max_over_ranks(status))
        return {"rel_l2": rel_l2, "max_ratio": ratio, "device_status": status,
                "ok": bool(rel_l2 <= 1e-2 and ratio <= 1.0 and status == 0),
                "rule": "|ep - single| <= 2e-2*|single| + 2e-2*max|single| and rel-L2 <= 1e-2, max over ranks; "
                        "single = yamoe_b200.experts on this rank's tokens with all experts resident"}

    def _ep_forward(self, tok, local_w):
        if self.peer_ctx is not None:
            return self.peer_ctx.forward(*tok, *local_w, self.cap)
        return self.ep.ep_experts(*tok, *local_w, self.cap, self.E, self.K, stats=self.ep_stats)

    def run(self, tok=None, grad=None):
        """One step on device-resident inputs (`tok` replaces the three per-token tensors)."""
        dev, cap, E, K, w = self.dev, self.cap, self.E, self.K, self.w
        a = list(tok) if tok is not None else dev[:3]
        g = grad if grad is not None else self.grad_out
        if self.use_ep and w["mode"] == "bwd":
            if self.peer_ctx is not None:
                return self.peer_ctx.backward(g, *a, *dev[3:], cap)[0]
            return self.ep.ep_experts_backward(g, *a, *dev[3:], cap, E, K)[0]
        if self.use_ep:
            return self._ep_forward(a, dev[3:])
        if w["mode"] == "bwd":
            return self.yamoe.experts_backward(g, *a, *dev[3:], cap, E, K)[0]
        if w["mode"] == "train":
            if tok is None:
                for i in (0, 2, 3, 4, 5, 6):
                    dev[i].grad = None
                out = self.yamoe.experts_autograd(*dev, cap, E, K, True, save_activations=bool(w.get("saved")))
                out.backward(g)
                return dev[0].grad
            x = a[0].detach().requires_grad_(True)
            out = self.yamoe.experts_autograd(x, a[1], a[2], *dev[3:], cap, E, K, False,
                                              save_activations=bool(w.get("saved")))
            out.backward(g)
            return x.grad
        return self.yamoe.experts(*a, *dev[3:], cap, E, K)

    def rows_processed(self):
        """Rows this rank's grouped GEMMs process per step."""
        if self.use_ep and self.peer_ctx is not None:
            lay_counts = self.peer_ctx.ctrl.view(-1)[: 2 * self.env.world * self.E].view(2, self.env.world, self.E)
            per = self.E // self.env.world
            epoch = int(self.peer_ctx.state[0])
            return int(lay_counts[epoch & 1, :, self.env.rank * per:(self.env.rank + 1) * per].sum().item())
        if self.use_ep:
            return int(self.ep_stats.get("rows_received", self.T * self.K))
        return self.T * self.K

    def uses_gemv(self):
        """The library's rule for decode-sized bf16 calls of these widths (gemv_preferred in csrc/gemv.cuh)."""
        S = self.T * self.K
        return self.decode and S <= min(256, 4 * self.E) and (S < self.E or S * self.H <= 80 * 1024)

    def launches(self):
        if self.uses_gemv():
            return LAUNCHES["decode"]
        if self.use_ep and self.peer_ctx is not None:
            return LAUNCHES["ep_" + self.mode]
        if self.mode == "fwd" and self.w.get("fp32"):
            return LAUNCHES["fwd_fp32"]
        saved = self.mode == "train" and self.w.get("saved")     # its backward skips routing, gather and gate_up
        routings = 2 if self.mode == "train" and not saved else 1
        return LAUNCHES[self.mode] - (3 if saved else 0) + (routings if self.T * self.K > 32768 else 0)


def time_resident(case: Case, steps: int, warmup: int, sample_clocks: bool = True):
    """Device-resident timing of `steps` steps: ms per step (max over ranks), the gate_up GEMM's
    device time inside every step (forward workloads), clock samples taken meanwhile."""
    from yamoe_b200 import _lib
    env, torch = case.env, case.env.torch
    L = _lib.lib()
    sampler = ClockSampler(env.local_rank).start() if sample_clocks else None
    for _ in range(warmup):
        case.run()
    env.sync_all()
    pairs = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
    for a, b in pairs:
        a.record(); b.record()           # forces creation of the underlying cudaEvent_t
    torch.cuda.synchronize()
    t_start, t_stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    env.sync_all()
    wall0 = time.time()
    eager_us = None
    if case.decode:
        # Touched weights (0.2 - 5.8 GB) are comparable to the 126 MB L2 at T=1: flush it between
        # steps and time every step by itself.  A call is ~50 us of GPU work but more than that of
        # Python dispatch, so the whole-call time is taken from a CUDA-graph replay of the same call
        # (the op issues only kernel launches); the gate_up kernel time comes from a second,
        # ungraphed pass with the stage events, which also gives the eager (ungraphed) call time.
        flush_buf = torch.empty(256 * 1024 * 1024, dtype=torch.uint8, device="cuda")
        flush_read = torch.zeros(64 * 1024 * 1024, dtype=torch.float32, device="cuda")
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            case.run()
        env.sync_all()
        step_ev = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in pairs]
        for s0, s1 in step_ev:
            flush_buf.fill_(1)             # 256 MB written: evicts the workload from the 126 MB L2 ...
            flush_read.sum()               # ... then 256 MB read: pushes the dirty lines out, so the timed
                                           # step does not pay for their write-back
            s0.record()
            graph.replay()
            s1.record()
        env.sync_all()
        ms_total = sum(s0.elapsed_time(s1) for s0, s1 in step_ev)
        eager = []
        for a, b in pairs:
            flush_buf.fill_(1)
            flush_read.sum()
            torch.cuda.synchronize()
            L.yamoe_b200_set_stage_events(a.cuda_event, b.cuda_event, 1)
            t0 = time.perf_counter()
            case.run()
            torch.cuda.synchronize()
            eager.append((time.perf_counter() - t0) * 1e6)
        eager_us = statistics.median(eager)
        env.sync_all()
        if sampler is not None:
            # the timed steps last microseconds: keep replaying the same call, untimed, for a few
            # sampling periods so that the clock record has samples under this load
            t_end = time.time() + 0.3
            while time.time() < t_end:
                for _ in range(50):
                    graph.replay()
                torch.cuda.synchronize()
        del flush_buf, flush_read
    else:
        # Expert-parallel steps launch the gate_up GEMM next to the dispatch kernel; an event record
        # between the two would undo that overlap, so there the GEMM's own time is taken from an
        # untimed repeat of the loop right after the timed one.
        stage_inside = not case.use_ep
        t_start.record()
        for a, b in pairs:
            if stage_inside:
                L.yamoe_b200_set_stage_events(a.cuda_event, b.cuda_event, 1)
            case.run()
        t_stop.record()
        env.sync_all()
        ms_total = t_start.elapsed_time(t_stop)
        if not stage_inside and case.mode == "fwd":
            for a, b in pairs:
                L.yamoe_b200_set_stage_events(a.cuda_event, b.cuda_event, 1)
                case.run()
            env.sync_all()
    L.yamoe_b200_set_stage_events(None, None, 0)
    wall1 = time.time()
    gemm_ms = [a.elapsed_time(b) for a, b in pairs] if case.mode == "fwd" else []
    ms_step = env.max_over_ranks(ms_total) / steps
    clocks = None
    if sampler is not None:
        if ms_step * steps < 250.0 and not case.decode:
            # the timed region was shorter than a few sampling periods: repeat the same loop, untimed
            # (the same number of steps on every rank), and take the clocks from both together
            for _ in range(int(300.0 / max(ms_step, 1e-3)) + 1):
                case.run()
            env.sync_all()
            clocks = dict(sampler.stop((wall0, time.time())),
                          note="timed region shorter than 0.25 s: sampled over it and an untimed repeat of the same "
                               "loop right after it")
        else:
            clocks = sampler.stop((wall0, wall1))
            if case.decode:
                clocks["note"] = "sampled over the timed steps and 0.3 s of untimed replays of the same call after them"
    status = case.peer_ctx.status() if case.peer_ctx is not None else 0
    return dict(ms_step=ms_step, gemm_ms=gemm_ms, clocks=clocks, eager_us=eager_us, device_status=status)


def time_e2e(case: Case, steps: int, warmup: int, eager: bool):
    """End to end: host inputs in, host result out, every step.  Returns (tokens/s over all ranks,
    h2d bytes, d2h bytes, description of the pipeline)."""
    env, torch = case.env, case.env.torch
    w, T, H, dtype = case.w, case.T, case.H, case.dtype
    host_in = [case.inp[k].pin_memory() for k in KEYS[:3]]
    host_out = torch.empty(T, H, dtype=dtype).pin_memory()
    host_go = case.inp["grad_out"].pin_memory() if w["mode"] in ("bwd", "train") else None
    h2d = sum(x.numel() * x.element_size() for x in host_in) + (host_go.numel() * host_go.element_size() if host_go is not None else 0)
    d2h = host_out.numel() * host_out.element_size()

    # Three streams pipeline consecutive steps: while step i computes, step i+1's inputs come in and
    # step i-1's result goes out (PCIe is full duplex).  Every step still copies its own inputs from
    # pinned host memory and its own result back.  Expert-parallel steps pipeline the same way: their
    # calls stay in order on the compute stream (all calls of a rank share its peer-writable
    # buffers), only the copies of the neighbouring steps move to the other two streams.
    pipelined = True
    cur = torch.cuda.current_stream()
    s_in, s_out = (torch.cuda.Stream(), torch.cuda.Stream()) if pipelined else (cur, cur)
    host_outs = [host_out, torch.empty_like(host_out).pin_memory()]
    in_ready = [torch.cuda.Event() for _ in range(2)]
    comp_done = [torch.cuda.Event() for _ in range(2)]
    out_done = [torch.cuda.Event() for _ in range(2)]
    keep = [None, None]
    dev_in = [[torch.empty_like(x, device="cuda") for x in host_in] for _ in range(2)]
    dev_go = [torch.empty_like(host_go, device="cuda") if host_go is not None else None for _ in range(2)]

    def e2e_step(i):
        b = i % 2
        with torch.cuda.stream(s_in):
            s_in.wait_event(comp_done[b])                 # device input buffers of step i-2 are free
            a, g = dev_in[b], dev_go[b]
            for d_, h_ in zip(a, host_in):
                d_.copy_(h_, non_blocking=True)
            if g is not None:
                g.copy_(host_go, non_blocking=True)
            in_ready[b].record(s_in)
        cur.wait_event(in_ready[b])
        out = case.run(a, g)
        comp_done[b].record(cur)
        with torch.cuda.stream(s_out):
            s_out.wait_event(comp_done[b])
            s_out.wait_event(out_done[b])                  # host buffer of step i-2 has been written
            host_outs[b].copy_(out, non_blocking=True)
            out_done[b].record(s_out)
        out.record_stream(s_out)
        keep[b] = out

    # Forward workloads on one GPU replay each step as a CUDA graph (host->device copies, the op
    # called through the public API, device->host copy): the host then issues one launch per step and
    # cannot fall behind the GPU.  Three graphs with their own buffers take turns on three streams,
    # so consecutive steps overlap as in the eager pipeline.  Anything else keeps the eager pipeline.
    graphs = None
    if not case.use_ep and w["mode"] == "fwd" and not eager:
        try:
            graphs = []
            g_streams = [s_in, s_out, torch.cuda.Stream()]
            g_in = dev_in + [[torch.empty_like(x, device="cuda") for x in host_in]]
            g_out = host_outs + [torch.empty_like(host_out).pin_memory()]
            for b in range(3):
                gph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(gph):
                    for d_, h_ in zip(g_in[b], host_in):
                        d_.copy_(h_, non_blocking=True)
                    g_out[b].copy_(case.run(g_in[b], None), non_blocking=True)
                graphs.append(gph)
        except Exception as exc:           # capture not possible here: time the eager pipeline
            sys.stderr.write(f"bench.py: CUDA-graph capture of the end-to-end step failed ({exc!r}); eager pipeline\n")
            graphs = None
            torch.cuda.synchronize()

    def graph_step(i):
        with torch.cuda.stream(g_streams[i % 3]):
            graphs[i % 3].replay()

    step_fn = graph_step if graphs is not None else e2e_step
    for i in range(min(warmup, 3) if graphs is None else 6):
        step_fn(i)
    env.sync_all()
    e_start, e_stop = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e_start.record()
    s_in.wait_event(e_start)
    s_out.wait_event(e_start)
    if graphs is not None:
        g_streams[2].wait_event(e_start)
    for i in range(steps):
        step_fn(i)
    cur.wait_stream(s_in)
    cur.wait_stream(s_out)
    if graphs is not None:
        cur.wait_stream(g_streams[2])
    e_stop.record()
    env.sync_all()
    ms = env.max_over_ranks(e_start.elapsed_time(e_stop))
    value = env.world * T / (ms / steps * 1e-3)
    how = ("every step is one CUDA-graph replay of (host->device copies, op, device->host copy); "
           "three such graphs take turns on three streams, so consecutive steps overlap"
           if graphs is not None else
           "host->device copy, op and device->host copy of consecutive steps overlap on three streams"
           if pipelined else "one stream, copies and op in sequence")
    return value, h2d, d2h, how


def roofline_of(case: Case, res, peaks, rows):
    """`roofline` object of the JSON line for the dominant kernel of a forward workload."""
    torch = case.env.torch
    gemm_ms, H = res["gemm_ms"], case.H
    if not gemm_ms:
        return None
    mean_ms = sum(gemm_ms) / len(gemm_ms)
    if case.decode:
        kbytes = case.distinct * (H * 2 * H * 2 + 2 * H * 2)          # gate_up weights + bias of the touched experts
        achieved = kbytes / (mean_ms * 1e-3) / 1e9
        return {"bound": "hbm", "kernel": ("gemv_kernel" if case.uses_gemv() else "umma_pair_kernel") + "<gate_up + bias + clamped SwiGLU>",
                "achieved": achieved, "peak": peaks["hbm_gbs"], "unit": "GB/s",
                "frac": achieved / peaks["hbm_gbs"], "traffic": None, "kernel_ms": mean_ms,
                "peak_source": peaks["source"] + " (copy bandwidth)",
                "frac_of_nominal_8000": achieved / 8000.0, "distinct_experts": case.distinct,
                "whole_op_gbs": case.distinct * 49783680 / (res["ms_step"] * 1e-3) / 1e9}
    if case.dtype == torch.float32:
        # fp32 runs as six bf16 products of three-part operands on the tensor cores
        achieved = 4.0 * rows * H * H / (mean_ms * 1e-3) / 1e12
        peak = peaks["bf16_tflops"] / 6
        return {"bound": "tensor", "kernel": "umma_f32_kernel<gate_up + bias + clamped SwiGLU> (three bf16 parts)",
                "achieved": achieved, "peak": peak, "unit": "TFLOP/s", "frac": achieved / peak,
                "traffic": None, "kernel_ms": mean_ms,
                "peak_source": peaks["source"] + " (burst bf16 matmul, a sixth of it)"}
    achieved = 4.0 * rows * H * H / (mean_ms * 1e-3) / 1e12
    tile_n = int(os.environ.get("YAMOE_B200_BN", "256") or 256)
    traffic, source = TRAFFIC.get((case.name, tile_n), (None, None)) if not case.use_ep else (None, None)
    out = {"bound": "tensor", "kernel": ("umma_gemm_kernel" if case.use_ep else "umma_pair_kernel") + "<gate_up + bias + clamped SwiGLU>",
           "achieved": achieved, "peak": peaks["bf16_tflops"], "unit": "TFLOP/s",
           "frac": achieved / peaks["bf16_tflops"], "traffic": traffic, "traffic_source": source,
           "kernel_ms": mean_ms, "peak_source": peaks["source"] + " (burst bf16 matmul)",
           "frac_of_nominal_2250": achieved / 2250.0, "rows": rows}
    if case.use_ep:
        out["timed"] = ("in an untimed repeat of the timed loop: the kernel is launched next to the dispatch kernel "
                        "and an event between the two would undo the overlap; its time includes waiting for rows")
    return out


def extras_single_gpu(env: Env, peaks):
    """Decode (T = 1, 4, 16, 64) and backward (T = 8192) under the same clock, one GPU."""
    out = {"decode": [], "bwd": None}
    weights = None
    for T in (1, 4, 16, 64):
        case = Case(env, f"gptoss120b_decode_t{T}", weights=weights)
        weights = case.dev[3:]               # 12.7 GB of expert weights: drawn once
        res = time_resident(case, 40, 5)
        roof = roofline_of(case, res, peaks, case.T * case.K)
        out["decode"].append({"T": T, "us": res["ms_step"] * 1e3, "distinct_experts": case.distinct,
                              "whole_op_gbs": roof["whole_op_gbs"],
                              "frac_of_measured_hbm": roof["whole_op_gbs"] / peaks["hbm_gbs"],
                              "gate_up_frac": roof["frac"], "eager_call_us": res["eager_us"],
                              "clocks": res["clocks"]})
        del case
    del weights
    env.torch.cuda.empty_cache()
    case = Case(env, "gptoss20b_bwd_t8192")
    res = time_resident(case, 10, 3)
    S = case.T * case.K
    tf = 16.0 * S * case.H * case.H / (res["ms_step"] * 1e-3) / 1e12
    out["bwd"] = {"workload": "gptoss20b_bwd_t8192", "ms": res["ms_step"], "tflops": tf,
                  "frac": tf / peaks["bf16_tflops"], "algorithmic_flops": "16*S*H^2", "clocks": res["clocks"]}
    del case
    env.torch.cuda.empty_cache()
    return out


def extras_multi_gpu(env: Env):
    """Strong-scaling expert-parallel workloads, peer-store and NCCL all-to-all exchange."""
    out = []
    for name in ("gptoss20b_fwd_t8192_ep", "gptoss20b_bwd_t8192_ep", "gptoss120b_prefill_t16384"):
        for mode in ("peer", "nccl"):
            case = Case(env, name, ep_mode=mode)
            res = time_resident(case, 10 if case.mode == "bwd" else 20, 3, sample_clocks=False)
            rows = case.rows_processed()
            out.append({"workload": name, "ep_mode": mode, "ms_per_step": res["ms_step"],
                        "tokens_per_s": WORKLOADS[name]["T"] / (res["ms_step"] * 1e-3),
                        "rank0_row_share": rows / float(WORKLOADS[name]["T"] * case.K),
                        "device_status": res["device_status"]})
            del case
            env.torch.cuda.empty_cache()
            env.sync_all()
    return out


def run_ours(args):
    env = Env()
    torch, dist = env.torch, env.dist
    world, rank, local_rank = env.world, env.rank, env.local_rank
    if not torch.cuda.is_available():
        raise RuntimeError("bench.py needs a CUDA device; yamoe_b200 has no CPU fallback")
    torch.cuda.set_device(local_rank)
    host_place = place_near_gpu(local_rank)
    allowed_cpus = host_place.pop("_allowed")
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local_rank))

    weak_ep = world > 1 and args.workload == DEFAULT
    case = Case(env, args.workload, ep_mode=args.ep_mode, weak=weak_ep)
    w, T, H, E, K, dtype = case.w, case.T, case.H, case.E, case.K, case.dtype
    if case.ep_check is not None and not case.ep_check["ok"]:
        if rank == 0:
            print(json.dumps({"metric": "moe_layer_tokens_per_s", "value": None, "n_gpus": world,
                              "ep_check": case.ep_check, "error": "expert-parallel output differs from the single-GPU op"}),
                  flush=True)
        dist.destroy_process_group()
        sys.exit(1)

    res = time_resident(case, args.steps, args.warmup)
    ms_step = res["ms_step"]
    value = world * T / (ms_step * 1e-3)
    rows = case.rows_processed()
    e2e_value, h2d, d2h, how = time_e2e(case, args.steps, args.warmup, args.eager_e2e)

    line = None
    if rank == 0:
        peaks = measured_peaks()
        if case.use_ep:
            exch = ("dispatch + combine as NVLink peer stores issued by the dispatch kernel and by the down GEMM's "
                    "epilogue, counts and phase boundaries as flags in symmetric memory, no collective call, no host sync"
                    if case.peer_ctx is not None else
                    "NCCL all-to-all dispatch + combine; rank-0 rows sent/received "
                    f"{case.ep_stats.get('rows_sent')}/{case.ep_stats.get('rows_received')}")
            par = (f"ep{world} (" + (f"{T} tokens per rank, " if weak_ep else "tokens sharded by rows, ")
                   + f"experts sharded contiguously {E // world} per rank; {exch})")
        else:
            par = f"dp{world} (token shards, replicated experts, no collective)"
        line = {
            "metric": "moe_layer_tokens_per_s", "value": value, "unit": "tokens/s", "n_gpus": world,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak" if (weak_ep or not case.use_ep) else "strong", "vs_baseline": None,
            "dtype": "bf16" if dtype == torch.bfloat16 else "f32",
            "data": "synthetic (seeded, shapes of the reference's own benchmarks)",
            "config": {"workload": args.workload, "tokens": T * world if weak_ep else w["T"], "tokens_per_rank": T,
                       "hidden": H, "experts": E, "top_k": K, "pass": w["mode"], "expert_capacity": case.cap,
                       "parallelism": par,
                       "l2": ("L2 flushed (256 MB write, then 256 MB read to drain the dirty lines) between steps; each step is a CUDA-graph replay of the op call timed by its own events" if case.decode
                              else f"expert weights ({case.weight_bytes / 1e9:.1f} GB) exceed the 126 MB L2; no flush")},
            "e2e": {"value": e2e_value, "unit": "tokens/s", "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "pipeline": how, "host": dict(host_place, **copy_bandwidth(torch))},
            "gpu_launches": args.steps * case.launches(),
            "clocks": res["clocks"],
            "achieved_tflops_whole_op": {"fwd": 6, "bwd": 16, "train": 22}[w["mode"]] * rows * H * H / (ms_step * 1e-3) / 1e12,
            "device_status": res["device_status"],
        }
        if case.ep_check is not None:
            line["ep_check"] = case.ep_check
        roof = roofline_of(case, res, peaks, rows)
        if roof is not None:
            line["roofline"] = roof
        if case.decode:
            line["eager_call_us"] = res["eager_us"]
    cpu_inp = {k: t.cpu() for k, t in case.inp.items()} if (rank == 0 and world == 1 and not args.no_cpu_baseline) else None
    del case
    torch.cuda.empty_cache()

    if not args.no_extras and args.workload == DEFAULT:
        try:
            extra = extras_single_gpu(env, measured_peaks()) if world == 1 else extras_multi_gpu(env)
        except Exception as exc:       # the headline numbers stand; say what went wrong
            extra = {"error": repr(exc)}
        if line is not None:
            line["extra"] = extra
    if line is not None:
        if cpu_inp is not None:
            os.sched_setaffinity(0, allowed_cpus)      # the CPU baseline may use every core again
            v, cores, sample, kind = cpu_reference_time(w, cpu_inp, dtype)
            line["cpu_baseline"] = {"value": v, "unit": "tokens/s", "cores": cores, "kind": kind, "sample": sample}
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    # A few dozen steps run at the boost clock; hundreds of back-to-back steps settle at the clock the
    # 1 kW power cap allows (about 1.5 GHz here, 15-20 % more time per step).
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default=DEFAULT, choices=sorted(WORKLOADS))
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-extras", action="store_true",
                    help="skip the `extra` measurements that follow the default workload")
    ap.add_argument("--eager-e2e", action="store_true",
                    help="time the end-to-end leg with eager calls on three streams instead of CUDA-graph replays")
    ap.add_argument("--ep-mode", default="peer", choices=["peer", "nccl"],
                    help="exchange used by the expert-parallel workloads on N > 1 GPUs")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
