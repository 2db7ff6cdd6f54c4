#!/usr/bin/env python
"""Benchmark of the ring-Ising structured-adjoint engine on B200.

Workload (one "step"): one energy_and_grad call of the ring-Ising VQE ansatz,
n=28 qubits, L=4 layers, h=J=1, complex128 statevector, angles seeded uniform
in [0, 2pi) (synthetic; the reference measures no dataset).  A circuit of so few
layers is contracted along the ring (rsv_ring.cu): its working set, a few MB,
fits L2, so a buffer larger than L2 is written between the timed steps, and the
calls go on behind them until the clocks have been sampled under load.  The HBM
roofline is that of the tile passes on the same circuit (``roofline.schedule``),
which hold three state vectors of 16*2^n bytes.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

``value`` is whole-job energy_and_grad/s with the parameters already in HBM
(device entry point, CUDA events, max over ranks); ``e2e`` is the same metric
through the public host API (host parameters in, host energy+gradient out,
copies inside the timed region).  ``--impl reference`` times the CPU
reference arm: the reference has no CPU implementation of this path, so the
arm runs the repository's CPU restatement of it (oracle/, OpenMP, every host
thread), one full energy_and_grad of the same n=28, L=4 circuit per step.
Beside it the arm records the reference's own CUDA code, rebuilt for sm_100a
from its sources (oracle/_ref), timed on the same GPU at n=28 and n=30, L=4
(``reference_gpu``).  With --gpus N > 1 (under torchrun) every rank evaluates
its own independent circuit (replicas, weak scaling; the path has no exchange
step).

Two further sections ride on the same JSON line: ``batch`` -- 4096 circuits
of uneven size per step through the batched kernels (one CUDA graph replay;
with N ranks a cost-balanced shard per rank plus a final all-gather), against a
per-circuit loop of the single-circuit entry point;
``warm_start`` -- plain VQE from seeded random angles vs from the warm-start
network's prediction at n=16, L=6 on 128 held-out fields (N=1 only);
``adam_n12_l3`` and ``autograd_n20_l8`` -- torch Adam loops through the
autograd Function at n=12, L=3 (20 steps) and n=20, L=8 (100 steps), with the
bare device entry point and the CPU oracle beside them (N=1 only);
``sharded`` -- one circuit split over 2^g ranks (gpu_simulation_b200/
sharded.py): with N > 1, n=30 over the N ranks (NCCL all-to-alls), against
the single-GPU engine's energy and gradient; with N = 1, the headline circuit
over two virtual ranks on the one GPU, and the per-rank kernels of an n=33
circuit over 8 ranks at their full shard size (2^30 amplitudes), timed alone.
"""

from __future__ import annotations

import argparse
import json
import os
import statistics
import subprocess
import sys
import tempfile
import time
from pathlib import Path

import numpy as np

ROOT = Path(__file__).resolve().parent
sys.path.insert(0, str(ROOT))

METRIC = "energy_and_grad/s at 24-30 qubits and % HBM peak; batched grads/s vs plain"
UNIT = "energy_and_grad/s"
FALLBACK_HBM_GBS = 6650.0


def parse_args():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=("ours", "reference"), default="ours")
    ap.add_argument("--qubits", type=int, default=28)
    ap.add_argument("--layers", type=int, default=4)
    ap.add_argument("--field", type=float, default=1.0)
    ap.add_argument("--no-sweep", action="store_true", help="skip the n=20/24/30 device-timed sweep")
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline sample")
    ap.add_argument("--no-batch", action="store_true", help="skip the 4096-circuit batched section")
    ap.add_argument("--no-warmstart", action="store_true", help="skip the warm-start section")
    ap.add_argument("--no-small", action="store_true", help="skip the n=12 Adam and n=20 autograd sections")
    ap.add_argument("--no-autotune", action="store_true", help="keep the planner's default plan (no autotune)")
    ap.add_argument("--no-sharded", action="store_true", help="skip the sharded single-circuit section")
    ap.add_argument("--shard-rank-kernels", default=None, metavar="N,G",
                    help="only time one rank's sharded kernels for N qubits over 2^G ranks, print them, exit")
    ap.add_argument("--no-reference-gpu", action="store_true",
                    help="reference arm: skip timing the reference's sm_100a rebuild on the GPU")
    return ap.parse_args()


def measured_peaks():
    p = ROOT / "MEASURED_PEAKS.json"
    if p.exists():
        d = json.loads(p.read_text())
        return float(d["hbm_gbs"]), "measured (MEASURED_PEAKS.json hbm_gbs)"
    return FALLBACK_HBM_GBS, "fallback 6.65 TB/s"


def workload_params(n, L, seed):
    return np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, 2 * n * L)


# --------------------------------------------------------------------- clocks
class ClockSampler:
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self):
        self.proc = None
        self.path = None

    def start(self):
        fd, self.path = tempfile.mkstemp(prefix="clocks_", suffix=".csv")
        os.close(fd)
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", f"--query-gpu={self.FIELDS}", "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=open(self.path, "w"), stderr=subprocess.DEVNULL)
        except OSError:
            self.proc = None

    def stop(self, gpu_indices):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        rows = []
        for line in Path(self.path).read_text().splitlines():
            parts = [x.strip() for x in line.split(",")]
            if len(parts) < 9:
                continue
            try:
                if int(parts[0]) not in gpu_indices:
                    continue
                rows.append(parts)
            except ValueError:
                continue
        os.unlink(self.path)
        if not rows:
            return None
        sm = [float(r[1]) for r in rows if r[1].replace(".", "").isdigit()]
        smax = [float(r[2]) for r in rows if r[2].replace(".", "").isdigit()]
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        reasons = sorted({names[i] for r in rows for i in range(4) if r[5 + i] == "Active"})
        under = [x for x in sm if smax and x > 0.5 * max(smax)] or sm
        return {"sm_mhz": statistics.median(under) if under else None,
                "sm_max_mhz": max(smax) if smax else None, "reasons": reasons, "samples": len(rows)}


# ------------------------------------------------------------- CPU baselines
def cpu_call(n, L, field, seed=7):
    """One full energy_and_grad of the workload on the oracle (the CPU
    restatement, every host thread); returns (seconds, threads, energy)."""
    import oracle

    threads = oracle.set_num_threads(0)
    p = workload_params(n, L, seed)
    t0 = time.perf_counter()
    e, _ = oracle.energy_and_grad(n, L, field, p)
    return time.perf_counter() - t0, threads, float(e)


def reference_gpu_times(L, field, sizes=(28, 30), warmup=2, reps=5):
    """The reference's own structured_adjoint CUDA code (its extension rebuilt
    for sm_100a from its sources into oracle/_ref), timed on this GPU through
    its public call energy_and_grad(params, True, False): host parameters in,
    energy and gradient out, synchronous, so a wall-clock interval per call is
    its end-to-end time.  Seed-7 angles as the workload."""
    from tests.refmod import load_reference_module

    ref = load_reference_module()
    if ref is None:
        return {"unavailable": "oracle/_ref was not built (make -C oracle ref)"}
    import gc

    out = {"what": "reference cpp/*.cu rebuilt for sm_100a (structured_adjoint, chunk width 8), "
                   "same GPU, median ms per energy_and_grad call (host params in, host results out)"}
    for n in sizes:
        p = workload_params(n, L, 7)
        try:
            rb = ref.RingIsingCudaBackend(n, L, field, "structured_adjoint", 8, False)
            for _ in range(warmup):
                r = rb.energy_and_grad(p, True, False)
            times = []
            for _ in range(reps):
                t0 = time.perf_counter()
                r = rb.energy_and_grad(p, True, False)
                times.append(time.perf_counter() - t0)
            ms = statistics.median(times) * 1e3
            out[f"n={n}"] = {"ms_per_call": ms, "energy_and_grad_per_s": 1000.0 / ms,
                             "energy": float(r["energy"]), "calls_timed": reps}
            del rb, r
            gc.collect()
        except Exception as exc:  # report, do not hide
            out[f"n={n}"] = {"error": str(exc)}
    return out


def run_reference_arm(args, rank, world):
    if rank != 0:
        return 0
    n, L = args.qubits, args.layers
    per_step = []
    energy = None
    for i in range(args.warmup + args.steps):
        t, threads, energy = cpu_call(n, L, args.field)
        if i >= args.warmup:
            per_step.append(t)
    sec = statistics.median(per_step)
    value = 1.0 / sec
    sample = (f"the full workload: one energy_and_grad at n={n}, L={L} per step on the CPU restatement "
              f"(oracle/, {threads} threads); median of {args.steps} steps after {args.warmup} warm-up steps")
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": sec * 1e3,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
        "data": "synthetic: seeded U[0,2pi) angles",
        "config": {"workload": f"structured_adjoint energy_and_grad n={n} L={L} h={args.field}",
                   "num_qubits": n, "num_layers": L, "field": args.field, "parallelism": "replicas"},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": threads, "kind": "port", "sample": sample},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "energy": energy,
    }
    if not args.no_reference_gpu:
        line["reference_gpu"] = reference_gpu_times(L, args.field)
    print(json.dumps(line), flush=True)
    return 0


def pennylane_baseline():
    """PennyLane lightning.qubit with adjoint differentiation on the host
    cores, the reported CPU baseline for the n=12, L=3 circuit, when PennyLane
    is installed; otherwise the reason it is not measured."""
    try:
        import pennylane as qml  # noqa: F401
    except Exception as exc:
        return {"unavailable": f"pennylane is not installed on this box ({type(exc).__name__}: {exc}); "
                               "the image has no network to install it"}
    n, L = 12, 3
    dev = qml.device("lightning.qubit", wires=n)
    ham = qml.Hamiltonian([-1.0] * n + [-1.0] * n,
                          [qml.PauliZ(i) @ qml.PauliZ((i + 1) % n) for i in range(n)]
                          + [qml.PauliX(i) for i in range(n)])

    @qml.qnode(dev, diff_method="adjoint")
    def circuit(x):
        for layer in range(L):
            for w in range(n):
                qml.RY(x[layer, w, 0], wires=w)
                qml.RZ(x[layer, w, 1], wires=w)
            for w in range(n):
                qml.CNOT(wires=[w, (w + 1) % n])
        return qml.expval(ham)

    from pennylane import numpy as pnp

    x = pnp.array(workload_params(n, L, 7).reshape(L, n, 2), requires_grad=True)
    grad = qml.grad(circuit)
    grad(x)
    t0 = time.perf_counter()
    reps = 5
    for _ in range(reps):
        grad(x)
    sec = (time.perf_counter() - t0) / reps
    return {"value": 1.0 / sec, "unit": "energy_and_grad/s", "cores": os.cpu_count(),
            "workload": f"n={n} L={L} h=1, lightning.qubit adjoint, seed 7"}


# ------------------------------------------------------- batched circuits
def fp64_peak_tflops():
    """FP64 throughput of a cuBLAS DGEMM (8192^3, best of 5) on this GPU."""
    import torch

    a = torch.randn(8192, 8192, dtype=torch.float64, device="cuda")
    b = torch.randn(8192, 8192, dtype=torch.float64, device="cuda")
    torch.matmul(a, b)
    s, e = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(5):
        s.record()
        torch.matmul(a, b)
        e.record()
        e.synchronize()
        best = min(best, s.elapsed_time(e))
    return 2.0 * 8192 ** 3 / (best * 1e-3) / 1e12


def batch_flops(ns, ls):
    """Algorithmic FP64 flops of energy_and_grad over a batch (FMA = 2):
    per circuit 2^(n-1) n L (24 forward + 80 backward) + 2^n (2n + 8)."""
    n = ns.astype(np.float64)
    L = ls.astype(np.float64)
    return float(np.sum(2.0 ** (n - 1) * n * L * 104.0 + 2.0 ** n * (2.0 * n + 8.0)))


def batch_section(args, rank, world, dist, barrier, max_over_ranks):
    """4096 circuits (n ~ U{6..16}, L ~ U{1..16}, h ~ U[0.2, 2)) per step, one
    CUDA-graph replay of the batched kernels (a launch a qubit count, or the
    persistent kernel where autotuning finds it faster); with N ranks every
    rank runs its cost-balanced shard and the results are all-gathered."""
    import torch

    from gpu_simulation_b200 import BatchEngine, Engine
    from gpu_simulation_b200.batch import gather_sharded, param_offsets, shard_circuits, synthetic_batch

    count = 4096
    ns, ls, hs, params = synthetic_batch(count, seed=7)
    off = param_offsets(ns, ls)
    shards = shard_circuits(ns, ls, world)
    mine = shards[rank]
    lo, hi = int(off[mine[0]]), int(off[mine[-1] + 1])
    eng = BatchEngine()
    eng.set_circuits(ns[mine], ls[mine], hs[mine])
    p = torch.from_numpy(params[lo:hi]).cuda()
    e = torch.empty(len(mine), dtype=torch.float64, device="cuda")
    g = torch.empty_like(p)
    tune = eng.autotune(p, e, g)
    graph = eng.capture_graph(p, e, g)

    def step():
        graph.replay()
        if world > 1:
            gather_sharded(e, g, shards, off)

    for _ in range(max(3, args.warmup)):
        step()
    barrier()
    s, t = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(args.steps):
        step()
    t.record()
    t.synchronize()
    ms = max_over_ranks(s.elapsed_time(t) / args.steps)

    # end to end through the host API (descriptors, parameters in; energies, gradients out)
    eng.energy_and_grad(ns[mine], ls[mine], hs[mine], params[lo:hi])
    barrier()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        eng.energy_and_grad(ns[mine], ls[mine], hs[mine], params[lo:hi])
    e2e_ms = max_over_ranks((time.perf_counter() - t0) * 1e3 / args.steps)

    flops = batch_flops(ns, ls)
    out = {
        "workload": f"{count} circuits per step: n~U{{6..16}}, L~U{{1..16}}, h~U[0.2,2), seed 7",
        "value": count * 1000.0 / ms, "unit": "circuits/s (energy+gradient)", "ms_per_step": ms,
        "gpu_launches_per_step": len(set(ns[mine].tolist())) if min(tune, key=tune.get) == "resident" else 1, "autotune_ms": tune,
        "l2": "no flush: every replay recomputes all states from the parameters; the states are meant to "
              "stay on chip / in L2",
        "flops_per_step": flops, "achieved_tflops": flops / (ms * 1e-3) / 1e12,
        "e2e": {"value": count * 1000.0 / e2e_ms, "unit": "circuits/s", "ms_per_step": e2e_ms,
                "h2d_bytes_per_step": int(8 * params.size + 16 * count),
                "d2h_bytes_per_step": int(8 * (params.size + count))},
    }
    if world == 1:
        peak = fp64_peak_tflops()
        out["fp64_peak_tflops"] = peak
        out["fp64_peak_source"] = "measured: cuBLAS DGEMM 8192^3, best of 5"
        out["frac_of_fp64_peak"] = out["achieved_tflops"] / peak
        # the per-circuit loop through the single-circuit device entry point
        engines = {}
        for c in range(count):
            k = (int(ns[c]), int(ls[c]))
            if k not in engines:
                engines[k] = Engine(k[0], k[1], 1.0)
        ee = torch.empty(count, dtype=torch.float64, device="cuda")
        gg = torch.empty_like(p)

        def loop():
            for c in range(count):
                en = engines[(int(ns[c]), int(ls[c]))]
                en.set_field(float(hs[c]))
                en.energy_and_grad_device(p[off[c]:off[c + 1]], ee[c:c + 1], gg[off[c]:off[c + 1]])

        loop()
        torch.cuda.synchronize()
        s.record()
        loop()
        t.record()
        t.synchronize()
        loop_ms = s.elapsed_time(t)
        out["per_circuit_loop_ms"] = loop_ms
        out["speedup_vs_per_circuit_loop"] = loop_ms / ms
        out["max_abs_diff_vs_loop"] = float(max((ee - e).abs().max().item(), (gg - g).abs().max().item()))
        for en in engines.values():
            en.close()
    del graph
    eng.close()
    return out


def adam_section(n, L, steps, seed, field=1.0):
    """``steps`` torch Adam steps (lr 0.05) on the autograd Function (forward
    sweep + energy, then the adjoint sweep as backward), angles U[0, 2 pi) from
    default_rng(seed).  Reports gradient evaluations/s of the loop and of the
    bare device entry point, and the CPU oracle on the same circuit."""
    import torch

    import oracle
    from gpu_simulation_b200 import Engine, ring_ising_energy

    eng = Engine(n, L, field)
    p0 = np.random.default_rng(seed).uniform(0.0, 2.0 * np.pi, (L, n, 2))
    x = torch.tensor(p0, device="cuda", requires_grad=True)
    opt = torch.optim.Adam([x], lr=0.05)

    def step():
        opt.zero_grad(set_to_none=False)
        e = ring_ising_energy(x, eng)
        e.backward()
        opt.step()
        return e

    for _ in range(3):
        step()
    with torch.no_grad():
        x.copy_(torch.tensor(p0, device="cuda"))
    opt = torch.optim.Adam([x], lr=0.05)
    torch.cuda.synchronize()
    s, t = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(steps):
        e = step()
    t.record()
    t.synchronize()
    loop_ms = s.elapsed_time(t)
    final = float(e.item())
    # bare device entry point
    flat = torch.tensor(p0.reshape(-1), device="cuda")
    ed = torch.empty(1, dtype=torch.float64, device="cuda")
    gd = torch.empty_like(flat)
    for _ in range(3):
        eng.energy_and_grad_device(flat, ed, gd)
    s.record()
    reps = 50
    for _ in range(reps):
        eng.energy_and_grad_device(flat, ed, gd)
    t.record()
    t.synchronize()
    dev_ms = s.elapsed_time(t) / reps
    # the same Adam loop on the device: energy_and_grad + fused Adam step, one
    # step captured as a CUDA graph and replayed (torch.optim.Adam's update)
    from gpu_simulation_b200.training import run_adam_device

    run_adam_device(eng, p0, 3, lr=0.05)  # warm-up (fresh optimiser state per call)
    dev_adam = run_adam_device(eng, p0, steps, lr=0.05)
    eng.close()
    threads = oracle.set_num_threads(0)
    oracle.energy_and_grad(n, L, field, p0.reshape(-1))
    t0 = time.perf_counter()
    creps = 3
    for _ in range(creps):
        oracle.energy_and_grad(n, L, field, p0.reshape(-1))
    cpu_s = (time.perf_counter() - t0) / creps
    return {
        "workload": f"n={n} L={L} h={field}, {steps} torch Adam steps (lr 0.05) through the autograd Function, seed {seed}",
        "adam_steps_per_s": steps * 1000.0 / loop_ms, "ms_per_adam_step": loop_ms / steps,
        "final_energy": final,
        "energy_and_grad_per_s_device": 1000.0 / dev_ms, "ms_per_energy_and_grad_device": dev_ms,
        "device_adam_graph": {"adam_steps_per_s": steps * 1000.0 / dev_adam["gpu_ms"],
                              "ms_per_adam_step": dev_adam["gpu_ms"] / steps,
                              "energy_at_last_step": float(dev_adam["energies"][-1]),
                              "torch_loop_energy_at_last_step": final},
        "cpu_baseline": {"value": 1.0 / cpu_s, "unit": "energy_and_grad/s", "cores": threads, "kind": "port",
                         "sample": f"{creps} energy_and_grad calls on the CPU restatement (oracle/)"},
    }


def warmstart_section():
    """Warm start (n=16, L=6): plain VQE (Adam lr 0.05, 300 steps) from seeded
    random angles vs from the network's prediction, on 128 held-out fields."""
    from gpu_simulation_b200.warmstart import warm_start_experiment

    r = warm_start_experiment()
    r.pop("steps_plain")
    r.pop("steps_warm")
    return r


def autotune_summary(eng, n, L, seed, repeats=2):
    """Autotune the engine on the workload's parameters (every plan candidate
    timed once per shape; the fastest kept) and summarise the report."""
    import re

    import torch

    p = torch.tensor(workload_params(n, L, seed), device="cuda")
    t0 = time.perf_counter()
    report = eng.autotune(p, repeats=repeats, force=True)
    tune_s = time.perf_counter() - t0
    cands = re.findall(r"^candidate (.*): ([0-9.eE+-]+) ms$", report, re.M)
    chosen = re.search(r"^chosen (.*): ([0-9.eE+-]+) ms$", report, re.M)
    spread = re.search(r"between candidates \(energy, gradient\): ([0-9.eE+-]+)", report)
    return {
        "candidates": [{"config": c, "ms": float(ms)} for c, ms in cands],
        "planner_default": {"config": cands[0][0], "ms": float(cands[0][1])} if cands else None,
        "chosen": {"config": chosen.group(1), "ms": float(chosen.group(2))} if chosen else None,
        "largest_difference_between_candidates": float(spread.group(1)) if spread else None,
        "tuning_s": tune_s,
    }


# ---------------------------------------------------------------- GPU arm
def sharded_section(args, rank, world, dist, barrier, max_over_ranks, single=None):
    """Sharded single circuit: timed energy_and_grad through ShardedEngine,
    compared with the single-GPU engine on the same parameters.  With several
    ranks every step that can fail on one rank alone (allocation, the
    single-GPU reference on rank 0) is followed by an agreement on its status,
    so all ranks take the same collectives or skip together."""
    import torch

    from gpu_simulation_b200 import Engine
    from gpu_simulation_b200.sharded import ShardedEngine

    L, h = args.layers, args.field
    out = {}

    def all_ok(ok):
        if dist is None:
            return ok
        flag = torch.tensor([1.0 if ok else 0.0], dtype=torch.float64, device="cuda")
        dist.all_reduce(flag, op=dist.ReduceOp.MIN)
        return flag.item() > 0.5

    if world > 1:
        n, kw, how = 30, dict(group=dist.group.WORLD), f"{world} ranks, NCCL all_to_all_single"
    else:
        n, kw, how = args.qubits, dict(virtual_ranks=2), "2 virtual ranks on one GPU (exchanges as device copies)"
    p = workload_params(n, L, 7)
    ref, ok = None, True
    try:
        if single is not None and single[0] == n:
            ref = single[1]
        elif rank == 0:
            e1 = Engine(n, L, h)
            ref = e1.energy_and_grad(p)
            e1.close()
            torch.cuda.empty_cache()
    except Exception as exc:  # report, do not hide
        out["reference_error"] = str(exc)
    sh = None
    try:
        sh = ShardedEngine(n, L, h, **kw)
    except Exception as exc:
        out["error"] = str(exc)
        ok = False
    if not all_ok(ok):
        out.setdefault("error", "a rank could not set up the sharded engine")
        return out
    e, g = sh.energy_and_grad(p)
    steps = max(2, min(args.steps, 5))
    barrier()
    s, t = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(steps):
        sh.energy_and_grad(p)
    t.record()
    torch.cuda.synchronize()
    ms = max_over_ranks(s.elapsed_time(t) / steps)
    out.update({"workload": f"energy_and_grad n={n} L={L} h={h}", "ranks": how, "ms_per_call": ms,
                "energy_and_grad_per_s": 1000.0 / ms, "energy": e,
                "timing": "CUDA events over host-parameter calls (host result), max over ranks"})
    if ref is not None:
        out["vs_single_gpu_engine"] = {"energy_abs_diff": abs(e - ref[0]),
                                       "grad_max_abs_diff": float(np.max(np.abs(g - ref[1])))}
    del sh
    torch.cuda.empty_cache()
    if world == 1:
        try:
            out["rank_kernels_n33_8_ranks"] = shard_rank_kernels(33, 3, L)
        except Exception as exc:  # report, do not hide
            out["rank_kernels_error"] = str(exc)
    return out


def shard_rank_kernels(n, g, L, reps=3):
    """One rank's kernels of a sharded call at full shard size (no exchange),
    and the exchange volume that the call's all-to-alls move per rank."""
    import torch

    from gpu_simulation_b200.sharded import CudaShardOps

    ops = CudaShardOps()
    local = 1 << (n - g)
    vec = lambda: torch.zeros(local, dtype=torch.complex128, device="cuda")  # noqa: E731
    psi, psi2, lam, lam2 = vec(), vec(), vec(), vec()
    psi.real.normal_()
    lam.real.normal_()
    p = torch.tensor(workload_params(n, L, 7), device="cuda")
    coef = torch.zeros(4 * n * L, dtype=torch.float64, device="cuda")
    ops.coef(n, L, p, coef)
    scratch = torch.zeros(ops.scratch_doubles(n, g), dtype=torch.float64, device="cuda")
    res = torch.zeros(2 + 2 * n * L, dtype=torch.float64, device="cuda")
    vbytes = local * 16
    peak, _ = measured_peaks()
    table = {}

    def timed(name, fn, vectors, per_call):
        fn()
        torch.cuda.synchronize()
        s, t = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        s.record()
        for _ in range(reps):
            fn()
        t.record()
        torch.cuda.synchronize()
        ms = s.elapsed_time(t) / reps
        gbs = vectors * vbytes / (ms * 1e-3) / 1e9
        table[name] = {"ms": ms, "per_call": per_call, "bytes": vectors * vbytes, "gbs": gbs, "frac_of_peak": gbs / peak}

    timed("rotate_local (wires 0..n-g-1, 4 tile passes)", lambda: ops.rotate_local(n, g, 1, coef, psi), 8, L)
    timed("ring_pack (wires n-g..n-1 + sort by destination)", lambda: ops.ring_pack(n, g, 0, 1, coef, psi, psi2), 2, L)
    timed("ring_unpack", lambda: ops.ring_unpack(n, g, 0, psi2, psi), 2, L)
    timed("energy_local (4 tile passes)", lambda: ops.energy_local(n, g, 0, 1.0, psi, lam, scratch, res), 11, 1)
    timed("ring_pack_adjoint", lambda: ops.ring_pack_adjoint(n, g, 0, psi, lam, psi2, lam2), 4, L)
    timed("ring_unpack_adjoint", lambda: ops.ring_unpack_adjoint(n, g, 0, L, 1, coef, 1.0, 0, psi2, lam2, psi, lam,
                                                                scratch, res), 4, L)
    timed("rotate_local_adjoint (4 tile passes)", lambda: ops.rotate_local_adjoint(n, g, L, 1, coef, psi, lam,
                                                                                  scratch, res), 16, L)
    kernels_ms = sum(v["ms"] * v["per_call"] for v in table.values())
    # all-to-alls per call: forward 2 vectors a layer, backward 4; (N-1)/N of
    # each crosses NVLink in each direction
    N = 1 << g
    cross = 6 * L * vbytes * (N - 1) / N
    link = 770.0  # GB/s per direction, measured peer copy on this pool's NVLink
    return {"shard_amplitudes": local, "ops": table, "kernels_ms_per_call": kernels_ms,
            "exchange_bytes_per_rank_per_call": cross,
            "exchange_ms_at_770_gbs": cross / (link * 1e9) * 1e3,
            "note": "per-rank kernels timed alone on one GPU (CUDA events); the all-to-alls are not run here"}


def pass_schedule(n, L):
    """An engine on the tile passes for a circuit that the default does not run on them."""
    from gpu_simulation_b200 import Engine

    eng = Engine(n, L, 1.0)
    eng.set_backward_mode("checkpoint" if n <= 30 else "uncompute")
    return eng


def on_passes(eng):
    return "the plan below is not used" not in eng.describe().splitlines()[0]


def device_time(eng, n, L, field, steps, warmup, seed, timing=False, flush=None, load_s=0.0):
    import torch

    dev = torch.device("cuda")
    p = torch.tensor(workload_params(n, L, seed), device=dev)
    e = torch.empty(1, dtype=torch.float64, device=dev)
    g = torch.empty_like(p)
    for _ in range(warmup):
        eng.energy_and_grad_device(p, e, g)
    torch.cuda.synchronize()
    if flush is not None:
        # the working set fits L2: each step alone, behind a write larger than L2
        k0 = eng.kernel_launches()
        marks = [(torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)) for _ in range(steps)]
        for s, t in marks:
            flush.fill_(0)
            s.record()
            eng.energy_and_grad_device(p, e, g)
            t.record()
        torch.cuda.synchronize()
        launched = eng.kernel_launches() - k0
        until = time.perf_counter() + load_s
        while time.perf_counter() < until:  # the same call, for the clock samples
            for _ in range(200):
                eng.energy_and_grad_device(p, e, g)
            torch.cuda.synchronize()
        return sum(s.elapsed_time(t) for s, t in marks) / steps, {"kernels_launched": launched}, float(e.item())
    if timing:
        eng.set_launch_timing(True)
    k0 = eng.kernel_launches()
    s, t = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    s.record()
    for _ in range(steps):
        eng.energy_and_grad_device(p, e, g)
    t.record()
    torch.cuda.synchronize()
    stats = None
    if timing:
        eng.set_launch_timing(False)
        stats = eng.launch_stats()
        stats["kernels_launched"] = eng.kernel_launches() - k0
    return s.elapsed_time(t) / steps, stats, float(e.item())


def main():
    args = parse_args()
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        return run_reference_arm(args, rank, world)

    import torch

    torch.cuda.set_device(local_rank)
    if args.shard_rank_kernels:
        ns, gs = (int(v) for v in args.shard_rank_kernels.split(","))
        print(json.dumps(shard_rank_kernels(ns, gs, args.layers)), flush=True)
        return 0
    dist = None
    if world > 1:
        import datetime

        import torch.distributed as dist

        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120),
                                device_id=torch.device("cuda", local_rank))

    from gpu_simulation_b200 import Engine

    n, L, h = args.qubits, args.layers, args.field
    eng = Engine(n, L, h)
    # one-time plan tuning (cached per shape), before any timed region
    tuned = autotune_summary(eng, n, L, seed=7 + rank) if not args.no_autotune else None

    def barrier():
        torch.cuda.synchronize()
        if dist is not None:
            dist.barrier()

    def max_over_ranks(x):
        if dist is None:
            return x
        t = torch.tensor([x], dtype=torch.float64, device="cuda")
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    # device-resident timed region (the headline value)
    barrier()
    sampler = ClockSampler() if rank == 0 else None
    if sampler:
        sampler.start()
    passes = on_passes(eng)
    flush = None if passes else torch.empty(1 << 28, dtype=torch.uint8, device="cuda")
    ms, stats, energy = device_time(eng, n, L, h, args.steps, args.warmup, seed=7 + rank, timing=True, flush=flush,
                                    load_s=1.0)
    barrier()
    clocks = sampler.stop(set(range(max(1, torch.cuda.device_count())))) if sampler else None
    ms_max = max_over_ranks(ms)
    value = world * 1000.0 / ms_max

    # end-to-end through the public host API: params from host, result to host
    p_host = workload_params(n, L, 7 + rank)
    eng.energy_and_grad(p_host)
    barrier()
    t0 = time.perf_counter()
    for _ in range(args.steps):
        eng.energy_and_grad(p_host)
    e2e_ms = (time.perf_counter() - t0) * 1e3 / args.steps
    e2e_ms = max_over_ranks(e2e_ms)

    peak, peak_src = measured_peaks()
    KERNEL_NAMES = {
        "backward_pass": "backward: bwd_tma_kernel<1> (phase pass, with the field terms of its tile), "
                         "bwd_tma_kernel<0>, bwd_tma_low_kernel, mps_grad4_kernel (+ its two small reductions)",
        "forward_pass": "fwd_pass_kernel (the first one evaluating the bond-4 matrix-product state)",
        "energy": "energy_kernel (diagonal and the field terms off the phase pass's tile; "
                  "energy_tile_kernel + energy_kernel without the fused energy)",
    }
    kernels_launched = int(stats.pop("kernels_launched"))
    pass_ms = ms_max
    if not passes:  # the roofline of the tile passes
        del flush
        ep = pass_schedule(n, L)
        pass_ms, stats, _ = device_time(ep, n, L, h, 3, 2, seed=7 + rank, timing=True)
        stats.pop("kernels_launched")
        ep.close()
    kinds = {k: v for k, v in stats.items() if v["launches"]}
    dom = max(kinds, key=lambda k: kinds[k]["ms"])
    d = kinds[dom]
    achieved = d["bytes"] / (d["ms"] * 1e-3) / 1e9
    total_ms = sum(v["ms"] for v in kinds.values())
    traffic = None
    tfile = ROOT / "profiles" / "traffic_per_launch.md"
    if tfile.exists():
        for row in tfile.read_text().splitlines():
            cells = [c.strip() for c in row.strip().strip("|").split("|")]
            if len(cells) == 3 and cells[0] == dom and cells[1] == str(n):
                traffic = float(cells[2])
    roofline = {
        "bound": "hbm", "kernel": KERNEL_NAMES.get(dom, dom), "achieved": achieved, "peak": peak,
        "unit": "GB/s", "frac": achieved / peak, "traffic": traffic,
        "peak_source": peak_src,
        "algorithmic_bytes_per_launch": d["bytes"] / d["launches"],
        "avg_launch_ms": d["ms"] / d["launches"],
        "schedule": "the timed call" if passes else f"tile passes (set_backward_mode), {pass_ms:.3f} ms a call; the timed "
                    "call reads no state vector and is bound by the latency of its chains of small products",
    }
    whole_bytes = sum(v["bytes"] for v in kinds.values())
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": ms_max, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f64", "data": "synthetic: seeded U[0,2pi) angles",
        "config": {
            "workload": f"structured_adjoint energy_and_grad n={n} L={L} h={h}",
            "num_qubits": n, "num_layers": L, "field": h,
            "parallelism": "replicas" if world > 1 else "single",
            "path": eng.describe().splitlines()[0],
            "l2": "no flush: inputs larger than L2 (3 state buffers of 16*2^n bytes)" if passes else
                  "flushed: 256 MiB written before every timed step; CUDA events around each step",
            "energy": energy,
        },
        "roofline": roofline,
        "whole_call": {
            "algorithmic_bytes": whole_bytes, "achieved_gbs": whole_bytes / (total_ms * 1e-3) / 1e9,
            "frac_of_peak": whole_bytes / (total_ms * 1e-3) / 1e9 / peak,
        },
        "kernels": kinds,
        "autotune": tuned,
        "gpu_launches": kernels_launched,
        "e2e": {"value": world * 1000.0 / e2e_ms, "unit": UNIT, "ms_per_step": e2e_ms,
                "h2d_bytes_per_step": n * L * 32, "d2h_bytes_per_step": (1 + 2 * n * L) * 8},
        "clocks": clocks,
    }
    if world == 1 and rank == 0 and not args.no_sweep:
        sweep = {}
        for ns in (20, 24, 30):
            if ns == n:
                continue
            try:
                e2 = Engine(ns, L, h)
                tuned_s = autotune_summary(e2, ns, L, seed=7) if not args.no_autotune else None
                if on_passes(e2):
                    fl, ep = None, e2
                else:
                    fl, ep = torch.empty(1 << 28, dtype=torch.uint8, device="cuda"), pass_schedule(ns, L)
                ms_s, st_s, _ = device_time(e2, ns, L, h, max(3, args.steps // 2), 2, seed=7, timing=True, flush=fl)
                if fl is not None:
                    del fl
                    ms_p, st_s, _ = device_time(ep, ns, L, h, 3, 2, seed=7, timing=True)
                    ep.close()
                else:
                    ms_p = ms_s
                st_s.pop("kernels_launched")
                byt = sum(v["bytes"] for v in st_s.values())
                tms = sum(v["ms"] for v in st_s.values())
                sweep[f"n={ns}"] = {"ms_per_call": ms_s, "energy_and_grad_per_s": 1000.0 / ms_s,
                                    "tile_passes_ms": ms_p,
                                    "tile_passes_frac_of_peak": byt / (tms * 1e-3) / 1e9 / peak,
                                    "autotune": tuned_s}
                e2.close()
            except Exception as exc:  # report, do not hide
                sweep[f"n={ns}"] = {"error": str(exc)}
        line["sweep"] = sweep
    if world == 1 and rank == 0 and not args.no_sweep:
        # the same call on the tile passes with fewer analytic leading layers
        # (matrix-product shortcut off): 0 = every layer on tile passes, as the
        # reference's schedule
        info = eng.analytic_layers()
        alt = {"default_max_layers": info["max_layers"], "used": info["used"]}
        for k in (0, 1, 2):
            eng.set_analytic_layers(k)
            ms_k, _, e_k = device_time(eng, n, L, h, max(3, args.steps // 2), 2, seed=7 + rank)
            alt[f"max_layers={k}"] = {"ms_per_call": ms_k, "energy_and_grad_per_s": 1000.0 / ms_k,
                                      "energy": e_k}
        eng.set_analytic_layers(info["max_layers"])
        line["analytic_layers"] = alt
    if world == 1 and rank == 0 and not args.no_cpu:
        t, threads, e_cpu = cpu_call(n, L, h)
        line["cpu_baseline"] = {
            "value": 1.0 / t, "unit": UNIT, "cores": threads, "kind": "port",
            "sample": f"one full energy_and_grad at n={n}, L={L} (the workload itself) on the CPU "
                      f"restatement (oracle/), {t:.2f} s, energy {e_cpu:.12f}",
        }
    if world == 1 and rank == 0:
        line["pennylane_lightning_qubit"] = pennylane_baseline()
    single = (n, eng.energy_and_grad(workload_params(n, L, 7))) if not args.no_sharded else None
    eng.close()
    if not args.no_sharded:
        import torch as _t

        _t.cuda.empty_cache()
        line["sharded"] = sharded_section(args, rank, world, dist, barrier, max_over_ranks, single)
    if not args.no_batch:
        line["batch"] = batch_section(args, rank, world, dist, barrier, max_over_ranks)
    if world == 1 and not args.no_warmstart:
        line["warm_start"] = warmstart_section()
    if world == 1 and not args.no_small:
        line["adam_n12_l3"] = adam_section(12, 3, 20, seed=7)
        line["autograd_n20_l8"] = adam_section(20, 8, 100, seed=7)
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()
    return 0


if __name__ == "__main__":
    sys.exit(main())
