#!/usr/bin/env python
"""Benchmark of the convolution hot path and of the CaffeNet training iteration built around it, on synthetic data,
one process per GPU.

    python bench.py [--gpus N] [--steps K] [--warmup W]           # one CaffeNet iteration, 256 images per GPU (default)
    python bench.py --workload alexnet_conv1|caffenet_conv2|lenet_conv1   # one convolution layer: forward + backward + SGD
    python bench.py --impl reference ...      # the reference's own CPU code (oracle/_ref) on the host cores

Prints ONE JSON line (rank 0).  `value` is whole-job images/s with inputs resident in HBM, device-timed, maximum over
ranks; `e2e` is the same metric with every step's inputs uploaded from pinned host memory and the loss (or the host-buffer
calls' outputs) read back inside the timed region; `roofline` describes the slowest contraction kernel group against
the tensor roofline of three 16-bit products per multiply-add; `cpu_baseline` is the reference CPU path timed on this box's host
cores in the same run.
"""
import argparse
import ctypes as C
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "conv_fwd_bwd_images_per_sec"
WORKLOADS = {
    # AlexNet conv1, batch 256 per GPU, X ~ N(0,1), W ~ N(0,0.01), bias 0, dY ~ N(0,1)
    "alexnet_conv1": dict(B=256, D=3, n=227, o=96, k=11, s=4, p=0, g=1, x="normal", bias="zero"),
    # BASELINE config 3 geometry: CaffeNet conv2 (grouped), post-ReLU inputs
    # (its backward runs fused: output gradient rebuilt from the 3x3/2 max-pool indices and the ReLU sign, input
    # gradient masked by the ReLU in front of the layer)
    "caffenet_conv2": dict(B=256, D=96, n=27, o=256, k=5, s=1, p=2, g=2, x="relu", bias="one", pool=(3, 2)),
    # LeNet conv1
    "lenet_conv1": dict(B=64, D=1, n=28, o=20, k=5, s=1, p=0, g=1, x="uniform", bias="normal"),
}
SOLVER = dict(base_lr=0.01, momentum=0.9, weight_decay=0.0005)  # caffenet solver values; lr kept small on purpose


def out_size(w):
    return (w["n"] + 2 * w["p"] - w["k"]) // w["s"] + 1


def gemm_flops(w):
    m = out_size(w)
    return 2.0 * w["o"] * (w["k"] ** 2 * w["D"] // w["g"]) * m * m * w["B"]


def synth(w, seed):
    rng = np.random.default_rng(seed)
    m = out_size(w)
    B, D, n, o, k, g = w["B"], w["D"], w["n"], w["o"], w["k"], w["g"]
    if w["x"] == "uniform":
        X = rng.random((B, D, n, n), dtype=np.float32)
    else:
        X = rng.standard_normal((B, D, n, n), dtype=np.float32)
        if w["x"] == "relu":
            np.maximum(X, 0, out=X)
    W = (0.01 * rng.standard_normal((o, D // g, k, k))).astype(np.float32)
    bias = {"zero": np.zeros(o, np.float32), "one": np.ones(o, np.float32),
            "normal": (0.01 * rng.standard_normal(o)).astype(np.float32)}[w["bias"]]
    dY = rng.standard_normal((B, o, m, m), dtype=np.float32)
    return X, W, bias, dY


def dram_traffic(workload, w, pass_name, batch):
    """DRAM bytes per launch of one pass, from the ncu captures summarised in profiles/dram_traffic.json: measured
    reads of the small-case capture scaled to this batch (they grow in proportion) plus the pass's output bytes (the
    small case's outputs stay in L2, so its write counter undercounts).  (None, None) for a pass never captured."""
    path = os.path.join(ROOT, "profiles", "dram_traffic.json")
    try:
        with open(path) as f:
            table = json.load(f)
    except OSError:
        return None, None
    entry = table.get(workload, {}).get(pass_name)
    if not entry:
        return None, None
    m = (w["n"] + 2 * w["p"] - w["k"]) // w["s"] + 1
    out_elems = {"forward": batch * w["o"] * m * m, "dgrad": batch * w["D"] * w["n"] * w["n"],
                 "wgrad": w["o"] * (w["D"] // w["g"]) * w["k"] * w["k"] + w["o"]}[pass_name]
    return entry["dram_read_bytes"] * batch / float(entry["batch"]) + 4.0 * out_elems, entry["source"]


def caffenet_traffic(kernel, batch):
    """DRAM bytes (read + write) of one launch of a CaffeNet kernel group ("conv2 dgrad", "fc6 forward", ...) from the
    batch-256 ncu capture summarised under profiles/, scaled by the batch ratio.  (None, None) if never captured."""
    try:
        with open(os.path.join(ROOT, "profiles", "dram_traffic.json")) as f:
            table = json.load(f).get("caffenet", {})
    except OSError:
        return None, None
    layer, _, what = kernel.partition(" ")
    entry = table.get("%s %s" % (layer, {"wgrad": "weight gradient", "dgrad": "data gradient"}.get(what, what)))
    if not entry:
        return None, None
    return (entry["dram_read_bytes"] + entry["dram_write_bytes"]) * batch / float(entry["batch"]), entry["source"]


def measure_tf32_peak(seconds=2.0):
    """Dense TF32 matmul throughput of this GPU, measured like the bf16 figures of MEASURED_PEAKS.json: a library
    8192^3 matmul with TF32 inputs, best of 10 (burst) and back to back for `seconds` (sustained).  Only a roofline
    denominator: nothing on the measured path calls a library GEMM."""
    import torch
    n = 8192
    prev = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = True
    try:
        a = torch.randn(n, n, device="cuda")
        b = torch.randn(n, n, device="cuda")
        c = torch.empty(n, n, device="cuda")
        for _ in range(3):
            torch.matmul(a, b, out=c)
        torch.cuda.synchronize()
        best = float("inf")
        for _ in range(10):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            torch.matmul(a, b, out=c)
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        reps = max(10, int(seconds * 1e3 / best))
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(reps):
            torch.matmul(a, b, out=c)
        e1.record()
        torch.cuda.synchronize()
        sustained = e0.elapsed_time(e1) / reps
        del a, b, c
        torch.cuda.empty_cache()
    finally:
        torch.backends.cuda.matmul.allow_tf32 = prev
    flops = 2.0 * n ** 3
    return flops / (best * 1e-3) / 1e12, flops / (sustained * 1e-3) / 1e12


def tensor_roofline(peaks, measure=True):
    """fp32-equivalent roofline in TFLOP/s: the measured rate of 16-bit matmuls / 3 (the larger contractions' three products of fp16 pairs; the
    others' are three of TF32, whose measured rate stands beside it)."""
    out = {"bf16_burst": peaks["bf16_tflops"], "bf16_sustained": peaks.get("bf16_tflops_sustained")}
    if measure:
        burst, sustained = measure_tf32_peak()
        out.update(tf32_burst=burst, tf32_sustained=sustained)
    else:
        out.update(tf32_burst=None, tf32_sustained=None)
    out.update(peak=peaks["bf16_tflops"] / 3.0, peak_sustained=(peaks.get("bf16_tflops_sustained") or 0) / 3.0,
               source="%s: 16-bit matmul burst %.1f, sustained %.1f TFLOP/s, / 3 - of measured%s" %
                      (peaks["source"], peaks["bf16_tflops"], peaks.get("bf16_tflops_sustained") or 0,
                       "; TF32 8192^3 library matmul in this run: burst %.1f, sustained %.1f" % (burst, sustained) if measure else ""))
    return out


def load_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(path):
        with open(path) as f:
            p = json.load(f)
        return dict(bf16_tflops=p["bf16_tflops"], bf16_tflops_sustained=p.get("bf16_tflops_sustained"),
                    hbm_gbs=p["hbm_gbs"], source="measured (MEASURED_PEAKS.json)")
    return dict(bf16_tflops=1590.0, bf16_tflops_sustained=1400.0, hbm_gbs=6650.0, source="fallback")


class ClockSampler:
    """Samples nvidia-smi clocks and throttle reasons every 200 ms while the timed region runs."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device_index):
        self.idx = device_index
        self.lines = []
        self.proc = None

    def start(self):
        try:
            self.proc = subprocess.Popen(["nvidia-smi", "--query-gpu=" + self.FIELDS, "--format=csv,noheader,nounits",
                                          "-lms", "100"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.thread = threading.Thread(target=self._pump, daemon=True)
            self.thread.start()
        except OSError:
            self.proc = None

    def _pump(self):
        for line in self.proc.stdout:
            self.lines.append(line)

    def stop(self):
        if not self.proc:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        time.sleep(0.25)
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        sm, smax, reasons = [], None, set()
        names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
        for line in self.lines:
            f = [x.strip() for x in line.split(",")]
            if len(f) < 9 or f[0] != str(self.idx):
                continue
            try:
                sm.append(float(f[1]))
                smax = float(f[2])
            except ValueError:
                continue
            for name, val in zip(names, f[5:9]):
                if val.lower().startswith("active"):
                    reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": smax, "samples": len(sm),
                "reasons": sorted(reasons)}


def cpu_reference_time(w, iters, warmup, with_update):
    """(images/s, cores, kind, sample) of the reference CPU path on this host; falls back to the C port."""
    from oracle import build as obuild, pyoracle
    X, W, bias, dY = synth(w, 1234)
    ref = pyoracle.reference()
    if ref is not None:
        parts = ref.default_partitions(w["B"])
        per_group = []
        g = w["g"]
        Dg, og = w["D"] // g, w["o"] // g
        for gi in range(g):  # the reference bridge has no group concept: one bridge per channel slice
            Xs = np.ascontiguousarray(X[:, gi * Dg:(gi + 1) * Dg])
            Ws = np.ascontiguousarray(W[gi * og:(gi + 1) * og])
            bs = np.ascontiguousarray(bias[gi * og:(gi + 1) * og])
            dYs = np.ascontiguousarray(dY[:, gi * og:(gi + 1) * og])
            per_group.append(ref.conv_time(Xs, Ws, bs, dYs, w["k"], w["s"], w["p"], parts, True, warmup, iters)[0])
        sec = sum(per_group)
        return dict(value=w["B"] / sec, unit="images/s", cores=parts, kind="reference",
                    sample="%d fwd+bwd passes over the full %d-image batch (median), %d batch partitions x 1 BLAS thread, "
                           "hardware_concurrency %d, %s" % (iters, w["B"], parts, ref.hardware_concurrency(),
                                                            ref.blas_config()),
                    seconds_per_step=sec)
    obuild.build_port()
    port = pyoracle.port()
    nb = max(1, min(w["B"], 8))
    Xs, dYs = X[:nb].copy(), dY[:nb].copy()
    t0 = time.perf_counter()
    port.conv_forward(Xs, W, bias, w["k"], w["s"], w["p"], w["g"])
    port.conv_backward(Xs, W, dYs, w["k"], w["s"], w["p"], w["g"])
    sec = time.perf_counter() - t0
    return dict(value=nb / sec, unit="images/s", cores=os.cpu_count(), kind="port",
                sample="1 fwd+bwd pass over %d images (plain-C restatement, OpenMP)" % nb, seconds_per_step=sec)


def run_reference_arm(args, w, rank, world):
    if rank != 0:
        return
    from oracle import pyoracle
    ref = pyoracle.reference()
    X, W, bias, dY = synth(w, 1234)
    if ref is None:
        base = cpu_reference_time(w, max(1, args.steps), max(0, args.warmup), True)
        ms = base["seconds_per_step"] * 1e3
        val = base["value"]
        cpu = base
    else:
        parts = ref.default_partitions(w["B"])
        g = w["g"]
        Dg, og = w["D"] // g, w["o"] // g
        handles = []
        for gi in range(g):
            h = ref.conv_create(w["B"], Dg, w["n"], og, w["k"], w["s"], w["p"], True, parts, True,
                                SOLVER["base_lr"], SOLVER["momentum"], SOLVER["weight_decay"])
            ref.lib.cctref_conv_set_model(h, pyoracle._p(np.ascontiguousarray(W[gi * og:(gi + 1) * og])),
                                          pyoracle._p(np.ascontiguousarray(bias[gi * og:(gi + 1) * og])))
            ref.lib.cctref_conv_load(h, pyoracle._p(np.ascontiguousarray(X[:, gi * Dg:(gi + 1) * Dg])),
                                     pyoracle._p(np.ascontiguousarray(dY[:, gi * og:(gi + 1) * og])))
            handles.append(h)
        def step():
            for h in handles:
                ref.lib.cctref_conv_step(h, 1)
        for _ in range(args.warmup):
            step()
        t0 = time.perf_counter()
        for _ in range(args.steps):
            step()
        sec = (time.perf_counter() - t0) / args.steps
        for h in handles:
            ref.conv_destroy(h)
        ms, val = sec * 1e3, w["B"] / sec
        cpu = dict(value=val, unit="images/s", cores=parts, kind="reference",
                   sample="each step = forward + backward + SGD update of the reference's ParallelizedBridge over one "
                          "%d-image batch (%d of the job's %d images), %d partitions x 1 BLAS thread, "
                          "hardware_concurrency %d, %s" % (w["B"], w["B"], w["B"] * world, parts,
                                                           ref.hardware_concurrency(), ref.blas_config()))
    line = {
        "impl": "reference", "metric": METRIC, "value": val, "unit": "images/s", "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": config_of(args, w, world), "tflops": 3 * gemm_flops(w) / (ms * 1e-3) / 1e12,
        "cpu_baseline": cpu,
        "e2e": {"value": val, "unit": "images/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


def preheat(step, warmup, seconds, stream, agree=None):
    """Untimed warm-up: at least `warmup` steps and at least `seconds` of device time, so that the timed steps that
    follow run at the clocks and power state of a long job and not in a cold burst.  Returns the steps run.  With
    several ranks every rank must run the same number of steps (each holds collectives): `agree(n)` returns the
    maximum of n over the ranks."""
    import torch
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    n0 = max(warmup, 3)
    for _ in range(2):  # the first steps carry one-off costs (module loading, communicator set-up)
        step()
    e0.record(stream)
    for _ in range(n0 - 2 if n0 > 2 else 1):
        step()
    e1.record(stream)
    torch.cuda.synchronize()
    per = max(e0.elapsed_time(e1) / max(n0 - 2, 1), 1e-3)
    more = max(0, int(seconds * 1e3 / per) - n0)
    if agree is not None:
        more = agree(more)
    for _ in range(more):
        step()
    torch.cuda.synchronize()
    return max(n0, 3) + more


# The five convolution layers of CaffeNet at batch 256 per GPU (BASELINE config 4 without the LRN / FC / softmax layers,
# which are outside this path): (name, D, n, o, k, s, p, g, pool behind the layer's ReLU or None, needs dX).
CAFFENET_CONVS = [
    ("conv1", 3, 227, 96, 11, 4, 0, 1, (3, 2), False),
    ("conv2", 96, 27, 256, 5, 1, 2, 2, (3, 2), True),
    ("conv3", 256, 13, 384, 3, 1, 1, 1, None, True),
    ("conv4", 384, 13, 384, 3, 1, 1, 2, None, True),
    ("conv5", 384, 13, 256, 3, 1, 1, 2, (3, 2), True),
]


def run_conv_stack(args, rank, world, local_rank):
    """All five CaffeNet convolution layers as one step: forward (+ReLU), fused backward (pooled gradient and ReLU
    masks folded in, conv1 without dX), gradient all-reduce (N>1) and SGD step per layer, on synthetic tensors of the
    layers' own shapes (the layers between them - LRN, pooling forward, FC - are not part of this path)."""
    import torch
    import torch.distributed as dist
    from caffecontroll_b200 import capi
    from caffecontroll_b200.bridge import Context, ConvolutionBridge, Layer, LogicalCube
    from caffecontroll_b200.parallel import DeviceOps, ParallelizedBridge, SolverParameter

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    stream = torch.cuda.current_stream()
    ctx = Context(local_rank, stream=stream.cuda_stream)
    lib, vp = ctx.lib, C.c_void_p
    B = args.batch or 256
    rng = np.random.default_rng(4000 + rank)
    layers, flops = [], 0.0
    for name, D, n, o, k, s_, p_, g, pool, needs_dx in CAFFENET_CONVS:
        m = (n + 2 * p_ - k) // s_ + 1
        X = rng.standard_normal((B, D, n, n), dtype=np.float32)
        if name != "conv1":
            X = np.maximum(X, 0)  # every later layer sees a ReLU output
        xin = Layer(LogicalCube.from_numpy(ctx, X), LogicalCube(ctx, n, n, D, B))
        out = Layer(LogicalCube(ctx, m, m, o, B), LogicalCube.from_numpy(ctx, rng.standard_normal((B, o, m, m), dtype=np.float32)))
        conv = ConvolutionBridge(xin, out, k, s_, p_, g, True, algo=args.algo)
        conv.needs_to_calc_backward_grad = needs_dx
        conv.fuse_relu = True
        conv.fuse_relu_backward = needs_dx
        conv.p_model_cube.upload((0.01 * rng.standard_normal((o, D // g, k, k))).astype(np.float32))
        conv.p_bias_cube.upload(np.zeros(o, np.float32) if name in ("conv1", "conv3") else np.ones(o, np.float32))
        pb = ParallelizedBridge(conv, SolverParameter(SOLVER["base_lr"], "step", 0.1, 100000, momentum=SOLVER["momentum"],
                                                      weight_decay=SOLVER["weight_decay"]), DeviceOps(ctx))
        if pool:
            pk, ps = pool
            mp = (m - pk) // ps + 1
            pooled, idx = LogicalCube(ctx, mp, mp, o, B), LogicalCube(ctx, mp, mp, o, B, np.int32)
            dP = LogicalCube.from_numpy(ctx, rng.standard_normal((B, o, mp, mp), dtype=np.float32))
            conv.forward()
            capi.check(lib.cct_maxpool_forward(ctx.h, vp(out.p_data_cube.ptr), vp(pooled.ptr), vp(idx.ptr), B * o, m, pk, ps),
                       "cct_maxpool_forward", ctx.h)
            conv.fuse_pool_relu_backward(dP, idx, pk, ps)
        F = 2.0 * o * (k * k * D // g) * m * m * B
        flops += (3 if needs_dx else 2) * F
        layers.append((name, pb, conv, F, needs_dx))

    def step():
        for _, pb, _, _, _ in layers:
            pb.forward()
        for _, pb, _, _, _ in reversed(layers):
            pb.backward()

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    for _ in range(max(args.warmup, 3)):
        step()
    barrier()
    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record(stream)
    counted = capi.kernel_launches()
    for _ in range(args.steps):
        step()
    timed_launches = capi.kernel_launches() - counted
    e1.record(stream)
    barrier()
    ms_total = e0.elapsed_time(e1)
    if world > 1:
        t = torch.tensor([ms_total], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_total = float(t.item())
    ms_step = ms_total / args.steps
    per_layer = {}
    for name, pb, conv, F, needs_dx in layers:
        lib.cct_conv_plan_enable_timing(conv.plan, 1)
    acc = {name: np.zeros(5) for name, *_ in layers}
    reps = min(args.steps, 5)
    for _ in range(reps):
        step()
        for name, pb, conv, F, needs_dx in layers:
            t5 = (C.c_float * 5)()
            capi.check(lib.cct_conv_plan_last_timings(conv.plan, t5), "timings", ctx.h)
            acc[name] += np.array(list(t5))
    clocks = sampler.stop() if rank == 0 else None
    for name, pb, conv, F, needs_dx in layers:
        k_ms = acc[name] / reps
        per_layer[name] = {"forward_ms": k_ms[0] + k_ms[4], "wgrad_ms": k_ms[1] + k_ms[2], "dgrad_ms": k_ms[3] if needs_dx else None,
                           "forward_tflops": F / (k_ms[0] * 1e-3) / 1e12, "wgrad_tflops": F / ((k_ms[1] + k_ms[2]) * 1e-3) / 1e12,
                           "dgrad_tflops": F / (k_ms[3] * 1e-3) / 1e12 if needs_dx and k_ms[3] > 0 else None}
    if rank == 0:
        peaks = load_peaks()
        peak = peaks["bf16_tflops"] / 3.0
        tf = world * flops / (ms_step * 1e-3) / 1e12
        line = {
            "metric": METRIC, "value": world * B / (ms_step * 1e-3), "unit": "images/s", "n_gpus": world,
            "steps": args.steps, "warmup": max(args.warmup, 3), "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "caffenet_convs (conv1-conv5, batch %d per GPU)" % B, "batch_per_gpu": B,
                       "global_batch": B * world, "step": "per layer: forward (+ReLU), fused backward (pooled gradient and ReLU masks folded in; conv1 "
                               "without dX), gradient all-reduce (N>1), SGD momentum step",
                       "l2": "inputs larger than L2 (2.4 GB of activations and gradients per step)", "parallelism": "dp%d" % world},
            "tflops": tf,
            "roofline": {"bound": "tensor", "kernel": "all contraction kernels of the five layers", "achieved": tf / world,
                         "peak": peak, "unit": "TFLOP/s", "frac": tf / world / peak, "traffic": None,
                         "peak_source": "%s: 16-bit matmul burst %.1f TFLOP/s / 3 - of measured; sustained figure %.1f" %
                                        (peaks["source"], peaks["bf16_tflops"], (peaks.get("bf16_tflops_sustained") or 0) / 3.0),
                         "flops_per_step": flops, "layers": per_layer},
            "cpu_baseline": None, "e2e": None, "clocks": clocks, "gpu_launches": timed_launches,
        }
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()
    ctx.close()


def caffenet_layer_table():
    """(name, kind, geometry) of every CaffeNet layer at the bench's shapes, for the reference arm."""
    return [
        ("conv1", "conv", dict(D=3, n=227, o=96, k=11, s=4, p=0, g=1, needs_dx=False)),
        ("relu1", "relu", dict(D=96, n=55)), ("pool1", "pool", dict(D=96, n=55)), ("norm1", "lrn", dict(D=96, n=27)),
        ("conv2", "conv", dict(D=96, n=27, o=256, k=5, s=1, p=2, g=2, needs_dx=True)),
        ("relu2", "relu", dict(D=256, n=27)), ("pool2", "pool", dict(D=256, n=27)), ("norm2", "lrn", dict(D=256, n=13)),
        ("conv3", "conv", dict(D=256, n=13, o=384, k=3, s=1, p=1, g=1, needs_dx=True)), ("relu3", "relu", dict(D=384, n=13)),
        ("conv4", "conv", dict(D=384, n=13, o=384, k=3, s=1, p=1, g=2, needs_dx=True)), ("relu4", "relu", dict(D=384, n=13)),
        ("conv5", "conv", dict(D=384, n=13, o=256, k=3, s=1, p=1, g=2, needs_dx=True)), ("relu5", "relu", dict(D=256, n=13)),
        ("pool5", "pool", dict(D=256, n=13)),
        ("fc6", "fc", dict(D=256, n=6, o=4096)), ("relu6", "relu", dict(D=4096, n=1)), ("drop6", "dropout", dict(D=4096, n=1)),
        ("fc7", "fc", dict(D=4096, n=1, o=4096)), ("relu7", "relu", dict(D=4096, n=1)), ("drop7", "dropout", dict(D=4096, n=1)),
        ("fc8", "fc", dict(D=4096, n=1, o=1000)), ("loss", "softmax", dict(D=1000, n=1)),
    ]


def caffenet_reference_seconds(B, iters, log=None, kinds=None):
    """Seconds of one CaffeNet iteration (forward + backward of every layer) on the host cores through the reference's
    own CPU bridges, one bridge at a time on synthetic tensors of the layer's shapes: convolutions through its
    ParallelizedBridge with the partition count DeepNet uses (grouped layers as one bridge per channel slice - the
    reference bridge has no group concept), fully connected layers with all hardware threads in BLAS as DeepNet gives
    them, the parameter-free bridges as plain bridges.  Median of `iters` passes per layer; returns (total, per layer)."""
    from oracle import pyoracle
    ref = pyoracle.reference()
    if ref is None:
        return None, None
    rng = np.random.default_rng(99)
    parts = ref.default_partitions(B)
    hc = ref.hardware_concurrency()
    per = {}
    for name, kind, g in caffenet_layer_table():
        if kinds is not None and kind not in kinds:
            continue
        D, n = g["D"], g["n"]
        X = np.maximum(rng.standard_normal((B, D, n, n), dtype=np.float32), 0) if name != "conv1" else \
            rng.standard_normal((B, D, n, n), dtype=np.float32)
        if kind == "conv":
            o, k, s_, p_, grp = g["o"], g["k"], g["s"], g["p"], g["g"]
            m = (n + 2 * p_ - k) // s_ + 1
            W = (0.01 * rng.standard_normal((o, D // grp, k, k))).astype(np.float32)
            bias = np.zeros(o, np.float32)
            dY = rng.standard_normal((B, o, m, m), dtype=np.float32)
            Dg, og = D // grp, o // grp
            sec = 0.0
            for gi in range(grp):
                sec += ref.conv_time(np.ascontiguousarray(X[:, gi * Dg:(gi + 1) * Dg]), np.ascontiguousarray(W[gi * og:(gi + 1) * og]),
                                     np.ascontiguousarray(bias[gi * og:(gi + 1) * og]),
                                     np.ascontiguousarray(dY[:, gi * og:(gi + 1) * og]), k, s_, p_, parts, g["needs_dx"], 1, iters)[0]
        elif kind == "relu":
            t0 = time.perf_counter()
            for _ in range(iters):
                ref.relu(X, dY=X)
            sec = (time.perf_counter() - t0) / iters
        elif kind == "pool":
            m = (n - 3) // 2 + 1
            dY = rng.standard_normal((B, D, m, m), dtype=np.float32)
            t0 = time.perf_counter()
            for _ in range(iters):
                ref.maxpool(X, 3, 2, dY=dY)
            sec = (time.perf_counter() - t0) / iters
        elif kind == "lrn":
            sec = ref.lrn(X, 5, 1e-4, 0.75, dY=X, time_iters=iters)[2]
        elif kind == "fc":
            o = g["o"]
            W = (0.01 * rng.standard_normal((o, D, n, n))).astype(np.float32)
            dY = rng.standard_normal((B, o, 1, 1), dtype=np.float32)
            sec = ref.fc(X, W, np.ones(o, np.float32), dY=dY, blas_threads=hc, time_iters=iters)[4]
        elif kind == "dropout":
            sec = ref.dropout(X, 0.5, 1, dY=X, time_iters=iters)[3]
        else:
            labels = rng.integers(0, D, B).astype(np.float32)
            sec = ref.softmax_loss(X, labels, time_iters=iters)[3]
        per[name] = sec
        if log:
            log("  reference %-6s %8.1f ms" % (name, sec * 1e3))
    return sum(per.values()), per


def run_caffenet(args, rank, world, local_rank):
    """BASELINE configs 4 (one GPU) and 5 (2 / 4 / 8 GPUs): one CaffeNet training iteration - forward, backward, gradient
    all-reduce over NCCL (N > 1), SGD momentum step - at batch 256 per GPU on synthetic 3 x 227 x 227 images, built from
    the package's prototxt by the network builder."""
    import torch
    import torch.distributed as dist
    from caffecontroll_b200 import capi
    from caffecontroll_b200.bridge import Context, LogicalCube
    from caffecontroll_b200.net import Net, parse_prototxt, solver_from_message
    from caffecontroll_b200.parallel import Communicator, DeviceOps

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    B = args.batch or 256
    if world > 1:
        # torch.distributed (gloo, host side) only carries the NCCL id and the timing reductions; the gradient sums are
        # NCCL all-reduces issued by the library's own communicator
        dist.init_process_group("gloo")
    stream = torch.cuda.current_stream()
    ctx = Context(local_rank, stream=stream.cuda_stream)
    comm = None
    if world > 1:
        ids = [Communicator.unique_id() if rank == 0 else None]
        dist.broadcast_object_list(ids, src=0)
        comm = Communicator(ctx, world, rank, ids[0])
    ops = DeviceOps(ctx, comm=comm)
    nets_dir = os.path.join(ROOT, "caffecontroll_b200", "nets")
    with open(os.path.join(nets_dir, "caffenet_train.prototxt")) as f:
        net_param = parse_prototxt(f.read())
    with open(os.path.join(nets_dir, "caffenet_solver.prototxt")) as f:
        solver = solver_from_message(parse_prototxt(f.read()))
    split = tuple(n for n in args.model_parallel.split(",") if n) if world > 1 else ()
    net = Net(ctx, net_param, solver, B, ops=ops, loss_batch=B * world, algo=args.algo, model_parallel=split)
    rng = np.random.default_rng(5000 + rank)
    X = rng.standard_normal((B, 3, 227, 227), dtype=np.float32)
    labels = rng.integers(0, 1000, B).astype(np.float32)
    net.set_input(X, labels)
    flops = net.flops_forward + net.flops_backward
    lib, vp = ctx.lib, C.c_void_p

    def barrier():
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()

    def max_over_ranks(v):
        if world == 1:
            return v
        t = torch.tensor([v], dtype=torch.float64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    roof = tensor_roofline(load_peaks(), measure=(rank == 0))
    warm_steps = preheat(net.step, args.warmup, args.preheat_s, stream, lambda n: int(max_over_ranks(float(n))))
    loss0 = net.get_loss()
    barrier()
    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record(stream)
    counted = capi.kernel_launches()
    for _ in range(args.steps):
        net.step()
    timed_launches = capi.kernel_launches() - counted
    e1.record(stream)
    barrier()
    ms_step = max_over_ranks(e0.elapsed_time(e1)) / args.steps
    clocks = sampler.stop() if rank == 0 else None
    loss1 = net.get_loss()

    # ---- per-layer device times: the same steps again with events around every bridge pass
    prof_steps = max(1, min(args.steps, 5))
    names = net.names
    fwd_ms, bwd_ms = np.zeros(len(names)), np.zeros(len(names))
    plan_ms = {}
    for i, br in enumerate(net.bridges):
        if net.types[i] == "Convolution":
            lib.cct_conv_plan_enable_timing(br.plan, 1)
        elif net.types[i] == "InnerProduct" and br.plan:
            lib.cct_fc_plan_enable_timing(br.plan, 1)
    upd_ms = 0.0
    for _ in range(prof_steps):
        evs = []
        for i, br in enumerate(net.bridges):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream); br.forward(); b.record(stream)
            evs.append(("f", i, a, b))
        for i in range(len(net.bridges) - 1, -1, -1):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record(stream)
            (net.pbridges[i] if i in net.pbridges else net.bridges[i]).backward()
            b.record(stream)
            evs.append(("b", i, a, b))
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(stream)
        ops.allreduce_wait()
        for i in sorted(net.pbridges, reverse=True):
            net.pbridges[i].apply_update()
        b.record(stream)
        torch.cuda.synchronize()
        upd_ms += a.elapsed_time(b)
        for kind, i, a, b in evs:
            (fwd_ms if kind == "f" else bwd_ms)[i] += a.elapsed_time(b)
        for i, br in enumerate(net.bridges):
            t5 = (C.c_float * 5)()
            if net.types[i] == "Convolution":
                lib.cct_conv_plan_last_timings(br.plan, t5)
            elif net.types[i] == "InnerProduct" and br.plan:
                lib.cct_fc_plan_last_timings(br.plan, t5)
            else:
                continue
            plan_ms[i] = plan_ms.get(i, np.zeros(5)) + np.array(list(t5))
    fwd_ms /= prof_steps; bwd_ms /= prof_steps; upd_ms /= prof_steps
    for i, br in enumerate(net.bridges):  # the plans' own events sit between their kernels: off again for what follows
        if net.types[i] == "Convolution":
            lib.cct_conv_plan_enable_timing(br.plan, 0)
        elif net.types[i] == "InnerProduct" and br.plan:
            lib.cct_fc_plan_enable_timing(br.plan, 0)
    # N > 1: the step's gradient reductions on their own (nothing beside them), to compare with the backward pass they
    # hide behind: every layer's flat gradient buffer, begun back to back, one wait.
    ar_alone_ms = None
    if world > 1:
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        barrier()
        a.record(stream)
        for _, pb in reversed(net.param_bridges()):
            pb.begin_allreduce()
        net.ops.allreduce_wait()
        b.record(stream)
        torch.cuda.synchronize()
        ar_alone_ms = max_over_ranks(a.elapsed_time(b))
    layers, contraction = {}, []
    hbm = load_peaks()["hbm_gbs"]
    for i, name in enumerate(names):
        rec = {"type": net.types[i], "forward_ms": float(fwd_ms[i]), "backward_ms": float(bwd_ms[i])}
        if i in plan_ms:
            k = plan_ms[i] / prof_steps
            br = net.bridges[i]
            F = (2.0 * br.oD * (br.K * br.K * br.iD // br.group) * br.oR * br.oC * B if net.types[i] == "Convolution"
                 else 2.0 * br.oD * br.in_features * B)
            rec.update(forward_kernel_ms=float(k[0]), wgrad_kernel_ms=float(k[1] + k[2]), dgrad_kernel_ms=float(k[3]),
                       gflop_per_pass=F / 1e9)
            for pname, ms in (("forward", k[0]), ("wgrad", k[1] + k[2]), ("dgrad", k[3])):
                if ms > 0:
                    rec[pname + "_tflops"] = F / (ms * 1e-3) / 1e12
                    contraction.append((ms, F, "%s %s" % (name, pname)))
        layers[name] = rec
    dom_ms, dom_F, dom_name = max(contraction) if contraction else (0.0, 0.0, "")
    hbm_passes = {}
    for i, name in enumerate(names):  # the HBM-bound bridges: algorithmic bytes over measured time
        br, t = net.bridges[i], net.types[i]
        n_in = br.iB * br.iD * br.iR * br.iC
        n_out = br.oB * br.oD * br.oR * br.oC
        if t == "Pooling":
            hbm_passes[name + " forward"] = (4.0 * n_in + 8.0 * n_out, fwd_ms[i])
        elif t == "LRN":
            kept = 4.0 if br.denoms is not None else 0.0  # the denominator cube: written forward, read backward
            hbm_passes[name + " forward"] = ((8.0 + kept) * n_in, fwd_ms[i])
            hbm_passes[name + " backward"] = ((12.0 + kept) * n_in, bwd_ms[i])  # X, dY (, scale) in, dX out
    hbm_table = {k: {"ms": float(ms), "bytes": b, "achieved_gbs": b / ms / 1e6, "frac": b / ms / 1e6 / hbm}
                 for k, (b, ms) in hbm_passes.items() if ms > 0}

    # ---- end to end: every step uploads its images and labels from pinned host memory and reads the loss back
    hX = torch.from_numpy(X).pin_memory()
    hL = torch.from_numpy(labels).pin_memory()
    copy_stream = torch.cuda.Stream()
    cctx = Context(local_rank, stream=copy_stream.cuda_stream)
    stage = [LogicalCube(ctx, 227, 227, 3, B), LogicalCube(ctx, 227, 227, 3, B)]
    stage_l = [LogicalCube(ctx, 1, 1, 1, B), LogicalCube(ctx, 1, 1, 1, B)]
    main_ptr, main_labels_ptr = net.input.p_data_cube.ptr, net.labels.ptr
    up_done = [torch.cuda.Event(), torch.cuda.Event()]
    used = [torch.cuda.Event(), torch.cuda.Event()]

    up_begin = [torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)]
    up_end = [torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)]

    def upload(slot):  # next batch -> staging buffer `slot`, on the copy stream
        copy_stream.wait_event(used[slot])
        up_begin[slot].record(copy_stream)
        capi.check(lib.cct_memcpy_h2d(cctx.h, vp(stage[slot].ptr), vp(hX.data_ptr()), X.nbytes), "h2d", cctx.h)
        capi.check(lib.cct_memcpy_h2d(cctx.h, vp(stage_l[slot].ptr), vp(hL.data_ptr()), labels.nbytes), "h2d", cctx.h)
        up_end[slot].record(copy_stream)
        up_done[slot].record(copy_stream)

    # The loss of every step is read back into pinned host memory by a copy queued behind the step; the host looks at it
    # one step later (after that copy's event), so it keeps queueing the next iteration's launches meanwhile.
    loss_host = C.c_void_p()
    capi.check(lib.cct_malloc_host(ctx.h, 8, C.byref(loss_host)), "cct_malloc_host", ctx.h)
    loss_view = (C.c_float * 2).from_address(loss_host.value)
    loss_done = [torch.cuda.Event(), torch.cuda.Event()]
    e2e_losses = []

    def e2e_step(slot, prev):
        stream.wait_event(up_done[slot])
        net.input.p_data_cube.ptr, net.labels.ptr = stage[slot].ptr, stage_l[slot].ptr
        net.loss_bridge.p_data_labels = net.labels
        net.step()
        used[slot].record(stream)
        net.read_loss_into(loss_host.value + 4 * slot)  # device -> host read of the step's result
        loss_done[slot].record(stream)
        upload(slot ^ 1)  # the next step's batch travels while this step computes
        if prev is not None:
            loss_done[prev].synchronize()
            e2e_losses.append(float(loss_view[prev]))

    for e in used:
        e.record(stream)
    upload(0)
    e2e_step(0, None)
    # The per-layer passes above ran with pauses, so the GPU is cooler than in the device-timed loop and would run the
    # next few dozen steps at a higher clock: the same number of untimed steps as that loop's pre-heat comes first.
    k = 0
    for _ in range(warm_steps if args.e2e_steps > 1 else 0):
        e2e_step((k + 1) & 1, k & 1)
        k += 1
    barrier()
    e2e_losses.clear()
    t0 = time.perf_counter()
    for _ in range(args.e2e_steps):
        e2e_step((k + 1) & 1, k & 1)
        k += 1
    torch.cuda.synchronize()
    e2e_losses.append(float(loss_view[k & 1]))  # the last step's loss: its copy has completed
    e2e_s = max_over_ranks((time.perf_counter() - t0) / args.e2e_steps)
    h2d_ms = max(up_begin[i].elapsed_time(up_end[i]) for i in (0, 1))  # the last two uploads, device-timed
    capi.check(lib.cct_free_host(ctx.h, loss_host), "cct_free_host", ctx.h)
    net.input.p_data_cube.ptr, net.labels.ptr = main_ptr, main_labels_ptr
    torch.cuda.synchronize()

    if rank == 0:
        cpu = None
        if world == 1 and not args.no_cpu_baseline:
            total, per = caffenet_reference_seconds(B, 1)
            if total:
                from oracle import pyoracle
                ref = pyoracle.reference()
                cpu = dict(value=B / total, unit="images/s", cores=ref.hardware_concurrency(), kind="reference",
                           sample="one forward + backward pass of every CaffeNet layer over a %d-image batch through the "
                                  "reference's CPU bridges, one bridge at a time (convolutions: %d partitions x 1 BLAS thread; "
                                  "fully connected: %d BLAS threads), times summed; %s" %
                                  (B, ref.default_partitions(B), ref.hardware_concurrency(), ref.blas_config()),
                           seconds_per_step=total)
        tf = world * flops / (ms_step * 1e-3) / 1e12
        ach = dom_F / (dom_ms * 1e-3) / 1e12 if dom_ms > 0 else 0.0
        dom_traffic, dom_traffic_source = caffenet_traffic(dom_name, B)
        line = {
            "metric": METRIC, "value": world * B / (ms_step * 1e-3), "unit": "images/s", "n_gpus": world,
            "steps": args.steps, "warmup": warm_steps, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "caffenet (BASELINE config %d: full CaffeNet iteration, batch %d per GPU)" % (4 if world == 1 else 5, B),
                       "batch_per_gpu": B, "global_batch": B * world,
                       "step": "forward + backward of all 23 layers + NCCL all-reduce of the %.1f M parameter gradients (N>1, "
                               "begun per layer, overlapping the layers below) + SGD momentum step" % (net.num_parameters() / 1e6),
                       "fusions": net.fused, "l2": "inputs larger than L2 (%.1f GB of activations and gradients per step)" %
                       (sum(c.n_elements * 4 for c in net._cubes) / 1e9),
                       "parallelism": "dp%d" % world + (" + %s split by output depth" % "/".join(split) if split else "")},
            "tflops": tf, "flops_per_step": flops,
            "roofline": {"bound": "tensor", "kernel": dom_name, "achieved": ach, "peak": roof["peak"], "unit": "TFLOP/s",
                         "frac": ach / roof["peak"] if roof["peak"] else None, "traffic": dom_traffic,
                         "peak_source": roof["source"], "peak_sustained": roof["peak_sustained"],
                         "frac_of_sustained": ach / roof["peak_sustained"] if roof["peak_sustained"] else None,
                         "whole_step_achieved": tf / world, "whole_step_frac": tf / world / roof["peak"],
                         "whole_step_frac_of_sustained": tf / world / roof["peak_sustained"] if roof["peak_sustained"] else None,
                         "flops_per_launch": dom_F, "ms_per_launch": dom_ms,
                         "timing": "CUDA events on the launching stream around every kernel group, mean of %d steps run "
                                   "right after the timed region" % prof_steps},
            "layers": layers, "update_ms": upd_ms, "hbm_bound_passes": hbm_table,
            "loss": {"after_warmup": loss0, "after_timed_steps": loss1},
            "cpu_baseline": cpu,
            "e2e": {"value": world * B / e2e_s, "unit": "images/s", "h2d_bytes_per_step": int(X.nbytes + labels.nbytes),
                    "d2h_bytes_per_step": 4, "ms_per_step": e2e_s * 1e3, "steps": args.e2e_steps,
                    "how": "each step: images and labels copied from pinned host memory (double-buffered on a copy stream), "
                           "the iteration, the loss copied back to pinned host memory and read by the host one step later",
                    "last_loss": e2e_losses[-1] if e2e_losses else None, "h2d_ms_per_upload": h2d_ms,
                    "h2d_gbs": X.nbytes / (h2d_ms * 1e-3) / 1e9 if h2d_ms > 0 else None},
            "clocks": clocks, "gpu_launches": timed_launches,
            "allreduce_bytes_per_step": 4 * net.num_parameters() if world > 1 else 0,
            "allreduce_ms_alone": ar_alone_ms,
        }
        if cpu:
            cpu.pop("seconds_per_step", None)
        if dom_traffic is not None:
            line["roofline"]["traffic_source"] = ("ncu dram__bytes_read.sum + dram__bytes_write.sum of this kernel at "
                                                  "batch 256, scaled by the batch ratio: " + dom_traffic_source)
        print(json.dumps(line), flush=True)
    for c in stage + stage_l:
        c.free()
    cctx.close()
    net.close()
    if comm is not None:
        comm.close()
    if world > 1:
        dist.destroy_process_group()
    ctx.close()


def run_caffenet_reference_arm(args, rank, world):
    if rank != 0:
        return
    # A step of this arm is a bounded sample of the workload: one forward + backward pass of every layer over B images,
    # B = 256 cut down (in multiples of 16, the reference's partition count) until `steps` of them fit in about 150 s at
    # the ~45 images/s these host cores deliver; images/s barely depends on the batch on the CPU.
    steps = max(1, args.steps)
    B = args.batch or max(16, min(256, (150 * 45 // steps) // 16 * 16))
    log = lambda m: print(m, file=sys.stderr, flush=True)
    total, per = caffenet_reference_seconds(B, steps, log)
    if total is None:
        print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libcct_ref.so (the reference's CPU code) is not built"}))
        return
    from oracle import pyoracle
    ref = pyoracle.reference()
    val = B / total
    cpu = dict(value=val, unit="images/s", cores=ref.hardware_concurrency(), kind="reference",
               sample="each step = forward + backward of every CaffeNet layer over one %d-image batch through the reference's "
                      "CPU bridges, one bridge at a time, median of %d passes per layer, times summed (convolutions: %d "
                      "partitions x 1 BLAS thread, fully connected: %d BLAS threads); %s" %
                      (B, max(1, args.steps), ref.default_partitions(B), ref.hardware_concurrency(), ref.blas_config()))
    line = {"impl": "reference", "metric": METRIC, "value": val, "unit": "images/s", "n_gpus": args.gpus, "steps": args.steps,
            "warmup": args.warmup, "ms_per_step": total * 1e3, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": {"workload": "caffenet (BASELINE config %d: full CaffeNet iteration, batch %d per GPU)" % (4 if world == 1 else 5, B),
                       "batch_per_gpu": B, "global_batch": B * world, "parallelism": "dp%d" % world},
            "layers_ms": {k: v * 1e3 for k, v in per.items()}, "cpu_baseline": cpu,
            "e2e": {"value": val, "unit": "images/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}, "gpu_launches": 0}
    print(json.dumps(line), flush=True)


def config_of(args, w, world):
    return {"workload": args.workload, "batch_per_gpu": w["B"], "global_batch": w["B"] * world,
            "in": "%dx%dx%d" % (w["D"], w["n"], w["n"]), "filters": "%d x %dx%d stride %d pad %d groups %d" %
            (w["o"], w["k"], w["k"], w["s"], w["p"], w["g"]),
            "step": ("forward (+ReLU) + fused backward (dY from max-pool indices and ReLU sign; dX masked by the input's "
                     "sign; dW, db) + gradient all-reduce (N>1) + SGD momentum step") if w.get("pool") else
            "forward + backward (dX, dW, db) + gradient all-reduce (N>1) + SGD momentum step",
            "l2": "inputs larger than L2 (X + dY per step exceed 126 MB)" if
            4 * w["B"] * (w["D"] * w["n"] ** 2 + w["o"] * out_size(w) ** 2) > 126e6 else "L2 flushed between steps",
            "parallelism": "dp%d" % world}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--workload", default="caffenet", choices=["caffenet"] + sorted(WORKLOADS) + ["caffenet_convs"])
    ap.add_argument("--algo", type=int, default=0, help="0 auto, 1 SIMT fp32, 2 tcgen05 3xTF32")
    ap.add_argument("--e2e-steps", type=int, default=20)
    ap.add_argument("--preheat-s", type=float, default=1.0,
                    help="untimed warm-up runs until at least this much device time has passed (and --warmup steps)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--batch", type=int, default=0, help="override the per-GPU batch (profiling on a small case)")
    ap.add_argument("--model-parallel", default="", help="comma-separated InnerProduct layers to split over the ranks by "
                    "output depth instead of by batch (N > 1 only; the default and the BASELINE configs are data parallel)")
    args = ap.parse_args()
    args.warmup = max(args.warmup, 3) if args.impl == "ours" else args.warmup
    if args.workload == "caffenet":
        env = [int(os.environ.get(k, d)) for k, d in (("RANK", "0"), ("WORLD_SIZE", "1"), ("LOCAL_RANK", "0"))]
        if args.impl == "reference":
            run_caffenet_reference_arm(args, env[0], env[1])
        else:
            run_caffenet(args, env[0], env[1], env[2])
        return
    if args.workload == "caffenet_convs":
        if args.impl == "reference":
            if int(os.environ.get("RANK", "0")) == 0:  # the five convolution bridges of the reference, one at a time
                steps = max(1, args.steps)
                B = args.batch or max(16, min(256, (150 * 60 // steps) // 16 * 16))
                total, per = caffenet_reference_seconds(B, steps, lambda m: print(m, file=sys.stderr, flush=True), kinds=("conv",))
                if total is None:
                    print(json.dumps({"impl": "reference", "unavailable": "oracle/_ref/libcct_ref.so (the reference's CPU code) is not built"}))
                    return
                from oracle import pyoracle
                ref = pyoracle.reference()
                print(json.dumps({
                    "impl": "reference", "metric": METRIC, "value": B / total, "unit": "images/s", "n_gpus": args.gpus,
                    "steps": args.steps, "warmup": args.warmup, "ms_per_step": total * 1e3, "higher_is_better": True,
                    "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
                    "config": {"workload": "caffenet_convs (conv1-conv5, batch %d per GPU)" % B, "batch_per_gpu": B},
                    "layers_ms": {k: v * 1e3 for k, v in per.items()},
                    "cpu_baseline": {"value": B / total, "unit": "images/s", "cores": ref.hardware_concurrency(), "kind": "reference",
                                     "sample": "each step = forward + backward of the five convolution layers over one %d-image "
                                               "batch through the reference's ParallelizedBridge, one layer at a time" % B},
                    "e2e": {"value": B / total, "unit": "images/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
                    "gpu_launches": 0}), flush=True)
            return
        run_conv_stack(args, int(os.environ.get("RANK", "0")), int(os.environ.get("WORLD_SIZE", "1")),
                       int(os.environ.get("LOCAL_RANK", "0")))
        return
    w = dict(WORKLOADS[args.workload])
    if args.batch:
        w["B"] = args.batch
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local_rank = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        run_reference_arm(args, w, rank, world)
        return

    import torch
    import torch.distributed as dist
    from caffecontroll_b200 import capi
    from caffecontroll_b200.bridge import Context

    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    if world > 1:
        dist.init_process_group("nccl", device_id=dev)
    stream = torch.cuda.current_stream()
    ctx = Context(local_rank, stream=stream.cuda_stream)
    lib = ctx.lib

    B, D, n, o, k, g = w["B"], w["D"], w["n"], w["o"], w["k"], w["g"]
    m = out_size(w)
    X, W, bias, dY = synth(w, 1000 * (rank + 1))
    nw = W.size
    # This rank's partition of the mini-batch, resident in HBM before the timed region starts.
    from caffecontroll_b200.bridge import ConvolutionBridge, Layer, LogicalCube
    from caffecontroll_b200.parallel import DeviceOps, ParallelizedBridge, SolverParameter
    xin = Layer(LogicalCube.from_numpy(ctx, X), LogicalCube(ctx, n, n, D, B))
    out = Layer(LogicalCube(ctx, m, m, o, B), LogicalCube.from_numpy(ctx, dY))
    conv = ConvolutionBridge(xin, out, k, w["s"], w["p"], g, True, algo=args.algo)
    pbridge = ParallelizedBridge(conv, SolverParameter(SOLVER["base_lr"], "step", 0.1, 100000, momentum=SOLVER["momentum"],
                                                       weight_decay=SOLVER["weight_decay"]), DeviceOps(ctx))
    conv.p_model_cube.upload(W)
    conv.p_bias_cube.upload(bias)
    plan = conv.plan
    algo = C.c_int(conv.algo)
    vp = C.c_void_p

    remnants = {}
    if w.get("pool"):
        # conv -> ReLU -> max-pool behind the layer: the pooled gradient dP ~ N(0,1) is what arrives from above.
        pk, ps = w["pool"]
        mp = (m - pk) // ps + 1
        conv.fuse_relu, conv.fuse_relu_backward = True, True
        pooled, idx = LogicalCube(ctx, mp, mp, o, B), LogicalCube(ctx, mp, mp, o, B, np.int32)
        dP = LogicalCube.from_numpy(ctx, np.random.default_rng(1000 * (rank + 1) + 7).standard_normal(
            (B, o, mp, mp), dtype=np.float32))
        conv.forward()
        capi.check(lib.cct_maxpool_forward(ctx.h, vp(out.p_data_cube.ptr), vp(pooled.ptr), vp(idx.ptr), B * o, m, pk, ps),
                   "cct_maxpool_forward", ctx.h)
        conv.fuse_pool_relu_backward(dP, idx, pk, ps)
        # The mask pass alone (HBM-bound): reads A, idx, dP once, writes dY once.
        ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
        scratch = LogicalCube(ctx, m, m, o, B)
        for it in range(13):
            if it == 3:
                ev[0].record(stream)
            capi.check(lib.cct_pool_relu_backward(ctx.h, vp(out.p_data_cube.ptr), vp(idx.ptr), vp(dP.ptr), vp(scratch.ptr),
                                                  B * o, m, pk, ps), "cct_pool_relu_backward", ctx.h)
        ev[1].record(stream)
        torch.cuda.synchronize()
        ms = ev[0].elapsed_time(ev[1]) / 10
        nbytes = 4.0 * B * o * (2 * m * m + 2 * mp * mp)
        hbm = load_peaks().get("hbm_gbs")
        remnants["pool_relu_mask_pass"] = {"ms": ms, "bytes": nbytes, "achieved_gbs": nbytes / ms / 1e6,
                                           "peak_gbs": hbm, "frac": nbytes / ms / 1e6 / hbm if hbm else None}
        scratch.free()

    def step():
        pbridge.forward()   # cct_conv_forward
        pbridge.backward()  # cct_conv_backward (dX, dW, db) -> all-reduce(SUM) of dW|db over ranks -> cct_sgd_step x2

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    roof = tensor_roofline(load_peaks(), measure=(rank == 0))
    def agree(n):
        if world == 1:
            return n
        t = torch.tensor([n], device=dev, dtype=torch.int64)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return int(t.item())

    warm_steps = preheat(step, args.warmup, args.preheat_s, stream, agree)
    barrier()
    sampler = ClockSampler(local_rank)
    if rank == 0:
        sampler.start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record(stream)
    counted = capi.kernel_launches()
    for _ in range(args.steps):
        step()
    timed_launches = capi.kernel_launches() - counted
    e1.record(stream)
    barrier()
    ms_total = e0.elapsed_time(e1)
    if world > 1:
        t = torch.tensor([ms_total], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_total = float(t.item())
    ms_step = ms_total / args.steps

    # Per-kernel durations: same steps again with CUDA events around each kernel group on the launching stream.
    lib.cct_conv_plan_enable_timing(plan, 1)
    acc = np.zeros(5)
    prof_steps = min(args.steps, 10)
    for _ in range(prof_steps):
        step()
        t5 = (C.c_float * 5)()
        capi.check(lib.cct_conv_plan_last_timings(plan, t5), "timings", ctx.h)
        acc += np.array(list(t5))
    lib.cct_conv_plan_enable_timing(plan, 0)
    clocks = sampler.stop() if rank == 0 else None
    k_ms = acc / prof_steps
    F = gemm_flops(w)
    passes = {"forward": k_ms[0], "wgrad": k_ms[1], "dgrad": k_ms[3]}
    wg_gather = (D // g) * k * k >= 512  # the library's rule: long lowered matrices take the gather-kernel weight gradient
    tensor_peak = roof["peak"]
    dom = max(passes, key=lambda x: passes[x])
    ach = F / (passes[dom] * 1e-3) / 1e12 if passes[dom] > 0 else 0.0
    traffic, traffic_source = dram_traffic(args.workload, w, dom, B) if algo.value == 2 else (None, None)
    roofline = {
        "bound": "tensor", "kernel": {"forward": "gather_conv_kernel (forward)", "dgrad": "gather_conv_kernel (data gradient)",
                                      "wgrad": "split_dy_kernel + gather_conv_kernel (weight gradient)" if wg_gather else "wgrad_kernel"}[dom] if algo.value == 2 else "simt_%s" % dom,
        "pass": dom, "achieved": ach, "peak": tensor_peak, "unit": "TFLOP/s", "frac": ach / tensor_peak,
        "traffic": traffic,
        "peak_source": roof["source"], "peak_sustained": roof["peak_sustained"],
        "frac_of_sustained": ach / roof["peak_sustained"] if roof["peak_sustained"] else None,
        "whole_step_frac": (3 * F / (ms_step * 1e-3) / 1e12) / tensor_peak,
        "flops_per_launch": F, "ms_per_launch": passes[dom],
        "timing": "CUDA events around each kernel group on the launching stream, mean of %d steps run right after the "
                  "timed region" % prof_steps,
        "passes_ms": {"forward": k_ms[0], "wgrad": k_ms[1], "wgrad_reduce": k_ms[2], "dgrad": k_ms[3],
                      "forward_repack": k_ms[4]},
        "passes_tflops": {p: (F / (v * 1e-3) / 1e12 if v > 0 else None) for p, v in passes.items()},
    }
    if traffic is not None:
        roofline["traffic_source"] = ("ncu dram__bytes_read.sum of the small-case capture scaled by the batch ratio, plus "
                                      "the pass's output bytes: " + traffic_source)

    # End to end through the host-buffer C-ABI calls: pinned host memory, copies inside the timed region.
    hX, hW, hb, hdY = (torch.from_numpy(a).pin_memory() for a in (X, W, bias, dY))
    hY = torch.empty((B, o, m, m)).pin_memory()
    hdX, hdW, hdb = torch.empty(X.shape).pin_memory(), torch.empty(W.shape).pin_memory(), torch.empty(o).pin_memory()

    def e2e_step():
        capi.check(lib.cct_conv_forward_host(plan, vp(hX.data_ptr()), vp(hW.data_ptr()), vp(hb.data_ptr()),
                                             vp(hY.data_ptr()), 0), "forward_host", ctx.h)
        capi.check(lib.cct_conv_backward_host(plan, None, None, vp(hdY.data_ptr()), vp(hdX.data_ptr()),
                                              vp(hdW.data_ptr()), vp(hdb.data_ptr())), "backward_host", ctx.h)
        return float(hdb[0])  # the step's result is read on the host

    e2e_step()
    barrier()
    t0 = time.perf_counter()
    for _ in range(args.e2e_steps):
        e2e_step()
    torch.cuda.synchronize()
    e2e_s = (time.perf_counter() - t0) / args.e2e_steps
    if world > 1:
        t = torch.tensor([e2e_s], device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        e2e_s = float(t.item())
    h2d = 4 * (X.size + W.size + bias.size + dY.size)
    d2h = 4 * (hY.numel() + X.size + W.size + bias.size)

    conv.close()
    if rank == 0:
        cpu = None
        if world == 1 and not args.no_cpu_baseline:
            cpu = cpu_reference_time(w, 3, 1, False)
            cpu.pop("seconds_per_step", None)
        line = {
            "metric": METRIC, "value": world * B / (ms_step * 1e-3), "unit": "images/s", "n_gpus": world,
            "steps": args.steps, "warmup": warm_steps, "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": dict(config_of(args, w, world), algo={1: "simt_fp32", 2: "tcgen05_3xtf32"}[algo.value]),
            "tflops": world * 3 * F / (ms_step * 1e-3) / 1e12,
            "roofline": roofline, "cpu_baseline": cpu,
            "e2e": {"value": world * B / e2e_s, "unit": "images/s", "h2d_bytes_per_step": h2d,
                    "d2h_bytes_per_step": d2h, "ms_per_step": e2e_s * 1e3, "steps": args.e2e_steps},
            "clocks": clocks, "gpu_launches": timed_launches,
        }
        if remnants:
            line["hbm_bound_passes"] = remnants
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()
    ctx.close()


if __name__ == "__main__":
    main()
