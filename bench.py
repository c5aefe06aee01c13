#!/usr/bin/env python
"""Benchmark of the spatial-graph hot path: binned kNN query points per second.

    python bench.py --gpus N --steps K --warmup W            # this implementation (sm_100a)
    python bench.py --impl reference --steps K --warmup W     # the reference's CPU path

A step is one forward + backward pass of binned_select_knn over one batch of synthetic
input: the single-event workload of the headline metric (200 000 points, D = 4, K = 32,
50-component Gaussian mixture; fastgraphcompute_b200.synthetic.c2_gaussian_mixture).
With N > 1 every rank (one process per GPU, launched by torch.distributed.run) works on
its own event of that size -- events are independent, so there is no data-path
collective -- and the reported value is the whole-job aggregate (weak scaling).

One JSON line is printed by rank 0.  `value` is measured with the inputs resident in
HBM; `e2e` is measured through the public API from pinned HOST buffers (host->device
copies of coordinates, row splits and upstream gradient, device->host copies of
indices, squared distances and coordinate gradients inside the timed region).
"""
import argparse
import json
import os
import statistics
import subprocess
import sys
import threading
import time

ROOT = os.path.dirname(os.path.abspath(__file__))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

METRIC = "binned_knn_query_points_per_sec_K32_D4"
UNIT = "points/s"
WORKLOAD = "c2: single-event binned kNN fwd+bwd, N=200000, D=4, K=32, 50-component Gaussian mixture sigma=0.02"
L2_FLUSH_BYTES = 256 << 20

# DRAM traffic of the 33 launches of one forward on this workload (search by groups): dram__bytes_read.sum +
# dram__bytes_write.sum of the ncu capture summarised in profiles/knn_c2_step_launch_list.md, caches cold for every launch.
FORWARD_DRAM_TRAFFIC_BYTES = 133900000


def env_int(name, default):
    try:
        return int(os.environ.get(name, default))
    except ValueError:
        return default


def measured_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return 6650.0, "fallback"


class ClockSampler:
    """SM clock and throttle-reason samples during the timed region.  Reads NVML directly
    (a few hundred samples per second, read-only queries); falls back to `nvidia-smi -lms`."""

    REASONS = {0x8: "hw_slowdown", 0x40: "hw_thermal_slowdown", 0x20: "sw_thermal_slowdown", 0x4: "sw_power_cap"}

    def __init__(self, gpu_uuid):
        self.samples = []          # (time, sm_mhz, reasons bitmask)
        self.max_mhz = None
        self._stop = False
        self.proc = None
        self.thread = None
        try:
            import pynvml
            pynvml.nvmlInit()
            h = pynvml.nvmlDeviceGetHandleByUUID(gpu_uuid)
            self.max_mhz = float(pynvml.nvmlDeviceGetMaxClockInfo(h, pynvml.NVML_CLOCK_SM))

            def loop():
                while not self._stop:
                    try:
                        mhz = pynvml.nvmlDeviceGetClockInfo(h, pynvml.NVML_CLOCK_SM)
                        try:
                            rs = pynvml.nvmlDeviceGetCurrentClocksEventReasons(h)
                        except Exception:
                            rs = pynvml.nvmlDeviceGetCurrentClocksThrottleReasons(h)
                        self.samples.append((time.time(), float(mhz), int(rs)))
                    except Exception:
                        pass
                    time.sleep(0.004)

            self.thread = threading.Thread(target=loop, daemon=True)
            self.thread.start()
        except Exception:
            self._start_smi(gpu_uuid)

    def _start_smi(self, gpu_id):
        fields = ("clocks.sm,clocks.max.sm,clocks_event_reasons.hw_slowdown,"
                  "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
                  "clocks_event_reasons.sw_power_cap")
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(gpu_id), "--query-gpu=" + fields, "--format=csv,noheader,nounits",
                 "-lms", "20"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)

            def read():
                bits = (0x8, 0x40, 0x20, 0x4)
                for line in self.proc.stdout:
                    parts = [p.strip() for p in line.split(",")]
                    try:
                        mask = sum(b for b, v in zip(bits, parts[2:6]) if v.lower() == "active")
                        self.max_mhz = float(parts[1])
                        self.samples.append((time.time(), float(parts[0]), mask))
                    except (ValueError, IndexError):
                        continue

            self.thread = threading.Thread(target=read, daemon=True)
            self.thread.start()
        except Exception:
            self.proc = None

    def stop(self):
        self._stop = True
        if self.proc is not None:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self, t0, t1):
        under = [r for r in self.samples if t0 <= r[0] <= t1 + 0.02] or list(self.samples)
        if not under:
            return {"sm_mhz": None, "sm_max_mhz": self.max_mhz, "reasons": [], "samples": 0}
        mask = 0
        for r in under:
            mask |= r[2]
        reasons = sorted(name for bit, name in self.REASONS.items() if mask & bit)
        return {"sm_mhz": statistics.median(r[1] for r in under), "sm_max_mhz": self.max_mhz,
                "reasons": reasons, "samples": len(under)}


def gpu_identifier(torch, dev_index):
    try:
        u = str(torch.cuda.get_device_properties(dev_index).uuid)
        return u if u.startswith("GPU-") else "GPU-" + u
    except Exception:
        vis = os.environ.get("CUDA_VISIBLE_DEVICES")
        if vis:
            return vis.split(",")[dev_index]
        return str(dev_index)


# --------------------------------------------------------------------------- reference arm

def cpu_reference_fwd_bwd(workload, torch):
    """One forward + backward of the reference's own CPU ops (oracle/_ref) or, where that
    library is absent, of the C restatement (oracle/).  Returns (seconds, kind)."""
    from oracle import ref_ops
    if ref_ops.available():
        coords = workload.coords.clone().requires_grad_(True)
        t0 = time.perf_counter()
        idx, dist = ref_ops.ref_binned_select_knn(workload.K, coords, workload.row_splits)
        (dist * workload.grad_distsq).sum().backward()
        return time.perf_counter() - t0, "reference"
    from oracle import oracle
    c = workload.coords.numpy()
    t0 = time.perf_counter()
    idx, dist = oracle.binned_select_knn(workload.K, c, workload.row_splits.numpy())
    oracle.binned_select_knn_grad(workload.grad_distsq.numpy(), idx, c)
    return time.perf_counter() - t0, "port"


def load_synthetic_standalone():
    """The workload generators, loaded from their file without importing the package around them
    (the package loads the CUDA library on import; the reference arm must not map it)."""
    import importlib.util
    spec = importlib.util.spec_from_file_location(
        "fgc_bench_synthetic", os.path.join(ROOT, "fastgraphcompute_b200", "synthetic.py"))
    mod = importlib.util.module_from_spec(spec)
    sys.modules[spec.name] = mod       # dataclasses looks the defining module up by name
    spec.loader.exec_module(mod)
    return mod


def run_reference(args):
    """The reference's own CPU ops on the full headline workload, every step the same 200 000
    points as the GPU arm (about 4 s per step on one core; its loops are single-threaded)."""
    rank = env_int("RANK", 0)
    if rank != 0:
        return
    import torch
    synthetic = load_synthetic_standalone()
    w = synthetic.c2_gaussian_mixture()
    kind = "reference"
    for _ in range(args.warmup):
        cpu_reference_fwd_bwd(w, torch)
    times = []
    for _ in range(args.steps):
        t, kind = cpu_reference_fwd_bwd(w, torch)
        times.append(t)
    total = sum(times)
    value = w.n_points * args.steps / total
    sample = "the full workload every step (%d points, forward + backward), %d steps" % (w.n_points, args.steps)
    line = {
        "impl": "reference", "metric": METRIC, "value": value, "unit": UNIT,
        "n_gpus": args.gpus, "steps": args.steps, "warmup": args.warmup,
        "ms_per_step": 1e3 * total / args.steps, "higher_is_better": True, "scaling": "weak",
        "vs_baseline": None, "dtype": "f32", "data": "synthetic",
        "config": {"workload": WORKLOAD, "device": "host CPU", "n_points_per_step": w.n_points},
        "cpu_baseline": {"value": value, "unit": UNIT, "cores": 1, "kind": kind, "sample": sample,
                         "aten_threads": torch.get_num_threads(),
                         "note": "the reference's kNN, binning and gradient loops are single-threaded"},
        "e2e": {"value": value, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
        "gpu_launches": 0,
    }
    print(json.dumps(line), flush=True)


# --------------------------------------------------------------------------- this implementation

def run_b200(args):
    import torch
    import torch.distributed as dist

    world = env_int("WORLD_SIZE", 1)
    rank = env_int("RANK", 0)
    local_rank = env_int("LOCAL_RANK", 0)
    if not torch.cuda.is_available():
        raise SystemExit("bench.py: no CUDA device; this implementation has no CPU path")
    torch.cuda.set_device(local_rank)
    dev = torch.device("cuda", local_rank)
    if world > 1:
        pg_options = None
        if os.environ.get("FGC_BENCH_NCCL_HIGH_PRIORITY", "1") != "0":
            # the exchange of finished rows runs beside the search of the next group, which fills
            # every SM: NCCL's kernels get their CTAs sooner from a high-priority stream
            try:
                pg_options = dist.ProcessGroupNCCL.Options(is_high_priority_stream=True)
            except Exception:             # noqa: BLE001
                pg_options = None
        dist.init_process_group("nccl", device_id=dev, pg_options=pg_options)

    import fastgraphcompute_b200 as fgc
    from fastgraphcompute_b200 import _cabi, synthetic

    sections = set() if args.no_gravnet else {x for x in args.sections.split(",") if x and x != "none"}

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize(dev)

    def max_over_ranks(x):
        if world == 1:
            return x
        t = torch.tensor([x], dtype=torch.float64, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
        return float(t.item())

    w = synthetic.c2_gaussian_mixture(seed=rank)
    n, K = w.n_points, w.K
    h_coords = w.coords.pin_memory()
    h_rs = w.row_splits.pin_memory()
    h_grad = w.grad_distsq.pin_memory()
    d_coords = h_coords.to(dev)
    d_rs = h_rs.to(dev)
    d_grad = h_grad.to(dev)
    flush = torch.empty(L2_FLUSH_BYTES, dtype=torch.uint8, device=dev)

    fwd_marks = []

    def step_resident(mark=False):
        c = d_coords.detach().requires_grad_(True)
        idx, dsq = fgc.binned_select_knn(K, c, d_rs)
        if mark:
            e = torch.cuda.Event(enable_timing=True)
            e.record()
            fwd_marks.append(e)
        dsq.backward(d_grad)
        return idx, dsq, c.grad

    sampler = ClockSampler(gpu_identifier(torch, local_rank)) if rank == 0 else None

    # ---- device-resident timing ("value") ----------------------------------------------------
    for _ in range(max(args.warmup, 3)):
        flush.zero_()
        step_resident()
    barrier()
    t_load0 = time.time()
    pairs = []
    for _ in range(args.steps):
        flush.zero_()                       # evict the 3.2 MB inputs and the outputs from L2
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        step_resident(mark=True)
        e1.record()
        pairs.append((e0, e1))
    barrier()
    t_load1 = time.time()
    step_ms = [a.elapsed_time(b) for a, b in pairs]
    total_ms = max_over_ranks(sum(step_ms))
    value = world * n * args.steps / (total_ms * 1e-3)

    fwd_ms = statistics.median(a.elapsed_time(m_) for (a, _), m_ in zip(pairs, fwd_marks))
    phases = {"fwd_ms_median": fwd_ms,
              "bwd_ms_median": statistics.median(m_.elapsed_time(b) for (_, b), m_ in zip(pairs, fwd_marks)),
              "fwd_bwd_ms_median": statistics.median(step_ms)}

    # ---- end to end from host buffers ("e2e") --------------------------------------------------
    o_idx = torch.empty((n, K), dtype=torch.int64).pin_memory()
    o_dsq = torch.empty((n, K), dtype=torch.float32).pin_memory()
    o_grad = torch.empty((n, w.coords.shape[1]), dtype=torch.float32).pin_memory()

    copy_stream = torch.cuda.Stream(device=dev)

    def step_e2e():
        # The way a host-side caller would drive it: inputs come from pinned host memory, results
        # go back to pinned host memory, and the copies that nothing waits for run on a second
        # stream (upstream gradient in while the forward runs, indices/distances out while the
        # backward runs).  Everything is inside the timed region.
        main = torch.cuda.current_stream(dev)
        c = h_coords.to(dev, non_blocking=True).requires_grad_(True)
        rs = h_rs.to(dev, non_blocking=True)
        copy_stream.wait_stream(main)
        with torch.cuda.stream(copy_stream):
            g = h_grad.to(dev, non_blocking=True)
            g_ready = torch.cuda.Event()
            g_ready.record(copy_stream)
        idx, dsq = fgc.binned_select_knn(K, c, rs)
        fwd_done = torch.cuda.Event()
        fwd_done.record(main)
        with torch.cuda.stream(copy_stream):
            copy_stream.wait_event(fwd_done)
            o_idx.copy_(idx, non_blocking=True)
            o_dsq.copy_(dsq.detach(), non_blocking=True)
        main.wait_event(g_ready)            # the gradient has to be on the device by now ...
        g.record_stream(main)
        dsq.backward(g)
        o_grad.copy_(c.grad, non_blocking=True)
        idx.record_stream(copy_stream)
        dsq.record_stream(copy_stream)
        main.wait_stream(copy_stream)       # ... and the step ends when every copy has landed

    for _ in range(3):
        step_e2e()
    barrier()
    pairs = []
    for _ in range(args.steps):
        flush.zero_()
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        step_e2e()
        e1.record()
        pairs.append((e0, e1))
    barrier()
    e2e_single_ms = max_over_ranks(sum(a.elapsed_time(b) for a, b in pairs)) / args.steps

    # The same calls as a STREAM of batches, the way a host-side caller with a queue of events
    # drives the library: three sets of pinned result buffers, the result copies of batch i run
    # while batch i+1 is searched, and the host waits for the copies of batch i-3 before it
    # hands that buffer set out again.  Timed from the first input copy to the moment the last
    # result has landed; the L2 flush of every step is inside the timed region.
    h2d_stream = torch.cuda.Stream(device=dev)
    d2h_stream = torch.cuda.Stream(device=dev)
    n_sets = 3
    outs = [(o_idx, o_dsq, o_grad)] + [
        (torch.empty_like(o_idx).pin_memory(), torch.empty_like(o_dsq).pin_memory(),
         torch.empty_like(o_grad).pin_memory()) for _ in range(n_sets - 1)]
    landed = [None] * n_sets

    def submit(i):
        s_ = i % n_sets
        if landed[s_] is not None:
            landed[s_].synchronize()        # buffer set s_ is free again
        b_idx, b_dsq, b_grad = outs[s_]
        main = torch.cuda.current_stream(dev)
        flush.zero_()
        c = h_coords.to(dev, non_blocking=True).requires_grad_(True)
        rs = h_rs.to(dev, non_blocking=True)
        with torch.cuda.stream(h2d_stream):
            g = h_grad.to(dev, non_blocking=True)
            g_ready = torch.cuda.Event()
            g_ready.record(h2d_stream)
        idx, dsq = fgc.binned_select_knn(K, c, rs)
        fwd_done = torch.cuda.Event()
        fwd_done.record(main)
        with torch.cuda.stream(d2h_stream):
            d2h_stream.wait_event(fwd_done)
            b_idx.copy_(idx, non_blocking=True)
            b_dsq.copy_(dsq.detach(), non_blocking=True)
        main.wait_event(g_ready)
        g.record_stream(main)
        dsq.backward(g)
        bwd_done = torch.cuda.Event()
        bwd_done.record(main)
        grad = c.grad
        with torch.cuda.stream(d2h_stream):
            d2h_stream.wait_event(bwd_done)
            b_grad.copy_(grad, non_blocking=True)
            ev = torch.cuda.Event()
            ev.record(d2h_stream)
        for t in (idx, dsq, grad):
            t.record_stream(d2h_stream)
        landed[s_] = ev

    def run_stream(k):
        for j in range(n_sets):
            landed[j] = None
        main = torch.cuda.current_stream(dev)
        e0 = torch.cuda.Event(enable_timing=True)
        e1 = torch.cuda.Event(enable_timing=True)
        e0.record()
        for i in range(k):
            submit(i)
        main.wait_stream(d2h_stream)
        main.wait_stream(h2d_stream)
        e1.record()
        torch.cuda.synchronize(dev)
        return e0.elapsed_time(e1)

    # warm-up long enough for the caching allocator to settle with n_sets batches in flight
    # (a cudaMalloc inside the timed region would stall the pipeline)
    run_stream(max(args.warmup, 3) + 4 * n_sets)
    run_stream(2 * n_sets)
    barrier()
    e2e_ms = max_over_ranks(run_stream(args.steps))
    barrier()
    e2e_value = world * n * args.steps / (e2e_ms * 1e-3)
    h2d = h_coords.numel() * 4 + h_rs.numel() * 8 + h_grad.numel() * 4
    d2h = o_idx.numel() * 8 + o_dsq.numel() * 4 + o_grad.numel() * 4

    clocks = sampler.summary(t_load0, t_load1) if sampler else None
    if sampler:
        sampler.stop()

    # ---- GravNet layer (second half of the headline metric) -------------------------------
    gravnet = None
    if "gravnet" in sections:
        from fastgraphcompute_b200.gnn_ops import GravNetOp
        from fastgraphcompute_b200 import event_sharding as event_sharding_mod
        gw = synthetic.c4_gravnet(seed=rank)
        m = synthetic.init_gravnet_weights(
            GravNetOp(gw.in_channels, gw.out_channels, gw.space_dimensions, gw.propagate_dimensions,
                      gw.k)).to(dev)
        x = gw.x.to(dev).requires_grad_(True)
        rs = gw.row_splits.to(dev)

        def gstep():
            for p in m.parameters():
                p.grad = None
            x.grad = None
            out = m(x, rs)[0]
            (out ** 2).sum().backward()
            if world > 1:
                # data-parallel over the event shards: one all-reduce of the parameter gradients
                event_sharding_mod.allreduce_gradients(m.parameters())

        for _ in range(3):
            gstep()
        barrier()
        gp = []
        for _ in range(5):
            e0 = torch.cuda.Event(enable_timing=True)
            e1 = torch.cuda.Event(enable_timing=True)
            e0.record()
            gstep()
            e1.record()
            gp.append((e0, e1))
        barrier()
        g_ms = max_over_ranks(sum(a.elapsed_time(b) for a, b in gp)) / 5
        gravnet = {"fwd_bwd_ms": g_ms, "n_gpus": world,
                   "config": "c4: GravNetOp(64->64, space 4, propagate 32, k 40), 16 events x 100000 points per GPU, loss sum(out^2)"
                             + ("; parameter gradients summed over the ranks by one all-reduce per step" if world > 1 else ""),
                   "inputs": "x 410 MB per GPU (larger than L2)", "steps": 5, "warmup": 3}
        del x, m

    # The two sections below are additions to the headline numbers: a rank that fails in its local
    # part reports it, all ranks agree (one all-reduce that every rank always reaches) and the
    # section is dropped from the line instead of taking the whole run down.
    def all_ranks_ok(ok):
        if world == 1:
            return bool(ok)
        t = torch.tensor([1 if ok else 0], dtype=torch.int32, device=dev)
        dist.all_reduce(t, op=dist.ReduceOp.MIN)
        return bool(int(t.item()))

    # ---- stacked-GravNet model: the reference's own end-to-end benchmark --------------------
    # (performance/gravnet_perfm.py:100-160: 64 input features, 4 GravNet layers with k = 64,
    # propagate 32, space 4, hidden 128, 10 outputs; one step = forward, sum(output)*0 backward,
    # SGD step, on a fresh randn input of n_nodes points in one event; largest size of its sweep)
    stacked = None
    if "stacked" in sections:
        n_nodes = 200000
        s_local = None
        try:
            from fastgraphcompute_b200.gravnet_model import GravNetModel
            torch.manual_seed(1000 + rank)
            sm = GravNetModel(64, 32, 4, 64, 128, 10).to(dev)
            opt = torch.optim.SGD(sm.parameters(), lr=0.01)
            srs = torch.tensor([0, n_nodes], dtype=torch.int64, device=dev)
            xs = [torch.randn((n_nodes, 64), device=dev) for _ in range(4)]

            def sstep(i):
                opt.zero_grad(set_to_none=True)
                out = sm(xs[i % len(xs)], srs)
                (torch.sum(out) * 0.0).backward()
                opt.step()
                return out

            for i in range(3):
                sstep(i)
            torch.cuda.synchronize(dev)
            sp = []
            for i in range(5):
                flush.zero_()
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record()
                sstep(i)
                e1.record()
                sp.append((e0, e1))
            torch.cuda.synchronize(dev)
            s_local = sum(a.elapsed_time(b) for a, b in sp) / 5
            del sm, opt, xs
        except Exception as exc:          # noqa: BLE001
            print("bench.py: stacked-GravNet section failed on rank %d: %r" % (rank, exc), file=sys.stderr)
        if all_ranks_ok(s_local is not None):
            stacked = {"train_step_ms": max_over_ranks(s_local), "n_gpus": world, "n_nodes_per_gpu": n_nodes,
                       "config": "GravNetModel(in 64, propagate 32, space 4, k 64, hidden 128, out 10, 4 GravNet "
                                 "layers), one event, forward + backward + SGD step as performance/gravnet_perfm.py",
                       "steps": 5, "warmup": 3}

    # ---- event-batched workload C3 sharded by event over the ranks (strong scaling) ----------
    # Every rank holds the batch and searches the events the partition table gives it.  Three
    # ways to end: rows stay on the rank that computed them (no collective), rows of all ranks on
    # every rank, rows of all ranks on rank 0.  The exchange is per-event point-to-point blocks
    # straight into the final tensors, ids as int32 on the wire, events searched in three groups
    # so that finished rows travel while the next group is searched.  With more than one rank
    # the gathered result is compared with a single-GPU search of the whole batch on every rank.
    def same_neighbour_rows(idx_a, dsq_a, idx_b, dsq_b):
        """Two searches of the same points on different grids: the sorted squared distances of
        every row must be bit-identical; the neighbour ids too, except that a row may hold a
        different one of several candidates that tie exactly at its largest distance."""
        if not torch.equal(torch.sort(dsq_a, 1).values, torch.sort(dsq_b, 1).values):
            return False
        differ = (torch.sort(idx_a, 1).values != torch.sort(idx_b, 1).values).any(1).nonzero().flatten()
        if differ.numel() > max(1000, idx_a.shape[0] // 1000):
            return False
        for r in differ.tolist():
            ia, ib = idx_a[r].tolist(), idx_b[r].tolist()
            da, db = dsq_a[r].tolist(), dsq_b[r].tolist()
            kth = max(da)
            only_a = [d for i, d in zip(ia, da) if i not in set(ib)]
            only_b = [d for i, d in zip(ib, db) if i not in set(ia)]
            if len(only_a) != len(only_b) or any(d != kth for d in only_a + only_b):
                return False
        return True

    c3 = None
    if "c3" in sections:
        c3_local = None
        c3_reps = 3
        try:
            from fastgraphcompute_b200 import event_sharding
            w3 = synthetic.c3_event_batch(seed=0)
            part = event_sharding.partition_events(w3.row_splits, world)
            c3_coords = w3.coords.to(dev)
            c3_rs = w3.row_splits.to(dev)

            def c3_run(mode, chunks, exchange="auto"):
                if world == 1 or mode == "none":
                    return event_sharding.local_binned_select_knn(w3.K, c3_coords, w3.row_splits, part.events[rank])
                return event_sharding.sharded_binned_select_knn(w3.K, c3_coords, w3.row_splits, gather=mode,
                                                                n_chunks=chunks, check=False, exchange=exchange)

            def c3_time(mode, chunks, exchange="auto"):
                for _ in range(3):        # (the first collective of a kind and size sets up its connections)
                    res = c3_run(mode, chunks, exchange)
                del res
                barrier()
                e0 = torch.cuda.Event(enable_timing=True)
                e1 = torch.cuda.Event(enable_timing=True)
                e0.record()
                for _ in range(c3_reps):
                    res = c3_run(mode, chunks, exchange)
                e1.record()
                torch.cuda.synchronize(dev)
                del res
                return e0.elapsed_time(e1) / c3_reps

            c3_local = {"none": c3_time("none", 1)}
            if world > 1:
                c3_local["all"] = c3_time("all", 3)
                c3_local["all_one_group"] = c3_time("all", 1)
                c3_local["all_p2p"] = c3_time("all", 3, "p2p")
                c3_local["root"] = c3_time("root", 3)
                # correctness of the exchange, on every rank: same distances bit for bit and same
                # neighbour sets as one GPU searching the whole batch
                g_idx, g_dsq = c3_run("all", 3)
                r_idx, r_dsq = fgc.binned_select_knn(w3.K, c3_coords, c3_rs)
                c3_local["equal"] = same_neighbour_rows(g_idx, g_dsq, r_idx, r_dsq)
                del g_idx, g_dsq, r_idx, r_dsq
        except Exception as exc:          # noqa: BLE001
            c3_local = None
            print("bench.py: C3 section failed on rank %d: %r" % (rank, exc), file=sys.stderr)
        if all_ranks_ok(c3_local is not None):
            c3_ms = max_over_ranks(c3_local["none"])
            c3 = {"config": "c3: 64 events of 50000..150000 uniform points, D=3, K=64, forward, sharded by event "
                            "(greedy longest-processing-time on point counts)",
                  "n_points": w3.n_points, "n_gpus": world, "search_ms": c3_ms,
                  "points_per_s": w3.n_points / (c3_ms * 1e-3), "scaling": "strong",
                  "largest_shard_points": max(part.points),
                  "note": "search_ms: local search + local->global ids, rows stay sharded, max over ranks"}
            if world > 1:
                c3["search_and_gather_all_ms"] = max_over_ranks(c3_local["all"])
                c3["search_and_gather_all_one_group_ms"] = max_over_ranks(c3_local["all_one_group"])
                c3["search_and_gather_all_point_to_point_ms"] = max_over_ranks(c3_local["all_p2p"])
                c3["search_and_gather_root_ms"] = max_over_ranks(c3_local["root"])
                c3["gathered_equals_single_gpu"] = all_ranks_ok(c3_local["equal"])
                c3["gather_note"] = ("search + exchange of idx (int32 on the wire, widened to int64 on receipt) and "
                                     "distsq; 'all': every rank ends with all rows -- one NCCL all-gather per group "
                                     "of events into a staging buffer, then a placing pass, three groups per rank so "
                                     "that transfers overlap the search ('point_to_point': per-event blocks sent "
                                     "straight into the final tensors instead); 'root': rank 0 only, point-to-point")
        c3_coords = None

    # ---- object-condensation index matrices (the loss-side consumer of the same row splits) --
    oc = None
    if "oc" in sections:
        oc_local = None
        try:
            import ctypes
            g_oc = torch.Generator().manual_seed(3 + rank)
            n_sp, per_sp = 16, 100000
            asso = torch.randint(-20, 200, (n_sp * per_sp,), generator=g_oc).to(dev)
            rs_oc = torch.arange(0, n_sp * per_sp + 1, per_sp, dtype=torch.int64).to(dev)
            n_oc = asso.shape[0]
            nb = _cabi.lib.fgc_oc_workspace_bytes(n_oc)
            ws_oc = torch.empty(nb, dtype=torch.uint8, device=dev)
            per_oc = torch.empty(n_sp, dtype=torch.int64, device=dev)
            st_oc = ctypes.c_int32(0)
            sz_oc = (ctypes.c_int64 * 3)()
            stream = _cabi.current_stream(dev)

            def oc_prepare():
                _cabi.check(_cabi.lib.fgc_oc_prepare(_cabi.ptr(asso), n_oc, _cabi.ptr(rs_oc), n_sp + 1, _cabi.ptr(ws_oc),
                                                     nb, _cabi.ptr(per_oc), stream), "fgc_oc_prepare")

            oc_prepare()
            _cabi.check(_cabi.lib.fgc_oc_read_sizes(_cabi.ptr(ws_oc), ctypes.byref(st_oc), sz_oc, stream), "sizes")
            nu, nq, nr = int(sz_oc[0]), int(sz_oc[1]), int(sz_oc[2])
            M_oc = torch.empty((nu, nq), dtype=torch.int64, device=dev)
            Mn_oc = torch.empty((nu, nr), dtype=torch.int64, device=dev)

            def oc_fill():
                _cabi.check(_cabi.lib.fgc_oc_fill(_cabi.ptr(ws_oc), nb, n_oc, _cabi.ptr(rs_oc), nu, nq, nr,
                                                  _cabi.ptr(M_oc), _cabi.ptr(Mn_oc), stream), "fgc_oc_fill")

            for _ in range(2):
                oc_prepare()
                oc_fill()
            torch.cuda.synchronize(dev)
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(3)]
            reps = 5
            t_prep = t_fill = 0.0
            for _ in range(reps):
                flush.zero_()
                ev[0].record()
                oc_prepare()
                ev[1].record()
                oc_fill()
                ev[2].record()
                torch.cuda.synchronize(dev)
                t_prep += ev[0].elapsed_time(ev[1])
                t_fill += ev[1].elapsed_time(ev[2])
            fill_bytes = 8 * nu * (nq + nr)
            oc_local = (t_prep / reps, t_fill / reps, fill_bytes, nu, nq, nr)
            del M_oc, Mn_oc, ws_oc
        except Exception as exc:          # noqa: BLE001
            print("bench.py: oc_helper section failed on rank %d: %r" % (rank, exc), file=sys.stderr)
        if all_ranks_ok(oc_local is not None):
            peak_oc, peak_oc_kind = measured_peaks()
            fill_ms = max_over_ranks(oc_local[1])
            oc = {"config": "oc_helper_matrices: 16 row splits x 100000 points, truth index uniform in [-20, 200) "
                            "(200 objects per row split + noise)",
                  "n_gpus": world, "prepare_ms": max_over_ranks(oc_local[0]), "fill_ms": fill_ms,
                  "shape": {"n_objects": oc_local[3], "n_max_points_per_object": oc_local[4],
                            "n_max_points_per_row_split": oc_local[5]},
                  "roofline": {"bound": "hbm", "kernel": "k_oc_fill_m + k_oc_fill_m_not",
                               "algorithmic_bytes": oc_local[2],
                               "achieved": oc_local[2] / (fill_ms * 1e-3) / 1e9, "peak": peak_oc, "unit": "GB/s",
                               "frac": oc_local[2] / (fill_ms * 1e-3) / 1e9 / peak_oc,
                               "peak_source": "of " + peak_oc_kind}}

    # ---- the reference's own published kNN timings, same configurations ------------------------
    # (forward only, one event, timer around the public call plus a device
    # synchronise as in performance/generate_faiss_performance.py:68-92; the published figures
    # come from an unspecified GPU and are quoted for orientation, not as a like-for-like ratio)
    published = None
    if "published" in sections and rank == 0:
        try:
            rows = []
            for tag, n_p, d_p, k_p, ref_ms, src in (
                    ("K=40 D=5 N=100000 randn", 100000, 5, 40, 72.3, "performance/faiss_data_sizes.csv:20"),
                    ("K=40 D=5 N=1000000 randn", 1000000, 5, 40, 2035.0, "performance/faiss_data_sizes.csv:33"),
                    ("K=40 D=5 N=3000000 randn", 3000000, 5, 40, 13288.0, "performance/faiss_data_sizes.csv:43"),
                    ("K=40 D=4 N=1000000 randn", 1000000, 4, 40, 993.6, "graphing/master_data.csv:668"),
                    ("K=40 D=4 N=5000000 randn", 5000000, 4, 40, 10232.0, "graphing/master_data.csv:1477"),
                    ("K=40 D=3 N=700000 randn", 700000, 3, 40, 148.5, "graphing/master_data.csv:566")):
                gp = torch.Generator().manual_seed(42)
                cp = torch.randn((n_p, d_p), generator=gp).to(dev)
                rp = torch.tensor([0, n_p], dtype=torch.int64, device=dev)
                for _ in range(2):
                    fgc.binned_select_knn(k_p, cp, rp)
                torch.cuda.synchronize(dev)
                ts = []
                for _ in range(3):
                    t0 = time.perf_counter()
                    out_p = fgc.binned_select_knn(k_p, cp, rp)
                    torch.cuda.synchronize(dev)
                    ts.append(1e3 * (time.perf_counter() - t0))
                    del out_p
                rows.append({"config": tag, "forward_ms": statistics.median(ts), "reference_published_ms": ref_ms,
                             "reference_source": src})
                del cp
            published = {"method": "wall clock around binned_select_knn + synchronize, median of 3 after 2 warm-ups, "
                                   "standard-normal coordinates, one row split",
                         "note": "published figures: the reference's CUDA path on an unspecified GPU",
                         "rows": rows}
        except Exception as exc:          # noqa: BLE001
            print("bench.py: published-config section failed: %r" % (exc,), file=sys.stderr)

    # ---- CPU baseline beside it (rank 0, single-GPU runs only) -----------------------------
    cpu_baseline = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        wb = synthetic.c2_gaussian_mixture(seed=0)
        t, kind = cpu_reference_fwd_bwd(wb, torch)
        cpu_baseline = {"value": wb.n_points / t, "unit": UNIT, "cores": 1, "kind": kind,
                        "sample": "the full workload once (200000 points, fwd+bwd, %.1f s)" % t,
                        "aten_threads": torch.get_num_threads(),
                        "note": "the reference's kNN, binning and gradient loops are single-threaded"}
        # distance evaluations of the reference's own shell walk at its default binning, counted
        # by the instrumented C restatement on the same workload
        try:
            from oracle import oracle as _oracle
            t0 = time.time()
            _, _, c_ref = _oracle.binned_select_knn(wb.K, wb.coords.numpy(), wb.row_splits.numpy(), return_evals=True)
            cpu_baseline["reference_binning_evals_per_query"] = c_ref / wb.n_points
            cpu_baseline["reference_binning_evals_note"] = (
                "C restatement of the reference forward with its default n_bins, %.1f s" % (time.time() - t0))
        except Exception as exc:      # noqa: BLE001
            cpu_baseline["reference_binning_evals_per_query"] = None
            cpu_baseline["reference_binning_evals_note"] = "not counted: %r" % (exc,)

    if rank == 0:
        peak, peak_kind = measured_peaks()
        d = w.coords.shape[1]
        alg_bytes = n * (4 * d + 8 * K + 4 * K)          # coords read + int64 idx + fp32 distsq written
        achieved = alg_bytes / (fwd_ms * 1e-3) / 1e9
        launches_per_step = _cabi.KERNELS_TREE_FORWARD + _cabi.KERNELS_TREE_SECOND_LOOK + _cabi.KERNELS_KNN_BWD
        line = {
            "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
            "warmup": max(args.warmup, 3), "ms_per_step": total_ms / args.steps,
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f32",
            "data": "synthetic",
            "config": {"workload": WORKLOAD, "points_per_gpu": n, "sharding": "one event per GPU, no data-path collective",
                       "l2": "flushed between steps by a 256 MiB write outside the timed events (inputs are 3.2 MB)",
                       "timing": "CUDA events per step on the launching stream, summed; max over ranks"},
            "e2e": {"value": e2e_value, "unit": UNIT, "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h,
                    "ms_per_step": e2e_ms / args.steps,
                    "mode": "a stream of batches from pinned host buffers, three sets of pinned result buffers: "
                            "the result copies of batch i overlap the search of batch i+1; timed from the "
                            "first input copy until the last result has landed, L2 flush of every step included",
                    "single_batch_ms": e2e_single_ms},
            "gpu_launches": launches_per_step * args.steps,
            "roofline": {"bound": "hbm", "kernel": "binned_select_knn forward: search by groups, 33 launches", "achieved": achieved,
                         "peak": peak, "unit": "GB/s", "frac": achieved / peak,
                         "peak_source": "of " + peak_kind, "traffic": FORWARD_DRAM_TRAFFIC_BYTES,
                         "algorithmic_bytes_per_launch": alg_bytes, "kernel_ms": fwd_ms,
                         "note": "not HBM-bound: k_tree_rows, its longest kernel, keeps 86 % of the issue slots busy "
                                 "(profiles/knn_c2_step_launch_list.md); tree and second look are chains of short launches"},
            "clocks": clocks,
        }
        line["phases"] = phases
        if cpu_baseline:
            line["cpu_baseline"] = cpu_baseline
        if c3:
            line["c3_event_sharded"] = c3
        if gravnet:
            line["gravnet"] = gravnet
        if stacked:
            line["stacked_gravnet"] = stacked
        if oc:
            line["oc_helper_matrices"] = oc
        if published:
            line["published_configs"] = published      # the long table last
        print(json.dumps(line), flush=True)
    if world > 1:
        dist.destroy_process_group()


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=50)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="b200", choices=["b200", "reference"])
    ap.add_argument("--no-gravnet", action="store_true", help="headline workload only (same as --sections none)")
    ap.add_argument("--sections", default="gravnet,stacked,c3,oc,published",
                    help="additional workloads to time after the headline one: any of gravnet, stacked, c3, oc, published")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
    else:
        run_b200(args)


if __name__ == "__main__":
    main()
