"""Benchmark: 3D layered shell time steps per second on GB300.

Workload (default): the 3D layered spherical shell -- icosphere level 5
(10242 surface vertices) x 9 node layers (8 prism layers, 3 tets each) =
92178 nodes, 491520 P1 tets, 3 material layers, Fisher-KPP + isotropic
elasticity, block-Jacobi PCG tolerance 1e-8, dt 0.01, plain FP64.  A "step" is
one time step of the forward model (velocity solve, node update,
reaction-diffusion solve).  Inputs are synthetic (seeded mesh + bump), the
per-step working set (operator blocks, geometry, CG vectors, ~0.3 GB) is
larger than the 129 MB L2.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--precision fp64|mixed]
  python bench.py --impl reference ...   # CPU restatement on the host cores

With N > 1 (torchrun) every rank runs its own replica of the workload (the
model does not shard: independent solves only), value = sum over ranks of
steps / max-over-ranks time.
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

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "3D shell steps/s"
WORKLOAD = ("3D layered spherical shell: icosphere level 5 x 8 prism layers, 92178 nodes, 491520 P1 tets, "
            "3 material layers, Fisher-KPP + layered isotropic elasticity, block-Jacobi PCG 1e-8, dt 0.01")


def dist_init():
    ws = int(os.environ.get("WORLD_SIZE", "1"))
    if ws <= 1:
        return 0, 0, 1, None
    import torch
    import torch.distributed as dist
    rank, local = int(os.environ["RANK"]), int(os.environ.get("LOCAL_RANK", "0"))
    backend = "nccl" if torch.cuda.is_available() else "gloo"
    if backend == "nccl":
        torch.cuda.set_device(local)
    dist.init_process_group(backend)
    return rank, local, ws, dist


def reduce_max(x: float, dist, local: int) -> float:
    if dist is None:
        return x
    import torch
    dev = f"cuda:{local}" if dist.get_backend() == "nccl" else "cpu"
    t = torch.tensor([x], dtype=torch.float64, device=dev)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def barrier(dist):
    if dist is not None:
        dist.barrier()


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        with open(p) as f:
            d = json.load(f)
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


class ClockSampler:
    """nvidia-smi sampling of SM clocks and throttle reasons during the timed region (every 50 ms: the default
    timed region of 20 steps lasts about a third of a second)."""

    Q = ("clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu: int):
        self.gpu, self.proc, self.path = gpu, None, None

    def start(self):
        try:
            fd, self.path = tempfile.mkstemp(suffix=".csv")
            os.close(fd)
            self.fh = open(self.path, "w")
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                          "-lms", "50", "-i", str(self.gpu)], stdout=self.fh,
                                         stderr=subprocess.DEVNULL)
        except (OSError, FileNotFoundError):
            self.proc = None

    def stop(self):
        if self.proc is None:
            return None
        self.proc.terminate()
        try:
            self.proc.wait(timeout=5)
        except subprocess.TimeoutExpired:
            self.proc.kill()
        self.fh.close()
        sm, mx, reasons = [], 0.0, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for line in open(self.path):
            f = [x.strip() for x in line.split(",")]
            if len(f) < 7:
                continue
            try:
                sm.append(float(f[0]))
                mx = max(mx, float(f[1]))
            except ValueError:
                continue
            for n, v in zip(names, f[3:7]):
                if v.lower() == "active":
                    reasons.add(n)
        os.unlink(self.path)
        if not sm:
            return None
        return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm)}


# element-object arrays the layered forward call reads (the frame model's tan/nml and tsv arrays and the
# boundary-segment arrays are not uploaded for it)
LAYERED_OBJ_KEYS = ("elmVtxMat", "vtxElmMat", "btmVtxMat", "vtxBtmMat", "femVtxMat", "femIfoMat", "vfdVtxMat",
                    "elmLyrVec")


def pinned_inputs(spec):
    """The spec with every array the call uploads copied into page-locked host memory (the inputs of the
    end-to-end leg), and the bytes the call copies to the device."""
    import torch

    def pin(a, dtype):
        return torch.from_numpy(np.ascontiguousarray(np.asarray(a, dtype=dtype))).pin_memory().numpy()

    s = dict(spec)
    obj = dict(spec["elmObj"])
    for k in LAYERED_OBJ_KEYS:
        if k in obj:
            obj[k] = pin(obj[k], np.int32)
    s["elmObj"] = obj
    if "elmLyrVec" in spec:
        s["elmLyrVec"] = pin(spec["elmLyrVec"], np.int32)
    s["lmkIniMat"] = pin(spec["lmkIniMat"], np.float64)
    s["tgt"] = tuple(pin(a, np.float64) for a in spec["tgt"])
    s["tauVarVec"] = pin(spec["tauVarVec"], np.float64)
    h2d = s["lmkIniMat"].nbytes + sum(obj[k].nbytes for k in LAYERED_OBJ_KEYS if k in obj) + \
        sum(a.nbytes for a in s["tgt"]) + s["tauVarVec"].nbytes
    return s, h2d


def spec_for(args, steps: int):
    from shape_atrophy_gb300 import problems
    if args.workload == "annulus":
        spec = problems.annulus_layered(steps=steps)
    else:
        spec = problems.shell_layered(steps=steps)
    spec["cgKernel"] = getattr(args, "cg_kernel", "auto")
    return spec


def cpu_sample(spec_full, steps: int = 8, warm: int = 3):
    """Time the CPU oracle (its -O3 -march=native -fopenmp timing build, all host cores) on time steps
    warm+1 .. warm+steps of the same workload, as the GPU steps are timed after warm-up steps: one run of
    warm + steps time steps, each step timed inside the oracle.  Returns (steps/s, cores, sample label)."""
    from oracle import build_oracle
    from oracle.oracle import Problem
    spec = dict(spec_full)
    spec["timeNum"] = warm + steps + 1
    P = Problem(spec, fast=True)
    t0 = time.perf_counter()
    r = P.forward(spec["tauVarVec"], with_obj=False)
    wall = time.perf_counter() - t0
    if r["status"] != 0:
        raise RuntimeError("oracle solve failed")
    dt = float(np.sum(r["stepSec"][warm:warm + steps]))
    cores = int(os.environ.get("OMP_NUM_THREADS", os.cpu_count() or 1))
    flags = " ".join(build_oracle.fast_flags())
    return steps / dt, cores, (f"time steps {warm + 1}-{warm + steps} of the same workload after {warm} warm-up "
                               f"steps (as the GPU steps), {dt:.1f} s timed, {wall:.1f} s run; oracle built "
                               f"gcc {flags}, {cores} OpenMP threads")


SERVED = ("Poisson stream of forward solves: 3D layered shells, icosphere level 3-5 x 4/8/12 prism layers "
          "(3210-133146 nodes), 20-60 steps each, random bump centre, Lame (lambda, mu=lambda/2) log-uniform in "
          "[0.5, 10] and diffusivity log-uniform in [0.005, 0.1] per material layer, Matern-3/2 varifold objective; "
          "the same stream served in FP64 and in mixed precision")


SERVED_FULL = ("Poisson stream of forward solves over the whole served range: 3D layered shells, icosphere "
               "level 3-6 x 4-12 prism layers (up to 532k nodes, 2.95M tets), 20-100 steps each, random bump, "
               "Lame and diffusivity per layer; served in FP64 and in mixed precision")


def served_requests(n: int, seed: int = 7, mean_gap_s: float = 0.04, full: bool = False):
    """Seeded request stream (specs + Poisson inter-arrival gaps); meshes are shared between requests.
    full=True draws from the whole served range (icosphere 3-6, 4-12 layers, 20-100 steps)."""
    import numpy as np
    from shape_atrophy_gb300 import problems
    rng = np.random.default_rng(seed)
    cache, out = {}, []
    for _ in range(n):
        if full:
            level = int(rng.choice([3, 4, 5, 6], p=[0.3, 0.3, 0.25, 0.15]))
            layers = int(rng.integers(4, 13))
            steps = int(rng.integers(20, 101))
        else:
            level = int(rng.choice([3, 4, 5], p=[0.4, 0.4, 0.2]))
            layers = int(rng.choice([4, 8, 12]))
            steps = int(rng.integers(20, 61))
        key = (level, layers)
        if key not in cache:
            cache[key] = problems.shell_layered(level=level, lyrCntNum=layers + 1, steps=steps, native=True)
        sp = dict(cache[key])
        sp["timeNum"] = steps + 1
        lam = 10.0 ** rng.uniform(np.log10(0.5), 1.0, 3)
        sp["modVec"] = np.column_stack([lam, lam / 2]).reshape(-1)
        sp["spdLyrVec"] = 10.0 ** rng.uniform(np.log10(0.005), np.log10(0.1), 3)
        c = rng.normal(size=3)
        c /= np.linalg.norm(c)
        sp["tauVarVec"] = np.array([c[0], c[1], c[2], 1.0, 0.15])
        out.append((sp, float(rng.exponential(mean_gap_s))))
    return out


def served_leg(device: int, n: int = 32, full: bool = False):
    """The same Poisson stream through the continuous-batching server in FP64 and in mixed precision."""
    import numpy as np
    from shape_atrophy_gb300 import api
    reqs = served_requests(n, full=full)
    runs = {}
    for prec in ("fp64", "mixed"):
        sv = api.Server(hbm_budget=200e9, max_instances=64, device=device)
        t0 = time.perf_counter()
        t_next, ids = t0, []
        for sp, gap in reqs:
            t_next += gap
            now = time.perf_counter()
            if t_next > now:
                time.sleep(t_next - now)
            ids.append(sv.submit(sp, precision=prec))
        res = [sv.result(i) for i in ids]
        wall = time.perf_counter() - t0
        st = sv.stats()
        sv.close()
        lat = np.array([r["latency_ms"] for r in res])
        runs[prec] = dict(res=res, line={
            "solves_per_s": len(res) / wall, "p50_ms": float(np.percentile(lat, 50)),
            "p99_ms": float(np.percentile(lat, 99)), "wall_s": wall,
            "steps_per_s": sum(sp["timeNum"] - 1 for sp, _ in reqs) / wall,
            "ok": int(sum(r["info"]["status"] == 0 for r in res)), "peak_device_gb": st["peakBytes"] / 1e9,
            "ticks": st["ticks"]})
    ep = eo = 0.0
    for a, b in zip(runs["mixed"]["res"], runs["fp64"]["res"]):
        ep = max(ep, float(np.abs(a["lmk"] - b["lmk"]).max() / np.abs(b["lmk"]).max()))
        eo = max(eo, abs(a["obj"] - b["obj"]) / abs(b["obj"]))
    return {"workload": SERVED_FULL if full else SERVED, "requests": n, "mean_gap_ms": 40.0,
            "fp64": runs["fp64"]["line"],
            "mixed": runs["mixed"]["line"],
            "mixed_over_fp64_solves": runs["mixed"]["line"]["solves_per_s"] / runs["fp64"]["line"]["solves_per_s"],
            "mixed_vs_fp64_max_rel_err": {"positions": ep, "objective": eo}}


BATCHED = ("Batched solves: 256 seeded instances submitted at once to the continuous-batching server (batched "
           "persistent CG launches per tick); half 2D layered annuli (node counts log-uniform in 2k-40k, radial:angular "
           "nodes 1:16, 2-6 material layers), half 3D layered shells (icosphere level 3-4 x 4-8 prism layers, 3 "
           "material layers); Lame (lambda, mu = lambda/2) log-uniform in [0.5, 10] and diffusivity in [0.005, 0.1] "
           "per material layer, random bump on the outer boundary, 50 steps each, varifold objective; the same batch "
           "in FP64 and in mixed precision")


def batched_requests(n: int = 256, seed: int = 13, steps: int = 50):
    """Seeded batch of 2D annuli and 3D shells (meshes shared between requests of the same size)."""
    import numpy as np
    from shape_atrophy_gb300 import problems
    rng = np.random.default_rng(seed)
    cache, out = {}, []
    for _ in range(n):
        if rng.random() < 0.5:
            nodes = 10.0 ** rng.uniform(np.log10(2000.0), np.log10(40000.0))
            L = int(rng.integers(2, 7))
            rad = max(L + 1, int(round(np.sqrt(nodes / 16.0))))
            ang = max(16, int(round(nodes / rad / 16.0)) * 16)
            key = ("a", ang, rad, L)
            if key not in cache:
                cache[key] = problems.annulus_layered(angNum=ang, radNum=rad, steps=steps, layers=L, native=True)
            sp = dict(cache[key])
            th = rng.uniform(0.0, 2.0 * np.pi)
            sp["tauVarVec"] = np.array([np.cos(th), np.sin(th), 1.0, 0.1])
        else:
            level, layers, L = int(rng.integers(3, 5)), int(rng.integers(4, 9)), 3
            key = ("s", level, layers)
            if key not in cache:
                cache[key] = problems.shell_layered(level=level, lyrCntNum=layers + 1, steps=steps, native=True)
            sp = dict(cache[key])
            c = rng.normal(size=3)
            c /= np.linalg.norm(c)
            sp["tauVarVec"] = np.array([c[0], c[1], c[2], 1.0, 0.15])
        lam = 10.0 ** rng.uniform(np.log10(0.5), 1.0, L)
        sp["modVec"] = np.column_stack([lam, lam / 2]).reshape(-1)
        sp["spdLyrVec"] = 10.0 ** rng.uniform(np.log10(0.005), np.log10(0.1), L)
        out.append(sp)
    return out


def batched_leg(device: int, n: int = 256):
    """The batch through the server in FP64 and in mixed precision: solves/s, latency, error of mixed vs FP64."""
    import numpy as np
    from shape_atrophy_gb300 import api
    reqs = batched_requests(n)
    runs = {}
    for prec in ("fp64", "mixed"):
        sv = api.Server(hbm_budget=200e9, max_instances=n, device=device)
        t0 = time.perf_counter()
        ids = [sv.submit(sp, precision=prec) for sp in reqs]
        res = [sv.result(i) for i in ids]
        wall = time.perf_counter() - t0
        st = sv.stats()
        sv.close()
        lat = np.array([r["latency_ms"] for r in res])
        runs[prec] = dict(res=res, line={
            "solves_per_s": len(res) / wall, "p50_ms": float(np.percentile(lat, 50)),
            "p99_ms": float(np.percentile(lat, 99)), "wall_s": wall,
            "steps_per_s": sum(sp["timeNum"] - 1 for sp in reqs) / wall,
            "ok": int(sum(r["info"]["status"] == 0 for r in res)), "peak_device_gb": st["peakBytes"] / 1e9,
            "ticks": st["ticks"]})
    ep = eo = 0.0
    for a, b in zip(runs["mixed"]["res"], runs["fp64"]["res"]):
        ep = max(ep, float(np.abs(a["lmk"] - b["lmk"]).max() / np.abs(b["lmk"]).max()))
        eo = max(eo, abs(a["obj"] - b["obj"]) / abs(b["obj"]))
    return {"workload": BATCHED, "requests": n, "fp64": runs["fp64"]["line"], "mixed": runs["mixed"]["line"],
            "mixed_over_fp64_solves": runs["mixed"]["line"]["solves_per_s"] / runs["fp64"]["line"]["solves_per_s"],
            "mixed_vs_fp64_max_rel_err": {"positions": ep, "objective": eo}}


def oracle_run(args, steps: int = 20):
    """One run of the CPU oracle (timing build, all host cores) over the first `steps` steps of the workload:
    its trajectory is the FP64 reference of the mixed-error leg, its per-step times the CPU baseline."""
    from oracle.oracle import Problem
    spec = spec_for(args, steps)
    P = Problem(spec, fast=True)
    t0 = time.perf_counter()
    r = P.forward(spec["tauVarVec"], with_obj=False)
    r["wall"] = time.perf_counter() - t0
    if r["status"] != 0:
        raise RuntimeError("oracle solve failed")
    r["problem"] = P
    return r


def cpu_from_run(r, warm: int = 3):
    """CPU baseline from an oracle run: steps after `warm` warm-up steps, each timed inside the oracle."""
    from oracle import build_oracle
    sec = r["stepSec"][warm:]
    dt = float(np.sum(sec))
    cores = int(os.environ.get("OMP_NUM_THREADS", os.cpu_count() or 1))
    flags = " ".join(build_oracle.fast_flags())
    return {"value": sec.size / dt, "unit": "steps/s", "cores": cores, "kind": "port",
            "sample": f"time steps {warm + 1}-{warm + sec.size} of the same workload after {warm} warm-up steps "
                      f"(as the GPU steps), {dt:.1f} s timed, {r['wall']:.1f} s run; oracle built gcc {flags}, "
                      f"{cores} OpenMP threads"}


def mixed_error_leg(args, device: int, ref, every: int = 10):
    """Mixed precision and FP64 on the GPU against the FP64 CPU oracle (`ref` = oracle_run) at every 10th step
    of the shell: node positions, concentration and objective (the oracle's varifold of its own shape)."""
    from shape_atrophy_gb300 import api
    T = ref["lmkStk"].shape[0] - 1
    spec = spec_for(args, T)
    P = ref["problem"]
    sess = {p: api.Session(spec, precision=p, objective=True, device=device) for p in ("fp64", "mixed")}
    rows = []
    for t in range(every, T + 1, every):
        x_o, u_o = ref["lmkStk"][t], ref["tauMat"][t]
        o_o = P.varifold(x_o)
        row = {"step": t}
        for p, sv in sess.items():
            sv.step(every)
            x, u, _ = sv.state()
            o = sv.objective()
            row[p] = {"positions": float(np.abs(x - x_o).max() / np.abs(x_o).max()),
                      "concentration": float(np.abs(u - u_o).max() / max(np.abs(u_o).max(), 1e-300)),
                      "objective": abs(o - o_o) / abs(o_o)}
        rows.append(row)
    for sv in sess.values():
        sv.close()
    worst = {p: {k: max(r[p][k] for r in rows) for k in ("positions", "concentration", "objective")}
             for p in ("fp64", "mixed")}
    return {"steps": T, "every": every, "reference": "FP64 CPU oracle, same workload and steps",
            "max_rel_err": worst["mixed"], "fp64_max_rel_err": worst["fp64"], "tolerance": 1e-6,
            "within": all(v <= 1e-6 for v in worst["mixed"].values()), "per_step": rows}


def mixed_drift_leg(args, device: int, steps: int = 100, every: int = 10):
    """Mixed precision against FP64, both on the GPU, over the workload's 100 steps (beyond what the oracle
    runs in the bench's time)."""
    from shape_atrophy_gb300 import api
    spec = spec_for(args, steps)
    s64 = api.Session(spec, precision="fp64", objective=True, device=device)
    s32 = api.Session(spec, precision="mixed", objective=True, device=device)
    worst = {"positions": 0.0, "concentration": 0.0, "objective": 0.0}
    for t in range(every, steps + 1, every):
        s64.step(every)
        s32.step(every)
        x64, u64, _ = s64.state()
        x32, u32, _ = s32.state()
        o64, o32 = s64.objective(), s32.objective()
        worst["positions"] = max(worst["positions"], float(np.abs(x32 - x64).max() / np.abs(x64).max()))
        worst["concentration"] = max(worst["concentration"],
                                     float(np.abs(u32 - u64).max() / max(np.abs(u64).max(), 1e-300)))
        worst["objective"] = max(worst["objective"], abs(o32 - o64) / abs(o64))
    s64.close()
    s32.close()
    return {"steps": steps, "every": every, "reference": "FP64 GPU path", "max_rel_err": worst}


def algorithmic_bytes(N: int, E: int, D: int, elt: int = 8) -> dict:
    """Compulsory HBM bytes of the operators, matrix-free recompute formulation: per application x read, y
    written and the coordinates read once (elt bytes per value), connectivity (4 B x E x V) and the element's
    layer id (4 B) read once; per CG iteration five N-vectors beside it.  Per step the geometry/right-hand-side
    passes read the coordinates twice, the connectivity once and write the element loads."""
    V = D + 1
    matvec = 3 * elt * N * D + 4 * E * V + 4 * E
    rd_matvec = 2 * elt * N + 4 * E * V + elt * N * D + 4 * E
    return {"elt": elt, "matvec": matvec, "iteration": matvec + 5 * elt * N * D,
            "rd_iteration": rd_matvec + 5 * elt * N, "per_step": 2 * 8 * N * D + 4 * E * V + 8 * E * V * D}


def run_reference(args, rank, ws, dist):
    """The model on the host cores: the CPU oracle, a restatement of the reference's element-loop operators
    (the reference is MATLAB MEX code with no CPU path of its own and an empty layered branch), timed on
    exactly --steps time steps after --warmup warm-up steps of the same workload."""
    if rank != 0:
        return
    K, W = args.steps, max(3, args.warmup)
    value, cores, sample = cpu_sample(spec_for(args, W + K), steps=K, warm=W)
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "steps/s", "n_gpus": args.gpus,
            "steps": K, "warmup": W, "ms_per_step": 1000.0 / value, "higher_is_better": True,
            "scaling": "weak", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": WORKLOAD, "precision": "fp64"},
            "cpu_baseline": {"value": value, "unit": "steps/s", "cores": cores, "kind": "port", "sample": sample},
            "e2e": {"value": value, "unit": "steps/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--precision", default="fp64", choices=["fp64", "mixed"])
    ap.add_argument("--workload", default="shell", choices=["shell", "annulus"])
    ap.add_argument("--cg-kernel", default="auto", choices=["auto", "persistent", "two-kernel", "persistent-global"])
    ap.add_argument("--no-cpu", action="store_true", help="skip the CPU baseline leg")
    ap.add_argument("--no-e2e", action="store_true", help="skip the end-to-end leg")
    ap.add_argument("--no-served", action="store_true", help="skip the served-stream leg")
    ap.add_argument("--no-batched", action="store_true", help="skip the batched-instances leg")
    ap.add_argument("--batched-requests", type=int, default=256)
    ap.add_argument("--no-mixed-error", action="store_true", help="skip the mixed-vs-FP64 error leg")
    ap.add_argument("--no-gradient", action="store_true", help="skip the objective-gradient leg")
    ap.add_argument("--oracle-steps", type=int, default=20,
                    help="steps of the CPU oracle run (mixed-error reference and CPU baseline)")
    ap.add_argument("--served-requests", type=int, default=None,
                    help="length of the served stream (default 24 over the whole range, 32 with --served-short)")
    ap.add_argument("--served-short", action="store_true",
                    help="served stream over icosphere levels 3-5 and 20-60 steps instead of the whole served range")
    args = ap.parse_args()
    rank, local, ws, dist = dist_init()
    if args.impl == "reference":
        run_reference(args, rank, ws, dist)
        if dist is not None:
            dist.destroy_process_group()
        return

    import __graft_entry__
    __graft_entry__.build()
    from shape_atrophy_gb300 import api

    K, W = args.steps, max(3, args.warmup)
    spec = spec_for(args, W + K)
    sess = api.Session(spec, precision=args.precision, objective=True, device=local)
    sess.step(W)                                       # untimed warm-up steps
    sess.profile(1)                                    # CUDA-event timing of the velocity CG kernel
    info0 = sess.info()
    launches0, iters0 = info0["kernelLaunches"], info0["cgIterTotal"]
    clk = ClockSampler(local)
    clk.start()
    barrier(dist)
    done = sess.step(K)                                # timed: device events around exactly K steps
    info = sess.info()
    clocks = clk.stop()
    if done != K or info["status"] != 0:
        raise RuntimeError(f"solve stopped after {done} of {K} steps, status {info['status']}")
    ms_dev = info["lastStepMs"]
    ms_max = reduce_max(ms_dev, dist, local)
    barrier(dist)
    k_ms, k_cnt, k_bytes, k_flops = sess.profile(0)
    launches = info["kernelLaunches"] - launches0
    cg_iters = info["cgIterTotal"] - iters0
    # the objective (varifold of the current shape against the target): pair evaluations per second
    objective = None
    if rank == 0:
        sess.objective()                               # warm-up
        ts = []
        for _ in range(3):
            t0 = time.perf_counter()
            sess.objective()
            ts.append(time.perf_counter() - t0)
        Vd = spec["elmObj"]["vfdVtxMat"].shape[1]
        Vt = np.asarray(spec["tgt"][2]).size
        pairs = float(Vd + Vt) ** 2
        t_obj = statistics.median(ts)
        evaluated = 0.5 * Vd * (Vd + 1) + float(Vd) * Vt      # symmetric DD half + DT; TT rows cached
        objective = {"kernel": ("k_vfd_rows_fix" if args.precision == "fp64" else "k_vfd_rows") +
                     " (varifold pair sums, Matern-3/2 x Binet)", "deformed": Vd, "target": Vt,
                     "pairs": pairs, "evaluated_pairs": evaluated, "ms": t_obj * 1e3, "pairs_per_s": pairs / t_obj,
                     "evaluated_pairs_per_s": evaluated / t_obj,
                     "what": "one sa_session_objective call (synchronous, host clock), median of 3 after one "
                             "warm-up; pairs = (Vd + Vt)^2 as the reference evaluates them"}
    sess.close()

    value = ws * K / (ms_max / 1000.0)
    hbm, peak_kind = peaks()
    persistent = 0 < 4 * k_cnt < cg_iters              # one launch per solve, not one per iteration
    N_, E_ = spec["lmkIniMat"].shape[1], spec["elmObj"]["elmVtxMat"].shape[1]
    D_ = int(spec["dim"])
    # the kernel that ran: the fixed-point solver reports the FP64 flops of its vector work alone, 2 (7 + D) per entry and
    # iteration; above 19 32-row slices per SM it is the form with several chunks per CTA
    kernel = "k_cg_persist" if persistent else "k_cg_spmv"
    if persistent and args.precision == "fp64" and abs(k_flops / cg_iters - 2.0 * (7 + D_) * N_ * D_) < 1.0:
        kernel = "k_cg_fix" if N_ <= 32 * 19 * api.device_name(local)[1] else "k_cg_fix_many"
    kname = kernel + (" (whole velocity CG solve: matvec, vector updates, dots)" if persistent else
                      " (velocity block matvec + dot)")
    avg_launch_s = (k_ms / k_cnt) / 1000.0 if k_cnt else float("nan")
    alg = algorithmic_bytes(N_, E_, D_, 4 if args.precision == "mixed" else 8)
    iters_per_launch = cg_iters / k_cnt if (k_cnt and persistent) else 1.0
    bytes_per_launch = alg["iteration"] * iters_per_launch if persistent else alg["matvec"]
    achieved = bytes_per_launch / avg_launch_s / 1e9 if k_cnt else None
    traffic = None
    tfile = os.path.join(ROOT, "profiles", f"{kernel}_shell_l5_{args.precision}_traffic.txt")
    if os.path.exists(tfile) and args.workload == "shell":
        for line in open(tfile):
            if line.startswith("dram_bytes_per_iteration:") and cg_iters:
                traffic = float(line.split(":")[1]) * (iters_per_launch if persistent else 1.0)
    roofline = {"bound": "hbm", "achieved": achieved, "peak": hbm, "unit": "GB/s",
                "frac": (achieved / hbm) if achieved else None, "traffic": traffic,
                "kernel": kname, "peak_source": f"{peak_kind} (MEASURED_PEAKS.json hbm_gbs)",
                "bytes_per_launch": bytes_per_launch, "avg_launch_us": avg_launch_s * 1e6, "launches": k_cnt,
                "iters_per_launch": iters_per_launch,
                "bytes_model": "algorithmic bytes of the matrix-free operator, recompute formulation, per CG "
                               "iteration: x + y + coordinates (%d B x N x D each) + elmVtx (4 B x E x V) + layer id "
                               "(4 B x E) + 5 CG vectors (%d B x N x D) = %.2f MB" % (
                                   alg["elt"], alg["elt"], alg["iteration"] / 1e6),
                "l2_operator_bytes_per_launch": k_bytes / k_cnt if k_cnt else None,
                "l2_operator_note": "the assembled 3x3-block operator (values, as digits on the FP64 path), read each "
                                    "iteration: the part that stays in shared and tensor memory from there, the "
                                    "rest from L2, so these bytes are on-chip traffic, not HBM"}
    # whole step, the same accounting (velocity CG + reaction-diffusion CG + per-step element passes)
    rd_iters = info["rdIterTotal"] - info0["rdIterTotal"]
    b_step = (cg_iters * alg["iteration"] + rd_iters * alg["rd_iteration"]) / K + alg["per_step"]
    roofline["step"] = {"bytes_per_step": b_step, "achieved": b_step / (ms_max / K / 1e3) / 1e9,
                        "frac": b_step / (ms_max / K / 1e3) / 1e9 / hbm, "velocity_iters_per_step": cg_iters / K,
                        "rd_iters_per_step": rd_iters / K}
    if k_cnt:
        fl = k_flops / k_cnt / avg_launch_s / 1e12
        fp64 = args.precision == "fp64"
        pk = api.fma_peak(fp64=fp64, device=local)
        sms = api.device_name(local)[1]
        # the pipe's rate per SM clock (clock64 in the FMA loop) at the SM clock sampled during the timed steps
        mhz = (clocks or {}).get("sm_mhz") or pk["sm_mhz"]
        peak_at_clock = pk["flops_per_clock_sm"] * sms * mhz * 1e6 / 1e12
        roofline["fp64_pipe" if fp64 else "fp32_pipe"] = {
            "achieved_tflops": fl, "peak_tflops": peak_at_clock, "frac": fl / peak_at_clock,
            "peak_flops_per_clock_sm": pk["flops_per_clock_sm"], "peak_clock_mhz": mhz,
            "fma_loop_tflops": pk["tflops"], "fma_loop_sm_mhz": pk["sm_mhz"],
            "peak_source": "measured in this run: sa_selftest_fma_peak (independent FMA chains per thread, "
                           "256-thread CTAs, 2/4/8 CTAs per SM, best launch), its rate per SM clock x SMs x the "
                           "SM clock sampled during the timed steps",
            "flops_model": ("2 x 10 x vector entries per CG iteration (per entry the x, r, p, s updates, three dot terms "
                            "and a row of the 3x3 block-Jacobi inverse); the operator's products are summed on the "
                            "integer pipes" if kernel.startswith("k_cg_fix") else
                            "2 x (9 x operator slots + 10 x vector entries) per CG iteration (assembled 3x3 blocks; "
                            "per entry the x, r, p, s updates, three dot terms and a row of the 3x3 block-Jacobi "
                            "inverse)")}

    e2e = None
    if not args.no_e2e and rank == 0:
        spec_e, h2d = pinned_inputs(spec_for(args, K))
        # one untimed call of the same entry point first (a single step): loads the objective's kernels, which
        # the timed step leg above does not launch, so the timed call measures a user's repeated calls
        api.forward(dict(spec_e, timeNum=2), trajectory=True, objective=True, precision=args.precision, device=local)
        walls, devs = [], []
        for _ in range(3):                      # a single call varies by a few % (host set-up on the CPU)
            t0 = time.perf_counter()
            r = api.forward(spec_e, trajectory=True, objective=True, precision=args.precision, device=local)
            walls.append(time.perf_counter() - t0)
            devs.append(r["info"]["elapsedMs"])
        wall = sorted(walls)[1]
        d2h = r["lmkStk"].nbytes + r["tauMat"].nbytes + r["obj"].nbytes
        e2e = {"value": K / wall, "unit": "steps/s", "h2d_bytes_per_step": h2d // K, "d2h_bytes_per_step": d2h // K,
               "what": f"one sa_forward call ({K} steps + objective) with its inputs in pinned host memory: mesh "
                       "upload and set-up, solve, trajectory download; median of 3 calls after one untimed "
                       "one-step call",
               "calls_s": [round(w, 4) for w in walls],
               "device_ms": [round(t, 2) for t in devs],
               "device_ms_what": "the call's device time from its first step to its objective (CUDA events on the "
                                 "library's stream): the rest of the call is upload, set-up and download"}

    served = None
    if not args.no_served and rank == 0 and args.workload == "shell":
        n_req = args.served_requests or (32 if args.served_short else 24)
        served = served_leg(local, n_req, full=not args.served_short)
    batched = None
    if not args.no_batched and rank == 0 and args.workload == "shell":
        batched = batched_leg(local, args.batched_requests)

    mixed_error = None
    ref_run = None
    if rank == 0 and ws == 1 and args.workload == "shell" and not (args.no_cpu and args.no_mixed_error):
        ref_run = oracle_run(args, args.oracle_steps)
    if not args.no_mixed_error and rank == 0 and args.workload == "shell":
        if ref_run is not None:
            mixed_error = mixed_error_leg(args, local, ref_run)
        mixed_error = dict(mixed_error or {}, drift_100_steps=mixed_drift_leg(args, local))

    gradient = None
    if not args.no_gradient and rank == 0 and args.precision == "fp64":
        # objective + gradient with respect to the bump parameters (tangent-linear model) against one forward
        # solve with objective, same K steps, host buffers, both synchronous calls timed on the host clock
        spec_g = spec_for(args, K)
        api.forward(spec_g, trajectory=False, objective=True, device=local)        # warm-up
        t0 = time.perf_counter()
        api.forward(spec_g, trajectory=False, objective=True, device=local)
        t_fwd = time.perf_counter() - t0
        t0 = time.perf_counter()
        gr = api.gradient(spec_g, device=local)
        t_grad = time.perf_counter() - t0
        t0 = time.perf_counter()
        ad = api.adjoint(spec_g, device=local)
        t_adj = time.perf_counter() - t0
        D_, N_ = int(spec_g["dim"]), spec_g["lmkIniMat"].shape[1]
        n_bump, n_all = D_ + 2, D_ + 2 + ad["grad_layer"].size + N_ + D_ * N_
        per_param = (t_grad - t_fwd) / n_bump            # the tangent model's cost per parameter
        gradient = {"what": f"sa_objective_gradient ({K} steps, objective and d obj / d [c, h, sigma], "
                            "tangent-linear model of every step) and sa_objective_adjoint (discrete adjoint: the "
                            "same and per-layer lambda, mu, D, every node's initial concentration and position) "
                            "beside one sa_forward of the same steps",
                    "params": int(gr["grad"].size), "s": t_grad, "forward_s": t_fwd, "vs_forward": t_grad / t_fwd,
                    "status": gr["info"]["status"],
                    "adjoint": {"s": t_adj, "vs_forward": t_adj / t_fwd, "params": int(n_all),
                                "status": ad["info"]["status"],
                                "bump_grad_vs_tangent_max_rel": float(np.abs(ad["grad"] - gr["grad"]).max() /
                                                                      np.abs(gr["grad"]).max())},
                    "tangent_at_20_params_s_extrapolated": t_fwd + 20 * per_param,
                    "tangent_at_all_adjoint_params_s_extrapolated": t_fwd + n_all * per_param}

    cpu = None
    if not args.no_cpu and rank == 0 and ws == 1:
        if ref_run is not None:
            cpu = cpu_from_run(ref_run)
        else:
            v, cores, sample = cpu_sample(spec_for(args, 12), steps=8, warm=3)
            cpu = {"value": v, "unit": "steps/s", "cores": cores, "kind": "port", "sample": sample}

    if rank == 0:
        line = {"metric": METRIC, "value": value, "unit": "steps/s", "n_gpus": ws, "steps": K, "warmup": W,
                "ms_per_step": ms_max / K, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
                "dtype": "f64" if args.precision == "fp64" else "f32+f64", "data": "synthetic",
                "config": {"workload": WORKLOAD if args.workload == "shell" else "2D layered annulus 4096 nodes",
                           "precision": args.precision, "nodes": spec["lmkIniMat"].shape[1],
                           "elements": spec["elmObj"]["elmVtxMat"].shape[1], "cg_iters_per_step": cg_iters / K,
                           "l2": "per-step working set (~0.3 GB) larger than the 129 MB L2",
                           "parallelism": f"replicas x{ws}"},
                "roofline": roofline, "cpu_baseline": cpu, "e2e": e2e, "objective": objective, "gradient": gradient,
                "mixed_error": mixed_error, "served": served, "batched": batched,
                "clocks": clocks,
                "gpu_launches": launches}
        print(json.dumps(line), flush=True)
    if dist is not None:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
