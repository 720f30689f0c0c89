#!/usr/bin/env python
"""Benchmark of the LRes-DFT window solve on one GB300.

Workload (the 1024-electron batched configuration): periodic 8x8x8 H2 crystal,
a = 4.5 bohr, bond 1.4 bohr, molecular centres jittered by U(-0.1, 0.1) bohr per axis,
bond axes uniform on the sphere (seed 0), 64^3 grid (dx = 0.5625 bohr), default s/p
Gaussian basis (6144 functions), one window per atom with R_w = 8 bohr (1024 windows,
n_W 264-312), M = 64 poles (32 upper-half-plane solves per window).  Inputs are
synthetic (seeded geometry; potential = that of the uniform starting density).

One step = one density evaluation at fixed (mu, e_lo) from the potential: H(v) assembly by
atom pairs, gather of the 1024 dense window blocks, the standard-form transform, and then on
the default tridiagonal route the Householder reduction of every window, the owned rows
through its reflectors and the fused shifted-solve + pole-sum kernel over all 1024 x 32
window-pole pairs (on the LDL^T route: one fused LDL^T per window-pole item and the pole
sums).  Metric: window-pole solves per second (1024 * 32 per step).  `value` is measured
with the potential resident on the GPU and the density left there; `e2e` goes through the
public drop-in API with a host potential in and a host density out every step.  Inputs
(window blocks ~0.7 GB) are larger than L2, so no L2 flush is needed between steps.

    python bench.py [--steps K] [--warmup W] [--precision mixed|fp64] [--route auto|tridiag|ldl]
                    [--impl ours|reference]
"""
from __future__ import annotations

import argparse
import datetime
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

WORKLOAD = dict(workload="8x8x8 H2 crystal, 1024 electrons, a=4.5, jitter U(+-0.1), R_w=8, M=64, 64^3 grid",
                natoms=1024, nwin=1024, poles_per_window=32, M=64, R_w=8.0, basis_functions=6144,
                grid="64^3", l2="inputs larger than L2 (no flush)", parallelism="single GPU")
SCF_ITERS = 4           # the fixed SCF window of the GPU and CPU s/iter figures


def build_system(cells=8, assembly="native", tabulation="numpy"):
    from lresdft_gb300 import system
    cr = system.jittered_h2((cells,) * 3, a=4.5, bond=1.4, pts_per_cell=8, jitter=0.1, seed=0)
    return cr, system.LCAOBasis(cr, assembly=assembly, tabulation=tabulation)


def read_peaks():
    try:
        return json.load(open(os.path.join(ROOT, "MEASURED_PEAKS.json")))
    except Exception:
        return None


class Clocks:
    """nvidia-smi sampler (every 50 ms, timestamped) started before the warm-up; the clocks
    reported are those of the samples taken inside the timed region (begin() / end()), or the
    sample nearest to its middle when the region is shorter than the sampling interval."""
    Q = ("timestamp,index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
         "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
         "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")
    NAMES = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]

    def __init__(self):
        self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
        self.p = None
        self.t0 = self.t1 = None

    def start(self):
        try:
            self.p = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits",
                                       "-lms", "50"], stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.p = None

    def begin(self):
        self.t0 = datetime.datetime.now()

    def end(self):
        self.t1 = datetime.datetime.now()

    @classmethod
    def summarise(cls, lines, t0, t1):
        """Clock record of the CSV lines of the samples within [t0, t1]."""
        rows = []
        for line in lines:
            r = [x.strip() for x in line.split(",")]
            if len(r) < 10:
                continue
            try:
                ts = datetime.datetime.strptime(r[0], "%Y/%m/%d %H:%M:%S.%f")
                rows.append((ts, float(r[2]), float(r[3]), [r[6 + i] == "Active" for i in range(4)]))
            except ValueError:
                continue
        if not rows:
            return {"sm_mhz": None, "sm_max_mhz": None, "samples": 0, "reasons": ["no nvidia-smi samples"]}
        inside = [x for x in rows if t0 <= x[0] <= t1]
        if not inside:
            mid = t0 + (t1 - t0) / 2
            inside = [min(rows, key=lambda x: abs((x[0] - mid).total_seconds()))]
        reasons = sorted({cls.NAMES[i] for x in inside for i in range(4) if x[3][i]})
        return {"sm_mhz": float(np.median([x[1] for x in inside])), "sm_max_mhz": max(x[2] for x in inside),
                "samples": len(inside), "sampled_every_ms": 50, "reasons": reasons}

    def stop(self):
        if self.p is None:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["nvidia-smi unavailable"]}
        self.p.terminate()
        self.p.wait()
        self.f.flush()
        lines = open(self.f.name).read().strip().splitlines()
        os.unlink(self.f.name)
        t1 = self.t1 or datetime.datetime.now()
        return self.summarise(lines, self.t0 or t1, t1)


def max_over_ranks(x, dist, device):
    """The largest value of x over the ranks of the job (x itself without torch.distributed):
    every timed leg reports the slowest rank's time, so that the whole-job rate is the units of
    all ranks over the time the last of them needed."""
    if not dist:
        return float(x)
    import torch
    t = torch.tensor([float(x)], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item())


def algorithmic_flops(nW, npoles):
    """(32/3) n^3 real flops per window-pole solve (complex LU + full inverse), fixed."""
    return float(npoles * (32.0 / 3.0) * np.sum(np.asarray(nW, float) ** 3))


def kernel_work(name, nW, mW, P, nnz_h):
    """Algorithmic work of one launch (per step) of each kernel, with the roofline that bounds
    it: ("flop", F) for compute kernels, ("byte", B) for bandwidth kernels."""
    n = np.asarray(nW, float)
    m = np.asarray(mW, float)
    if name == "tri_reduce":          # Householder tridiagonalisation: (4/3) n^3 per window
        return "flop", float(np.sum(4.0 / 3.0 * n ** 3))
    if name == "tri_rows":            # Y = F^ Q: 2 m n^2 per window
        return "flop", float(np.sum(2.0 * m * n ** 2))
    if name == "transform":           # L^-1 H L^-T: n^3/2 + n^3/6 multiply-adds per window
        return "flop", float(np.sum(4.0 / 3.0 * n ** 3))
    if name == "pole_kernel_tri":     # per (pole, row, step): complex multiply-add + u^2/D (20 flops)
        return "flop", float(P * np.sum(20.0 * m * n))
    if name == "pole_kernel_ldl":     # the fixed unit: (32/3) n^3 per window-pole solve
        return "flop", algorithmic_flops(nW, P)
    if name == "assemble_h":          # read the common-point slots, v and basis values, write H
        return "byte", float(nnz_h * 8 * 2 + 0.3e9)
    if name == "gather":              # window blocks written (FP64) and the atom-pair blocks read
        return "byte", float(np.sum(n ** 2) * 8 * 2)
    return None, None


FP32_SIMT_TFLOPS = round(152 * 128 * 2 * 2.07e9 / 1e12, 1)     # 80.5


def roofline_of(name, ms, nW, mW, P, nnz_h, peaks):
    kind, work = kernel_work(name, nW, mW, P, nnz_h)
    if kind is None:
        return None
    if kind == "flop":
        achieved = work / (ms / 1e3) / 1e12
        peak = peaks.get("bf16_tflops_sustained") if peaks else 1700.0
        # these kernels run on the FP32 SIMT pipes; their own ceiling beside the tensor peak
        simt = FP32_SIMT_TFLOPS
        return {"bound": "tensor", "achieved": round(achieved, 3), "peak": peak, "unit": "TFLOP/s",
                "frac": round(achieved / peak, 5), "traffic": None, "kernel_ms": round(ms, 3),
                "algorithmic_flop_per_launch": work,
                "peak_source": "MEASURED_PEAKS.json bf16_tflops_sustained (of measured)" if peaks else "fallback",
                "fp32_simt": {"peak": simt, "frac": round(achieved / simt, 4),
                              "peak_source": "nominal: 152 SMs x 128 FP32 FMA/clk x 2 x 2.07 GHz"}}
    achieved = work / (ms / 1e3) / 1e9
    peak = peaks.get("hbm_gbs") if peaks else 6800.0
    return {"bound": "hbm", "achieved": round(achieved, 1), "peak": peak, "unit": "GB/s",
            "frac": round(achieved / peak, 5), "traffic": None, "kernel_ms": round(ms, 3),
            "algorithmic_bytes_per_launch": work,
            "peak_source": "MEASURED_PEAKS.json hbm_gbs (of measured)" if peaks else "fallback"}


def oz_launches(nwin, m, n, k, gram=False, balance=False):
    """Launches of one FP64 product of all windows on the tensor cores (csrc/oz_gemm.cu): the balance
    of the terms (standard form), the digits of both operands (one of a Gram product) and the product,
    per batch of 1 GB of digits."""
    up = lambda x, t: -(-max(x, 1) // t) * t
    per_window = 18 * (up(m, 64) + up(n, 64)) * up(k, 32) + 4 * (up(m, 64) + up(n, 64) + up(k, 32))
    batch = min(nwin, max((1 << 30) // per_window, 1))
    return ((2 if gram else 3) + balance) * -(-nwin // batch)


def launches_per_step(route, precision, tile_config=0, standard_form="simt", nW=(), mW=()):
    """Our kernels in one step (H(v) + window blocks + standard form + pass)."""
    nwin, n, m = len(nW), int(max(nW, default=0)), int(max(mW, default=0))
    if route == "tridiag":
        # assemble_h, gather, 2 standard-form GEMMs, reduction, rows, pole nodes, pass, window
        # sums; + the FP32 potential per slot, + V^T V and the T factors of the
        # resident-row application (every configuration but 2), + the FP32 copy of the H
        # blocks that the SIMT standard form's FP32 windows are gathered from, + the first columns
        # of windows beyond 384 functions
        if precision == "mixed":
            return 10 + 2 * (tile_config != 2) + (standard_form == "simt") + (tile_config in (0, 4) and n > 384)
        # FP64: assemble_h, gather, symmetric part, reduction, T factors, pole nodes, diagonals of G, P, rows' sums
        # (V a batch of windows at a time, 1 GB), window sums; the products: 2 of the standard form,
        # V^T V and 3 of the rows per panel of 128 reflectors, V = Y P
        total = 10 + 2 * oz_launches(nwin, n, n, n, balance=True)
        for j0 in range(0, n - 2, 128):
            q, r = min(128, n - 2 - j0), n - 1 - j0
            total += oz_launches(nwin, q, q, r, gram=True) + oz_launches(nwin, m, q, r)
            total += oz_launches(nwin, m, q, q) + oz_launches(nwin, m, r, q)
        vb = max(1, min(nwin, (1 << 27) // max(m * n, 1)))
        batches = -(-nwin // vb)
        return total + (batches - 1) + sum(oz_launches(min(vb, nwin - i * vb), m, n, n) for i in range(batches))
    # assemble_h, gather, [split + 2 double-float GEMMs], pole nodes, LDL^T kernel, pole sums
    return 8 if precision == "mixed" else 5


def cpu_leg(b, v, s, mu, e_lo, workers=None):
    from oracle import cpu_baseline
    H = b.H(v)
    r = cpu_baseline.run(H, b.S, b.Xr, s.Wflat, s.Woff, s.Oflat, s.Ooff, mu, e_lo, s.M, b.cr.dV, workers=workers)
    return r


def adjoint_leg(s, s64, mu, e_lo):
    """Band-energy adjoint at fixed N (dE/dv, dE/dH_W, dE/dS_W) on the benchmark potential:
    wall time of one call through the C ABI (pole pass with kept factors, back-substitution,
    accumulation, contraction to the grid; host copy of dv) for the mixed and the FP64 path,
    and the mixed gradient's error against the FP64 one."""
    out = {}
    s.adjoint(mu, e_lo)                         # first call: inverse maps and buffers
    t = time.perf_counter()
    am = s.adjoint(mu, e_lo)
    out["mixed_s"] = round(time.perf_counter() - t, 3)
    t = time.perf_counter()
    a64 = s64.adjoint(mu, e_lo)
    out["fp64_s_first_call"] = round(time.perf_counter() - t, 3)
    out["mixed_speedup"] = round(out["fp64_s_first_call"] / out["mixed_s"], 2)
    dv, dv64 = am["dv"].ravel(), a64["dv"].ravel()
    out["mixed_dv_err_rel"] = float(np.max(np.abs(dv - dv64)) / np.max(np.abs(dv64)))
    out["mixed_kappa_err"] = abs(am["kappa"] - a64["kappa"])
    out["dv_integral_over_N"] = float(np.sum(dv64) / a64["N"])
    return out


def published_leg():
    """The reference's published 1024-electron LRes SCF (benchmarks/scaling_rigorous.py:33-38,
    results/scaling_rigorous.json, n = 8): 512 H2 cells, a = 6, 10 points per cell (80^3 grid),
    rc = 0.6, benchmark basis (rcut 4.5, s 1.2/0.4/0.15, p 0.5), windows on the cell centres with
    R_w = 12.1, M = 64, SCF tol 1e-6 with the reference's mixer.  Timed like the reference's `wall`:
    solver construction + SCF (the basis tabulation before it is excluded there too)."""
    from lresdft_gb300 import LResGPU, system
    from lresdft_gb300.scf import scf_lcao
    cr = system.h2_crystal((8, 8, 8), a=6.0, pts_per_cell=10, rc=0.6)
    b = system.LCAOBasis(cr, rcut=4.5, s_exps=(1.2, 0.4, 0.15), p_exps=(0.5,))
    t0 = time.perf_counter()
    s = LResGPU(b, system.cell_centres((8, 8, 8), 6.0), R_w=12.1, M=64, precision="mixed", tile_config="auto")
    t1 = time.perf_counter()
    st = []
    r = scf_lcao(cr, s, tol=1e-6, step_times=st)
    t2 = time.perf_counter()
    E_pub = -298.93659450240705
    out = {"workload": "8x8x8 H2 cells, a=6, 80^3 grid, cell windows R_w=12.1 (n_W %d-%d), M=64, tol 1e-6, mixed"
                       % (int(s.nW.min()), int(s.nW.max())),
           "wall_s": round(t2 - t0, 2), "scf_wall_s": round(t2 - t1, 2), "iterations": r["iterations"],
           "converged": bool(r["converged"]), "warm_step_s": round(float(np.median(st[1:])), 3) if len(st) > 1 else None,
           "passes": s.passes, "energy": r["energy"], "energy_err_per_e_vs_published": abs(r["energy"] - E_pub) / cr.n_elec,
           "reference_published": {"wall_s": 125.4, "scf_wall_s": 115.0, "iterations": 11, "warm_step_s": 6.3,
                                   "energy": E_pub, "hardware": "1 CPU thread (results/scaling_rigorous.json, median of 3)"},
           "speedup_wall_vs_published": round(125.4 / (t2 - t0), 1)}
    s.close()
    return out


def run_ours(args):
    import torch
    from lresdft_gb300 import LResGPU
    from lresdft_gb300.scf import GridOps, scf_lcao

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    dist = None
    if world > 1:
        import torch.distributed as dist
        dist.init_process_group("nccl")
    t_setup = time.perf_counter()
    cr, b = build_system(args.cells, tabulation="gpu")     # GPU tabulation, native sparse assembly
    basis_s = time.perf_counter() - t_setup
    if args.cells != 8:
        WORKLOAD.update(workload=f"{args.cells}^3 H2 crystal (profiling size), {cr.n_elec} electrons",
                        natoms=len(cr.pos), nwin=len(cr.pos), basis_functions=6 * len(cr.pos), grid=f"{cr.shape[0]}^3")
    if world > 1:
        WORKLOAD.update(parallelism=f"{world} replicas")
    s = LResGPU(b, cr.pos, R_w=8.0, M=64, precision=args.precision, route=args.route,
                tile_config="auto" if args.tile_config is None else args.tile_config)
    s.set_standard_form(args.standard_form)
    route = s.route
    go = GridOps(s)
    vion = go.ion_potential()
    d0 = np.full(cr.shape, cr.n_elec / (cr.ng * cr.dV))
    exc, vxc, vh = go.lda_hartree(d0)
    v = vion + vh + vxc
    # mu and e_lo of this potential: one cold density call through the drop-in API
    dens0, eb0, mu = s.density(v)
    e_lo = s.e_lo
    setup_s = time.perf_counter() - t_setup
    err = None
    try:
        g = np.load(os.path.join(ROOT, "tests", "golden", "jit8.npz"))
        err = {"eband_per_e_vs_reference": abs(eb0 - float(g["eband"])) / cr.n_elec,
               "mu_vs_reference": abs(mu - float(g["mu"])),
               "dens_max_vs_reference": float(np.max(np.abs(dens0.ravel()[g["sample"]] - g["dens_sample"])))}
    except Exception:
        pass

    dev = torch.device("cuda", local)
    v_dev = torch.from_numpy(np.ascontiguousarray(v.ravel())).to(dev)
    nW = s.ctx_nW
    mW = np.array([len(o) for o in s.ctx_own])
    P = s.M // 2
    units = len(s.nW) * P
    lps = launches_per_step(route, args.precision, s.tile_config if isinstance(s.tile_config, int) else 0,
                            args.standard_form, nW, mW)

    def step():
        s.set_potential_device(v_dev.data_ptr())
        return s.pole_pass_device(mu, e_lo)

    clocks = Clocks()
    clocks.start()                        # running before the timed region begins
    for _ in range(args.warmup):
        step()
    torch.cuda.synchronize()
    names = ("pole_kernel", "pole_sums", "assemble_h", "gather", "transform", "tri_reduce", "tri_rows")
    per = {k: [] for k in names}
    if dist:
        dist.barrier()
    torch.cuda.synchronize()
    clocks.begin()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(args.steps):
        step()
        t = s.timings()
        for k in names:
            per[k].append(t[k])
    e1.record()
    torch.cuda.synchronize()
    clocks.end()
    clk = clocks.stop()
    ms_total = max_over_ranks(e0.elapsed_time(e1), dist, dev)
    ms_step = ms_total / args.steps
    value = units * world / (ms_step / 1e3)
    breakdown = {k: round(float(np.mean(x)), 3) for k, x in per.items() if np.mean(x) >= 0}

    # e2e through the drop-in API: host potential in, host density out, every step
    for _ in range(max(1, args.warmup // 2)):
        s.set_potential(v)
        s.pole_pass(mu, e_lo)
    torch.cuda.synchronize()
    if dist:
        dist.barrier()
    t = time.perf_counter()
    for _ in range(args.steps):
        s.set_potential(v)
        dens, N, eb = s.pole_pass(mu, e_lo)
    torch.cuda.synchronize()
    e2e_ms = max_over_ranks((time.perf_counter() - t) * 1e3 / args.steps, dist, dev)
    h2d = cr.ng * 8 + 3 * 16 * P
    d2h = cr.ng * 8 + 2 * 8 * len(nW) + 4

    # one more mu trial on the same Hamiltonian (what each extra pass of a density call costs)
    torch.cuda.synchronize()
    t = time.perf_counter()
    for k in range(args.steps):
        s.pole_pass_device(mu + 1e-4 * (k % 3), e_lo)
    torch.cuda.synchronize()
    pass_ms = (time.perf_counter() - t) * 1e3 / args.steps

    # the same step as one CUDA graph (H(v) from device v + capturable pass, N and E_band
    # left on the device): replayed K times, timed on the replay stream
    graph_leg = None
    try:
        out_dev = torch.zeros(2, dtype=torch.float64, device=dev)
        side = torch.cuda.Stream(device=dev)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            st = side.cuda_stream
            s.set_potential_device(v_dev.data_ptr(), st)
            s.pass_async(mu, e_lo, out_dev.data_ptr(), st)
        side.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            st = torch.cuda.current_stream().cuda_stream
            s.set_potential_device(v_dev.data_ptr(), st)
            s.pass_async(mu, e_lo, out_dev.data_ptr(), st)
        for _ in range(args.warmup):
            graph.replay()
        torch.cuda.synchronize()
        g0, g1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        g0.record()
        for _ in range(args.steps):
            graph.replay()
        g1.record()
        torch.cuda.synchronize()
        g_ms = g0.elapsed_time(g1) / args.steps
        gN = float(out_dev[0].item())
        if s.status() != 0 or abs(gN - cr.n_elec) > 1e-3:
            raise RuntimeError(f"graph replay gave N={gN}, status {s.status()}")
        graph_leg = {"value": round(units / (g_ms / 1e3), 1), "unit": "window-pole solves/s",
                     "ms_per_step": round(g_ms, 3), "launches_per_step": lps + 1}
        del graph
    except Exception as exc:          # reported, never silently replaced
        graph_leg = {"error": str(exc)[:200]}

    # roofline of the dominant kernel of the step (largest device time), with its own
    # algorithmic work; the fixed (32/3) n^3 unit of the whole step beside it
    peaks = read_peaks()
    nnz_h = float(b.S.nnz)
    cand = {k: breakdown[k] for k in ("pole_kernel", "transform", "tri_reduce", "tri_rows", "assemble_h", "gather")
            if k in breakdown}
    # kernels of the chosen tridiagonal configuration (TriCfg in csrc/tridiag.cu): mixed
    # configurations 0 and 4 reduce with the window on its SM, all but 2 apply with resident rows
    mixed = args.precision == "mixed"
    cfg = s.tile_config if isinstance(s.tile_config, int) else 0
    kernel_names = {"pole_kernel": ("tri_pass_kernel" if mixed else "tri_pmat_kernel")
                    if route == "tridiag" else "ldl_left_kernel",
                    "transform": ("gemm_tc_kernel" if args.standard_form == "tensor" else "gemm_f32blk_kernel")
                    if (route == "tridiag" and mixed)
                    else ("oz_gemm_kernel (standard form)" if args.precision == "fp64" else "gemm_df64_kernel"),
                    "tri_reduce": "tri_reduce_reg_kernel" if (mixed and cfg in (0, 4)) else "tri_reduce_kernel",
                    "tri_rows": ("tri_apply_res_kernel" if cfg != 2 else "tri_apply_kernel") if mixed else "oz_gemm_kernel (rows)",
                    "assemble_h": "assemble_h32_kernel" if mixed else "assemble_h_kernel",
                    "gather": "gather_windows_kernel"}

    def work_name(k):
        return {"pole_kernel": "pole_kernel_tri" if route == "tridiag" else "pole_kernel_ldl"}.get(k, k)
    dom = max(cand, key=cand.get)
    roof = roofline_of(work_name(dom), cand[dom], nW, mW, P, nnz_h, peaks)
    roof["kernel"] = kernel_names[dom]
    try:
        tr = json.load(open(os.path.join(ROOT, "profiles", "traffic.json")))
        roof["traffic"] = tr.get(f"{args.precision}/{route}/{roof['kernel']}")
    except Exception:
        pass
    others = {}
    for k in cand:
        if k != dom:
            r = roofline_of(work_name(k), cand[k], nW, mW, P, nnz_h, peaks)
            if r:
                others[kernel_names[k]] = {x: r[x] for x in ("bound", "achieved", "unit", "frac", "kernel_ms")}
    flops_step = algorithmic_flops(nW, P)

    line = {
        "metric": "window-pole solves/s", "value": round(value, 1), "unit": "window-pole solves/s",
        "n_gpus": world, "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(ms_step, 3),
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
        "dtype": "c64 (FP32 reduction, FP64 sums)" if args.precision == "mixed" else "c128",
        "precision": args.precision, "route": route,
        "data": "synthetic (seeded H2 crystal, potential of the uniform starting density)",
        "config": dict(WORKLOAD),
        "e2e": {"value": round(units * world / (e2e_ms / 1e3), 1), "unit": "window-pole solves/s",
                "ms_per_step": round(e2e_ms, 3), "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h)},
        "gpu_launches": lps * args.steps,
        "roofline": roof,
        "roofline_other_kernels": others,
        "equivalent_work": {"unit": "(32/3) n_W^3 real flops per window-pole solve (fixed)",
                            "flop_per_step": flops_step,
                            "tflops_per_s": round(flops_step / (ms_step / 1e3) / 1e12, 2)},
        "clocks": clk,
        "breakdown_ms": breakdown,
        "standard_form": s.standard_form,
        "tile_config": {"chosen": s.tile_config,
                        "ms_per_config": None if getattr(s, "tune_ms", None) is None
                        else [round(float(x), 3) for x in s.tune_ms]},
        "extra_pass_ms": round(pass_ms, 3),
        "cuda_graph": graph_leg,
        "setup_s": round(setup_s, 2), "basis_s": round(basis_s, 2), "basis_tabulation": "gpu", "accuracy": err,
    }

    # FP64 path on the same potential (the target ratio is mixed vs FP64)
    if args.precision == "mixed" and args.fp64_steps > 0:
        s64 = LResGPU(b, cr.pos, R_w=8.0, M=64, precision="fp64", route=args.route, tile_config=3)
        s64.set_potential_device(v_dev.data_ptr())
        s64.pole_pass_device(mu, e_lo)
        torch.cuda.synchronize()
        a0, a1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a0.record()
        for _ in range(args.fp64_steps):
            s64.set_potential_device(v_dev.data_ptr())
            N64, E64 = s64.pole_pass_device(mu, e_lo)
        a1.record()
        torch.cuda.synchronize()
        ms64 = a0.elapsed_time(a1) / args.fp64_steps
        t64 = s64.timings()
        _, N32, E32 = s.pole_pass(mu, e_lo)
        line["fp64"] = {"route": s64.route, "value": round(units / (ms64 / 1e3), 1), "ms_per_step": round(ms64, 2),
                        "mixed_speedup": round(ms64 / ms_step, 2),
                        "breakdown_ms": {k: round(float(t64[k]), 3) for k in names if t64[k] >= 0},
                        "mixed_eband_err_per_e": abs(E32 - E64) / cr.n_elec,
                        "mixed_count_err": abs(N32 - N64)}
        # the LDL^T route on the same potential (SIMT tile configuration 1 and the tensor-core
        # configuration 4), for comparison with the default route
        if route == "tridiag" and args.ldl_leg:
            ldl = {}
            try:
                s.set_route("ldl")
                for cfg in (1, 4):
                    s.autotune(mu, e_lo, config=cfg)
                    s.pole_pass(mu, e_lo)
                    _, Nl, El = s.pole_pass(mu, e_lo)
                    ldl[f"config{cfg}"] = {"pole_kernel_ms": round(s.timings()["pole_kernel"], 2),
                                           "eband_err_per_e_vs_fp64": abs(El - E64) / cr.n_elec}
                ldl["note"] = "LDL^T route (one fused factorisation per window-pole item); config4 = tcgen05 3xTF32"
            except Exception as exc:
                ldl["error"] = str(exc)[:200]
            finally:
                s.set_route("tridiag")
            line["ldl_route"] = ldl
        if args.adjoint:
            line["adjoint"] = adjoint_leg(s, s64, mu, e_lo)
        s64.close()

    # SCF seconds per iteration: the same fixed iteration window from the same start for the
    # mixed and the FP64 solver (the 1024-electron SCF does not converge with the reference
    # mixer, so a fixed window is timed); median of iterations 3..end; energies after the
    # window compared per electron
    if args.scf_iters > 0:
        scf = {}
        for prec in ("mixed", "fp64") if args.precision == "mixed" and args.fp64_scf else (args.precision,):
            st = []
            s_scf = LResGPU(b, cr.pos, R_w=8.0, M=64, precision=prec, route=args.route)
            r = scf_lcao(cr, s_scf, tol=1e-12, maxiter=args.scf_iters, vion=vion, step_times=st)
            scf[prec] = {"s_per_iter": round(float(np.median(st[2:])) if len(st) > 2 else float(np.median(st)), 4),
                         "iterations": len(st), "passes": s_scf.passes, "first_iter_s": round(st[0], 3),
                         "energy": r["energy"]}
            s_scf.close()
        if "fp64" in scf and "mixed" in scf:
            scf["mixed_speedup_per_iter"] = round(scf["fp64"]["s_per_iter"] / scf["mixed"]["s_per_iter"], 2)
            scf["energy_diff_per_e"] = abs(scf["mixed"]["energy"] - scf["fp64"]["energy"]) / cr.n_elec
        scf["note"] = (f"fixed window of {args.scf_iters} SCF iterations from the uniform start (reference "
                       "Pulay mixer, tol not reached at 1024 e); s/iter = median of iterations 3..end")
        line["scf"] = scf

    if rank == 0 and world == 1 and args.published:
        try:
            line["published_scf_1024"] = published_leg()
        except Exception as exc:
            line["published_scf_1024"] = {"error": str(exc)[:200]}

    if rank == 0 and world == 1 and not args.no_cpu:
        try:
            c = cpu_leg(b, v, s, mu, e_lo)
            line["cpu_baseline"] = {"value": round(c["eig_rate"], 1), "unit": "window-pole solves/s (equivalent)",
                                    "cores": c["workers"], "kind": "port",
                                    "sample": f"one full eigen-route window pass over all {c['nwin']} windows "
                                              f"({c['eig_wall']:.2f} s wall), dsygvx below c+1.5R per window",
                                    "pole_route_value": round(c["pole_rate"], 1),
                                    "pole_route_sample": f"scipy solve per window-pole on {c['pole_windows']} windows"}
            if args.cpu_scf and args.scf_iters > 0:
                from oracle import cpu_baseline
                cs = cpu_baseline.scf_window(cr, b, vion, 8.0, 64, args.scf_iters)
                line["cpu_baseline"]["scf"] = dict(cs, unit="s/iter", iterations=args.scf_iters,
                                                   note="reference SCF (eigen route, reuse_vectors=False) over the "
                                                        "same fixed iteration window, window passes on all cores")
                if "scf" in line and "mixed" in line["scf"]:
                    line["cpu_baseline"]["scf"]["gpu_mixed_speedup_per_iter"] = round(
                        cs["s_per_iter"] / line["scf"]["mixed"]["s_per_iter"], 1)
        except Exception as ex:   # the CPU leg must not hide the GPU result
            line["cpu_baseline"] = {"value": None, "error": repr(ex)}
    s.close()
    if rank == 0:
        print(json.dumps(line), flush=True)
    if dist:
        dist.destroy_process_group()


def run_reference(args):
    """The reference's CPU algorithm for the path (the eigen route of _lrft_cpp.lrft_windows,
    restated in oracle/, windows spread over all host cores), timed on the same workload and
    metric; nothing of the GPU library is imported."""
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    from oracle import cpu_baseline
    from oracle import lrft_oracle as orc
    cr, b = build_system(assembly="scipy")      # the reference's own scipy assembly
    # the potential and (mu, e_lo) of the reference's own cold call (tests/golden/jit8.npz)
    g = np.load(os.path.join(ROOT, "tests", "golden", "jit8.npz"))
    vion = orc.ion_potential(cr)
    v = orc.guess_potential(cr, vion)
    windows, own, _ = orc.window_setup(b, cr.pos, 8.0)

    class W:
        pass
    s = W()
    s.M = 64
    s.Wflat = np.concatenate(windows).astype(np.int64)
    s.Woff = np.concatenate([[0], np.cumsum([len(w) for w in windows])]).astype(np.int64)
    s.Oflat = np.concatenate(own).astype(np.int64)
    s.Ooff = np.concatenate([[0], np.cumsum([len(o) for o in own])]).astype(np.int64)
    rates = []
    for i in range(args.warmup + args.steps):
        c = cpu_leg(b, v, s, float(g["mu"]), float(g["e_lo"]))
        if i >= args.warmup:
            rates.append(c["eig_rate"])
    val = float(np.median(rates))
    line = {"impl": "reference", "metric": "window-pole solves/s", "value": round(val, 1),
            "unit": "window-pole solves/s", "n_gpus": int(os.environ.get("WORLD_SIZE", "1")),
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": round(1024 * 32 / val * 1e3, 2),
            "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "f64",
            "precision": "fp64 eigen route (reference algorithm)",
            "data": "synthetic (seeded H2 crystal, potential of the uniform starting density)",
            "config": dict(WORKLOAD),
            "cpu_baseline": {"value": round(val, 1), "unit": "window-pole solves/s (equivalent)",
                             "cores": c["workers"], "kind": "port",
                             "sample": f"full eigen-route window pass over {c['nwin']} windows per step"},
            "e2e": {"value": round(val, 1), "unit": "window-pole solves/s", "h2d_bytes_per_step": 0,
                    "d2h_bytes_per_step": 0}}
    iters = getattr(args, "scf_iters", SCF_ITERS)
    if getattr(args, "cpu_scf", True) and iters > 0:
        try:
            cs = cpu_baseline.scf_window(cr, b, vion, 8.0, 64, iters)
            line["cpu_baseline"]["scf"] = dict(cs, unit="s/iter", iterations=iters)
        except Exception as ex:
            line["cpu_baseline"]["scf"] = {"error": repr(ex)}
    print(json.dumps(line), flush=True)


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=30)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", choices=["ours", "reference"], default="ours")
    ap.add_argument("--precision", choices=["mixed", "fp64"], default="mixed")
    ap.add_argument("--fp64-steps", type=int, default=2)
    ap.add_argument("--scf-iters", type=int, default=SCF_ITERS)
    ap.add_argument("--route", choices=["auto", "tridiag", "ldl"], default="auto")
    ap.add_argument("--no-ldl-leg", dest="ldl_leg", action="store_false",
                    help="skip the LDL^T-route comparison passes")
    ap.add_argument("--no-cpu-scf", dest="cpu_scf", action="store_false",
                    help="skip the reference SCF s/iter on the host cores (about a minute at 1024 electrons)")
    ap.add_argument("--no-fp64-scf", dest="fp64_scf", action="store_false",
                    help="skip the FP64 SCF window (about a minute at 1024 electrons)")
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-published", dest="published", action="store_false",
                    help="skip the reference's published 1024-electron SCF setting")
    ap.add_argument("--no-adjoint", dest="adjoint", action="store_false",
                    help="skip the band-energy adjoint leg (mixed and FP64)")
    ap.add_argument("--cells", type=int, default=8, help="crystal of cells^3 H2 (8 = the benchmark workload)")
    ap.add_argument("--tile-config", type=int, default=None, help="force a pole-kernel tile configuration")
    ap.add_argument("--standard-form", choices=["simt", "tensor"], default="simt",
                    help="kernel of the mixed standard form (SIMT FP32 GEMMs or tcgen05 3xTF32)")
    args = ap.parse_args()
    if args.warmup < 3:
        args.warmup = 3
    if args.impl == "reference":
        run_reference(args)
    else:
        run_ours(args)


if __name__ == "__main__":
    main()
