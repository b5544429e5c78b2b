#!/usr/bin/env python
"""Throughput of the 3-phonon scattering path on B200: one JSON line on stdout.

Workload: fcc rocksalt 2-atom cell (a = 4.21 A, Mg/O), seeded spring-model FC2
and FC3, 24^3 Gamma-centred mesh (13824 q, 413 irreducible q0), T = 100/300/700 K,
Gaussian smearing sigma = 2 cm^-1.  One step = the whole path for all
temperatures: device phonons for the grid and the irreducible set, pair
enumeration for every q0, V3 -> W -> Gaussian delta sum for every pair, RTA
kappa (symmetrised).  V3 runs on the tensor cores (--precision, default the
compensated BF16x3; phonons, deltas, rates and kappa stay FP64); the plain FP64
path is timed in the same run, and the line reports the time-to-kappa of both
and the largest linewidth and kappa error of the measured path against FP64.

metric: 3-phonon scattering evaluations per second, one evaluation = one mode
triple (s0,s1,s2) of one enumerated pair (sum over q0 of npairs * Ndof^3 per
step; the three temperatures reuse the same V3).

--impl reference times the CPU restatement of the reference (the oracle; the
Fortran reference cannot be built on this image) on a bounded sample of the
same workload, with all host threads.

Extra legs on the other configurations (--legs, default all four): c2 iterative
kappa at 24^3 (T = 100/300/700 K, tolerance 1e-6); c3 three- plus four-phonon
plus isotope kappa at 16^3 with the tensor-core V4 (FP64 four-phonon time from
sampled q0 unless --c3-fp64 full); c4 the batched uneven workload and 200 path
points; c5 the surrogate-screened four-phonon run (trained at 12^3, screened at
20^3, T = 300 and 900 K).  Each reports its own times and errors in the line.
"""
from __future__ import annotations

import argparse
import csv
import io
import json
import os
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

MESH = 24
TEMPS = [100.0, 300.0, 700.0]
SIGMA = 0.3767          # 2 cm^-1 in rad/ps
DELTA = "gauss"
WORKLOAD = "rocksalt2-fcc-24x24x24-3ph-gauss-T100/300/700"
METRIC = "3ph scattering evals/s"


def parse():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=10)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--mesh", type=int, default=MESH)
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--legs", default="c2,c3,c4,c5",
                    help="extra legs on their own configurations: c2 iterative kappa (24^3), c3 four-phonon + "
                         "isotope (16^3), c4 batched workloads + path points, c5 surrogate screening (12^3 -> 20^3); "
                         "'none' for the main leg alone (all four take about two minutes on one B200)")
    ap.add_argument("--mesh4", type=int, default=16, help="mesh of the four-phonon leg")
    ap.add_argument("--c3-fp64", default="sample", choices=["sample", "full", "off"],
                    help="FP64 comparison of the four-phonon leg: 'sample' times 8 evenly spaced q0 and "
                         "extrapolates by quartet count (kappa error not reported), 'full' runs every q0")
    ap.add_argument("--precision", default="bf16x3", choices=["fp64", "bf16", "bf16x3"],
                    help="arithmetic of V3 on the measured path (FP64 is always timed beside it)")
    return ap.parse_args()


def algorithmic_flops_per_pair(ndof, na3_counts):
    """V3 in the factored form: phase-weighted FC sum 4*27*sum_mu Na3^2, three
    eigenvector contractions 3*8*Ndof^4, |Phi|^2 scaling 3*Ndof^3."""
    return 4 * 27 * int(np.sum(np.asarray(na3_counts) ** 2)) + 3 * 8 * ndof ** 4 + 3 * ndof ** 3


FALLBACK_PEAKS = {"hbm_gbs": 6650.0, "bf16_tflops": 1590.0}  # the pool's earlier measurement


def measured_peaks():
    """Roofline denominators: the driver-written MEASURED_PEAKS.json beside this file when present
    ("of measured"), else the pool's earlier measurement ("of fallback")."""
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        with open(path) as f:
            d = json.load(f)
        flat = {}

        def walk(x, pre=""):
            if isinstance(x, dict):
                for k, v in x.items():
                    walk(v, f"{pre}{k}.")
            elif isinstance(x, (int, float)) and not isinstance(x, bool):
                flat[pre[:-1]] = float(x)
        walk(d)

        def pick(*keys):
            for k in keys:
                for fk, v in flat.items():
                    if fk == k or fk.endswith("." + k):
                        return v
            return None
        bf = pick("bf16_tflops", "bf16_dense_tflops")
        hbm = pick("hbm_gbs", "hbm_copy_gbs")
        if bf:
            return {"bf16_tflops": bf, "hbm_gbs": hbm or FALLBACK_PEAKS["hbm_gbs"],
                    "source": "MEASURED_PEAKS.json bf16_tflops (burst, cuBLAS bf16 GEMM), of measured"}
    except (OSError, ValueError):
        pass
    return dict(FALLBACK_PEAKS, source="no MEASURED_PEAKS.json: the pool's earlier 1.59 PFLOP/s bf16, of fallback")

# DRAM bytes per tiled pair of the tensor-core pass (read + write), from one ncu capture of the
# 16^3 rocksalt launch (140,383 of its 297,076 pairs have a mode triple inside the delta window and
# are tiled; 61.0 MB read, 0.68 MB written: the operand tables and mode records in, the sums out)
TC_DRAM_BYTES_PER_TILED_PAIR = (60.978176e6 + 0.677120e6) / 140383


def tc_issued_flops_per_tile(passes):
    """Two basis atoms x 3 K-steps x passes MMAs of M128 N48 K16."""
    return 2 * 3 * passes * 2 * 128 * 48 * 16




class Clocks:
    """SM clock and clock-event reasons sampled through NVML by a background thread while a timed
    region is open (begin/end around each one); median SM clock under load, max clock and the
    reasons seen.  Falls back to nvidia-smi polling when the NVML bindings are missing."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")

    def __init__(self, index, bus_id=None):
        import threading
        self.index, self.bus_id = index, bus_id
        self.rows = []
        self.lock = threading.Lock()
        self.active = threading.Event()
        self.done = threading.Event()
        self.thread = None
        self.p = None
        self.f = None

    def _query(self, nv, h):
        names = {"hw_slowdown": nv.nvmlClocksEventReasonHwSlowdown,
                 "hw_thermal_slowdown": nv.nvmlClocksEventReasonHwThermalSlowdown,
                 "sw_thermal_slowdown": nv.nvmlClocksEventReasonSwThermalSlowdown,
                 "sw_power_cap": nv.nvmlClocksEventReasonSwPowerCap}
        smax = nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM)
        sm = nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)
        r = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
        return (float(sm), float(smax), sorted(k for k, v in names.items() if r & v))

    def _nvml_loop(self, nv, h):
        while not self.done.is_set():
            if not self.active.wait(0.05) or self.done.is_set():
                continue
            with self.lock:  # a query that began inside the timed region is kept, however short it is
                self.rows.append(self._query(nv, h))
            time.sleep(0.002)

    def sample(self):
        """One query from the calling thread, made while the GPU runs the step just queued (a timed
        region of a few milliseconds can fall between two of the background thread's queries)."""
        if self.thread is not None and self.active.is_set():
            with self.lock:
                self.rows.append(self._query(self.nv, self.h))

    def start(self):
        try:
            import pynvml as nv
            nv.nvmlInit()
            h = (nv.nvmlDeviceGetHandleByPciBusId(self.bus_id) if self.bus_id
                 else nv.nvmlDeviceGetHandleByIndex(self.index))
            self.nv, self.h = nv, h
            import threading
            self.thread = threading.Thread(target=self._nvml_loop, args=(nv, h), daemon=True)
            self.thread.start()
        except Exception:
            self.thread = None
            self.f = tempfile.NamedTemporaryFile("w+", suffix=".csv", delete=False)
            try:
                self.p = subprocess.Popen(["nvidia-smi", "-i", str(self.index), f"--query-gpu={self.Q}",
                                           "--format=csv,noheader,nounits", "-lms", "100"], stdout=self.f,
                                          stderr=subprocess.DEVNULL)
            except OSError:
                self.p = None

    def begin(self):
        self.active.set()

    def end(self):
        self.active.clear()
        with self.lock:  # let a query in flight finish and be recorded
            pass

    def stop(self):
        rows = []
        if self.thread is not None:
            self.done.set()
            self.active.set()
            self.thread.join(timeout=5)
            rows = self.rows
        elif self.p is not None:
            self.p.terminate()
            try:
                self.p.wait(timeout=5)
            except subprocess.TimeoutExpired:
                self.p.kill()
            self.f.flush()
            names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
            with open(self.f.name) as fh:
                for r in csv.reader(fh):
                    r = [x.strip() for x in r]
                    if len(r) >= 9 and r[1].replace(".", "").isdigit() and r[2].replace(".", "").isdigit():
                        rows.append((float(r[1]), float(r[2]), [names[k] for k in range(4) if r[5 + k].lower() == "active"]))
            os.unlink(self.f.name)
        if not rows:
            return None
        smax = max(r[1] for r in rows)
        sm = [r[0] for r in rows]
        load = [x for x in sm if x > 0.5 * smax] or sm
        reasons = sorted({k for r in rows for k in r[2]})
        return {"sm_mhz": float(np.median(load)), "sm_max_mhz": smax, "reasons": reasons, "samples": len(rows),
                "source": "nvml" if self.thread is not None else "nvidia-smi"}


def pci_bus_id(torch, index):
    """NVML bus id ('dddddddd:bb:dd.0') of a CUDA device, so the sampler reads the GPU this process
    runs on whatever CUDA_VISIBLE_DEVICES maps; None when torch does not expose it."""
    try:
        p = torch.cuda.get_device_properties(index)
        return f"{p.pci_domain_id:08x}:{p.pci_bus_id:02x}:{p.pci_device_id:02x}.0"
    except Exception:
        return None


def fp64_peak_tflops(torch):
    """Measured FP64 ceiling of this GPU in this run: cuBLAS DGEMM 8192^3, best of 5."""
    n = 8192
    a = torch.randn(n, n, dtype=torch.float64, device="cuda")
    b = torch.randn(n, n, dtype=torch.float64, device="cuda")
    torch.matmul(a, b)
    best = 0.0
    for _ in range(5):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        torch.matmul(a, b)
        e1.record()
        torch.cuda.synchronize()
        best = max(best, 2.0 * n ** 3 / (e0.elapsed_time(e1) * 1e-3) / 1e12)
    del a, b
    torch.cuda.empty_cache()
    return best


def cpu_baseline(cr, mesh, temps, ph_grid, ph_irr, irr_int, sample, threads_note, lw_out=None):
    """The oracle (CPU restatement of the reference loops) on a sample of q0: enumeration,
    naive V3 (ScatterMatEl loop order) and the Gaussian sum at every temperature.  lw_out (a
    dict) receives the oracle linewidths of each sampled q0, [T][s]."""
    from oracle import driver as D
    qi, qf, _ = D.make_tetrahedron(mesh, cr.G)
    evals = 0
    t0 = time.perf_counter()
    for i0 in sample:
        A, perm, cnt = D.momentum3(mesh, qi, irr_int[i0])
        sctr = D.scatter_w3(cr, qf, qi, irr_int[i0], ph_irr["evec"][i0], ph_irr["onebyomega"][i0], ph_grid["evec"],
                            ph_grid["onebyomega"], perm)
        lws = []
        for it in range(len(temps)):
            r = D.lw3_gauss(ph_irr["omega"][i0], ph_grid["omega"], ph_grid["nbe"][it], sctr, A, qi, SIGMA)
            lws.append(np.asarray(r[0] if isinstance(r, tuple) else r))
        if lw_out is not None:
            lw_out[i0] = np.array(lws)
        evals += cnt[0] * cr.ndof ** 3
    dt = time.perf_counter() - t0
    return evals / dt, dt, D.lib().orc_num_threads()


def run_reference(args):
    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return 0
    from oracle import driver as D
    from oracle import phonons as P
    from spring_b200 import synthetic as S
    cr = S.build("rocksalt2")
    mesh = (args.mesh,) * 3
    qi, qf, _ = D.make_tetrahedron(mesh, cr.G)
    W, _ = S.point_group(cr)
    ir = D.irr_q(mesh, W, qi)
    irr = ir["irr_q_pnt_int"]
    irq = ((cr.G / np.array(mesh)[None, :]) @ irr.T.astype(float)).T
    args_ph = (cr.latvec, cr.mass, cr.fc2_atm_num, cr.fc2_atm_indx, cr.fc2)
    ph_grid = P.get_phonon(*args_ph, qf, TEMPS)
    ph_irr = P.get_phonon(*args_ph, irq, TEMPS)
    nq0 = irr.shape[0]
    order = [(7 * k + 1) % nq0 for k in range(args.steps + args.warmup)]
    for k in range(args.warmup):
        cpu_baseline(cr, mesh, TEMPS, ph_grid, ph_irr, irr, [order[k]], "")
    evals, secs = 0, 0.0
    threads = 1
    for k in range(args.steps):
        i0 = order[args.warmup + k]
        v, dt, threads = cpu_baseline(cr, mesh, TEMPS, ph_grid, ph_irr, irr, [i0], "")
        evals += v * dt
        secs += dt
    value = evals / secs
    line = {"impl": "reference", "metric": METRIC, "value": value, "unit": "evals/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1e3 * secs / args.steps,
            "higher_is_better": True, "scaling": "strong", "vs_baseline": None, "dtype": "f64", "data": "synthetic",
            "config": {"workload": WORKLOAD, "mesh": list(mesh), "temperatures": TEMPS, "sigma_rad_ps": SIGMA,
                       "sample": "one irreducible q0 per step"},
            "cpu_baseline": {"value": value, "unit": "evals/s", "cores": threads, "kind": "port",
                             "sample": f"{args.steps} of {nq0} irreducible q0 (one per step): enumeration, V3 in "
                                       "the reference loop order, Gaussian sum at 3 T; phonons excluded"},
            "e2e": {"value": value, "unit": "evals/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}}
    print(json.dumps(line), flush=True)
    return 0


def _ev_ms(torch, fn):
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record()
    r = fn()
    e1.record()
    torch.cuda.synchronize()
    return r, e0.elapsed_time(e1)


def _kdiag(k):
    return np.array([k[0], k[4], k[8]])


def fourph_c3_leg(torch, mesh=16, prec4="bf16x3", fp64="sample"):
    """Three-phonon + four-phonon + isotope kappa of the rocksalt cell with FC4 at mesh^3, 300 K,
    Gaussian 2 cm^-1, isotope g2 = 1e-3 on both atoms.  Timed from the phonons to kappa with the
    tensor-core V3 (BF16x3) and V4 (prec4).  The plain FP64 path (k_v3s + k_v4) beside it: 'full'
    runs it for every q0 (times and kappa, rate and linewidth errors), 'sample' runs the FP64
    four-phonon rates of 8 evenly spaced q0 (their errors, and the FP64 four-phonon time
    extrapolated by quartet count), 'off' skips it."""
    from spring_b200 import synthetic as S
    from spring_b200.api import from_crystal
    cr = S.build("rocksalt2", fc4=True)
    T = [300.0]
    g2 = [1e-3, 1e-3]
    ctx, info = from_crystal(cr, (mesh,) * 3, T, with_fc4=True)
    counts = np.array([ctx.count4(i + 1)[0] for i in range(ctx.nq0)], dtype=np.int64)
    quartets = int(counts.sum())

    def run(p3, p4):
        def step():
            ctx.compute_phonons(T)
            ctx.reset_linewidths()
            ctx.set_precision(p3)
            ctx.linewidth3(1, ctx.nq0, "gauss", SIGMA, want=False)
            ctx.linewidth_iso(1, ctx.nq0, g2, delta="gauss", sigma=SIGMA, want=False)
            ctx.set_precision(p4)
            r4 = ctx.linewidth4(1, ctx.nq0, "gauss", SIGMA)
            return r4, ctx.get_linewidths(), ctx.kappa_rta(info["Rxyz"])[0]
        return _ev_ms(torch, step)

    ctx.set_precision(prec4)
    ctx.linewidth4(1, 1, "gauss", SIGMA)  # warm-up (allocations, tables)
    ctx.set_profiling(True)
    (r4m, lwm, km), ms_m = run("bf16x3", prec4)
    v4_ms, v4_n = ctx.kernel_time("k_v4tc")
    ctx.set_profiling(False)
    out = {"mesh": [mesh] * 3, "temperature": 300.0, "isotope_g2": g2, "sigma_rad_ps": SIGMA,
           "irreducible_q0": int(ctx.nq0), "quartets": quartets, "v4_arithmetic": prec4,
           "time_to_kappa_ms": ms_m, "v4tc_kernel_ms": v4_ms, "v4tc_launches": v4_n,
           "evals_per_s_4ph": quartets * 6 ** 4 / (v4_ms * 1e-3) if v4_ms else None,
           "kappa_diag": _kdiag(km).tolist(),
           "what": "phonons + 3ph (bf16x3 V3) + isotope + 4ph (tensor-core V4) + RTA kappa, every q0; one 4ph eval = "
                   "one (s0..s3) of one quartet"}
    if fp64 == "full":
        (r4f, lwf, kf), ms_f = run("fp64", "fp64")
        big = r4f > 1e-3 * r4f.max()
        lbig = lwf > 1e-3 * lwf.max()
        out.update({"fp64_time_to_kappa_ms": ms_f, "fp64_over_mixed": ms_f / ms_m,
                    "kappa_max_rel_err_vs_fp64": float(np.abs(_kdiag(km) / _kdiag(kf) - 1).max()),
                    "linewidth_max_rel_err_vs_fp64": float((np.abs(lwm[lbig] - lwf[lbig]) / lwf[lbig]).max()),
                    "rate4_max_rel_err_vs_fp64": float((np.abs(r4m[big] - r4f[big]) / r4f[big]).max()),
                    "fp64_kappa_diag": _kdiag(kf).tolist()})
    elif fp64 == "sample":
        ctx.set_precision("fp64")
        sample = list(np.linspace(0, ctx.nq0 - 1, 8).round().astype(int))
        f_ms, err = 0.0, 0.0
        for i in sample:
            r, ms = _ev_ms(torch, lambda: ctx.linewidth4(int(i) + 1, 1, "gauss", SIGMA))
            f_ms += ms
            ref = r[0, 0]
            big = ref > 1e-3 * ref.max()
            if big.any():
                err = max(err, float((np.abs(r4m[0, i][big] - ref[big]) / ref[big]).max()))
        fp64_4ph_ms = f_ms * quartets / counts[sample].sum()
        out.update({"fp64_4ph_ms_extrapolated": fp64_4ph_ms, "fp64_sample_q0": [int(i) + 1 for i in sample],
                    "fp64_sample_ms": f_ms, "fp64_4ph_over_v4tc": fp64_4ph_ms / v4_ms if v4_ms else None,
                    "rate4_max_rel_err_vs_fp64_sample": err,
                    "fp64_note": "FP64 four-phonon time of the whole leg extrapolated from the sampled q0 by their "
                                 "quartet counts; rate errors over the sampled q0"})
    ctx.close()
    return out


def surrogate_c5_leg(torch, train_mesh=12, mesh=20, frac=0.25, members=3):
    """Surrogate-screened four-phonon kappa: a network ensemble (5-128-128-128-1, SiLU, trained on
    the GPU with the library's kernels on the exact rates of a train_mesh^3 mesh at 300 and 900 K)
    ranks the (q0, branch) blocks of the mesh^3 mesh; exact tensor-core V4 runs for the top `frac`
    of them and the prediction (BF16 tensor-core inference) stands in elsewhere.  Compared with the
    full exact four-phonon kappa on the same GPU, and with a network-free estimate
    (log r4 = a + b log r3 fitted on the same training rates) given the same exact budget."""
    from spring_b200 import surrogate as SG
    from spring_b200 import synthetic as S
    from spring_b200.api import from_crystal
    cr = S.build("rocksalt2", fc4=True)
    T = [300.0, 900.0]

    def mesh_data(N):
        ctx, info = from_crystal(cr, (N, N, N), T, with_fc4=True)
        ctx.set_precision("bf16x3")
        ctx.reset_linewidths()
        lw3 = ctx.linewidth3(1, ctx.nq0, "gauss", SIGMA)[0]
        ph = ctx.get_phonons(1)
        q = ((cr.G / N) @ info["irr_q_pnt_int"].T.astype(float)).T
        X = [SG.mode_features(ph["omega"], ph["grp_vel"], 2.0 * lw3[t], q) for t in range(len(T))]
        return ctx, info, lw3, ph, X

    ct, _, lw_t, _, X_t = mesh_data(train_mesh)
    r_t, train_exact_ms = _ev_ms(torch, lambda: ct.linewidth4(1, ct.nq0, "gauss", SIGMA))
    X_all = np.concatenate(X_t)
    y_all = r_t.reshape(-1)
    m = (y_all > 0) & (X_all[:, 2] > 0)
    sur = SG.Surrogate(ct, seed=1, members=members)
    _, train_ms = _ev_ms(torch, lambda: sur.fit(X_all[m], np.log(y_all[m]), epochs=300, batch=64, lr=2e-3))
    pl = SG.PowerLaw().fit(X_all[:, 2], y_all)

    c, info, lw3, ph, X = mesh_data(mesh)
    quartets = sum(c.count4(i + 1)[0] for i in range(c.nq0))
    r_ex, exact_ms = _ev_ms(torch, lambda: c.linewidth4(1, c.nq0, "gauss", SIGMA))

    def predict():
        out = [sur.predict(X[t], bf16=True) for t in range(len(T))]
        return (np.exp(np.array([o[0] for o in out])).reshape(len(T), c.nq0, -1),
                np.array([o[1] for o in out]).reshape(len(T), c.nq0, -1))
    (pred, spread), pred_ms = _ev_ms(torch, predict)
    pred_pl = np.array([pl.predict(2.0 * lw3[t]) for t in range(len(T))])
    w = np.array([SG.kappa_weight(ph["omega"], ph["nbe"][t], ph["grp_vel"], info["multiplicity"]) for t in range(len(T))])

    def kappa(r4):
        c.set_linewidths(lw3 + 0.5 * r4)
        return c.kappa_rta(info["Rxyz"])

    def screened(p, unc):
        sc = np.max([SG.mode_scores(2.0 * lw3[t], p[t], w[t], None if unc is None else unc[t])
                     for t in range(len(T))], axis=0)
        masks, sel = SG.select_modes(sc, frac)
        (r, _), ms = _ev_ms(torch, lambda: SG.screened_rates4(c, p, masks, sigma=SIGMA))
        return r, ms

    r_net, scr_ms = screened(pred, spread)
    r_pl, _ = screened(pred_pl, None)
    k_ex, k_net, k_pl = kappa(r_ex), kappa(r_net), kappa(r_pl)
    err = lambda k: [float(np.abs(_kdiag(k[t]) / _kdiag(k_ex[t]) - 1).max()) for t in range(len(T))]
    ok = (r_ex > 0) & (np.stack([x[:, 2] for x in X]).reshape(r_ex.shape) > 0)
    out = {"train_mesh": [train_mesh] * 3, "mesh": [mesh] * 3, "temperatures": T, "irreducible_q0": int(c.nq0),
           "quartets": int(quartets), "fraction_exact_blocks": frac, "ensemble_members": members,
           "exact_ms": exact_ms, "screened_ms": scr_ms + pred_ms, "exact_over_screened": exact_ms / (scr_ms + pred_ms),
           "screened_exact_part_ms": scr_ms, "prediction_ms": pred_ms, "train_ms": train_ms,
           "train_exact_rates_ms": train_exact_ms,
           "kappa_exact_diag": [_kdiag(k).tolist() for k in k_ex],
           "kappa_rel_err_screened": err(k_net), "kappa_rel_err_network_free_same_budget": err(k_pl),
           "median_abs_log_err_prediction": float(np.median(np.abs(np.log(pred[ok]) - np.log(r_ex[ok])))),
           "v4_arithmetic": "bf16x3",
           "what": "blocks = (irreducible q0, branch s0) of the quartet sum; ranked by predicted kappa impact x "
                   "(1 + ensemble spread of the log prediction); exact V4 (spring_linewidth4_modes) on the top "
                   "fraction, network (BF16 tensor-core inference) elsewhere"}
    c.close()
    ct.close()
    return out


def bte_c2_leg(torch, ctx, mesh):
    """Iterative (non-RTA) kappa of the benchmark context (mesh^3, T = 100/300/700 K) to the
    tolerance 1e-6, in the Gaussian operator form (delta weights of width SIGMA).  FP64 operator:
    first call (time-reversal pairs, operator build with the FP64 V3 of every pair, the entries
    inside the delta window, row sort, iterations), then the iterations alone on the kept operator,
    and the operator pass's achieved HBM bandwidth.  Then the same with the operator entries from
    the BF16x3 tensor-core pass (the iterations, deltas and occupations stay FP64), against the
    FP64 operator's kappa."""
    prec = ctx.precision
    ctx.set_precision("fp64")
    r1, first_ms = _ev_ms(torch, lambda: ctx.kappa_iter_gauss(SIGMA, eps_k=1e-6))
    r2, iter_ms = _ev_ms(torch, lambda: ctx.kappa_iter_gauss(SIGMA, eps_k=1e-6))
    ctx.set_profiling(True)
    ctx.kappa_iter_gauss(SIGMA, eps_k=1e-6)
    rows_ms, rows_n = ctx.kernel_time("k_bteg_rows<dF>")
    ctx.set_profiling(False)
    E = r2["entries"]
    n_iter = int(r2["iters"].sum())
    # per operator pass: (k1, k2) and the coefficient of every entry, the row offsets, dF out
    ntr_rows = (mesh ** 3 // 2 + 8) * 6
    bytes_pass = E * (8 + 8) + ntr_rows * (4 + 24)
    per_ms = rows_ms / rows_n if rows_n else None
    peaks = measured_peaks()
    ctx.set_precision("bf16x3")
    t1, tc_first_ms = _ev_ms(torch, lambda: ctx.kappa_iter_gauss(SIGMA, eps_k=1e-6))
    t2, tc_iter_ms = _ev_ms(torch, lambda: ctx.kappa_iter_gauss(SIGMA, eps_k=1e-6))
    ctx.set_precision(prec)
    kerr = float(np.abs(t1["kappa"] - r2["kappa"]).max() / np.abs(r2["kappa"]).max())
    kerr0 = float(np.abs(t1["kappa_rta"] - r2["kappa_rta"]).max() / np.abs(r2["kappa_rta"]).max())
    tc = {"first_call_ms": tc_first_ms, "iterations_only_ms": tc_iter_ms, "operator_entries": t1["entries"],
          "iterations": t1["iters"].tolist(), "first_call_fp64_over_this": first_ms / tc_first_ms,
          "kappa_max_rel_diff_vs_fp64_operator": kerr, "kappa_rta_max_rel_diff_vs_fp64_operator": kerr0,
          "kappa_diag": [_kdiag(k).tolist() for k in t1["kappa"]],
          "what": "operator entries from the tensor-core V3 pass (BF16x3) over the time-reversal pairs, "
                  "window and cuts as in FP64; the same FP64 iterations"}
    return {"mesh": [mesh] * 3, "temperatures": TEMPS, "sigma_rad_ps": SIGMA, "eps_k": 1e-6,
            "tensor_core_operator": tc,
            "operator_entries": E, "pairs": r2["pairs"], "iterations": r2["iters"].tolist(),
            "converged": bool((r2["iters"] <= 1000).all()),
            "first_call_ms": first_ms, "iterations_only_ms": iter_ms,
            "ms_per_iteration": iter_ms / max(n_iter, 1),
            "operator_pass_ms": per_ms,
            "operator_pass_gbs": bytes_pass / (per_ms * 1e-3) / 1e9 if per_ms else None,
            "operator_pass_frac_hbm": (bytes_pass / (per_ms * 1e-3) / 1e9) / peaks["hbm_gbs"] if per_ms else None,
            "kappa_diag": [_kdiag(k).tolist() for k in r2["kappa"]],
            "kappa_rta_diag": [_kdiag(k).tolist() for k in r2["kappa_rta"]],
            "same_as_first_call": bool(np.array_equal(r1["kappa"], r2["kappa"])),
            "what": "spring_kappa_iter_gauss: F <- F0 + tau sum over both channels until max|dkappa| < 1e-6; "
                    "operator = one entry per pair and mode triple inside the exp(-40) window, kept in HBM"}


BATCH_CELLS = (("rocksalt2", 12), ("rocksalt2", 16), ("rocksalt2", 20), ("rocksalt8", 8), ("rocksalt8", 10))
# Gamma-X-W-K-Gamma-L in the fractional reciprocal basis, 200 points
PATH_NODES = np.array([[0.0, 0.0, 0.0, 0], [0.0, 0.5, 0.5, 50], [0.25, 0.625, 0.625, 25], [0.375, 0.75, 0.375, 18],
                       [0.0, 0.0, 0.0, 53], [0.5, 0.5, 0.5, 54]])


def batched_leg(torch, steps=3):
    """Batched uneven workload: the 2-atom cell at 12^3/16^3/20^3 and the 8-atom cubic cell at
    8^3/10^3, 9 temperatures (100-900 K), Gaussian three-phonon linewidths of every irreducible q0
    of all five in one batch run with the autotuned configuration; then
    Gaussian linewidths at 200 path points (Gamma-X-W-K-Gamma-L) on the 2-atom 12^3 context.
    Compared with each context's own spring_linewidth3 call (FP64) one after the other."""
    from spring_b200 import synthetic as S
    from spring_b200.api import Batch, from_crystal
    temps = [100.0 * k for k in range(1, 10)]
    cells = []
    evals = 0
    for name, N in BATCH_CELLS:
        cr = S.build(name)
        ctx, info = from_crystal(cr, (N, N, N), temps)
        npairs = sum(ctx.enumerate3(i + 1)[2][0] for i in range(ctx.nq0))
        evals += npairs * cr.ndof ** 3
        cells.append((name, N, ctx, npairs))

    def ev_ms(fn):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        torch.cuda.synchronize()
        e0.record()
        fn()
        e1.record()
        torch.cuda.synchronize()
        return e0.elapsed_time(e1)

    def separate():
        for _, _, ctx, _ in cells:
            ctx.reset_linewidths()
            ctx.linewidth3(1, ctx.nq0, "gauss", SIGMA, want=False)
        for _, _, ctx, _ in cells:
            ctx.synchronize()

    separate()
    sep = min(ev_ms(separate) for _ in range(steps))
    ref = [ctx.get_linewidths() for _, _, ctx, _ in cells]
    b = Batch()
    for _, _, ctx, _ in cells:
        b.add_linewidth3(ctx, 1, ctx.nq0, SIGMA)
    b.run()
    cfg, tuned_ms, tried = b.tune()
    for _, _, ctx, _ in cells:
        ctx.reset_linewidths()
    b.run()  # capture with the tuned configuration
    err = max(float(np.abs(b.result(k)[0] - ref[k]).max() / np.abs(ref[k]).max()) for k in range(len(cells)))
    runs = []
    for _ in range(steps):
        b.run()
        runs.append(b.result(0)[2])
    batch_ms = min(runs)
    ctx12 = cells[0][2]
    q, _, z = ctx12.path_qpoints(PATH_NODES)
    ctx12.linewidth_path(q, z, delta="gauss", sigma=SIGMA)
    path_ms = min(ev_ms(lambda: ctx12.linewidth_path(q, z, delta="gauss", sigma=SIGMA)) for _ in range(steps))
    b.close()
    # Mixed precision: the two-atom contexts on BF16x3 (tensor-core pass), the 8-atom ones on FP64;
    # single calls plus the path call, against one batch holding all of it (path points in its graph).
    for name, _, ctx, _ in cells:
        if name == "rocksalt2":
            ctx.set_precision("bf16x3")
    path_lw = [None]

    def separate_mixed():
        for _, _, ctx, _ in cells:
            ctx.reset_linewidths()
            ctx.linewidth3(1, ctx.nq0, "gauss", SIGMA, want=False)
        path_lw[0] = ctx12.linewidth_path(q, z, delta="gauss", sigma=SIGMA)[0]
        for _, _, ctx, _ in cells:
            ctx.synchronize()

    separate_mixed()
    sep_mixed = min(ev_ms(separate_mixed) for _ in range(steps))
    ref_m = [ctx.get_linewidths() for _, _, ctx, _ in cells]
    bm = Batch()
    for _, _, ctx, _ in cells:
        bm.add_linewidth3(ctx, 1, ctx.nq0, SIGMA)
    ip = bm.add_path(ctx12, q, z, SIGMA)
    bm.set_config(*cfg)
    runs_m = []
    for _ in range(steps + 1):
        for _, _, ctx, _ in cells:
            ctx.reset_linewidths()
        bm.run()
        runs_m.append(bm.result(0)[2])
    batch_mixed = min(runs_m[1:])
    err_m = max(float(np.abs(bm.result(k)[0] - ref_m[k]).max() / np.abs(ref_m[k]).max()) for k in range(len(cells)))
    lwp = bm.path_result(ip)[0]
    err_p = float(np.abs(lwp - path_lw[0]).max() / np.abs(path_lw[0]).max())
    bm.close()
    for _, _, ctx, _ in cells:
        ctx.close()
    nq12 = 12 ** 3
    path_evals = int(len(q)) * nq12 * 6 ** 3
    return {"workloads": [f"{n}-{N}^3" for n, N, _, _ in cells], "temperatures": temps,
            "pairs": [int(p) for *_, p in cells], "evals_per_T": int(evals),
            "batch_ms": batch_ms, "separate_calls_ms": sep, "separate_over_batch": sep / batch_ms,
            "evals_per_s_batch": evals / (batch_ms * 1e-3),
            "max_rel_diff_vs_separate": err,
            "tuned_config": {"two_atom_layout": cfg[0], "ctas_per_sm": cfg[1], "s0_block_ndof24": cfg[2],
                             "items_per_step": cfg[3]},
            "tuning": {"configs_tried": tried, "best_trial_ms": tuned_ms},
            "path_points": int(len(q)), "path_ms": path_ms, "path_mesh": [12, 12, 12],
            "what": "one FP64 batch run over all five workloads, each cell's own kernel after the graph; path points "
                    "on the 12^3 context afterwards",
            "mixed": {"batch_ms": batch_mixed, "separate_calls_ms": sep_mixed,
                      "separate_over_batch": sep_mixed / batch_mixed,
                      "evals_per_s_batch": (evals + path_evals) / (batch_mixed * 1e-3),
                      "evals_per_s_separate": (evals + path_evals) / (sep_mixed * 1e-3),
                      "path_evals_per_T": path_evals,
                      "max_rel_diff_vs_separate": err_m, "path_max_rel_diff_vs_separate": err_p,
                      "what": "two-atom workloads on BF16x3 through the tensor-core pass (the kernel of "
                              "spring_linewidth3), 8-atom workloads in their FP64 matrix kernel, the 200 "
                              "path points inside the batch's CUDA graph; against each context's own call "
                              "with the same precision plus the path call, one after the other"}}


def run_ours(args):
    import torch
    import torch.distributed as dist
    from spring_b200 import distributed as DD
    from spring_b200 import synthetic as S
    from spring_b200.api import Context

    world = int(os.environ.get("WORLD_SIZE", "1"))
    rank = int(os.environ.get("RANK", "0"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    torch.cuda.set_device(local)
    if world > 1:
        import datetime
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))
    dev = torch.device("cuda", local)
    stream = torch.cuda.Stream(device=dev)

    cr = S.build("rocksalt2")
    W, Rxyz = S.point_group(cr)
    mesh = (args.mesh,) * 3
    ctx = Context(cr.nbasis, mesh, len(TEMPS), device=local)
    ctx.set_stream(stream.cuda_stream)
    ctx.set_crystal(cr.latvec, cr.mass)
    ctx.set_fc2(cr.fc2_atm_num, cr.fc2_atm_indx, cr.fc2)
    ctx.set_fc3(cr.fc3_atm_num, cr.fc3_atm_indx, cr.fc3)
    ctx.make_mesh(want=False)
    irr = ctx.find_irr_q(W)
    nq0 = ctx.nq0
    ctx.compute_phonons(TEMPS)
    enum = [ctx.enumerate3(i + 1) for i in range(nq0)]
    counts = np.array([e[2][0] for e in enum])
    lo, hi = DD.partition_by_cost(counts, world, rank)
    my_pairs = int(counts[lo:hi].sum())
    del enum
    evals_total = int(counts.sum()) * cr.ndof ** 3
    flops_pair = algorithmic_flops_per_pair(cr.ndof, cr.fc3_atm_num)
    flush = torch.empty(256 << 20, dtype=torch.uint8, device=dev)
    kap_dev = torch.zeros(len(TEMPS), 9, dtype=torch.float64, device=dev)

    def step():
        ctx.compute_phonons(TEMPS)
        ctx.prepare3()
        ctx.reset_linewidths()
        if hi > lo:
            ctx.linewidth3(lo + 1, hi - lo, delta=DELTA, sigma=SIGMA, want=False)
        if world > 1:
            ctx.set_linewidths(DD.allreduce_linewidths(ctx.get_linewidths()[:, lo:hi], lo, hi, nq0, device=dev))
        ctx.kappa_rta(Rxyz, want=False)

    def timed(prec, clocks=None):
        """K steps of the whole path with V3 in `prec`: (ms per step, launches, kernel times, lw, kappa)."""
        ctx.set_precision(prec)
        for _ in range(args.warmup):
            step()
        torch.cuda.synchronize()
        if world > 1:
            dist.barrier()
        if clocks:
            clocks.start()
            clocks.begin()
        ctx.set_profiling(True)
        l0 = ctx.kernel_launches()
        times = []
        for _ in range(args.steps):
            flush.zero_()           # L2 flush, outside the timed events
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            step()
            e1.record(stream)
            if clocks:
                clocks.sample()     # while the step's kernels run
            e1.synchronize()
            times.append(e0.elapsed_time(e1))
        torch.cuda.synchronize()
        launches = ctx.kernel_launches() - l0
        kt = {k: ctx.kernel_time(k) for k in ("k_v3tc<", "k_v3s", "k_v3<", "k_phonons", "k_tc_tab",
                                              "k_kappa")}
        ctx.set_profiling(False)
        if clocks:
            clocks.end()
        clk = clocks.stop() if clocks else None
        ms = float(np.sum(times)) / args.steps
        if world > 1:
            t = torch.tensor([ms], dtype=torch.float64, device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            ms = float(t.item())
            dist.barrier()
        lw = ctx.get_linewidths()
        kap = ctx.kappa_rta(Rxyz)
        return ms, launches, kt, lw, kap, clk

    with torch.cuda.stream(stream):
        ms64, _, kt64, lw64, kap64, _ = timed("fp64")
        # the FP64 path on the pairs that the delta-window pre-screen keeps (the same pre-screen as
        # the tensor-core path's): the strongest FP64 baseline
        from spring_b200 import _lib as L
        ctx.set_option(L.SPRING_OPT_FP64_PRESCREEN, 1)
        ms64p, _, kt64p, lw64p, _, _ = timed("fp64")
        ctx.set_option(L.SPRING_OPT_FP64_PRESCREEN, 0)
        big64 = lw64 > 1e-3 * lw64.max(axis=(1, 2), keepdims=True)
        lw64p_err = float((np.abs(lw64p - lw64)[big64] / lw64[big64]).max())
        clocks = Clocks(local, pci_bus_id(torch, local))
        ms, launches, kt, lw_p, kap_p, clk = timed(args.precision, clocks)
        tc_tiles_run, tc_pairs_run = ctx.tc_stats() if args.precision != "fp64" else (0, 0)
        big = lw64 > 1e-3 * lw64.max(axis=(1, 2), keepdims=True)
        lw_err = float((np.abs(lw_p - lw64)[big] / lw64[big]).max())
        diag = [0, 4, 8]
        k_err = float(np.abs(kap_p[:, diag] / kap64[:, diag] - 1.0).max())
        main_kernel = "k_v3tc<" if args.precision != "fp64" else "k_v3s"
        v3_ms, v3_n = kt[main_kernel] if kt[main_kernel][1] else kt["k_v3<"]

        # end to end through the public API: host inputs, pinned, copied every step
        pin = lambda a: torch.from_numpy(np.ascontiguousarray(a)).pin_memory().numpy()
        h_lat, h_mass = pin(cr.latvec), pin(cr.mass)
        h_f2 = (pin(cr.fc2_atm_num), pin(cr.fc2_atm_indx), pin(cr.fc2))
        h_f3 = (pin(cr.fc3_atm_num), pin(cr.fc3_atm_indx), pin(cr.fc3))
        h_W = pin(W)
        h_lw = pin(np.zeros((len(TEMPS), max(hi - lo, 1), cr.ndof)))
        h_kap = pin(np.zeros((len(TEMPS), 9)))
        nq = int(np.prod(mesh))
        h2d = (h_lat.nbytes + h_mass.nbytes + sum(a.nbytes for a in h_f2) + sum(a.nbytes for a in h_f3) + h_W.nbytes
               + 8 * len(TEMPS))
        d2h = (4 * nq + 12 * nq          # irreducible map and grid addresses (find_irr_q)
               + 8 + 4 * (nq0 + 1)       # pair count and offsets (prepare3)
               + h_lw.nbytes + h_kap.nbytes)

        def step_e2e():
            ctx.set_crystal(h_lat, h_mass)
            ctx.set_fc2(*h_f2)
            ctx.set_fc3(*h_f3)
            ctx.make_mesh(want=False)
            ctx.find_irr_q(h_W)
            ctx.compute_phonons(TEMPS)
            ctx.prepare3()
            ctx.reset_linewidths()
            if hi > lo:
                ctx.linewidth3(lo + 1, hi - lo, delta=DELTA, sigma=SIGMA, out=h_lw)
            if world > 1:
                ctx.set_linewidths(DD.allreduce_linewidths(h_lw[:, : hi - lo], lo, hi, nq0, device=dev))
            ctx.kappa_rta(Rxyz, out=h_kap)

        ctx.set_precision(args.precision)
        for _ in range(max(1, args.warmup)):
            step_e2e()
        torch.cuda.synchronize()
        et = []
        for _ in range(args.steps):
            flush.zero_()
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record(stream)
            step_e2e()
            e1.record(stream)
            e1.synchronize()
            et.append(e0.elapsed_time(e1))
        e2e_ms = float(np.mean(et))
        if world > 1:
            t = torch.tensor([e2e_ms], dtype=torch.float64, device=dev)
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
            e2e_ms = float(t.item())

    peak = fp64_peak_tflops(torch) if rank == 0 else None
    legs = set(x.strip() for x in args.legs.split(",")) if rank == 0 and world == 1 else set()
    four = fourph_c3_leg(torch, args.mesh4, fp64=args.c3_fp64) if "c3" in legs else None
    sur = surrogate_c5_leg(torch) if "c5" in legs else None
    batched = batched_leg(torch) if "c4" in legs else None
    bte = bte_c2_leg(torch, ctx, mesh[0]) if "c2" in legs else None
    cpu = None
    oracle_check = None
    if rank == 0 and world == 1 and not args.no_cpu_baseline:
        ph_grid, ph_irr = ctx.get_phonons(0), ctx.get_phonons(1)
        sample = [1, nq0 // 2, nq0 - 1]
        lw_orc = {}
        v, dt, thr = cpu_baseline(cr, mesh, TEMPS, ph_grid, ph_irr, irr["irr_q_pnt_int"], sample, "", lw_orc)
        cpu = {"value": v, "unit": "evals/s", "cores": thr, "kind": "port",
               "sample": f"{len(sample)} of {nq0} irreducible q0: enumeration, V3 in the reference loop order, "
                         f"Gaussian sum at 3 T; phonons excluded ({dt:.1f} s)"}
        # parity at the full size: the measured path's and the FP64 path's linewidths of the sampled q0
        # against the oracle's (same device phonons), every mode above 1e-3 of the q0's largest
        def max_rel(lw_gpu):
            e = 0.0
            for i0, ref in lw_orc.items():
                g = lw_gpu[:, i0 - lo] if lo <= i0 < hi else None
                if g is None:
                    continue
                big = ref > 1e-3 * ref.max()
                e = max(e, float((np.abs(g[big] - ref[big]) / ref[big]).max()))
            return e
        oracle_check = {"q0": [int(i) for i in sample], "mesh": list(mesh),
                        "lw_max_rel_err_measured_path": max_rel(lw_p),
                        "lw_max_rel_err_fp64_path": max_rel(lw64),
                        "what": "GPU linewidths of these irreducible q0 at every temperature against the oracle "
                                "(CPU restatement of the reference loops, FP64) on the device phonons"}
    if rank == 0:
        value = evals_total / (ms * 1e-3)
        v3_per_launch = v3_ms / max(v3_n, 1)
        fp64_kernel_ms = kt64["k_v3s"][0] / max(kt64["k_v3s"][1], 1) if kt64["k_v3s"][1] else None
        if args.precision == "fp64":
            achieved = flops_pair * my_pairs / (v3_per_launch * 1e-3) / 1e12 if v3_n else None
            roof = {"kernel": "k_v3s<gauss>", "bound": "fp64", "achieved": achieved, "peak": peak, "unit": "TFLOP/s",
                    "frac": (achieved / peak) if (achieved and peak) else None, "traffic": None,
                    "peak_source": "cuBLAS FP64 GEMM 8192^3 measured in this run (MEASURED_PEAKS.json holds no FP64)"}
        else:
            passes = 3 if args.precision == "bf16x3" else 1
            issued = tc_issued_flops_per_tile(passes) * tc_tiles_run
            algo = flops_pair * tc_pairs_run
            sec = v3_per_launch * 1e-3
            achieved = algo / sec / 1e12 if v3_n else None
            pk = measured_peaks()
            roof = {"kernel": f"k_v3tc<{args.precision}>", "bound": "tensor", "achieved": achieved,
                    "peak": pk["bf16_tflops"], "unit": "TFLOP/s",
                    "frac": (achieved / pk["bf16_tflops"]) if achieved else None,
                    "traffic": TC_DRAM_BYTES_PER_TILED_PAIR * tc_pairs_run,
                    "pairs_tiled": tc_pairs_run, "tiles": tc_tiles_run, "pairs_all": my_pairs,
                    "peak_source": pk["source"],
                    "algorithmic_flops_per_launch": algo,
                    "issued_mma_tflops": issued / sec / 1e12 if v3_n else None,
                    "issued_flops_per_launch": issued,
                    "traffic_note": "dram read + write bytes per tiled pair from an ncu capture of the 16^3 "
                                    "launch, scaled by the tiled pairs of this launch",
                    "note": "achieved = algorithmic V3 flops (42336 per pair) x the pairs the kernel computes "
                            "(pairs_tiled: those with a mode triple inside the delta window; the pre-screen "
                            "drops the others, whose every weight is below the exp(-40) cut) / kernel time; "
                            "issued_mma_tflops counts the tcgen05 MMAs as issued (M128 N48 K16, padding "
                            "included) over its tiles.  The kernel is bound by its epilogue (accumulator "
                            "reads, window masks, |Phi|^2 of the active triples and their FP64 delta/rate "
                            "evaluation), not by the tensor pipe"}
        roof.update({"kernel_ms_per_launch": v3_per_launch, "kernel_share_of_step": v3_per_launch / ms,
                     "algorithmic_fp64_flops_per_pair": flops_pair})
        line = {"metric": METRIC, "value": value, "unit": "evals/s", "n_gpus": world, "steps": args.steps,
                "warmup": args.warmup, "ms_per_step": ms, "higher_is_better": True, "scaling": "strong",
                "vs_baseline": None, "dtype": args.precision, "data": "synthetic",
                "config": {"workload": WORKLOAD, "mesh": list(mesh), "irreducible_q0": nq0,
                           "pairs": int(counts.sum()), "temperatures": TEMPS, "sigma_rad_ps": SIGMA,
                           "delta": DELTA, "parallelism": f"q0-partition x{world}",
                           "v3_arithmetic": args.precision,
                           "fp64_parts": "phonons, deltas, rates and kappa",
                           "l2": "256 MiB buffer written between timed steps, outside the events"},
                "time_to_kappa": {"ms": ms, "fp64_gpu_ms": ms64, "fp64_gpu_over_this": ms64 / ms,
                                  "fp64_prescreened_gpu_ms": ms64p, "fp64_prescreened_over_this": ms64p / ms,
                                  "fp64_prescreened_lw_max_rel_diff_vs_fp64": lw64p_err,
                                  "kappa_max_rel_err_vs_fp64": k_err, "linewidth_max_rel_err_vs_fp64": lw_err,
                                  "fp64_v3_kernel_ms": fp64_kernel_ms,
                                  "what": "one step = phonons + pairs + linewidths at 3 T + RTA kappa; errors over "
                                          "every mode with a linewidth above 1e-3 of the largest, kappa diagonal"},
                "fp64_path": {"value": evals_total / (ms64 * 1e-3), "unit": "evals/s", "ms_per_step": ms64},
                "fourph_c3": four,
                "surrogate_c5": sur,
                "batched": batched,
                "bte_c2": bte,
                "roofline": roof,
                "cpu_baseline": cpu,
                "oracle_check_24": oracle_check,
                "e2e": {"value": evals_total / (e2e_ms * 1e-3), "unit": "evals/s", "ms_per_step": e2e_ms,
                        "h2d_bytes_per_step": int(h2d), "d2h_bytes_per_step": int(d2h)},
                "gpu_launches": int(launches),
                "clocks": clk}
        print(json.dumps(line), flush=True)
    ctx.close()
    if world > 1:
        dist.barrier()
        dist.destroy_process_group()
    return 0


def main():
    args = parse()
    if args.impl == "reference":
        return run_reference(args)
    return run_ours(args)


if __name__ == "__main__":
    sys.exit(main())
