#!/usr/bin/env python
"""Benchmark of the quantised matmul hot path on B200.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl ours|reference]

Workload: Q4_K prefill GEMM, M = 8192 tokens x K = 5120 -> N = 17408, synthetic seeded data
with the configured distributions.  One step = quantise the f32 activations per 32-block + the GEMM.
  value   tokens/s with the f32 activations already in HBM (CUDA events, K steps, max over ranks)
  e2e     the same through the host-buffer C-ABI call (izb_matmul_host): pinned host activations in, f32 outputs back,
          both copies inside the timed region
  roofline  the dominant kernel (the tcgen05 GEMM): 2*M*N*K integer ops per launch / its CUDA-event duration, against the
          measured dense 16-bit tensor peak (the MMA kind the kernel issues), plus the fraction of the nominal int8 peak
  cpu_baseline  the reference's own CPU code (tools/ref_forward.cpp matmul via oracle/_ref) on a bounded sample
With --gpus N > 1 (launched by torchrun) the weight rows are split over the ranks as the reference's tensor-parallel
mode splits a gate/up projection (column parallel, no exchange): strong scaling of the same GEMM.
`--impl reference` times the reference's CPU implementation on the host cores for the same metric.
"""
from __future__ import annotations

import argparse
import json
import os
import subprocess
import sys
import tempfile
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

M, N, K = 8192, 17408, 5120
QT = 12
SEED = 20261125
WORKLOAD = "config2: Q4_K prefill GEMM M=8192 N=17408 K=5120 (quantiser + GEMM per step: one izb_quant_matmul call)"
NOMINAL_INT8_TOPS = 4500.0
NCU_TRAFFIC_BYTES_PER_TILE = (159.7e6 + 121.0e6) / (16 * 136)       # gemm_fold: ncu capture of 16 x 136 tiles of 128 x 128


def peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return d["hbm_gbs"], d["bf16_tflops"], d["bf16_tflops_sustained"], "measured"
    return 6650.0, 1590.0, 1400.0, "fallback"


def _rel(got, ref) -> float:
    """The reference's error form (bench/gemv_bench.cpp:199-214): max|got - ref| / max|ref|."""
    return float(np.abs(got.astype(np.float64) - ref.astype(np.float64)).max() / max(1e-30, float(np.abs(ref).max())))


class ClockSampler:
    """SM clock and throttle reasons sampled while the timed region runs: NVML read-only queries from a thread every
    few milliseconds (nvidia-smi every 100 ms when the NVML binding is missing)."""

    Q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, gpu_index: int, pci_bus_id: str | None = None):
        self.idx, self.pci, self.rows, self.proc = gpu_index, pci_bus_id, [], None
        self.sm, self.mx, self.reasons, self.stop_flag, self.thread, self.source = [], [], set(), False, None, None

    def _nvml_loop(self, nv, h):
        names = (("hw_slowdown", nv.nvmlClocksEventReasonHwSlowdown), ("hw_thermal_slowdown", nv.nvmlClocksEventReasonHwThermalSlowdown),
                 ("sw_thermal_slowdown", nv.nvmlClocksEventReasonSwThermalSlowdown), ("sw_power_cap", nv.nvmlClocksEventReasonSwPowerCap))
        while not self.stop_flag:
            try:
                self.sm.append(float(nv.nvmlDeviceGetClockInfo(h, nv.NVML_CLOCK_SM)))
                r = nv.nvmlDeviceGetCurrentClocksEventReasons(h)
                for n, bit in names:
                    if r & bit:
                        self.reasons.add(n)
            except Exception:
                break
            time.sleep(0.004)

    def start(self):
        try:
            import pynvml as nv
            nv.nvmlInit()
            h = nv.nvmlDeviceGetHandleByPciBusId(self.pci.encode()) if self.pci else nv.nvmlDeviceGetHandleByIndex(self.idx)
            self.mx = [float(nv.nvmlDeviceGetMaxClockInfo(h, nv.NVML_CLOCK_SM))]
            self.source = "nvml"
            self.thread = threading.Thread(target=self._nvml_loop, args=(nv, h), daemon=True)
            self.thread.start()
            return
        except Exception:
            self.source = "nvidia-smi"
        try:
            self.proc = subprocess.Popen(["nvidia-smi", f"--query-gpu={self.Q}", "--format=csv,noheader,nounits", "-lms", "100",
                                          "-i", str(self.idx)], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            threading.Thread(target=self._read, daemon=True).start()
        except OSError:
            self.proc = None

    def _read(self):
        for line in self.proc.stdout:
            self.rows.append([c.strip() for c in line.split(",")])

    def stop(self) -> dict:
        if self.thread:
            self.stop_flag = True
            self.thread.join(timeout=2)
            return {"sm_mhz": float(np.median(self.sm)) if self.sm else None, "sm_max_mhz": max(self.mx) if self.mx else None,
                    "reasons": sorted(self.reasons), "samples": len(self.sm), "source": self.source}
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=2)
            except Exception:
                pass
        sm = [float(r[1]) for r in self.rows if len(r) >= 9 and r[1].replace(".", "").isdigit()]
        mx = [float(r[2]) for r in self.rows if len(r) >= 9 and r[2].replace(".", "").isdigit()]
        reasons = set()
        for r in self.rows:
            if len(r) >= 9:
                for name, v in zip(("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"), r[5:9]):
                    if v.lower().startswith("active"):
                        reasons.add(name)
        return {"sm_mhz": float(np.median(sm)) if sm else None, "sm_max_mhz": max(mx) if mx else None,
                "reasons": sorted(reasons), "samples": len(sm), "source": self.source}


def cpu_baseline(seconds_target: float = 15.0) -> dict:
    """tok/s of the reference's CPU path on a sample of the workload: M_s tokens x N_s weight rows x full K, scaled to the
    full N.  kind "reference" = tools/ref_forward.cpp matmul() (oracle/_ref); "port" = the C restatement."""
    from arcinferzero_b200 import synth as S
    from oracle import oracle as O
    Ms, Ns = 64, 1024
    w = S.make_weight(QT, Ns, K, SEED)
    x = S.make_act(Ms, K, SEED + 1)
    # Every host core the process may use, set explicitly: a launcher (torch.distributed.run) exports OMP_NUM_THREADS=1,
    # which would otherwise time the reference on one thread.
    cores = len(os.sched_getaffinity(0)) if hasattr(os, "sched_getaffinity") else (os.cpu_count() or 1)
    cores = O.set_threads(cores)
    if O.ref() is not None:
        kind = "reference"
        d = tempfile.mkdtemp()
        path = os.path.join(d, "s.gguf")
        S.write_gguf(path, {"w": (QT, w, Ns, K)})

        def run(ms):
            return O.ref_forward_matmul(path, "w", x[:ms] if ms <= Ms else np.tile(x, (ms // Ms, 1)), Ns, threads=cores)
    else:
        kind = "port"

        def run(ms):
            xx = x[:ms] if ms <= Ms else np.tile(x, (ms // Ms, 1))
            aq, asc, _ = O.quantize_act(xx)
            return O.matmul(QT, w, K, aq, asc, xx.shape[0], "gemm")
    run(8)
    t0 = time.perf_counter()
    run(Ms)
    t1 = time.perf_counter() - t0
    reps = int(min(128, max(1, seconds_target / max(t1, 1e-3))))
    ms = Ms * reps
    t0 = time.perf_counter()
    run(ms)
    t = time.perf_counter() - t0
    tok_s = ms / (t * (N / Ns))
    return {"value": tok_s, "unit": "tok/s", "cores": cores, "kind": kind,
            "sample": f"{ms} tokens x {Ns} of {N} weight rows x K={K} in {t:.2f} s, scaled by N/{Ns}"}


def gemv_section(izb, torch, hbm_peak: float, peak_src: str, lite: bool = False) -> list:
    """Decode GEMV: batch 1 and 2, K = 5120; Q4_K N = 5120 and 17408, Q8_0 N = 151936.
    Each launch reads a different copy of the weights (enough copies to exceed the 126 MB L2), so the bytes come from
    HBM; GB/s = (weight bytes + activation bytes + output bytes) / mean launch time over the timed launches."""
    from arcinferzero_b200 import synth as S
    out = []
    # config 3's three matrices, then the down-projection shape of the same model (long rows: not in config 3)
    # ... and two Q6_K matrices (the type of the FFN down / output tensors of the common Q4_K_M files), held in the generic
    # packed device form (224 bytes per 256 weights for the file's 210): GB/s counted on the FILE's bytes
    # ... and the gate and up matrices of one layer loaded as ONE weight of 2 x 17408 rows (izb_weight_create_stack): one
    # launch where the separate matrices take two
    for qt, Nn, Kk, parts in ((12, 5120, K, 1), (12, 17408, K, 1), (8, 151936, K, 1), (12, 5120, 17408, 1), (14, 17408, K, 1), (14, 151936, K, 1),
                              (12, 34816, K, 2)):
        ws = [S.make_weight(qt, Nn // parts, Kk, SEED + Nn + (0 if Kk == K else Kk) + 7 * p) for p in range(parts)]
        wbytes = sum(w.size for w in ws)
        dev_bytes = wbytes if qt in (8, 12) else Nn * (Kk // 256) * (224 if qt == 14 else 304)
        copies = max(1, -(-300_000_000 // dev_bytes)) if dev_bytes < 400_000_000 else 2
        Ws = [izb.Weight(qt, ws[0], Nn, Kk) if parts == 1 else izb.stacked_weight(qt, ws, Kk) for _ in range(copies)]
        # rows the oracle checks after the timed launches: the first 1024 and the last 256 of the matrix
        chk_rows = np.concatenate([np.arange(min(1024, Nn)), np.arange(max(Nn - 256, 0), Nn)])
        w_chk = np.ascontiguousarray((ws[0] if parts == 1 else np.concatenate(ws))[chk_rows])
        del ws
        # (the output head once more with its logit soft-cap, as the reference's Gemma head runs: GEMV, then cap * tanh(v / cap))
        for T, cap in ((1, 0.0), (2, 0.0)) + (((1, 30.0),) if qt == 8 else ()):
            x = torch.from_numpy(S.make_act(T, Kk, SEED + T)).cuda()
            aq, asc, _ = izb.quantize_act(x, Mp=16)
            y = torch.empty((T, Nn), dtype=torch.float32, device="cuda")
            def launch(i):
                izb.gemv(Ws[i % copies], aq, asc, T, out=y)
                if cap > 0:
                    izb.softcap_rows(y, T, Nn, cap)

            for i in range(max(3, copies)):
                launch(i)
            torch.cuda.synchronize()
            # the launches of one sweep over the copies are captured in a CUDA graph, so that the host's per-call cost
            # (Python + ctypes) is not what is measured
            launches = copies if lite else max(20, 4 * copies)  # lite: few launches, for a profiler's launch list
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph):
                for i in range(launches):
                    launch(i)
            graph.replay()
            torch.cuda.synchronize()
            reps = 1 if lite else 5
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for _ in range(reps):
                graph.replay()
            e1.record()
            torch.cuda.synchronize()
            us = e0.elapsed_time(e1) * 1e3 / (launches * reps)
            # parity of this shape (checker only, outside the timed launches): one more launch against the oracle's f64 model
            from oracle import oracle as O
            launch(0)
            got = y.cpu().numpy()[:, chk_rows]
            ref = O.matmul(qt, w_chk, Kk, aq.cpu().numpy(), asc.cpu().numpy(), T, "f64")
            if cap > 0:
                ref = (np.float32(cap) * np.tanh(ref.astype(np.float64) / cap)).astype(np.float32)
            par = _rel(got, ref)
            nbytes = wbytes + T * (Kk + Kk // 32 * 4) + T * Nn * 4 * (3 if cap > 0 else 1)  # (the cap reads and writes the row again)
            gbs = nbytes / (us * 1e-6) / 1e9
            out.append({"type": {12: "Q4_K", 8: "Q8_0", 14: "Q6_K"}[qt], "device_weight_bytes": dev_bytes, "N": Nn, "K": Kk, "stacked_parts": parts, "batch": T, "softcap": cap,
                        "in_config3": Kk == K and cap == 0 and qt != 14 and parts == 1, "us_per_launch": us,
                        "bytes_per_launch": nbytes, "GBps": gbs, "frac_of_hbm_peak": gbs / hbm_peak, "parity_max_rel": par, "parity_tolerance": 1e-5,
                        "parity_rows_checked": int(len(chk_rows)),
                        "peak": f"{hbm_peak} GB/s {peak_src} copy", "weight_copies_in_rotation": copies})
        for W_ in Ws:
            W_.close()
    return out


def moe_section(izb, torch, tc_peak: float, peak_src: str, iters: int = 10) -> dict:
    """4096 tokens, hidden 2048, 128 experts (gate / up 768 x 2048, down 2048 x 768, Q4_K), top-8
    routing from softmax of N(0,1) logits.  One pass = route, sort by expert, grouped gate/up GEMM with the SwiGLU store,
    quantise, grouped down GEMM scaled by the router weights, weighted sum per token.  Device-timed."""
    from arcinferzero_b200 import synth as S
    T, E, F, NE, NU, TM = 4096, 2048, 768, 128, 8, 128
    rng = np.random.default_rng(SEED + 9)
    wg, wu, wd = S.make_weight(QT, NE * F, E, SEED + 11), S.make_weight(QT, NE * F, E, SEED + 12), S.make_weight(QT, NE * E, F, SEED + 13)
    Wgu = izb.gateup_weight(QT, wg, wu, F, E, n_mats=NE)  # gate | up rows interleaved: one grouped GEMM, SwiGLU in its epilogue
    Wd = izb.Weight(QT, wd, E, F, n_mats=NE)
    x = torch.from_numpy(S.make_act(T, E, SEED + 14)).cuda()
    logits = torch.from_numpy(rng.standard_normal((T, NE), dtype=np.float32)).cuda()
    Sn = T * NU
    Sp = izb.pad_rows(Sn)
    out = torch.empty_like(x)

    keep = {}

    def one_pass():
        out.copy_(x)
        aq, asc, _ = izb.quantize_act(x, Mp=T)
        ids, wts, counts = izb.moe_route(logits, NU)
        offs, tiles, max_tiles, stok, swt, inv = izb.moe_sort(ids, wts, counts, TM)
        h = izb.moe_gateup(Wgu, None, aq, asc, tiles, max_tiles, TM, stok, Sn)
        hq, hsc, _ = izb.quantize_act(h, Mp=Sp)
        y = izb.moe_down(Wd, hq, hsc, tiles, max_tiles, TM, swt, Sn)
        izb.moe_combine(out, y, inv, NU)
        keep.update(aq=aq, asc=asc, ids=ids, offs=offs, stok=stok, swt=swt, h=h, hq=hq, hsc=hsc, y=y)
        return counts

    def parity() -> dict:
        """Stage-wise, teacher-forced, on sampled slots against the CPU oracle (checker only, after the timed region)."""
        from oracle import oracle as O
        k = {n: v.cpu().numpy() for n, v in keep.items()}
        rid, _, _ = O.moe_route(logits.cpu().numpy(), NU)
        se = O.slot_experts(k["offs"])
        smp = np.unique(np.concatenate([k["offs"][[0, 1, 64, 127]], k["offs"][[1, 65, 128]] - 1, rng.integers(0, Sn, 20)]))
        rh = O.moe_gateup(QT, wg, wu, F, E, k["aq"], k["asc"], se[smp], k["stok"][smp])
        rq, rs, _ = O.quantize_act(k["h"][smp])
        ry = O.moe_down(QT, wd, E, F, rq, rs, se[smp], k["swt"][smp])
        return {"parity_max_rel": max(_rel(k["h"][smp], rh), _rel(k["y"][smp], ry)), "parity_tolerance": 1e-5,
                "routing_ids_exact": bool((k["ids"] == rid).all()),
                "int8_rows_exact": bool(np.array_equal(k["hq"][smp], rq) and np.array_equal(k["hsc"][:, smp].view(np.uint32), rs.view(np.uint32))),
                "parity_slots_sampled": int(len(smp))}

    for _ in range(3):
        counts = one_pass()
    torch.cuda.synchronize()
    l0 = izb.launch_count()
    izb.profile_start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(iters):
        one_pass()
    e1.record()
    torch.cuda.synchronize()
    prof = izb.profile_stop()
    ms = e0.elapsed_time(e1) / iters
    launches = (izb.launch_count() - l0) // iters
    ops = 2.0 * Sn * 3 * F * E
    c = counts.cpu().numpy()
    tc_ms = sum(v["ms"] for k, v in prof.items() if k == "gemm_tc") / iters
    res = {"workload": "config 4: 4096 tokens x top-8 of 128 experts, hidden 2048, expert FFN 768, Q4_K",
           "ms_per_pass": ms, "tokens_per_s": T / (ms * 1e-3), "tops": ops / (ms * 1e-3) / 1e12,
           "grouped_gemm_ms_per_pass": tc_ms, "grouped_gemm_tops": ops / (tc_ms * 1e-3) / 1e12 if tc_ms > 0 else None,
           "frac_of_tensor_peak_grouped_gemm": (ops / (tc_ms * 1e-3) / 1e12) / tc_peak if tc_ms > 0 else None,
           "peak": f"{tc_peak} TFLOP/s {peak_src} dense 16-bit sustained", "gpu_launches_per_pass": launches,
           "expert_load": {"max": int(c.max()), "min": int(c.min()), "mean": float(c.mean())},
           "kernel_ms_per_pass": {k: v["ms"] / iters for k, v in prof.items()},
           "finite": bool(torch.isfinite(out).all().item())}
    res.update(parity())
    for W in (Wgu, Wd):
        W.close()
    return res


def q8_config1_section(izb, torch, tc_peak: float, iters: int = 20) -> dict:
    """BASELINE.json config 1 (the reference's CPU-runnable case): one Q8_0 GEMM, M = 512, N = K = 4096, through the same
    tensor-core kernel; device-timed, quantiser included."""
    from arcinferzero_b200 import synth as S
    Mq, Nq, Kq = 512, 4096, 4096
    W = izb.Weight(8, S.make_weight(8, Nq, Kq, SEED + 21), Nq, Kq)
    x = torch.from_numpy(S.make_act(Mq, Kq, SEED + 22)).cuda()
    out = torch.empty((Mq, Nq), dtype=torch.float32, device="cuda")
    aq = torch.empty((Mq, Kq), dtype=torch.int8, device="cuda")
    asc = torch.empty((Kq // 32, Mq), dtype=torch.float32, device="cuda")
    for _ in range(3):
        izb.quantize_act(x, Mp=Mq, out=(aq, asc, None))
        izb.matmul(W, aq, asc, Mq, out=out)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record()
    for _ in range(iters):
        izb.quantize_act(x, Mp=Mq, out=(aq, asc, None))
        izb.matmul(W, aq, asc, Mq, out=out)
    e1.record()
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / iters
    tops = 2.0 * Mq * Nq * Kq / (ms * 1e-3) / 1e12
    W.close()
    return {"workload": "config 1: Q8_0 GEMM M=512 N=4096 K=4096 (quantize_act + GEMM)", "ms_per_step": ms,
            "tokens_per_s": Mq / (ms * 1e-3), "tops": tops, "frac_of_tensor_peak": tops / tc_peak,
            "note": "128 tiles on 148 SMs: a single partial wave, host launch cost included"}


def tp_stack_parity(st, torch, dist, x_in) -> dict:
    """One teacher-forced layer of the stack on sampled token rows against the CPU oracle (checker only, outside every
    timed region): each projection from the GPU's own quantised input, the sums from all ranks' partial outputs in rank
    order, the quantiser bit for bit, and a checksum of the quantised stream that must be equal on all ranks."""
    from arcinferzero_b200 import tp
    from oracle import oracle as O
    cfg, world, rank = st.cfg, st.world, st.rank
    QT, E = cfg.qtype, cfg.hidden
    st.set_input(x_in)
    trace = []
    st.forward(trace, layers=1)
    torch.cuda.synchronize()
    t = trace[0]
    # the same sample on every rank: two rows of every rank's share of the first and of the last chunk
    own = st.Tc // world
    idx = np.array(sorted({c * st.Tc + r * own + o for c in (0, st.chunks - 1) for r in range(world) for o in (0, own - 1)}))
    mine = np.intersect1d(idx, st.owned_rows())
    g = lambda k: t[k][torch.from_numpy(idx).to(t[k].device)].cpu().numpy()  # noqa: E731
    sh = tp.shard_rows(cfg, tp.layer_weights(cfg, 0), st.plan)
    nq = st.plan.q[1] - st.plan.q[0]
    rels, exact = {}, True
    xq0, xsc0 = g("xq0"), np.ascontiguousarray(t["xsc0"][:, torch.from_numpy(idx).to(t["xsc0"].device)].cpu().numpy())
    qkv = g("qkv")
    rels["qkv"] = _rel(qkv, O.matmul(QT, sh["qkv"][0], E, xq0, xsc0, len(idx)))
    hq, hsc, _ = O.quantize_act(np.ascontiguousarray(qkv[:, :nq]))
    rows, _, Kk, cr = sh["o"]
    o_part = g("o_part")
    rels["o_part"] = _rel(o_part, O.matmul(QT, tp.slice_cols(QT, rows, Kk, *cr), nq, hq, hsc, len(idx)))

    def all_parts(a):
        tt = torch.from_numpy(np.ascontiguousarray(a)).cuda()
        if world == 1:
            return a[None]
        out = [torch.empty_like(tt) for _ in range(world)]
        dist.all_gather(out, tt)
        return np.stack([o.cpu().numpy() for o in out])

    sel = np.searchsorted(idx, mine)
    x1 = g("x1")
    rels["x1"] = _rel(x1[sel], O.tp_add(g("x0"), all_parts(o_part))[sel])
    xq1 = g("xq1")
    xsc1 = np.ascontiguousarray(t["xsc1"][:, torch.from_numpy(idx).to(t["xsc1"].device)].cpu().numpy())
    rq, rs, _ = O.quantize_act(np.ascontiguousarray(x1[sel]))
    exact &= bool(np.array_equal(xq1[sel], rq) and np.array_equal(xsc1[:, sel].view(np.uint32), rs.view(np.uint32)))
    gate = O.matmul(QT, sh["gate"][0], E, xq1, xsc1, len(idx))
    up = O.matmul(QT, sh["up"][0], E, xq1, xsc1, len(idx))
    h = g("h")
    rels["h"] = _rel(h, (up * (gate / (np.float32(1) + np.exp(-gate, dtype=np.float32)))).astype(np.float32))
    hq, hsc, _ = O.quantize_act(h)
    rows, _, Kk, cr = sh["down"]
    d_part = g("down_part")
    rels["down_part"] = _rel(d_part, O.matmul(QT, tp.slice_cols(QT, rows, Kk, *cr), cr[1] - cr[0], hq, hsc, len(idx)))
    rels["x2"] = _rel(g("x2")[sel], O.tp_add(x1, all_parts(d_part))[sel])
    # the quantised stream every rank holds must be the same bytes
    chk = torch.stack([t["xq2"].view(torch.int64).sum(), t["xsc2"].view(torch.int32).to(torch.int64).sum(),
                       t["xq1"].view(torch.int64).sum(), t["xsc1"].view(torch.int32).to(torch.int64).sum()])
    same = True
    if world > 1:
        allc = [torch.empty_like(chk) for _ in range(world)]
        dist.all_gather(allc, chk)
        same = all(bool(torch.equal(allc[0], c)) for c in allc[1:])
    worst = torch.tensor([max(rels.values()), 0.0 if exact else 1.0, 0.0 if same else 1.0], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(worst, op=dist.ReduceOp.MAX)
    return {"parity_max_rel": float(worst[0].item()), "parity_tolerance": 1e-5, "parity_by_stage_rank0": rels,
            "int8_rows_exact": worst[1].item() == 0.0, "int8_identical_across_ranks": worst[2].item() == 0.0,
            "parity_rows_sampled": int(len(idx))}


def tp_stack_section(izb, torch, dist, world: int, rank: int, local: int, tokens: int, passes: int = 2) -> list:
    """the projections of 8 dense layers (Q4_K, hidden 5120, FFN 17408, 7168 QKV rows) over 32768
    token rows, split over the ranks as the reference's tensor-parallel mode splits them.  Three forms of
    arcinferzero_b200/tp.py: the two summation modes with everything on one stream, and the pipelined form (token chunks,
    the sums of one chunk on a second stream beside the GEMMs of the next, Q rows balanced against the FFN rows).
    Device-timed per pass, max over ranks; each entry carries the parity of one teacher-forced layer."""
    from arcinferzero_b200 import synth as S
    from arcinferzero_b200 import tp
    cfg = tp.StackConfig(tokens=tokens)
    x_in = torch.from_numpy(S.make_act(cfg.tokens, cfg.hidden, SEED + 5)).cuda() * 0.05
    out = []
    forms = [("allreduce", dict()), ("rs_quant_ag", dict()),
             # (SMs left to the collectives, swept at 8 ranks: 4 -> 138 ms, 8 -> 81, 12 -> 68.2, 16 -> 66.9, 20 -> 66.0,
             #  24 -> 70.4, 32 -> 74.4 per pass: too few and the sums become the critical path, too many and the GEMMs lose
             #  more than the sums gain; at 2 ranks the sums are 3 % of a pass)
             ("rs_quant_ag", dict(chunks=4, overlap=True, balance=True, comm_sms=8 if world <= 2 else 16 if world < 8 else 20)),
             # the same sums moved by the copy engines (izb_p2p_*): no SM is taken from the GEMMs
             ("p2p", dict(chunks=4, balance=True))]
    if world != 2:
        forms = forms[:3]   # (the copy-engine form is run at two ranks, where it has been verified and is the fastest)
    if world == 1:
        forms = forms[1:3]  # (one rank: the summation modes are the same work and nothing is moved)
    for mode, kw in forms:
        try:
            st = tp.Stack(cfg, world, rank, local, mode=mode, distinct_layers=False, **kw)
        except Exception as e:  # (a form this box cannot set up, e.g. no peer mappings between the GPUs: say so, go on)
            ok = torch.tensor([0], device="cuda")
            st = None
            err = f"{type(e).__name__}: {e}"[:300]
        else:
            ok = torch.tensor([1], device="cuda")
        if world > 1:
            dist.all_reduce(ok, op=dist.ReduceOp.MIN)
        if int(ok.item()) == 0:
            out.append({"mode": mode, "form": kw, "unavailable": err if st is None else "another rank could not set this form up"})
            st = None
            continue
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        ms = 0.0
        l0 = 0
        for p in range(1 + passes):
            st.set_input(x_in)
            if world > 1:
                dist.barrier()
            torch.cuda.synchronize()
            if p == 1:
                l0 = izb.launch_count()
            e0.record()
            st.forward()
            e1.record()
            torch.cuda.synchronize()
            if p >= 1:
                ms += e0.elapsed_time(e1)
        launches = izb.launch_count() - l0
        t = torch.tensor([ms / passes], dtype=torch.float64, device="cuda")
        if world > 1:
            dist.all_reduce(t, op=dist.ReduceOp.MAX)
        ms_pass = float(t.item())
        own = torch.from_numpy(st.owned_rows()).cuda()
        finite = bool(torch.isfinite(st.x[own]).all().item())
        nbytes = cfg.tokens * cfg.hidden * 4
        entry = {"mode": mode + ("+overlap" if kw.get("overlap") else ""), "form": kw or {"chunks": 1, "overlap": False, "balance": False},
                 "ms_per_pass": ms_pass, "tokens_per_s": cfg.tokens / (ms_pass * 1e-3),
                 "tops_all_ranks": cfg.ops_per_pass / (ms_pass * 1e-3) / 1e12, "sums_per_pass": 2 * cfg.layers,
                 "bytes_per_sum_f32": nbytes, "gpu_launches_per_pass": launches // passes, "finite": finite,
                 "workload": f"config 5: {cfg.layers} layers x (QKV 7168, O, gate, up, down) Q4_K, T={cfg.tokens}, hidden 5120, FFN 17408"}
        entry.update(tp_stack_parity(st, torch, dist, x_in))
        out.append(entry)
        st.close()
        del st
        torch.cuda.empty_cache()
    return out


def run_reference(args, rank: int) -> None:
    if rank != 0:
        return
    base, timed = None, []
    for i in range(args.warmup + args.steps):  # a step = one bounded sample of the workload (see cpu_baseline)
        base = cpu_baseline(seconds_target=4.0)
        if i >= args.warmup:
            timed.append(base["value"])
    vals = float(np.mean(timed)) if timed else base["value"]
    base = dict(base, value=vals)
    line = {"impl": "reference", "metric": "Q4_K prefill GEMM throughput", "value": vals, "unit": "tok/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000.0 * M / vals, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None, "dtype": "f64",
            "data": "synthetic", "config": {"workload": WORKLOAD}, "cpu_baseline": base,
            "e2e": {"value": vals, "unit": "tok/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0}, "gpu_launches": 0}
    print(json.dumps(line), flush=True)


def main() -> None:
    global M, WORKLOAD
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=20)
    ap.add_argument("--warmup", type=int, default=5)
    ap.add_argument("--impl", default="ours")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-gemv", action="store_true", help="skip the decode GEMV section (BASELINE.json config 3)")
    ap.add_argument("--no-moe", action="store_true", help="skip the MoE section (BASELINE.json config 4)")
    ap.add_argument("--moe-only", action="store_true", help="profiling only: run just the MoE section")
    ap.add_argument("--gemv-only", action="store_true", help="profiling only: run just the decode GEMV section")
    ap.add_argument("--lite", action="store_true", help="profiling only: few launches per GEMV shape")
    ap.add_argument("--no-tp-stack", action="store_true", help="skip the tensor-parallel projection stack (BASELINE.json config 5)")
    ap.add_argument("--tp-tokens", type=int, default=32768, help="profiling only: token rows of the stack section")
    ap.add_argument("--tokens", type=int, default=M, help="profiling only: fewer token rows than the configured 8192")
    args = ap.parse_args()
    if args.tokens != M:
        M = args.tokens
        WORKLOAD = WORKLOAD.replace("M=8192", f"M={M} (reduced for profiling)")
    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    if args.impl == "reference":
        run_reference(args, rank)
        return

    import torch
    import torch.distributed as dist

    import arcinferzero_b200 as izb
    from arcinferzero_b200 import synth as S

    assert torch.cuda.is_available(), "bench.py needs a GPU (the library has no CPU path)"
    torch.cuda.set_device(local)
    if args.moe_only:
        _, _, tc_sus, src = peaks()
        print(json.dumps({"moe": moe_section(izb, torch, tc_sus, src, iters=3)}), flush=True)
        return
    if args.gemv_only:
        hbm, _, _, src = peaks()
        print(json.dumps({"decode_gemv": gemv_section(izb, torch, hbm, src, lite=args.lite)}), flush=True)
        return
    if world > 1:
        dist.init_process_group("nccl", device_id=torch.device("cuda", local))

    # ---- this rank's rows of the weight (column-parallel split in units of 256 rows, zero/mgpu/engine_tp_shard.h:68-72)
    n0, n1 = izb.tp_range(N, 256, world, rank)
    Nr = n1 - n0
    w_full = S.make_weight(QT, N, K, SEED)
    W = izb.Weight(QT, w_full, N, K, device=local, row_range=(n0, n1))
    w_shard = np.ascontiguousarray(w_full[n0:n1]) if rank == 0 else None  # (for the parity field of the line)
    del w_full
    x_host = torch.from_numpy(S.make_act(M, K, SEED + 1)).pin_memory()
    x = x_host.cuda(non_blocking=True)
    Mp = izb.pad_rows(M)
    aq = torch.empty((Mp, K), dtype=torch.int8, device="cuda")
    asc = torch.empty((K // 32, Mp), dtype=torch.float32, device="cuda")
    out = torch.empty((Mp, Nr), dtype=torch.float32, device="cuda")
    out_host = torch.empty((M, Nr), dtype=torch.float32).pin_memory()
    izb.selfcheck(local)

    def step():
        # quant_rows + matmul as one call (izb_quant_matmul): the quantiser also writes the tensor-core GEMM's operand images
        izb.quant_matmul(W, x, M, Mp, out=out, qout=(aq, asc))

    def barrier():
        if world > 1:
            dist.barrier()
        torch.cuda.synchronize()

    for _ in range(max(3, args.warmup)):
        step()
    barrier()
    try:
        pr = torch.cuda.get_device_properties(local)
        pci = f"{pr.pci_domain_id:08x}:{pr.pci_bus_id:02x}:{pr.pci_device_id:02x}.0"
    except Exception:
        pci = None
    sampler = ClockSampler(local, pci)
    if rank == 0:
        sampler.start()
    launches0 = izb.launch_count()
    izb.profile_start()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    barrier()
    e0.record()
    for _ in range(args.steps):
        step()
    e1.record()
    barrier()
    ms_total = e0.elapsed_time(e1)
    prof = izb.profile_stop()
    launches = izb.launch_count() - launches0
    t = torch.tensor([ms_total], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_total = float(t.item())
    ms_step = ms_total / args.steps

    # ---- parity of what was just timed (rank 0; the oracle is the checker, outside the timed region): eight token rows of
    # the last step's output against the oracle's quantiser (int8 rows and scales exact) and its f64 model of the product
    parity = None
    if rank == 0:
        from oracle import oracle as O
        idx = np.array([0, 1, 127, 128, M // 2, M - 129, M - 2, M - 1])
        xs = x_host.numpy()[idx]
        oq, osc, _ = O.quantize_act(xs, Mp=16)
        tidx = torch.from_numpy(idx).cuda()
        gq, gsc = aq[tidx].cpu().numpy(), asc[:, tidx].cpu().numpy()
        ref = O.matmul(QT, w_shard, K, oq, osc, len(idx), "f64")
        parity = {"parity_max_rel": _rel(out[tidx].cpu().numpy(), ref), "parity_tolerance": 1e-5,
                  "int8_rows_exact": bool((gq == oq[:len(idx)]).all() and (gsc.view(np.uint32) == osc[:, :len(idx)].view(np.uint32)).all()),
                  "rows_checked": int(len(idx)), "columns_checked": int(Nr)}
        del w_shard

    # ---- end to end through the host-buffer C-ABI call
    for _ in range(2):
        izb.matmul_host(W, x_host, out_host)
    barrier()
    e_steps = max(2, min(args.steps, 5))
    t0 = time.perf_counter()
    e0.record()
    for _ in range(e_steps):
        izb.matmul_host(W, x_host, out_host)
    e1.record()
    barrier()
    ms_e2e = e0.elapsed_time(e1) / e_steps
    t = torch.tensor([ms_e2e], dtype=torch.float64, device="cuda")
    if world > 1:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_e2e = float(t.item())
    clocks = sampler.stop() if rank == 0 else None
    tp_stack = None
    if not args.no_tp_stack:
        W.close()
        del x, aq, asc, out
        torch.cuda.empty_cache()
        tp_stack = tp_stack_section(izb, torch, dist, world, rank, local, args.tp_tokens)
    # the device's own tensor-core rates: a TMEM-resident tcgen05.mma loop per MMA kind, a short burst and ~0.5 s sustained
    tc_peaks = None
    if rank == 0:
        tc_peaks = {}
        for name, kind in (("f16", 0), ("i8", 1)):
            burst, clk = izb.tensor_peak(local, kind, 4096, 2)
            sus, _ = izb.tensor_peak(local, kind, 4096, 400 if kind == 0 else 800)
            tc_peaks[name] = {"burst_tops": burst, "sustained_tops": sus, "sm_clocks_per_128x256_mma": clk}
    status = izb.device_status(local)

    if rank == 0:
        hbm, tc_burst, tc_sus, src = peaks()
        kname = next((k for k in ("gemm_fold", "gemm_tc", "gemm_core") if k in prof), "gemm_tc")
        g = prof.get(kname) or {"launches": 0, "ms": 0.0}
        per_tile = NCU_TRAFFIC_BYTES_PER_TILE
        ms_kernel = g["ms"] / max(1, g["launches"])
        ops = 2.0 * M * Nr * K
        achieved = ops / (ms_kernel * 1e-3) / 1e12 if ms_kernel > 0 else 0.0
        total_prof = sum(v["ms"] for v in prof.values()) or 1.0
        line = {
            "metric": "Q4_K prefill GEMM throughput", "value": M / (ms_step * 1e-3), "unit": "tok/s", "n_gpus": world,
            "steps": args.steps, "warmup": max(3, args.warmup), "ms_per_step": ms_step, "higher_is_better": True,
            "scaling": "strong", "vs_baseline": None,
            "dtype": "int8",
            "data": "synthetic",
            "config": {"workload": WORKLOAD,
                       "arithmetic": ("int8 x 4-bit dot products per 32-block with the block scales in the operands (activations as two fp16 terms, 23 to 24 bits; "
                                      "weight sub-scale x quant exact in fp16; f32 TMEM accumulators per 256 of K), f32 combine"),
                       "parallelism": f"weight rows split over {world} rank(s), no exchange",
                       "l2": "per step 168 MB of f32 activations in and 570 MB of outputs written: larger than the 126 MB L2",
                       "rows_per_rank": Nr},
            "roofline": {"bound": "tensor", "kernel": kname, "achieved": achieved, "peak": tc_sus, "unit": "TFLOP/s",
                         "frac": achieved / tc_sus, "peak_source": f"{src} dense bf16/fp16 (sustained; burst {tc_burst})",
                         "frac_of_burst_peak": achieved / tc_burst, "frac_of_nominal_int8": achieved / NOMINAL_INT8_TOPS,
                         "frac_of_measured_int8": achieved / tc_peaks["i8"]["burst_tops"], "frac_of_measured_f16_mma": achieved / tc_peaks["f16"]["burst_tops"],
                         "measured_tcgen05_peaks": dict(tc_peaks, method="izb_tensor_peak: tcgen05.mma 128x256 loop, operands in shared memory, accumulators in TMEM, all SMs"),
                         # DRAM bytes per launch: one ncu capture of the same kernel at 2048 token rows and all weight rows
                         # (read 159.7 MB + written 121.0 MB), scaled by the 128x128 tiles this launch runs
                         "traffic": per_tile * ((M + 127) // 128) * (Nr // 128),
                         "traffic_source": f"ncu dram__bytes_read+write of {kname} at M=2048, N=17408 (profiles/), per 128x128 tile x tiles",
                         "ms_per_launch": ms_kernel, "launches": g["launches"],
                         "kernel_shares": {k: v["ms"] / total_prof for k, v in prof.items()}},
            "e2e": {"value": M / (ms_e2e * 1e-3), "unit": "tok/s", "h2d_bytes_per_step": M * K * 4, "d2h_bytes_per_step": M * Nr * 4},
            "gpu_launches": launches, "clocks": clocks, "device_wait_errors": status, "parity": parity,
        }
        if tp_stack is not None:
            line["tp_stack"] = tp_stack
        if not args.no_moe and world == 1:
            line["moe"] = moe_section(izb, torch, tc_sus, src)
            line["q8_0_gemm_config1"] = q8_config1_section(izb, torch, tc_sus)
        if not args.no_gemv and world == 1:
            line["decode_gemv"] = gemv_section(izb, torch, hbm, src)
        if not args.no_cpu_baseline and world == 1:
            line["cpu_baseline"] = cpu_baseline()
        print(json.dumps(line), flush=True)
    W.close()
    if world > 1:
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
