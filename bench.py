#!/usr/bin/env python
"""Benchmark of the likelihood path on one B200 (or N, pattern-sharded).

Workload (the "FP64 vs mixed-precision DNA at scale" configuration): DNA GTR+G4 (Gamma shape
0.5) on a seeded 512-taxon tree with branch lengths ~Exp(0.05), 1,000,000 simulated sites
with 5% gap cells, compressed to unique patterns (with random gaps nearly every column is
unique).  A step is one full-tree log-likelihood evaluated from scratch: every partial of the
tree recomputed (510 node updates over all patterns), then the branch log-likelihood and its
pattern-weighted sum.  Both precision forms are timed in the same run:
  * fp64  -- the plain drop-in (eigen-space FP64 partials, reference arithmetic);
  * mixed -- FP32 real-space partials with per-pattern scaling, FP64 branch terms.
`value` is the mixed form's site-partial updates/s when its lnL is within 1e-6 relative of
the FP64 lnL of the same run (reported as `lnl_rel_err_mixed`), else the FP64 form's.
`e2e` runs the same step through the public PhyloTree API from pinned host buffers (tips and
weights up, pattern lnL down; computeLikelihoodFromHost, the tip upload overlapped with the
traversal in pattern chunks).  Timing uses CUDA events on the session's stream; the partial
buffers (65 GB FP64, 33 GB mixed) exceed L2 many times over, so no flush is needed.

Also reported (same run): one Newton branch optimisation (optimizeOneBranch) per branch; the
20-state protein +G4 configuration (128 taxa, 100,000 sites) FP64 vs mixed (tcgen05 split-TF32)
with its lnL error; 256 RELL reweightings; 64 candidate codon models (+G4 and +R8) on one
200-taxon, 4,000-site alignment in one batched tcgen05 launch; the serving loop on a seeded
request stream; the measured compute peaks.  `--block NAME` runs one of these alone.

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl gems|reference]

Under torchrun each rank holds its own 1,000,000-site slab of the same tree and model (weak
scaling); the per-evaluation exchange is one NCCL all-reduce of the lnL.  `--impl reference`
times the CPU restatement of the reference kernels (oracle/, FP64, all host threads) on the
same workload, bounded to a pattern sample per step.
"""
from __future__ import annotations

import argparse
import json
import os
import re
import statistics
import subprocess
import sys
import tempfile
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from gems_b200 import synth  # noqa: E402

NSITES = 1_000_000
NTAXA = 512
MIXED_RTOL = 1e-6

CONFIGS = {
    "dna512": "DNA GTR+G4 (alpha 0.5), 512 taxa, Exp(0.05) lengths, {sites} sites/rank with 5% "
              "gaps, from-scratch full-tree lnL",
    "protein128": "20-state protein +G4 (alpha 0.8), log-normal exchangeabilities, Dirichlet "
                  "frequencies, 128 taxa, Exp(0.15) lengths, {sites} sites/rank, from-scratch "
                  "full-tree lnL",
}


def update_bytes(s, n=4, C=4, safe=False):
    """Algorithmic bytes of one site-partial update: internal-internal 3*C*n*s + 3*sigma,
    tip-internal 2*C*n*s + 1 + 2*sigma, tip-tip C*n*s + 2 + sigma, with s = 8 (FP64) or 4
    (FP32 partials) and sigma = 2 B (NORM counter) or 2*C B (SAFE counters)."""
    sig = 2 * C if safe else 2
    return 3 * C * n * s + 3 * sig, 2 * C * n * s + 1 + 2 * sig, C * n * s + 2 + sig


def required_bytes(P, nops, ntaxa, s, n=4, C=4, safe=False):
    """DRAM bytes a from-scratch traversal cannot avoid: every internal partial and its scale
    counters written once (they are the stored result later calls read), every tip byte read
    once.  Child partials read back by the op that consumes them are not counted: a kernel
    that keeps them on chip never reads them from DRAM."""
    sig = 2 * C if safe else 2
    return P * (nops * (C * n * s + sig) + ntaxa)


def _r(x, d=4):
    return float(f"{x:.{d}g}") if isinstance(x, (int, float)) and x is not None else x


def compact_line(line):
    """The bench line the driver parses: the contract's keys and a short summary of every
    block, small enough to stay whole in a 3,000-character output tail."""
    keep = ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step",
            "higher_is_better", "scaling", "vs_baseline", "dtype", "data", "gpu_launches",
            "clocks")
    out = {k: line[k] for k in keep if k in line}
    cfg = line["config"]
    out["config"] = {"workload": cfg["workload"], "npat_per_rank": cfg["npat_per_rank"],
                     "parallelism": cfg["parallelism"], "precision": cfg.get("precision"),
                     "l2": "inputs > L2, no flush"}
    rf = line["roofline"]
    out["roofline"] = {k: _r(rf[k]) for k in ("bound", "achieved", "peak", "unit", "frac",
                                               "traffic", "frac_required_bytes")}
    # frac counts every child partial as an HBM read (the per-update figure of the algorithm);
    # the kernel keeps children on chip, so the bytes it must move are the partial writes and
    # the tip reads: frac_required_bytes is the fraction of the peak on those
    out["roofline"]["basis"] = ("frac: algorithmic bytes (children counted as HBM reads); "
                                "frac_required_bytes: bytes the launch must move")
    e = line["e2e"]
    out["e2e"] = {k: _r(e[k]) for k in ("value", "unit", "h2d_bytes_per_step",
                                        "d2h_bytes_per_step", "ms_per_step", "h2d_copy_alone_ms")
                  if k in e}
    forms = {}
    for k, f in line.get("forms", {}).items():
        forms[k] = {"ms": _r(f["ms_per_step"]), "frac": _r(f["roofline"]["frac"]),
                    "frac_req": _r(f["roofline"]["frac_required_bytes"])}
        if "newton" in f:
            forms[k]["newton_ms_per_branch"] = _r(f["newton"]["ms_per_branch"])
        if "lnl_rel_err_vs_fp64" in f:
            forms[k]["lnl_rel_err_vs_fp64"] = _r(f["lnl_rel_err_vs_fp64"], 2)
    out["forms"] = forms
    if "parity" in line:
        p = line["parity"]
        out["parity_vs_oracle"] = {"patterns": p["patterns"], **{
            k: {"lnl": _r(p[k]["lnl_rel_err_vs_oracle"], 2),
                "df/ddf": _r(p[k]["df_err_over_ddf"], 2), "ddf": _r(p[k]["ddf_rel_err"], 2)}
            for k in ("fp64", "mixed")}}
    if "protein20" in line:
        p = line["protein20"]
        out["protein20"] = {"fp64_ms": _r(p["fp64"]["ms_per_step"]),
                            "tcgen05_ms": _r(p["mixed_tcgen05"]["ms_per_step"]),
                            "speedup_vs_fp64": _r(p["mixed_tcgen05"]["speedup_vs_fp64"]),
                            "lnl_rel_err_vs_fp64": _r(p["mixed_tcgen05"]["lnl_rel_err_vs_fp64"], 2),
                            "tensor_frac": _r(p["mixed_tcgen05"]["compute"]["frac"], 3),
                            "hbm_frac": _r(p["mixed_tcgen05"]["roofline"]["frac"], 3)}
    if "codon64" in line:
        out["codon64"] = {k: {"batched_ms": _r(c["batched_wall_ms"]),
                              "kernel_ms": _r(c["batched_traversal_kernel_ms"]),
                              "fp64_one_ms": _r(c["fp64_one_model_ms"]),
                              "speedup": _r(c["speedup_vs_fp64_one_by_one"], 3),
                              "err": _r(c["lnl_rel_err_model0_vs_fp64"], 2)}
                          for k, c in line["codon64"].items()}
    if "rell" in line:
        r = line["rell"]
        out["rell"] = {"ms": _r(r["ms_per_call"]), "frac": _r(r["roofline"]["frac"], 3),
                       "err": _r(r["max_rel_err_vs_fp64_dot"], 2)}
    if "serving" in line:
        sv = line["serving"]
        out["serving"] = {"req_s": _r(sv["throughput_req_s"]),
                          "capacity_req_s": _r(sv["capacity_req_s"]),
                          "p50_ms": _r(sv["latency_ms"]["p50"]),
                          "p99_ms": _r(sv["latency_ms"]["p99"]), "load": sv["load"]}
        if "at_half_capacity" in sv:
            h = sv["at_half_capacity"]
            out["serving"]["p99_ms_at_0.5"] = _r(h["latency_ms"]["p99"])
    if "ingest" in line:
        g = line["ingest"]
        out["ingest"] = {"device_ms": _r(g["device_path_ms"]), "host_ms": _r(g["host_path_ms"]),
                         "identical": g["identical_to_host"]}
    if "cpu_baseline" in line:
        c = line["cpu_baseline"]
        out["cpu_baseline"] = {"value": _r(c["value"]), "unit": c["unit"], "cores": c["cores"],
                               "kind": c["kind"], "sample": c["sample"]}
    return out


def update_flops(n=4, C=4):
    """Algorithmic flops of one site-partial update (eigen-space form): 6*C*n^2 + C*n."""
    return 6 * C * n * n + C * n


def env_rank():
    return (int(os.environ.get("RANK", 0)), int(os.environ.get("WORLD_SIZE", 1)),
            int(os.environ.get("LOCAL_RANK", 0)))


def op_kinds(tree):
    """(internal-internal, tip-internal, tip-tip) node updates of a from-scratch
    computeLikelihood, rooted at the leaf that findFarthestLeaf returns."""
    n = tree.nnodes
    adj = [[] for _ in range(n)]
    for u, v in zip(tree.eu, tree.ev):
        adj[int(u)].append(int(v))
        adj[int(v)].append(int(u))
    h = [0] * n
    sys.setrecursionlimit(10000)

    def far(node, dad):
        if dad >= 0 and len(adj[node]) == 1:
            h[node] = 0
            return node
        res = -1
        h[node] = 0
        for c in adj[node]:
            if c == dad:
                continue
            lf = far(c, node)
            if h[node] < h[c] + 1:
                h[node] = h[c] + 1
                res = lf
        return res

    root = far(0, -1)
    counts = [0, 0, 0]
    stack = [(adj[root][0], root)]
    while stack:
        node, dad = stack.pop()
        kids = [c for c in adj[node] if c != dad]
        if not kids:
            continue
        nleaf = sum(1 for c in kids if len(adj[c]) == 1)
        counts[nleaf] += 1
        stack.extend((c, node) for c in kids)
    return counts


def read_peaks():
    path = os.path.join(ROOT, "MEASURED_PEAKS.json")
    try:
        d = json.load(open(path))
        return float(d["hbm_gbs"]), float(d.get("bf16_tflops", 1590.0)), "measured"
    except Exception:
        return 6650.0, 1590.0, "fallback"


def read_traffic(name):
    """traffic (DRAM bytes per launch, scaled to this workload) from the committed ncu summary."""
    path = os.path.join(ROOT, "profiles", name)
    try:
        m = re.search(r"traffic_bytes_per_launch:\s*([0-9.eE+]+)", open(path).read())
        return float(m.group(1)) if m else None
    except OSError:
        return None


class Clocks:
    """nvidia-smi sampling during the timed region."""

    def __init__(self, index):
        self.index = index
        self.proc = None
        self.path = os.path.join(tempfile.gettempdir(), f"clocks_bench_{os.getpid()}.csv")

    def __enter__(self):
        try:
            os.makedirs(os.path.dirname(self.path), exist_ok=True)
            self.f = open(self.path, "w")
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.index),
                 "--query-gpu=clocks.sm,clocks.max.sm,power.draw,"
                 "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
                 "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap",
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=self.f, stderr=subprocess.DEVNULL)
        except Exception:
            self.proc = None
        return self

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            self.proc.wait()
            self.f.close()

    def summary(self):
        try:
            rows = [r.split(",") for r in open(self.path).read().strip().split("\n") if r]
            sm = [float(r[0]) for r in rows]
            reasons = set()
            names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
            for r in rows:
                for k, nm in enumerate(names):
                    if "Active" in r[3 + k] and "Not" not in r[3 + k]:
                        reasons.add(nm)
            return {"sm_mhz": statistics.median(sm), "sm_max_mhz": float(rows[0][1]),
                    "reasons": sorted(reasons), "samples": len(rows)}
        except Exception:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": [], "samples": 0}


def make_workload(rank, nsites, config="dna512"):
    """Same tree and model on every rank; each rank simulates its own site slab."""
    if config == "protein128":
        rng = np.random.default_rng(3)
        model = synth.protein(rng, 4, 0.8)
        tree = synth.random_tree(128, 0.15, 14)
        aln = synth.simulate(tree, model, nsites, 26 + 1000 * rank)
        return tree, model, aln
    rng = np.random.default_rng(2)
    model = synth.dna_gtr(rng, 4, 0.5)
    tree = synth.random_tree(NTAXA, 0.05, 13)
    aln = synth.simulate(tree, model, nsites, 25 + 1000 * rank, gap_frac=0.05)
    return tree, model, aln


def config_block(args, aln, nops):
    return {"workload": CONFIGS[args.config].format(sites=f"{args.sites:,}"),
            "npat_per_rank": aln.npat, "node_updates_per_step": nops,
            "parallelism": f"pattern-shard x{env_rank()[1]}",
            "l2": "inputs larger than L2 (partials 33-65 GB), no flush needed"}


def cpu_sample(model, aln, nsamp=40_000):
    """The first nsamp patterns of the workload, as an alignment of their own."""
    nsamp = min(aln.npat, nsamp)
    return synth.Alignment(aln.ntaxa, model.nstates, int(aln.weights[:nsamp].sum()),
                           np.ascontiguousarray(aln.patterns[:, :nsamp]), aln.weights[:nsamp])


def cpu_baseline(tree, model, aln, target_s=12.0, sub=None):
    """The oracle (CPU restatement of the reference kernels) on a bounded pattern sample."""
    from oracle import oracle as orc
    threads = os.cpu_count() or 1
    orc.set_threads(threads)
    sub = sub if sub is not None else cpu_sample(model, aln)
    nsamp = sub.npat
    ot = orc.OracleTree(tree, model, sub)
    nops = sum(op_kinds(tree))
    ot.computeLikelihood()  # warm-up (allocation of the oracle's buffers)
    t0 = time.perf_counter()
    k = 0
    while True:
        ot.clearAllPartialLH()
        ot.computeLikelihood()
        k += 1
        el = time.perf_counter() - t0
        if el > target_s or k >= 50:
            break
    ups = k * nops * nsamp / el
    return {"value": ups, "unit": "site-partial updates/s", "cores": threads, "kind": "port",
            "sample": f"{nsamp} of {aln.npat} patterns, {k} from-scratch lnL evaluations "
                      f"({nops} node updates each), oracle FP64 (scalar C, -O3, no FMA "
                      f"contraction), {threads} threads",
            "lnl_evals_per_s": k / el}


def slice_parity(tree, model, sub, local, nbranch=8):
    """Parity at the bench's own tree and model on the CPU sample: the oracle's lnL, pattern
    lnL and derivatives on `nbranch` branches against the FP64 and mixed GPU forms evaluated on
    the same patterns (a session over the sample)."""
    from gems_b200 import PhyloTree
    from oracle import oracle as orc
    ot = orc.OracleTree(tree, model, sub)
    lo, plo = ot.computeLikelihood(pattern_lh=True)
    edges = list(range(0, tree.nedges, max(1, tree.nedges // nbranch)))[:nbranch]
    dref = []
    for e in edges:
        u, v = int(tree.eu[e]), int(tree.ev[e])
        f, df = ot.computeFuncDerv(u, v, float(tree.length[e]), new_branch=True)
        dref.append((-f, -df))
    out = {"patterns": sub.npat, "oracle_lnl": lo, "branches_with_derivatives": len(edges)}
    for prec in ("fp64", "mixed"):
        gt = PhyloTree.from_case(tree, model, sub, precision=prec, device=local)
        lg, plg = gt.computeLikelihood(pattern_lh=True)
        d1e = d2e = 0.0
        for e, (r1, r2) in zip(edges, dref):
            u, v = int(tree.eu[e]), int(tree.ev[e])
            f, df = gt.computeFuncDerv(u, v, float(tree.length[e]), new_branch=True)
            d1e = max(d1e, abs(-f - r1) / abs(r2))
            d2e = max(d2e, abs(-df - r2) / abs(r2))
        out[prec] = {"lnl_rel_err_vs_oracle": abs(lg - lo) / abs(lo),
                     "pattern_lnl_max_abs_err": float(np.max(np.abs(plg - plo))),
                     "df_err_over_ddf": d1e, "ddf_rel_err": d2e}
        gt.close()
        gt.session.close()
    return out


def run_reference(args):
    rank, world, _ = env_rank()
    if rank != 0:
        return
    tree, model, aln = make_workload(0, args.sites, args.config)
    cpu_baseline(tree, model, aln, target_s=1.0)  # warm-up
    res = [cpu_baseline(tree, model, aln, target_s=max(3.0, 30.0 / args.steps))
           for _ in range(args.steps)]
    v = statistics.median(r["value"] for r in res)
    nops = sum(op_kinds(tree))
    line = {
        "impl": "reference", "metric": "site-partial updates/s", "value": v,
        "unit": "site-partial updates/s", "n_gpus": 0, "steps": args.steps,
        "warmup": args.warmup, "higher_is_better": True, "scaling": "weak",
        "ms_per_step": 1e3 * nops * aln.npat / v, "vs_baseline": None, "dtype": "f64",
        "data": "synthetic (seeded generator; no public dataset)",
        "config": config_block(args, aln, nops),
        "cpu_baseline": {**res[0], "value": v},
        "e2e": {"value": v, "unit": "site-partial updates/s", "h2d_bytes_per_step": 0,
                "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line), flush=True)


def time_lnl(gt, steps, warmup, stream, dist, lnl_buf):
    """K from-scratch lnL evaluations timed with CUDA events on the session stream; returns
    (ms per step (max over ranks), lnL, traversal kernel ms per launch, launches)."""
    import torch
    s = gt.session

    def step():
        gt.clearAllPartialLH()
        v = gt.computeLikelihood()
        if dist is not None:
            lnl_buf.fill_(v)
            dist.all_reduce(lnl_buf)
            return float(lnl_buf.item())
        return v

    for _ in range(warmup):
        step()
    torch.cuda.synchronize()
    if dist is not None:
        dist.barrier()
    s.profile(True)
    s.profile_read(0)
    l0 = s.launch_count()
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    e0.record(stream)
    for _ in range(steps):
        lnl = step()
    e1.record(stream)
    torch.cuda.synchronize()
    s.profile(False)
    ms = e0.elapsed_time(e1) / steps
    trav_ms, trav_n = s.profile_read(0)
    launches = s.launch_count() - l0
    t = torch.tensor([ms], dtype=torch.float64, device=lnl_buf.device)
    if dist is not None:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    return float(t.item()), lnl, trav_ms / max(trav_n, 1), launches


def time_newton(gt, tree, stream, nbranch=24):
    """optimizeOneBranch on nbranch branches (traversal of stale partials, theta, the whole
    Newton loop on device); ms per branch."""
    import torch
    gt.clearAllPartialLH()
    gt.computeLikelihood()
    br = [(int(u), int(v)) for u, v in zip(tree.eu, tree.ev)][:nbranch]
    gt.optimizeOneBranch(*br[0])  # warm-up
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    torch.cuda.synchronize()
    e0.record(stream)
    nev = 0
    for u, v in br:
        gt.optimizeOneBranch(u, v)
        nev += gt.stats()[1]
    e1.record(stream)
    torch.cuda.synchronize()
    return {"branches": len(br), "ms_per_branch": e0.elapsed_time(e1) / len(br),
            "derivative_evals_per_branch": nev / len(br)}


def protein_comparison(args, local, peaks):
    """20-state +G4: FP64 vs mixed (tcgen05 split-TF32) and mixed on CUDA cores, each with its
    HBM roofline (algorithmic bytes) and compute roofline (algorithmic flops 6Cn^2 + Cn per
    update, credited alike to every form, against the measured peak of the unit it runs on)."""
    import torch
    from gems_b200 import PhyloTree
    tree, model, aln = make_workload(0, 100_000, "protein128")
    out = {"workload": CONFIGS["protein128"].format(sites="100,000"), "npat": aln.npat}
    kinds = op_kinds(tree)
    nops = sum(kinds)
    hbm_peak, _, peak_src = read_peaks()
    n, C = model.nstates, model.ncat
    flops = aln.npat * nops * update_flops(n, C)
    lnl_buf = torch.zeros(1, dtype=torch.float64, device=f"cuda:{local}")
    res = {}
    for name, prec, tc in (("fp64", "fp64", True), ("mixed_tcgen05", "mixed", True),
                           ("mixed_cuda_cores", "mixed", False)):
        gt = PhyloTree.from_case(tree, model, aln, precision=prec, device=local)
        gt.session.set_tensor_cores(tc)
        stream = torch.cuda.ExternalStream(gt.session.stream_handle(), device=local)
        ms, lnl, kms, _ = time_lnl(gt, max(args.steps, 5), 3, stream, None, lnl_buf)
        b_ii, b_ti, b_tt = update_bytes(8 if prec == "fp64" else 4, n, C)
        alg = aln.npat * (kinds[0] * b_ii + kinds[1] * b_ti + kinds[2] * b_tt)
        unit, pk = {"fp64": ("fp64 mma.sync (the rate of fp64 FMA)", peaks["fp64_tflops"]),
                    "mixed_tcgen05": ("tcgen05 TF32 (3 products issued per credited one)",
                                      peaks["tf32_tflops"]),
                    "mixed_cuda_cores": ("fp32 FMA", peaks["fp32_tflops"])}[name]
        res[name] = {"ms_per_step": ms, "traverse_ms": kms,
                     "site_partial_updates_per_s": nops * aln.npat / (ms * 1e-3),
                     "lnl_evals_per_s": 1e3 / ms, "lnl": lnl,
                     "roofline": {"bound": "hbm", "achieved": alg / (kms * 1e-3) / 1e9,
                                  "peak": hbm_peak, "peak_source": peak_src, "unit": "GB/s",
                                  "frac": alg / (kms * 1e-3) / 1e9 / hbm_peak,
                                  "algorithmic_bytes_per_launch": alg,
                                  "traffic": read_traffic(f"traverse_{prec}_protein128.md")
                                  if tc else None},
                     "compute": {"unit_used": unit, "achieved_tflops": flops / (kms * 1e-3) / 1e12,
                                 "peak_tflops": pk, "frac": flops / (kms * 1e-3) / 1e12 / pk,
                                 "algorithmic_flops_per_launch": flops}}
        gt.close()
        gt.session.close()
    base = res["fp64"]
    for k in ("mixed_tcgen05", "mixed_cuda_cores"):
        res[k]["speedup_vs_fp64"] = base["ms_per_step"] / res[k]["ms_per_step"]
        res[k]["lnl_rel_err_vs_fp64"] = abs(res[k]["lnl"] - base["lnl"]) / abs(base["lnl"])
    out.update(res)
    return out


def rell_block(gt, aln, stream, R=256, reps=5):
    """UFBoot RELL on the resident pattern log-likelihoods: R multinomial reweightings
    (seeded) of the pattern counts, replicate lnL and derivative sums in one launch each."""
    import torch
    s = gt.session
    # multinomial resampling of the sites (as UFBoot draws them), counted per pattern
    rng = np.random.default_rng(11)
    site_ptn = np.repeat(np.arange(aln.npat), aln.weights.astype(np.int64))
    nsites = len(site_ptn)
    W = np.empty((R, aln.npat), np.float32)
    for r in range(R):
        W[r] = np.bincount(site_ptn[rng.integers(nsites, size=nsites)], minlength=aln.npat)
    s.upload_reweightings(W)
    _, plh = gt.computeLikelihood(pattern_lh=True)
    ref = W.astype(np.float64) @ plh
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    got = s.reweighted_lnl()
    torch.cuda.synchronize()
    e0.record(stream)
    for _ in range(reps):
        got = s.reweighted_lnl()
    e1.record(stream)
    torch.cuda.synchronize()
    ms = e0.elapsed_time(e1) / reps
    hbm_peak, _, _ = read_peaks()
    byts = R * aln.npat * 4 + aln.npat * 8
    return {"replicates": R, "npat": aln.npat, "ms_per_call": ms,
            "replicate_lnl_evals_per_s": R / (ms * 1e-3),
            "max_rel_err_vs_fp64_dot": float(np.max(np.abs(got - ref) / np.abs(ref))),
            "roofline": {"bound": "hbm", "achieved": byts / (ms * 1e-3) / 1e9, "peak": hbm_peak,
                         "unit": "GB/s", "frac": byts / (ms * 1e-3) / 1e9 / hbm_peak}}


def codon_batch_block(local, nmodels=64, reps=3):
    """64 candidate codon models (61 states, kappa ~ U[1,5], omega ~ U[0.1,1], Dirichlet
    frequencies; +G4 and +R8) on one 200-taxon, 4,000-site alignment: one batched tcgen05
    traversal over every (model, pattern tile) plus each model's branch lnL, against one model
    in the plain FP64 form (timed alone, as the reference evaluates candidates one by one)."""
    import torch
    from gems_b200 import PhyloTree, Session, branch_lnl_batch, full_traversal, traverse_batch
    out = {}
    for freerate in (False, True):
        tree, model, aln = synth.config_codon200(nsites=4000, freerate=freerate)
        C = model.ncat
        nops = sum(op_kinds(tree))
        rng = np.random.default_rng(17 + C)
        models = [model] + [synth.codon_gy(rng, C, float(rng.uniform(0.3, 1.5)), freerate=freerate)
                            for _ in range(nmodels - 1)]
        sessions = []
        for m in models:
            s = Session(tree.ntaxa, aln.npat, 61, C, tree.ntaxa - 2, "mixed", "safe", local)
            s.upload_tips(aln.patterns)
            s.upload_patterns(aln.weights)
            s.set_model(m.eval, m.evec, m.inv_evec, m.rates, m.props)
            sessions.append(s)
        ops, br = full_traversal(tree)
        lnl = branch_lnl_batch(sessions, ops, br)  # warm-up
        torch.cuda.synchronize()
        t0 = time.perf_counter()
        for _ in range(reps):
            lnl = branch_lnl_batch(sessions, ops, br)
        wall = (time.perf_counter() - t0) / reps
        s0 = sessions[0]
        s0.profile(True)
        s0.profile_read(0)
        traverse_batch(sessions, ops)
        kms, kn = s0.profile_read(0)
        s0.profile(False)
        for s in sessions:
            s.close()
        # model 0 in FP64, alone
        g64 = PhyloTree.from_case(tree, model, aln, precision="fp64", scaling="safe", device=local)
        l64 = g64.computeLikelihood()
        stream = torch.cuda.ExternalStream(g64.session.stream_handle(), device=local)
        lnl_buf = torch.zeros(1, dtype=torch.float64, device=f"cuda:{local}")
        ms64, _, _, _ = time_lnl(g64, 3, 1, stream, None, lnl_buf)
        g64.close()
        g64.session.close()
        kinds = op_kinds(tree)
        b_ii, b_ti, b_tt = update_bytes(4, 61, C, safe=True)
        alg = nmodels * aln.npat * (kinds[0] * b_ii + kinds[1] * b_ti + kinds[2] * b_tt)
        flops = nmodels * aln.npat * nops * update_flops(61, C)
        kt = kms / max(kn, 1) * 1e-3
        hbm_peak, _, peak_src = read_peaks()
        out[f"C{C}"] = {
            "model": "codon GY 61 states " + ("+R8" if freerate else "+G4"), "npat": aln.npat,
            "roofline": {"bound": "hbm", "kernel": "batched tcgen05 traversal",
                         "achieved": alg / kt / 1e9, "peak": hbm_peak, "peak_source": peak_src,
                         "unit": "GB/s", "frac": alg / kt / 1e9 / hbm_peak,
                         "algorithmic_bytes_per_launch": alg,
                         "traffic": read_traffic("traverse_tc61_codon200.md")
                         if (C == 4 and nmodels == 64) else None},
            "compute": {"unit_used": "tcgen05 TF32 (3 products issued per credited one)",
                        "achieved_tflops": flops / kt / 1e12,
                        "algorithmic_flops_per_launch": flops},
            "models": nmodels, "batched_wall_ms": wall * 1e3,
            "batched_traversal_kernel_ms": kms / max(kn, 1),
            "models_per_s": nmodels / wall,
            "site_partial_updates_per_s": nmodels * nops * aln.npat / wall,
            "fp64_one_model_ms": ms64,
            "speedup_vs_fp64_one_by_one": nmodels * ms64 / (wall * 1e3),
            "lnl_rel_err_model0_vs_fp64": abs(lnl[0] - l64) / abs(l64)}
    return out


def ingest_block(aln, local, reps=3):
    """Alignment ingest of the headline alignment (512 taxa x 1,000,000 sites): from host
    sequences to a session ready to evaluate, by the device path (sequences cross once; encoding,
    compression, tips, weights and +I terms on the GPU) and by the host path (host compressor, C
    with OpenMP hashing, then the uploads).  Both must produce the same patterns and weights."""
    from gems_b200 import Ingest, Session
    cols = synth.expand_patterns(aln)
    ntaxa, n = cols.shape[0], aln.nstates

    def host_path():
        h = synth.compress(cols, n)
        s = Session(ntaxa, h.npat, n, 4, 1, "mixed", "norm", local)  # loading only
        s.upload_tips(h.patterns)
        s.upload_patterns(h.weights)
        return h, s

    def device_path():
        g = Ingest(cols, n, encoded=True, device=local)
        s = Session(ntaxa, g.npat, n, 4, 1, "mixed", "norm", local)
        g.to_session(s)
        return g, s

    h, s = host_path()  # warm-up
    s.close()
    g, s = device_path()
    pat, w, _, _ = g.read()
    same = bool(np.array_equal(pat, h.patterns) and np.array_equal(w, h.weights))
    g.close()
    s.close()
    t = {}
    for name, fn in (("host", host_path), ("device", device_path)):
        t0 = time.perf_counter()
        for _ in range(reps):
            a, sess = fn()
            sess.sync()
            sess.close()
            if name == "device":
                a.close()
        t[name] = (time.perf_counter() - t0) / reps
    return {"ntaxa": int(ntaxa), "sites": int(cols.shape[1]), "npat": int(len(w)),
            "device_path_ms": t["device"] * 1e3, "host_path_ms": t["host"] * 1e3,
            "host_threads": os.cpu_count(), "speedup_vs_host": t["host"] / t["device"],
            "identical_to_host": same,
            "path": "host sequences -> session with tips, weights and +I terms loaded "
                    "(creation of a one-slot session included in both)"}


def serving_block(local, nsess=48, nreq=800, load=0.7, taxa=(8, 256), sites=(500, 50_000)):
    """The serving loop on a seeded stream: sessions of 8-256 taxa and 500-50,000 sites
    (log-uniform), 4/20/61 states, 1/4/8 categories, FP64/mixed; per request an NNI with Newton
    on the 5 branches around it, or (30%) an SPR with Newton on 4 branches, then the lnL.  Passes
    over the same stream, sessions opened before each: every request queued at once gives the
    capacity; Poisson arrivals at `load` and at half of the capacity give the request latency.
    Session open times (create, upload, first full lnL) are reported apart."""
    import torch
    from gems_b200 import serve
    kw = dict(seed=5, taxa=taxa, sites=sites)
    specs, reqs = serve.make_stream(nsess, nreq, 1.0, **kw)
    cases = {sp.sid: serve.build_case(sp) for sp in specs}
    torch.cuda.empty_cache()
    free_gb = torch.cuda.mem_get_info(local)[0] / 1e9
    srv = serve.Server(device=local, workers=16)
    # untimed warm-up over the first quarter of the stream: a running server has loaded its
    # kernels and tuned its launch shapes before the requests measured here arrive
    srv.run(specs, cases, [(0.0, sid) for _, sid in reqs[: max(1, nreq // 4)]], preopen=True)
    records, wall = srv.run(specs, cases, [(0.0, sid) for _, sid in reqs], preopen=True)
    cap = serve.summarize(records, wall, specs, cases)
    opened = np.array(srv.open_ms)
    rate = load * cap["throughput_req_s"]
    _, reqs = serve.make_stream(nsess, nreq, rate, **kw)
    records, wall = srv.run(specs, cases, reqs, preopen=True)
    out = serve.summarize(records, wall, specs, cases)
    # the same stream at half the capacity (per-session order serialises a session's requests,
    # so the open-loop capacity is below the closed-loop one)
    _, reqs = serve.make_stream(nsess, nreq, 0.5 * cap["throughput_req_s"], **kw)
    rec5, wall5 = srv.run(specs, cases, reqs, preopen=True)
    half = serve.summarize(rec5, wall5, specs, cases)
    out["at_half_capacity"] = {"offered_rate_req_s": 0.5 * cap["throughput_req_s"],
                               "throughput_req_s": half["throughput_req_s"],
                               "latency_ms": half["latency_ms"], "failed": half["failed"]}
    out.update({"capacity_req_s": cap["throughput_req_s"], "capacity_failed": cap["failed"],
                "capacity_rejected": cap["rejected"], "capacity_wall_s": cap["wall_s"],
                "offered_rate_req_s": rate, "load": load,
                "session_open_ms": {"p50": float(np.percentile(opened, 50)),
                                    "p99": float(np.percentile(opened, 99)),
                                    "max": float(opened.max())},
                "sessions": nsess, "workers": 16, "free_gb_at_start": free_gb,
                "budget_gb": srv.budget / 1e9, "pool_admissions": srv.pool_admissions,
                "evictions": srv.evictions,
                "stream": f"seeded; taxa {taxa[0]}-{taxa[1]}, sites {sites[0]:,}-{sites[1]:,} "
                          "(log-uniform), states {4,20,61}, categories {1,4,8}, fp64/mixed; "
                          "request = NNI + Newton on the 5 branches around it, or (30%) SPR "
                          "within radius 3 + Newton on 4 branches, then lnL; latency at "
                          "Poisson arrivals; sessions that fit the HBM budget opened first, the "
                          "others admitted as memory frees"})
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="gems", choices=["gems", "reference"])
    ap.add_argument("--sites", type=int, default=None)
    ap.add_argument("--config", default="dna512", choices=sorted(CONFIGS))
    ap.add_argument("--precision", default="both", choices=["fp64", "mixed", "both"])
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-extras", action="store_true",
                    help="skip the Newton timing and the protein comparison")
    ap.add_argument("--block", choices=["protein20", "codon64", "serving", "serving_full"],
                    default=None,
                    help="run only this block of the line and print it (profiling runs)")
    ap.add_argument("--codon-models", type=int, default=64,
                    help="candidate codon models in the batched block (small for profiling)")
    ap.add_argument("--e2e-chunks", type=int, default=16,
                    help="pattern chunks of the overlapped tip upload in the e2e measurement")
    ap.add_argument("--no-tc", action="store_true",
                    help="20-state mixed traversal on CUDA cores instead of tcgen05")
    ap.add_argument("--traversal-shape", type=int, default=None,
                    help="force shape k of the 4-state traversal's list instead of tuning "
                         "(profiling runs: the captured kernel is then known in advance)")
    args = ap.parse_args()
    if args.sites is None:
        args.sites = NSITES if args.config == "dna512" else 100_000
    if args.impl == "reference":
        return run_reference(args)

    import torch
    from gems_b200 import PhyloTree
    rank, world, local = env_rank()
    torch.cuda.set_device(local)
    if args.block is not None:
        from gems_b200 import measure_peaks
        fn = {"protein20": lambda: protein_comparison(args, local, measure_peaks(local)),
              "codon64": lambda: codon_batch_block(local, args.codon_models),
              "serving": lambda: serving_block(local),
              # the full serving stream: 200 sessions, 20,000 requests, up to 1024 taxa and
              # 500,000 sites (minutes; not part of the default line)
              "serving_full": lambda: serving_block(local, 200, 20_000, taxa=(8, 1024),
                                                    sites=(500, 500_000))}[args.block]
        print(json.dumps({args.block: fn()}), flush=True)
        return
    dist = None
    if world > 1:
        import datetime
        import torch.distributed as dist
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=120))

    from gems_b200 import measure_peaks
    peaks = measure_peaks(local)
    tree, model, aln = make_workload(rank, args.sites, args.config)
    kinds = op_kinds(tree)
    nops = sum(kinds)
    P = aln.npat
    lnl_buf = torch.zeros(1, dtype=torch.float64, device=f"cuda:{local}")
    hbm_peak, _, peak_src = read_peaks()
    precisions = ["fp64", "mixed"] if args.precision == "both" else [args.precision]
    forms = {}
    keep = None
    with Clocks(local) as clk:
        for prec in precisions:
            gt = PhyloTree.from_case(tree, model, aln, precision=prec, device=local)
            if args.no_tc:
                gt.session.set_tensor_cores(False)
            if args.traversal_shape is not None:
                gt.session.set_autotune(False, force_shape=args.traversal_shape)
            stream = torch.cuda.ExternalStream(gt.session.stream_handle(), device=local)
            ms, lnl, kms, launches = time_lnl(gt, args.steps, args.warmup, stream, dist, lnl_buf)
            s_bytes = 8 if prec == "fp64" else 4
            b_ii, b_ti, b_tt = update_bytes(s_bytes, model.nstates, model.ncat)
            alg = P * (kinds[0] * b_ii + kinds[1] * b_ti + kinds[2] * b_tt)
            ach = alg / (kms * 1e-3) / 1e9
            req = required_bytes(P, nops, tree.ntaxa, s_bytes, model.nstates, model.ncat)
            forms[prec] = {
                "ms_per_step": ms, "value": world * nops * P / (ms * 1e-3), "lnl": lnl,
                "gpu_launches": launches,
                "roofline": {"bound": "hbm", "kernel": "traversal (one launch per step)",
                             "achieved": ach, "peak": hbm_peak,
                             "peak_source": peak_src, "unit": "GB/s", "frac": ach / hbm_peak,
                             "algorithmic_bytes_per_launch": alg, "avg_launch_ms": kms,
                             "traffic": read_traffic(f"traverse_{prec}_{args.config}.md"),
                             "required_bytes_per_launch": req,
                             "frac_required_bytes": req / (kms * 1e-3) / 1e9 / hbm_peak},
            }
            pp, blocks, tuned = gt.session.traversal_shape()
            forms[prec]["launch_shape"] = {"patterns_per_lane_group": pp, "blocks_per_sm": blocks,
                                           "tuned": tuned}
            if not args.no_extras and rank == 0:
                forms[prec]["newton"] = time_newton(gt, tree, stream)
            if keep is not None:
                keep[0].close()
                keep[0].session.close()
            keep = (gt, stream, prec)
    fp = forms.get("fp64")
    mx = forms.get("mixed")
    head = "fp64"
    if mx is not None and fp is not None:
        err = abs(mx["lnl"] - fp["lnl"]) / abs(fp["lnl"])
        mx["lnl_rel_err_vs_fp64"] = err
        if err <= MIXED_RTOL:
            head = "mixed"
    elif mx is not None:
        head = "mixed"
    H = forms[head]

    # end to end through the public API from pinned host buffers, on the headline form
    gt, stream, prec = keep
    if prec != head:
        gt.close()
        gt.session.close()
        gt = PhyloTree.from_case(tree, model, aln, precision=head, device=local)
        stream = torch.cuda.ExternalStream(gt.session.stream_handle(), device=local)
    s = gt.session
    pin_pat = torch.empty(aln.patterns.shape, dtype=torch.uint8, pin_memory=True)
    pin_w = torch.empty(aln.weights.shape, dtype=torch.float64, pin_memory=True)
    pin_plh = torch.empty(P, dtype=torch.float64, pin_memory=True)
    pat_host, w_host, plh_host = pin_pat.numpy(), pin_w.numpy(), pin_plh.numpy()
    pat_host[:] = aln.patterns
    w_host[:] = aln.weights
    h2d = pat_host.nbytes + w_host.nbytes
    d2h = 8 * P + 8
    e2, e3 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    for _ in range(args.warmup):  # also creates the call's copy stream, events and pinned word
        gt.computeLikelihoodFromHost(pat_host, w_host, chunks=args.e2e_chunks, pattern_lh=plh_host)
    torch.cuda.synchronize()
    e2.record(stream)
    for _ in range(args.steps):
        gt.computeLikelihoodFromHost(pat_host, w_host, chunks=args.e2e_chunks, pattern_lh=plh_host)
    e3.record(stream)
    torch.cuda.synchronize()
    ms_e2e = e2.elapsed_time(e3) / args.steps
    t = torch.tensor([ms_e2e], dtype=torch.float64, device=f"cuda:{local}")
    if dist is not None:
        dist.all_reduce(t, op=dist.ReduceOp.MAX)
    ms_e2e = float(t.item())
    # the floor the upload sets: a plain copy of the same host bytes (pinned) to the device, on
    # a stream torch owns (the pinned allocator records the streams its buffers were copied on,
    # and the session's stream is destroyed when the session closes)
    dev_pat = torch.empty(aln.patterns.shape, dtype=torch.uint8, device=f"cuda:{local}")
    dev_w = torch.empty(aln.weights.shape, dtype=torch.float64, device=f"cuda:{local}")
    cs = torch.cuda.Stream(device=local)
    with torch.cuda.stream(cs):
        for _ in range(2):
            dev_pat.copy_(pin_pat, non_blocking=True)
            dev_w.copy_(pin_w, non_blocking=True)
        e2.record(cs)
        for _ in range(args.steps):
            dev_pat.copy_(pin_pat, non_blocking=True)
            dev_w.copy_(pin_w, non_blocking=True)
        e3.record(cs)
    torch.cuda.synchronize()
    ms_h2d = e2.elapsed_time(e3) / args.steps
    del dev_pat, dev_w
    rell = rell_block(gt, aln, stream) if (rank == 0 and not args.no_extras) else None
    gt.close()
    s.close()

    line = {
        "metric": "site-partial updates/s", "value": H["value"],
        "unit": "site-partial updates/s", "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": H["ms_per_step"], "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None,
        "dtype": "f64" if head == "fp64" else "f32 partials + f64 branch terms",
        "data": "synthetic (seeded generator; no public dataset)",
        "config": {**config_block(args, aln, nops), "precision": head},
        "lnl_evals_per_s": 1.0 / (H["ms_per_step"] * 1e-3), "lnl": H["lnl"],
        "gpu_launches": H["gpu_launches"],
        "e2e": {"value": world * nops * P / (ms_e2e * 1e-3), "unit": "site-partial updates/s",
                "h2d_bytes_per_step": h2d, "d2h_bytes_per_step": d2h, "ms_per_step": ms_e2e,
                "upload_chunks": args.e2e_chunks, "h2d_copy_alone_ms": ms_h2d,
                "h2d_copy_alone_gbs": h2d / (ms_h2d * 1e-3) / 1e9},
        "roofline": H["roofline"],
        "forms": forms,
        "clocks": clk.summary(),
        "peaks_measured": peaks,
    }
    if rell is not None:
        line["rell"] = rell
    # single-GPU blocks and the CPU baseline: one GPU only (under torchrun the other ranks would
    # wait for them at the closing barrier)
    if world == 1 and not args.no_extras and args.config == "dna512":
        line["protein20"] = protein_comparison(args, local, peaks)
        line["codon64"] = codon_batch_block(local, args.codon_models)
        line["ingest"] = ingest_block(aln, local)
        line["serving"] = serving_block(local)
    if world == 1 and not args.no_cpu:
        sub = cpu_sample(model, aln)
        line["parity"] = slice_parity(tree, model, sub, local)
        line["cpu_baseline"] = cpu_baseline(tree, model, aln, sub=sub)
    if rank == 0:
        # the full record first (stderr), then the one compact line the driver parses (stdout)
        print(json.dumps({"detail": line}), file=sys.stderr, flush=True)
        print(json.dumps(compact_line(line)), flush=True)
    if dist is not None:
        dist.barrier()
        dist.destroy_process_group()


if __name__ == "__main__":
    main()
