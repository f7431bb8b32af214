"""Benchmark of the RPD hot path on one GB300 (or N replicas).

Metric: RPD cells/sec -- one cell is one emitted (tet, site) restricted
convex cell, the unit of libmat's ConvexCellHost -- on the 1M-tet ellipsoid
workload (jittered-grid Delaunay ellipsoid, semi-axes 1.0/0.6/0.4, ~1M tets;
50,000 sites, 70% near the surface, radii lognormal(ln 0.01, 0.5)), seeded
synthetic data generated here.  One step = one rpd_compute: GPU kNN (k = 64),
candidate pairs by the reference's rule, clipping, compaction, from
device-resident mesh and sites to device-resident compact cells.

  value   fast path: FP32 filter + FP64 fallback predicates (reference signs),
          neighbours in ascending bisector distance with the security-radius
          certificate, first-pass list lengths chosen by the autotuner among
          16 / 32 / all neighbours and the k-predictor trained here (untimed
          set-up: 200k labelled cells of two meshes with other seeds)
  plain   the plain FP64 path: FP64 determinant on every predicate
  e2e     the fast path through the C ABI with host buffers: mesh + sites
          host->device, compute, every cell device->host, per step; two
          contexts, one host thread each, a step's copy back overlapping
          the other context's compute ("serial": one context, blocking copy)
  cpu_baseline / --impl reference: the oracle (CPU restatement of the
          reference's clipper and candidate rule, all host cores) on a
          bounded sample of the same workload's tets

    python bench.py [--gpus N] [--steps K] [--warmup W] [--impl reference]
"""
import argparse
import json
import os
import subprocess
import sys
import threading
import time

import numpy as np

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

METRIC = "RPD cells/sec at 1M tets (learned-k + FP32 filter vs plain FP64), exact topology"
UNIT = "cells/s"


def load_peaks():
    p = os.path.join(ROOT, "MEASURED_PEAKS.json")
    if os.path.exists(p):
        d = json.load(open(p))
        return float(d["hbm_gbs"]), "measured"
    return 6800.0, "fallback"


def compare_topology(ph_fast, hash_fast, ph_plain, hash_plain):
    """Cells of a fast run against the plain FP64 path's, pair by pair:
    canonical topology of the cells both emit, statuses elsewhere.  The
    reference's fixed capacities (64 planes, 96 vertices, 152 edges) drop
    cells whose clipping in site-id order overflows them; clipping in
    ascending bisector distance builds fewer intermediate vertices and edges
    and can emit those cells -- counted apart, not as differences."""
    assert np.array_equal(ph_fast["tet_id"], ph_plain["tet_id"])
    assert np.array_equal(ph_fast["site_id"], ph_plain["site_id"])
    sf, sp = ph_fast["status"], ph_plain["status"]
    both = (sf == 4) & (sp == 4)
    overflow = np.isin(sp, [0, 1, 7]) & (sf == 4)
    # a different emitted set, apart from the capacity drops above
    other = ((sf == 4) != (sp == 4)) & ~overflow
    n_topo = int((hash_fast[both] != hash_plain[both]).sum())
    kinds = {}
    for a_, b_ in zip(sp[sf != sp], sf[sf != sp]):
        key = "plain %d / fast %d" % (a_, b_)
        kinds[key] = kinds.get(key, 0) + 1
    return {"topology_bit_exact": bool(n_topo == 0 and not other.any()),
            "cells_topology_differing": n_topo, "emitted_set_differing": int(other.sum()),
            "status_differing_kinds": kinds,
            "reference_capacity_drops_emitted": int(overflow.sum())}


def replica_throughput(local_ms, local_cells, dist=None, device="cpu"):
    """Whole-job throughput of N replicas: cells of all ranks over the slowest
    rank's time (max over ranks, as the timing rules ask).  Returns (cells/s,
    max ms, total cells)."""
    if dist is None:
        return local_cells / (local_ms / 1000.0), local_ms, local_cells
    import torch

    t = torch.tensor([local_ms], dtype=torch.float64, device=device)
    n = torch.tensor([local_cells], dtype=torch.float64, device=device)
    dist.all_reduce(t, op=dist.ReduceOp.MAX)
    dist.all_reduce(n, op=dist.ReduceOp.SUM)
    return float(n.item()) / (float(t.item()) / 1000.0), float(t.item()), int(n.item())


def make_workload(args):
    from libmat_gb300 import workloads as W

    t0 = time.time()
    if args.config == "small":
        cfg = W.config_small_cube()
        name = "cube_20x20x20x6_48k_tets_2k_sites"
    elif args.config == "lattice":
        cfg = W.config_lattice(n=args.lattice_n, m=args.lattice_m)
        name = "lattice_%d^3_points_%d^3_sites_5pct_perturbed_1e-12" % (args.lattice_n,
                                                                       args.lattice_m)
    else:
        cfg = W.config_ellipsoid(target_tets=args.tets, n_site=args.sites, seed=2)
        name = "ellipsoid_%dk_tets_%dk_sites" % (round(args.tets / 1000), round(args.sites / 1000))
    return cfg, name, time.time() - t0


class ClockSampler:
    """nvidia-smi clocks and throttle reasons sampled during the timed region."""
    FIELDS = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,"
              "clocks_event_reasons.hw_slowdown,clocks_event_reasons.hw_thermal_slowdown,"
              "clocks_event_reasons.sw_thermal_slowdown,clocks_event_reasons.sw_power_cap")

    def __init__(self, device):
        self.device = device
        self.proc = None
        self.lines = []

    def __enter__(self):
        try:
            self.proc = subprocess.Popen(
                ["nvidia-smi", "-i", str(self.device), "--query-gpu=" + self.FIELDS,
                 "--format=csv,noheader,nounits", "-lms", "200"],
                stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
            self.t = threading.Thread(target=self._read, daemon=True)
            self.t.start()
        except Exception:
            self.proc = None
        return self

    def _read(self):
        for line in self.proc.stdout:
            self.lines.append(line.strip())

    def __exit__(self, *a):
        if self.proc:
            self.proc.terminate()
            try:
                self.proc.wait(timeout=5)
            except Exception:
                self.proc.kill()

    def summary(self):
        sm, mx, reasons = [], None, set()
        names = ["hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap"]
        for ln in self.lines:
            f = [x.strip() for x in ln.split(",")]
            if len(f) < 9:
                continue
            try:
                sm.append(float(f[1]))
                mx = float(f[2])
            except ValueError:
                continue
            for n, v in zip(names, f[5:9]):
                if v.lower() == "active":
                    reasons.add(n)
        if not sm:
            return {"sm_mhz": None, "sm_max_mhz": None, "reasons": ["unsampled"]}
        return {"sm_mhz": float(np.median(sm)), "sm_max_mhz": mx, "reasons": sorted(reasons),
                "samples": len(sm)}


def flush_l2(device_sync=True):
    """Writes 256 MB (> 129 MB L2) on the device between timed steps; waits
    for the whole device, or (device_sync=False) only for the write itself,
    so that copies in flight on the engines' streams keep running."""
    import torch

    if not hasattr(flush_l2, "buf"):
        flush_l2.buf = torch.empty(64 << 20, dtype=torch.int32, device="cuda")
    flush_l2.buf.fill_(1)
    if device_sync:
        torch.cuda.synchronize()
    else:
        torch.cuda.current_stream().synchronize()


def clip_algorithmic_bytes(cfg, n_pairs, k, topo_bytes):
    """Bytes the clip kernel must move at least once per launch: the mesh
    (float vertices, tets, face counts / ids, edge counts, vertex counts),
    the float sites, the distance-ordered lists and their keys, the pair
    list, the per-pair headers and the topology part of the emitted records
    (planes, plane ids, dual triangles, edges, face counts; the FP64
    coordinates are the epilogue kernel's)."""
    nv, nt, ns = cfg["vert3d"].shape[0], cfg["tets"].shape[0], cfg["sites"].shape[0]
    mesh = 12 * nv + 16 * nt + 32 * nt + 6 * nt + 4 * nv
    sites = 16 * ns
    return mesh + sites + 8 * k * ns + 8 * n_pairs + 32 * n_pairs + topo_bytes


# The first clipping pass by lanes (FP32-filter or exact predicates, whole base
# lists, at least CLIP_LANE_PAIRS pairs: kThreadsPairs of rpd_clip_thread.cu):
# DRAM traffic per candidate pair of its two launches -- ncu
# dram__bytes_read.sum + dram__bytes_write.sum of clip_threads_kernel and of
# clip_cells_kernel on the cells that go back, 200k-tet ellipsoid (the same
# workload family, scaled by the pass's pairs: its traffic grows with them) --
# and smsp__issue_active and threads per instruction of the first, from the same
# capture; its command is in profiles/clip_threads_kernel_ellipsoid_200k.md
CLIP_LANE_PAIRS = 20000
CLIP_DRAM_BYTES_PER_PAIR = 309.4
CLIP_ISSUE_ACTIVE = 0.518
CLIP_THREADS_PER_INST = 14.20


def clip_pass(n_pairs, shortened):
    """The kernels of a first clipping pass (ms_clip_kernel) and what was
    captured of them: counters for the lanes' kernels, none for the others."""
    if shortened or n_pairs < CLIP_LANE_PAIRS:
        return {"kernel": "clip_cells_kernel", "traffic": None, "issue_active_frac": None,
                "threads_per_inst": None}
    return {"kernel": "clip_threads_kernel + clip_cells_kernel",
            "traffic": CLIP_DRAM_BYTES_PER_PAIR * n_pairs,
            # what bounds it instead of HBM: instruction issue and latency
            # (of clip_threads_kernel)
            "issue_active_frac": CLIP_ISSUE_ACTIVE, "threads_per_inst": CLIP_THREADS_PER_INST}


def sample_tets(n_tet, n, seed):
    rng = np.random.default_rng(seed)
    return np.sort(rng.choice(n_tet, size=min(n, n_tet), replace=False))


def cpu_sample_run(cfg, adj, nbr, n_tets, seed=0, n_threads=None, clip_nbr=None):
    """The oracle on n_tets random tets: the reference's candidate rule over
    all sites with the lists nbr (brute force, as the reference) + clipping
    with FP64 predicates, with the lists clip_nbr (default nbr).  Returns
    (cells, seconds, pairs, details)."""
    from oracle import oracle as O

    sub = sample_tets(cfg["tets"].shape[0], n_tets, seed)
    tets = cfg["tets"][sub]
    mesh = dict(vert3d=cfg["vert3d"], tets=tets, v_adjs=adj["v_adjs"],
                e_adj6=adj["e_adj6"][sub], f_adjs=adj["f_adjs"][sub], f_ids=adj["f_ids"][sub])
    t0 = time.perf_counter()
    offs, ps = O.candidate_pairs(cfg["vert3d"].astype(np.float32), tets,
                                 cfg["sites"].astype(np.float32), cfg["flags"], nbr,
                                 n_threads=n_threads)
    h, p, _ = O.clip_cells(mesh, cfg["sites"], nbr if clip_nbr is None else clip_nbr, offs, ps,
                           pred_mode=0, n_threads=n_threads)
    dt = time.perf_counter() - t0
    return int((h["status"] == 4).sum()), dt, int(offs[-1]), dict(sub=sub, offs=offs, ps=ps, h=h,
                                                                  p=p)


def parity_vs_oracle(cfg, adj, base_nbr, final_nbr, gpu_offs, gpu_ps, gpu_ph, gpu_hash, gpu_p,
                     n_tets, seed=0):
    """The fast path's cells on a sample of tets against the oracle's (the
    reference's algorithm, FP64 predicates) with the same lists: the
    candidate pairs by the reference rule on the base lists, and every cell
    clipped with the list the GPU finally used for its site (its exact-lists
    extension where it got one).  Pairs and statuses compared one for one,
    emitted cells by their canonical topology (the certified path clips in
    ascending key and records fewer dead planes), FP64 vertices (as sorted
    rows) and volumes against the oracle's FP64 reconstruction.  Returns
    (report, cells, seconds)."""
    from oracle import oracle as O

    c, dt, npairs, d = cpu_sample_run(cfg, adj, base_nbr, n_tets, seed=seed, clip_nbr=final_nbr)
    sub, offs, ps, oh, op = d["sub"], d["offs"], d["ps"], d["h"], d["p"]
    # the GPU's pairs of the sampled tets, in the same CSR order
    idx = np.concatenate([np.arange(gpu_offs[t], gpu_offs[t + 1]) for t in sub]).astype(np.int64)
    pairs_equal = bool(np.array_equal(np.diff(offs), np.diff(gpu_offs)[sub]) and
                       np.array_equal(ps, gpu_ps[idx]))
    rep = {"sample_tets": int(len(sub)), "pairs": int(npairs), "pairs_equal": pairs_equal}
    if not pairs_equal:
        return rep, c, dt
    gh = gpu_ph[idx]
    rep["status_differing"] = int((gh["status"] != oh["status"]).sum())
    ok = (gh["status"] == 4) & (oh["status"] == 4)
    ohash = O.topology_hashes(oh, op)
    rep["cells_compared"] = int(ok.sum())
    rep["cells_topology_differing"] = int((ohash[ok] != gpu_hash[idx][ok]).sum())
    vmax = vsq = 0.0
    vn = 0
    wmax = wsq = 0.0
    nw = 0
    tmax = 0.0
    tv = cfg["vert3d"][cfg["tets"][sub].astype(np.int64)]
    tvol = np.abs(np.einsum("ij,ij->i", np.cross(tv[:, 1] - tv[:, 0], tv[:, 2] - tv[:, 0]),
                            tv[:, 3] - tv[:, 0])) / 6.0
    pair_tvol = np.repeat(tvol, np.diff(offs))
    for j in np.flatnonzero(ok):
        q = idx[j]
        a = _xyz(gpu_p, gpu_ph, q)
        b = _xyz(op, oh, j)
        if a.shape != b.shape:
            continue
        a = a[np.lexsort(a.T[::-1])]
        b = b[np.lexsort(b.T[::-1])]
        dv = np.abs(a - b) / 1000.0  # relative to the coordinate scale (libmat's [0, 1000])
        vmax = max(vmax, float(dv.max()))
        vsq += float((dv * dv).sum())
        vn += dv.size
        dvol = abs(gh["volume"][j] - oh["volume"][j])
        tmax = max(tmax, dvol / pair_tvol[j])
        # relative error of the cells that hold at least 1e-6 of their tet
        # (below, the FP64 volume of a cell whose topology the float planes
        # decide is itself at the level of the coordinates' rounding)
        if abs(oh["volume"][j]) >= 1e-6 * pair_tvol[j]:
            rv = dvol / abs(oh["volume"][j])
            wmax = max(wmax, rv)
            wsq += rv * rv
            nw += 1
    rep.update({"vertex_max_rel": vmax, "vertex_rms_rel": (vsq / max(vn, 1)) ** 0.5,
                "volume_max_rel": wmax, "volume_rms_rel": (wsq / max(nw, 1)) ** 0.5,
                "volume_cells": nw, "volume_max_err_of_tet": tmax})
    return rep, c, dt


def true_rpd_check(cfg, adj, rpd, fast_ph, fast_hash):
    """The fast path's cells against the exact restricted power diagram: the
    oracle's power neighbours of every site (the stand-in for libmat's
    regular triangulation, exact signs) clipped by the engine's reference
    path (user lists in site-id order, as libmat runs them; hidden spheres
    unflagged, as libmat's is_rt_valid).  Cells compared by (tet, site) and
    canonical topology."""
    from oracle import oracle as O

    t0 = time.perf_counter()
    s4 = cfg["sites"].astype(np.float32)
    v = cfg["vert3d"]
    nbr, cnt = O.power_neighbors(s4, v.min(0), v.max(0), max_nbr=256)
    pn_s = time.perf_counter() - t0
    k = max(int(cnt.max()), 1)
    flags = cfg["flags"].copy()
    flags[cnt < 0] = 0
    with rpd.RPD(predicate_mode=rpd.PRED_FP32_FILTER, neighbor_source=rpd.NEIGH_USER,
                 topology_hash=True) as r:
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], flags)
        r.set_neighbors(np.ascontiguousarray(nbr[:, :k]))
        r.compute()
        ph = r.pair_headers()
        hs = r.topology_hashes()

    def keyed(h, hh):
        ok = h["status"] == rpd.SUCCESS
        key = (h["tet_id"][ok].astype(np.int64) << 32) | h["site_id"][ok].astype(np.int64)
        o = np.argsort(key)
        return key[o], hh[ok][o]

    ka, ha = keyed(fast_ph, fast_hash)
    kb, hb = keyed(ph, hs)
    common, ia, ib = np.intersect1d(ka, kb, assume_unique=True, return_indices=True)
    n_topo = int((ha[ia] != hb[ib]).sum())
    # cells the reference's capacities (64 planes, 96 vertices, 152 edges)
    # drop when it clips in site-id order, and the fast path emits
    drop = np.isin(ph["status"], [0, 1, 7])
    kd = (ph["tet_id"][drop].astype(np.int64) << 32) | ph["site_id"][drop].astype(np.int64)
    extra = np.setdiff1d(ka, common, assume_unique=True)
    n_drop = int(np.isin(extra, kd).sum())
    return {"cells": int(len(ka)), "reference_cells": int(len(kb)),
            "cells_missing": int(len(kb) - len(common)), "cells_extra": int(len(extra) - n_drop),
            "reference_capacity_drops_emitted": n_drop,
            "cells_topology_differing": n_topo,
            "true_rpd_differing": int(len(kb) - len(common) + len(extra) - n_drop + n_topo),
            "hidden_sites": int((cnt == -1).sum()), "capacity_sites": int((cnt < -1).sum()),
            "power_neighbours_mean": float(cnt[cnt >= 0].mean()),
            "power_neighbours_s": round(pn_s, 2)}


def run_reference(args):
    """--impl reference: the reference's CPU path restated (oracle port; the
    reference's own clipper builds only where its sources are, not on the GPU
    machines), all host threads, bounded sample per step."""
    from libmat_gb300 import workloads as W  # noqa: F401
    from oracle import oracle as O

    rank = int(os.environ.get("RANK", "0"))
    if rank != 0:
        return
    cfg, name, gen_s = make_workload(args)
    adj = O.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    nbr, _ = O.knn(cfg["sites"].astype(np.float32), args.k)
    nbr = np.sort(nbr, axis=1)
    cores = O.nthreads()
    sample = args.ref_sample
    for w in range(args.warmup):
        cpu_sample_run(cfg, adj, nbr, max(sample // 8, 100), seed=100 + w)
    cells = 0
    secs = 0.0
    for s in range(args.steps):
        c, dt, _, _ = cpu_sample_run(cfg, adj, nbr, sample, seed=s)
        cells += c
        secs += dt
    v = cells / secs
    line = {
        "impl": "reference", "metric": METRIC, "value": v, "unit": UNIT, "n_gpus": args.gpus,
        "steps": args.steps, "warmup": args.warmup, "ms_per_step": 1000 * secs / args.steps,
        "higher_is_better": True, "scaling": "weak", "vs_baseline": None, "dtype": "fp32+fp64",
        "data": "synthetic (seeded)",
        "config": {"workload": name, "n_tet": int(cfg["tets"].shape[0]),
                   "n_site": int(cfg["sites"].shape[0]), "knn_k": args.k},
        "cpu_baseline": {"value": v, "unit": UNIT, "cores": cores, "kind": "port",
                         "sample": "%d random tets per step: reference candidate rule over all "
                                   "sites + clipping (FP64 predicates)" % sample},
        "e2e": {"value": v, "unit": UNIT, "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
    }
    print(json.dumps(line))


def train_predictor(args, r, rpd, W):
    """Untimed set-up of the learned list length: labelled cells (the
    certifying list length of every cell of the plain method) from training
    meshes of the same distribution with other seeds, then training on the
    GPU with the engine's own kernels.  Leaves the engine on the training
    set's last mesh; the caller loads the evaluation inputs."""
    t0 = time.time()
    n = 0
    per = args.train_cells // len(args.train_seeds)
    for seed in args.train_seeds:
        tc = W.config_ellipsoid(target_tets=args.tets, n_site=args.sites, seed=seed)
        ta = rpd.mesh_adjacency(tc["vert3d"].shape[0], tc["tets"])
        r.set_mesh(tc["vert3d"], tc["tets"], ta["v_adjs"], ta["e_adj6"], ta["f_adjs"], ta["f_ids"])
        r.set_sites(tc["sites"], tc["flags"])
        n = r.mlp_collect(per)
    rep = r.mlp_train(epochs=args.epochs, batch=512, lr=2e-3, miss_target=args.miss_target,
                      seed=7)
    return {"samples": int(n), "train_meshes": ["ellipsoid seed %d" % s for s in args.train_seeds],
            "report": rep.as_dict(), "setup_s": round(time.time() - t0, 2)}


def _clip_ms(r, reps=3):
    ts, st = [], None
    for _ in range(reps):
        st = r.compute()
        ts.append(st.ms_clip)
    return float(np.median(ts)), st


def run_ours(args):
    from libmat_gb300 import rpd
    from libmat_gb300 import workloads as W

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))
    dist = None
    if world > 1:
        import torch
        import torch.distributed as tdist

        torch.cuda.set_device(local)
        tdist.init_process_group("nccl" if torch.cuda.is_available() else "gloo")
        dist = tdist

    def barrier():
        if dist is not None:
            dist.barrier()

    cfg, name, gen_s = make_workload(args)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    nt, nv, ns = cfg["tets"].shape[0], cfg["vert3d"].shape[0], cfg["sites"].shape[0]

    def load(r):
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])

    def engine(pred, certify, k=None):
        r = rpd.RPD(device=local if world > 1 else 0, predicate_mode=pred,
                    neighbor_source=rpd.NEIGH_KNN, knn_k=k or args.k,
                    clip_order=rpd.ORDER_SITE_ID, certify=certify)
        load(r)
        return r

    def timed(r, steps, warmup):
        for _ in range(warmup):
            r.compute()
        ms, cells, st_last = [], 0, None
        for _ in range(steps):
            flush_l2()
            barrier()
            st = r.compute()
            ms.append(st.ms_total)
            cells += st.n_cells
            st_last = st
        return ms, cells, st_last

    # ---- fast path (the metric): FP32-filter predicates, neighbours in
    # ascending bisector distance, the security-radius certificate, and the
    # learned per-cell list length trained here (untimed set-up)
    fast = rpd.RPD(device=local if world > 1 else 0, predicate_mode=rpd.PRED_FP32_FILTER,
                   neighbor_source=rpd.NEIGH_KNN, knn_k=args.k, clip_order=rpd.ORDER_SITE_ID,
                   certify=True)
    learned = None
    if not args.no_learned:
        learned = train_predictor(args, fast, rpd, W)
    load(fast)
    # the project's autotuner picks the clip kernel's block size, register
    # (and so shared-memory) budget and the first-pass list length (16, 32,
    # all neighbours, or the predictor's per-cell lengths) on this workload
    tuning = fast.autotune(repeats=1).as_dict() if not args.no_tune else None
    if args.force_learned and learned is not None:
        fast.mlp_enable(True)
    fast.configure(topology_hash=0)  # a validation aid, not part of the path
    barrier()
    with ClockSampler(local) as clk:
        ms, cells, st = timed(fast, args.steps, args.warmup)
    value, total_ms, _ = replica_throughput(sum(ms), cells, dist, "cuda")
    used_learned = bool(fast.config().learned_k)

    # ---- validation run of the same configuration with topology hashes
    fast.configure(topology_hash=1)
    fast.compute()
    fast_ph = fast.pair_headers()
    fast_hash = fast.topology_hashes()
    fast_h, fast_p = fast.cells()
    final_lists = fast.site_lists_padded(ns)
    base_lists = fast.neighbor_lists(ns)
    offs_g, ps_g = fast.pairs(nt)
    # ---- per-cell topology of the emitted cells (what libmat's consumers
    # rebuild on the host: active planes and edges, face cycles, Euler
    # numbers), on the device; reported beside the step, not inside it
    topo_ms = sorted(fast.compute_topology() for _ in range(3))[1]
    topo_h, topo_rec = fast.topology()
    topology = {"ms": topo_ms, "cells_per_s": len(topo_h) / (topo_ms / 1000.0),
                "record_bytes": int(topo_rec.size), "flagged": int((topo_h["flags"] != 0).sum())}

    # ---- what the learned lengths do on this (unseen) mesh: clip stage
    # with them, with the certificate tested as each cell is clipped (no
    # network), and with the whole list (no certificate, no network)
    if learned is not None:
        base_cfg = fast.config()
        fast.configure(learned_k=1, topology_hash=0)
        ms_l, st_l = _clip_ms(fast)
        klen = fast.mlp_klen()
        fast.configure(learned_k=0)
        fast.set_site_k(None)
        ms_e, st_e = _clip_ms(fast)
        fast.set_pair_k(np.full(st_e.n_pairs, args.k, np.int32))
        ms_f, _ = _clip_ms(fast)
        fast.set_pair_k(None)
        fast.set_config(base_cfg)
        learned["eval"] = {
            "miss_rate": st_l.n_reclipped / max(st_l.n_pairs, 1),
            "reclipped": int(st_l.n_reclipped), "mean_list_length": float(klen.mean()),
            "const_k_same_miss_rate": learned["report"]["const_k"],
            "ms_clip_learned": ms_l, "ms_predict": st_l.ms_predict,
            "ms_clip_certificate_no_net": ms_e, "ms_clip_whole_list": ms_f,
            "used_in_timed_runs": used_learned}

    # ---- plain FP64 path: whole list in site-id order, FP64 determinant on
    # every predicate
    # (the same base lists as the fast path: its tuned k)
    plain = engine(rpd.PRED_FP64, False, k=fast.config().knn_k)
    plain_tuning = plain.autotune(repeats=1).as_dict() if not args.no_tune else None
    plain.configure(topology_hash=0)
    pms, pcells, pst = timed(plain, max(1, args.steps // 2), 1)
    plain_value = pcells / (sum(pms) / 1000.0)
    plain.configure(topology_hash=1)
    plain.compute()
    plain_ph = plain.pair_headers()
    plain_hash = plain.topology_hashes()
    plain_h, plain_p = plain.cells()
    plain.close()
    # exact topology: same pairs, statuses and canonical topology of every
    # cell (the certified path's records list fewer dead planes, so the raw
    # bytes differ; the vertices' face-key triples do not)
    cmp = compare_topology(fast_ph, fast_hash, plain_ph, plain_hash)
    topo_ok, n_topo_diff = cmp["topology_bit_exact"], cmp["cells_topology_differing"]
    geo = _geometry_error(fast_ph, fast_p, plain_ph, plain_p)

    # ---- end to end through the C ABI with host buffers, same configuration
    e2e = _e2e(args, cfg, adj, rpd, fast)

    # ---- roofline of the clip kernel
    peak, peak_src = load_peaks()
    ok = fast_ph["status"] == 4
    xyz_bytes = 24 * int(fast_ph["nb_v"][ok].astype(np.int64).sum())
    alg = clip_algorithmic_bytes(cfg, st.n_pairs, st.knn_k, st.payload_bytes - xyz_bytes)
    achieved = alg / (st.ms_clip_kernel / 1000.0) / 1e9
    shortened = used_learned or bool(tuning and tuning["k_bucket"])

    cpu = parity = true_rpd = None
    if rank == 0 and not args.no_cpu:
        from oracle import oracle as O

        # the oracle (test infrastructure) as the checker, and as the CPU
        # baseline on the same sample.  Base lists as built (site-id order,
        # -1 padded) for the candidate rule; the sites without an extension
        # clip with them in that order, the others with their extended list
        # in ascending key (as the plain FP64 path does)
        base = base_lists
        kb = base.shape[1]
        clip_lists = np.full((ns, max(kb, final_lists.shape[1])), -1, np.int32)
        clip_lists[:, :final_lists.shape[1]] = final_lists
        is_base = (final_lists >= 0).sum(axis=1) <= kb
        clip_lists[is_base] = -1
        clip_lists[is_base, :kb] = base[is_base]
        parity, c, dt = parity_vs_oracle(cfg, adj, base, clip_lists, offs_g, ps_g, fast_ph,
                                         fast_hash, fast_p, args.cpu_sample)
        cpu = {"value": c / dt, "unit": UNIT, "cores": O.nthreads(), "kind": "port",
               "sample": "%d random tets: reference candidate rule over all sites + clipping "
                         "with FP64 predicates and the GPU's final lists, oracle on all host "
                         "threads" % args.cpu_sample}
        if not args.no_true_rpd:
            true_rpd = true_rpd_check(cfg, adj, rpd, fast_ph, fast_hash)
    fast.close()
    if rank != 0:
        return
    line = {
        "metric": METRIC, "value": value, "unit": UNIT, "n_gpus": world, "steps": args.steps,
        "warmup": args.warmup, "ms_per_step": total_ms / args.steps, "higher_is_better": True,
        "scaling": "weak", "vs_baseline": None, "dtype": "fp32+fp64",
        "data": "synthetic (seeded jittered-grid Delaunay ellipsoid and sites; no dataset)",
        "config": {"workload": name, "n_tet": nt, "n_vert": nv, "n_site": ns, "knn_k": st.knn_k,
                   "n_pairs": st.n_pairs, "n_cells": st.n_cells,
                   "predicates": "fp32 filter, fp64 det when undecided",
                   "neighbours": "gpu kNN base lists (the k smallest power-bisector "
                                 "distances, k autotuned) + exact-lists rounds (sites of "
                                 "uncertified cells get every site whose key lies below the "
                                 "cells' radius bound; those cells are clipped again)",
                   "clipping": "ascending bisector distance, security-radius certificate",
                   "learned_k": used_learned, "l2": "flushed between steps (256 MB write)",
                   "parallelism": "replicas" if world > 1 else "single gpu",
                   "generation_s": round(gen_s, 2)},
        "plain": {"value": plain_value, "ms_per_step": sum(pms) / len(pms),
                  "speedup_fast_over_plain": value / world / plain_value,
                  "topology_bit_exact": bool(topo_ok), "cells_topology_differing": n_topo_diff,
                  "emitted_set_differing": cmp["emitted_set_differing"],
                  "reference_capacity_drops_emitted": cmp["reference_capacity_drops_emitted"],
                  "predicates_evaluated": int(pst.n_predicates), "tuning": plain_tuning},
        "geometry_vs_plain": geo,
        "tuning": tuning,
        "learned": learned,
        "reclipped": int(st.n_reclipped),
        # emitted cells whose certificate failed after the rounds (sites
        # beyond their list might cut them); 0 = every cell is exact
        "uncertified_cells": int(st.n_uncertified),
        "exact_lists": {"extended_sites": int(st.n_extended_sites),
                        "cells_reclipped": int(st.n_cert_reclipped),
                        "rounds": int(st.n_extend_rounds), "longest": int(st.ext_longest),
                        "ms": st.ms_extend, "ms_lists": st.ms_extend_lists},
        "parity_vs_oracle": parity,
        "true_rpd": true_rpd,
        "stage_ms": {"knn": st.ms_knn, "pairs": st.ms_pairs, "clip": st.ms_clip,
                     "clip_kernel": st.ms_clip_kernel, "epilogue": st.ms_epilogue,
                     "exact_lists": st.ms_extend, "predict": st.ms_predict,
                     "compact": st.ms_compact},
        "predicates": {"evaluated": st.n_predicates, "escalated_fp64": st.n_escalated,
                       "escalation_rate": st.n_escalated / max(st.n_predicates, 1)},
        "status_counts": {rpd.STATUS_NAMES[i]: int(st.status_counts[i]) for i in range(10)
                          if st.status_counts[i]},
        "e2e": e2e,
        "topology": topology,
        "gpu_launches": int(st.n_launches) * args.steps,
        "roofline": {"bound": "hbm", "achieved": achieved, "peak": peak, "unit": "GB/s",
                     "frac": achieved / peak, "peak_source": peak_src,
                     "algorithmic_bytes": alg, **clip_pass(st.n_pairs, shortened)},
        "cpu_baseline": cpu,
        "clocks": clk.summary(),
    }
    print(json.dumps(line))


def run_stress(args):
    """Near-degenerate predicate stress (--config lattice): lattice cube mesh,
    lattice sites with equal radii (exact ties), 5% perturbed by N(0, 1e-12).
    Measures how many predicates the FP32 filter escalates to FP64 and how
    many FP64 signs are uncertain (decided exactly in RPD_PRED_EXACT), and
    checks the FP32-filter path's topology against the FP64 path's."""
    from libmat_gb300 import rpd

    cfg, name, gen_s = make_workload(args)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])

    def engine(pred, certify=False):
        r = rpd.RPD(predicate_mode=pred, neighbor_source=rpd.NEIGH_KNN, knn_k=args.k,
                    clip_order=rpd.ORDER_SITE_ID, certify=certify)
        r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
                   adj["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        return r

    out = {}
    for label, pred, cert in (("plain_fp64", rpd.PRED_FP64, False),
                              ("fp32_filter", rpd.PRED_FP32_FILTER, False),
                              ("fp32_filter_certified", rpd.PRED_FP32_FILTER, True),
                              ("exact", rpd.PRED_EXACT, False)):
        r = engine(pred, cert)
        r.configure(topology_hash=0)
        for _ in range(args.warmup):
            r.compute()
        ms, cells = [], 0
        for _ in range(args.steps):
            st = r.compute()
            ms.append(st.ms_total)
            cells += st.n_cells
        r.configure(topology_hash=1)
        st = r.compute()
        out[label] = {"cells_per_s": cells / (sum(ms) / 1000.0), "ms_per_step": float(np.median(ms)),
                      "n_pairs": st.n_pairs, "n_cells": st.n_cells,
                      "predicates": st.n_predicates, "escalated_fp64": st.n_escalated,
                      "escalated_fraction": st.n_escalated / max(st.n_predicates, 1),
                      "fp64_uncertain_exact": st.n_fp64_uncertain,
                      "exact_fraction": st.n_fp64_uncertain / max(st.n_predicates, 1),
                      "exact_flips": st.n_exact_flips,
                      "status": r.pair_headers()["status"], "hash": r.topology_hashes()}
        r.close()
    base = out["plain_fp64"]
    for label, o in out.items():
        o["same_status_as_fp64"] = bool(np.array_equal(o["status"], base["status"]))
        o["cells_topology_differing_from_fp64"] = int((o["hash"] != base["hash"]).sum())
    for o in out.values():
        del o["status"], o["hash"]
    print(json.dumps({"workload": name, "n_tet": int(cfg["tets"].shape[0]),
                      "n_site": int(cfg["sites"].shape[0]), "knn_k": args.k,
                      "generation_s": round(gen_s, 2), "runs": out}))


def run_batch(args):
    """Batched uneven workload (--config batch): 256 independent meshes (cube
    or ellipsoid, random rotation and scale, tets log-uniform in [2k, 200k],
    sites log-uniform in [100, 20k], uniform in the volume, radii U[0.005,
    0.04]) in one batch: the per-mesh front end replayed from a CUDA graph,
    one persistent clip launch for all meshes, autotuned.  Beside it: the
    same batch with the front end launched directly, a loop of single-mesh
    computes, and the plain FP64 batch (topology reference).  Exact lists
    are on in every form (the cells are the exact restricted cells)."""
    from libmat_gb300 import rpd
    from libmat_gb300 import workloads as W

    t0 = time.time()
    ms = W.config_batch(n_mesh=args.batch_meshes, seed=3)
    for cfg in ms:
        cfg["adj"] = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    gen_s = time.time() - t0
    n_tet = sum(m["tets"].shape[0] for m in ms)
    n_site = sum(m["sites"].shape[0] for m in ms)

    def make(pred, certify, graph=True):
        b = rpd.Batch(predicate_mode=pred, knn_k=args.k, certify=certify, use_graph=graph,
                      topology_hash=False)
        for cfg in ms:
            a = cfg["adj"]
            b.add_mesh(cfg["vert3d"], cfg["tets"], a["v_adjs"], a["e_adj6"], a["f_adjs"],
                       a["f_ids"], cfg["sites"], cfg["flags"])
        return b

    def timed(b):
        for _ in range(args.warmup):
            b.compute()
        ms_, cells, st = [], 0, None
        for _ in range(args.steps):
            flush_l2()
            st = b.compute()
            ms_.append(st.ms_total)
            cells += st.n_cells
        return cells / (sum(ms_) / 1000.0), float(np.median(ms_)), st

    out = {}
    fast = make(rpd.PRED_FP32_FILTER, True)
    tuning = fast.autotune(repeats=1).as_dict() if not args.no_tune else None
    with ClockSampler(0) as clk:
        v, m_, st = timed(fast)
    out["batch_graph"] = {"cells_per_s": v, "ms_per_step": m_, "n_launches": int(st.n_launches),
                          "stage_ms": {"front_end": st.ms_knn, "pairs_csr": st.ms_pairs,
                                       "clip": st.ms_clip, "clip_kernel": st.ms_clip_kernel,
                                       "epilogue": st.ms_epilogue, "compact": st.ms_compact,
                                       "exact_lists": st.ms_extend},
                          "uncertified_cells": int(st.n_uncertified),
                          "exact_lists": {"extended_sites": int(st.n_extended_sites),
                                          "cells_reclipped": int(st.n_cert_reclipped),
                                          "rounds": int(st.n_extend_rounds)}}
    n_cells, n_pairs = int(st.n_cells), int(st.n_pairs)
    fast.configure(topology_hash=1)
    fast.compute()
    fh, fph = fast.topology_hashes(), fast.pair_headers()
    fast.close()
    nog = make(rpd.PRED_FP32_FILTER, True, graph=False)
    v, m_, st = timed(nog)
    out["batch_no_graph"] = {"cells_per_s": v, "ms_per_step": m_}
    nog.close()
    # one single-mesh compute per mesh (same configuration), back to back
    singles = []
    for cfg in ms:
        a = cfg["adj"]
        r = rpd.RPD(predicate_mode=rpd.PRED_FP32_FILTER, neighbor_source=rpd.NEIGH_KNN,
                    knn_k=args.k, certify=True, topology_hash=False)
        r.set_mesh(cfg["vert3d"], cfg["tets"], a["v_adjs"], a["e_adj6"], a["f_adjs"], a["f_ids"])
        r.set_sites(cfg["sites"], cfg["flags"])
        if tuning:
            r.configure(warps_per_block=tuning["warps_per_block"], clip_variant=tuning["clip_variant"])
        singles.append(r)
    for r in singles:
        r.compute()
    t1 = time.perf_counter()
    cells = 0
    for _ in range(args.steps):
        for r in singles:
            cells += r.compute().n_cells
    out["per_mesh_loop"] = {"cells_per_s": cells / (time.perf_counter() - t1),
                            "note": "host wall clock over 256 rpd_compute calls per step"}
    for r in singles:
        r.close()
    plain = make(rpd.PRED_FP64, False)
    v, m_, st = timed(plain)
    out["plain_fp64_batch"] = {"cells_per_s": v, "ms_per_step": m_}
    plain.configure(topology_hash=1)
    plain.compute()
    ph, pph = plain.topology_hashes(), plain.pair_headers()
    plain.close()
    cmp = compare_topology(fph, fh, pph, ph)
    print(json.dumps({
        "workload": "batch_%d_meshes_cube_or_ellipsoid_tets_2k-200k_sites_100-20k" % len(ms),
        "n_mesh": len(ms), "n_tet": n_tet, "n_site": n_site, "n_pairs": n_pairs,
        "n_cells": n_cells, "knn_k": args.k, "generation_s": round(gen_s, 1), "tuning": tuning,
        "vs_plain_fp64": cmp, "runs": out,
        "clocks": clk.summary()}))


def run_fast_only(args):
    """Set-up plus warmup + steps computes of the fast path, nothing else:
    the command profiled by ncu (launch lists and kernel captures)."""
    from libmat_gb300 import rpd

    cfg, name, _ = make_workload(args)
    adj = rpd.mesh_adjacency(cfg["vert3d"].shape[0], cfg["tets"])
    r = rpd.RPD(predicate_mode=rpd.PRED_FP32_FILTER, neighbor_source=rpd.NEIGH_KNN,
                knn_k=args.k, clip_order=rpd.ORDER_SITE_ID, certify=True,
                clip_variant=args.clip_variant, topology_hash=False)
    r.set_mesh(cfg["vert3d"], cfg["tets"], adj["v_adjs"], adj["e_adj6"], adj["f_adjs"],
               adj["f_ids"])
    r.set_sites(cfg["sites"], cfg["flags"])
    out = []
    for i in range(args.warmup + args.steps):
        st = r.compute()
        out.append(st.as_dict())
    if args.topology or args.power_cells:
        out[-1]["ms_topology"] = r.compute_topology()
    if args.power_cells:  # get_all_voro_info + the connected components
        nb = int((adj["f_adjs"] == 1).sum())
        out[-1]["ms_power_cells"] = r.compute_power_cells(nb - 1)
    r.close()
    print(json.dumps({"workload": name, "last": out[-1]}))


def _geometry_error(h1, p1, h2, p2, n=20000):
    """Max / RMS difference of FP64 vertex coordinates (relative to the
    coordinate scale) and of cell volumes between two runs, on a sample of
    cells with the same topology (vertex order may differ: compared as
    sorted coordinate rows)."""
    from libmat_gb300 import rpd

    ok = np.flatnonzero(h1["status"] == rpd.SUCCESS)
    if len(ok) == 0:
        return None
    rng = np.random.default_rng(1)
    pick = rng.choice(ok, size=min(n, len(ok)), replace=False)
    vmax, vsq, vn, wmax, wsq = 0.0, 0.0, 0, 0.0, 0.0
    for q in pick:
        a = _xyz(p1, h1, q)
        b = _xyz(p2, h2, q)
        if a.shape != b.shape:
            continue
        a = a[np.lexsort(a.T[::-1])]
        b = b[np.lexsort(b.T[::-1])]
        d = np.abs(a - b) / 1000.0
        vmax = max(vmax, float(d.max()))
        vsq += float((d * d).sum())
        vn += d.size
        rv = abs(h1["volume"][q] - h2["volume"][q]) / max(abs(h2["volume"][q]), 1e-30)
        wmax = max(wmax, rv)
        wsq += rv * rv
    return {"vertex_max_rel": vmax, "vertex_rms_rel": (vsq / max(vn, 1)) ** 0.5,
            "volume_max_rel": wmax, "volume_rms_rel": (wsq / len(pick)) ** 0.5,
            "cells_sampled": int(len(pick))}


def _xyz(p, h, q):
    nv, np_, ne = int(h["nb_v"][q]), int(h["nb_p"][q]), int(h["nb_e"][q])
    a = lambda x: (x + 15) // 16 * 16  # noqa: E731
    start = int(h["offset"][q]) + 16 * np_ + a(8 * np_) + a(4 * nv) + a(4 * ne) + a(np_)
    return p[start:start + 24 * nv].view(np.float64).reshape(-1, 3)


def _sample_topology_equal(h1, p1, h2, p2, n=20000):
    from libmat_gb300 import rpd

    ok = np.flatnonzero(h1["status"] == rpd.SUCCESS)
    if len(ok) == 0:
        return True
    rng = np.random.default_rng(0)
    pick = rng.choice(ok, size=min(n, len(ok)), replace=False)
    for q in pick:
        nv, np_, ne = int(h1["nb_v"][q]), int(h1["nb_p"][q]), int(h1["nb_e"][q])
        sz = rpd.payload_bytes(nv, np_, ne) - ((24 * nv + 15) // 16) * 16
        a = p1[int(h1["offset"][q]):int(h1["offset"][q]) + sz]
        b = p2[int(h2["offset"][q]):int(h2["offset"][q]) + sz]
        if not np.array_equal(a, b):
            return False
    return True


def pipelined_steps(first, n, upload, compute, copy_back, finish, n_ctx=2, timeout=300.0):
    """Steps first .. first + n - 1 on n_ctx contexts, step i on context
    (i - first) % n_ctx, each context driven by its own host thread.
    upload(e) and compute(e) of the steps take turns in step order (two
    contexts' kernels on one GPU time-slice rather than run side by side);
    copy_back(e, compute's result) queues the step's copy back and returns
    at once, so the copy runs while the next steps upload and compute;
    finish(e) after a context's last step waits for its copies.  Returns the
    wall time from the threads' start to the last finish and, per step,
    (seconds waiting for the turn, uploading, computing, copy_back's value).
    The first error of any thread stops the others at their next turn and is
    raised here."""
    go = threading.Barrier(n_ctx + 1)
    turn = threading.Condition()
    nxt = [first]  # the step whose turn it is
    errors = []
    records = {}

    def worker(e):
        try:
            go.wait()
            for i in range(first + e, first + n, n_ctx):
                t0 = time.perf_counter()
                with turn:
                    if not turn.wait_for(lambda: nxt[0] == i or bool(errors), timeout=timeout):
                        raise RuntimeError("pipelined steps: no turn for step %d" % i)
                    if errors:
                        return
                t1 = time.perf_counter()
                try:
                    upload(e)
                    t2 = time.perf_counter()
                    res = compute(e)
                finally:
                    with turn:
                        nxt[0] = i + 1
                        turn.notify_all()
                t3 = time.perf_counter()
                records[i] = (t1 - t0, t2 - t1, t3 - t2, copy_back(e, res))
            finish(e)
        except BaseException as ex:
            with turn:
                errors.append(ex)
                turn.notify_all()

    ths = [threading.Thread(target=worker, args=(e,)) for e in range(n_ctx)]
    for th in ths:
        th.start()
    go.wait()
    t0 = time.perf_counter()
    for th in ths:
        th.join()
    if errors:
        raise errors[0]
    return time.perf_counter() - t0, [records[i] for i in sorted(records)]


def _e2e(args, cfg, adj, rpd, tuned):
    """The same metric through the C ABI with host buffers (page-locked): per
    step rpd_set_mesh + rpd_set_sites (host->device), rpd_compute, and the
    device->host copy of every cell.  Two contexts take the steps in turn,
    each driven by its own host thread, uploads and computes one after the
    other (pipelined_steps): a step's copy back
    (rpd_copy_cells_to_host_async) and its host round trips overlap the
    other context's upload and kernels, and the timed region ends when the
    last step's cells have landed.  No L2 flush between the steps: each step writes 1.7
    GB of cells (> 129 MB L2).  "serial" is one context with the blocking
    copy (rpd_copy_cells_to_host)."""
    nt, nv, ns = cfg["tets"].shape[0], cfg["vert3d"].shape[0], cfg["sites"].shape[0]
    pins = {}

    def pin(name, a):
        pa = rpd.PinnedArray(a.shape, a.dtype)
        pa.array[...] = a
        pins[name] = pa
        return pa.array

    v = pin("v", cfg["vert3d"])
    t = pin("t", cfg["tets"])
    va = pin("va", adj["v_adjs"])
    e6 = pin("e6", adj["e_adj6"])
    fa = pin("fa", adj["f_adjs"])
    fi = pin("fi", adj["f_ids"])
    s = pin("s", cfg["sites"])
    fl = pin("fl", cfg["flags"])
    h2d = (v.nbytes + t.nbytes + va.nbytes + e6.nbytes + fa.nbytes + fi.nbytes + s.nbytes +
           fl.nbytes)

    def engine():
        r = rpd.RPD(predicate_mode=rpd.PRED_FP32_FILTER, neighbor_source=rpd.NEIGH_KNN,
                    knn_k=args.k, clip_order=rpd.ORDER_SITE_ID, certify=True)
        # the fast engine's tuned configuration and trained predictor
        tc = tuned.config()
        tc.topology_hash = 0
        r.set_config(tc)
        try:
            params, margin = tuned.mlp_params()
            r.mlp_set_params(params, margin)
        except rpd.RPDError:
            pass
        r.set_mesh(v, t, va, e6, fa, fi)
        r.set_sites(s, fl)
        st = r.compute()
        hbuf = rpd.PinnedArray((int(st.n_cells * 1.1) + 1024,), rpd.HEADER_DTYPE)
        pbuf = rpd.PinnedArray((int(st.payload_bytes * 1.1) + (1 << 20),), np.uint8)
        return r, hbuf, pbuf

    def upload_compute(r):
        r.set_mesh(v, t, va, e6, fa, fi)
        r.set_sites(s, fl)
        return r.compute()

    engines = [engine(), engine()]
    # ---- serial: one context, blocking copy
    r0, hb0, pb0 = engines[0]
    for _ in range(args.warmup):
        upload_compute(r0)
        r0.cells(hb0.array, pb0.array)
    serial_secs, serial_cells = 0.0, 0
    parts = np.zeros(3)
    for _ in range(args.steps):
        flush_l2()
        t0 = time.perf_counter()
        r0.set_mesh(v, t, va, e6, fa, fi)
        r0.set_sites(s, fl)
        t1 = time.perf_counter()
        st = r0.compute()
        t2 = time.perf_counter()
        h, p = r0.cells(hb0.array, pb0.array)
        t3 = time.perf_counter()
        parts += (t1 - t0, t2 - t1, t3 - t2)
        serial_secs += t3 - t0
        serial_cells += st.n_cells
    copy_bytes = h.nbytes + p.nbytes
    # ---- pipelined (pipelined_steps): two contexts, one host thread each;
    # a step's copy back runs while the other context uploads and computes
    def run(first, n):
        def upload(e):
            r = engines[e][0]
            r.set_mesh(v, t, va, e6, fa, fi)
            r.set_sites(s, fl)

        def copy_back(e, st):
            r, hb, pb = engines[e]
            h, p = r.cells_async(hb.array, pb.array)
            return st.n_cells, h.nbytes + p.nbytes, st.ms_total / 1000.0

        return pipelined_steps(first, n, upload, lambda e: engines[e][0].compute(), copy_back,
                               lambda e: engines[e][0].synchronize())

    run(0, max(2, args.warmup))
    flush_l2()
    # a pipeline fills (the first upload) and drains (the last copy back)
    # outside any overlap: at least 16 steps, so that these two ends weigh
    # little against the steady state
    n_pipe = max(args.steps, 16)
    secs, recs = run(args.warmup, n_pipe)
    cells = sum(rec[3][0] for rec in recs)
    d2h_total = sum(rec[3][1] for rec in recs)
    pparts = np.array([[rec[0], rec[1], rec[2], rec[3][2]] for rec in recs]).mean(axis=0)
    for r, hb, pb in engines:
        r.close()
        hb.free()
        pb.free()
    for pa in pins.values():
        pa.free()
    return {"value": cells / secs, "unit": UNIT, "h2d_bytes_per_step": int(h2d),
            "d2h_bytes_per_step": int(d2h_total // n_pipe),
            "ms_per_step": 1000 * secs / n_pipe, "steps": n_pipe,
            "pipelined": "2 contexts, one host thread each, upload + compute in turn",
            "l2": "not flushed between pipelined steps: each writes 1.7 GB of cells (> 129 MB)",
            "parts_ms": {"wait_turn": 1000 * pparts[0], "upload": 1000 * pparts[1],
                         "compute_wall": 1000 * pparts[2], "compute_device": 1000 * pparts[3]},
            "serial": {"value": serial_cells / serial_secs,
                       "ms_per_step": 1000 * serial_secs / args.steps,
                       "upload_ms": 1000 * parts[0] / args.steps,
                       "compute_ms": 1000 * parts[1] / args.steps,
                       "copy_ms": 1000 * parts[2] / args.steps,
                       "copy_gbps": copy_bytes / (parts[2] / args.steps) / 1e9}}


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=5)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--impl", default="ours", choices=["ours", "reference"])
    ap.add_argument("--config", default="ellipsoid",
                    choices=["ellipsoid", "small", "lattice", "batch"])
    ap.add_argument("--batch-meshes", type=int, default=256)
    ap.add_argument("--lattice-n", type=int, default=100, help="lattice mesh grid points per axis")
    ap.add_argument("--lattice-m", type=int, default=50, help="lattice sites per axis")
    ap.add_argument("--tets", type=int, default=1_000_000)
    ap.add_argument("--sites", type=int, default=50_000)
    ap.add_argument("--k", type=int, default=64)
    ap.add_argument("--cpu-sample", type=int, default=20000)
    ap.add_argument("--ref-sample", type=int, default=20000)
    ap.add_argument("--no-cpu", action="store_true")
    ap.add_argument("--no-tune", action="store_true", help="skip the autotuner")
    ap.add_argument("--no-true-rpd", action="store_true",
                    help="skip the comparison with the power-neighbour lists")
    ap.add_argument("--no-learned", action="store_true", help="skip training the k-predictor")
    ap.add_argument("--force-learned", action="store_true",
                    help="time the learned lengths even if the autotuner prefers others")
    ap.add_argument("--train-seeds", type=int, nargs="+", default=[41, 42])
    ap.add_argument("--train-cells", type=int, default=200_000)
    ap.add_argument("--epochs", type=int, default=20)
    ap.add_argument("--miss-target", type=float, default=0.02)
    ap.add_argument("--clip-variant", type=int, default=2,
                    help="--fast-only: clip kernel register budget (2 = the tuned choice)")
    ap.add_argument("--topology", action="store_true",
                    help="--fast-only: also run the per-cell topology pass after the last step")
    ap.add_argument("--power-cells", action="store_true",
                    help="--fast-only: also run the topology and power-cell passes after the last step")
    ap.add_argument("--fast-only", action="store_true",
                    help="only the timed fast path (for profiler launch lists)")
    args = ap.parse_args()
    if args.impl == "reference":
        run_reference(args)
    elif args.config == "lattice":
        from __graft_entry__ import build

        build()
        run_stress(args)
    elif args.config == "batch":
        from __graft_entry__ import build

        build()
        run_batch(args)
    elif args.fast_only:
        from __graft_entry__ import build

        build()
        run_fast_only(args)
    else:
        from __graft_entry__ import build

        build()
        run_ours(args)


if __name__ == "__main__":
    main()
