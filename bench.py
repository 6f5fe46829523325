"""Benchmark of the Gaussian-field path tracer: forward + adjoint path segments per second.

A step is one inverse-rendering training iteration on the workload: LBVH refit, forward trace of
every (view, sample) path, the loss (the terms of PTIR's default training loss that the tracer's
outputs feed: L1 on pbr against a target render, L2 albedo and roughness prior regularisation on
the material output), the path-replay adjoint, and the fused selective Adam step of the material
and environment. The default workload is field-1m (1M Gaussians, 8 views of 1024x768 at 16 spp,
4 bounces, 512x1024 environment; see ptir_b200/synthetic.py) with BF16 attribute storage and FP32
arithmetic; --storage fp32 gives the plain FP32 drop-in. The metric counts the forward path
segments of a step (the adjoint replays each of them) over the step's device time.

  python bench.py [--gpus N] [--steps K] [--warmup W] [--workload NAME] [--storage bf16|fp16|fp32]
                  [--impl ours|reference]

One JSON line on rank 0. Multi-GPU runs (torchrun) are data parallel over views: every rank
traces its own views of the same scene (weak scaling) and the material / environment
gradients are summed with one NCCL all-reduce per step.

--impl reference times the reference path's CPU restatement (the oracle port in FP32, all
host threads) on a bounded sample of the same workload with the same loss, the reference's
OptiX build being unavailable here (no OptiX SDK headers).
"""
from __future__ import annotations

import argparse
import json
import math
import os
import statistics
import subprocess
import sys
import threading
import time

import numpy as np
import torch

ROOT = os.path.dirname(os.path.abspath(__file__))
sys.path.insert(0, ROOT)

from ptir_b200 import dist as pdist  # noqa: E402
from ptir_b200 import envmap, synthetic  # noqa: E402
from ptir_b200.optim import selective_adam_  # noqa: E402

METRIC = "fwd+bwd path segments/s at 1M Gaussians"


def metric_of(wl) -> str:
    """The metric's name: the headline's for the 1M-Gaussian workload, else named for the workload."""
    if wl.name == "field-1m":
        return METRIC
    return f"{'fwd+bwd' if wl.backward else 'fwd'} path segments/s ({wl.name}, {wl.n:,} Gaussians)"
ADAM_LR = 1e-3
PEAKS_PATH = os.path.join(ROOT, "MEASURED_PEAKS.json")
HBM_FALLBACK_GBS = 6650.0


def _peaks():
    try:
        with open(PEAKS_PATH) as f:
            p = json.load(f)
        return float(p["hbm_gbs"]), "measured"
    except Exception:
        return HBM_FALLBACK_GBS, "fallback"


# ------------------------------------------------------------------------------------------
# workload setup
def workload_of(args):
    """The named workload, optionally shrunk for profiling (--views/--res/--spp; these make every
    view alike)."""
    wl = synthetic.workload(args.workload)
    if not any(getattr(args, k, None) for k in ("res", "spp", "views")):
        return wl
    w, h, spp = wl.views[0]
    if getattr(args, "res", None):
        w, h = (int(v) for v in args.res.lower().split("x"))
    if getattr(args, "spp", None):
        spp = int(args.spp)
    views = int(args.views) if getattr(args, "views", None) else len(wl.views)
    wl.views = [(w, h, spp)] * views
    return wl


class Setup:
    def __init__(self, wl, rank: int, device):
        self.wl = wl
        self.device = device
        f = synthetic.make_field(wl.n, seed=wl.seed, layout=wl.layout, scale_range=wl.scale_range, sh_full=wl.sh_full)
        self.field = f
        d = lambda t: t.to(device).contiguous()  # noqa: E731
        self.pos, self.rot, self.scl, self.dns = d(f["pos"]), d(f["rot"]), d(f["scl"]), d(f["dns"])
        self.density = d(synthetic.density_tensor(f))
        self.material = d(synthetic.material_tensor(f))
        self.sph, self.snrm = d(f["sph"]), d(f["snrm"])
        env = synthetic.make_environment(*wl.env_hw, seed=wl.seed)
        self.env = d(env)
        self.alias = envmap.pack(envmap.build(env), device)
        # With W ranks the job has W x views views; this rank traces its share, balanced by the
        # views' samples (the estimate of their path segments).
        world = int(os.environ.get("WORLD_SIZE", "1"))
        job_views = list(wl.views) * world
        all_eyes = synthetic.camera_positions(len(job_views), seed=wl.seed)
        mine = pdist.shard_weighted([w * h * spp for w, h, spp in job_views], rank, world)
        eyes = all_eyes[mine]
        self.my_views = [job_views[i] for i in mine]
        self.t2w = torch.eye(4, device=device).reshape(1, 4, 4).contiguous()
        self.batched = any(v != self.my_views[0] for v in self.my_views)
        oris, dirs = [], []
        if not self.batched:
            # one launch: z = sample * views + view (the reference's order)
            w, h, spp = self.my_views[0]
            for eye in eyes:
                o, dr = synthetic.view_rays_device(w, h, spp, eye, device)
                oris.append(o)
                dirs.append(dr)
            self.ray_ori = torch.stack(oris, 1).reshape(spp * len(eyes), h, w, 3).contiguous()
            self.ray_dir = torch.stack(dirs, 1).reshape(spp * len(eyes), h, w, 3).contiguous()
        else:
            # views of their own resolution and spp, one batch: rays flat in view order
            self.views = []
            for v, ((w, h, spp), eye) in enumerate(zip(self.my_views, eyes)):
                o, dr = synthetic.view_rays_device(w, h, spp, eye, device)
                oris.append(o.reshape(-1, 3))
                dirs.append(dr.reshape(-1, 3))
                self.views.append((v, self.t2w, spp, h, w))
            self.ray_ori = torch.cat(oris).contiguous()
            self.ray_dir = torch.cat(dirs).contiguous()
        del oris, dirs
        self.samples = int(self.ray_ori.numel() // 3)
        e = lambda *s, dt=torch.float32: torch.empty(s, dtype=dt, device=device)  # noqa: E731
        self.lights = (e(0, 9), e(5, 0), e(0, 3), e(0, 3, dt=torch.int32), e(0, 8), e(3, 0))

    def tracer(self, **kw):
        from ptir_b200 import OptixTracer

        return OptixTracer("", "", "reference", "referenceBwd", "instances", 4, 0.0113, True, 3, True, True, True,
                           False, False, **kw)

    def trace(self, tr, material=None, ray_ori=None, ray_dir=None, frame=0, env=None):
        ori = self.ray_ori if ray_ori is None else ray_ori
        drs = self.ray_dir if ray_dir is None else ray_dir
        mat = self.material if material is None else material
        scene = (self.density, mat, self.sph, self.snrm, self.env if env is None else env, self.alias, *self.lights, 0,
                 3, 0.001, self.wl.max_bounces)
        if self.batched:
            return tr.trace_views(self.views, ori, drs, *scene)
        return tr.trace(frame, self.t2w, ori, drs, *scene)

    def trace_bwd(self, tr, fwd, pbr_grad, material_grad=None, ray_ori=None, ray_dir=None, frame=0, material=None,
                  env=None):
        (rad, dns, hit, hit2, dist, nrm, snrm, mat, hits, vis, pbr, light, comps) = fwd
        z = self._zeros
        ori = self.ray_ori if ray_ori is None else ray_ori
        drs = self.ray_dir if ray_dir is None else ray_dir
        args = (rad, dns, hit, hit2, dist, nrm, snrm, mat, pbr, light, self.density,
                self.material if material is None else material, self.sph, self.snrm, self.env if env is None else env,
                self.alias, *self.lights, z["rad"], z["dns"], z["hit"], z["hit2"], z["dist"], z["nrm"], z["snrm"],
                z["mat"] if material_grad is None else material_grad, pbr_grad, z["light"], 0, 3, 0.001,
                self.wl.max_bounces)
        if self.batched:
            return tr.trace_bwd_views(self.views, ori, drs, *args)
        return tr.trace_bwd(frame, self.t2w, ori, drs, *args)

    def prepare_grads(self, fwd):
        (rad, dns, hit, hit2, dist, nrm, snrm, mat, hits, vis, pbr, light, comps) = fwd
        self._zeros = dict(rad=torch.zeros_like(rad), dns=torch.zeros_like(dns), hit=torch.zeros_like(hit),
                           hit2=torch.zeros_like(hit2), dist=torch.zeros_like(dist), nrm=torch.zeros_like(nrm),
                           snrm=torch.zeros_like(snrm), mat=torch.zeros_like(mat), light=torch.zeros_like(light))


def _clock_sampler(out: list, stop: threading.Event, gpu_index: int):
    q = ("index,clocks.sm,clocks.max.sm,power.draw,clocks_event_reasons.active,clocks_event_reasons.hw_slowdown,"
         "clocks_event_reasons.hw_thermal_slowdown,clocks_event_reasons.sw_thermal_slowdown,"
         "clocks_event_reasons.sw_power_cap")
    try:
        p = subprocess.Popen(["nvidia-smi", f"--id={gpu_index}", f"--query-gpu={q}", "--format=csv,noheader,nounits",
                              "-lms", "200"], stdout=subprocess.PIPE, stderr=subprocess.DEVNULL, text=True)
    except Exception:
        return
    try:
        while not stop.is_set():
            line = p.stdout.readline()
            if not line:
                break
            out.append(line.strip())
    finally:
        p.terminate()
        try:
            p.wait(timeout=5)
        except Exception:
            p.kill()


def _clock_summary(lines: list):
    sm, mx, reasons = [], None, set()
    names = ("hw_slowdown", "hw_thermal_slowdown", "sw_thermal_slowdown", "sw_power_cap")
    for ln in lines:
        f = [x.strip() for x in ln.split(",")]
        if len(f) < 9:
            continue
        try:
            sm.append(float(f[1]))
            mx = float(f[2])
        except ValueError:
            continue
        for name, v in zip(names, f[5:9]):
            if v.lower().startswith("active"):
                reasons.add(name)
    if not sm:
        return None
    return {"sm_mhz": statistics.median(sm), "sm_max_mhz": mx, "reasons": sorted(reasons), "samples": len(sm)}


# ------------------------------------------------------------------------------------------
STAGES = ("intersect", "shadow", "replay", "shading", "megakernel", "sort")
KERNEL_OF_STAGE = {"intersect": "k_wf_trace_near/quad", "shadow": "k_wf_shadow", "replay": "k_wb_replay",
                   "shading": "k_wf_camera/primary/bounce", "megakernel": "k_trace_fwd/k_trace_bwd",
                   "sort": "k_wf_sort_keys + radix sort"}
ACCEL_KERNELS_PER_BUILD = 6  # the step's refit: k_prep, k_bounds_partial, k_bounds_final, k_gather, k_refit, k_emit4


def stage_bytes(stage: str, c: dict, rec: dict) -> float:
    """Algorithmic HBM bytes of one stage's work from its device counters: per segment 24 B of
    ray, a geometry record per candidate, and per composited hit the material, SH and shading
    normal records (`rec`: 48 / 20 / 192 / 12 B in FP32 storage, half in 16-bit storage); a replay
    writes 20 B of material gradient per hit. BVH node fetches are implementation overhead and
    not counted."""
    hit = rec["mat"] + rec["sh"] + rec["nrm"]
    if stage == "intersect":
        return 24.0 * c["segments"] + rec["geo"] * c["candidates"] + hit * c["accepted"]
    if stage == "shadow":
        return 24.0 * c["segments"] + rec["geo"] * c["candidates"]
    if stage == "replay":
        return 24.0 * c["replay"] + rec["geo"] * c["candidates"] + 40.0 * c["replay_accepted"]
    if stage == "shading":
        return 64.0 * c["env_lookups"]
    if stage == "sort":
        return 36.0 * c["segments"]
    return 24.0 * c["segments"] + rec["geo"] * c["candidates"] + hit * c["accepted"] + 64.0 * c["env_lookups"]


def record_bytes(storage: str) -> dict:
    f = 2 if storage in ("bf16", "fp16") else 1
    return {"geo": 48 // f, "mat": 20 // f, "sh": 192 // f, "nrm": 12 // f}


def algorithmic_bytes(fc: dict, bc: dict, samples: int):
    """Per-launch algorithmic HBM bytes of the forward and backward kernels.

    forward, per segment 24 B ray + 48 B per candidate (geometry record) + 224 B per composited
    hit (material 20 + SH 192 + shading normal 12) + 64 B per bilinear environment lookup, plus
    128 B of per-sample outputs. backward: the same for its replay of the forward path, plus per
    gradient re-traversal 24 B, 20 B read + 20 B written per hit receiving a material gradient,
    48 B of atomics per environment lookup, and 68 B of per-sample inputs (pbr, light and their
    gradients, material gradient)."""
    fwd = 24 * fc["segments"] + 48 * fc["candidates"] + 224 * fc["accepted"] + 64 * fc["env_lookups"] + 128 * samples
    bwd = (24 * (bc["segments"] + bc["replay"]) + 48 * bc["candidates"] + 224 * bc["accepted"]
           + 40 * bc["replay_accepted"] + (64 + 48) * bc["env_lookups"] + 68 * samples)
    return fwd, bwd


def tune_launch_shape(S, args, device) -> dict:
    """Autotune the launch shape on a sample of the workload (a thirty-second of its rays, or its
    first view; forward + adjoint), cached in _autotune.json beside this file. The default sweep
    keeps the reference's k-buffer of 16, whose results are the reference's, and sweeps block
    {64, 128} x refill {16, 32}. --autotune-full also sweeps k-buffer {8, 16, 32} and the chunk size.
    Other k-buffer sizes cull at another distance and keep another set of grazing candidates, which
    changes the image (on the 300k-Gaussian config-4 scene, 0.3 % of samples at 32)."""
    from ptir_b200 import autotune

    tr0 = S.tracer(storage=args.storage)
    tr0.build_bvh(S.pos, S.rot, S.scl, S.dns, True, True)
    del tr0
    if S.batched:
        frame, t2w, z, h, w = S.views[0]
        n = z * h * w
        ori, drs = S.ray_ori[:n], S.ray_dir[:n]
        views = [S.views[0]]
    else:
        z = max(1, S.ray_ori.shape[0] // 32)
        ori, drs, views = S.ray_ori[:z], S.ray_dir[:z], None

    def run(tr):
        tr.build_bvh(S.pos, S.rot, S.scl, S.dns, True, True)
        scene = (S.density, S.material, S.sph, S.snrm, S.env, S.alias, *S.lights, 0, 3, 0.001, S.wl.max_bounces)
        f = tr.trace_views(views, ori, drs, *scene) if views else tr.trace(0, S.t2w, ori, drs, *scene)
        z_ = torch.zeros_like
        g = torch.sign(f[10] - 0.5) * 1e-6
        args_b = (*f[:8], f[10], f[11], *scene[:12], z_(f[0]), z_(f[1]), z_(f[2]), z_(f[3]), z_(f[4]), z_(f[5]),
                  z_(f[6]), z_(f[7]), g, z_(f[11]), *scene[12:])
        if views:
            tr.trace_bwd_views(views, ori, drs, *args_b)
        else:
            tr.trace_bwd(0, S.t2w, ori, drs, *args_b)

    shapes = autotune.space() if args.autotune_full else autotune.space(kbuffers=(16,), blocks=(64, 128),
                                                                          chunks=(0,), refills=(16, 32))
    sig = (f"{S.wl.name}|n={S.wl.n}|samples={S.samples}|bounces={S.wl.max_bounces}|storage={args.storage}"
           f"|shapes={len(shapes)}")
    tuner = autotune.Autotuner(os.path.join(ROOT, "_autotune.json"))
    best, _ = tuner.tune(sig, lambda **kw: S.tracer(storage=args.storage, **kw), run, shapes=shapes)
    return best.launch()


def _view_config(views):
    if all(v == views[0] for v in views):
        return {"resolution": list(views[0][:2]), "spp": views[0][2]}
    return {"views": [list(v) for v in views]}


# The loss of the timed training iteration: the terms of PTIR's default training loss
# (configs/base_ptir.yaml:74-100, threedgrut/trainer.py:932-1125) that the tracer's outputs feed:
# L1 on pred_pbr against the target render (lambda_l1 0.8), and the albedo and roughness prior
# regularisations, L2 of pred_material against a prior image (lambda_init 0.5 and 0.2; the prior
# here is the material image of the target scene). The prior terms give every primary interaction
# a material gradient, so the adjoint re-traverses those segments even where no light reaches the
# camera (the 1M-Gaussian scene's opaque shell keeps its pbr image black).
LOSS_L1, LOSS_ALBEDO, LOSS_ROUGHNESS = 0.8, 0.5, 0.2
# dram__bytes_read.sum + dram__bytes_write.sum of the intersection kernels per segment they intersect, from
# an ncu capture of a forward pass's launches on 2 views of 512x384x4 (5,223,165,184 bytes over 2,479,466 segments)
DRAM_BYTES_PER_INTERSECT_SEGMENT = 2106.6
STEP_DESC = ("lbvh refit + forward + loss (0.8 L1(pbr, target) + 0.5 L2(albedo, prior) + 0.2 L2(roughness, prior)) "
             "+ adjoint + selective adam (material, env)")


def loss_terms(pbr, material, target_pbr, prior_material):
    """The iteration's loss and its gradients w.r.t. the per-sample pbr and material outputs."""
    d = pbr - target_pbr
    da = material[..., 0:3] - prior_material[..., 0:3]
    dr = material[..., 3:4] - prior_material[..., 3:4]
    loss = LOSS_L1 * d.abs().mean() + LOSS_ALBEDO * (da * da).mean() + LOSS_ROUGHNESS * (dr * dr).mean()
    pbr_grad = torch.sign(d) * (LOSS_L1 / d.numel())
    mat_grad = torch.zeros_like(material)
    mat_grad[..., 0:3] = da * (2.0 * LOSS_ALBEDO / da.numel())
    mat_grad[..., 3:4] = dr * (2.0 * LOSS_ROUGHNESS / dr.numel())
    return loss, pbr_grad, mat_grad


def loss_terms_np(pbr, material, target_pbr, prior_material):
    """loss_terms() in numpy for the CPU legs: (pbr_grad, material_grad) float32."""
    d = pbr.astype(np.float64) - target_pbr
    da = material[..., 0:3].astype(np.float64) - prior_material[..., 0:3]
    dr = material[..., 3:4].astype(np.float64) - prior_material[..., 3:4]
    mat_grad = np.zeros(material.shape, np.float32)
    mat_grad[..., 0:3] = da * (2.0 * LOSS_ALBEDO / da.size)
    mat_grad[..., 3:4] = dr * (2.0 * LOSS_ROUGHNESS / dr.size)
    return (np.sign(d) * (LOSS_L1 / d.size)).astype(np.float32), mat_grad


def perturbed_material(material: torch.Tensor) -> torch.Tensor:
    """The target scene's material: albedo + N(0, 0.02), seeded (the same bytes on every device)."""
    gen = torch.Generator(device="cpu").manual_seed(1234)
    mat_t = material.detach().cpu().clone()
    mat_t[:, :3] += 0.02 * torch.randn(mat_t[:, :3].shape, generator=gen)
    return mat_t.to(material.device)


def bench_config(wl, args, world: int) -> dict:
    """The `config` object shared by both arms (ours and the reference's CPU restatement)."""
    return {"workload": wl.name, "storage": args.storage, "gaussians": wl.n, "views_per_gpu": len(wl.views),
            **_view_config(wl.views), "max_bounces": wl.max_bounces, "env": list(wl.env_hw),
            "step": (STEP_DESC if wl.backward else "lbvh refit + forward") + (" + grad all-reduce" if world > 1 else ""),
            "parallelism": f"dp{world} over views"}


def run_ours(args, rank, world, device):
    import torch.distributed as dist

    S = Setup(workload_of(args), rank, device)
    shape = {}
    if not args.no_autotune:
        shape = tune_launch_shape(S, args, device)
    if args.kbuffer:
        shape = dict(shape, kbuffer=args.kbuffer)
    if args.no_warp_aggregate:
        shape = dict(shape, warp_aggregate=False)
    if args.schedule == "megakernel":
        shape = dict(shape, schedule="megakernel")
    if args.chunk_tiles:
        shape = dict(shape, chunk_tiles=args.chunk_tiles)
    if args.exact_candidates:
        shape = dict(shape, exact_candidates=True)
    if args.resume_rounds is not None:
        shape = dict(shape, resume_rounds=args.resume_rounds)
    if args.bvh_builder != "default":
        shape = dict(shape, bvh_builder=args.bvh_builder)
    if args.refill_lanes:
        shape = dict(shape, refill_lanes=args.refill_lanes)
    if args.block_size:
        shape = dict(shape, block_size=args.block_size)
    tr = S.tracer(collect_timings=True, storage=args.storage, **shape)
    stream = torch.cuda.current_stream()
    backward = S.wl.backward
    tr.build_bvh(S.pos, S.rot, S.scl, S.dns, True, True)
    if backward:
        # target image and material prior: the same scene with albedo perturbed by N(0, 0.02)
        tgt = S.trace(tr, material=perturbed_material(S.material))
        target, prior = tgt[10].clone(), tgt[7].clone()
        del tgt
    torch.cuda.synchronize()

    # the trained attributes, material [N,5] and environment [He,We,4], and their optimizer state
    material = S.material.clone().requires_grad_(backward)
    env = S.env.clone().requires_grad_(backward)
    adam = {k: (torch.zeros_like(t), torch.zeros_like(t)) for k, t in (("material", material), ("env", env))}
    bucket = pdist.GradientBucket()  # the all-reduce's flat buffer, allocated once
    # the step's ray inputs (device buffers, refilled from pinned host memory every timed step)
    ori_d, dir_d = S.ray_ori.clone(), S.ray_dir.clone()
    use_autograd = backward and not S.batched and not args.graph
    if use_autograd:
        from ptir_b200.tracer import LightBuffers, Tracer

        lights = LightBuffers(*S.lights)

    def step(events=None, on_fwd=None, on_bwd=None):
        """One training iteration: LBVH refit, forward, loss, adjoint, selective Adam. The eager
        single-batch step goes through the reference-facing autograd entry (Tracer._Autograd: the
        torch.autograd.Function of threedgptir_tracer/tracer.py:137-384) and loss.backward(); a
        batch of views, or a step captured in a CUDA graph, calls trace / trace_bwd directly with
        the same loss gradients."""
        tr.build_bvh(S.pos, S.rot, S.scl, S.dns, False, True)
        if events:
            events[0].record(stream)
        if not backward:
            fwd = S.trace(tr, material=material, ray_ori=ori_d, ray_dir=dir_d)
            if events:
                events[1].record(stream)
            if on_fwd:
                on_fwd()
            return fwd[10].mean()
        if use_autograd:
            out = Tracer._Autograd.apply(tr, 0, S.t2w, ori_d, dir_d, S.pos, S.rot, S.scl, S.dns, S.sph, S.snrm,
                                         material[:, 0:3], material[:, 3:4], material[:, 4:5], env, S.alias, lights,
                                         0, 3, 0.001, S.wl.max_bounces)
            if events:
                events[1].record(stream)
            if on_fwd:
                on_fwd()
            loss = loss_terms(out[10], out[7], target, prior)[0]
            if events:
                events[2].record(stream)
            loss.backward()
            mg, eg, vis = material.grad, env.grad, out[9]
        else:
            fwd = S.trace(tr, material=material.detach(), ray_ori=ori_d, ray_dir=dir_d)
            if events:
                events[1].record(stream)
            if on_fwd:
                on_fwd()
            loss, pbr_grad, mat_grad = loss_terms(fwd[10], fwd[7], target, prior)
            if not hasattr(S, "_zeros"):
                S.prepare_grads(fwd)
            if events:
                events[2].record(stream)
            _, mg, _, _, eg = S.trace_bwd(tr, fwd, pbr_grad, material_grad=mat_grad, ray_ori=ori_d, ray_dir=dir_d,
                                          material=material.detach(), env=env.detach())
            vis = fwd[9]
        if events:
            events[3].record(stream)
        if on_bwd:
            on_bwd()
        if world > 1:
            bucket.allreduce([mg, eg])
        with torch.no_grad():
            selective_adam_(material, mg, *adam["material"], vis.view(torch.int32) != 0, lr=ADAM_LR)
            selective_adam_(env, eg, *adam["env"], None, lr=ADAM_LR)
        material.grad = None
        env.grad = None
        return loss.detach()

    # warm-up (also reads the deterministic per-launch counters, in total and per stage)
    got = {}

    def read(tag):
        got[tag] = tr.counters()
        got[tag + "_stages"] = {st: tr.counters(st) for st in STAGES}

    for i in range(args.warmup):
        if i == 0:
            step(on_fwd=lambda: read("fwd"), on_bwd=(lambda: read("bwd")) if backward else None)
        else:
            step()
    zero = {k: 0 for k in got["fwd"]}
    fc, fcs = got["fwd"], got["fwd_stages"]
    bc, bcs = got.get("bwd", zero), got.get("bwd_stages", {st: zero for st in STAGES})
    torch.cuda.synchronize()
    status = tr.device_status()
    if status != 0:
        raise RuntimeError(f"device loop bound hit during warm-up (status {status})")

    graph, stage_t, stage_steps = None, None, args.steps
    if args.graph:
        if world > 1:
            raise SystemExit("--graph runs on one GPU")
        # stage times of one eager step (no events can be recorded inside the graph), then the
        # whole iteration is captured once and replayed
        tr.stage_times()
        step()
        torch.cuda.synchronize()
        stage_t, stage_steps = tr.stage_times(), 1
        tr.set_collect_timings(False)
        side = torch.cuda.Stream()
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            step()
        torch.cuda.current_stream().wait_stream(side)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            graph_loss = step()
        torch.cuda.synchronize()

    # Timed region: K steps. Every step copies its rays from pinned host memory into the input
    # buffers and reads its loss back (the end-to-end figure, e2e); the step's own device time,
    # inputs resident, is bracketed by events after the copy and before the read (value).
    ori_h = S.ray_ori.cpu().pin_memory()
    dir_h = S.ray_dir.cpu().pin_memory()
    loss_h = torch.empty((args.steps,), dtype=torch.float32).pin_memory()
    clock_lines, stop = [], threading.Event()
    sampler = threading.Thread(target=_clock_sampler, args=(clock_lines, stop, torch.cuda.current_device()), daemon=True)
    sampler.start()
    time.sleep(0.3)
    if graph is None:
        tr.stage_times()  # forget the warm-up launches
    ev = [[torch.cuda.Event(enable_timing=True) for _ in range(4)] for _ in range(args.steps)]
    s0 = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    s1 = [torch.cuda.Event(enable_timing=True) for _ in range(args.steps)]
    t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    if world > 1:
        dist.barrier()
    torch.cuda.synchronize()
    t0.record(stream)
    for k in range(args.steps):
        ori_d.copy_(ori_h, non_blocking=True)
        dir_d.copy_(dir_h, non_blocking=True)
        s0[k].record(stream)
        if graph is not None:
            graph.replay()
            loss = graph_loss
        else:
            loss = step(events=ev[k])
        s1[k].record(stream)
        loss_h[k:k + 1].copy_(loss.reshape(1), non_blocking=True)
    t1.record(stream)
    torch.cuda.synchronize()
    if world > 1:
        dist.barrier()
    stop.set()
    sampler.join(timeout=10)
    e2e_ms = t0.elapsed_time(t1) / args.steps
    ms_total = sum(a.elapsed_time(b) for a, b in zip(s0, s1))
    if not all(math.isfinite(float(v)) for v in loss_h):
        raise RuntimeError("non-finite loss in the timed steps")
    if graph is None:
        stage_t = tr.stage_times()  # {stage: (ms, launches)} over the timed steps
        fwd_ms = statistics.mean(e[0].elapsed_time(e[1]) for e in ev)
        bwd_ms = statistics.mean(e[2].elapsed_time(e[3]) for e in ev) if backward else None
    else:
        fwd_ms = bwd_ms = None
    del graph

    status = tr.device_status()
    if status != 0:
        raise RuntimeError(f"device loop bound hit (status {status})")

    segs = fc["segments"]
    stats = torch.tensor([ms_total, e2e_ms * args.steps, float(segs)], dtype=torch.float64, device=device)
    if world > 1:
        mx = stats.clone()
        dist.all_reduce(mx, op=dist.ReduceOp.MAX)
        sm = stats.clone()
        dist.all_reduce(sm, op=dist.ReduceOp.SUM)
        ms_total, e2e_ms, total_segs = float(mx[0]), float(mx[1]) / args.steps, float(sm[2])
    else:
        total_segs = float(segs)
    if rank != 0:
        return None
    ms_step = ms_total / args.steps
    # the dominant kernel: the stage with the most device time; its algorithmic bytes per launch
    # (forward + backward work of the stage per step / its launches per step) over its mean launch time
    dom = max(STAGES, key=lambda st: stage_t[st][0])
    dom_ms_total, dom_launches = stage_t[dom]
    rec = record_bytes(args.storage)
    dom_bytes_step = stage_bytes(dom, fcs[dom], rec) + stage_bytes(dom, bcs[dom], rec)
    launches_step = dom_launches / stage_steps
    dom_bytes = dom_bytes_step / launches_step
    dom_ms = dom_ms_total / dom_launches
    peak, peak_kind = _peaks()
    achieved = dom_bytes / (dom_ms * 1e-3) / 1e9
    # DRAM traffic of the intersection kernel per launch, scaled from an ncu capture of a smaller
    # case by the segments the launch intersects
    traffic = None
    if dom == "intersect":
        isect_segs = fcs[dom].get("segments", 0) + bcs[dom].get("segments", 0)
        traffic = DRAM_BYTES_PER_INTERSECT_SEGMENT * isect_segs / launches_step
    launches_per_step = ACCEL_KERNELS_PER_BUILD + sum(n for _, n in stage_t.values()) / stage_steps
    h2d = int(S.ray_ori.numel() * 4 * 2)
    res = {
        "metric": metric_of(S.wl),
        "value": total_segs / (ms_step * 1e-3),
        "unit": "segments/s",
        "n_gpus": world,
        "steps": args.steps,
        "warmup": args.warmup,
        "ms_per_step": ms_step,
        "higher_is_better": True,
        "scaling": "weak",
        "vs_baseline": None,
        "dtype": "f32",
        "data": "synthetic",
        "config": {**bench_config(S.wl, args, world), "launch": shape or "defaults", "cuda_graph": bool(args.graph),
                   "api": "Tracer._Autograd + loss.backward()" if use_autograd else "OptixTracer.trace / trace_bwd",
                   "samples_per_gpu": S.samples, "segments_per_step_per_gpu": segs,
                   "l2": "inputs larger than L2 (scene + BVH records ~400 MB)"},
        "pass_ms": {"forward": fwd_ms, "backward": bwd_ms},
        "stages_ms_per_step": {KERNEL_OF_STAGE[st]: stage_t[st][0] / stage_steps for st in STAGES if stage_t[st][1]},
        "roofline": {"bound": "hbm", "kernel": KERNEL_OF_STAGE[dom], "achieved": achieved, "peak": peak,
                     "unit": "GB/s", "frac": achieved / peak, "peak_source": peak_kind, "traffic": traffic,
                     "algorithmic_bytes_per_launch": dom_bytes, "ms_per_launch": dom_ms,
                     "launches_per_step": launches_step},
        "counters": {"forward": fc, "backward": bc, "forward_by_stage": fcs, "backward_by_stage": bcs},
        "e2e": {"value": total_segs / (e2e_ms * 1e-3), "unit": "segments/s", "h2d_bytes_per_step": h2d,
                "d2h_bytes_per_step": 4, "ms_per_step": e2e_ms, "steps": args.steps,
                "timing": "the same K steps: rays copied from pinned host memory and the loss read back every step"},
        "gpu_launches": int(round(launches_per_step * args.steps)),
        "clocks": _clock_summary(clock_lines),
    }
    return res, S


def cpu_sample(args, S=None, threads=0, budget_s=15.0, repeats=1):
    """Time the oracle's FP32 instantiation (the reference path restated on the CPU) on a bounded
    sample of the workload: a block of rows of every view's first sample plane, forward and (for
    workloads with a backward) the adjoint of the benchmark's loss. The loss's target render and
    material prior (the same scene with perturbed albedo) are rendered by the oracle first, outside
    the timed part. With `repeats` > 1 the sized sample is timed that many times and the value is
    the median."""
    from oracle import oracle as O

    wl = workload_of(args)
    f = synthetic.make_field(wl.n, seed=wl.seed, layout=wl.layout, scale_range=wl.scale_range, sh_full=wl.sh_full)
    env = synthetic.make_environment(*wl.env_hw, seed=wl.seed)
    alias = envmap.pack(envmap.build(env)).numpy()
    w, h, spp = wl.views[0]
    eyes = synthetic.camera_positions(len(wl.views), seed=wl.seed)
    material = synthetic.material_tensor(f)
    base = dict(build_pos=f["pos"].numpy(), build_rot=f["rot"].numpy(), build_scl=f["scl"].numpy(),
                build_dns=f["dns"].numpy(), density=synthetic.density_tensor(f).numpy(),
                material=material.numpy(), sph=f["sph"].numpy(), shading_normal=f["snrm"].numpy(),
                environment=env.numpy(), alias_table=alias, ray_to_world=np.eye(4, dtype=np.float32)[None], frame=0,
                sph_degree=3, min_transmittance=0.001, max_bounces=wl.max_bounces)
    cfg = O.OracleConfig()
    jitter = synthetic.SPP_PATTERNS.get(spp, ((0.5, 0.5),))[0]
    targets = {}

    def run(rows):
        oris, dirs = [], []
        for eye in eyes:
            o, d = synthetic.pinhole_rays(w, h, eye, jitter=jitter)
            r0 = (h - rows) // 2
            oris.append(o[r0:r0 + rows])
            dirs.append(d[r0:r0 + rows])
        s = dict(base, ray_ori=np.stack(oris), ray_dir=np.stack(dirs))
        zhw = s["ray_ori"].shape[:3]
        if wl.backward and rows not in targets:
            targets[rows], _, _ = O.trace(cfg, dict(s, material=perturbed_material(material).numpy()), "f32",
                                          threads=threads)
        tgt = targets.get(rows)
        t = time.perf_counter()
        out, _, st = O.trace(cfg, s, "f32", threads=threads)
        if wl.backward:
            pbr_g, mat_g = loss_terms_np(out["pbr"], out["material"], tgt["pbr"], tgt["material"])
            g = dict(pbr=pbr_g, light=np.zeros(zhw + (3,), np.float32), material=mat_g)
            O.trace_bwd(cfg, s, out, g, "f32", threads=threads)
        return time.perf_counter() - t, st.segments, int(np.prod(zhw))

    rows = 2
    dt, segs, paths = run(rows)
    target_rows = int(min(h, max(rows, rows * budget_s / max(dt, 1e-3))))
    if target_rows > rows:
        dt, segs, paths = run(target_rows)
        rows = target_rows
    times = [dt] + [run(rows)[0] for _ in range(repeats - 1)]
    dt = statistics.median(times)
    n_threads = threads or O.num_threads()
    what = "fwd + adjoint of the benchmark loss" if wl.backward else "fwd"
    return {"value": segs / dt, "unit": "segments/s", "cores": n_threads, "kind": "port",
            "sample": f"{paths} paths ({len(eyes)} views x {rows} rows x {w} px, first sample of each pixel), "
                      f"{what}, oracle FP32, {dt:.1f} s (median of {len(times)})", "seconds": dt,
            "segments": segs}


def accuracy_sample(args, shape: dict, device, name: str = "field-300k-sh", res=(128, 96)) -> dict:
    """Image and gradient error of the tracer (the run's launch shape) against the FP64 oracle fed
    the same per-path sample sequences, for each attribute storage: config 4 of the benchmark (the
    300k-Gaussian scene with degree-3 SH, 512x1024 environment, 3 bounces) on one view of res at
    1 spp, since the full view is beyond the oracle's reach. (The timed 1M-Gaussian scene is no use
    here: its background shell is opaque, so no light reaches the camera and its PBR image is
    black.) With 16-bit storage the oracle gets the attributes rounded as the tracer holds them.
    Both backward passes start from the oracle's forward values with the same seeded pbr
    gradient.

    The error is split by the paths' decision signatures (oracle/compare.py): "flipped" paths took
    another discrete branch than the FP64 evaluation somewhere (and differ by whole
    contributions), "agree" paths took the same branches. The gradients are reported for the
    seeded gradient on every path ("grad_all") and with it zeroed on the flipped paths
    ("grad_agree"). The oracle's own FP32 build, the same estimator in float32 on the CPU, is the
    yardstick of float32's distance from FP64 ("oracle_fp32_vs_fp64")."""
    from oracle import compare as K
    from oracle import oracle as O
    from ptir_b200 import OptixTracer

    wl = synthetic.workload(name)
    f = synthetic.make_field(wl.n, seed=wl.seed, layout=wl.layout, scale_range=wl.scale_range, sh_full=wl.sh_full)
    env = synthetic.make_environment(*wl.env_hw, seed=wl.seed)
    alias = envmap.pack(envmap.build(env))
    w, h = res
    o, d = synthetic.pinhole_rays(w, h, synthetic.camera_positions(1, seed=wl.seed)[0])
    attrs = dict(build_pos=f["pos"], build_rot=f["rot"], build_scl=f["scl"], build_dns=f["dns"],
                 density=synthetic.density_tensor(f), material=synthetic.material_tensor(f), sph=f["sph"],
                 shading_normal=f["snrm"])
    g = np.random.default_rng(7).standard_normal((1, h, w, 3)).astype(np.float32) / float(h * w)
    dev = lambda t: t.to(device).contiguous()  # noqa: E731
    ori, drs = dev(torch.from_numpy(o[None].astype(np.float32))), dev(torch.from_numpy(d[None].astype(np.float32)))
    e_env, e_alias, t2w = dev(env), dev(alias), torch.eye(4, device=device).reshape(1, 4, 4)
    e = lambda *sh, dt=torch.float32: torch.empty(sh, dtype=dt, device=device)  # noqa: E731
    lights = (e(0, 9), e(5, 0), e(0, 3), e(0, 3, dt=torch.int32), e(0, 8), e(3, 0))

    out = {"reference": "FP64 oracle, same sample sequences",
           "sample": f"{wl.name} (config 4 scene): 1 view {w}x{h} at 1 spp, {wl.max_bounces} bounces",
           "tolerance": f"per sample |x - ref| <= {K.TOL_ABS} + {K.TOL_REL} |ref|"}
    t0 = time.perf_counter()
    for storage, rnd in (("fp32", None), ("bf16", torch.bfloat16), ("fp16", torch.float16)):
        held = {k: (t if rnd is None else t.to(rnd).float()) for k, t in attrs.items()}
        scene = dict({k: t.numpy() for k, t in held.items()}, environment=env.numpy(), alias_table=alias.numpy(),
                     ray_to_world=np.eye(4, dtype=np.float32)[None], frame=0, sph_degree=3, min_transmittance=0.001,
                     max_bounces=wl.max_bounces, ray_ori=o[None].astype(np.float32), ray_dir=d[None].astype(np.float32))
        cfg = O.OracleConfig()
        ref, _, _ = O.trace(cfg, scene, "f64")
        tr = OptixTracer("", "", "reference", "referenceBwd", "instances", 4, 0.0113, True, 3, True, True, True,
                         False, False, storage=storage, **shape)
        tr.build_bvh(dev(f["pos"]), dev(f["rot"]), dev(f["scl"]), dev(f["dns"]), True, True)
        scene_t = (dev(attrs["density"]), dev(attrs["material"]), dev(f["sph"]), dev(f["snrm"]), e_env, e_alias,
                   *lights)
        sig_t = torch.zeros((1, h, w), dtype=torch.int32, device=device)
        fwd = list(tr.trace(0, t2w, ori, drs, *scene_t, 0, 3, 0.001, wl.max_bounces, path_signature=sig_t))
        pbr = fwd[10].cpu().numpy()
        sig = sig_t.cpu().numpy().view(np.uint32)
        fwd[10] = torch.from_numpy(ref["pbr"]).to(device)
        fwd[11] = torch.from_numpy(ref["light"]).to(device)
        z = torch.zeros_like

        def gpu_bwd(grad):
            bw = tr.trace_bwd(0, t2w, ori, drs, *fwd[:8], fwd[10], fwd[11], *scene_t, z(fwd[0]), z(fwd[1]),
                              z(fwd[2]), z(fwd[3]), z(fwd[4]), z(fwd[5]), z(fwd[6]), z(fwd[7]),
                              torch.from_numpy(grad).to(device), z(fwd[11]), 0, 3, 0.001, wl.max_bounces)
            return bw[1].cpu().numpy(), bw[4].cpu().numpy()

        g_m = K.masked_grad(g, sig, ref["path_sig"])
        rep = K.image_report(pbr, ref["pbr"], sig, ref["path_sig"])
        rep["grad_all"] = K.grad_report(*gpu_bwd(g), *O.trace_bwd(cfg, scene, ref, dict(pbr=g), "f64")[:2])
        rep["grad_agree"] = K.grad_report(*gpu_bwd(g_m), *O.trace_bwd(cfg, scene, ref, dict(pbr=g_m), "f64")[:2])
        if storage == "fp32":
            # yardstick: the same estimator in float32 on the CPU (the oracle's FP32 instantiation)
            r32, _, _ = O.trace(cfg, scene, "f32")
            y = K.image_report(r32["pbr"], ref["pbr"], r32["path_sig"], ref["path_sig"])
            g32 = K.masked_grad(g, r32["path_sig"], ref["path_sig"])
            y["grad_all"] = K.grad_report(*O.trace_bwd(cfg, scene, ref, dict(pbr=g), "f32")[:2],
                                          *O.trace_bwd(cfg, scene, ref, dict(pbr=g), "f64")[:2])
            y["grad_agree"] = K.grad_report(*O.trace_bwd(cfg, scene, ref, dict(pbr=g32), "f32")[:2],
                                            *O.trace_bwd(cfg, scene, ref, dict(pbr=g32), "f64")[:2])
            out["oracle_fp32_vs_fp64"] = y
            out["gpu_fp32_vs_oracle_fp32"] = K.image_report(pbr, r32["pbr"], sig, r32["path_sig"])
        out[storage] = rep
        del tr
    out["seconds"] = round(time.perf_counter() - t0, 1)
    return out


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--gpus", type=int, default=1)
    ap.add_argument("--steps", type=int, default=3)
    ap.add_argument("--warmup", type=int, default=3)
    ap.add_argument("--workload", default="field-1m")
    # shrink the workload for profiling captures (the default bench line uses the full workload)
    ap.add_argument("--views", type=int, default=None)
    ap.add_argument("--res", default=None, help="WxH")
    ap.add_argument("--spp", type=int, default=None)
    ap.add_argument("--impl", default="ours", choices=("ours", "reference"))
    ap.add_argument("--graph", action="store_true", help="capture the training iteration in a CUDA graph")
    ap.add_argument("--no-autotune", action="store_true", help="use the default launch shape (k-buffer 16)")
    ap.add_argument("--autotune-full", action="store_true",
                    help="sweep k-buffer, block, chunk and refill (default: k-buffer and block)")
    ap.add_argument("--storage", default="bf16", choices=("fp32", "bf16", "fp16"),
                    help="attribute storage of the tracer (arithmetic is FP32 in every case)")
    ap.add_argument("--no-cpu-baseline", action="store_true")
    ap.add_argument("--no-accuracy", action="store_true", help="skip the error report against the FP64 oracle")
    ap.add_argument("--chunk-tiles", type=int, default=0, help="8x4 pixel tiles per wavefront chunk (0: tuned / default)")
    ap.add_argument("--schedule", default="wavefront", choices=("wavefront", "megakernel"),
                    help="megakernel: one thread per whole path, the plain drop-in schedule (use with --no-autotune)")
    ap.add_argument("--no-warp-aggregate", action="store_true",
                    help="one gradient atomic per lane and term (default: warp-aggregated rows)")
    ap.add_argument("--kbuffer", type=int, default=0, choices=(0, 8, 16, 24, 32),
                    help="candidates per traversal (0: the tuned or default size)")
    ap.add_argument("--resume-rounds", type=int, choices=(0, 1, 2), default=None,
                    help="k-buffer rounds resumed from the previous round's frontier: 0 backward replay (default), "
                         "1 none, 2 replay and intersection")
    ap.add_argument("--refill-lanes", type=int, default=0, help="waiting lanes before a warp refills (0: tuned / 32)")
    ap.add_argument("--block-size", type=int, default=0, choices=(0, 64, 128, 256),
                    help="threads per block of the wavefront stages (0: tuned / 128)")
    ap.add_argument("--bvh-builder", default="default", choices=("default", "morton", "ploc"),
                    help="hierarchy of the rebuild before the warm-up (the timed steps refit it)")
    ap.add_argument("--exact-candidates", action="store_true",
                    help="every traversal returns exactly the K nearest candidates (order independent)")
    args = ap.parse_args()

    rank = int(os.environ.get("RANK", "0"))
    world = int(os.environ.get("WORLD_SIZE", "1"))
    local = int(os.environ.get("LOCAL_RANK", "0"))

    if args.impl == "reference":
        if rank != 0:
            return
        # one bounded sample sized to ~budget seconds, timed once per step (median)
        steps = max(1, args.steps)
        base = cpu_sample(args, budget_s=max(3.0, min(10.0, 150.0 / steps)), repeats=steps)
        v = base["value"]
        wl = workload_of(args)
        print(json.dumps({
            "impl": "reference", "metric": metric_of(wl), "value": v, "unit": "segments/s", "n_gpus": args.gpus,
            "steps": args.steps, "warmup": args.warmup, "higher_is_better": True, "scaling": "weak",
            "vs_baseline": None, "dtype": "f32", "data": "synthetic",
            "config": dict(bench_config(wl, args, world), storage="fp32"),
            "cpu_baseline": {"value": v, "unit": "segments/s", "cores": base["cores"], "kind": "port",
                             "sample": base["sample"]},
            "e2e": {"value": v, "unit": "segments/s", "h2d_bytes_per_step": 0, "d2h_bytes_per_step": 0},
            "note": "the reference's OptiX tracer cannot be built here (OptiX SDK headers absent); its per-ray "
                    "math restated in C++ (oracle/oracle.cpp) runs on the host cores instead, in FP32 (the "
                    "reference's arithmetic and storage)",
        }))
        return

    if world > 1:
        import datetime

        import torch.distributed as dist

        torch.cuda.set_device(local)
        dist.init_process_group("nccl", timeout=datetime.timedelta(seconds=300))
    device = torch.device("cuda", local)
    torch.cuda.set_device(device)
    out = run_ours(args, rank, world, device)
    if world > 1:
        import torch.distributed as dist

        dist.barrier()
        dist.destroy_process_group()
    if rank == 0 and out is not None:
        res, S = out
        if world == 1 and not args.no_cpu_baseline:
            cb = cpu_sample(args, S)
            res["cpu_baseline"] = {k: cb[k] for k in ("value", "unit", "cores", "kind", "sample")}
        if world == 1 and not args.no_accuracy:
            shape = res["config"]["launch"] if isinstance(res["config"].get("launch"), dict) else {}
            res["accuracy"] = accuracy_sample(args, shape, device)
        print(json.dumps(res))


if __name__ == "__main__":
    main()
