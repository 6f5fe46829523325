"""Performance cases of the path tracer: the calls a program makes through the public entry points, over
the range of sizes, types and options in which they are used.

A case is a dict of plain values. ``prepare(case, seed)`` makes on the GPU what the program holds before
the call (scene, rays, tracer with its acceleration structure, light tables, optimizer state); ``run``
is one call of it. Kinds of case:

  forward    one image: Tracer's autograd function on an OptixTracer, one launch [spp, h, w]
  step       the traced part of a training step, the same way: refit of the acceleration structure,
             forward, and the backward of the gradients a loss hands back
  views      a training step over a batch of views of mixed resolution and sample count, on
             OptixTracer's trace_views and trace_bwd_views
  frame      one evaluation frame on the reference-facing Tracer: build_acc, then render
  iteration  one training iteration on Tracer: build_acc, render(train=True), the loss, backward()
  rebuild    a new acceleration structure (after the Gaussians were split, pruned or loaded) and a
             small preview image
  adam       the fused optimizer step of the SH and material groups for the Gaussians in view
  envmap     the importance table of an environment that a step has changed

Scenes follow ptir_b200/synthetic.py (uniform fields, and the cluster-and-shell field of a million
Gaussians; kernel degree 4, MIS and normals on), generated on the GPU. ``clamp`` is the density
clamping of the kernel support (particle_kernel_density_clamping): a program that has it on
rebuilds its structure every iteration (Tracer.build_acc), one that has it off refits.

A ray that leaves the field without becoming opaque ends at the last Gaussian it met, and with
clamping a Gaussian can be composited outside its own box; which of those a traversal reaches depends
on the order of the rays in the launch. In a launch larger than the device's resident threads (about
94,000 paths) that order differs from run to run, and with it about one path in 100,000. So the launches
above that size here are of the clustered field, whose shell is opaque, without clamping (or are
forward only), and the others stay below it.
"""
from __future__ import annotations

import math
from types import SimpleNamespace

import numpy as np
import torch

from ptir_b200 import OptixTracer, envmap, synthetic
from ptir_b200.lights import light_buffers
from ptir_b200.optim import SelectiveAdam
from ptir_b200.tracer import LightBuffers, Tracer

DEV = "cuda"
SPP = (1, 2, 4, 8)
STORAGES = ("fp32", "bf16", "fp16")


def _scene(name, kind, n, w, h, spp, bounces, env_h, env_w, clamp, layout="uniform", sh=False, storage="fp32",
           lights=False):
    return dict(name=name, kind=kind, n=n, w=w, h=h, spp=spp, bounces=bounces, env_h=env_h, env_w=env_w, clamp=clamp,
                layout=layout, sh=sh, storage=storage, lights=lights)


def listed():
    return [
        # a thumbnail of a small object while it is edited: the smallest call, latency alone
        _scene("preview-2k", "forward", 2_000, 61, 47, 1, 3, 32, 64, True),
        # the 10k-Gaussian field at 128x128, forward only (benchmark workload field-10k)
        _scene("field-10k", "forward", 10_000, 128, 128, 1, 2, 64, 128, True),
        # a training iteration at an early, coarse stage; clamped, so that each one rebuilds the structure
        _scene("iteration-20k", "iteration", 20_000, 151, 133, 4, 3, 64, 128, True),
        # an evaluation frame at an odd size with point, sphere and mesh lights
        _scene("frame-lights-30k", "frame", 30_000, 417, 333, 2, 3, 64, 128, False, lights=True),
        # a training iteration on the 100k-Gaussian field (benchmark workload field-100k), on an image crop
        _scene("iteration-100k", "iteration", 100_000, 200, 112, 4, 3, 256, 512, False),
        # a training step with degree-3 SH in 16-bit attribute storage (field-300k-sh), a crop of its 800x800
        _scene("step-300k-sh", "step", 300_000, 300, 300, 1, 3, 512, 1024, False, sh=True, storage="fp16"),
        # a batch of views of mixed resolution and spp in one launch sequence (as field-300k-mv)
        _scene("views-600k", "views", 600_000, 400, 256, 2, 3, 512, 1024, False, layout="cluster_shell"),
        # a training step of the headline workload, one of its views at 1 spp (field-1m)
        _scene("step-1m", "step", 1_000_000, 1024, 768, 1, 4, 512, 1024, False, layout="cluster_shell", storage="bf16"),
        # the structure of a million Gaussians after densification, and a thumbnail of it
        _scene("rebuild-1m", "rebuild", 1_000_000, 64, 48, 1, 2, 32, 64, True, layout="cluster_shell"),
        # the optimizer step of a medium scene: 48 SH coefficients and 5 material values a Gaussian
        dict(name="adam-300k", kind="adam", n=300_000, row=48, visible=0.6),
        # the importance table of a 512x1024 environment under optimisation, once a step
        dict(name="envmap-512", kind="envmap", h=512, w=1024, cube=False),
        # and of a cube map, whose table has a cell a texel
        dict(name="envmap-cube-48", kind="envmap", h=288, w=48, cube=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("forward", "forward", "step", "step", "views", "frame", "iteration", "rebuild", "adam", "envmap"))
    if kind == "adam":
        return dict(kind=kind, n=_log_int(rng, 1_000, 400_000), row=rng.choice((3, 4, 12, 27, 48)),
                    visible=round(rng.uniform(0.2, 1.0), 3))
    if kind == "envmap":
        if rng.random() < 0.4:
            fs = rng.randint(8, 48)
            return dict(kind=kind, h=6 * fs, w=fs, cube=True)
        h = _log_int(rng, 32, 512)
        return dict(kind=kind, h=h, w=2 * h + rng.choice((0, 0, 1, 6)), cube=False)
    # launches of about 2k to 250k paths; a million Gaussians only in the clustered layout they come in
    layout = rng.choice(("uniform", "uniform", "cluster_shell"))
    n = _log_int(rng, 2_000, 300_000) if layout == "uniform" else _log_int(rng, 200_000, 1_000_000)
    spp = rng.choice(SPP[:3])
    clamp = rng.random() < 0.5
    large = not clamp and (kind in ("forward", "frame") or n >= 600_000)
    most = 8_000 if kind == "rebuild" else 250_000 if large else 85_000
    px = _log_int(rng, 2_000, max(3_000, most // (spp + 5 if kind == "views" else spp)))
    w = max(8, int(round(math.sqrt(px * rng.uniform(0.6, 1.8)))))
    h = max(8, px // w)
    env_h = rng.choice((32, 64, 128, 256))
    return dict(kind=kind, n=n, w=w, h=h, spp=spp, bounces=rng.choice((2, 3, 3, 4)), env_h=env_h, env_w=2 * env_h,
                clamp=clamp, layout=layout, sh=rng.random() < 0.3,
                storage="fp32" if kind in ("frame", "iteration") or w * h * spp > 85_000 else rng.choice(STORAGES),
                lights=kind == "frame" and rng.random() < 0.5)


# ------------------------------------------------------------------------------------------
# inputs
def _unit(g, n, d):
    v = torch.randn((n, d), generator=g, device=DEV)
    return v / v.norm(dim=1, keepdim=True)


def _field(case, g):
    """The Gaussian field of synthetic.make_field, from a CUDA generator."""
    n = case["n"]
    rnd = lambda *s: torch.rand(s, generator=g, device=DEV)  # noqa: E731
    if case["layout"] == "cluster_shell":
        nc = int(round(0.7 * n))
        shell = _unit(g, n - nc, 3) * (5.0 + 15.0 * rnd(n - nc, 1))
        pos = torch.cat([torch.randn((nc, 3), generator=g, device=DEV), shell])
        lo, hi = 0.002, 0.2
    else:
        pos = 2.0 * rnd(n, 3) - 1.0
        lo, hi = (0.01, 0.08) if n < 10_000 else (0.005, 0.05)
    sph = torch.zeros((n, 48), device=DEV)
    if case["sh"]:
        sph.normal_(0.0, 0.1, generator=g)
    else:
        sph[:, :3].normal_(0.0, 0.5, generator=g)
    return dict(pos=pos.contiguous(), rot=_unit(g, n, 4),
                scl=torch.exp(math.log(lo) + (math.log(hi) - math.log(lo)) * rnd(n, 3)),
                dns=torch.sigmoid(torch.randn((n, 1), generator=g, device=DEV)), albedo=rnd(n, 3),
                roughness=0.05 + 0.95 * rnd(n, 1), metallic=rnd(n, 1), snrm=_unit(g, n, 3), sph=sph)


def _environment(h, w, g):
    env = torch.ones((h, w, 4), device=DEV)
    env[..., :3].log_normal_(0.0, 1.0, generator=g)
    return env


def _eyes(count, g):
    return (3.0 * _unit(g, count, 3)).cpu().numpy().astype(np.float64)


def _lights(env):
    return light_buffers([dict(type="point", position=(0.3, 1.5, -0.2), intensity=(2.0, 1.5, 1.0)),
                          dict(type="sphere", center=(-1.0, 1.2, 0.5), radius=0.25, radiance=(3.0, 3.0, 2.5)),
                          dict(type="sphere", center=(0.8, 0.9, 1.3), radius=0.1, radiance=(10.0, 2.0, 1.0), two_sided=True),
                          dict(type="mesh", vertices=[[-0.5, 2.0, -0.5], [0.5, 2.0, -0.5], [0.5, 2.0, 0.5], [-0.5, 2.0, 0.5]],
                               triangles=[[0, 1, 2], [0, 2, 3]], radiance=(4.0, 3.5, 3.0), two_sided=False)],
                         environment=env.cpu(), device=DEV)


class _Model:
    """The accessors Tracer reads from the program's Gaussian model."""

    n_active_features = 3
    rotation_activation = scale_activation = density_activation = staticmethod(lambda x: x)

    def __init__(self, f, env, table):
        self.positions, self.rotation, self.scale, self.density = f["pos"], f["rot"], f["scl"], f["dns"]
        self.features, self.snrm = f["sph"], f["snrm"]
        self.albedo, self.roughness, self.metallic, self.env = f["albedo"], f["roughness"], f["metallic"], env
        self.environment_alias_table = SimpleNamespace(
            prob=table["prob"].to(DEV), alias=table["alias"].to(DEV), pdf=table["pdf"].to(DEV), height=table["height"],
            width=table["width"])

    def trained(self):
        return self.albedo, self.roughness, self.env

    get_rotation = lambda self: self.rotation  # noqa: E731
    get_scale = lambda self: self.scale  # noqa: E731
    get_density = lambda self: self.density  # noqa: E731
    get_features = lambda self: self.features  # noqa: E731
    get_shading_normal = lambda self: self.snrm  # noqa: E731
    get_material_albedo = lambda self: self.albedo  # noqa: E731
    get_material_roughness = lambda self: self.roughness  # noqa: E731
    get_material_metallic = lambda self: self.metallic  # noqa: E731
    get_environment = lambda self: self.env  # noqa: E731

    def background(self, t2w, rays_dir, rgb, opacity, train):
        return rgb, opacity


def _conf(case):
    r = SimpleNamespace(pipeline_type="reference", backward_pipeline_type="referenceBwd", primitive_type="instances",
                        particle_kernel_degree=4, particle_kernel_min_response=0.0113,
                        particle_kernel_density_clamping=case["clamp"], particle_radiance_sph_degree=3, enable_normals=True,
                        enable_hitcounts=True, enable_mis=True, min_transmittance=0.001, max_bounces=case["bounces"],
                        max_consecutive_bvh_update=15, inversion_spp=case["spp"], render_spp=case["spp"],
                        filter_type="none", visualize_lights=case["lights"])
    return SimpleNamespace(render=r, model=SimpleNamespace(optimize_material_metallic=False), loss=None)


def _camera_batch(case, eye, lights):
    """A pinhole camera as the program's data loader hands it over: camera-space rays, the pose, the
    pixel coordinates and the intrinsics that Tracer expands the samples with."""
    w, h = case["w"], case["h"]
    fwd = -eye / np.linalg.norm(eye)
    up = np.array([0.0, 0.0, 1.0]) if abs(fwd[2]) < 0.999 else np.array([0.0, 1.0, 0.0])
    right = np.cross(fwd, up)
    right /= np.linalg.norm(right)
    pose = np.eye(4)
    pose[:3, 0], pose[:3, 1], pose[:3, 2], pose[:3, 3] = right, np.cross(fwd, right), fwd, eye
    focal = 0.5 * h / math.tan(math.radians(20.0))
    ys, xs = torch.meshgrid(torch.arange(h, device=DEV), torch.arange(w, device=DEV), indexing="ij")
    pix = torch.stack([xs, ys], -1).float().unsqueeze(0) + 0.5
    d = torch.stack([(pix[..., 0] - 0.5 * w) / focal, (pix[..., 1] - 0.5 * h) / focal, torch.ones((1, h, w), device=DEV)], -1)
    d = torch.nn.functional.normalize(d, dim=-1)
    extra = {}
    if lights is not None:
        extra = dict(lights=lights.lights, light_alias_table=lights.alias_table, mesh_light_vertices=lights.mesh_vertices,
                     mesh_light_triangles=lights.mesh_triangles, mesh_lights=lights.mesh_lights,
                     mesh_light_triangle_alias_table=lights.mesh_triangle_alias_table)
    return SimpleNamespace(rays_ori=torch.zeros_like(d), rays_dir=d, pixel_coords=pix,
                           intrinsics=torch.tensor([focal, focal, 0.5 * w, 0.5 * h], device=DEV),
                           T_to_world=torch.tensor(pose, dtype=torch.float32, device=DEV).unsqueeze(0), **extra)


def prepare(case, seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    kind = case["kind"]
    if kind == "adam":
        n = case["n"]
        params = [torch.nn.Parameter(torch.randn((n, k), generator=g, device=DEV)) for k in (case["row"], 5)]
        for p in params:
            p.grad = 1e-3 * torch.randn(p.shape, generator=g, device=DEV)
        visible = (torch.rand((n, 1), generator=g, device=DEV) < case["visible"]).float()
        return dict(kind=kind, params=params, visible=visible,
                    adam=SelectiveAdam([{"params": [p], "lr": 2.5e-3} for p in params], eps=1e-15))
    if kind == "envmap":
        return dict(kind=kind, env=_environment(case["h"], case["w"], g))

    f = _field(case, g)
    env = _environment(case["env_h"], case["env_w"], g)
    table = envmap.build(env)
    if kind in ("frame", "iteration"):
        model = _Model(f, env, table)
        batch = _camera_batch(case, _eyes(1, g)[0], _lights(env) if case["lights"] else None)
        tracer = Tracer(_conf(case))
        if kind == "frame":
            return dict(kind=kind, tracer=tracer, model=model, batch=batch)
        for p in model.trained():
            p.requires_grad_(True)
        shape = (1, case["h"], case["w"], 3)
        return dict(kind=kind, tracer=tracer, model=model, batch=batch,
                    target=torch.rand(shape, generator=g, device=DEV), prior=torch.rand(shape, generator=g, device=DEV))

    views = [(case["w"], case["h"], case["spp"])]
    if kind == "views":
        views = [(case["w"], case["h"], case["spp"]), (case["h"], case["w"], 1), (case["w"], case["w"], 2)]
    eyes = _eyes(len(views), g)
    rays = [synthetic.view_rays_device(w, h, spp, eye, DEV) for (w, h, spp), eye in zip(views, eyes)]
    t2w = torch.eye(4, device=DEV).reshape(1, 4, 4)
    if kind == "views":
        ori, dirs = (torch.cat([r[k].reshape(-1, 3) for r in rays]) for k in (0, 1))
        table_of_views = [(k, t2w, spp, h, w) for k, (w, h, spp) in enumerate(views)]
    else:
        (ori, dirs), table_of_views = rays[0], None
    e = lambda *s, dt=torch.float32: torch.empty(s, dtype=dt, device=DEV)  # noqa: E731
    none = (e(0, 9), e(5, 0), e(0, 3), e(0, 3, dt=torch.int32), e(0, 8), e(3, 0))
    tracer = OptixTracer("", "", "reference", "referenceBwd", "instances", 4, 0.0113, case["clamp"], 3, True, True, True,
                         False, False, storage=case["storage"])
    geometry = (f["pos"], f["rot"], f["scl"], f["dns"])
    state = dict(kind=kind, tracer=tracer, geometry=geometry, t2w=t2w, ori=ori, dirs=dirs, opts=(0, 3, 0.001, case["bounces"]))
    if kind != "rebuild":
        tracer.build_bvh(*geometry, True, True)
    if kind != "forward" and kind != "rebuild":
        # what an L1 loss on the image and an L2 loss on the material hand back
        lead, total = ori.shape[:-1], ori.numel() // 3
        state["pbr_grad"] = torch.sign(torch.randn((*lead, 3), generator=g, device=DEV)) * (0.8 / (3 * total))
        state["material_grad"] = torch.randn((*lead, 5), generator=g, device=DEV) / (5 * total)
        state["material_grad"][..., 4] = 0.0
    alias = envmap.pack(table, DEV)
    if kind == "views":
        state["views"] = table_of_views
        state["zeros"] = {c: torch.zeros((*lead, c), device=DEV) for c in (1, 2, 3)}
        state["scene"] = (torch.cat([f["pos"], f["dns"], f["rot"], f["scl"], torch.zeros_like(f["dns"])], 1),
                          torch.cat([f["albedo"], f["roughness"], f["metallic"]], 1), f["sph"], f["snrm"], env, alias, *none)
        return state
    state["trained"] = (f["albedo"], f["roughness"], env) if kind == "step" else ()
    for p in state["trained"]:
        p.requires_grad_(True)
    state["scene"] = (f["pos"], f["rot"], f["scl"], f["dns"], f["sph"], f["snrm"], f["albedo"], f["roughness"],
                      f["metallic"], env, alias, LightBuffers(*none))
    return state


# ------------------------------------------------------------------------------------------
# calls
def _trace(s):
    return Tracer._Autograd.apply(s["tracer"], 0, s["t2w"], s["ori"], s["dirs"], *s["scene"], *s["opts"])


def run(s):
    kind = s["kind"]
    if kind == "adam":
        s["adam"].step(s["visible"])
        return [(p.detach(), s["adam"].state[p]["exp_avg"], s["adam"].state[p]["exp_avg_sq"]) for p in s["params"]]
    if kind == "envmap":
        t = envmap.build_device(s["env"])
        return dict(prob=t[0], alias=t[1], pdf=t[2])
    if kind == "forward":
        return _trace(s)
    if kind == "rebuild":
        s["tracer"].build_bvh(*s["geometry"], True, True)
        return _trace(s)
    if kind == "frame":
        s["tracer"].build_acc(s["model"])
        with torch.no_grad():
            out = s["tracer"].render(s["model"], s["batch"], train=False, frame_id=3)
        return {k: v for k, v in out.items() if isinstance(v, torch.Tensor)}
    if kind == "iteration":
        model = s["model"]
        for p in model.trained():
            p.grad = None
        s["tracer"].build_acc(model, rebuild=False)
        out = s["tracer"].render(model, s["batch"], train=True, frame_id=3)
        loss = 0.8 * (out["pred_pbr"] - s["target"]).abs().mean() + 0.5 * (
            out["pred_material"][..., :3] - s["prior"]).square().mean()
        loss.backward()
        return dict(loss=loss.detach(), pbr=out["pred_pbr"].detach(), material=out["pred_material"].detach(),
                    opacity=out["pred_opacity"].detach(), grads=[p.grad for p in model.trained()])
    s["tracer"].build_bvh(*s["geometry"], False, True)
    if kind == "step":
        for p in s["trained"]:
            p.grad = None
        out = _trace(s)
        torch.autograd.backward([out[10], out[7]], [s["pbr_grad"], s["material_grad"]])
        return dict(forward=[t.detach() for t in out], grads=[p.grad for p in s["trained"]])
    fwd = s["tracer"].trace_views(s["views"], s["ori"], s["dirs"], *s["scene"], *s["opts"])
    (rad, dns, hit, hit2, dist, nrm, snrm, mat, _, _, pbr, light, _) = fwd
    z = s["zeros"]
    bwd = s["tracer"].trace_bwd_views(
        s["views"], s["ori"], s["dirs"], rad, dns, hit, hit2, dist, nrm, snrm, mat, pbr, light, *s["scene"], z[3], z[1],
        z[2], z[1], z[1], z[3], z[3], s["material_grad"], s["pbr_grad"], z[3], *s["opts"])
    return dict(forward=fwd, material_grad=bwd[1], environment_grad=bwd[4])


def exact(case, seed):
    """The optimizer step and the environment's pdf in 64 bits. The traced kinds have no such value: a path
    is a chain of discrete draws, which another precision takes differently. Neither have the alias
    table's cells, whose pairing any change of the weights' last bits reorders."""
    if case["kind"] == "adam":
        s = prepare(case, seed)
        out = []
        for p in s["params"]:
            g, vis = p.grad.double(), s["visible"] != 0
            m, v = 0.1 * g, 0.001 * g * g
            q = p.detach().double() - 2.5e-3 * m / (v.sqrt() + 1e-15)
            z = torch.zeros_like(g)
            out.append((torch.where(vis, q, p.detach().double()), torch.where(vis, m, z), torch.where(vis, v, z)))
        return out
    if case["kind"] == "envmap":
        env = prepare(case, seed)["env"][..., :3].double().cpu().numpy()
        if case["cube"]:
            fs = case["w"]
            edge = np.linspace(-1.0, 1.0, fs + 1)
            area = lambda u, v: np.arctan2(u * v, np.sqrt(u * u + v * v + 1.0))  # noqa: E731
            u0, u1, v0, v1 = edge[None, :-1], edge[None, 1:], edge[:-1, None], edge[1:, None]
            solid = np.tile(area(u1, v1) - area(u0, v1) - area(u1, v0) + area(u0, v0), (6, 1))
        else:
            th, tw = 64, 128
            h, w = env.shape[:2]
            cum = np.zeros((h + 1, w + 1, 3))
            cum[1:, 1:] = env.cumsum(0).cumsum(1)
            y0, x0 = np.arange(th) * h // th, np.arange(tw) * w // tw
            y1, x1 = -(-(np.arange(1, th + 1) * h) // th), -(-(np.arange(1, tw + 1) * w) // tw)
            total = cum[y1][:, x1] - cum[y0][:, x1] - cum[y1][:, x0] + cum[y0][:, x0]
            env = total / ((y1 - y0)[:, None, None] * (x1 - x0)[None, :, None])
            e = (np.arange(th + 1) / th - 0.5) * np.pi
            solid = np.repeat((2.0 * np.pi / tw) * (np.sin(e[1:]) - np.sin(e[:-1]))[:, None], tw, 1)
        weight = (env @ np.array([0.2126, 0.7152, 0.0722])) * solid
        return dict(prob=None, alias=None, pdf=weight / (weight.sum() * solid))
    return None


def work(case):
    """Bytes: every input read once and every output written once. Flops of a traced path: 32 composited
    Gaussians a segment at about 150 operations, over the segments of its bounces and shadow ray (the
    adjoint visits them again)."""
    kind = case["kind"]
    if kind == "adam":
        rows = case["n"] * (case["row"] + 5)
        return dict(bytes=4.0 * case["n"] + 28.0 * rows * case["visible"], flops=12.0 * rows * case["visible"])
    if kind == "envmap":
        cells = case["h"] * case["w"] if case["cube"] else 64 * 128
        return dict(bytes=16.0 * case["h"] * case["w"] + 12.0 * cells, flops=6.0 * case["h"] * case["w"] + 20.0 * cells)
    w, h, spp = case["w"], case["h"], case["spp"]
    paths = w * h * spp + (w * h + 2 * w * w if kind == "views" else 0)
    attribute = 4.0 * case["n"] * (12 + 5 + 48 + 3)
    env = 16.0 * case["env_h"] * case["env_w"]
    flops = 4800.0 * paths * (case["bounces"] + 1)
    total = attribute + env + 24.0 * paths + 124.0 * paths + 4.0 * case["n"]
    if kind in ("step", "views", "iteration"):
        total += attribute + env + 68.0 * paths + 20.0 * case["n"] + env
        flops *= 2.0
    if kind in ("rebuild", "frame", "iteration"):
        # the Gaussians' transforms in, leaves (64 bytes) and 4-wide nodes (59 bytes a leaf) out
        total += case["n"] * (44.0 + 64.0 + 59.0)
        flops += 200.0 * case["n"]
    return dict(bytes=total, flops=flops)
