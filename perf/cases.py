"""Cases of the framework's work: what its users have it do, as calls of the
public API on the GPU, over the range of sizes and options that the bundled
configurations, tests and benchmark use.

Kinds of case (``case["kind"]``):

``step``     one optimisation step of a volume scene through the plain API:
             parameter update (state rotation, packing), two-state render with
             the control variate, L2 loss, adjoint and Adam.  ``adjoint`` names
             the adjoint integrator: path replay (``prb``) or the DRT adjoint
             (``volpathsimple``) that the grid experiments pair with it.
             ``views`` > 0 gives a batch film in a translated and scaled box,
             ``envmap`` an environment map, ``factor`` a majorant supergrid,
             ``albedo`` a constant, a grid of the density's resolution
             (``grid``) or of its own (``own``).
``surface``  the same step of the textured surface scene.
``target``   a single-state render with many samples per pixel (reference and
             validation images).
``batched``  one step of a mix of uneven jobs in the batched engine (graph).
``pixels``   the elementwise part of a step alone: loss with its gradient,
             Adam, and the control variate's statistics of two images.

The learning rates are those of the end of a schedule, so that the work of a
pass does not drift with the number of passes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import recursive_control_variates_gb300 as rcv
from recursive_control_variates_gb300 import core, scenes
from recursive_control_variates_gb300.batch import BatchedCV, CVJob

DEV = "cuda"
LR = 1e-4


def _step(name, dims, film, spp, depth, albedo="const", adjoint="prb", views=0, envmap=0, factor=0, blobs=8):
    return {"name": name, "kind": "step", "dx": dims[0], "dy": dims[1], "dz": dims[2], "width": film[0],
            "height": film[1], "spp": spp, "depth": depth, "albedo": albedo, "adjoint": adjoint, "views": views,
            "envmap": envmap, "factor": factor, "blobs": blobs}


def listed():
    return [
        # previews and unit-sized problems, of which a user runs thousands: launches and latency
        _step("step_16_64px", (16, 16, 16), (64, 64), 4, 16),
        # the first configuration of the benchmark: an interactive problem
        _step("step_32_128px", (32, 32, 32), (128, 128), 4, 16),
        # the headline configuration: density and RGB albedo, deep paths
        _step("step_64_512px", (64, 64, 64), (512, 512), 16, 64, albedo="grid"),
        # the largest served jobs
        _step("step_256_1024px", (256, 256, 256), (1024, 1024), 16, 32),
        # a captured scene: ragged grids of two resolutions in a placed box, several cameras, lit by a map
        _step("step_views_envmap", (67, 41, 53), (107, 83), 6, 24, albedo="own", views=5, envmap=256),
        # a mostly empty medium, for which the supergrid is switched on
        _step("step_sparse_supergrid", (128, 128, 128), (512, 512), 16, 64, factor=8, blobs=1),
        # the pairing of the grid experiments: two-state primal, DRT adjoint, cameras around a map-lit volume
        _step("drt_views_envmap", (72, 60, 72), (128, 128), 8, 32, albedo="grid", adjoint="volpathsimple", views=3,
              envmap=256),
        # the DRT adjoint on the headline configuration
        _step("drt_64_512px", (64, 64, 64), (512, 512), 16, 64, albedo="grid", adjoint="volpathsimple"),
        # texture recovery on the surface scene, the benchmark's configuration
        {"name": "surface_1024px", "kind": "surface", "width": 1024, "height": 1024, "tex": 512, "spp": 8, "depth": 8,
         "rr": 5},
        # a reference image of the headline medium
        {"name": "target_512px_256spp", "kind": "target", "dx": 64, "dy": 64, "dz": 64, "width": 512, "height": 512,
         "spp": 256, "depth": 64, "albedo": "grid", "envmap": 0, "blobs": 8},
        # many small and middle-sized jobs advanced together
        {"name": "batched_24_jobs", "kind": "batched", "jobs": 24, "mix": 4, "max_film": 512, "max_grid": 128,
         "depth": 32},
        # what is left of a step when the images are there
        {"name": "pixels_1023x767", "kind": "pixels", "width": 1023, "height": 767},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "step", "drt", "surface", "target", "batched", "pixels"])
    if kind in ("step", "drt"):
        drt = kind == "drt"
        most = 512 * 512 * (16 if drt else 48)  # paths of one pass
        d = _log_int(rng, 16, 128 if drt else 224)
        dims = tuple(max(8, int(d * rng.uniform(0.7, 1.0))) if rng.random() < 0.6 else d for _ in range(3))
        views = rng.choice([0, 0, 0, 2, 3, 6])
        w, spp = _log_int(rng, 48, 512 if drt else 1024), rng.choice([1, 2, 4, 5, 8, 16])
        h = max(16, int(w * rng.uniform(0.6, 1.1)))
        if views:
            w, h = max(24, w // 3), max(24, h // 3)
        spp = max(1, min(spp, most // (max(1, views) * w * h)))
        albedo = rng.choice(["const", "const", "grid", "own"])
        factor = rng.choice([0, 0, 0, 4, 8]) if min(dims) >= 32 else 0
        c = _step("", dims, (w, h), spp, rng.choice([8, 16, 24, 32, 48]), albedo,
                  "volpathsimple" if drt else "prb", views, rng.choice([0, 0, 64, 512]), factor, rng.choice([1, 4, 8]))
        del c["name"]
        return c
    if kind == "surface":
        w, spp = _log_int(rng, 64, 1024), rng.choice([1, 2, 3, 4, 8])
        return {"kind": "surface", "width": w, "height": max(32, int(w * rng.uniform(0.5, 1.0))),
                "tex": _log_int(rng, 32, 700), "spp": spp, "depth": rng.choice([3, 4, 6, 8]), "rr": rng.choice([3, 5])}
    if kind == "target":
        w = _log_int(rng, 64, 512)
        d = _log_int(rng, 16, 128)
        return {"kind": "target", "dx": d, "dy": max(8, int(d * rng.uniform(0.7, 1.0))), "dz": d, "width": w,
                "height": max(32, int(w * rng.uniform(0.6, 1.0))), "spp": _log_int(rng, 16, 256),
                "depth": rng.choice([8, 16, 32, 64]), "albedo": rng.choice(["const", "grid"]),
                "envmap": rng.choice([0, 0, 128]), "blobs": rng.choice([1, 8])}
    if kind == "batched":
        return {"kind": "batched", "jobs": rng.randint(2, 24), "mix": rng.randrange(1 << 16),
                "max_film": rng.choice([128, 256, 512]), "max_grid": rng.choice([32, 64, 128]),
                "depth": rng.choice([8, 16, 32])}
    w = _log_int(rng, 32, 2048)
    return {"kind": "pixels", "width": w, "height": max(17, int(w * rng.uniform(0.5, 1.0)))}


# ------------------------------------------------------------------- inputs
def blobs(dx, dy, dz, n, rng):
    """(dz, dy, dx, 1) sum of n Gaussian blobs, the family of scenes.blob_density."""
    centre, sigma, amp = rng.uniform(0.2, 0.8, (n, 3)), rng.uniform(0.05, 0.15, n), rng.uniform(5.0, 20.0, n)
    x, y, z = (torch.arange(d, device=DEV, dtype=torch.float32).add_(0.5).div_(d) for d in (dx, dy, dz))
    out = torch.zeros((dz, dy, dx), device=DEV)
    for (cx, cy, cz), s, a in zip(centre.tolist(), sigma.tolist(), amp.tolist()):
        gx, gy, gz = (torch.exp((c - m).square_() * (-0.5 / s ** 2)) for c, m in ((x, cx), (y, cy), (z, cz)))
        out += a * gz[:, None, None] * gy[None, :, None] * gx[None, None, :]
    return out[..., None]


def smooth_albedo(dx, dy, dz, seed):
    """(dz, dy, dx, 3) uniform values in [0.3, 0.95], smoothed by a Gaussian of two voxels."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    a = 0.3 + 0.65 * torch.rand((dz, dy, dx, 3), device=DEV, generator=g)
    weights = [math.exp(-0.5 * (k / 2.0) ** 2) for k in range(-4, 5)]
    for axis, n in enumerate((dz, dy, dx)):
        at = torch.arange(n, device=DEV)
        out = torch.zeros_like(a)
        for k, w in zip(range(-4, 5), weights):
            out += (w / sum(weights)) * a.index_select(axis, (at + k).clamp_(0, n - 1))
        a = out
    return a


def sky(width, rng):
    """(width / 2, width, 3) sky gradient with a soft sun: linear radiance."""
    h = width // 2
    v = (torch.arange(h, device=DEV, dtype=torch.float32) + 0.5) / h
    u = (torch.arange(width, device=DEV, dtype=torch.float32) + 0.5) / width
    su, sv = rng.uniform(0.2, 0.8), rng.uniform(0.15, 0.45)
    sun = torch.exp(-((u[None, :] - su) ** 2 + (v[:, None] - sv) ** 2) / (2 * 0.03 ** 2))
    base = 0.4 + 0.6 * (1.0 - v)[:, None].expand(h, width)
    return torch.stack([base * 0.7 + 12.0 * sun, base * 0.8 + 10.0 * sun, base + 7.0 * sun], dim=-1)


def _albedo(case, rng):
    if case["albedo"] == "const":
        return 0.8
    f = 0.6 if case["albedo"] == "own" else 1.0
    dims = [max(6, int(case[k] * f)) for k in ("dx", "dy", "dz")]
    return smooth_albedo(*dims, int(rng.integers(1 << 30)))


def _volume_scene(case, density, albedo, env, two_state):
    box = views = None
    if case.get("views"):
        box = core.T.translate((-0.6, 0.1, -0.5)).scale((1.3, 0.9, 1.1))
        views = scenes.orbit_views(box, case["views"], distance=2.2, height=0.3)
    d = scenes.scene_dict(density, 0.8, res=case["width"], height=case["height"], two_state=two_state,
                          spp=case["spp"], box=box, views=views)
    if isinstance(albedo, torch.Tensor):
        grid = {"type": "gridvolume", "data": albedo, **({"to_world": box} if box is not None else {})}
        interior = d["object"]["interior"]
        for medium in [interior["old"], interior["new"], interior["incoming"]] if two_state else [interior]:
            medium["albedo"] = grid
    if env is not None:
        d["emitter"] = {"type": "envmap", "data": env}
    return rcv.load_dict(d, device=DEV)


def _prepare_step(case, seed):
    rng = np.random.default_rng(seed)
    true = blobs(case["dx"], case["dy"], case["dz"], case["blobs"], rng)
    alb = _albedo(case, rng)
    env = sky(case["envmap"], rng) if case["envmap"] else None
    depth = {"max_depth": case["depth"], "rr_depth": case["depth"]}
    target = rcv.load_dict({"type": "prbvolpath", **depth}).render(_volume_scene(case, true, alb, env, False), 0,
                                                                 seed=seed % 65536 + 17, spp=8)
    scene = _volume_scene(case, true * 0.78, alb, env, True)
    if case["factor"]:
        scene.named_shapes()["object"].interior_medium().set_majorant_resolution_factor(case["factor"])
    cv = {"type": "cv", "integrator": {"type": "twostateprbvolpath", **depth}}
    if case["adjoint"] != "prb":
        cv["adjoint_integrator"] = {"type": case["adjoint"], **depth}
    integrator = rcv.load_dict(cv)
    params = rcv.traverse(scene)
    opt = rcv.ad.Adam(lr=LR)
    opt[scenes.DENSITY_KEY] = true * 0.78
    opt.set_bounds(scenes.DENSITY_KEY, 0.0, 250.0)
    if case["albedo"] != "const":
        opt[scenes.ALBEDO_KEY] = alb * 0.9
    params.update(opt)
    params.update(opt)
    opt[scenes.DENSITY_KEY] = true * 0.8  # the next iterate: old and new differ as in a running optimisation
    if case["albedo"] != "const":
        opt[scenes.ALBEDO_KEY] = alb * 0.91
    return {"kind": "step", "scene": scene, "params": params, "opt": opt, "integrator": integrator, "target": target,
            "spp": case["spp"], "i": seed % 10007}


def _prepare_surface(case, seed):
    tex = torch.as_tensor(scenes.value_noise(case["tex"], seed % 65536), device=DEV)
    d = scenes.surface_scene_dict(tex, case["width"], seed=seed % 65536, spp=case["spp"])
    d["sensor"]["film"]["height"] = case["height"]
    depth = {"max_depth": case["depth"], "rr_depth": case["rr"]}
    scene = rcv.load_dict(d, device=DEV)
    params = rcv.traverse(scene)
    target = rcv.load_dict({"type": "twostateprb", **depth}).render(scene, 0, seed=seed % 65536 + 17, spp=8)
    opt = rcv.ad.Adam(lr=LR)
    opt[scenes.TEXTURE_KEY] = 0.5 + 0.4 * (tex - 0.5)
    opt.set_bounds(scenes.TEXTURE_KEY, 0.0, 1.0)
    params.update(opt)
    params.update(opt)
    opt[scenes.TEXTURE_KEY] = 0.5 + 0.42 * (tex - 0.5)
    integrator = rcv.load_dict({"type": "cv", "integrator": {"type": "twostateprb", **depth}})
    return {"kind": "step", "scene": scene, "params": params, "opt": opt, "integrator": integrator, "target": target,
            "spp": case["spp"], "i": seed % 10007}


def _prepare_target(case, seed):
    rng = np.random.default_rng(seed)
    env = sky(case["envmap"], rng) if case["envmap"] else None
    scene = _volume_scene(case, blobs(case["dx"], case["dy"], case["dz"], case["blobs"], rng), _albedo(case, rng), env,
                          False)
    integrator = rcv.load_dict({"type": "prbvolpath", "max_depth": case["depth"], "rr_depth": case["depth"]})
    return {"kind": "target", "scene": scene, "integrator": integrator, "spp": case["spp"], "i": seed % 10007}


def _mix(case):
    """The size mix of a batch: grids, films and sample counts of the batched configuration."""
    rng = np.random.default_rng(case["mix"])
    grids = [g for g in (16, 32, 64, 128) if g <= case["max_grid"]]
    films = [f for f in (64, 128, 256, 512) if f <= case["max_film"]]
    return [(int(rng.choice(grids)), int(rng.choice(films)), int(rng.choice([4, 8, 16]))) for _ in range(case["jobs"])]


def _prepare_batched(case, seed):
    rng = np.random.default_rng(seed)
    depth = {"max_depth": case["depth"], "rr_depth": case["depth"]}
    base = rcv.load_dict({"type": "prbvolpath", **depth})
    jobs = []
    for k, (grid, film, spp) in enumerate(_mix(case)):
        true = blobs(grid, grid, grid, 8, rng)
        scene = rcv.load_dict(scenes.scene_dict(true, 0.8, res=film, two_state=False), device=DEV)
        target = base.render(scene, 0, seed=17843 + k, spp=8)
        jobs.append(CVJob(true * 0.8, 0.8, target, scene.sensors()[0], spp=spp, seed=seed % 65536 + 1000 * k, lr=LR,
                          density_bounds=(0.0, 250.0), device=DEV, **depth))
    return {"kind": "batched", "batch": BatchedCV(jobs), "jobs": jobs}


def _pixels_inputs(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    shape = (case["height"], case["width"], 3)
    img, ref, *renders = (torch.rand(shape, device=DEV, generator=g) for _ in range(6))
    return img, ref, renders


def _prepare_pixels(case, seed):
    img, ref, (h0, f0, h1, f1) = _pixels_inputs(case, seed)
    opt = rcv.ad.Adam(lr=0.02)
    opt["image"] = img
    stats = rcv.plugins.welford.StatisticsEstimator(0.9, 0.999)
    stats.update(h0, f0)  # the previous iteration's images
    return {"kind": "pixels", "opt": opt, "ref": ref, "H": h1, "F": f1, "stats": stats}


def prepare(case, seed):
    return {"step": _prepare_step, "surface": _prepare_surface, "target": _prepare_target,
            "batched": _prepare_batched, "pixels": _prepare_pixels}[case["kind"]](case, int(seed))


# --------------------------------------------------------------------- passes
def _run_step(s):
    opt = s["opt"]
    s["params"].update(opt)
    img = rcv.render(s["scene"], s["params"], integrator=s["integrator"], seed=s["i"], spp=s["spp"])
    loss = rcv.l2_loss(img, s["target"])
    loss.backward()
    opt.step()
    s["i"] += 1
    # the updated parameters and the moments, the first of which holds the gradient
    out = {"image": img.detach(), "loss": loss.detach(), "old": s["integrator"].H, "new": s["integrator"].F}
    for k, key in enumerate(sorted(opt.keys())):
        out["parameter%d" % k] = opt[key].detach()
        out["gradient_mean%d" % k] = opt.state[key][1]
    return out


def _run_target(s):
    return s["integrator"].render(s["scene"], 0, seed=s["i"], spp=s["spp"])


def _run_batched(s):
    s["batch"].step()
    return {"images": [j.image() for j in s["jobs"]],
            "densities_and_gradient_means": torch.cat([t.reshape(-1) for j in s["jobs"]
                                                       for t in (j.params(), j.density_m)])}


def _run_pixels(s):
    opt, stats = s["opt"], s["stats"]
    loss = rcv.l2_loss(opt["image"], s["ref"])
    loss.backward()
    opt.step()
    stats.update(s["H"], s["F"])
    vx, vy, cov = stats.get()
    return {"loss": loss.detach(), "image": opt["image"].detach(), "m": opt.state["image"][1], "v": opt.state["image"][2],
            "vx": vx, "vy": vy, "cov": cov}


def run(state):
    return {"step": _run_step, "target": _run_target, "batched": _run_batched, "pixels": _run_pixels}[state["kind"]](
        state)


# ----------------------------------------------------------- work and values
# Float operations of a free-flight step (random numbers, logarithm, position,
# trilinear lookup, weights) and of a surface bounce (two intersections with
# the scene, light and direction sampling), and how many of them an average
# path of these scenes takes (most camera rays miss the medium).
STEP_FLOPS, STEPS_PER_PATH, BOUNCE_FLOPS, BOUNCES_PER_PATH = 120, 8, 300, 2.5


def work(case):
    pixels = case.get("width", 0) * case.get("height", 0) * max(1, case.get("views") or 0)
    if case["kind"] == "pixels":
        n = 3.0 * pixels
        # read image, target, H, F; write the loss gradient, parameter, moments, statistics and their values
        return {"bytes": 4 * n * (4 + 1 + 3 + 5 + 3), "flops": 40 * n}
    if case["kind"] == "surface":
        return {"bytes": 4 * 3 * (pixels * 12.0 + case["tex"] ** 2 * 8.0),
                "flops": 2.0 * pixels * case["spp"] * BOUNCES_PER_PATH * BOUNCE_FLOPS}
    if case["kind"] == "batched":
        jobs = _mix(case)
        return {"bytes": sum(4.0 * 36 * f * f + 4.0 * 8 * g ** 3 for g, f, _ in jobs),
                "flops": sum(2.0 * f * f * spp for _, f, spp in jobs) * STEPS_PER_PATH * STEP_FLOPS}
    voxels = float(case["dx"] * case["dy"] * case["dz"]) * (1 if case["albedo"] == "const" else 4)
    if case["kind"] == "target":
        return {"bytes": 4 * (voxels + 3.0 * pixels), "flops": 1.0 * pixels * case["spp"] * STEPS_PER_PATH * STEP_FLOPS}
    times = 2.0 if case["adjoint"] == "prb" else 3.0  # the DRT adjoint traces a second path from each
    return {"bytes": 4 * (8 * voxels + 36.0 * pixels),
            "flops": times * pixels * case["spp"] * STEPS_PER_PATH * STEP_FLOPS}


def exact(case, seed):
    """The elementwise cases in 64 bits.  A traced image has no such value: the
    decisions of a path (real or null collision) are taken on its 32-bit
    numbers, and another rounding takes another path."""
    if case["kind"] != "pixels":
        return None
    img, ref, renders = _pixels_inputs(case, int(seed))
    f32 = lambda x: float(np.float32(x))  # noqa: E731  (the library's scalars are 32-bit numbers)
    b1, b2, eps = f32(0.9), f32(0.999), f32(1e-8)
    img, ref = img.double(), ref.double()
    diff = img - ref
    g = 2.0 * diff / img.numel()
    m, v = (1.0 - b1) * g, (1.0 - b2) * g * g
    new = img - f32(0.02) * math.sqrt(1.0 - b2) / (1.0 - b1) * m / (v.sqrt() + eps)
    # two EMA-Welford updates: deviations from the bias-corrected means before and after each
    h0, f0, h1, f1 = (t.double() for t in renders)
    mx, my = torch.zeros_like(img), torch.zeros_like(img)
    vx, vy, cov = torch.zeros_like(img), torch.zeros_like(img), torch.zeros_like(img)
    for n, (x, y) in enumerate(((h0, f0), (h1, f1))):
        prev = 1.0 - b1 ** n if n else 1.0
        dx, dy = x - mx / prev, y - my / prev
        mx, my = b1 * mx + (1.0 - b1) * x, b1 * my + (1.0 - b1) * y
        ex, ey = x - mx / (1.0 - b1 ** (n + 1)), y - my / (1.0 - b1 ** (n + 1))
        vx, vy = b2 * vx + (1.0 - b2) * dx * ex, b2 * vy + (1.0 - b2) * dy * ey
        cov = b2 * cov + (1.0 - b2) * dx * ey
    d2 = 1.0 - b2 ** 2
    return {"loss": diff.square().mean(), "image": new, "m": m, "v": v, "vx": vx / d2, "vy": vy / d2, "cov": cov / d2}
