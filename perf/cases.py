"""What is measured of the surfel tracer: the work a user's program has it do, over the range of sizes it is used at.

A case is one iteration of such a program: rendering one view of a finished scene, or one training step (bring the
hierarchy up to date, trace, back-propagate). The scenes are the four kinds this repository's configurations are made of:

    ball       a small ball of large overlapping surfels (first steps of a reconstruction, smoke tests)
    object     surfels on the surface of one object against the void
    unbounded  a dense core inside a shell that reaches 50 units out, with a specularity per surfel for reflection bounces
    street     a ground plane and the faces of boxes, seen by spinning LiDARs (linear ray lists, precomputed colours)

Everything is made on the GPU from the seed: surfels, camera position, upstream gradients.

Fields of a case: scene; surfels; views x height x width rays (street: views sweeps of height beams x width azimuths);
layout "image" (one view), "batch" (views x (height*width) whole images) or "pixels" (random pixels of random views, as
a ray-batch trainer draws them); patch (an image that is a crop of a 1920-wide view: the same pixel spacing); task "train" or "render"; structure "keep" (static hierarchy), "refit" or "rebuild" on every
pass; calls (traces of one step before its backward); sh (degree the coefficient tensor holds, -1: precomputed colours) and
active (degree in use); bounces; white (background); distortion.
"""
import math
import os
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "diff-surfel-tracing_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

from diff_surfel_tracing import SurfelTracer, SurfelTracingSettings  # noqa: E402

_BASE = dict(views=1, layout="image", patch=False, task="train", structure="keep", calls=1, sh=3, active=3, bounces=0, white=False, distortion=False)


def _case(**kw):
    return {**_BASE, **kw}


def listed():
    return [
        # the smallest call there is: a thumbnail of a tiny scene; launches and host work are what it takes
        _case(name="tiny-render", scene="ball", surfels=10_000, height=64, width=64, task="render", sh=0, active=0),
        # the first steps of a small reconstruction: the same scene, forward and backward
        _case(name="tiny-train", scene="ball", surfels=10_000, height=128, width=128, sh=0, active=0),
        # a finished object shown in a viewer
        _case(name="object-render", scene="object", surfels=500_000, height=800, width=800, task="render", white=True),
        # training on one object: the surfels move a little every step, so the hierarchy is refitted
        _case(name="object-train", scene="object", surfels=500_000, height=800, width=800, structure="refit"),
        # two views, one loss: both are traced before the backward; early in training (degree 1 of a degree-3 tensor), with the
        # distortion regulariser switched on
        _case(name="object-two-views", scene="object", surfels=200_000, height=400, width=400, calls=2, active=1, white=True, distortion=True),
        # full-size training step of an unbounded scene with one reflection (the configuration of the headline benchmark)
        _case(name="reflective-train", scene="unbounded", surfels=3_000_000, height=1080, width=1920, bounces=1),
        # rendering such a scene at an odd size
        _case(name="reflective-render", scene="unbounded", surfels=1_000_003, height=721, width=1283, task="render", bounces=1),
        # patch-based training of a large scene after densification or pruning: full rebuild, few rays
        _case(name="reflective-patch", scene="unbounded", surfels=3_000_000, height=200, width=200, patch=True, structure="rebuild", bounces=1),
        # ray-batch training: random pixels of many views, nothing coherent between neighbours
        _case(name="ray-batch", scene="unbounded", surfels=500_000, views=8, height=1, width=30_000, layout="pixels", structure="refit", bounces=1),
        # four full LiDAR sweeps, colour and depth supervised
        _case(name="lidar-train", scene="street", surfels=1_000_000, views=4, height=64, width=2048, layout="sweeps", sh=-1, active=0),
        # one sweep of a smaller scanner, simulated in a finished scene
        _case(name="lidar-render", scene="street", surfels=300_000, height=32, width=900, layout="sweeps", task="render", sh=-1, active=0),
        # one GPU's share of the scale-out configuration: whole images in a batch, two reflections, rebuilt every step
        _case(name="scale-out-train", scene="unbounded", surfels=6_000_000, views=4, height=540, width=960, layout="batch", structure="rebuild", bounces=2),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    scene = rng.choice(["ball", "object", "object", "unbounded", "unbounded", "unbounded", "street"])
    c = _case(scene=scene, task=rng.choice(["train", "train", "render"]), structure="keep", white=rng.random() < 0.3)
    if scene == "street":
        c.update(surfels=_log(rng, 100_000, 2_000_000), views=rng.randint(1, 4), height=rng.choice([16, 32, 64]), width=_log(rng, 300, 2048),
                 layout="sweeps", sh=-1, active=0)
    else:
        lo, hi = {"ball": (2_000, 40_000), "object": (50_000, 1_000_000), "unbounded": (200_000, 5_000_000)}[scene]
        rays = _log(rng, 2_000, {"ball": 100_000, "object": 1_500_000, "unbounded": 1_000_000}[scene])
        aspect = rng.uniform(0.5, 1.2)
        h = max(16, int(math.sqrt(rays * aspect)))
        c.update(surfels=_log(rng, lo, hi), height=h, width=max(16, rays // h), sh=rng.choice([0, 3, 3]) if scene == "ball" else 3)
        c["active"] = rng.randint(0, c["sh"]) if rng.random() < 0.3 else c["sh"]
        if scene == "unbounded":
            c["bounces"] = rng.choice([0, 1, 1, 2])
            if rng.random() < 0.25:
                c.update(layout="pixels", views=8, height=1, width=min(rays, 60_000))
            elif rays < 100_000 and rng.random() < 0.5:
                c["patch"] = True
            elif rays > 100_000 and rng.random() < 0.3:
                c.update(layout="batch", views=2, height=h // 2)
    if c["task"] == "train":
        c["structure"] = rng.choice(["keep", "refit", "rebuild"])
        if scene == "object":
            c["distortion"] = rng.random() < 0.3
            if rng.random() < 0.2:
                c.update(calls=2, height=max(16, c["height"] // 2))
    return c


# ---- scenes ---------------------------------------------------------------------------------------------------

def _unit(n, g):
    d = torch.randn((n, 3), generator=g, device="cuda")
    return d / d.norm(dim=-1, keepdim=True)


def _quaternion_to(normal):
    """Rotations (w, x, y, z) that take the z axis to `normal`."""
    w = 1.0 + normal[:, 2:3]
    q = torch.cat([w, -normal[:, 1:2], normal[:, 0:1], torch.zeros_like(w)], dim=-1)
    q = torch.where(w < 1e-6, torch.tensor([0.0, 1.0, 0.0, 0.0], device="cuda"), q)
    return q / q.norm(dim=-1, keepdim=True)


def _scene(case, g):
    P, scene = case["surfels"], case["scene"]
    rn = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    ru = lambda *s: torch.rand(s, generator=g, device="cuda")  # noqa: E731
    if scene == "ball":
        means, scales = _unit(P, g) * ru(P, 1) ** (1 / 3), torch.exp(-4.0 + 0.5 * rn(P, 2))
        rots, opac = rn(P, 4), torch.sigmoid(1.5 * rn(P, 1))
    elif scene == "object":
        n = _unit(P, g)
        means, scales = n * (1.0 + 0.02 * rn(P, 1)), torch.exp(-5.0 + 0.4 * rn(P, 2))
        tilted = n + 0.1 * rn(P, 3)
        rots, opac = _quaternion_to(tilted / tilted.norm(dim=-1, keepdim=True)), torch.sigmoid(1.0 + rn(P, 1))
    elif scene == "unbounded":
        inner = torch.arange(P, device="cuda")[:, None] < 2 * P // 3
        u = ru(P, 1)
        r_out = torch.exp(math.log(2.0) + math.log(25.0) * u)
        means = _unit(P, g) * torch.where(inner, u ** (1 / 3), r_out)
        scales = torch.where(inner, torch.exp(-5.5 + 0.5 * rn(P, 2)), r_out * torch.exp(-4.0 + 0.5 * rn(P, 2)))
        rots, opac = rn(P, 4), torch.sigmoid(0.5 + 1.5 * rn(P, 1))
    else:
        flat = torch.arange(P, device="cuda") < P // 2
        centre, size = (ru(200, 3) - 0.5) * 90.0, 1.0 + 9.0 * ru(200, 3)
        centre[:, 2] = 0.5 * size[:, 2]
        box = torch.randint(0, 200, (P,), generator=g, device="cuda")
        axis = torch.randint(0, 3, (P,), generator=g, device="cuda")
        side = torch.randint(0, 2, (P,), generator=g, device="cuda").float() * 2 - 1
        onehot = torch.nn.functional.one_hot(axis, 3).float()
        on_box = centre[box] + torch.where(onehot > 0, 0.5 * side[:, None], ru(P, 3) - 0.5) * size[box]
        ground = torch.cat([(ru(P, 2) - 0.5) * 100.0, torch.zeros((P, 1), device="cuda")], dim=-1)
        normal = torch.where(flat[:, None], torch.tensor([0.0, 0.0, 1.0], device="cuda"), onehot * side[:, None])
        means, scales = torch.where(flat[:, None], ground, on_box), torch.exp(-3.0 + 0.4 * rn(P, 2))
        rots, opac = _quaternion_to(normal), torch.sigmoid(2.0 + rn(P, 1))
    s = dict(means3D=means, scales=scales, rotations=rots / rots.norm(dim=-1, keepdim=True), opacities=opac)
    if case["sh"] >= 0:
        shs = 0.05 * rn(P, (case["sh"] + 1) ** 2, 3)
        shs[:, 0] = 0.5 + 0.2 * rn(P, 3)
        s["shs"] = shs
    else:
        s["colors_precomp"] = ru(P, 3)
    if scene == "unbounded":
        s["others_precomp"] = ru(P, 2)
    return {k: v.contiguous() for k, v in s.items()}


# ---- rays -----------------------------------------------------------------------------------------------------

def _camera(case, height, width, angle):
    """K, R, T of a pinhole camera on a ring around the scene, looking at its centre."""
    radius, fov = {"ball": (3.0, 60.0), "object": (4.0, 40.0), "unbounded": (4.0, 50.0)}[case["scene"]]
    pos = torch.tensor([radius * math.sin(angle), -radius * math.cos(angle), 0.0])
    fwd = -pos / pos.norm()
    right = torch.linalg.cross(fwd, torch.tensor([0.0, 0.0, 1.0]))
    R = torch.stack([right, torch.linalg.cross(fwd, right), fwd])
    f = 0.5 * (1920 if case["patch"] else max(width, height)) / math.tan(math.radians(fov / 2))
    return torch.tensor([[f, 0.0, 0.5 * width], [0.0, f, 0.5 * height], [0.0, 0.0, 1.0]]), R, -(R @ pos)


def _rays(case, tracer, g, angles):
    """ray_o, ray_d of every trace call of one pass, the image size the settings name, and the camera of a single view."""
    V, H, W = case["views"], case["height"], case["width"]
    if case["layout"] == "sweeps":
        el, az = torch.deg2rad(torch.linspace(-25.0, 3.0, H, device="cuda"))[:, None], torch.arange(W, device="cuda") * (2 * math.pi / W)
        d = torch.stack([el.cos() * az.cos(), el.cos() * az.sin(), el.sin().expand(H, W)], dim=-1).reshape(1, H * W, 3)
        pos = torch.cat([(torch.rand((V, 2), generator=g, device="cuda") - 0.5) * 60.0, torch.full((V, 1), 1.8, device="cuda")], dim=-1)
        return [(pos[:, None].expand(V, H * W, 3).contiguous(), d.expand(V, -1, -1).contiguous())], (0, 0), None
    if case["layout"] == "image":
        cams = [_camera(case, H, W, a) for a in angles[: case["calls"]]]
        return [tracer.get_rays(H, W, *c) for c in cams], (H, W), cams[0]
    h, w = (H, W) if case["layout"] == "batch" else (1080, 1920)
    o, d = tracer.get_rays(h, w, *(torch.stack(x) for x in zip(*(_camera(case, h, w, a) for a in angles[:V]))))
    o, d = o.reshape(V, h * w, 3), d.reshape(V, h * w, 3)
    if case["layout"] == "batch":
        return [(o, d)], (h, w), None
    pick = torch.randint(0, V * h * w, (W,), generator=g, device="cuda")
    return [(o.reshape(-1, 3)[pick][None].contiguous(), d.reshape(-1, 3)[pick][None].contiguous())], (0, 0), None


# ---- one pass -------------------------------------------------------------------------------------------------

_OUTPUTS = ("rgb", "dpt", "acc", "norm", "dist", "aux", "mid", "wet")


def _supervised(case):
    """Outputs of a training step that receive a gradient."""
    if case["scene"] == "street":
        return ("rgb", "dpt")
    if case["scene"] == "object":
        return ("rgb", "acc", "norm") + (("dist",) if case["distortion"] else ())
    return ("rgb", "norm") if case["bounces"] else ("rgb",)


def prepare(case, seed):
    g = torch.Generator("cuda").manual_seed(seed)
    start = 2 * math.pi * ((seed * 0.6180339887) % 1.0)
    angles = [start + 2 * math.pi * k / 8 for k in range(max(case["views"], case["calls"], 1))]
    train = case["task"] == "train"
    tracer = SurfelTracer().train(train)
    if case["distortion"]:
        tracer.enable_distortion()
    params = _scene(case, g)
    rays, (ih, iw), camera = _rays(case, tracer, g, angles)
    bg = torch.full((3,), 1.0 if case["white"] else 0.0, device="cuda")
    eye = torch.eye(4, device="cuda")
    settings = SurfelTracingSettings(image_height=ih, image_width=iw, tanfovx=1.0, tanfovy=1.0, bg=bg, scale_modifier=1.0, viewmatrix=eye,
                                     projmatrix=eye, sh_degree=case["active"], campos=torch.zeros(3, device="cuda"), prefiltered=False,
                                     debug=False, max_trace_depth=case["bounces"], specular_threshold=0.3 if case["bounces"] == 2 else 0.5)
    vertices = tracer.build_from_surfels(params["means3D"], params["scales"], params["rotations"], rebuild=True)
    s = dict(case=case, tracer=tracer, params=params, rays=rays, camera=camera, settings=settings, vertices=vertices,
             grads3D=torch.zeros_like(params["means3D"]))
    if train:
        for p in (*params.values(), s["grads3D"]):
            p.requires_grad_(True)
        shapes = dict(rgb=3, dpt=1, acc=1, norm=3, dist=1)
        s["upstream"] = [[torch.randn((*o.shape[:2], shapes[n]), generator=g, device="cuda") for n in _supervised(case)] for o, _ in rays]
    return s


def run(s):
    case, tracer, p = s["case"], s["tracer"], s["params"]
    if case["structure"] != "keep":
        tracer.build_from_surfels(p["means3D"], p["scales"], p["rotations"], rebuild=case["structure"] == "rebuild", vertices=s["vertices"])
    if case["task"] == "render":
        with torch.no_grad():
            if s["camera"] is not None:
                out = tracer.forward_camera(case["height"], case["width"], *s["camera"], s["vertices"], grads3D=s["grads3D"], tracer_settings=s["settings"], **p)
            else:
                out = tracer(*s["rays"][0], s["vertices"], grads3D=s["grads3D"], tracer_settings=s["settings"], **p)
        return dict(zip(_OUTPUTS, out))
    outs = [dict(zip(_OUTPUTS, tracer(o, d, s["vertices"], grads3D=s["grads3D"], tracer_settings=s["settings"], **p))) for o, d in s["rays"]]
    names = _supervised(case)
    grads = torch.autograd.grad([o[n] for o in outs for n in names], [*p.values(), s["grads3D"]], [u for up in s["upstream"] for u in up])
    result = {"d_" + n: gr for n, gr in zip([*p, "grads3D"], grads)}
    for k, o in enumerate(outs):
        result.update({n + str(k): v.detach() for n, v in o.items()})
    return result


# ---- bounds and tolerance -------------------------------------------------------------------------------------

def _rays_of(case):
    return case["calls"] * (case["width"] if case["layout"] == "pixels" else case["views"] * case["height"] * case["width"])


def work(case):
    """Bytes: rays, surfel parameters and gradients each moved once (a rebuild reads the corners and writes the quads of the
    hierarchy on top). Operations: the contributions a ray of the scene composites (means of the listed cases) at about 150
    operations each, twice that again for their gradients; the search for them is left out."""
    R, P, train = _rays_of(case), case["surfels"], case["task"] == "train"
    floats = 3 + 2 + 4 + 1 + (3 * (case["active"] + 1) ** 2 if case["sh"] >= 0 else 3) + (2 if case["scene"] == "unbounded" else 0)
    stored = 3 + 2 + 4 + 1 + (3 * (case["sh"] + 1) ** 2 if case["sh"] >= 0 else 3) + (2 if case["scene"] == "unbounded" else 0) + 3
    outputs = 3 + 1 + 1 + 3 + 1 + 2 + 16 * max(2, case["bounces"] + 1)
    upstream = {"rgb": 3, "norm": 3}
    per_ray = 4 * (6 + outputs + (sum(upstream.get(n, 1) for n in _supervised(case)) if train else 0))
    per_surfel = 4 * (floats + ((stored + 1) if train else 0)) + (48 if case["structure"] != "keep" else 0)
    hits = {"ball": 6, "object": 20, "unbounded": (50, 80, 160)[case["bounces"]], "street": 10}[case["scene"]]
    return {"bytes": float(R * per_ray + P * per_surfel), "flops": float(R * hits * 150 * (3 if train else 1))}


def tolerance(case):
    """Per-surfel gradients and weights are 32-bit sums of up to some ten thousand terms of both signs, in no fixed order."""
    return {"rel": 1e-4, "max": 1e-2} if case["task"] == "train" else {"rel": 1e-5, "max": 1e-3}
