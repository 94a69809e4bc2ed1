"""Performance cases of the differentiable renderer: what its users' programs
call, over the sizes they call it with.

A case is a plain dict: which entry point (`call`), which scene, and the
render's size and options.  `listed()` gives the fixed cases, `draw(rng)` one
more of the same ranges, `prepare(case, seed)` the state a user's program holds
before the call (a device scene, an image adjoint, host tensors), `run(state)`
one pass through the public entry points, `work(case)` the bytes and
operations a pass cannot do without, `exact(case, seed)` the results in 64 bits
where plain torch gives them.

Entry points:
* step      Scene.forward and Scene.backward on a scene that is kept, as an
            optimisation loop over materials or lights calls them
* forward   Scene.forward alone (final-quality and target images)
* apply     RenderFunction.apply and loss.backward() on host tensors, the
            drop-in interface: every call uploads and builds its scene
* fit       one view's part of an inverse-rendering step: Scene.update with new
            positions, forward, image loss, backward, with the unbiased
            estimator options of delta_ray_b200.inverse
* views     Scene.backward_views, several cameras of uneven size in one call
* proposal  Scene.backward with edges drawn through a trained edge proposal
* trace     Scene.trace, closest hits of a batch of rays
"""
import math

import numpy as np
import torch

from delta_ray_b200 import _abi, inverse, proposal, workloads
from delta_ray_b200.camera import Camera
from delta_ray_b200.light import Light
from delta_ray_b200.material import Material
from delta_ray_b200.render_pytorch import RenderFunction, RenderOptions, Scene
from delta_ray_b200.shape import Shape


def _case(name, call, scene, width, height, spp, bounces, **more):
    c = dict(call=call, scene=scene, width=width, height=height, spp=spp, bounces=bounces)
    c.update(more)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the reference's first demo at its own size: calls of well under a
        # millisecond of GPU work, where launches and synchronisation count
        _case("triangle step", "step", "triangle", 256, 256, 4, 1),
        # the soft-shadow demo: few triangles, many samples, direct lighting
        _case("soft shadow step", "step", "shadow", 512, 512, 16, 1),
        # the same demo through the drop-in interface, at a preview's odd size
        _case("soft shadow apply", "apply", "shadow", 201, 133, 4, 2),
        # a room of smooth spheres (shading normals, textures, two lobes, one
        # near-mirror): medium meshes, two bounces
        _case("room step", "step", "room", 320, 240, 4, 2, spheres=12, subdiv=2),
        # one multi-view call over the room, cameras of uneven size
        _case("room views", "views", "room", 128, 96, 2, 2, spheres=12, subdiv=2, views=6),
        # the glossy heightfield of the benchmark (130,050 triangles, three
        # bounces) at preview size and at full size, one sample per pixel each
        _case("heightfield preview step", "step", "heightfield", 160, 120, 1, 3, grid=256, ggx=False),
        _case("heightfield step", "step", "heightfield", 640, 480, 1, 3, grid=256, ggx=False),
        # its images: forward only
        _case("heightfield image", "forward", "heightfield", 640, 480, 16, 3, grid=256, ggx=False),
        # a smaller mesh with GGX lobes at a ragged size through the drop-in
        # interface (scene build and upload per call)
        _case("ggx heightfield apply", "apply", "heightfield", 203, 149, 2, 2, grid=128, ggx=True),
        # one view of the inverse-rendering loop at its default setting
        _case("heightfield fit", "fit", "heightfield", 128, 96, 8, 1, grid=64, ggx=False),
        # edges drawn through the learned proposal
        _case("heightfield proposal", "proposal", "heightfield", 160, 120, 1, 2, grid=64, ggx=False),
        # picking and visibility queries against the large mesh
        _case("heightfield rays", "trace", "heightfield", 0, 0, 0, 0, grid=256, ggx=False, rays=400_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: an entry point, a scene it is used with, and a size
    (odd ones included), no more costly than the largest listed case."""
    call = rng.choice(["step", "step", "step", "forward", "apply", "apply", "fit", "views", "proposal", "trace"])
    scene = {"fit": ["heightfield"], "proposal": ["heightfield"], "trace": ["heightfield", "room"],
             "views": ["room", "heightfield"]}.get(call, ["triangle", "shadow", "room", "heightfield", "heightfield"])
    scene = rng.choice(scene)
    more = {}
    if scene == "heightfield":
        more = dict(grid=_log_int(rng, 24, 64 if call in ("fit", "proposal") else 256), ggx=rng.random() < 0.3)
    elif scene == "room":
        more = dict(spheres=rng.randint(4, 16), subdiv=rng.randint(1, 3))
    if call == "views":
        more["views"] = rng.randint(2, 8)
    if call == "trace":
        return _case(None, call, scene, 0, 0, 0, 0, rays=_log_int(rng, 1000, 400_000), **more)
    most = {"triangle": 3e6, "shadow": 3e6, "room": 3e5, "heightfield": 2.5e5}[scene]
    if call == "forward":
        most = 4e6
    if call == "views":
        most /= more["views"]
    while True:
        width = _log_int(rng, 24, 640)
        height = max(16, int(round(width * rng.uniform(0.5, 1.1))))
        spp = rng.choice([1, 2, 3, 4, 8, 16])
        if 500 <= width * height * spp <= most:
            break
    return _case(None, call, scene, width, height, spp, 1 if call == "fit" else rng.choice([1, 2, 3, 4]), **more)


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _f32(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, np.float32)))


def _i32(a):
    return torch.from_numpy(np.ascontiguousarray(np.asarray(a, np.int32)))


def _camera(eye, look, fov, width, height):
    return Camera(position=_f32(eye), look_at=_f32(look), up=_f32([0, 1, 0]), cam_to_world=None, fov=_f32([fov]),
                  clip_near=_f32([0.01]), clip_far=_f32([10000.0]), resolution=[width, height])


def _icosphere(levels):
    t = (1.0 + 5.0 ** 0.5) / 2.0
    v = np.array([[-1, t, 0], [1, t, 0], [-1, -t, 0], [1, -t, 0], [0, -1, t], [0, 1, t], [0, -1, -t], [0, 1, -t],
                  [t, 0, -1], [t, 0, 1], [-t, 0, -1], [-t, 0, 1]], np.float64)
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    f = np.array([[0, 11, 5], [0, 5, 1], [0, 1, 7], [0, 7, 10], [0, 10, 11], [1, 5, 9], [5, 11, 4], [11, 10, 2],
                  [10, 7, 6], [7, 1, 8], [3, 9, 4], [3, 4, 2], [3, 2, 6], [3, 6, 8], [3, 8, 9], [4, 9, 5],
                  [2, 4, 11], [6, 2, 10], [8, 6, 7], [9, 8, 1]])
    for _ in range(levels):
        side = np.sort(np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]]), axis=1)
        uniq, inv = np.unique(side, axis=0, return_inverse=True)
        mid = v[uniq[:, 0]] + v[uniq[:, 1]]
        mid /= np.linalg.norm(mid, axis=1, keepdims=True)
        ab, bc, ca = np.split(inv.reshape(-1) + len(v), 3)
        v = np.concatenate([v, mid])
        a, b, c = f.T
        f = np.concatenate([np.stack(s, 1) for s in ((a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca))])
    return v, f


def _wall(center, ax, ay, facing):
    c, ax, ay = (np.asarray(x, np.float64) for x in (center, ax, ay))
    v = np.stack([c - ax - ay, c + ax - ay, c - ax + ay, c + ax + ay])
    f = np.array([[0, 1, 2], [1, 3, 2]])
    if np.dot(np.cross(v[f[0, 1]] - v[f[0, 0]], v[f[0, 2]] - v[f[0, 0]]), facing) < 0:
        f = f[:, [0, 2, 1]]
    return _f32(v), _i32(f)


def _room(case, seed):
    """A closed room with a textured floor, a ceiling light and smooth spheres
    (shading normals); the first sphere is a near-mirror."""
    rng = np.random.default_rng(seed)
    floor = Material(diffuse_reflectance=_f32(rng.uniform(0.2, 0.9, (16, 16, 3))),
                     specular_reflectance=_f32(rng.uniform(0.0, 0.3, (8, 8, 3))),
                     roughness=_f32(rng.uniform(0.1, 0.6, (8, 8, 1))), diffuse_uv_scale=_f32([2.0, 2.0]))
    mats = [Material(diffuse_reflectance=_f32([0.6, 0.6, 0.55]), two_sided=True), floor,
            Material(diffuse_reflectance=_f32([0.0, 0.0, 0.0]))]
    h = 5.0
    walls = [([0, 0, 0], [h, 0, 0], [0, 0, h], [0, 1, 0]), ([0, 2 * h, 0], [h, 0, 0], [0, 0, h], [0, -1, 0]),
             ([-h, h, 0], [0, 0, h], [0, h, 0], [1, 0, 0]), ([h, h, 0], [0, 0, h], [0, h, 0], [-1, 0, 0]),
             ([0, h, -h], [h, 0, 0], [0, h, 0], [0, 0, 1]), ([0, h, h], [h, 0, 0], [0, h, 0], [0, 0, -1])]
    shapes = []
    for k, w in enumerate(walls):
        v, f = _wall(*w)
        uv = (v[:, [0, 2]] + h) / (2 * h) if k == 0 else None
        shapes.append(Shape(v, f, uv, None, 1 if k == 0 else 0))
    v, f = _wall([0, 2 * h - 0.01, 0], [1.5, 0, 0], [0, 0, 1.5], [0, -1, 0])
    shapes.append(Shape(v, f, None, None, 2))
    lights = [Light(len(shapes) - 1, _f32([12.0, 12.0, 12.0]))]
    sv, sf = _icosphere(case["subdiv"])
    for k in range(case["spheres"]):
        rough = 0.006 if k == 0 else rng.uniform(0.1, 0.5)
        mats.append(Material(diffuse_reflectance=_f32(rng.uniform(0.1, 0.8, 3)),
                             specular_reflectance=_f32(rng.uniform(0.1, 0.4, 3)), roughness=_f32([rough])))
        r = rng.uniform(0.3, 1.2)
        c = np.array([rng.uniform(-3.5, 3.5), rng.uniform(r, 4.0), rng.uniform(-2.0, 3.5)])
        shapes.append(Shape(_f32(sv * r + c), _i32(sf), None, _f32(sv), len(mats) - 1))
    cam = _camera([0, 5, -4.5], [0, 3, 0], 60.0, max(1, case["width"]), max(1, case["height"]))
    return workloads.Workload("room", cam, mats, shapes, lights, [case["width"], case["height"]], case["spp"],
                              case["bounces"])


def _workload(case, seed):
    size = dict(resolution=(max(1, case["width"]), max(1, case["height"])), spp=max(1, case["spp"]),
                max_bounces=max(1, case["bounces"]))
    if case["scene"] == "triangle":
        return workloads.single_triangle(seed=seed, **size)
    if case["scene"] == "shadow":
        return workloads.soft_shadow(seed=seed, **size)
    if case["scene"] == "room":
        return _room(case, seed)
    return workloads.heightfield(seed=seed, grid=case["grid"], patch=max(8, case["grid"] // 8),
                                 microfacet="ggx" if case["ggx"] else "blinn_phong", **size)


def _views(case, seed):
    """Cameras of uneven resolution and sample count around the scene."""
    out = []
    for k in range(case["views"]):
        shrink = (1.0, 0.75, 1.25, 0.5)[k % 4]
        w, h = max(16, int(case["width"] * shrink)), max(16, int(case["height"] * shrink))
        if case["scene"] == "room":
            a = 2 * math.pi * k / case["views"]
            cam = _camera([4.2 * math.sin(a), 5.0, -4.2 * math.cos(a)], [0, 2.5, 0], 60.0, w, h)
        else:
            cam = inverse.view_cameras(case["views"], (w, h))[k]
        out.append(dict(camera=cam, width=w, height=h, spp=case["spp"] + (k % 2), max_bounces=case["bounces"],
                        seed=1000 * seed + k))
    return out


# ---------------------------------------------------------------------------
# state and passes
# ---------------------------------------------------------------------------
def _adjoint(height, width, gen):
    """The image adjoint of a mean squared error against a target."""
    return torch.randn(height, width, 3, generator=gen, device="cuda") * (2.0 * 0.1 / (3 * width * height))


def _rays(wl, n, gen):
    """Half from above the scene towards it, half from within it in all directions."""
    v = torch.cat([s.vertices for s in wl.shapes]).cuda()
    lo, hi = v.min(0).values, v.max(0).values
    o = lo + (hi - lo) * torch.rand(n, 3, generator=gen, device="cuda")
    d = torch.randn(n, 3, generator=gen, device="cuda")
    m = n // 2
    target = lo + (hi - lo) * torch.rand(m, 3, generator=gen, device="cuda")
    o[:m, 1] = hi[1] + 0.1 * (hi[1] - lo[1])
    d[:m] = target - o[:m]
    return torch.cat([o, torch.nn.functional.normalize(d, dim=1)], 1).contiguous()


def prepare(case, seed):
    wl = _workload(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    state = dict(call=case["call"], size=(case["width"], case["height"], case["spp"], case["bounces"]),
                 seed=seed % 1_000_003)
    if case["call"] == "apply":
        args = wl.serialize()
        leaves = [t for m in wl.materials for t in (m.diffuse_reflectance, m.specular_reflectance, m.roughness)]
        ids = {id(t) for t in leaves + [s.vertices for s in wl.shapes] + [light.intensity for light in wl.lights]}
        state["leaves"] = []
        for i, a in enumerate(args):
            if id(a) in ids:
                args[i] = a.detach().clone().requires_grad_(True)
                state["leaves"].append(args[i])
        state["args"] = args
        state["target"] = 0.5 * torch.rand(case["height"], case["width"], 3, generator=gen, device="cuda")
        return state
    cam, mats, shapes, lights = _abi.scene_dicts(wl.camera, wl.materials, wl.shapes, wl.lights)
    state["scene"] = Scene(cam, mats, shapes, lights, torch.cuda.current_device())
    if case["call"] == "trace":
        state["rays"] = _rays(wl, case["rays"], gen)
    elif case["call"] == "views":
        state["views"] = _views(case, seed % 1_000_003)
        for v in state["views"]:
            v["d_image"] = _adjoint(v["height"], v["width"], gen)
    elif case["call"] == "fit":
        # the positions the update brings: the heights of a fit under way
        rng = np.random.default_rng(seed + 1)
        moved = []
        for s in wl.shapes[:-2]:
            v = s.vertices.clone()
            v[:, 1] += _f32(rng.normal(0.0, 0.01, v.shape[0]))
            moved.append(Shape(v, s.indices, s.uvs, s.normals, s.mat_id))
        state["update"] = _abi.scene_dicts(wl.camera, wl.materials, moved + wl.shapes[-2:], wl.lights)
        state["target"] = 0.5 * torch.rand(case["height"], case["width"], 3, generator=gen, device="cuda")
        state["options"] = RenderOptions(dp_mode=_abi.DR_DP_SUM, detached_pdf=True, edge_lobe_mis=True,
                                         full_pixel_jitter=True)
    else:
        state["options"] = RenderOptions(learned_proposal=case["call"] == "proposal")
        state["d_image"] = _adjoint(max(1, case["height"]), max(1, case["width"]), gen)
        if case["call"] == "proposal":
            state["scene"].set_proposal(train=False, mix=0.8, params=proposal.init_params(seed))
    return state


def run(state):
    call, (width, height, spp, bounces), seed = state["call"], state["size"], state["seed"]
    if call == "apply":
        img = RenderFunction.apply(seed, *state["args"])
        loss = (img - state["target"]).square().mean()
        grads = torch.autograd.grad(loss, state["leaves"])
        return dict(image=img.detach(), loss=loss.detach(), grad=torch.cat([g.reshape(-1) for g in grads]))
    scene = state["scene"]
    if call == "trace":
        tri, t = scene.trace(state["rays"])
        return dict(tri=tri, t=t)
    if call == "views":
        grad, camera = scene.backward_views(state["views"])
        return dict(grad=grad, camera=camera)
    if call == "fit":
        scene.update(*state["update"])
        img = scene.forward(width, height, spp, bounces, seed, state["options"])
        diff = img - state["target"]
        grad, _ = scene.backward(width, height, spp, bounces, seed, (2.0 / diff.numel()) * diff, state["options"])
        return dict(image=img, grad=grad)
    out = {}
    if call in ("step", "forward"):
        out["image"] = scene.forward(width, height, spp, bounces, seed, state["options"])
    if call != "forward":
        out["grad"], _ = scene.backward(width, height, spp, bounces, seed, state["d_image"], state["options"])
    return out


# ---------------------------------------------------------------------------
# work and exact values
# ---------------------------------------------------------------------------
def _triangles(case):
    if case["scene"] == "triangle":
        return 3
    if case["scene"] == "shadow":
        return 8
    if case["scene"] == "room":
        return 14 + case["spheres"] * 20 * 4 ** case["subdiv"]
    return 2 * (case["grid"] - 1) ** 2 + 4


def _edges_per_sample(case):
    """Edges the edge-tree estimator samples per pixel sample (it walks every
    branch whose bound is high, so the count grows with the mesh's edges).
    Counted on these scenes (Scene.last_counts)."""
    if case["scene"] == "triangle":
        return 1.0
    if case["scene"] == "shadow":
        return 9.8
    if case["scene"] == "room":
        return 0.002 * _triangles(case)
    return 158.0 * (_triangles(case) / 7942.0) ** 0.84


def work(case):
    """bytes: the scene's arrays read and the image and gradients written, once
    each.  flops: float operations of the samples' rays (a box pair per level
    of a binary tree over the triangles and one triangle test), shading, and
    the edge samples (line sample, two rays, the walk's decisions)."""
    tris = _triangles(case)
    level = max(1.0, math.log2(tris))
    ray = 48.0 * level + 60.0
    mesh = 12.0 * (0.5 * tris + 2) + 12.0 * tris
    if case["call"] == "trace":
        return dict(bytes=case["rays"] * 32.0 + mesh, flops=case["rays"] * ray)
    samples = float(case["width"] * case["height"] * case["spp"])
    pixels = 12.0 * case["width"] * case["height"]
    if case["call"] == "views":
        scale = sum((1.0, 0.5625, 1.5625, 0.25)[k % 4] * (case["spp"] + k % 2) / case["spp"]
                    for k in range(case["views"]))
        samples *= scale
        pixels *= scale
    path = (1 + 2 * case["bounces"]) * ray + 300.0 * case["bounces"]
    flops = samples * path if case["call"] not in ("views", "proposal") else 0.0
    moved = mesh + pixels
    if case["call"] != "forward":
        edge = 300.0 + 0.25 * ray
        flops += samples * (2.0 * path + 2.0 * path + _edges_per_sample(case) * edge)
        moved += pixels + mesh
    return dict(bytes=moved, flops=flops)


def exact(case, seed):
    """Hit distances in 64 bits by testing every triangle.  The renders are
    Monte Carlo estimates over the renderer's own random streams, whose
    branches (hits, edge choices) are decided sample by sample: they have no
    value of their own in 64 bits."""
    if case["call"] != "trace":
        return None
    wl = _workload(case, seed)
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rays = _rays(wl, case["rays"], gen).double()
    tri = torch.cat([s.vertices.cuda().double()[s.indices.cuda().long()] for s in wl.shapes])
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    # Moeller-Trumbore's four numbers are linear in (d, o x d) and (o, 1):
    # det = -d.n, u det = d.(a x e2) + (o x d).e2, v det = d.(e1 x a) - (o x d).e1, t det = (o - a).n
    n = torch.cross(e1, e2, dim=1)
    mu = torch.cat([torch.cross(a, e2, dim=1), e2], 1)
    mv = torch.cat([torch.cross(e1, a, dim=1), -e1], 1)
    na = (n * a).sum(1)
    out = []
    for r in rays.split(max(1, int(5e8 // len(tri)))):
        o, d = r[:, :3], r[:, 3:]
        dm = torch.cat([d, torch.cross(o, d, dim=1)], 1)
        inv = -1.0 / (d @ n.T)
        u = (dm @ mu.T) * inv
        miss = u < 0
        v = (dm @ mv.T) * inv
        miss |= v < 0
        miss |= (u + v) > 1
        t = (o @ n.T - na) * inv
        miss |= ~(t > 1e-3)
        out.append(t.masked_fill_(miss, math.inf).min(1).values)
    return dict(tri=None, t=torch.cat(out))
