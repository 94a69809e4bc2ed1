"""The warp walk of large edge trees (k_edge_walk) against the depth-first
two-stage walk: the node decisions share their rules and the draws are keyed
by node, so both sample the same edges (equal counts and images) and the
gradients agree to the order of float atomic sums.  Sizes around what the walk
is cut by: calls of one point, fewer points than a batch, many points per
batch; both trees, both lobes, the learned proposal, leaves of several edges,
and walks long enough to be handed on in rounds."""
import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _stack(n=40):
    """n coincident copies of a small fan above a heightfield: each of its edges
    has n - 1 others with the same midpoint, so the edge tree's nodes over them
    cannot be split further and become leaves of n edges."""
    from delta_ray_b200 import workloads
    from delta_ray_b200.shape import Shape
    wl = workloads.heightfield(seed=2, resolution=(24, 20), spp=2, max_bounces=2, grid=64, patch=16)
    fan = workloads.soft_shadow(3, (24, 20)).shapes[1]
    for _ in range(n):
        wl.shapes.append(Shape(fan.vertices, fan.indices, None, None, 0))
    return wl


def _case(name):
    import scenes
    from delta_ray_b200 import workloads
    if name.startswith("heightfield"):
        res = {"1": (1, 1), "3": (3, 1), "many": (160, 120)}[name.split()[1]]
        wl = workloads.heightfield(seed=2, resolution=res, spp=1 if res[0] < 9 else 3, max_bounces=2, grid=64,
                                   patch=16, microfacet="ggx" if name.endswith("ggx") else "blinn_phong")
        for m in wl.materials[:3]:  # narrow lobes: long walks beside short ones
            m.roughness = torch.tensor([0.02])
        return wl
    if name == "room":  # the normal tree's cone and direction tests; the silhouette tree is small
        return scenes.icosphere_room(seed=3, n_spheres=8, subdiv=(2, 3), max_bounces=2, resolution=(37, 29))
    return _stack()


@pytest.mark.parametrize("name", ["heightfield 1", "heightfield 3", "heightfield many", "heightfield many ggx",
                                  "room", "stack"])
@pytest.mark.parametrize("learned", [False, True])
def test_warp_walk_samples_the_depth_first_walks_edges(name, learned):
    from delta_ray_b200 import _abi
    from delta_ray_b200.render_pytorch import RenderOptions, Scene
    wl = _case(name)
    cam, mats, shps, lts = _abi.scene_dicts(wl.camera, wl.materials, wl.shapes, wl.lights)
    W, H = wl.resolution
    d_image = torch.from_numpy(np.random.default_rng(5).uniform(0.5, 1.5, (H, W, 3)).astype(np.float32)).cuda()
    opts = RenderOptions(learned_proposal=learned)
    sc = Scene(cam, mats, shps, lts, 0)
    try:
        if learned:
            sc.set_proposal(train=False, mix=0.7)
        got = []
        for depth_first in (1, 0, 0):
            sc.set_tuning(depth_first=depth_first)
            g, img = sc.backward(W, H, wl.spp, wl.max_bounces, 11, d_image, opts, want_image=True)
            got.append((g.cpu().numpy(), img.cpu().numpy(), tuple(sc.last_counts()), sc.last_work()))
        g0, img0, c0, w0 = got[0]
        assert w0["tasks"] > 0 or c0[0] == 0  # the trees are walked in two stages
        for g, img, c, w in got[1:]:
            # GGX peaks of the narrowest lobes give NaN samples, the same ones each time
            assert c == c0 and np.array_equal(img, img0, equal_nan=True)
            assert w["survivors"] == w0["survivors"] and w["shaded"] == w0["shaded"]
            # both sum the same float terms in another order (test_streaming_gpu.py's bound)
            fine = np.isfinite(g0)
            assert np.array_equal(fine, np.isfinite(g)) and rel_err(g[fine], g0[fine]) < 1e-5
    finally:
        sc.close()
