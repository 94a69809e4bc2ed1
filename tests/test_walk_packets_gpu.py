"""The warp walk of large edge trees (k_edge_walk) when its rounds cannot hand
their pending nodes on: with room for one packet, or for a few, warps walk on
themselves with their stacks nearly full, and sample the same edges as the
depth-first walk (equal counts and images, gradients to the order of float
sums).  Narrow lobes give walks long enough to be handed on; a roughness of 0
gives infinite and undefined bounds; the learned proposal a third share per
node."""
import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _case(name):
    import scenes
    from delta_ray_b200 import workloads
    if name == "room":
        return scenes.icosphere_room(seed=3, n_spheres=8, subdiv=(2, 3), max_bounces=2, resolution=(37, 29))
    wl = workloads.heightfield(seed=2, resolution=(61, 47), spp=2, max_bounces=2, grid=64, patch=16)
    for k, m in enumerate(wl.materials[:8]):
        m.roughness = torch.tensor([0.0 if name == "zero roughness" and k % 4 == 0 else 0.02])
    return wl


@pytest.mark.parametrize("name", ["narrow lobes", "zero roughness", "room"])
@pytest.mark.parametrize("learned", [False, True])
def test_walks_without_room_sample_the_same_edges(name, learned):
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

        def call(depth_first, packets):
            sc.set_tuning(depth_first=depth_first)
            sc.set_walk_packets(packets)
            g, img = sc.backward(W, H, wl.spp, wl.max_bounces, 11, d_image, opts, want_image=True)
            return g.cpu().numpy(), img.cpu().numpy(), tuple(sc.last_counts()), sc.last_work()
        g0, img0, c0, w0 = call(1, 0)
        fine = np.isfinite(g0)
        assert w0["packets"] == 0 and c0[1] > 0
        for packets in (0, 1, 7, 200):
            g, img, c, w = call(0, packets)
            assert c == c0 and np.array_equal(img, img0, equal_nan=True)
            assert w["survivors"] == w0["survivors"] and w["shaded"] == w0["shaded"]
            # the same float terms summed in another order (test_streaming_gpu.py's bound)
            assert np.array_equal(fine, np.isfinite(g)) and rel_err(g[fine], g0[fine]) < 1e-5
            if name != "room":  # walks are handed on, and find no room (the room's end before)
                assert w["packets"] > (packets if packets < 200 else 0)
    finally:
        sc.close()


def test_negative_packet_bound_is_refused():
    import scenes
    from delta_ray_b200 import _abi, _lib
    from delta_ray_b200.render_pytorch import Scene
    wl = scenes.SCENES["glossy_shadow"](seed=1)
    sc = Scene(*_abi.scene_dicts(wl.camera, wl.materials, wl.shapes, wl.lights), 0)
    try:
        with pytest.raises(_lib.DrError):
            sc.set_walk_packets(-1)
    finally:
        sc.close()
