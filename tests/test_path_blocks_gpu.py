"""The path kernels' two block sizes against the kernel logic compiled for the
CPU.

The forward and backward path kernels run in one large block per SM, whose
warps a barrier per sample (per bounce in the forward image) keeps in step, from
2,048 path threads per SM on, and in small blocks below: images just above that
line on a 148-SM GPU (their last block partly empty), just below it, and of one
pixel.  The side radiance of sampled edges runs in one large block per SM at
any size, fewer sides than one round of it included.  The loss weights a sprinkle
of pixels, so that the CPU's edge sampling stays small; counts of shading points
and edges are compared exactly, images and gradients within the parity bounds
of the other device tests.
"""
import numpy as np
import pytest
import torch

from conftest import assert_grad_parity, assert_image_parity
from native import harness

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scene,width,height,spp,bounces", [
    ("soft_shadow", 611, 497, 1, 1), ("soft_shadow", 610, 496, 1, 1), ("soft_shadow", 1, 1, 3, 1),
    ("heightfield_small", 611, 497, 1, 3), ("heightfield_small", 610, 496, 1, 3), ("heightfield_small", 1, 1, 2, 3),
    ("mirror_shadow", 379, 401, 2, 3), ("mirror_shadow", 61, 37, 6, 3)])
def test_block_sizes_match_the_cpu_build(scene, width, height, spp, bounces):
    import scenes
    from delta_ray_b200 import _abi, ltc, workloads
    from delta_ray_b200.render_pytorch import RenderOptions, Scene
    build = workloads.soft_shadow if scene == "soft_shadow" else scenes.SCENES[scene]
    wl = build(seed=6, resolution=(width, height), spp=spp, max_bounces=bounces)
    rng = np.random.default_rng(2)
    d_image = rng.uniform(0.5, 1.5, (height, width, 3)).astype(np.float32)
    if width * height > 1:
        d_image *= rng.random((height, width, 1)) < 600.0 / (width * height)
    samples = 2000
    table = ltc.default_table(0)  # the scene's default
    ref = harness.render(wl, 19, d_image, ltc_table=table, primary_edge_samples=samples)
    cam, mats, shps, lts = _abi.scene_dicts(wl.camera, wl.materials, wl.shapes, wl.lights)
    sc = Scene(cam, mats, shps, lts, 0)
    try:
        grad, img = sc.backward(width, height, spp, bounces, 19, torch.from_numpy(d_image).cuda(),
                                RenderOptions(primary_edge_samples=samples), want_image=True)
        assert tuple(sc.last_counts()) == tuple(ref["stats"])
        assert_image_parity(img.cpu().numpy(), ref["image"])
        assert_grad_parity(grad.cpu().numpy(), ref["grad"])
        assert_image_parity(sc.forward(width, height, spp, bounces, 19).cpu().numpy(),
                            harness.render(wl, 19, ltc_table=table)["image"])
    finally:
        sc.close()
