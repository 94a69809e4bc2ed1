"""The line and ray stages of the sampled edges against the no-alloc backward,
whose line kernel takes one lane per item and drops nothing before the face
test: k_edge_line (phases over tiles of a warp's run, edges whose faces the
side rays surely miss dropped first, solves refilled lane by lane) must keep the
same samples.  Counts of kept and shaded samples are compared exactly, the
gradients to float round-off (atomic sums in another order).  Sizes: runs
shorter than a tile, one item more and less than a warp, many runs; meshes
whose faces are large and small against the rays' lean; both trees, both lobes
and the lobe mixture weight."""
import ctypes as C

import numpy as np
import pytest
import torch

from conftest import rel_err

pytestmark = pytest.mark.gpu


def _case(name):
    import scenes
    from delta_ray_b200 import workloads
    kind, res, spp = name.split()
    w, h = (int(x) for x in res.split("x"))
    if kind == "room":
        return scenes.icosphere_room(seed=3, n_spheres=8, subdiv=(1, 3), max_bounces=2, resolution=(w, h), spp=int(spp))
    grid = int(kind[2:])
    wl = workloads.heightfield(seed=2, resolution=(w, h), spp=int(spp), max_bounces=2, grid=grid, patch=16,
                               microfacet="ggx" if kind[0] == "g" else "blinn_phong")
    return wl


@pytest.mark.parametrize("name", ["hf24 1x1 1", "hf24 3x1 1", "hf24 33x17 2", "hf64 31x9 1", "hf128 24x20 1",
                                  "gf64 24x20 2", "room 37x29 2"])
@pytest.mark.parametrize("mis", [False, True])
def test_line_stage_keeps_the_samples_of_the_lane_per_item_kernel(name, mis):
    from delta_ray_b200 import _abi, _lib
    from delta_ray_b200.render_pytorch import RenderOptions, Scene
    wl = _case(name)
    cam, mats, shps, lts = _abi.scene_dicts(wl.camera, wl.materials, wl.shapes, wl.lights)
    W, H = wl.resolution
    d_image = torch.from_numpy(np.random.default_rng(5).uniform(0.5, 1.5, (H, W, 3)).astype(np.float32)).cuda()
    opts = RenderOptions(edge_lobe_mis=mis)
    sc = Scene(cam, mats, shps, lts, 0)
    try:
        g, _ = sc.backward(W, H, wl.spp, wl.max_bounces, 11, d_image, opts)
        work, counts = sc.last_work(), sc.last_counts()
        ref = torch.empty_like(g)
        L = _lib.lib()
        L.dr_render_backward_noalloc.argtypes = L.dr_render_backward.argtypes
        rd = _abi.render_desc(W, H, wl.spp, wl.max_bounces, 11, 0, opts.dp_mode, opts.flags)
        _lib.check(L.dr_render_backward_noalloc(sc.handle, C.byref(rd), C.c_void_p(d_image.data_ptr()),
                                                C.c_void_p(ref.data_ptr()), None, None))
        torch.cuda.synchronize()
        work0 = sc.last_work()
        assert sc.last_counts() == counts
        for k in ("survivors", "candidates", "shaded"):
            assert work[k] == work0[k], k
        # test_streaming_gpu.py's bound for the same terms summed in another order
        assert rel_err(g.cpu().numpy(), ref.cpu().numpy()) < 1e-5
    finally:
        sc.close()
