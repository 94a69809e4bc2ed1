"""Work counts of a backward call (Scene.last_work): the edges sampled by the
traversal's first stage are all of the call's where the traversal runs in one
stage (small trees, the warp walk of large ones, the no-alloc backward) and
fewer where it runs in two (the depth-first walk of large trees)."""
import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,stages", [(10, 1), (64, 1), (64, 2)])
def test_first_stage_edges(grid, stages):
    from delta_ray_b200 import _abi, _lib, workloads
    from delta_ray_b200.render_pytorch import Scene
    wl = workloads.heightfield(seed=2, resolution=(31, 23), spp=1, max_bounces=2, grid=grid, patch=16)
    sc = Scene(*_abi.scene_dicts(wl.camera, wl.materials, wl.shapes, wl.lights), 0)
    d_image = torch.ones(23, 31, 3, device="cuda")
    try:
        sc.set_tuning(depth_first=stages - 1)
        g, _ = sc.backward(31, 23, 1, 2, 11, d_image)
        w = sc.last_work()
        assert w["items"] > 0
        if stages == 1:
            assert w["items_first_stage"] == w["items"]
            L = _lib.lib()
            L.dr_render_backward_noalloc.argtypes = L.dr_render_backward.argtypes
            rd = _abi.render_desc(31, 23, 1, 2, 11, 0, 0, 0)
            _lib.check(L.dr_render_backward_noalloc(sc.handle, C.byref(rd), C.c_void_p(d_image.data_ptr()),
                                                    C.c_void_p(g.data_ptr()), None, None))
            torch.cuda.synchronize()
            w = sc.last_work()
            assert w["items_first_stage"] == w["items"] > 0
        else:
            assert w["items_first_stage"] < w["items"]  # none where every leaf lies deeper than its 8 levels
    finally:
        sc.close()
