"""The line stage on scenes of 1 to 3,000 units across: edges whose faces the side
rays surely miss are dropped by a bound in scene units (faces_out_of_reach), and
the same samples must be kept as by the no-alloc backward's line kernel, which
drops none before the face test.  Images of one, two and many pixels, item
counts that are no multiple of a warp among them."""
import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scale", [0.1, 1.0, 30.0, 100.0, 300.0])
@pytest.mark.parametrize("kind", ["heightfield", "room"])
def test_scaled_scenes_keep_the_same_samples(kind, scale):
    import scenes
    from delta_ray_b200 import _abi, _lib, workloads
    from delta_ray_b200.camera import Camera
    from delta_ray_b200.render_pytorch import Scene
    size, eye, look = (37, 23), [0, 7, -9], [0, 0, 0]
    if kind == "heightfield":
        wl = workloads.heightfield(seed=2, resolution=size, spp=1, max_bounces=2, grid=48, patch=16)
    else:
        wl = scenes.icosphere_room(seed=3, n_spheres=8, subdiv=(1, 3), max_bounces=2, resolution=size, spp=1)
        eye, look = [0, 5, -4.5], [0, 3, 0]
    f = lambda x: torch.tensor(x, dtype=torch.float32)
    wl.camera = Camera(position=f(eye) * scale, look_at=f(look) * scale, up=f([0.0, 1.0, 0.0]), cam_to_world=None,
                       fov=f([45.0]), clip_near=f([0.01]), clip_far=f([10000.0]), resolution=list(size))
    for sh in wl.shapes:
        sh.vertices = sh.vertices * scale
    sc = Scene(*_abi.scene_dicts(wl.camera, wl.materials, wl.shapes, wl.lights), 0)
    d_image = torch.from_numpy(np.random.default_rng(5).uniform(0.5, 1.5, (size[1], size[0], 3)).astype(np.float32)).cuda()
    L = _lib.lib()
    L.dr_render_backward_noalloc.argtypes = L.dr_render_backward.argtypes
    counts = set()
    try:
        for w, h in ((1, 1), (2, 1), size):
            d = d_image[:h, :w].contiguous()
            g, _ = sc.backward(w, h, 1, 2, 11, d)
            work = sc.last_work()
            rd = _abi.render_desc(w, h, 1, 2, 11, 0, 0, 0)
            _lib.check(L.dr_render_backward_noalloc(sc.handle, C.byref(rd), C.c_void_p(d.data_ptr()),
                                                    C.c_void_p(g.data_ptr()), None, None))
            torch.cuda.synchronize()
            work0 = sc.last_work()
            for k in ("items", "survivors", "candidates", "shaded"):
                assert work[k] == work0[k], (w, h, k)
            counts.add(work["items"] % 32 != 0)
        assert True in counts and work["survivors"] > 0
    finally:
        sc.close()
