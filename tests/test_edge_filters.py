"""Tests that decide an edge's or a node's fate before its exact evaluation,
compiled for the CPU and checked against that evaluation on random inputs and on
inputs near their margins, at scenes of very different sizes:

* bsdf_bound_side, a Blinn-Phong bound by its sides of 0 and 1 from fast
  divisions and roots (the device's errors of up to 2 ulps drawn at random);
* faces_out_of_reach, edges dropped because their samples' side rays cannot hit
  the edge's faces;
* fast_kids and leaf_entered, box tests with fused multiply-adds, against the
  binary walk.
"""
import numpy as np
import pytest

from native import harness


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


@pytest.mark.parametrize("scale", [0.01, 1.0, 300.0])
@pytest.mark.parametrize("ulps", [0, 2])
def test_side_bound_is_on_the_exact_bounds_side(scale, ulps):
    rng = np.random.default_rng([7, ulps])
    n = 200_000
    p = rng.uniform(-5, 5, (n, 3)) * scale
    normal = _unit(rng.normal(size=(n, 3)))
    cos = np.where(rng.random((n, 1)) < 0.5, rng.uniform(0, 1, (n, 1)),
                   1 - np.exp(rng.uniform(np.log(1e-6), 0, (n, 1))))  # towards normal incidence too
    wi = _unit(cos * normal + np.sqrt(1 - cos ** 2) * _unit(np.cross(normal, rng.normal(size=(n, 3)))))
    ext = np.exp(rng.uniform(np.log(1e-4), np.log(2), (n, 3))) * scale
    c = p + _unit(rng.normal(size=(n, 3))) * np.exp(rng.uniform(np.log(1e-2), np.log(12), (n, 1))) * scale
    rough = np.exp(rng.uniform(np.log(0.003), np.log(0.9), n))
    dl = np.where(rng.random(n) < 0.2, 0, rng.uniform(0, 1, n))
    sl = np.exp(rng.uniform(np.log(1e-3), 0, n))
    box = (c - ext, c + ext, p, normal, wi, dl)
    for near_one in (False, True):
        if near_one:  # reflectances that bring the exact bound within 1e-7 to 1e-2 of 1
            with np.errstate(all="ignore"):
                f = (1 - dl / np.pi) / (exact - dl / np.pi)
            off = np.exp(rng.uniform(np.log(1e-7), np.log(1e-2), n)) * rng.choice([-1, 1], n)
            sl = np.where(np.isfinite(f) & (f > 0), np.clip(sl * f * (1 + off), 1e-6, 1), sl)
        decided, side, margin, exact = harness.bound_side(*box, sl, rough, ulps)
        assert 0.3 < decided.mean() < 0.95
        assert np.array_equal(side[decided] > 1, exact[decided] > 1)
        assert np.array_equal(side[decided] <= 0, exact[decided] <= 0)
        assert (np.abs(side.astype(np.float64) - exact)[decided] <= (margin.astype(np.float64) * exact)[decided]).all()
    assert (np.abs(exact - 1) < 1e-2).mean() > 0.05


@pytest.mark.parametrize("scale", [0.1, 1.0, 10.0, 100.0, 300.0, 3000.0])
@pytest.mark.parametrize("squeeze", [1.0, 0.003])
def test_dropped_edges_have_no_face_hit(scale, squeeze):
    rng = np.random.default_rng([3, int(10 * scale)])
    n = 60_000
    p = rng.uniform(-1, 1, (n, 3)) * scale
    mid = p + _unit(rng.normal(size=(n, 3))) * scale * np.exp(rng.uniform(np.log(0.02), np.log(3), (n, 1)))
    size = scale * np.exp(rng.uniform(np.log(1e-4), 0, (n, 1)))
    half = _unit(rng.normal(size=(n, 3))) * size / 2
    v0, v1 = mid - half, mid + half
    normal = np.cross(v0 - p, v1 - p)
    normal /= np.maximum(np.linalg.norm(normal, axis=1, keepdims=True), 1e-30)
    dist = np.linalg.norm(mid - p, axis=1, keepdims=True)

    def opposite():  # out of the plane of p and the edge by a hundredth of the rays' lean to 30 times it
        q = mid + rng.normal(size=(n, 3)) * size * rng.choice([0.3, 1, 2], (n, 1))
        flat = q - ((q - mid) * normal).sum(1, keepdims=True) * normal
        out = 1e-3 * dist * dist * np.exp(rng.uniform(np.log(1e-2), np.log(30), (n, 1))) * rng.choice([-1, 1], (n, 1))
        return np.where(rng.random((n, 1)) < 0.8, flat + out * normal, q)
    a, b = opposite(), opposite()
    # lobe transforms: a rotation that brings the edge above the horizon, and a
    # lobe's stretch (squeeze: how narrow, at the least)
    rot, _ = np.linalg.qr(rng.normal(size=(n, 3, 3)))
    rot *= np.sign((rot[:, 2] * (mid - p)).sum(1))[:, None, None]
    lobe = np.zeros((n, 3, 3))
    stretch = np.exp(rng.uniform(np.log(squeeze), 0, (n, 2)))
    lobe[:, 0, 0], lobe[:, 1, 1], lobe[:, 2, 2] = stretch[:, 0], stretch[:, 1], 1
    lobe[:, 0, 2], lobe[:, 2, 0] = rng.uniform(-0.5, 0.5, (2, n))
    m = np.transpose(rot, (0, 2, 1)) @ lobe
    dropped, hits = harness.faces_reach(v0, v1, a, b, p, np.linalg.inv(m).reshape(n, 9), m.reshape(n, 9),
                                        [1e-4, 0.01, 0.2, 0.5, 0.8, 0.99, 0.9999])
    assert not (dropped & (hits > 0)).any()
    assert (hits > 0).mean() > 0.2 and dropped.any()


def test_fused_box_tests_answer_as_the_binary_walk():
    import scenes
    for wl in (scenes.heightfield_small(seed=1, grid=40), scenes.icosphere_room(seed=3, n_spheres=6, subdiv=(1, 2))):
        rng = np.random.default_rng(3)
        n = 8000
        rays = scenes.scene_rays(wl, n, 4)
        rays[: n // 8, 3 + rng.integers(0, 3)] = 0.0  # along a plane of the axes
        rays[n // 8: n // 4, 3:] = np.eye(3)[rng.integers(0, 3, n // 8)] * rng.choice([-1, 1], (n // 8, 1))
        verts = np.concatenate([np.asarray(s.vertices) for s in wl.shapes])
        rays[n // 4: n // 2, :3] = verts[rng.integers(0, len(verts), n // 4)]  # from the boxes' own corners
        tri, t, _ = harness.trace(wl, rays)
        hit = tri >= 0
        ta = np.where(hit, t, rng.uniform(1, 20, n)).astype(np.float32)
        ta = ta * rng.choice([1.0, 0.999, 1.001, 0.5], n).astype(np.float32)
        ida = np.where(hit, tri + rng.integers(-1, 2, n), rng.integers(0, 1000, n)).astype(np.int32)
        out = harness.trace_before_fast(wl, rays, ta, ida)
        assert np.array_equal(out[:, 0], out[:, 1]), int((out[:, 0] != out[:, 1]).sum())
        assert 0.02 < out[:, 0].mean() < 0.95  # both answers occur
