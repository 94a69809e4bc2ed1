"""bench.py's memory roofline (no GPU): a kernel whose profiled DRAM traffic is
far below the copy rate is not reported as bound by HBM, whatever its byte model
counts, and the byte model of the edge shading holds the multi-bounce rays of a
step once, in the kernel that traces them."""
import os
import sys

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
import bench  # noqa: E402


def test_bound_follows_the_profiled_traffic():
    r = bench.memory_roofline(300.0, 1.1e12, 35e9, 6470.0)
    assert r["bound"] != "hbm" and r["bytes"] != "model" and abs(r["achieved"] - 35e9 / 0.3 / 1e9) < 1e-6
    assert abs(r["frac"] - r["achieved"] / 6470.0) < 1e-12
    assert bench.memory_roofline(1.0, 0, 5e9, 6470.0)["bound"] == "hbm"
    assert bench.memory_roofline(1.0, 5e9, None, 6470.0) == {
        "bound": "hbm", "achieved": 5000.0, "frac": 5000.0 / 6470.0, "bytes": "model"}
    assert bench.memory_roofline(0.0, 5e9, None, 6470.0)["achieved"] == 0.0


def test_paths_of_the_sides_are_counted_once():
    class Wl:
        resolution, spp, max_bounces, num_triangles = (64, 48), 1, 3, 130054
    work = {"points": 10, "items": 100, "shaded": 7}
    ray = bench.ray_bytes(Wl.num_triangles)
    radiance = bench.kernel_bytes("k_edge_radiance", Wl, work)
    assert radiance >= 7 * 10 * ray
    assert bench.kernel_bytes("k_edge_shade", Wl, work) < 7 * 3 * ray
