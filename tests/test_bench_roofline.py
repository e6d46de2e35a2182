"""The bench's bytes per ray follow the trees that the rays walked: binary nodes of 64 bytes for closest hits
under closest_traversal 0, 4-wide nodes of 128 bytes for every other ray."""
import importlib.util
import pathlib
import types

import pytest

ROOT = pathlib.Path(__file__).resolve().parent.parent


@pytest.mark.parametrize("closest,node", [(0, 64), (6, 128)])
def test_bytes_per_ray_follow_the_tree(closest, node):
    spec = importlib.util.spec_from_file_location("bench_module", ROOT / "bench.py")
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    counted = types.SimpleNamespace(node_visits=1000, tri_tests=200, closest_rays=100, shadow_node_visits=300,
                                    shadow_tri_tests=30, shadow_rays=50)
    r = bench.traversal_roofline(closest, counted, 4000, 2000, 0.5)
    closest_bytes = 10 * node + 2 * 48 + 32 + 16 + 4      # nodes, triangles, ray, hit, queue entry
    shadow_bytes = 6 * 128 + 0.6 * 48 + 64 + 4            # nodes, triangles, record, queue entry
    assert r["bytes_per_ray"] == pytest.approx(closest_bytes)
    assert r["any_hit_bytes_per_ray"] == pytest.approx(shadow_bytes)
    assert r["achieved"] == pytest.approx((4000 * closest_bytes + 2000 * shadow_bytes) / 0.5e-3 / 1e9)
    assert ("kIntersectBinary" in r["kernel"]) == (closest == 0)
    assert bench.traversal_roofline(closest, counted, 4000, 2000, 0.0)["achieved"] is None
