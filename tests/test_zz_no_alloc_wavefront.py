"""The no-allocation tile on the bounce-by-bounce wavefront: with the tail threshold below the tile's
paths its waves go through the queues, bins and shadow records of the fixed scratch.  The film does not
depend on the threshold, so it equals the allocating entry point's of the same traversal bit for bit
(the two traversals may settle ties between triangles differently, the tail kernel's is the 4-wide one's).
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind):
    S = importlib.import_module("photon_engine_b200.scenes")
    if kind == "cornell":
        return S.cornell_box(300, 200, 4, 8, seed=0)
    if kind == "grid":
        return S.instanced_grid_scene(300, 200, 4, 12, nx=2, nz=2, nu=128, nv=16, env_size=(64, 33))
    return S.media_scene(300, 200, 4, 16, n_leds=100, sphere_res=(48, 24), cyl_res=(48, 8), slab_res=6)


@pytest.mark.parametrize("kind", ["cornell", "grid", "media"])
def test_tile_wavefront_matches_allocating_entry_point(pe, device, kind):
    import torch

    scene, cam, st = _scene(kind)
    scene.build_accelerator()
    device.set_scene(scene)
    try:
        # part of a wave, a wave that fills the scratch's 32768 slots, several waves
        for x0, y0, w, h, spp in ((16, 8, 65, 41, 2), (40, 60, 256, 128, 1), (3, 5, 97, 113, 5)):
            wholes = {}
            for closest in (6, 0):
                device.set_tuning(tail_paths=0, closest_traversal=closest)
                wholes[closest] = pe.Film(st.width, st.height)
                device.render(cam, st, pe.RenderTargets(beauty=wholes[closest]), 0, spp)
            for tail, closest in ((0, 6), (1000, 6), (16576, 6), (-1, 6), (0, 0)):
                device.set_tuning(tail_paths=tail, closest_traversal=closest)
                whole = wholes[closest]
                s = torch.zeros((st.height, st.width, 3), dtype=torch.float32, device="cuda")
                c = torch.zeros((st.height, st.width), dtype=torch.int32, device="cuda")
                q = torch.zeros((st.height, st.width), dtype=torch.float32, device="cuda")
                torch.cuda.synchronize()
                device.render_tile_noalloc(cam, st, x0, y0, w, h, 0, spp, s.data_ptr(), c.data_ptr(), q.data_ptr())
                device.synchronize()
                tile = (slice(y0, y0 + h), slice(x0, x0 + w))
                got = {"sum": s.cpu().numpy(), "count": c.cpu().numpy().astype(np.uint32), "sum_sq": q.cpu().numpy()}
                for name, film in got.items():
                    expect = np.zeros_like(film)
                    expect[tile] = getattr(whole, name)[tile]
                    assert np.array_equal(film.view(np.uint32), expect.view(np.uint32)), (w, h, spp, tail, closest, name)
    finally:
        device.set_tuning()
