"""The queues' edges: frames whose path counts fall short of, fill and exceed a warp, a block of the
binning kernel (1024 entries) and a band of four pixel rows, on scenes that take each traversal
and shading kernel (plain surfaces, a sky, instances, media and subsurface walks).

The general path is the whole wavefront (no tail).  The tail kernels run the same shading code on the same
rays, and a region's pixels take the frame's samples, so films are equal bit for bit: no tolerance.
"""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scene(kind):
    S = importlib.import_module("photon_engine_b200.scenes")
    if kind == "cornell":
        return S.cornell_box(64, 64, 4, 8)
    if kind == "knot":
        return S.torus_knot_scene(64, 64, 4, 12, nu=256, nv=16, env_size=(97, 41))
    if kind == "grid":
        return S.instanced_grid_scene(64, 64, 4, 12, nx=2, nz=2, nu=128, nv=16, env_size=(64, 33))
    return S.media_scene(64, 64, 4, 24, n_leds=100, sphere_res=(48, 24), cyl_res=(32, 6), slab_res=4)


def _same(a, b):
    return all(np.array_equal(x.view(np.uint32), y.view(np.uint32)) for x, y in
               ((a.sum, b.sum), (a.sum_sq, b.sum_sq), (a.count, b.count)))


@pytest.mark.parametrize("kind", ["cornell", "knot", "grid", "media"])
def test_queue_edges(pe, device, kind):
    scene, cam, st = _scene(kind)
    scene.build_accelerator()
    device.set_scene(scene)
    try:
        for w, h, spp in ((1, 1, 1), (5, 3, 2), (31, 33, 1), (32, 32, 1), (41, 25, 1), (259, 130, 3)):
            st.width, st.height = w, h
            films = {}
            for tail in (0, 1 << 40, 1000, -1):
                device.set_tail_paths(tail)
                films[tail] = pe.Film(w, h)
                device.render(cam, st, pe.RenderTargets(beauty=films[tail]), 0, spp)
            for tail, f in films.items():
                assert _same(films[0], f), (w, h, tail)
            # a region that starts and ends inside bands of rows
            x0, y0, rw, rh = w // 3, h // 3, max(1, w // 2), max(1, h // 2)
            part = pe.Film(w, h)
            device.render_region(cam, st, part, (x0, y0, rw, rh), 0, spp)
            inside = np.zeros((h, w), bool)
            inside[y0:y0 + rh, x0:x0 + rw] = True
            for name in ("sum", "sum_sq", "count"):
                whole, got = getattr(films[0], name), getattr(part, name)
                assert np.array_equal(whole[inside], got[inside]), (w, h, name)
                assert not got[~inside].any(), (w, h, name)
            # the denoiser's films beside the beauty, traced by the wavefront and by the tail
            aovs = {}
            for tail in (0, 1 << 40):
                device.set_tail_paths(tail)
                t = pe.RenderTargets(beauty=pe.Film(w, h), aovs=pe.AovFilms(w, h))
                device.render(cam, st, t, 0, spp)
                aovs[tail] = t
            for name in ("albedo", "normal", "alpha"):
                assert _same(getattr(aovs[0].aovs, name), getattr(aovs[1 << 40].aovs, name)), (w, h, name)
            assert _same(films[0], aovs[0].beauty), (w, h)
    finally:
        device.set_tail_paths(-1)
