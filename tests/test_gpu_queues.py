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


@pytest.mark.parametrize("kind", ["cornell", "knot", "grid", "media", "room_guided"])
def test_feature_kernels_equal_the_full_kernel(pe, device, kind):
    """Waves are shaded by kernels that carry their scene's features only; a counting device takes the
    kernels with all of them, over the same paths: the films are equal bit for bit.  The guided wave is
    a fresh network's first, whose training step comes after it."""
    if kind == "room_guided":
        S = importlib.import_module("photon_engine_b200.scenes")
        scene, cam, st = S.room_scene(64, 36, 4, 8)
    else:
        scene, cam, st = _scene(kind)
    scene.build_accelerator()
    device.set_scene(scene)
    films = []
    try:
        device.set_tail_paths(0)
        for counting in (False, True):
            if kind == "room_guided":
                device.set_guiding(0)
                device.set_guiding(1, 0, 0.0)
                pe._capi.check(pe._capi.load().pe_device_guide_reset(device.handle, 7, None, None))
            device.set_counting(counting)
            films.append(pe.Film(st.width, st.height))
            device.render(cam, st, pe.RenderTargets(beauty=films[-1]), 0, 4)
    finally:
        device.set_counting(False)
        device.set_tail_paths(-1)
        device.set_guiding(0)
    assert _same(*films)


def test_tail_vertices_stay_unguided(pe, device):
    """The tail kernel runs no inference.  A camera that sees a small mirror and nothing else has no
    guidable first vertex, and the few paths left go to the tail after it: the guided film is the plain one."""
    S = importlib.import_module("photon_engine_b200.scenes")
    scene = pe.Scene()
    grey = pe.Lambertian((0.6, 0.5, 0.4))
    for p, u, v, mat in (((-0.5, 0, 3), (1, 0, 0), (0, 1, 0), pe.Mirror((0.9, 0.9, 0.9))),
                         ((-9, -9, -6), (18, 0, 0), (0, 18, 0), grey), ((-9, -2, -9), (18, 0, 0), (0, 0, 9), grey)):
        pos, idx = S._wall_grid(tuple(map(float, p)), tuple(map(float, u)), tuple(map(float, v)), 4, 4, None)
        scene.add_shape(pe.TriangleMesh(pos, None, None, idx, mat))
    scene.add_light(pe.AreaLight((-1.0, 4.0, -3.0), (2.0, 0.0, 0.0), (0.0, 0.0, 2.0), (9.0, 9.0, 8.0)))
    scene.build_accelerator()
    device.set_scene(scene)
    st = pe.RenderSettings(width=64, height=64, max_bounces=6, seed=3)
    cam = pe.PerspectiveCamera((0.0, 0.5, 0.0), (0.0, 0.5, 3.0), (0.0, 1.0, 0.0), 40.0, 1.0)
    films = []
    try:
        for guided in (False, True):
            device.set_guiding(1 if guided else 0, 0, 0.0)
            films.append(pe.Film(64, 64))
            device.render(cam, st, pe.RenderTargets(beauty=films[-1]), 0, 1)
            if guided:
                assert 0 < device.last_stats().tail_paths <= 2048
    finally:
        device.set_guiding(0)
    assert films[0].sum.max() > 0.0
    assert _same(*films)


def test_moving_instances_in_a_regenerating_wave(pe, device):
    """Waves over moving instances trace their shadow rays before a slot is handed on and flush ended
    paths bounce by bounce, to the last one: 3.3M paths through 1M slots give the film of a wave whose
    paths all start at once."""
    scene, cam, st = importlib.import_module("test_instances").moving_cornell(pe, 64, 64, 8, 6)
    st.motion_blur = True
    st.width, st.height = 1100, 1000
    scene.build_accelerator()
    device.set_scene(scene)
    films = []
    try:
        for slots, tail in ((1 << 23, -1), (1 << 20, -1), (1 << 20, 0)):
            device.set_tuning(wave_slots=slots, tail_paths=tail)
            films.append(pe.Film(1100, 1000))
            device.render(cam, st, pe.RenderTargets(beauty=films[-1]), 0, 3)
            assert _same(films[0], films[-1]), (slots, tail)
    finally:
        device.set_tuning()
