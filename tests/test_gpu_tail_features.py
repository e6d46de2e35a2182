"""Scenes whose waves take the full-feature shading kernels, shadow rays of their own or inline ones: the film does
not depend on where a wave hands over to its tail kernel.  The tail runs the wavefront's shading code on
the same rays in the same order of terms, so films are equal bit for bit: no tolerance."""
import importlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _scenes():
    return importlib.import_module("photon_engine_b200.scenes")


def _transmitters(pe):
    return importlib.import_module("test_gpu_transmit")._scene(pe)


def _links(pe):
    return importlib.import_module("test_gpu_light_links")._scene(pe, True)


def _catcher(pe):
    return importlib.import_module("test_gpu_aovs")._open_scene(pe, "catcher")


def _moving(pe):
    scene, cam, st = importlib.import_module("test_instances").moving_cornell(pe, 64, 64, 8, 6)
    st.motion_blur = True
    return scene, cam, st


def _rounded(pe):
    S = _scenes()
    scene, cam, st = S.cornell_box(64, 64, 8, 8, seed=0)
    m = pe.Lambertian((0.6, 0.6, 0.7))
    m.set_round_edge_radius(0.25)
    p, n, i = S.grid_box((2.2, 0.8, 2.0), (1.6, 1.6, 1.6), 2)
    scene.add_shape(pe.TriangleMesh(p, n, None, i, m))
    st.ao_strength = 0.7
    return scene, cam, st


def _mipmapped(pe):
    S = _scenes()
    scene, cam, st = S.cornell_box(64, 64, 8, 8, seed=0)
    m = pe.DisneyMaterial((0.8, 0.8, 0.8), 0.0, 0.4)
    image = np.random.default_rng(5).uniform(0.05, 0.95, (32, 32, 3)).astype(np.float32)
    m.set_albedo_image(image, mipmaps=True)
    pos, nrm, idx = S.uv_sphere((2.78, 1.2, 2.2), 0.9, 32, 16)
    scene.add_shape(pe.TriangleMesh(pos, nrm, None, idx, m))
    return scene, cam, st


@pytest.mark.parametrize("make", [_transmitters, _links, _catcher, _moving, _rounded, _mipmapped],
                         ids=["transmitters", "links", "catcher", "moving", "rounded", "mipmapped"])
def test_film_does_not_depend_on_the_tail(pe, device, make):
    scene, cam, st = make(pe)
    st.width, st.height = 65, 47
    scene.build_accelerator()
    device.set_scene(scene)
    try:
        for quality in (1, 3):
            st.shadow_quality = quality
            films = []
            for tail in (0, 100, 1000, -1, 1 << 40):
                device.set_tail_paths(tail)
                films.append(pe.Film(st.width, st.height))
                device.render(cam, st, pe.RenderTargets(beauty=films[-1]), 0, 3)
                for name in ("sum", "sum_sq", "count"):
                    assert np.array_equal(getattr(films[0], name).view(np.uint32), getattr(films[-1], name).view(np.uint32)), \
                        (quality, tail, name)
    finally:
        device.set_tail_paths(-1)
