"""What the autotuner chooses from: whatever is in force when it starts, both closest-hit kernels and the
thresholds around the default of the scene that it renders."""
import importlib

import pytest

pytestmark = pytest.mark.gpu


def _probes(device, knob):
    times = {}
    for line in device.autotune_log().splitlines():
        name, ms = line.split()[:2]
        if name.startswith(knob + "="):
            times[int(name.split("=")[1])] = float(ms)
    return times


@pytest.mark.parametrize("in_force,wide", [(0, 6), (6, 6), (3, 3)])
def test_both_closest_hit_kernels_are_probed(pe, device, in_force, wide):
    scene, cam, st = importlib.import_module("photon_engine_b200.scenes").cornell_box(64, 64, 1, 4)
    scene.build_accelerator()
    device.set_scene(scene)
    try:
        device.set_tuning(closest_traversal=in_force)
        device.autotune(cam, st, 1)
        times = _probes(device, "closest_traversal")
        assert set(times) == {0, wide}
        assert device.tuning()["closest_traversal"] == min(times, key=times.get)
    finally:
        device.set_tuning()


def test_default_tail_threshold_is_the_scenes(pe, device):
    """448 live paths per SM in scenes of plain surfaces, 224 in others and in waves whose settings need
    more than plain shading; the autotuner probes 1/4, 1/2, 1 and 2 times the default of what it renders."""
    import torch

    S = importlib.import_module("photon_engine_b200.scenes")
    sm = torch.cuda.get_device_properties(0).multi_processor_count
    media = S.media_scene(64, 64, 1, 4, n_leds=100, sphere_res=(24, 12), cyl_res=(24, 4), slab_res=3)
    try:
        for (scene, cam, st), ao, per_sm, default in ((S.cornell_box(64, 64, 1, 4), 0.0, 448, 448), (media, 0.0, 224, 224),
                                                      (S.cornell_box(64, 64, 1, 4), 0.5, 224, 448)):
            scene.build_accelerator()
            device.set_tuning()
            device.set_scene(scene)
            assert device.tail_paths == default * sm
            st.ao_strength = ao
            device.autotune(cam, st, 1)
            line = per_sm * sm
            assert set(_probes(device, "tail_paths")) == {line // 4, line // 2, line, 2 * line}
            device.set_tail_paths(1234)
            assert device.tail_paths == 1234
    finally:
        device.set_tuning()
