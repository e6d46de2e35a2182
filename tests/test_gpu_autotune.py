"""What the autotuner chooses from: whatever is in force when it starts, both closest-hit kernels are
probed, and the faster one is kept."""
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
