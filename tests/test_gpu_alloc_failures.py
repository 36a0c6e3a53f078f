"""Renders during which a device allocation fails, and the renders after them.

Every allocation of a first render is made to fail once, one after another (the library reports
that there is no memory without asking the GPU).  The render then either raises an out-of-memory
error or, where the memory was optional (the bounding spheres and second record queue of the packed
kernels, pixel lists), gives the same image through kernels that do without; the next render must
give the image of an undisturbed one through the same kernels, with nothing left half built.
"""

import numpy
import pytest

import fresnel_b200 as fresnel
from fresnel_b200 import workloads

pytestmark = pytest.mark.gpu


def _fail(after, count=1):
    return fresnel._gpu.debugFailAllocations(after, count)


def _parts(dev):
    return workloads.config3(dev, scale=0.004)


def _spheres(dev):
    return workloads.random_spheres(dev, 3000, 20.0, seed=3)


SIZE = (160, 130)
CASES = {  # scene, samples (2M path slots and more), light samples, device options
    "parts": (_parts, 100, 1, {}),
    "parts_lights": (_parts, 100, 2, {}),
    "spheres_lists": (_spheres, 100, 2, {"pixel_lists": 1}),
    "parts_short": (_parts, 3, 1, {}),
}


def _setup(name):
    make, spp, lights, options = CASES[name]
    dev = fresnel.Device(mode="gpu")
    for key, value in options.items():
        dev._device.setOption(key, value)
    scene = make(dev)
    tracer = fresnel.tracer.Path(dev, *SIZE)

    def render():
        before = tracer._tracer.getStats()["kernel_launches"]
        tracer.seed = 9
        tracer.sample(scene, spp, light_samples=lights)
        return (tracer.linear_output[:].copy(),
                tracer._tracer.getStats()["kernel_launches"] - before)

    return dev, scene, render


@pytest.mark.parametrize("name", sorted(CASES))
def test_render_after_a_failed_allocation(gpu_device, name):
    _, _, render = _setup(name)
    image, launches = render()
    raised = served = 0
    for k in range(200):
        _, _, render = _setup(name)
        _fail(k)
        try:
            first, _ = render()
        except RuntimeError as e:
            assert "memory" in str(e)
            first = None
        failed = _fail(0, 0)
        if first is not None:
            numpy.testing.assert_array_equal(first, image)
        if not failed:
            break
        raised += first is None
        served += first is not None
        again, n = render()
        numpy.testing.assert_array_equal(again, image)
        assert n == launches
    else:
        pytest.fail("the render allocates without end")
    assert raised > 10
    # bounding spheres; they and three record arrays; three record arrays and the lists; none
    assert served == {"parts": 1, "parts_lights": 4, "spheres_lists": 4, "parts_short": 0}[name]
