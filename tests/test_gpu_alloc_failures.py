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


def _batch(dev, batch, scenes, spp, lights):
    tracers = []
    for i, scene in enumerate(scenes):
        t = fresnel.tracer.Path(dev, *SIZE)
        t.seed = 4 + i
        batch.add(t, scene, samples=spp, light_samples=lights)
        tracers.append(t)
    batch.render()
    return [t.linear_output[:].copy() for t in tracers]


@pytest.mark.parametrize("wave", [0, 1])
def test_batch_after_a_failed_allocation(gpu_device, wave):
    """A small batch (captured as a graph), then larger ones whose allocations fail one after
    another, each followed by the small one again: its graph must not run over arrays that moved.
    """
    def setup():
        dev = fresnel.Device(mode="gpu")
        dev._device.setOption("wave", wave)
        dev._device.setOption("pixel_lists", 1)
        scenes = [_parts(dev), _parts(dev), _spheres(dev)]
        for i, s in enumerate(scenes):
            s.background_color = (0.1 * i, 0.2, 0.3)
        return dev, scenes, fresnel.tracer.PathBatch(dev)

    dev, scenes, batch = setup()
    small = _batch(dev, batch, scenes[:1], 2, 1)
    large = _batch(dev, batch, scenes, 100, 2)
    raised = 0
    for k in range(200):
        dev, scenes, batch = setup()
        _batch(dev, batch, scenes[:1], 2, 1)
        _fail(k + 9)  # (after the images and counters of the three tracers)
        try:
            images = _batch(dev, batch, scenes, 100, 2)
        except RuntimeError as e:
            assert "memory" in str(e)
            images = None
            raised += 1
        failed = _fail(0, 0)
        if images is not None:
            for a, b in zip(images, large):
                numpy.testing.assert_array_equal(a, b)
        if not failed:
            break
        for a, b in zip(_batch(dev, batch, scenes[:1], 2, 1), small):
            numpy.testing.assert_array_equal(a, b)
        for a, b in zip(_batch(dev, batch, scenes, 100, 2), large):
            numpy.testing.assert_array_equal(a, b)
    else:
        pytest.fail("the batch allocates without end")
    assert raised > 10


def test_optional_arrays_make_room(gpu_device):
    """Pixel lists and second record queues stay with a device and its batches between renders; an
    allocation that then fails once succeeds without them, whichever it is."""
    def run(k):
        dev = fresnel.Device(mode="gpu")
        dev._device.setOption("pixel_lists", 1)
        scene = _spheres(dev)
        t = fresnel.tracer.Path(dev, *SIZE)
        t.seed = 9
        t.sample(scene, 100, light_samples=2)
        batch = fresnel.tracer.PathBatch(dev)
        _batch(dev, batch, [scene], 100, 2)
        if k is not None:
            _fail(k)
        parts = _parts(dev)  # every array of a scene, a larger image, more path slots, a batch
        large = fresnel.tracer.Path(dev, 210, 170)
        large.seed = 5
        large.sample(parts, 70)
        small = fresnel.tracer.Preview(dev, 64, 48, anti_alias=True)
        small.render(parts)
        images = [large.linear_output[:].copy(), small.linear_output[:].copy()]
        images += _batch(dev, fresnel.tracer.PathBatch(dev), [parts, scene], 70, 1)
        dev._device.setOption("accel", 0)  # trees
        large.seed = 5
        large.sample(parts, 3)
        images.append(large.linear_output[:].copy())
        return images, _fail(0, 0)

    wanted, _ = run(None)
    for k in range(200):
        images, failed = run(k)
        for a, b in zip(images, wanted):
            numpy.testing.assert_array_equal(a, b)
        if not failed:
            break
    assert 40 < k < 199


@pytest.mark.parametrize("failures", [1, 2])
def test_resize_that_finds_no_memory(gpu_device, failures):
    """A tracer whose resize fails keeps an image of its old size; when there is no memory even for
    that, it renders nothing until a resize succeeds."""
    dev = fresnel.Device(mode="gpu")
    scene = _spheres(dev)
    for kind in (fresnel.tracer.Path, fresnel.tracer.Preview):
        t = kind(dev, 64, 48)
        t.seed = 3
        t.render(scene)
        image = t.linear_output[:].copy()
        batch = fresnel.tracer.PathBatch(dev)
        if kind is fresnel.tracer.Path:
            batch.add(t, scene, samples=1)
        _fail(0, failures)
        with pytest.raises(RuntimeError, match="memory"):
            t.resize(640, 480)
        assert _fail(0, 0) == failures
        if failures == 1:
            assert not t.linear_output[:].any() and t.linear_output[:].shape == image.shape
        else:
            with pytest.raises(RuntimeError, match="no memory to resize"):
                t.render(scene)
            if kind is fresnel.tracer.Path:
                with pytest.raises(RuntimeError, match="no memory to resize"):
                    batch.render()
                with pytest.raises(RuntimeError, match="no memory to resize"):
                    batch.add(t, scene, samples=1)
        t.resize(64, 48)
        if kind is fresnel.tracer.Path:
            t.reset()
        t.seed = 3
        t.render(scene)
        numpy.testing.assert_array_equal(t.linear_output[:], image)
