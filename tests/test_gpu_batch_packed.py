"""Batches whose renders go over packed queues side by side against the batch's graph.

Both follow the same paths with the same arithmetic, so images and ray counts must be equal bit
for bit: more renders than run at once, renders of several sizes, one and several light samples,
a tracer that takes part twice and a wavefront too small for all (the renders then come in several
waves, each with a share of the samples), camera rays answered by pixel lists, and grids over
parts.
"""

import numpy
import pytest

pytestmark = pytest.mark.gpu


def _scenes(dev):
    import fresnel_b200 as fresnel
    from fresnel_b200 import workloads
    scenes = []
    for seed, n in ((1, 4000), (2, 900)):
        rng = numpy.random.default_rng(seed)
        scene = fresnel.Scene(dev, lights=fresnel.light.cloudy())
        g = fresnel.geometry.Sphere(scene, position=rng.uniform(-9, 9, (n, 3)).astype(numpy.float32),
                                    radius=0.6, outline_width=0.02 * seed)
        g.color[:] = rng.uniform(0.2, 1, (n, 3))
        g.material = fresnel.material.Material(primitive_color_mix=1.0, roughness=0.5,
                                               spec_trans=0.1)
        scene.camera = fresnel.camera.Orthographic.fit(scene)
        scenes.append(scene)
    scenes.append(workloads.config3(dev, scale=0.01))
    return scenes


CASES = {  # (scene, w, h, samples, light samples) per render, option path_slots, pixel_lists
    "many": ([(0, 131, 97, 45, 1), (1, 300, 200, 9, 1)] * 17 + [(0, 257, 129, 20, 1)], None, 2),
    "lights": ([(0, 256, 200, 45, 2), (1, 301, 190, 40, 3)], None, 2),
    "parts": ([(2, 256, 256, 12, 1), (0, 256, 200, 16, 1), (2, 190, 130, 40, 1)], None, 2),
    "lists": ([(0, 256, 200, 18, 1), (2, 256, 256, 17, 1), (1, 300, 200, 16, 1)], None, 1),
    "waves": ([(0, 256, 256, 40, 1), (1, 256, 256, 24, 1), (0, 300, 200, 50, 1)], 1 << 21, 1),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_packed_batch_gives_the_graphs_images(gpu_device, name):
    import fresnel_b200 as fresnel
    renders, slots, lists = CASES[name]
    option = gpu_device._device.setOption
    before = gpu_device._device.getOption("path_slots")
    scenes = _scenes(gpu_device)
    got = []
    try:
        if slots:
            option("path_slots", slots)
        option("pixel_lists", lists)
        for wave in (1, 0):
            option("wave", wave)
            batch = fresnel.tracer.PathBatch(gpu_device)
            tracers = []
            for i, (k, w, h, spp, ls) in enumerate(renders):
                t = fresnel.tracer.Path(gpu_device, w, h)
                t.seed = 3 + i
                batch.add(t, scenes[k], samples=spp, light_samples=ls)
                tracers.append(t)
            if name == "waves":
                batch.add(tracers[1], scenes[0], samples=30, reset=False)
            batch.render()
            assert (batch.stats["graph_launches"] == 0) == bool(wave)
            assert (batch.stats["waves"] > 1) == (name == "waves")
            got.append([(t.linear_output[:].copy(), t.output[:].copy(),
                         t._tracer.getStats()["rays"]) for t in tracers])
        for (image, srgb, rays), (image0, srgb0, rays0) in zip(*got):
            numpy.testing.assert_array_equal(image, image0)
            numpy.testing.assert_array_equal(srgb, srgb0)
            assert rays == rays0
    finally:
        option("wave", 1)
        option("pixel_lists", 2)
        option("path_slots", before)


@pytest.mark.parametrize("lights,height,packed", [(1, 40.0, True), (2, 40.0, True),
                                                  (1, 4000.0, True), (2, 4000.0, False)])
def test_batches_that_miss_take_the_graph(gpu_device, lights, height, packed):
    """With several light samples a packed render's passes are worth their launches only where
    enough camera rays hit: the same batch with the scene filling the image, and as a few pixels
    in its middle."""
    import fresnel_b200 as fresnel
    scene = _scenes(gpu_device)[0]
    scene.camera = fresnel.camera.Orthographic(position=(60, 50, 70), look_at=(0, 0, 0),
                                               up=(0, 1, 0), height=height)
    option = gpu_device._device.setOption
    got = []
    try:
        for wave in (1, 0):
            option("wave", wave)
            batch = fresnel.tracer.PathBatch(gpu_device)
            t = fresnel.tracer.Path(gpu_device, 256, 256)
            t.seed = 8
            batch.add(t, scene, samples=36, light_samples=lights)
            batch.render()
            assert (batch.stats["graph_launches"] == 0) == (packed and wave == 1)
            got.append(t.linear_output[:].copy())
    finally:
        option("wave", 1)
    numpy.testing.assert_array_equal(got[0], got[1])


def test_packed_batch_lists_take_a_lane_each(gpu_device):
    """The pixel lists of a batch's renders take memory for those that run at once (32 streams), not
    for all of its renders."""
    import gc
    import torch
    import fresnel_b200 as fresnel
    gc.collect()  # (what earlier tests left would be freed between the two readings)
    dev = fresnel.Device(mode="gpu")
    scene = _scenes(dev)[0]
    batch = fresnel.tracer.PathBatch(dev)
    tracers = [fresnel.tracer.Path(dev, 192, 192) for _ in range(96)]
    images, free = [], []
    for lists in (0, 1):
        dev._device.setOption("pixel_lists", lists)
        for i, t in enumerate(tracers):
            t.seed = i
            batch.add(t, scene, samples=15)
        batch.render()
        assert batch.stats["graph_launches"] == 0 and batch.stats["waves"] == lists + 1
        images.append([t.linear_output[:].copy() for t in tracers])
        free.append(torch.cuda.mem_get_info()[0])
    for a, b in zip(*images):
        numpy.testing.assert_array_equal(a, b)
    # 32 lists of 128 bytes per pixel, and as much again for what else the second render may take
    assert 0 < free[0] - free[1] < 2 * 32 * 128 * 192 * 192
