"""Tree-traced sphere scenes whose remaining bounces run in the tail kernel against pass-by-pass ones.

The tail follows the same paths with the same arithmetic, so images and ray counts must be equal
for every number of passes before it (option tail), for wavefronts of one path up to several
hundred thousand, an empty queue (every ray misses) and both leaf layouts (one sphere, many).
"""

import numpy
import pytest

pytestmark = pytest.mark.gpu

CASES = {  # spheres, image, samples, camera distance
    "one": (1, (33, 17), 5, 6.0),
    "pixel": (40, (1, 1), 1, 20.0),
    "cluster": (5000, (161, 99), 24, 30.0),
    "inside": (3000, (128, 64), 40, 0.5),
    "miss": (30, (64, 48), 3, None),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_tail_gives_the_passes_images(gpu_device, name):
    import fresnel_b200 as fresnel
    n, size, samples, at = CASES[name]
    option = gpu_device._device.setOption
    rng = numpy.random.default_rng(21)
    option("accel", 0)
    try:
        scene = fresnel.Scene(gpu_device, lights=fresnel.light.cloudy())
        pos = (rng.normal(0, 3, (n, 3)) if n > 1 else numpy.zeros((1, 3))).astype(numpy.float32)
        g = fresnel.geometry.Sphere(scene, position=pos, radius=0.5, outline_width=0.03)
        g.color[:] = rng.uniform(0.2, 1, (n, 3))
        g.material = fresnel.material.Material(primitive_color_mix=1.0, roughness=0.4,
                                               spec_trans=0.2)
        look, p = ((0, 0, 0), (0, 0, at)) if at else ((0, 0, 100), (0, 0, 50))
        scene.camera = fresnel.camera.Perspective(position=p, look_at=look, up=(0, 1, 0),
                                                  focal_length=0.5, height=0.5)
        got = []
        for tail in (-1, 0, 1, 3):
            option("tail", tail)
            t = fresnel.tracer.Path(gpu_device, *size)
            t.seed = 5
            t.sample(scene, samples)
            got.append((t.linear_output[:].copy(), t.output[:].copy(),
                        t._tracer.getStats()["rays"]))
        for image, srgb, rays in got[1:]:
            numpy.testing.assert_array_equal(image, got[0][0])
            numpy.testing.assert_array_equal(srgb, got[0][1])
            assert rays == got[0][2]
    finally:
        option("tail", 1)
        option("accel", 2)


def test_tail_kernel_runs(gpu_device):
    """The cases above compare two routes only if the tail takes the place of later passes."""
    import fresnel_b200 as fresnel
    n, size, samples, at = CASES["cluster"]
    option = gpu_device._device.setOption
    rng = numpy.random.default_rng(21)
    option("accel", 0)
    launches = {}
    try:
        scene = fresnel.Scene(gpu_device, lights=fresnel.light.cloudy())
        fresnel.geometry.Sphere(scene, position=rng.normal(0, 3, (n, 3)).astype(numpy.float32),
                                radius=0.5)
        scene.camera = fresnel.camera.Perspective(position=(0, 0, at), look_at=(0, 0, 0),
                                                  up=(0, 1, 0), focal_length=0.5, height=0.5)
        for tail in (-1, 0, 1, 3):
            option("tail", tail)
            t = fresnel.tracer.Path(gpu_device, *size)
            t.sample(scene, samples)
            launches[tail] = t._tracer.getStats()["kernel_launches"]
    finally:
        option("tail", 1)
        option("accel", 2)
    # camera pass, tail, fold, and two launches for each pass before the tail
    assert launches[0] == 3 and launches[1] == 5 and launches[3] == 9
    assert launches[-1] > launches[3]
