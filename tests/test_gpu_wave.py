"""Bounces over packed queues (device option wave) against the fused bounce and tail kernels.

Both follow the same paths with the same arithmetic, so images and ray counts must be equal bit
for bit: wavefronts long enough for several trace-and-shade passes and ones the tail kernel takes
after the first, one and several light samples per camera ray (the second packed queue then lies
in arrays of its own, and a lane restarts light samples), image sizes that are no multiple of a
tile, a single sphere, and rays that leave the scene at once; spheres, and grids over parts with
every type of primitive, whose own tests wait for one another there.
"""

import numpy
import pytest

pytestmark = pytest.mark.gpu


def _scene(dev, n, box, radius, at, outline=0.0):
    import fresnel_b200 as fresnel
    rng = numpy.random.default_rng(17)
    scene = fresnel.Scene(dev, lights=fresnel.light.cloudy())
    pos = rng.uniform(-box / 2, box / 2, (n, 3)).astype(numpy.float32)
    g = fresnel.geometry.Sphere(scene, position=pos, radius=radius, outline_width=outline)
    g.color[:] = rng.uniform(0.2, 1, (n, 3))
    g.material = fresnel.material.Material(primitive_color_mix=1.0, roughness=0.5, spec_trans=0.1)
    scene.background_color = (0.3, 0.5, 0.7)
    scene.background_alpha = 0.5
    d = float(numpy.linalg.norm(at))
    scene.camera = fresnel.camera.Perspective(position=at, look_at=(0, 0, 0), up=(0, 1, 0),
                                              focal_length=0.25 * d, focus_distance=d,
                                              height=0.25 * 1.2 * box)
    return scene


def _mixed(dev, scale=0.01):
    from fresnel_b200 import workloads
    return workloads.config3(dev, scale=scale)


def _layers(dev):
    from fresnel_b200 import workloads
    return workloads.polygons(dev, nx=20, ny=16, spheres=300)


def _odd_cubes(dev):
    """Cubes whose stated bounding radius is too small, some of them scaled by their quaternions."""
    import fresnel_b200 as fresnel
    from fresnel_b200 import workloads
    rng = numpy.random.default_rng(8)
    scene = fresnel.Scene(dev, lights=fresnel.light.rembrandt())
    info = workloads.unit_cube_planes()
    info["radius"] = 0.6
    pos = rng.uniform(-5, 5, (700, 3)).astype(numpy.float32)
    q = workloads.random_quaternions(rng, 700)
    q[::3] *= 0.8
    fresnel.geometry.ConvexPolyhedron(scene, info, position=pos, orientation=q,
                                      color=(0.7, 0.4, 0.2), outline_width=0.02)
    scene.camera = fresnel.camera.Orthographic.fit(scene)
    return scene


CASES = {  # scene, image size, samples, light samples
    "mixed": (_mixed, (160, 130), 250, 1),
    "mixed_lights": (_mixed, (161, 97), 150, 2),
    "layers": (_layers, (160, 128), 220, 1),
    "odd_cubes": (_odd_cubes, (130, 130), 200, 1),
    "dense": (dict(n=6000, box=20.0, radius=0.6, at=(20.0, 12.0, 26.0)), (161, 129), 250, 1),
    "dense_lights": (dict(n=6000, box=20.0, radius=0.6, at=(20.0, 12.0, 26.0), outline=0.05),
                     (161, 129), 120, 3),
    "inside": (dict(n=3000, box=20.0, radius=0.5, at=(0.4, 0.2, 0.3)), (97, 101), 230, 2),
    "sparse": (dict(n=60, box=20.0, radius=0.4, at=(24.0, 15.0, 30.0)), (130, 128), 150, 1),
    "one": (dict(n=1, box=2.0, radius=0.7, at=(4.0, 3.0, 5.0)), (128, 128), 140, 4),
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_packed_queues_give_the_fused_kernels_images(gpu_device, name):
    import fresnel_b200 as fresnel
    args, size, samples, lights = CASES[name]
    option = gpu_device._device.setOption
    scene = args(gpu_device) if callable(args) else _scene(gpu_device, **args)
    out = []
    try:
        for wave in (0, 1):
            option("wave", wave)
            t = fresnel.tracer.Path(gpu_device, *size)
            t.seed = 23
            t.sample(scene, samples, light_samples=lights)
            t.sample(scene, 3, reset=False, light_samples=lights)  # a short wavefront after it
            out.append((t.linear_output[:], t._tracer.getStats()))
    finally:
        option("wave", 1)
    (a, sa), (b, sb) = out
    assert sa["rays"] == sb["rays"] and sa["paths"] == sb["paths"]
    assert sa["kernel_launches"] != sb["kernel_launches"]  # the two forms did run
    numpy.testing.assert_array_equal(a.view(numpy.uint32), b.view(numpy.uint32))
