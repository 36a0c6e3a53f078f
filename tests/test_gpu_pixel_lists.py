"""Per-pixel primitive lists (device option pixel_lists) against the walk they stand in for.

A list may only answer a camera ray as the walk of the acceleration structure would, so every
image must be the same bit for bit with the lists and without them, over every kind of structure,
camera and primitive the lists take, and where they must decline: a camera among the primitives, a
bounding radius smaller than the polyhedron, quaternions that are not of unit length.
"""

import math

import numpy
import pytest

pytestmark = pytest.mark.gpu


def _spheres(dev, n=4000, box=22.0, camera="perspective", radii=0.5, f_stop=math.inf, at=None):
    import fresnel_b200 as fresnel
    rng = numpy.random.default_rng(3)
    scene = fresnel.Scene(dev, lights=fresnel.light.cloudy())
    pos = rng.uniform(-box / 2, box / 2, (n, 3)).astype(numpy.float32)
    r = numpy.full(n, radii) if numpy.isscalar(radii) else rng.uniform(*radii, n)
    g = fresnel.geometry.Sphere(scene, position=pos, radius=r.astype(numpy.float32),
                                outline_width=0.05)
    g.color[:] = rng.uniform(0, 1, (n, 3))
    g.material = fresnel.material.Material(primitive_color_mix=1.0, roughness=0.4)
    where = numpy.array((1.1 * box, 0.8 * box, 1.3 * box) if at is None else at, float)
    if camera == "perspective":
        d = float(numpy.linalg.norm(where))
        scene.camera = fresnel.camera.Perspective(position=where, look_at=(0, 0, 0), up=(0, 1, 0),
                                                  focal_length=0.25 * d, focus_distance=d,
                                                  f_stop=f_stop, height=0.3 * box)
    else:
        scene.camera = fresnel.camera.Orthographic(position=where, look_at=(0, 0, 0),
                                                   up=(0, 1, 0), height=1.3 * box)
    return scene


def _cubes(dev, radius=None, scale=1.0):
    """Cubes and bonds; radius: the stated bounding radius, scale: the quaternions' length."""
    import fresnel_b200 as fresnel
    from fresnel_b200 import workloads
    rng = numpy.random.default_rng(8)
    scene = fresnel.Scene(dev, lights=fresnel.light.rembrandt())
    info = workloads.unit_cube_planes()
    if radius is not None:
        info["radius"] = radius
    pos = rng.uniform(-7, 7, (500, 3)).astype(numpy.float32)
    fresnel.geometry.ConvexPolyhedron(scene, info, position=pos, color=(0.7, 0.4, 0.2),
                                      orientation=workloads.random_quaternions(rng, 500) * scale,
                                      outline_width=0.03)
    pts = numpy.stack([pos[:200], pos[200:400]], axis=1) * 0.5
    fresnel.geometry.Cylinder(scene, points=pts, radius=0.1, color=(0.2, 0.3, 0.8))
    scene.camera = fresnel.camera.Orthographic.fit(scene)
    return scene


def _mixed(dev):
    from fresnel_b200 import workloads
    return workloads.config3(dev, scale=0.004)


def _layers(dev):
    from fresnel_b200 import workloads
    return workloads.polygons(dev, nx=12, ny=9, spheres=150)


SCENES = {
    "grid": (_spheres, {}),
    "grid_ortho": (_spheres, dict(camera="orthographic")),
    "grid_lens": (_spheres, dict(f_stop=4.0)),
    "grid_radii": (_spheres, dict(radii=(0.02, 1.5), n=1500)),
    "grid_inside": (_spheres, dict(at=(0.3, 0.2, 0.4))),
    "grid_distant": (_spheres, dict(at=(900.0, 0.0, 10.0))),
    "grid_one": (_spheres, dict(n=1)),
    "tree": (_spheres, dict(accel=0)),
    "tree_lens": (_spheres, dict(accel=0, f_stop=8.0, radii=(0.02, 1.5))),
    "tree_ortho": (_spheres, dict(accel=0, camera="orthographic")),
    "mixed": (_mixed, {}),
    "layers": (_layers, {}),
    "cubes": (_cubes, {}),
    "cubes_small_radius": (_cubes, dict(radius=0.4)),
    "cubes_scaled": (_cubes, dict(scale=1.4)),
}


@pytest.mark.parametrize("name", sorted(SCENES))
@pytest.mark.parametrize("size", [(97, 61), (8, 4), (33, 1)])
def test_lists_give_the_walks_images(gpu_device, name, size):
    import fresnel_b200 as fresnel
    make, args = SCENES[name]
    args = dict(args)
    option = gpu_device._device.setOption
    option("accel", args.pop("accel", 2))
    try:
        scene = make(gpu_device, **args)
        images = []
        for lists in (0, 1):
            option("pixel_lists", lists)
            path = fresnel.tracer.Path(gpu_device, *size)
            path.seed = 11
            path.sample(scene, 40)
            preview = fresnel.tracer.Preview(gpu_device, *size, anti_alias=True)
            preview.seed = 5
            preview.render(scene)
            images.append((path.linear_output[:], preview.linear_output[:], path._tracer.getStats()))
    finally:
        option("pixel_lists", 2)
        option("accel", 2)
    numpy.testing.assert_array_equal(images[0][0].view(numpy.uint32),
                                     images[1][0].view(numpy.uint32))
    numpy.testing.assert_array_equal(images[0][1].view(numpy.uint32),
                                     images[1][1].view(numpy.uint32))
    for key in ("rays", "paths"):
        assert images[0][2][key] == images[1][2][key]
    if name == "grid" and size == (97, 61):  # the lists are in use
        assert images[1][2]["box_tests"] < 0.8 * images[0][2]["box_tests"]


@pytest.mark.parametrize("bonds", [False, True])
@pytest.mark.parametrize("half", [0.5, 2.0, 8.0])
def test_lists_with_primitives_behind_the_camera(gpu_device, bonds, half):
    """A camera among the spheres, from a moderate to a very wide angle: the line of a pixel's axis
    also meets spheres behind the camera, which hide nothing."""
    import fresnel_b200 as fresnel
    rng = numpy.random.default_rng(12)
    option = gpu_device._device.setOption
    scene = fresnel.Scene(gpu_device, lights=fresnel.light.cloudy())
    pos = rng.uniform(-6, 6, (400, 3)).astype(numpy.float32)
    # one right behind the camera, in the cells around it, and none that holds it
    pos = numpy.concatenate([pos[numpy.linalg.norm(pos, axis=1) > 1.2],
                             [[-0.75, 0.02, 0.01]]]).astype(numpy.float32)
    fresnel.geometry.Sphere(scene, position=pos, radius=0.5)
    if bonds:
        fresnel.geometry.Cylinder(scene, points=numpy.stack([pos[:60] * 1.3, pos[60:120]], 1),
                                  radius=0.1)
    scene.camera = fresnel.camera.Perspective(position=(0, 0, 0), look_at=(1, 0, 0), up=(0, 0, 1),
                                              focal_length=1.0, height=2 * half)
    images = []
    try:
        for lists in (0, 1):
            option("pixel_lists", lists)
            t = fresnel.tracer.Preview(gpu_device, 480, 320, anti_alias=True)
            t.render(scene)
            images.append((t.linear_output[:].copy(), t._tracer.getStats()["box_tests"]))
    finally:
        option("pixel_lists", 2)
    numpy.testing.assert_array_equal(images[0][0], images[1][0])
    assert images[1][1] < images[0][1]  # lists were in use


@pytest.mark.parametrize("case", [(12, 2136, 0.2, 30.0), (7, 2046, 0.05, 0.0), (5, 5000, 0.05, 0.0)])
def test_lists_of_grazed_cylinders(gpu_device, case):
    """Long cylinders along an axis, seen obliquely from afar: the distance at which a ray that
    grazes one meets it may lie just before its box, where another primitive is hit."""
    import fresnel_b200 as fresnel
    seed, n, radius, at = case
    option = gpu_device._device.setOption
    box = (n / 0.1) ** (1 / 3)
    for k in range(6):
        rng = numpy.random.default_rng([seed, k])
        pos = rng.uniform(-box / 2, box / 2, (n, 3)) + at
        axis = numpy.array([1.0, 0, 0]) + 1e-3 * rng.normal(size=(n, 3))
        scene = fresnel.Scene(gpu_device, lights=fresnel.light.cloudy())
        fresnel.geometry.Cylinder(scene, points=numpy.stack([pos, pos + 4 * axis], 1).astype(
            numpy.float32), radius=(radius * rng.uniform(0.5, 1.5, n)).astype(numpy.float32))
        scene.camera = fresnel.camera.Orthographic(
            position=numpy.array([at] * 3) + 6 * box / math.sqrt(3), look_at=[at] * 3,
            up=(0.1, 1, 0.05), height=1.2 * box)
        hits = []
        try:
            for lists in (0, 1):
                option("pixel_lists", lists)
                t = fresnel.tracer.Preview(gpu_device, 320, 240, anti_alias=True)
                hits.append(numpy.array(t._tracer.renderHitIds(scene._scene)))
        finally:
            option("pixel_lists", 2)
        assert (hits[0] != hits[1]).any(-1).sum() == 0


def test_lists_of_cylinders_among_polyhedra(gpu_device):
    """Short cylinders among bricks, seen from afar: a ray accepted beside a cylinder can meet its box
    only behind the next brick, so that whether the walk tests the cylinder depends on which of
    the two it comes to first."""
    import fresnel_b200 as fresnel
    from fresnel_b200 import workloads
    option = gpu_device._device.setOption
    found = 0
    for seed in range(3):
        rng = numpy.random.default_rng([78, seed])
        scene = fresnel.Scene(gpu_device, lights=fresnel.light.cloudy())
        n, box = 4800, 30.0
        info = workloads.unit_cube_planes()
        info["face_origin"] = (info["face_origin"] * (0.2, 1, 1)).astype(numpy.float32)
        info["radius"] = 0.71415
        pos = rng.uniform(-box / 2, box / 2, (n, 3))
        d = rng.normal(size=(n, 3))
        d /= numpy.linalg.norm(d, axis=1, keepdims=True)
        fresnel.geometry.Cylinder(scene, points=numpy.stack([pos, pos + d], 1).astype(numpy.float32),
                                  radius=0.1)
        fresnel.geometry.ConvexPolyhedron(
            scene, info, position=rng.uniform(-box / 2, box / 2, (n, 3)).astype(numpy.float32),
            orientation=workloads.random_quaternions(rng, n))
        scene.camera = fresnel.camera.Perspective(position=(0, 0, 6 * box), look_at=(0, 0, 0),
                                                  up=(0.1, 1, 0.07), focal_length=1.0,
                                                  height=1 / 6)
        hits = []
        try:
            for lists in (0, 1):
                option("pixel_lists", lists)
                t = fresnel.tracer.Preview(gpu_device, 640, 361, anti_alias=True)
                t.seed = seed
                hits.append(numpy.array(t._tracer.renderHitIds(scene._scene)))
        finally:
            option("pixel_lists", 2)
        found += (hits[0] != hits[1]).any(-1).sum()
    assert found == 0
