"""Where frames take per-pixel primitive lists by themselves (device option pixel_lists 2).

Camera rays answered by a list do not walk the grid, so a frame with lists counts fewer box tests
(cells) than one without, and a frame that declines them counts the same number.  The image is the
same either way.
"""

import numpy
import pytest

import fresnel_b200 as fresnel
from fresnel_b200 import workloads

pytestmark = pytest.mark.gpu


def _cubes(dev, n=500, odd=0.0, radius=None, faces=6):
    """n cubes at 0.3 per unit volume; `odd`: the share whose quaternions have norm 0.95."""
    rng = numpy.random.default_rng(2)
    box = (n / 0.3) ** (1 / 3)
    scene = fresnel.Scene(dev, lights=fresnel.light.rembrandt())
    info = workloads.unit_cube_planes()
    if faces > 6:  # a ball of planes tangent to a sphere of radius 0.5
        i = numpy.arange(faces) + 0.5
        z, a = 1 - 2 * i / faces, numpy.pi * (1 + 5**0.5) * i
        n_ = numpy.stack([numpy.sqrt(1 - z * z) * numpy.cos(a),
                          numpy.sqrt(1 - z * z) * numpy.sin(a), z], 1).astype(numpy.float32)
        info = dict(face_origin=0.5 * n_, face_normal=n_,
                    face_color=numpy.full((faces, 3), 0.9, numpy.float32), radius=0.6)
    if radius is not None:
        info["radius"] = radius
    q = workloads.random_quaternions(rng, n)
    q[:int(odd * n)] *= 0.95
    fresnel.geometry.ConvexPolyhedron(
        scene, info, position=rng.uniform(-box / 2, box / 2, (n, 3)).astype(numpy.float32),
        orientation=q, color=(0.8, 0.3, 0.2))
    scene.camera = fresnel.camera.Orthographic(position=(40, 40, 40), look_at=(0, 0, 0),
                                               up=(0, 1, 0), height=1.8 * box)
    return scene


CASES = {  # scene, image, lists are used
    "cubes": (dict(), (480, 360), True),
    "few_odd": (dict(odd=0.05), (480, 360), True),
    "odd": (dict(odd=0.4), (480, 360), False),
    "small_radius": (dict(radius=0.8), (480, 360), False),
    "faces_48": (dict(faces=48), (480, 360), True),
    "faces_49": (dict(faces=49), (480, 360), False),  # (its bounds are not checked)
}


@pytest.mark.parametrize("name", sorted(CASES))
def test_frames_with_lists(gpu_device, name):
    args, size, used = CASES[name]
    scene = _cubes(gpu_device, **args)
    option = gpu_device._device.setOption
    got = []
    try:
        for lists in (0, 2):
            option("pixel_lists", lists)
            t = fresnel.tracer.Preview(gpu_device, *size, anti_alias=True)
            t.render(scene)
            got.append((t.linear_output[:].copy(), t._tracer.getStats()["box_tests"]))
    finally:
        option("pixel_lists", 2)
    numpy.testing.assert_array_equal(got[0][0], got[1][0])
    assert (got[1][1] < 0.8 * got[0][1]) if used else (got[1][1] == got[0][1])


def _spheres_and_bonds(dev, m=14):
    rng = numpy.random.default_rng(4)
    ijk = numpy.stack(numpy.meshgrid(*[numpy.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pos = ((ijk - (m - 1) / 2) * 2.0 + rng.uniform(-0.3, 0.3, (m**3, 3))).astype(numpy.float32)
    scene = fresnel.Scene(dev, lights=fresnel.light.rembrandt())
    fresnel.geometry.Sphere(scene, position=pos, radius=0.4, color=(0.4, 0.5, 0.6))
    i = numpy.flatnonzero(ijk[:, 2] < m - 1)
    fresnel.geometry.Cylinder(scene, points=numpy.stack([pos[i], pos[i + 1]], 1), radius=0.1,
                              color=(0.3, 0.3, 0.8))
    scene.camera = fresnel.camera.Orthographic(position=(4 * m, 4 * m, 4 * m), look_at=(0, 0, 0),
                                               up=(0, 1, 0), height=3.6 * m)
    return scene


@pytest.mark.parametrize("kind,size,used", [
    ("cubes", (1000, 700), True), ("cubes", (260, 200), False), ("cubes_dense", (260, 200), False),
    ("bonds", (640, 480), True), ("bonds", (260, 200), False)])
def test_beams_that_suit_the_primitives(gpu_device, kind, size, used):
    """Lists over parts ask for thinner beams (more pixels) than lists over spheres, the thinner the
    fewer rays there are."""
    scene = (_spheres_and_bonds(gpu_device) if kind == "bonds" else
             _cubes(gpu_device, n=500 if kind == "cubes" else 20000))
    option = gpu_device._device.setOption
    got = []
    try:
        for lists in (0, 2):
            option("pixel_lists", lists)
            t = fresnel.tracer.Preview(gpu_device, *size, anti_alias=True)
            t.render(scene)
            got.append((t.linear_output[:].copy(), t._tracer.getStats()["box_tests"]))
    finally:
        option("pixel_lists", 2)
    numpy.testing.assert_array_equal(got[0][0], got[1][0])
    assert (got[1][1] < 0.8 * got[0][1]) if used else (got[1][1] == got[0][1])


def test_trees_take_no_lists(gpu_device):
    """Lists are of grid references: over trees the option changes nothing."""
    scene = _cubes(gpu_device)
    option = gpu_device._device.setOption
    option("accel", 0)
    counts = []
    try:
        for lists in (0, 1):
            option("pixel_lists", lists)
            t = fresnel.tracer.Preview(gpu_device, 160, 120, anti_alias=True)
            t.render(scene)
            counts.append(t._tracer.getStats()["box_tests"])
    finally:
        option("pixel_lists", 2)
        option("accel", 2)
    assert counts[0] == counts[1] > 0


def test_path_images_over_parts_take_lists(gpu_device):
    scene = _spheres_and_bonds(gpu_device)  # (beams of 0.13 mean radii, 21M rays: 0.2 allowed)
    option = gpu_device._device.setOption
    counts = []
    try:
        for lists in (0, 2):
            option("pixel_lists", lists)
            t = fresnel.tracer.Path(gpu_device, 1000, 700)
            t.seed = 3
            t.sample(scene, 30)
            counts.append((t._tracer.getStats()["box_tests"], t.linear_output[:].copy()))
    finally:
        option("pixel_lists", 2)
    assert counts[1][0] < counts[0][0]
    numpy.testing.assert_array_equal(counts[0][1], counts[1][1])


def test_tiles_that_reach_the_budget(gpu_device):
    """A very wide tile over many small spheres ends after a few thousand references; its lists then
    answer up to there only."""
    rng = numpy.random.default_rng(6)
    scene = fresnel.Scene(gpu_device, lights=fresnel.light.cloudy())
    fresnel.geometry.Sphere(scene, position=rng.uniform(-20, 20, (60000, 3)).astype(numpy.float32),
                            radius=0.15)
    scene.camera = fresnel.camera.Orthographic(position=(50, 60, 70), look_at=(0, 0, 0),
                                               up=(0, 1, 0), height=70.0)
    option = gpu_device._device.setOption
    images = []
    try:
        for lists in (0, 1):
            option("pixel_lists", lists)
            t = fresnel.tracer.Preview(gpu_device, 40, 24, anti_alias=True)
            t.render(scene)
            images.append(t.linear_output[:].copy())
    finally:
        option("pixel_lists", 2)
    numpy.testing.assert_array_equal(images[0], images[1])
