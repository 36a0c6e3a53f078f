"""The sRGB bytes of rendered images against the double-precision curve.

The engine decides most bytes with single-precision powers and the close ones with the power in
double precision, so every byte must be the one the double-precision formula gives for the linear
output: over dark and bright images (values across the linear segment's end, up to and above 1)
and both the Preview and the Path output kernels.
"""

import numpy
import pytest

pytestmark = pytest.mark.gpu


def _bytes(linear):
    x = linear.astype(numpy.float32)
    with numpy.errstate(invalid="ignore"):
        power = numpy.power(x.astype(numpy.float64),
                            numpy.float64(numpy.float32(1.0) / numpy.float32(2.4)))
    f = numpy.float32
    y = numpy.where(x < f(0.0031308), f(12.92) * x,
                    (f(1.0) + f(0.055)) * power.astype(numpy.float32) - f(0.055))
    y = numpy.where(y > f(1.0), f(1.0), y).astype(numpy.float32)
    return (y * f(255.0) + f(0.5)).astype(numpy.uint8)


@pytest.mark.parametrize("bright", [0.01, 0.4, 1.0, 6.0])
@pytest.mark.parametrize("kind", ["preview", "path"])
def test_bytes_are_the_double_curves(gpu_device, kind, bright):
    import fresnel_b200 as fresnel
    rng = numpy.random.default_rng(4)
    light = fresnel.light.Light(direction=(0.3, 0.8, 0.6), color=(bright, 0.7 * bright, 0.9 * bright),
                                theta=0.8)
    scene = fresnel.Scene(gpu_device, lights=[light, fresnel.light.Light(direction=(0, 0, 1),
                                              color=(0.2 * bright,) * 3, theta=numpy.pi)])
    pos = rng.uniform(-8, 8, (1500, 3)).astype(numpy.float32)
    g = fresnel.geometry.Sphere(scene, position=pos, radius=0.6)
    g.color[:] = rng.uniform(0, 1, (1500, 3))
    g.material = fresnel.material.Material(primitive_color_mix=1.0, roughness=0.3)
    scene.background_color = (0.002 * bright, 0.0032 * bright, 0.5 * bright)
    scene.camera = fresnel.camera.Orthographic.fit(scene)
    t = (fresnel.tracer.Preview(gpu_device, 641, 483) if kind == "preview"
         else fresnel.tracer.Path(gpu_device, 641, 483))
    if kind == "preview":
        t.render(scene)
    else:
        t.sample(scene, 24)
    numpy.testing.assert_array_equal(t.output[:][..., :3], _bytes(t.linear_output[:][..., :3]))
