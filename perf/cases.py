"""Rendering workloads to time: what programs that use fresnel_b200 have it do.

Every case is one call (or the few calls) a program makes per image through the public API, on a
scene it has built, ending with the image as a numpy array on the host:

* ``preview``  `tracer.Preview.render`: the quick look at a scene, with or without 8 x 8
  anti-aliasing;
* ``path``     `tracer.Path.sample`: an image of ``spp`` samples per pixel, each with
  ``light_samples`` light paths;
* ``frames``   a trajectory: the particles of the next frame are written into the scene (whose
  acceleration structure is then rebuilt) before `tracer.Path.sample`;
* ``batch``    `tracer.PathBatch`: images of several scenes traced together.

`listed` names twelve of them, from a thumbnail to the benchmark frame; `draw` gives
others of the same ranges; `prepare` builds the scene, `run` is one pass, `work` the bytes and
operations a pass cannot do without, and `exact` renders sphere scenes in 64 bits with plain
torch where brute force can.
"""

import math
import random

import numpy as np
import torch

RHO = 1e6 / 140.0**3  # spheres per unit volume of the 1M-sphere benchmark scene


def listed():
    return [
        # the six spheres with outlines of fresnel's own test fixture as a thumbnail: launches and
        # host calls
        dict(name="preview_thumbnail", kind="preview", scene="hexagon", n=6, w=101, h=75, aa=0,
             read="linear"),
        # the look at a large particle configuration before its path-traced image: 1M spheres,
        # full HD, 8 x 8 anti-aliasing
        dict(name="preview_1m", kind="preview", scene="spheres", n=1_000_000, w=1920, h=1080,
             aa=1, read="srgb"),
        # a crystal of outlined cubes (hard-particle simulations), orthographic, in a window of odd
        # size
        dict(name="preview_cubes", kind="preview", scene="cubes", n=8000, w=903, h=677, aa=1,
             camera="orthographic", outline=0.04, read="srgb"),
        # an interactive view: one sample per pixel after each camera move
        dict(name="path_interactive", kind="path", scene="spheres", n=50_000, w=1280, h=720,
             spp=1, light_samples=1, read="linear"),
        # fresnel's default `pathtrace` (600 x 370, 64 samples) of a ball-and-stick molecule,
        # outlined, with depth of field
        dict(name="path_molecule", kind="path", scene="sticks", n=3000, w=600, h=370, spp=64,
             light_samples=1, outline=0.05, f_stop=4.0, read="srgb"),
        # 1000 spheres with many light samples per camera ray (a figure for a paper)
        dict(name="path_1k_lights", kind="path", scene="spheres", n=1000, rho=0.125, w=580,
             h=580, spp=64, light_samples=32, outline=0.1, lights="cloudy", read="srgb"),
        # the headline benchmark frame: 1M spheres, full HD, 256 samples
        dict(name="path_1m", kind="path", scene="spheres", n=1_000_000, w=1920, h=1080, spp=256,
             light_samples=1, read="srgb"),
        # spheres, bonds, cubes and icosahedra together (the mixed benchmark scene)
        dict(name="path_mixed", kind="path", scene="mixed", n=280_000, w=1280, h=720, spp=128,
             light_samples=1, lights="rembrandt", read="srgb"),
        # droplets in a vapour (nucleation): clustered particles, an odd image size
        dict(name="path_droplets", kind="path", scene="droplets", n=100_000, w=641, h=479, spp=64,
             light_samples=1, read="linear"),
        # a two-dimensional packing of rounded polygons seen from above
        dict(name="path_polygons", kind="path", scene="polygons", n=10_000, w=800, h=800, spp=32,
             light_samples=1, camera="orthographic", outline=0.05, lights="rembrandt",
             read="srgb"),
        # the next frame of a trajectory: new positions, a movie-quality image
        dict(name="frames_200k", kind="frames", scene="spheres", n=200_000, w=1024, h=768,
             spp=16, light_samples=1, read="srgb"),
        # images of several small configurations at once
        dict(name="batch_small", kind="batch", scene="spheres", n=20_000, frames=8, w=384, h=384,
             spp=16, light_samples=1, read="srgb"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: a kind, a scene and sizes of the ranges the listed cases stand for."""
    c = dict(kind=rng.choice(["preview", "preview", "path", "path", "path", "frames", "batch"]))
    c["scene"] = rng.choice(["spheres", "spheres", "spheres", "cubes", "sticks", "mixed",
                             "droplets", "polygons"])
    if c["kind"] in ("frames", "batch"):
        c["scene"] = "spheres"
    most = dict(spheres=1_000_000, cubes=20_000, sticks=100_000, mixed=280_000, droplets=200_000,
                polygons=20_000)[c["scene"]]
    c["n"] = _log(rng, 500, most)
    c["w"], c["h"] = _log(rng, 96, 1920), _log(rng, 72, 1080)
    c["lights"] = rng.choice(["lightbox", "cloudy", "rembrandt"])
    c["read"] = rng.choice(["srgb", "linear"])
    if rng.random() < 0.3 or c["scene"] == "polygons":
        c["camera"] = "orthographic"
    if rng.random() < 0.3:
        c["outline"] = round(rng.uniform(0.02, 0.1), 3)
    if c["scene"] == "spheres":
        c["rho"] = round(RHO * math.exp(rng.uniform(-1.5, 0.5)), 4)
    if c["kind"] == "preview":
        c["aa"] = rng.choice([0, 1])
        return c
    c["light_samples"] = rng.choice([1, 1, 1, 4, 13])
    c["spp"] = _log(rng, 1, 256)
    if rng.random() < 0.2 and "camera" not in c:
        c["f_stop"] = round(rng.uniform(2.0, 16.0), 2)
    if c["kind"] == "batch":
        c["n"] = min(c["n"], 200_000)
        c["frames"] = rng.randint(2, 12)
        c["w"], c["h"] = min(c["w"], 768), min(c["h"], 768)
    # no more paths than a drawn case may cost
    most_paths = 2e8 if c["scene"] == "spheres" else 5e7
    per_spp = c["w"] * c["h"] * c["light_samples"] * c.get("frames", 1)
    c["spp"] = max(1, min(c["spp"], int(most_paths / per_spp)))
    return c


# ---------------------------------------------------------------------------------------------
# scenes: plain numpy arrays made from the seed
# ---------------------------------------------------------------------------------------------
def _unit(v):
    v = np.asarray(v, np.float64)
    return v / np.linalg.norm(v)


def _quaternions(rng, n):
    q = rng.normal(size=(n, 4))
    return (q / np.linalg.norm(q, axis=1, keepdims=True)).astype(np.float32)


def _arrays(case, seed):
    """The particles of a case's scene (float32 arrays) and the half width of its box."""
    rng = np.random.default_rng([int(seed), 11])
    n, kind = case["n"], case["scene"]
    if kind == "hexagon":
        a = np.arange(6) * (2 * math.pi / 6) + rng.uniform(-0.1, 0.1)
        pos = np.stack([2 * np.cos(a), 2 * np.sin(a), 0 * a], axis=1).astype(np.float32)
        return dict(pos=pos, radius=np.ones(6, np.float32),
                    color=np.full((6, 3), 0.5, np.float32), half=(3.0, 3.0, 1.0))
    if kind in ("spheres", "mixed", "sticks"):
        if kind == "spheres":
            n_s, rho = n, case.get("rho", RHO)
        elif kind == "mixed":  # 200k spheres, 50k bonds, 20k cubes, 10k icosahedra per 280k
            n_s, rho = max(1, n * 5 // 7), 0.2
        else:
            n_s, rho = max(2, n // 2), 0.125
        box = (n_s / rho) ** (1 / 3)
        if kind == "sticks":  # atoms on a jittered lattice, a bond to the next one along x
            m = math.ceil(n_s ** (1 / 3))
            ijk = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)
            pos = ((ijk[:n_s] - (m - 1) / 2) * (box / m) + rng.uniform(-0.3, 0.3, (n_s, 3)))
            pos = pos.astype(np.float32)
            radius = rng.choice([0.3, 0.4, 0.5], n_s).astype(np.float32)
        else:
            pos = rng.uniform(-box / 2, box / 2, (n_s, 3)).astype(np.float32)
            radius = np.full(n_s, 0.5, np.float32)
        out = dict(pos=pos, radius=radius, half=(box / 2,) * 3,
                   color=rng.uniform(0, 1, (n_s, 3)).astype(np.float32))
        if kind == "sticks":
            i = np.flatnonzero(ijk[:n_s, 2] < m - 1)
            i = i[i + 1 < n_s]
            out["bonds"] = np.stack([pos[i], pos[i + 1]], axis=1)
        if kind == "mixed":
            from fresnel_b200.workloads import near_bonds
            out["radius"] = np.exp(rng.uniform(math.log(0.3), math.log(0.7), n_s)).astype(
                np.float32)
            pairs = near_bonds(rng, pos, n_s // 4)
            out["bonds"] = np.stack([pos[pairs[:, 0]], pos[pairs[:, 1]]], axis=1)
            n_c, n_m = max(1, n_s // 10), max(1, n_s // 20)
            out["cubes"] = rng.uniform(-box / 2, box / 2, (n_c, 3)).astype(np.float32)
            out["cubes_q"] = _quaternions(rng, n_c)
            out["meshes"] = rng.uniform(-box / 2, box / 2, (n_m, 3)).astype(np.float32)
            out["meshes_q"] = _quaternions(rng, n_m)
        return out
    if kind == "droplets":  # nine of ten particles in dense droplets, the others as vapour
        box = (n * 0.5236 / 0.004) ** (1 / 3)
        k = max(2, min(24, n // 2000))
        centres = rng.uniform(-0.4 * box, 0.4 * box, (k, 3))
        share = rng.multinomial(n * 9 // 10, rng.dirichlet(np.full(k, 3.0)))
        parts = []
        for c, m in zip(centres, share):
            r = (m / 0.85 * 3 / (4 * math.pi)) ** (1 / 3)
            d = rng.normal(size=(m, 3))
            d /= np.linalg.norm(d, axis=1, keepdims=True)
            parts.append(c + d * (r * rng.uniform(0, 1, (m, 1)) ** (1 / 3)))
        parts.append(rng.uniform(-box / 2, box / 2, (n - n * 9 // 10, 3)))
        pos = np.concatenate(parts).astype(np.float32)
        return dict(pos=pos, radius=np.full(n, 0.5, np.float32), half=(box / 2,) * 3,
                    color=rng.uniform(0, 1, (n, 3)).astype(np.float32))
    if kind == "cubes":
        m = math.ceil(n ** (1 / 3))
        ijk = np.stack(np.meshgrid(*[np.arange(m)] * 3, indexing="ij"), -1).reshape(-1, 3)[:n]
        pos = (ijk - (m - 1) / 2) * 1.6 + rng.uniform(-0.1, 0.1, (n, 3))
        return dict(cubes=pos.astype(np.float32), cubes_q=_quaternions(rng, n),
                    half=(0.8 * m,) * 3)
    if kind == "polygons":
        m = math.ceil(math.sqrt(n))
        ij = np.stack(np.meshgrid(np.arange(m), np.arange(m), indexing="ij"), -1).reshape(-1, 2)
        pos = (ij[:n] - (m - 1) / 2) * 1.6 + rng.uniform(-0.15, 0.15, (n, 2))
        return dict(polygons=pos.astype(np.float32),
                    angle=rng.uniform(-math.pi, math.pi, n).astype(np.float32),
                    color=rng.uniform(0, 1, (n, 3)).astype(np.float32),
                    half=(0.8 * m, 0.8 * m, 0.1))
    raise ValueError(kind)


_LIGHTS = {  # direction in camera space, colour, half angle
    "lightbox": [((0, 0, 1), (0.9, 0.9, 0.9), math.pi)],
    "cloudy": [((0, 1, 0), (0.9, 0.9, 0.9), math.pi / 2), ((0, -1, 0), (0.1, 0.1, 0.1),
                                                           math.pi / 2)],
    "rembrandt": [((0.664463, 0.342020, 0.664463), (1.0, 1.0, 1.0), math.pi / 4),
                  ((-0.707107, 0.0, 0.707107), (0.1, 0.1, 0.1), math.pi / 2)],
}


def _material(case):
    if case["scene"] == "hexagon":
        return dict(color=(1.0, 0.74, 0.02), roughness=0.3, specular=0.5, primitive_color_mix=0.0)
    if case["scene"] == "cubes":
        return dict(color=(0.8, 0.3, 0.2), roughness=0.3, specular=0.5, metal=0.5)
    return dict(color=(0.9, 0.9, 0.9), roughness=0.4, specular=0.5, primitive_color_mix=1.0)


def _view(case, half):
    """Camera of a case: the whole box in the image, from the front for flat scenes, else along
    the diagonal."""
    half = np.asarray(half, np.float64)
    flat = half[2] < 0.51 * half[0]
    v, up = (((0, 0, 1), (0, 1, 0)) if flat else ((1, 1, 1), (-1, 2, -1)))
    v, up = _unit(v), _unit(up)
    corners = np.array([[x, y, z] for x in (-1, 1) for y in (-1, 1) for z in (-1, 1)]) * half
    height = 2.1 * np.abs(corners @ up).max()
    distance = 1.1 * (corners @ v).max() + (1.0 if flat else 0.0)
    view = dict(position=v * distance, look_at=np.zeros(3), up=up, height=float(height),
                model=case.get("camera", "perspective"))
    if view["model"] == "perspective":
        f = 0.25 * distance  # the focal plane through the middle shows `height`
        view.update(focal_length=float(f), focus_distance=float(distance),
                    f_stop=float(case.get("f_stop", math.inf)), height=float(height * f / distance))
    return view


# ---------------------------------------------------------------------------------------------
# one case through the framework
# ---------------------------------------------------------------------------------------------
_device = None


def _the_device():
    global _device
    if _device is None:  # a program makes one and keeps it
        import fresnel_b200
        _device = fresnel_b200.Device(mode="gpu")
    return _device


def _scene(case, seed):
    import fresnel_b200 as fresnel
    from fresnel_b200 import workloads
    a = _arrays(case, seed)
    scene = fresnel.Scene(_the_device(), lights=[
        fresnel.light.Light(direction=d, color=c, theta=t)
        for d, c, t in _LIGHTS[case.get("lights", "lightbox")]])
    scene.background_color = (1, 1, 1)
    scene.background_alpha = 0
    mat = fresnel.material.Material(**_material(case))
    outline = case.get("outline", 0.0)
    if "pos" in a:
        fresnel.geometry.Sphere(scene, position=a["pos"], radius=a["radius"], color=a["color"],
                                material=mat, outline_width=outline)
    if "bonds" in a and len(a["bonds"]):
        fresnel.geometry.Cylinder(scene, points=a["bonds"], radius=0.1, color=(0.3, 0.3, 0.8),
                                  material=mat, outline_width=outline)
    if "cubes" in a:
        g = fresnel.geometry.ConvexPolyhedron(scene, workloads.unit_cube_planes(),
                                              position=a["cubes"], orientation=a["cubes_q"],
                                              color=(0.8, 0.3, 0.2), outline_width=outline)
        g.material = fresnel.material.Material(color=(0.8, 0.3, 0.2), metal=0.5, roughness=0.3)
    if "meshes" in a:
        verts = workloads.icosahedron(0.5)
        fresnel.geometry.Mesh(scene, verts, position=a["meshes"], orientation=a["meshes_q"],
                              color=np.full((len(verts), 3), 0.7, np.float32))
    if "polygons" in a:
        fresnel.geometry.Polygon(scene,
                                 vertices=np.array(workloads.POLYGON_OUTLINE, np.float32) * 0.5,
                                 position=a["polygons"], angle=a["angle"], color=a["color"],
                                 rounding_radius=0.1, material=mat, outline_width=outline)
    view = _view(case, a["half"])
    model = view.pop("model")
    cls = {"perspective": fresnel.camera.Perspective,
           "orthographic": fresnel.camera.Orthographic}[model]
    scene.camera = cls(**view)
    return scene, a


def _seeds(seed, n):
    """Random seeds of a case's images."""
    r = random.Random(int(seed) * 7919 + 5)
    return [r.randrange(1, 1 << 30) for _ in range(n)]


def prepare(case, seed):
    import fresnel_b200 as fresnel
    dev = _the_device()
    n = case.get("frames", 1)
    made = [_scene(case, int(seed) * 64 + i) for i in range(n)]
    cls = fresnel.tracer.Preview if case["kind"] == "preview" else fresnel.tracer.Path
    more = dict(anti_alias=bool(case["aa"])) if case["kind"] == "preview" else {}
    s = dict(case=case, scenes=[m[0] for m in made], seeds=_seeds(seed, n),
             tracers=[cls(dev, case["w"], case["h"], **more) for _ in range(n)])
    if case["kind"] == "frames":
        s["next"] = _arrays(case, int(seed) * 64 + 63)["pos"]
    if case["kind"] == "batch":
        s["batch"] = fresnel.tracer.PathBatch(dev)
    return s


def run(state):
    case = state["case"]
    for t, seed in zip(state["tracers"], state["seeds"]):
        t.seed = seed
    tracer, scene = state["tracers"][0], state["scenes"][0]
    if case["kind"] == "preview":
        tracer.render(scene)
    elif case["kind"] == "batch":
        for t, sc in zip(state["tracers"], state["scenes"]):
            state["batch"].add(t, sc, case["spp"], light_samples=case["light_samples"])
        state["batch"].render()
    else:
        if case["kind"] == "frames":
            scene.geometry[0].position[:] = state["next"]
        tracer.sample(scene, case["spp"], light_samples=case["light_samples"])
    out = [t.linear_output[:] if case["read"] == "linear" else t.output[:]
           for t in state["tracers"]]
    return {case["read"]: out}


def work(case):
    """Every particle read once (its shape and colour) and the image written once; every sample's
    camera ray (random numbers, a camera model, one intersection) and, for a path, at least one
    shaded vertex per light path."""
    per = dict(cubes=40, polygons=24, mixed=32, sticks=34).get(case["scene"], 28)
    n, px = case["n"], case["w"] * case["h"]
    frames = case.get("frames", 1)
    size = 16 if case["read"] == "linear" else 4
    samples = px * (case.get("spp") or (64 if case["aa"] else 1))
    flops = samples * (80 + 150 * case.get("light_samples", 1))
    moved = 12 * n if case["kind"] == "frames" else 0
    return dict(bytes=float(frames * (per * n + moved + size * px)), flops=float(frames * flops))


# ---------------------------------------------------------------------------------------------
# sphere scenes in 64 bits: plain torch, every ray against every sphere
# ---------------------------------------------------------------------------------------------
_EPS = 1e-4  # a sphere is left at least this far along the ray


def _philox(c, k):
    """Philox4x32-10 (Salmon et al., SC'11) on int64 tensors holding 32-bit words."""
    mask = 0xFFFFFFFF

    def mul(m, x):  # 32 x 32 -> (high, low) words
        lo = (m & 0xFFFF) * x
        hi = (m >> 16) * x
        s = (lo >> 16) + (hi & 0xFFFF)
        return (hi >> 16) + (s >> 16), ((s & 0xFFFF) << 16) | (lo & 0xFFFF)

    c, k = list(c), list(k)
    for _ in range(10):
        h0, l0 = mul(0xD2511F53, c[0])
        h1, l1 = mul(0xCD9E8D57, c[2])
        c = [h1 ^ c[1] ^ k[0], l1, h0 ^ c[3] ^ k[1], l0]
        k = [(k[0] + 0x9E3779B9) & mask, (k[1] + 0xBB67AE85) & mask]
    return [x.double() * 2.0**-32 + 2.0**-33 for x in c]


def _dot(a, b):
    return (a * b).sum(-1)


def _norm(a):
    return a / _dot(a, a).sqrt()[..., None]


class _Exact:
    """A sphere scene, its camera and its lights in 64 bits."""

    def __init__(self, case, seed, dev):
        f64 = dict(dtype=torch.float64, device=dev)
        a = _arrays(case, seed)

        def t(x):
            return torch.tensor(np.asarray(np.asarray(x, np.float32), np.float64), **f64)

        self.dev, self.case = dev, case
        self.pos, self.rad, self.col = t(a["pos"]), t(a["radius"]), t(a["color"])
        m = dict(solid=0, color=(0.9, 0.9, 0.9), primitive_color_mix=0, roughness=0.3,
                 specular=0.5, metal=0)
        m.update(_material(case))
        self.mat = {k: t(v) for k, v in m.items()}
        self.outline = float(np.float32(case.get("outline", 0.0)))
        v = _view(case, a["half"])
        self.p = t(v["position"])
        d = _norm(t(v["look_at"]) - self.p)
        self.u = _norm(torch.linalg.cross(d, _norm(t(v["up"]))))
        self.v = _norm(torch.linalg.cross(self.u, d))
        self.w = -d
        self.model = v["model"]
        height = float(np.float32(v["height"]))
        self.focal_h, self.aperture = height, 0.0
        if self.model == "perspective":
            f, fd = float(np.float32(v["focal_length"])), float(np.float32(v["focus_distance"]))
            self.focal_h, self.focal_d = height / f * fd, fd
            if case["kind"] != "preview":
                self.aperture = f / float(np.float32(v["f_stop"]))
        self.lights = []
        for direction, color, theta in _LIGHTS[case.get("lights", "lightbox")]:
            x = _norm(t(direction))
            self.lights.append((x[0] * self.u + x[1] * self.v + x[2] * self.w, t(color),
                                float(np.float32(theta))))

    def camera(self, pixel, sample, seed, jitter):
        w, h = self.case["w"], self.case["h"]
        i, j = (pixel % w).double() + 0.5, torch.div(pixel, w, rounding_mode="floor").double() + 0.5
        zero = torch.zeros_like(pixel)
        if jitter:
            r = _philox([zero, zero, sample, zero + 0x22AB5871], [pixel, zero + seed])

            def tent(x):
                x = 2 * x
                return torch.where(x < 1, x.sqrt() - 1, 1 - (2 - x).clamp(min=0).sqrt())

            i, j = i + tent(r[0]) * math.sqrt(0.5), j + tent(r[1]) * math.sqrt(0.5)
        ys = -(j / h - 0.5)
        xs = i / h - 0.5 * w / h
        plane = (ys[:, None] * self.v + xs[:, None] * self.u) * self.focal_h
        if self.model == "orthographic":
            return self.p + plane, (-self.w).expand_as(plane)
        c = self.p - self.w * self.focal_d + plane
        o = self.p.expand_as(c)
        if self.aperture:
            r = _philox([zero, zero, sample, zero + 0x983ABC12], [pixel, zero + seed])
            theta, rad = (r[0] * 2 * math.pi)[:, None], (r[1] * self.aperture / 2)[:, None]
            o = o + rad * theta.cos() * self.u + rad * theta.sin() * self.v
        return o, _norm(c - o)

    def closest(self, o, d, near):
        """(distance, sphere) of each ray's closest hit; infinity where there is none."""
        best = torch.full((len(o),), math.inf, dtype=torch.float64, device=self.dev)
        prim = torch.zeros(len(o), dtype=torch.int64, device=self.dev)
        rows = max(1, int(6e7) // len(self.pos))
        pp = _dot(self.pos, self.pos)
        rr = self.rad * self.rad - pp
        for a in range(0, len(o), rows):
            oo, dd = o[a:a + rows], d[a:a + rows]
            b = dd @ self.pos.T - _dot(oo, dd)[:, None]
            det = (2 * oo) @ self.pos.T
            det += rr
            det -= _dot(oo, oo)[:, None]
            det += b * b  # b^2 - |p - o|^2 + r^2
            ok = det >= 0
            det.clamp_(min=0).sqrt_()
            t = b - det
            t = torch.where(t > _EPS, t, b.add_(det))
            t[~(ok & (t > max(near, _EPS)))] = math.inf
            best[a:a + rows], prim[a:a + rows] = t.min(dim=1)
        return best, prim

    def surface(self, o, d, t, prim):
        p, r = self.pos[prim], self.rad[prim]
        c = torch.linalg.cross(p - o, d)
        edge = r - _dot(c, c).sqrt()
        return _norm(o + t[:, None] * d - p), edge, self.col[prim]

    def base(self, color):
        m = self.mat
        return (1 - m["primitive_color_mix"]) * m["color"] + m["primitive_color_mix"] * color

    def brdf(self, l, v, n, color, half=None):
        """Diffuse and specular parts of the Disney BRDF (half: a light's half angle)."""
        m = self.mat
        h = _norm(l + v)
        ndotv, ndotl, ldoth, ndoth = _dot(n, v), _dot(n, l), _dot(l, h), _dot(n, h)
        base = self.base(color)
        schlick = lambda x: (1 - x) ** 5  # noqa: E731
        fl, fv, rr = schlick(ndotl), schlick(ndotv), 2 * m["roughness"] * ldoth * ldoth
        s = (1 - 0.5 * fl) * (1 - 0.5 * fv) + rr * (fl + fv + fl * fv * (rr - 1))
        f_d = base / math.pi * s[:, None] * (1 - m["metal"])
        alpha = m["roughness"] ** 2
        a2 = alpha * alpha
        dd = a2 / (math.pi * (1 + (a2 - 1) * ndoth * ndoth) ** 2)
        if half is not None:
            half = min(half, 0.99 * math.pi / 2)
            if half > 0:
                ap = torch.clamp(alpha + 0.5 * math.tan(half), max=1.0)
                dd = dd * a2 / (ap * ap)
        f0 = (1 - m["metal"]) * 0.08 * m["specular"] + m["metal"] * base
        fr = f0 + (1 - f0) * schlick(ldoth)[:, None]
        vis = (1 / (ndotv + (a2 + ndotv**2 - a2 * ndotv**2).sqrt()) /
               (ndotl + (a2 + ndotl**2 - a2 * ndotl**2).sqrt()))
        f_s = dd[:, None] * fr * vis[:, None]
        keep = (ndotv > 0)[:, None]
        return torch.where(keep, f_d, 0 * f_d), torch.where(keep, f_s, 0 * f_s)

    def preview(self, pixel, sample, seed, jitter):
        """RGBA of one Preview sample of each pixel (direct light by representative points)."""
        o, d = self.camera(pixel, sample, seed, jitter)
        t, prim = self.closest(o, d, 0.0)
        out = torch.ones(len(o), 4, dtype=torch.float64, device=self.dev)  # the background
        out[:, 3] = 0
        hit = torch.isfinite(t)
        d = d[hit]
        n, edge, color = self.surface(o[hit], d, t[hit], prim[hit])
        v = -_norm(d)
        c = torch.zeros_like(n)
        for l, lc, theta in self.lights:
            l = l.expand_as(n)
            r = 2 * n * _dot(n, v)[:, None] - v
            ldotr = _dot(l, r)
            ax = _norm(torch.linalg.cross(l, r))
            ang = (theta - torch.acos(ldotr.clamp(-1, 1)))[:, None]
            turned = (r * ang.cos() + torch.linalg.cross(ax, r) * ang.sin() +
                      ax * _dot(ax, r)[:, None] * (1 - ang.cos()))
            r = torch.where((ldotr < math.cos(theta))[:, None], turned, r)
            ndotl, ndotr = _dot(n, l)[:, None], _dot(n, r)[:, None]
            f_d = torch.where(ndotl >= 0, self.brdf(l, v, n, color)[0] * ndotl, 0 * n)
            f_s = torch.where(ndotr >= 0, self.brdf(r, v, n, color, theta)[1] * ndotr, 0 * n)
            c += (f_d + f_s) * math.pi * lc
        c[edge < self.outline] = 0  # the outline: solid black
        out[hit, :3], out[hit, 3] = c, 1.0
        return out

    def path(self, pixel, sample, light, lights, seed, first):
        """Radiance of one light path of each pixel sample (first: the camera ray's hit)."""
        o, d, t, prim = (x.clone() for x in first)
        result = torch.zeros(len(o), 3, dtype=torch.float64, device=self.dev)
        att = torch.ones_like(result)
        live = torch.arange(len(o), device=self.dev)
        s = (sample - 1) * lights + light
        m = self.mat
        alpha = m["roughness"] ** 2
        for depth in range(1 << 16):
            miss = ~torch.isfinite(t)
            gone = live[miss]
            if depth == 0:
                result[gone] = 1.0  # the background
            else:
                for l, lc, theta in self.lights:
                    lit = (_dot(d[miss], l) >= math.cos(theta)).double()[:, None]
                    result[gone] += lit * att[gone] * lc / math.sin(min(theta, math.pi / 2))
            live, o, d, t, prim = (x[~miss] for x in (live, o, d, t, prim))
            if not len(live):
                break
            n, edge, color = self.surface(o, d, t, prim)
            px, sm = pixel[live], s[live]
            zero = torch.zeros_like(px)
            x0, x1, pick, _ = _philox([zero, zero + depth, sm, zero + 0x8754ABCD],
                                      [px, zero + seed])
            v = -d
            diffuse = (pick <= 0.5)
            z_g = ((1 - x1) / (1 + (alpha * alpha - 1) * x1)).sqrt()
            rho = torch.where(diffuse, x0.sqrt(), (1 - z_g * z_g).clamp(min=0).sqrt())
            z = torch.where(diffuse, (1 - x0).sqrt(), z_g)
            ang = 2 * math.pi * torch.where(diffuse, x1, x0)
            up = torch.zeros_like(n)
            steep = n[:, 2].abs() > 0.999
            up[:, 2], up[:, 0] = (~steep).double(), steep.double()
            tx = _norm(torch.linalg.cross(up, n))
            ty = torch.linalg.cross(n, tx)
            w = (tx * (rho * ang.cos())[:, None] + ty * (rho * ang.sin())[:, None] +
                 n * z[:, None])
            l = torch.where(diffuse[:, None], w, 2 * _dot(v, w)[:, None] * w - v)
            h = _norm(l + v)
            ndotl, ndoth = _dot(n, l), _dot(n, h)
            p_d = (ndotl / math.pi).clamp(min=0)
            a2 = alpha * alpha
            dd = a2 / (math.pi * (1 + (a2 - 1) * ndoth * ndoth) ** 2)
            p_g = (dd * ndoth / (4 * _dot(l, h))).clamp(min=0)
            f_d, f_s = self.brdf(l, v, n, color)
            factor = 2 / (p_d + p_g)
            att[live] *= (f_d + f_s) * (ndotl * factor)[:, None]
            rr = _philox([zero, zero + depth, sm, zero + 0x54ABF853], [px, zero + seed])[0]
            prob = att[live].amax(-1).clamp(max=1)
            go = (_dot(n, v) > 0) & (ndotl > 0) & (rr <= prob) & (edge >= self.outline)
            att[live] /= prob[:, None]
            o, d = (o + t[:, None] * d)[go], l[go]
            live = live[go]
            if not len(live):
                break
            t, prim = self.closest(o, d, 1e-3)
        return result


def exact(case, seed):
    """What `run` returns for a scene of spheres, in 64 bits; None for other scenes, where every
    ray against every sphere takes too long, and for bytes."""
    if case["scene"] not in ("spheres", "hexagon") or case["kind"] not in ("preview", "path") or \
            case["read"] != "linear":
        return None
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    w, h = case["w"], case["h"]
    spp = case.get("spp") or (64 if case["aa"] else 1)
    lights = case.get("light_samples", 1)
    rays = w * h * spp * (1 if case["kind"] == "preview" else 1 + lights)
    if rays * case["n"] > (1.2e11 if dev.type == "cuda" else 2e9) or rays > 3e7:
        return None
    sc = _Exact(case, int(seed) * 64, dev)
    image_seed = _seeds(seed, 1)[0]
    pixel = torch.arange(w * h, device=dev)
    total = torch.zeros(w * h, 4, dtype=torch.float64, device=dev)
    for k in range(spp):
        if case["kind"] == "preview":
            total += sc.preview(pixel, torch.full_like(pixel, k), image_seed, bool(case["aa"]))
            continue
        sample = torch.full_like(pixel, k + 1)
        o, d = sc.camera(pixel, sample, image_seed + 1, True)  # `sample` advances the seed
        first = (o, d) + sc.closest(o, d, 1e-3)
        for ls in range(lights):
            total[:, :3] += sc.path(pixel, sample, ls, lights, image_seed + 1, first) / lights
        total[:, 3] += torch.isfinite(first[2]).double()
    return {"linear": [(total / spp).reshape(h, w, 4).cpu().numpy()]}
