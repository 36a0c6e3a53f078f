// lists.cu -- building the per-pixel primitive lists of beam.cuh.
//
// Grids: one warp per tile of 8 x 4 pixels.  The warp walks the tile's beam through the grid slab by
// slab along the beam's main axis; the references of a slab's cells are tested against the tile's
// beam by all lanes side by side (one reference per lane), and each survivor is then tested by
// every lane against its own pixel's beam and kept in the lane's list.  One walk serves 32 pixels
// and all their samples: on the 1M-sphere frame at 1920x1080 the lists of a frame take about 0.5 ms.
//
// A beam is an axis (o, d) and a radius R(tau) about the axis point at distance tau that covers
// every ray of the beam at the same parameter: the jitter (perspective: growing with tau;
// parallel projection: constant), the lens (shrinking towards the focal plane, growing behind
// it) and the rounding of positions.  A ray's own distance t to such a point is tau times a factor
// within 1 -+ g.
#include <algorithm>
#include <cmath>

#include "beam.cuh"

namespace fr {

namespace {

constexpr float INF = __builtin_huge_valf();

// Largest jitter of a camera ray about its pixel's centre, in pixels: the tent filter reaches
// 0.70711 along each axis, 1 along the diagonal (and the rounding of pixel coordinates).
constexpr float PIXEL_REACH = 1.003f;
// The same about the centre of a tile of 8 x 4 pixels: (3.5 + 0.7072, 1.5 + 0.7072).
constexpr float TILE_REACH = 4.76f;

// Square root to a few units in the last place: every bound here is widened by far more.
__device__ __forceinline__ float root(float x)
{
    float y;
    asm("sqrt.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

struct Beam {
    V3 o, d;         // axis, d of unit length
    float lens;      // radius of the beam's origin about o
    float inv_focus; // 1 / distance along the axis at which the lens's part vanishes
    float grow;      // radius gained per unit of tau
    float base;      // constant part of the radius
    float g;         // spread of t / tau
    __device__ __forceinline__ float at(float tau) const
    {
        return fabsf(1.0f - tau * inv_focus) * lens + tau * grow + base;
    }
    // largest radius over [a, b] (the radius is convex in tau)
    __device__ __forceinline__ float over(float a, float b) const { return fmaxf(at(a), at(b)); }
};

// The beam of all camera rays within `reach` pixels of image position (x, y) (pixel centres at
// half-integers): camera_ray's geometry without the jitter.
__device__ __forceinline__ Beam make_beam(const CamK& k, float x, float y, float reach)
{
    const float ys = -1.0f * (y / float(k.height) - 0.5f);
    const float xs = x / float(k.height) - 0.5f * float(k.width) / float(k.height);
    const V3 plane = ys * k.v + xs * k.u;
    const float rho = reach * fabsf(k.focal_h) / float(k.height);
    Beam b;
    if (k.model == 0) {
        b.o = k.p + plane * k.focal_h;
        b.d = -k.w;
        b.lens = 0.0f;
        b.inv_focus = 0.0f;
        b.grow = 0.0f;
        b.base = rho;
        b.g = 1e-6f;
        return b;
    }
    b.o = k.p;
    const V3 D = k.p - k.w * k.focal_d + plane * k.focal_h - k.p;
    const float L = root(dot(D, D));
    b.d = D * (1.0f / L);
    b.lens = 0.5f * fabsf(k.aperture) * 1.0001f;
    b.inv_focus = 1.0f / L;
    // the focal point's coordinates are rounded before the direction is taken
    const float m = fmaxf(fmaxf(fabsf(k.p.x), fabsf(k.p.y)), fabsf(k.p.z));
    b.grow = rho / L + 4e-7f * (m + L) / L;
    b.base = 0.0f;
    b.g = (rho + b.lens) / L + 1e-6f;
    return b;
}

// Adds the rounding of positions up to `far` from the axis's origin to the radius; false when
// the beam is too wide (or not a number) for the bounds used here.
__device__ __forceinline__ bool finish_beam(Beam& b, float far)
{
    const float m = fmaxf(fmaxf(fabsf(b.o.x), fabsf(b.o.y)), fabsf(b.o.z));
    b.base += 4e-6f * (m + far);
    return b.g < 0.1f && far < 1e30f && b.at(far) < far;
}

// One pixel's list while it is built: entries in shared memory, nearest first.
struct ListBuilder {
    uint2* e;        // entry k of this lane at e[k * 32]
    uint32_t n;
    float complete;  // every possible hit nearer than this is listed
    float certain;   // every ray of the beam is hit nearer than this
    __device__ __forceinline__ void start(uint2* entries)
    {
        e = entries;
        n = 0;
        complete = INF;
        certain = INF;
    }
    // distances beyond this cannot matter any more
    __device__ __forceinline__ float reach() const { return fminf(complete, certain); }
    __device__ __forceinline__ void add(uint32_t slot, float t_lo)
    {
        if (t_lo > reach())
            return;
        if (n == LIST_MAX) {  // the farthest entry leaves: the list is complete up to it
            const float last = __uint_as_float(e[(n - 1u) * 32u].y);
            complete = fminf(complete, fmaxf(last, t_lo));
            if (t_lo >= last)
                return;
            --n;
        }
        uint32_t k = n;
        while (k > 0u && __uint_as_float(e[(k - 1u) * 32u].y) > t_lo) {
            e[k * 32u] = e[(k - 1u) * 32u];
            --k;
        }
        e[k * 32u] = make_uint2(slot, __float_as_uint(t_lo));
        ++n;
    }
    __device__ __forceinline__ void store(uint2* out) const
    {
        // entries beyond `certain` or `complete` are never needed, and a ray that no entry answers
        // nearer than that walks: only a list with neither bound can tell that a ray misses
        uint32_t m = n;
        while (m > 0u && __uint_as_float(e[(m - 1u) * 32u].y) > reach())
            --m;
        out[0] = make_uint2(m, __float_as_uint(reach()));
        for (uint32_t k = 0; k < m; ++k)
            out[k + 1u] = e[k * 32u];
    }
};

// What deciding whether a beam meets a sphere takes besides the distance of the sphere's centre
// from the beam's axis.  The pixels of a tile share it: their rays start at one point (or within
// `spread` of it: the lens), or in one plane along parallel axes.
struct SphereBounds {
    float reach;    // some ray may be accepted by the float test if the distance is at most
    float t_lo;     // this, and then not nearer than t_lo
    float inner2;   // every ray is hit before t_hi if the squared distance is at most this and
                    // the centre lies ahead of the beam's origin
    float t_hi;
    float hi;       // no ray is hit beyond this
};

// radius(tau) bounds the radius of the beams in question.
template <class Radius>
__device__ __forceinline__ SphereBounds sphere_bounds(const Beam& b, bool parallel, float spread,
                                                      V3 c, float r, const Radius& radius)
{
    SphereBounds s;
    const V3 v = c - b.o;
    const float far = root(dot(v, v)) * (1.0f + 1e-6f);
    const float dist = parallel ? dot(v, b.d) : far;
    const float slack = SPHERE_SLACK * (far + spread) * (far + spread) + 1e-12f;
    const float round = 2e-6f * (far + spread);
    const float re = root(r * r + slack) * (1.0f + 1e-6f) + round;
    const float lo = fmaxf(dist - re - b.lens, 0.0f);
    s.hi = (fmaxf(dist, 0.0f) + re + b.lens) * (1.0f + 1.2f * b.g);
    const float R = fmaxf(radius(lo * (1.0f - 1.1f * b.g)), radius(s.hi));
    s.reach = (re + R + round) * (1.0f + 1e-5f);
    s.t_lo = lo * (1.0f - 1e-5f);
    const float solid = r * r - slack;
    const float inner = solid > 0.0f ? root(solid) * (1.0f - 1e-6f) - R - round : -1.0f;
    s.inner2 = (inner > 0.0f && lo > 0.02f) ? inner * inner * (1.0f - 1e-5f) : -1.0f;
    s.t_hi = (dist + b.lens) * (1.0f + 1e-5f);
    return s;
}

// Squared distance of c from the line of the beam's axis; tau: of its foot along the axis.
__device__ __forceinline__ float axis_dist2(const Beam& b, V3 c, float& tau)
{
    const V3 v = c - b.o;
    tau = fmaf(v.x, b.d.x, fmaf(v.y, b.d.y, v.z * b.d.z));
    const float x = fmaf(-tau, b.d.x, v.x), y = fmaf(-tau, b.d.y, v.y), z = fmaf(-tau, b.d.z, v.z);
    return fmaf(x, x, fmaf(y, y, z * z));
}

// The same for a box (centre c, half extents e): the axis against the box widened by R; t_lo: some
// ray may reach a cell that the box lies in from there on.
__device__ __forceinline__ bool beam_box(const Beam& b, const RayK& axis, V3 c, V3 e, float R,
                                         const GridDev& G, float& t_lo)
{
    const float scale = fmaxf(fmaxf(fabsf(c.x) + e.x, fabsf(c.y) + e.y), fabsf(c.z) + e.z);
    const float w = R + 2e-4f * scale + 2e-5f;  // beyond the padding of the walk's own box test
    const float4 lo = make_float4(c.x - e.x - w, c.y - e.y - w, c.z - e.z - w, 0.0f);
    const float4 hi = make_float4(c.x + e.x + w, c.y + e.y + w, c.z + e.z + w, 0.0f);
    float t;
    if (!slab(axis, lo, hi, INF, t))
        return false;
    const float p = w - R;  // the padding alone
    float4 cl = make_float4(c.x - e.x - p, c.y - e.y - p, c.z - e.z - p, 0.0f);
    float4 ch = make_float4(c.x + e.x + p, c.y + e.y + p, c.z + e.z + p, 0.0f);
    cells_of(G, cl, ch);
    slab(axis, make_float4(cl.x - w, cl.y - w, cl.z - w, 0.0f),
         make_float4(ch.x + w, ch.y + w, ch.z + w, 0.0f), INF, t);
    t_lo = t * (1.0f - b.g) * (1.0f - 1e-5f);
    return true;
}

__device__ __forceinline__ float comp(V3 a, int k) { return k == 0 ? a.x : (k == 1 ? a.y : a.z); }

// A reference of a grid over parts as the shape the beams are tested against.
struct PartShape {
    V3 c, e;          // sphere: e.x is its radius; else a box of half extents e
    bool sphere;
    bool regular;     // its surface lies within the shape, so no hit comes before the shape's
};

__device__ __forceinline__ PartShape part_shape(const SceneDev& sc, uint32_t s, uint32_t gw)
{
    PartShape p;
    const uint32_t gi = gw & ((1u << PART_TYPE_SHIFT) - 1u);
    const int type = int(gw >> PART_TYPE_SHIFT);
    const float4 a = ldg4(sc.leaf_data + 2 * size_t(s));
    p.c = v3(a.x, a.y, a.z);
    p.sphere = true;
    p.regular = true;
    p.e = v3(a.w, a.w, a.w);
    if (type == FR_GEOM_SPHERE)
        return p;
    const float4 b = ldg4(sc.leaf_data + 2 * size_t(s) + 1);
    const GeomDev& g = sc.geoms[gi];
    p.sphere = false;
    if (type == FR_GEOM_CYLINDER) {
        const float r = fabsf(a.w);
        p.c = v3(0.5f * (a.x + b.x), 0.5f * (a.y + b.y), 0.5f * (a.z + b.z));
        p.e = v3(0.5f * fabsf(a.x - b.x) + r, 0.5f * fabsf(a.y - b.y) + r,
                 0.5f * fabsf(a.z - b.z) + r);
        p.regular = a.w >= 0.0f;
        return p;
    }
    const float q2 = b.x * b.x + b.y * b.y + b.z * b.z + b.w * b.w;
    p.regular = g.bounded != 0u && fabsf(q2 - 1.0f) < UNIT_SLACK;
    float r = g.bound_radius;
    if (type == FR_GEOM_MESH)
        r = r * fmaxf(q2, 1.0f) * 1.0001f;
    p.e = v3(r, r, r);
    if (type == FR_GEOM_POLYGON) {
        p.c.z = 0.0f;
        p.e.z = 0.0f;
    }
    return p;
}

// Index of the cell holding coordinate x along axis k (clamped).
__device__ __forceinline__ int clamp_cell(float x, float lo, float ih, uint32_t n)
{
    return int(fminf(fmaxf(floorf((x - lo) * ih), 0.0f), float(n - 1u)));
}

constexpr float BOX = -2.0f;            // marks a box record (a sphere's inner2 is -1 or more)
constexpr uint32_t LIST_BUDGET = 4096;  // cells and references a tile's walk may visit

template <bool PARTS>
__global__ void __launch_bounds__(128, 6) k_pixel_lists_grid(FrameParams P, uint2* out)
{
    __shared__ uint2 entries[4][LIST_MAX * 32];
    __shared__ float4 found_rec[4][32], found_bnd[4][32];
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t tiles_x = (P.w + 7u) >> 3;
    const uint32_t tile = blockIdx.x * 4u + warp;
    const uint32_t ty = tile / tiles_x, tx = tile - ty * tiles_x;
    const uint32_t i = tx * 8u + (lane & 7u), j = ty * 4u + (lane >> 3);
    if (ty * 4u >= P.h)
        return;  // warp-uniform
    const bool valid = i < P.w && j < P.h;
    const SceneDev& sc = P.scene;
    const GridDev& G = sc.grid;

    Beam tb = make_beam(P.cam, float(tx * 8u) + 4.0f, float(ty * 4u) + 2.0f, TILE_REACH);
    Beam pb = make_beam(P.cam, float(i) + 0.5f, float(j) + 0.5f, PIXEL_REACH);
    const V3 gc = v3(0.5f * (G.lox + G.hix), 0.5f * (G.loy + G.hiy), 0.5f * (G.loz + G.hiz));
    const V3 ge = v3(0.5f * (G.hix - G.lox), 0.5f * (G.hiy - G.loy), 0.5f * (G.hiz - G.loz));
    const V3 oc = gc - tb.o;
    const float far = root(dot(oc, oc)) + root(dot(ge, ge));
    // the walks' padding scales with the coordinates; a camera far outside them could make the
    // rounding of its distances exceed it
    const float scale = fmaxf(fmaxf(fmaxf(fabsf(G.lox), fabsf(G.hix)),
                                    fmaxf(fabsf(G.loy), fabsf(G.hiy))),
                              fmaxf(fabsf(G.loz), fabsf(G.hiz)));
    ListBuilder L;
    L.start(entries[warp] + lane);
    const bool parallel = P.cam.model == 0;
    const bool fits = finish_beam(tb, far) && far <= 16.0f * scale;
    const bool fits_lane = finish_beam(pb, far);
    if (!__all_sync(0xffffffffu, fits && (fits_lane || !valid))) {
        L.complete = 0.0f;
        if (valid)
            L.store(out + size_t(LIST_WORDS) * (size_t(j) * P.w + i));
        return;
    }
    const RayK tile_axis = make_rayk(tb.o, tb.d), axis = make_rayk(pb.o, pb.d);
    const float tile_R = tb.over(0.0f, far * (1.0f + 2.0f * tb.g));
    const float R = pb.over(0.0f, far * (1.0f + 2.0f * pb.g));
    // a bound on the radius of every pixel's beam of the tile, and how much wider the tile's is
    const float narrow = PIXEL_REACH / TILE_REACH;
    const float spread = parallel ? tile_R : tb.lens;
    auto pixel_radius = [&](float tau) {
        const float f = tau * tb.inv_focus;
        return (fabsf(1.0f - f) + 2.0f * f * tb.g) * tb.lens +
               tau * tb.grow * (narrow * (1.0f + 4.0f * tb.g) + 0.01f) +
               (parallel ? tb.base * (narrow + 0.01f) : tb.base);
    };

    // the tile's beam within the grid, and the axis it advances fastest along (in cells)
    float t_in = 0.0f, t_out = 0.0f;
    bool inside = false;
    {
        const float4 lo = make_float4(G.lox - tile_R, G.loy - tile_R, G.loz - tile_R, 0.0f);
        const float4 hi = make_float4(G.hix + tile_R, G.hiy + tile_R, G.hiz + tile_R, 0.0f);
        inside = slab(tile_axis, lo, hi, INF, t_in);
        const float x0 = fmaf(lo.x, tile_axis.inv.x, tile_axis.oinv.x);
        const float x1 = fmaf(hi.x, tile_axis.inv.x, tile_axis.oinv.x);
        const float y0 = fmaf(lo.y, tile_axis.inv.y, tile_axis.oinv.y);
        const float y1 = fmaf(hi.y, tile_axis.inv.y, tile_axis.oinv.y);
        const float z0 = fmaf(lo.z, tile_axis.inv.z, tile_axis.oinv.z);
        const float z1 = fmaf(hi.z, tile_axis.inv.z, tile_axis.oinv.z);
        t_out = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fmaxf(z0, z1));
    }
    if (inside) {
        const float ax = fabsf(tb.d.x) * G.ihx, ay = fabsf(tb.d.y) * G.ihy, az = fabsf(tb.d.z) * G.ihz;
        const int k = (ax >= ay && ax >= az) ? 0 : (ay >= az ? 1 : 2);
        const int a = k == 0 ? 1 : 0, b = k == 2 ? 1 : 2;  // the lateral axes
        const V3 glo = v3(G.lox, G.loy, G.loz), gh = v3(G.hx, G.hy, G.hz), gih = v3(G.ihx, G.ihy, G.ihz);
        const uint32_t nk = k == 0 ? G.nx : (k == 1 ? G.ny : G.nz);
        const uint32_t na = a == 0 ? G.nx : G.ny, nb = b == 1 ? G.ny : G.nz;
        const uint32_t sk = k == 0 ? 1u : (k == 1 ? G.nx : G.nx * G.ny);
        const uint32_t sa = a == 0 ? 1u : G.nx, sb = b == 1 ? G.nx : G.nx * G.ny;
        const float ok = comp(tb.o, k), oa = comp(tb.o, a), ob = comp(tb.o, b);
        const float dk = comp(tb.d, k), da = comp(tb.d, a), db = comp(tb.d, b);
        const int step = dk >= 0.0f ? 1 : -1;
        const float sg = dk >= 0.0f ? 1.0f : -1.0f, idk = 1.0f / fabsf(dk);
        const float lok = comp(glo, k), hk = comp(gh, k);
        int m = clamp_cell(ok + t_in * dk - sg * tile_R, lok, comp(gih, k), nk);
        uint32_t work = 0;
        uint32_t seen_g = MISS, seen_p = MISS, n_seen = 0;  // the last 32 survivors, one per lane
        while (m >= 0 && m < int(nk)) {
            // the slab's two planes, in the order the beam meets them
            const float xa = lok + float(step > 0 ? m : m + 1) * hk;
            const float xb = lok + float(step > 0 ? m + 1 : m) * hk;
            const float ta0 = ((xa - ok) * sg - tile_R) * idk;
            if (ta0 > t_out)
                break;
            const float tb0 = fminf(((xb - ok) * sg + tile_R) * idk, far);
            const float Rs = fminf(tile_R, tb.over(fmaxf(ta0, 0.0f), fmaxf(tb0, 0.0f)));
            const float ta = fmaxf(((xa - ok) * sg - Rs) * idk, 0.0f);
            const float tz = fmaxf(((xb - ok) * sg + Rs) * idk, 0.0f);
            const float a0 = fminf(oa + ta * da, oa + tz * da) - Rs, a1 = fmaxf(oa + ta * da, oa + tz * da) + Rs;
            const float b0 = fminf(ob + ta * db, ob + tz * db) - Rs, b1 = fmaxf(ob + ta * db, ob + tz * db) + Rs;
            const float la = comp(glo, a), lb = comp(glo, b);
            const float ha = a == 0 ? G.hix : G.hiy, hb = b == 1 ? G.hiy : G.hiz;
            if (a1 >= la && a0 <= ha && b1 >= lb && b0 <= hb) {
                const uint32_t ia0 = uint32_t(clamp_cell(a0, la, comp(gih, a), na));
                const uint32_t ib0 = uint32_t(clamp_cell(b0, lb, comp(gih, b), nb));
                const uint32_t wa = uint32_t(clamp_cell(a1, la, comp(gih, a), na)) - ia0 + 1u;
                const uint32_t wb = uint32_t(clamp_cell(b1, lb, comp(gih, b), nb)) - ib0 + 1u;
                const uint32_t cells = wa * wb;
                work += cells;
                for (uint32_t c0 = 0; c0 < cells && work < LIST_BUDGET; c0 += 32u) {
                    uint32_t first = 0, cnt = 0;
                    if (c0 + lane < cells) {
                        const uint32_t cb = (c0 + lane) / wa, ca = (c0 + lane) - cb * wa;
                        const uint32_t id = uint32_t(m) * sk + (ia0 + ca) * sa + (ib0 + cb) * sb;
                        first = __ldg(G.cell_start + id);
                        cnt = __ldg(G.cell_start + id + 1u) - first;
                    }
                    uint32_t upto = cnt;  // references of this lane's cell and those before it
                    for (uint32_t off = 1; off < 32u; off <<= 1) {
                        const uint32_t v = __shfl_up_sync(0xffffffffu, upto, off);
                        if (lane >= off)
                            upto += v;
                    }
                    const uint32_t total = __shfl_sync(0xffffffffu, upto, 31);
                    work += total;
                    for (uint32_t r0 = 0; r0 < total; r0 += 32u) {
                        const uint32_t r = r0 + lane;
                        uint32_t own = 0;  // the cell reference r belongs to
                        for (uint32_t bit = 16; bit; bit >>= 1) {
                            const uint32_t v = __shfl_sync(0xffffffffu, upto, own + bit - 1u);
                            if (v <= r)
                                own += bit;
                        }
                        own = min(own, 31u);
                        const uint32_t f = __shfl_sync(0xffffffffu, first, own);
                        const uint32_t u = __shfl_sync(0xffffffffu, upto, own);
                        const uint32_t n_own = __shfl_sync(0xffffffffu, cnt, own);
                        const uint32_t ref = f + (r - (u - n_own));
                        bool pass = false, regular = true;
                        // the record the lanes test: a sphere's centre, reach^2 and bounds, or
                        // (bounds.inner2 = BOX) a box's centre and half extents
                        float4 rec = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        float4 bnd = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        uint32_t key_g = 0, key_p = 0;
                        if (r < total) {
                            key_p = __ldg((PARTS ? sc.order : G.ref_prim) + ref);
                            V3 c;
                            float rad = 0.0f;
                            bool sphere = true;
                            PartShape sh;
                            if (PARTS) {
                                key_g = __ldg(sc.leaf_geom + ref);
                                sh = part_shape(sc, ref, key_g);
                                c = sh.c;
                                rad = sh.e.x;
                                sphere = sh.sphere;
                                regular = sh.regular;
                            } else {
                                const float4 q = ldg4(G.ref_sphere + ref);
                                c = v3(q.x, q.y, q.z);
                                rad = q.w;
                            }
                            if (sphere) {
                                const SphereBounds sb =
                                    sphere_bounds(tb, parallel, spread, c, rad, pixel_radius);
                                const float w = sb.reach + tb.over(sb.t_lo * (1.0f - 1.2f * tb.g), sb.hi);
                                float tau;
                                pass = axis_dist2(tb, c, tau) <= w * w;
                                rec = make_float4(c.x, c.y, c.z, sb.reach * sb.reach);
                                bnd = make_float4(sb.t_lo, sb.inner2, sb.t_hi, 0.0f);
                            } else {
                                float t_lo;
                                pass = beam_box(tb, tile_axis, c, sh.e, tile_R, G, t_lo);
                                rec = make_float4(c.x, c.y, c.z, sh.e.x);
                                bnd = make_float4(sh.e.y, BOX, sh.e.z, 0.0f);
                            }
                            if (!regular)
                                rec.w = -rec.w - 1e-30f;
                        }
                        uint32_t left = __ballot_sync(0xffffffffu, pass);
                        if (pass) {
                            const uint32_t k = __popc(left & ((1u << lane) - 1u));
                            found_rec[warp][k] = rec;
                            found_bnd[warp][k] = make_float4(bnd.x, bnd.y, bnd.z, __uint_as_float(ref));
                        }
                        __syncwarp();
                        for (uint32_t k = 0; left; ++k) {
                            const int from = __ffs(left) - 1;
                            left &= left - 1u;
                            const uint32_t p = __shfl_sync(0xffffffffu, key_p, from);
                            const uint32_t gw = PARTS ? __shfl_sync(0xffffffffu, key_g, from) : 0u;
                            if (__any_sync(0xffffffffu, seen_p == p && seen_g == gw))
                                continue;  // met in another cell just before
                            if (lane == (n_seen & 31u)) {
                                seen_p = p;
                                seen_g = gw;
                            }
                            ++n_seen;
                            const float4 q = found_rec[warp][k], u = found_bnd[warp][k];
                            const V3 c = v3(q.x, q.y, q.z);
                            float t_lo = u.x;
                            bool hit;
                            if (!PARTS || u.y != BOX) {
                                float tau;
                                const float a2 = axis_dist2(pb, c, tau);
                                hit = a2 <= q.w;
                                if (a2 <= u.y && tau > 0.0f)
                                    L.certain = fminf(L.certain, u.z);
                            } else {
                                const bool odd = q.w < 0.0f;
                                hit = beam_box(pb, axis, c, v3(odd ? -q.w : q.w, u.x, u.z), R, G,
                                               t_lo);
                                if (odd)
                                    t_lo = 0.0f;
                            }
                            if (hit)
                                L.add(__float_as_uint(u.w), t_lo);
                        }
                        __syncwarp();
                    }
                }
            }
            // every hit nearer than this lies in the slabs walked so far
            const float upto_t = fmaxf(((xb - ok) * sg - Rs) * idk, 0.0f) * (1.0f - tb.g) *
                                 (1.0f - 1e-5f);
            if (work >= LIST_BUDGET) {  // this slab may be unfinished
                L.complete = fminf(L.complete, fmaxf(((xa - ok) * sg - Rs) * idk, 0.0f) *
                                                   (1.0f - tb.g) * (1.0f - 1e-5f));
                break;
            }
            if (__all_sync(0xffffffffu, !valid || L.reach() <= upto_t || L.n >= P.list_enough)) {
                L.complete = fminf(L.complete, upto_t);
                break;
            }
            m += step;
        }
    }
    if (valid)
        L.store(out + size_t(LIST_WORDS) * (size_t(j) * P.w + i));
}

__global__ void __launch_bounds__(256) k_part_bounds(SceneDev sc, uint32_t n, float4* bound)
{
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n)
        return;
    const uint32_t gw = __ldg(sc.leaf_geom + s);
    const PartShape p = part_shape(sc, s, gw);
    if (p.sphere) {
        bound[s] = make_float4(p.c.x, p.c.y, p.c.z, p.e.x);
        return;
    }
    float r;
    if (int(gw >> PART_TYPE_SHIFT) == FR_GEOM_CYLINDER) {
        const float4 a = ldg4(sc.leaf_data + 2 * size_t(s)), b = ldg4(sc.leaf_data + 2 * size_t(s) + 1);
        const V3 h = v3(b.x - a.x, b.y - a.y, b.z - a.z);
        r = 0.5f * root(dot(h, h)) + fabsf(a.w);
    } else {
        r = p.e.x;  // a bounding radius about the position
        // The polyhedron test stops, and accepts, once the entry and the exit found so far are
        // equal, without looking at the planes left: a ray that crosses the extension of an edge
        // can be hit outside the polyhedron, though (as the test's own box test asks) only if it
        // meets the box of that radius.
        if (int(gw >> PART_TYPE_SHIFT) == FR_GEOM_POLYHEDRON)
            r *= 1.7320509f;
    }
    const float scale = fmaxf(fmaxf(fabsf(p.c.x), fabsf(p.c.y)), fabsf(p.c.z)) + r;
    r = r * (1.0f + 1e-5f) + 2e-4f * scale + 2e-5f;
    bound[s] = make_float4(p.c.x, p.c.y, p.c.z, p.regular && r < INF ? -r : -INF);
}

}  // namespace

// Camera rays per pixel, and in all, from which building the lists pays (16 samples of a 200k-sphere
// frame at 1024x768: lists 0.2 ms, camera pass 0.83 -> 0.49 ms; a few million rays take less than
// the walk of the slowest tile).
constexpr uint32_t LIST_MIN_SAMPLES = 16;
constexpr uint64_t LIST_MIN_RAYS = 3u << 20;
// Widest beam, in mean primitive radii: with 15 entries a beam as wide as the spheres leaves a
// few percent of its rays to their own walks, one twice as wide a fifth, and its tiles span many
// cells (313k spheres at 186x97 with a lens, beams of several radii: 0.39 ms without lists, 1.79 ms
// with them; no frame of 150 drawn ones with beams below this was slower by more than 1%).
constexpr double LIST_WIDEST = 0.6;
// The same for the other types, per cell that a ray crosses between two of their boxes: a list then
// also holds what lies in the cells of what it meets (parts_cell_test), the more the closer
// together the boxes are, no sphere's solid inside ends it, and a box holds less of a cylinder than
// of a polyhedron or a mesh.  Scenes of several types take the harmonic mean over their primitives,
// and few rays, over which the lists' own time counts for more, the fourth root of their number
// less.  Preview at 1000x700 against no lists: 20k cubes at 0.3 per unit volume (0.57 cells), beams
// of 0.087, 0.90x; 500 of them (0.025) 1.45x; 5k at 1.0 (0.25 cells, 0.037) 0.94x; a crystal at 0.24
// (0.65 cells, 0.068) 1.23x.  Cylinders at 0.3 (1.7 cells) 0.044 1.76x and 0.15 0.89x; meshes 0.044
// 1.41x and 0.15 1.05x, at 1.0 (0.77 cells) 0.064 1.17x.  Spheres and bonds (2.9 cells) 0.2 1.20x; the
// mixed scene (five in seven are spheres, 1.8 cells) in a Path image of 118M rays, 0.35, 1.15x.
constexpr double LIST_WIDEST_SOLIDS = 0.1;
constexpr double LIST_WIDEST_CYLINDERS = 0.055;
constexpr double LIST_WIDEST_PARTS = 0.12;  // (cubes at 0.05, 1.9 cells, 0.16: 0.93x)
constexpr double LIST_WIDEST_RAYS = 1 << 24;
// Share of the references (1 in so many) that may be odd: nothing is known of how near one can be
// hit, so every ray of the beam tests it, and a list of 15 of them is complete nowhere.  Preview of
// 5000 primitives at 1000x700, cubes with quaternions of norm 0.95 among cubes: 8% of them 6.8 ms
// with lists and 8.0 without, 30% 7.8 and 7.8, all 11.7 and 7.3; 20000 of a third that density, 8%
// 8.1 and 8.4, 15% 8.4 and 8.3, 30% 9.0 and 8.2.
constexpr uint32_t LIST_ODD_SHARE = 8;

bool lists_possible(const FrameParams& P)
{
    return P.scene.grid.n_cells != 0;
}

bool lists_pay(const FrameParams& P, uint32_t samples)
{
    if (samples < LIST_MIN_SAMPLES || uint64_t(P.w) * P.h * samples < LIST_MIN_RAYS)
        return false;
    const GridDev& G = P.scene.grid;
    if (flat_layer(G))
        return false;  // a camera ray crosses only a cell or two of a flat layer
    if (uint64_t(G.n_odd) * LIST_ODD_SHARE > G.n_refs)
        return false;
    // the beam's radius in the middle of the grid: one pixel, and the lens away from the focus
    const CamK& k = P.cam;
    double rho = std::fabs(double(k.focal_h)) / k.height;
    if (k.model != 0) {
        const double c[3] = {0.5 * (G.lox + G.hix) - k.p.x, 0.5 * (G.loy + G.hiy) - k.p.y,
                             0.5 * (G.loz + G.hiz) - k.p.z};
        const double s = std::sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]) /
                         std::fabs(double(k.focal_d));
        const double e[3] = {G.hix - G.lox, G.hiy - G.loy, G.hiz - G.loz};
        const double half = 0.25 * std::sqrt(e[0] * e[0] + e[1] * e[1] + e[2] * e[2]) /
                            std::fabs(double(k.focal_d));
        rho = rho * s + 0.5 * std::fabs(double(k.aperture)) * std::max(std::fabs(1.0 - s), half);
    }
    double widest = G.list_widest;
    if (G.parts)
        widest = std::min(LIST_WIDEST, widest * std::pow(double(P.w) * P.h * samples /
                                                             LIST_WIDEST_RAYS, 0.25));
    return rho <= widest * G.mean_radius;
}

float list_widest(const uint64_t (&of_type)[5], float free_cells)
{
    double n = 0.0, inverse = 0.0;
    for (int type = 0; type < 5; ++type) {
        const bool solid = type == FR_GEOM_POLYHEDRON || type == FR_GEOM_MESH;
        const double widest =
            type == FR_GEOM_SPHERE
                ? LIST_WIDEST
                : std::min(LIST_WIDEST_PARTS, double(free_cells) * (solid ? LIST_WIDEST_SOLIDS
                                                                          : LIST_WIDEST_CYLINDERS));
        n += double(of_type[type]);
        if (of_type[type])
            inverse += of_type[type] / std::max(widest, 1e-6);
    }
    return float(n > 0.0 ? n / inverse : LIST_WIDEST);
}

void launch_part_bounds(const SceneDev& sc, uint32_t n, float4* bound, cudaStream_t st)
{
    if (n)
        k_part_bounds<<<(n + 255) / 256, 256, 0, st>>>(sc, n, bound);
}

size_t pixel_list_words(const FrameParams& P)
{
    return size_t(LIST_WORDS) * P.w * P.h;
}

void launch_pixel_lists(const FrameParams& P, uint2* lists, cudaStream_t st)
{
    const uint32_t tiles = ((P.w + 7u) >> 3) * ((P.h + 3u) >> 2);
    const uint32_t blocks = (tiles + 3u) / 4u;
    if (P.scene.grid.parts)
        k_pixel_lists_grid<true><<<blocks, 128, 0, st>>>(P, lists);
    else
        k_pixel_lists_grid<false><<<blocks, 128, 0, st>>>(P, lists);
}

}  // namespace fr
