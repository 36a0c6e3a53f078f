// beam.cuh -- per-pixel lists of the primitives a pixel's camera rays can meet.
//
// The camera rays of one pixel (its anti-aliasing or Monte Carlo samples) form a thin beam: all of
// them meet the same few primitives.  k_pixel_lists_grid (lists.cu) walks the acceleration structure
// once per beam and stores, per pixel, the primitives some ray of the beam may hit, nearest first,
// and a depth up to which that list is complete; list_hit then finds a sample's closest hit by
// testing the listed primitives alone, with the tests and the acceptance rule of the structure's
// own walk, instead of walking the structure for every sample.
//
// A list answers a ray only where its answer is provably the walk's:
//   * every primitive a walk of the ray would test and could accept closer than `complete` is
//     listed (the beam is widened by the jitter, the lens, and the rounding of the float tests);
//   * the closest listed hit lies nearer than `complete` and its point lies inside the primitive's
//     own bounding box by more than the walk's rounding, so that the walk, which tests every
//     primitive whose box the ray enters before its closest hit, tests this one too; and the
//     list holds every primitive that the walk may test before it ends (parts_cell_test).
// Any other ray takes the walk itself (list_hit returns false), so images are identical with and
// without lists.
#ifndef FR_BEAM_CUH
#define FR_BEAM_CUH

#include "render.hpp"

namespace fr {

// A pixel's list: LIST_WORDS uint2; word 0 is (entries, bits of the distance up to which the list
// answers: it is complete, or every ray hit, nearer than that), the others (slot, bits of the nearest
// distance a ray can be hit at: over parts, of the cells of any but spheres).  Slots number the
// grid's references.  128 bytes: one line per pixel.
constexpr uint32_t LIST_WORDS = 16;
constexpr uint32_t LIST_MAX = LIST_WORDS - 1;

// Widening of a sphere's squared radius, per squared distance: the float sphere test evaluates
// b*b - |v|^2 + r*r with errors of up to about 20 half-ulps of |v|^2 (the direction's norm 9, b*b
// 7, |v|^2 3), so it can accept a ray that passes outside the sphere by that much.
constexpr float SPHERE_SLACK = 1.25e-6f;

// Whether the closest hit h of a listed primitive, at distance t, lies inside that primitive's
// bounding box by more than the rounding of a walk's cell boundaries.
template <uint32_t MASK>
__device__ __forceinline__ bool hit_inside_box(const SceneDev& sc, const Hit& h, V3 o, V3 d,
                                               float t)
{
    const V3 x = o + d * t;
    const float m = 1e-6f * (t + fmaxf(fmaxf(fabsf(o.x), fabsf(o.y)), fabsf(o.z)));
    const GeomDev& g = sc.geoms[h.geom];
    auto in3 = [&](V3 c, float r) {
        return fmaxf(fmaxf(fabsf(x.x - c.x), fabsf(x.y - c.y)), fabsf(x.z - c.z)) <= r - m;
    };
    if constexpr ((MASK & MASK_ALL) == 0u) {
        return in3(load3(g.position, h.prim), __ldg(g.radius + h.prim));
    } else {
        if (g.type == FR_GEOM_SPHERE)
            return in3(load3(g.position, h.prim), __ldg(g.radius + h.prim));
        if (g.type == FR_GEOM_CYLINDER) {
            const V3 a = load3(g.points, 2 * h.prim), b = load3(g.points, 2 * h.prim + 1);
            const float r = __ldg(g.radius + h.prim) - m;
            return x.x >= fminf(a.x, b.x) - r && x.x <= fmaxf(a.x, b.x) + r &&
                   x.y >= fminf(a.y, b.y) - r && x.y <= fmaxf(a.y, b.y) + r &&
                   x.z >= fminf(a.z, b.z) - r && x.z <= fmaxf(a.z, b.z) + r;
        }
        if (g.type == FR_GEOM_POLYHEDRON)
            return in3(load3(g.position, h.prim), g.bound_radius);
        if (g.type == FR_GEOM_POLYGON) {
            const float r = g.bound_radius - m;
            return fabsf(x.x - __ldg(g.position + 2 * size_t(h.prim))) <= r &&
                   fabsf(x.y - __ldg(g.position + 2 * size_t(h.prim) + 1)) <= r;
        }
        // a mesh's triangle (flat: the point may lie off it by the rounding of t)
        const uint32_t inst = h.prim / g.n_faces, face = h.prim - inst * g.n_faces;
        const V3 pos = load3(g.position, inst);
        const Qt q = loadq(g.orientation, inst);
        V3 lo, hi;
        for (uint32_t k = 0; k < 3; ++k) {
            const V3 v = rotate(q, load3(g.vertices, 3 * face + k)) + pos;
            lo = k ? v3(fminf(lo.x, v.x), fminf(lo.y, v.y), fminf(lo.z, v.z)) : v;
            hi = k ? v3(fmaxf(hi.x, v.x), fmaxf(hi.y, v.y), fmaxf(hi.z, v.z)) : v;
        }
        return x.x >= lo.x - m && x.x <= hi.x + m && x.y >= lo.y - m && x.y <= hi.y + m &&
               x.z >= lo.z - m && x.z <= hi.z + m;
    }
}

// Closest hit of the ray (o, d) from its pixel's list; false when the list cannot answer it.
template <uint32_t MASK>
__device__ __forceinline__ bool list_hit(const FrameParams& P, const uint2* list, V3 o, V3 d,
                                         float tnear, TraceCount& tc, Hit& h)
{
    const SceneDev& sc = P.scene;
    const uint2 head = __ldg(list);
    const float complete = __uint_as_float(head.y);
    float tmax = __int_as_float(0x7f800000);  // +inf
    h.geom = MISS;
    h.prim = 0;
    if constexpr (MASK == MASK_GRID) {
        const GridDev& G = sc.grid;
        uint32_t slot = MISS;
        for (uint32_t e = 1; e <= head.x; ++e) {
            const uint2 c = __ldg(list + e);
            if (tmax < __uint_as_float(c.y))
                break;
            ++tc.prim;
            const float4 q = ldg4(G.ref_sphere + c.x);
            float t;
            if (sphere_t(o, d, v3(q.x, q.y, q.z), q.w, t) && (tnear < t) &&
                ((t < tmax) || (t == tmax && slot != MISS &&
                                __ldg(G.ref_prim + c.x) < __ldg(G.ref_prim + slot)))) {
                tmax = t;
                slot = c.x;
            }
        }
        if (slot == MISS)
            return complete == __int_as_float(0x7f800000);
        h.geom = G.geom;
        h.prim = __ldg(G.ref_prim + slot);
    } else {
        const RayK ray = make_rayk(o, d);
        uint32_t hg = MISS, hp = 0, last_g = MISS, last_p = 0;
        for (uint32_t e = 1; e <= head.x; ++e) {
            const uint2 c = __ldg(list + e);
            if (tmax < __uint_as_float(c.y))
                break;
            parts_cell_test<MASK & MASK_ALL, true>(sc, ray, c.x, c.x + 1u, tnear, tmax, hg, hp,
                                                   last_g, last_p, tc);
        }
        if (hg == MISS)
            return complete == __int_as_float(0x7f800000);
        h.geom = hg;
        h.prim = hp;
    }
    return tmax < complete && hit_inside_box<MASK>(sc, h, o, d, tmax);
}

// The list of pixel (i, j).
__device__ __forceinline__ const uint2* pixel_list(const FrameParams& P, uint32_t i, uint32_t j)
{
    return P.lists + size_t(LIST_WORDS) * (size_t(j) * P.w + i);
}

// No ray of the pixel meets anything.
__device__ __forceinline__ bool list_empty(const uint2* list)
{
    const uint2 head = __ldg(list);
    return head.x == 0u && __uint_as_float(head.y) == __int_as_float(0x7f800000);
}

}  // namespace fr

#endif
