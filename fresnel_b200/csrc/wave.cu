// wave.cu -- extension rays over packed queues: tracing and shading in passes of their own.
//
// The fused bounce kernels (render.cu) trace a ray and shade its hit in one thread, so a warp walks
// as long as its longest ray: with 32 rays the longest walk is some four times the mean, and
// the walk ran with 7 of 32 lanes active.  Here
//   k_wave_trace  walks the rays of a queue with per-lane refill: every iteration of a lane tests
//                 up to two spheres of its current cell and, once those are done, steps to the
//                 next cell; a lane whose ray is finished stores the hit and, once WAVE_REFILL
//                 lanes of its warp are idle, takes the next ray of the queue;
//   k_wave_shade  shades the hits in queue order and appends the continuing paths to the other
//                 queue;
//   k_wave_tail   follows the last paths to their end, one path per lane, state in registers.
// A queue holds whole path records (48 bytes: ray, throughput, slot, depth, light sample), written
// and read in order, instead of slot numbers that lead to scattered state: the first shading pass
// of a 200k-sphere frame moves 334 MB instead of 914 MB through HBM (0.17 against 0.28 ms).
// Against the fused bounce and tail kernels: 1M spheres 1080p, 256 samples 54.4 -> 44.4 ms a frame;
// 1000 spheres with 32 light samples 50.8 -> 34.5 ms; 200k spheres, 16 samples 2.87 -> 2.72 ms.
// The mixed scene of 280k primitives, 1280x720, 128 samples: 51.4 -> 31.3 ms.
// What bounds k_wave_trace now: issue (62-72%), with 13 to 15 of 32 lanes active on average (a lane's
// iteration takes the test, the square root or the step, and not all need each); over parts 7 to 8
// lanes at 66%.
#include "path_device.cuh"

namespace fr {

namespace {

// Idle lanes of a warp before they take new rays (one atomic per refill).
constexpr uint32_t WAVE_REFILL = 8;

// Walk of one ray through a grid, one iteration at a time.  Each axis keeps the plane the ray
// leaves the current cell through as a whole number of cells (p), so that the distance to it is
// recomputed from the plane's position at every step, exactly as grid_walk_visit does.
struct CellWalk {
    RayK ray;
    float tmax;          // distance of the closest hit so far
    float px, py, pz;    // exit planes of the cell last stepped to (the one after the current)
    float tx, ty, tz;    // distances to them
    float t_out;         // distance at which the ray leaves the grid
    float t_cell;        // exit distance of the current cell
    bool more;           // there is a cell after it
    uint32_t id;         // that cell
    uint32_t k, end;     // references of the current cell still to test
    uint32_t nk, nend;   // references of the cell after it

    // steps past the current cell and loads the reference range of the cell there, which the
    // tests of the current cell's spheres then overlap
    __device__ __forceinline__ void look_ahead(const GridDev& G)
    {
        const bool ux = ray.inv.x >= 0.0f, uy = ray.inv.y >= 0.0f, uz = ray.inv.z >= 0.0f;
        t_cell = fminf(tx, fminf(ty, tz));
        const bool sx = tx <= ty && tx <= tz, sy = !sx && ty <= tz, sz = !sx && !sy;
        const float lx = ux ? float(G.nx) : 0.0f, ly = uy ? float(G.ny) : 0.0f,
                    lz = uz ? float(G.nz) : 0.0f;
        more = t_cell < t_out && !((sx && px == lx) || (sy && py == ly) || (sz && pz == lz));
        if (sx) {
            px += ux ? 1.0f : -1.0f;
            id += ux ? 1u : ~0u;
        }
        if (sy) {
            py += uy ? 1.0f : -1.0f;
            id += uy ? G.nx : 0u - G.nx;
        }
        if (sz) {
            pz += uz ? 1.0f : -1.0f;
            id += uz ? G.nx * G.ny : 0u - G.nx * G.ny;
        }
        if (more) {
            nk = __ldg(G.cell_start + id);
            nend = __ldg(G.cell_start + id + 1);
        }
        tx = fmaf(fmaf(px, G.hx, G.lox), ray.inv.x, ray.oinv.x);
        ty = fmaf(fmaf(py, G.hy, G.loy), ray.inv.y, ray.oinv.y);
        tz = fmaf(fmaf(pz, G.hz, G.loz), ray.inv.z, ray.oinv.z);
    }
    // false: the ray misses the grid
    __device__ __forceinline__ bool begin_cells(const GridDev& G, V3 o, V3 d, TraceCount& tc)
    {
        ray = make_rayk(o, d);
        tmax = __int_as_float(0x7f800000);
        GridWalk W;
        if (!grid_walk_begin(G, ray, W))
            return false;
        px = float(W.ix + (ray.inv.x >= 0.0f ? 1 : 0));
        py = float(W.iy + (ray.inv.y >= 0.0f ? 1 : 0));
        pz = float(W.iz + (ray.inv.z >= 0.0f ? 1 : 0));
        tx = W.tnx;
        ty = W.tny;
        tz = W.tnz;
        t_out = W.t_out;
        id = grid_cell_id(G, W.ix, W.iy, W.iz);
        k = W.first;
        end = W.last;
        look_ahead(G);
        tc.box += 1;
        tc.prim += end - k;
        return true;
    }
    // the next cell, once every reference of the current one is tested; false when the walk is over
    __device__ __forceinline__ bool next_cell(const GridDev& G, TraceCount& tc)
    {
        if (tmax <= t_cell || !more)
            return false;
        k = nk;
        end = nend;
        look_ahead(G);
        tc.box += 1;
        tc.prim += end - k;
        return true;
    }
};

// The line distance test of sphere_t for the spheres (c, r) of two references, up to its square
// root: most lines miss, and of the spheres they meet half lie behind (b < 0 and |b| above the
// root by more than its rounding, so that both distances are negative).
struct LineTest {
    float b, d;  // projection of the centre, discriminant
    bool c;      // the sphere may be hit
    __device__ __forceinline__ LineTest(const RayK& ray, V3 centre, float r)
    {
        const V3 v = centre - ray.o;
        b = dot(v, ray.d);
        const float s = b * b;
        d = s - dot(v, v) + r * r;
        c = !(d < 0) && !(b < 0.0f && d < 0.999998f * s);
    }
    // sphere_t's distance; false when it has none
    __device__ __forceinline__ static bool distance(float b, float d, float& t)
    {
        const float root = sqrtf(d);
        t = b - root;
        if (!(t > SPHERE_EPS))
            t = b + root;
        return t > SPHERE_EPS;
    }
};

struct SphereWalk : CellWalk {
    static constexpr bool DEFERS = false;
    uint32_t slot;  // reference of the closest hit so far

    __device__ __forceinline__ bool begin(const FrameParams& P, V3 o, V3 d, TraceCount& tc)
    {
        slot = MISS;
        return begin_cells(P.scene.grid, o, d, tc);
    }
    // one iteration; false once the walk is over
    __device__ __forceinline__ bool step(const FrameParams& P, float tnear, TraceCount& tc)
    {
        const GridDev& G = P.scene.grid;
        // exact tie with the closest hit so far: the lower sphere index wins (one geometry)
        const auto tie = [&](uint32_t r) {
            return slot != MISS && __ldg(G.ref_prim + r) < __ldg(G.ref_prim + slot);
        };
        if (k < end) {
            const bool two = k + 1u < end;
            const float4 q0 = ldg4(G.ref_sphere + k);
            const float4 q1 = ldg4(G.ref_sphere + (two ? k + 1u : k));
            LineTest l0(ray, v3(q0.x, q0.y, q0.z), q0.w), l1(ray, v3(q1.x, q1.y, q1.z), q1.w);
            l1.c = l1.c && two;
            // one section for either sphere, which a warp enters once per iteration (a second
            // time where a lane needs both)
            while (l0.c || l1.c) {
                float t;
                const bool hit = LineTest::distance(l0.c ? l0.b : l1.b, l0.c ? l0.d : l1.d, t);
                const uint32_t r = l0.c ? k : k + 1u;
                if (l0.c)
                    l0.c = false;
                else
                    l1.c = false;
                if (hit && tnear < t && (t < tmax || (t == tmax && tie(r)))) {
                    tmax = t;
                    slot = r;
                }
            }
            k += 2u;
        }
        return k < end || next_cell(G, tc);
    }
    __device__ __forceinline__ uint2 hit(const FrameParams& P) const
    {
        const GridDev& G = P.scene.grid;
        return slot == MISS ? make_uint2(MISS, 0u) : make_uint2(G.geom, __ldg(G.ref_prim + slot));
    }
};

// Walk through a grid over parts.  Every reference is first tested by a sphere (GridDev::ref_bound:
// the sphere itself, or one around the primitive, its radius negative), two references per
// iteration as above; a primitive of another type whose sphere the ray meets waits (pend) until
// enough lanes of the warp hold one, and then its own test, with its own box test before it,
// runs for all of them together (parts_cell_test).
template <uint32_t TYPES>
struct PartsWalk : CellWalk {
    static constexpr bool DEFERS = true;
    uint32_t hg, hp;          // closest hit so far
    uint32_t last_g, last_p;  // see parts_cell_test
    uint32_t pend;            // reference whose test waits (MISS: none)

    __device__ __forceinline__ bool begin(const FrameParams& P, V3 o, V3 d, TraceCount& tc)
    {
        hg = last_g = pend = MISS;
        hp = last_p = 0;
        return begin_cells(P.scene.grid, o, d, tc);
    }
    // Sphere test of reference r: true for a primitive of another type to test.
    __device__ __forceinline__ LineTest line(const FrameParams& P, uint32_t r, float& radius) const
    {
        const float4 q = ldg4(P.scene.grid.ref_bound + r);
        const V3 c = v3(q.x, q.y, q.z);
        radius = q.w;
        if (q.w < 0.0f) {
            // widened by what the primitive's own test may be off by
            const V3 v = c - ray.o;
            const float far = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fabsf(v.z));
            radius = fmaf(far, PART_SLACK, -q.w);
        }
        LineTest l(ray, c, radius);
        if (q.w < 0.0f) {
            if (l.b - radius > tmax)
                l.c = false;  // wholly beyond the closest hit
            radius = -1.0f;
        }
        return l;
    }
    __device__ __forceinline__ bool step(const FrameParams& P, float tnear, TraceCount& tc)
    {
        const SceneDev& sc = P.scene;
        if (k < end) {
            const bool two = k + 1u < end;
            float r0, r1;
            LineTest l0 = line(P, k, r0), l1 = line(P, two ? k + 1u : k, r1);
            l1.c = l1.c && two;
            while (l0.c || l1.c) {
                const bool first = l0.c;
                const uint32_t r = first ? k : k + 1u;
                if ((first ? r0 : r1) < 0.0f) {
                    pend = r;
                    k = r + 1u;  // the references after it wait with it
                    return true;
                }
                float t;
                const bool hit = LineTest::distance(first ? l0.b : l1.b, first ? l0.d : l1.d, t);
                if (first)
                    l0.c = false;
                else
                    l1.c = false;
                if (hit && tnear < t && t <= tmax) {
                    const uint32_t g = __ldg(sc.leaf_geom + r) & ((1u << PART_TYPE_SHIFT) - 1u);
                    const uint32_t p = __ldg(sc.order + r);
                    if (t < tmax || tie_wins(g, hg, [&]() { return p; }, [&]() { return hp; })) {
                        tmax = t;
                        hg = g;
                        hp = p;
                    }
                }
            }
            k += 2u;
        }
        return k < end || next_cell(sc.grid, tc);
    }
    // the waiting primitive's own test
    __device__ __forceinline__ void resolve(const FrameParams& P, float tnear)
    {
        TraceCount none;  // counted with its cell
        parts_cell_test<TYPES>(P.scene, ray, pend, pend + 1u, tnear, tmax, hg, hp, last_g, last_p,
                               none);
        pend = MISS;
    }
    __device__ __forceinline__ uint2 hit(const FrameParams&) const
    {
        return make_uint2(hg, hg == MISS ? 0u : hp);
    }
};

// Lanes of a warp with a waiting primitive before their tests run.
constexpr uint32_t WAVE_PENDING = 8;  // (the primitives' own tests ran with some 2 lanes of a warp
                                     // in the fused kernels' walk)

template <class Walk>
__global__ void __launch_bounds__(256, Walk::DEFERS ? 3 : 4) k_wave_trace(FrameParams P, PathState S, int q)
{
    const uint32_t count = S.ctr[q];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        S.ctr[q ^ 1] = 0;  // consumed by the pass that filled q
        atomicAdd(P.stats + 0, (unsigned long long)count);
    }
    const float4* rec_o = S.rec_o[q];
    const float4* rec_d = S.rec_d[q];
    const uint32_t lane = lane_id();
    const uint32_t below = (1u << lane) - 1u;
    TraceCount tc;
    Walk W;
    bool active = false, exhausted = count == 0u;
    uint32_t i = 0;
    while (true) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !active);
        if (!exhausted && (__popc(idle) >= int(WAVE_REFILL))) {
            const uint32_t n = uint32_t(__popc(idle));
            uint32_t base = 0;
            if (lane == 0)
                base = atomicAdd(S.ctr + 2, n);
            base = __shfl_sync(0xffffffffu, base, 0);
            exhausted = base + n >= count;
            if (!active) {
                i = base + uint32_t(__popc(idle & below));
                if (i < count) {
                    active = W.begin(P, xyz(ld_cs(rec_o + i)), xyz(ld_cs(rec_d + i)), tc);
                    if (!active)
                        st_cs(S.hit + i, make_uint2(MISS, 0u));
                }
            }
        } else if (idle == 0xffffffffu) {
            break;
        }
#pragma unroll 1
        for (int r = 0; r < 3; ++r) {
            bool walks = active;
            if constexpr (Walk::DEFERS)
                walks = active && W.pend == MISS;
            if (walks && !W.step(P, PATH_TNEAR, tc)) {
                st_cs(S.hit + i, W.hit(P));
                active = false;
            }
        }
        if constexpr (Walk::DEFERS) {
            const bool waits = active && W.pend != MISS;
            const uint32_t n = uint32_t(__popc(__ballot_sync(0xffffffffu, waits)));
            if (n && (n >= WAVE_PENDING || !__any_sync(0xffffffffu, active && !waits)) && waits)
                W.resolve(P, PATH_TNEAR);
        }
    }
    flush_counts(tc, P.tests);
}

// The record i of queue q as a lane to shade (its hit still to be set).
__device__ __forceinline__ void load_record(const FrameParams& P, const PathState& S, int q,
                                            uint32_t i, ShadeLane& L)
{
    const float4 o = ld_cs(S.rec_o[q] + i), d = ld_cs(S.rec_d[q] + i), a = ld_cs(S.rec_a[q] + i);
    L.p = __float_as_uint(o.w);
    const PrimaryItem pi = primary_item(L.p, P.w, P.h, P.batch, P.tile_log2);
    L.pixel = pi.j * P.w + pi.i;
    L.n_samples = P.n_samples + pi.k;
    L.ls = __float_as_uint(a.w);
    L.s.depth = __float_as_uint(d.w);
    L.s.result = P.light_samples > 1u ? rgb3(ld_cs(S.result + L.p)) : c3(0.0f, 0.0f, 0.0f);
    L.s.att = rgb3(a);
    L.s.origin = v3(0, 0, 0);
    L.s.dir = v3(0, 0, 0);
    L.ph = make_uint2(0u, 0u);
    L.ro = xyz(o);
    L.rd = xyz(d);
    L.have_sf = false;
}

// Shades the hits of queue q, continuing paths into queue q ^ 1.  The lanes of a warp first take
// records (of the warp's share: groups of 32, warp w owning groups w, w + n_warps, ...) until
// most hold a hit, finishing those that missed on the way, and then shade their hits together;
// a slot's light samples that end at its primary vertex are shaded one after another by the
// same lane while the others take new records.
constexpr uint32_t SHADE_FULL = 24;  // lanes with a hit before a warp shades

__global__ void __launch_bounds__(256, 3) k_wave_shade(FrameParams P, PathState S, int q)
{
    if (blockIdx.x == 0 && threadIdx.x == 0)
        S.ctr[2] = 0;  // work counter of the trace that follows
    const uint32_t count = S.ctr[q];
    const uint32_t lane = lane_id();
    const uint32_t below = (1u << lane) - 1u;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t n_warps = (gridDim.x * blockDim.x) >> 5;
    uint32_t taken = 0;  // positions of the warp's share handed out so far (warp-uniform)
    bool busy = false;   // the lane holds a record whose next vertex is a hit
    ShadeLane L;
    while (true) {
        while (true) {
            const uint32_t idle = __ballot_sync(0xffffffffu, !busy);
            // groups are handed out in order: once a position lies past the end, all later do
            const bool work = (warp + (taken >> 5) * n_warps) * 32u < count;
            if (!work || __popc(idle) <= int(32u - SHADE_FULL))
                break;
            if (!busy) {
                const uint32_t k = taken + __popc(idle & below);
                const uint32_t i = (warp + (k >> 5) * n_warps) * 32u + (k & 31u);
                if (i < count) {
                    load_record(P, S, q, i, L);
                    L.h = ld_cs(S.hit + i);
                    busy = L.h.x != MISS || shade_miss(P, S, L);
                }
            }
            taken += __popc(idle);
        }
        if (!__any_sync(0xffffffffu, busy))
            break;
        bool push = false;
        if (busy) {
            const ShadeStep r = shade_step<true>(P, S, L);
            busy = r == STEP_RESTART;
            push = r == STEP_CONTINUE;
        }
        const uint32_t m = __ballot_sync(0xffffffffu, push);
        if (m) {
            uint32_t at = 0;
            if (lane == 0)
                at = atomicAdd(S.ctr + (q ^ 1), uint32_t(__popc(m)));
            at = __shfl_sync(0xffffffffu, at, 0);
            if (push)
                store_record(S, q ^ 1, at + __popc(m & below), L);
        }
    }
}

// The remaining bounces of the paths of queue q, each lane following one path at a time with its
// state in registers (a path longer than TAIL_MAX_DEPTH further bounces is cut and reported).
template <uint32_t MASK>
__global__ void __launch_bounds__(256, fused_blocks(MASK)) k_wave_tail(FrameParams P, PathState S,
                                                                       int q)
{
    const uint32_t count = S.ctr[q];
    const uint32_t lane = lane_id();
    const uint32_t below = (1u << lane) - 1u;
    TraceCount tc;
    bool active = false, exhausted = count == 0u;
    uint32_t guard = 0;
    unsigned long long rays = 0;
    ShadeLane L;
    while (true) {
        const uint32_t idle = __ballot_sync(0xffffffffu, !active);
        if (idle && !exhausted) {
            const uint32_t n = uint32_t(__popc(idle));
            uint32_t base = 0;
            if (lane == 0)
                base = atomicAdd(S.ctr + 2, n);
            base = __shfl_sync(0xffffffffu, base, 0);
            exhausted = base + n >= count;
            if (!active) {
                const uint32_t i = base + uint32_t(__popc(idle & below));
                if (i < count) {
                    load_record(P, S, q, i, L);
                    active = true;
                    guard = TAIL_MAX_DEPTH;
                }
            }
        }
        if (__ballot_sync(0xffffffffu, active) == 0u)
            break;
        if (active) {
            ++rays;
            const Hit h = trace_closest<4, MASK>(P.scene, L.ro, L.rd, PATH_TNEAR, tc);
            L.h = make_uint2(h.geom, h.prim);
            L.have_sf = false;
            if (!shade_run<true>(P, S, L)) {
                active = false;
            } else if (--guard == 0u) {
                atomicOr(P.scene.status, ERR_ITERATION_CAP);
                active = false;
            } else {
                L.ro = L.s.origin;
                L.rd = L.s.dir;
            }
        }
    }
    for (int off = 16; off > 0; off >>= 1)
        rays += __shfl_xor_sync(0xffffffffu, rays, off);
    if (lane == 0 && rays)
        atomicAdd(P.stats + 0, rays);
    flush_counts(tc, P.tests);
}

constexpr uint32_t NO_MESH = MASK_GRID_PARTS_NO_MESH & MASK_ALL;

template <class K> int fill(K kernel, int num_sms)
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, 0);
    return num_sms * (n > 0 ? n : 1);
}

}  // namespace

void wave_launch_shape(int num_sms, LaunchShape& s)
{
    s.trace_grid[0] = fill(k_wave_trace<SphereWalk>, num_sms);
    s.trace_grid[1] = fill(k_wave_trace<PartsWalk<MASK_ALL>>, num_sms);
    s.trace_grid[2] = fill(k_wave_trace<PartsWalk<NO_MESH>>, num_sms);
    s.shade_rec_grid = fill(k_wave_shade, num_sms);
    s.tail_rec_grid[0] = fill(k_wave_tail<MASK_GRID>, num_sms);
    s.tail_rec_grid[1] = fill(k_wave_tail<MASK_GRID_PARTS>, num_sms);
    s.tail_rec_grid[2] = fill(k_wave_tail<MASK_GRID_PARTS_NO_MESH>, num_sms);
}

// 0: a sphere grid, 1: a grid over parts, 2: one without meshes.
static int wave_kind(const FrameParams& P)
{
    return !P.scene.grid.parts ? 0 : (P.type_mask & (1u << FR_GEOM_MESH)) ? 1 : 2;
}

void launch_wave_trace(const FrameParams& P, const PathState& S, int q, const LaunchShape& shape,
                       cudaStream_t st)
{
    const int gk = wave_kind(P);
    auto k = gk == 0   ? k_wave_trace<SphereWalk>
             : gk == 1 ? k_wave_trace<PartsWalk<MASK_ALL>>
                       : k_wave_trace<PartsWalk<NO_MESH>>;
    k<<<shape.trace_grid[gk], 256, 0, st>>>(P, S, q);
}

void launch_wave_shade(const FrameParams& P, const PathState& S, int q, const LaunchShape& shape,
                       cudaStream_t st)
{
    k_wave_shade<<<shape.shade_rec_grid, 256, 0, st>>>(P, S, q);
}

void launch_wave_tail(const FrameParams& P, const PathState& S, int q, const LaunchShape& shape,
                      cudaStream_t st)
{
    const int gk = wave_kind(P);
    auto k = gk == 0   ? k_wave_tail<MASK_GRID>
             : gk == 1 ? k_wave_tail<MASK_GRID_PARTS>
                       : k_wave_tail<MASK_GRID_PARTS_NO_MESH>;
    k<<<shape.tail_rec_grid[gk], 256, 0, st>>>(P, S, q);
}

}  // namespace fr
