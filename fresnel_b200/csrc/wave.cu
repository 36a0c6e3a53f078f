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
// What bounds k_wave_trace now: issue (72%), with 15 of 32 lanes active on average (a lane's
// iteration takes the test, the square root or the step, and not all need each).
#include "path_device.cuh"

namespace fr {

namespace {

// Idle lanes of a warp before they take new rays (one atomic per refill).
constexpr uint32_t WAVE_REFILL = 8;

// Walk of one ray through a sphere grid, one iteration at a time.  Each axis keeps the plane the
// ray leaves the current cell through as a whole number of cells (p), so that the distance to it is
// recomputed from the plane's position at every step, exactly as grid_walk_visit does.
struct SphereWalk {
    RayK ray;
    float tmax;
    uint32_t slot;       // reference of the closest hit so far
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
    __device__ __forceinline__ bool begin(const GridDev& G, V3 o, V3 d, TraceCount& tc)
    {
        ray = make_rayk(o, d);
        tmax = __int_as_float(0x7f800000);
        slot = MISS;
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
    // one iteration; false once the walk is over
    __device__ __forceinline__ bool step(const GridDev& G, float tnear, TraceCount& tc)
    {
        // exact tie with the closest hit so far: the lower sphere index wins (one geometry)
        const auto tie = [&](uint32_t r) {
            return slot != MISS && __ldg(G.ref_prim + r) < __ldg(G.ref_prim + slot);
        };
        if (k < end) {
            const bool two = k + 1u < end;
            const float4 q0 = ldg4(G.ref_sphere + k);
            const float4 q1 = ldg4(G.ref_sphere + (two ? k + 1u : k));
            // sphere_t of both, up to its square root: most lines miss, and of the spheres they
            // meet half lie behind (b < 0 and |b| above the root by more than its rounding, so
            // that both distances are negative); the rest is one section for either sphere, which
            // a warp enters once per iteration (a second time where a lane needs both)
            const V3 v0 = v3(q0.x, q0.y, q0.z) - ray.o, v1 = v3(q1.x, q1.y, q1.z) - ray.o;
            const float b0 = dot(v0, ray.d), b1 = dot(v1, ray.d);
            const float s0 = b0 * b0, s1 = b1 * b1;
            const float d0 = s0 - dot(v0, v0) + q0.w * q0.w, d1 = s1 - dot(v1, v1) + q1.w * q1.w;
            bool c0 = !(d0 < 0) && !(b0 < 0.0f && d0 < 0.999998f * s0);
            bool c1 = two && !(d1 < 0) && !(b1 < 0.0f && d1 < 0.999998f * s1);
            while (c0 || c1) {
                const float b = c0 ? b0 : b1, root = sqrtf(c0 ? d0 : d1);
                const uint32_t r = c0 ? k : k + 1u;
                if (c0)
                    c0 = false;
                else
                    c1 = false;
                float t = b - root;
                if (!(t > SPHERE_EPS))
                    t = b + root;
                if (t > SPHERE_EPS && tnear < t && (t < tmax || (t == tmax && tie(r)))) {
                    tmax = t;
                    slot = r;
                }
            }
            k += 2u;
        }
        if (k >= end) {
            if (tmax <= t_cell || !more)
                return false;
            k = nk;
            end = nend;
            look_ahead(G);
            tc.box += 1;
            tc.prim += end - k;
        }
        return true;
    }
    __device__ __forceinline__ uint2 hit(const GridDev& G) const
    {
        return slot == MISS ? make_uint2(MISS, 0u) : make_uint2(G.geom, __ldg(G.ref_prim + slot));
    }
};

template <class Walk>
__global__ void __launch_bounds__(256, 4) k_wave_trace(FrameParams P, PathState S, int q)
{
    const uint32_t count = S.ctr[q];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        S.ctr[q ^ 1] = 0;  // consumed by the pass that filled q
        atomicAdd(P.stats + 0, (unsigned long long)count);
    }
    const float4* rec_o = S.rec_o[q];
    const float4* rec_d = S.rec_d[q];
    const GridDev& G = P.scene.grid;
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
                    active = W.begin(G, xyz(ld_cs(rec_o + i)), xyz(ld_cs(rec_d + i)), tc);
                    if (!active)
                        st_cs(S.hit + i, make_uint2(MISS, 0u));
                }
            }
        } else if (idle == 0xffffffffu) {
            break;
        }
#pragma unroll 1
        for (int r = 0; r < 3; ++r) {
            if (active && !W.step(G, PATH_TNEAR, tc)) {
                st_cs(S.hit + i, W.hit(G));
                active = false;
            }
        }
    }
    flush_counts(tc, P.stats + 3);
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
    flush_counts(tc, P.stats + 3);
}

template <class K> int fill(K kernel, int num_sms)
{
    int n = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, 256, 0);
    return num_sms * (n > 0 ? n : 1);
}

}  // namespace

void wave_launch_shape(int num_sms, LaunchShape& s)
{
    for (int k = 0; k < 3; ++k) {
        s.trace_grid[k] = fill(k_wave_trace<SphereWalk>, num_sms);
        s.shade_rec_grid[k] = fill(k_wave_shade, num_sms);
        s.tail_rec_grid[k] = fill(k_wave_tail<MASK_GRID>, num_sms);
    }
}

void launch_wave_trace(const FrameParams& P, const PathState& S, int q, const LaunchShape& shape,
                       cudaStream_t st)
{
    k_wave_trace<SphereWalk><<<shape.trace_grid[0], 256, 0, st>>>(P, S, q);
}

void launch_wave_shade(const FrameParams& P, const PathState& S, int q, const LaunchShape& shape,
                       cudaStream_t st)
{
    k_wave_shade<<<shape.shade_rec_grid[0], 256, 0, st>>>(P, S, q);
}

void launch_wave_tail(const FrameParams& P, const PathState& S, int q, const LaunchShape& shape,
                      cudaStream_t st)
{
    k_wave_tail<MASK_GRID><<<shape.tail_rec_grid[0], 256, 0, st>>>(P, S, q);
}

}  // namespace fr
