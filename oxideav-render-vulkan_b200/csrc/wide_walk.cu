// Wide traversal of the wavefront plans: rays walk the four-wide tree with
// conservative box tests, and a warp tests the triangles of all its rays
// together. The answers are the reference walk's, bit for bit.
//
// What bounded the walks before (walk.cuh, 1.05 M triangles, 1080p): the
// L1's load pipe (92% busy in an any-hit launch of this kernel that still
// read the 128-byte float nodes) and instruction issue at 10 active lanes of
// 32, since lanes at nodes and lanes at leaves took turns. So:
// * Nodes are 64 bytes, two 32-byte loads, with child boxes as bytes
//   (bvh4_build.cu, wide_nodes). Near and far planes are picked by the ray's
//   direction signs and each child's pair is one fma.rn.f32x2.
// * Inner children are numbered in sequence, so a node leaves at most one
//   stack entry behind: the first child's index and a mask. The first SS
//   entries are shared memory columns (one conflict-free access a warp).
// * Leaves that pass are noted in the lane's column; when FLUSH are noted (or
//   no lane has node work) the warp tests one (ray, triangle) pair per lane:
//   full warps whatever the rays' mix of nodes and leaves is.
// * A node step is about 190 instructions: the stored corner lets one fused
//   operation place a plane, an any-hit walk takes its next node straight from
//   the group of waiting siblings (nearest first gained it nothing).
// A 64-spp 1080p frame of that scene: closest hits 89.9 -> 44 ms, shadow rays
// 135.9 -> 70 ms (18 and 22 of 32 lanes active; now bound by issue: 71 and 73%
// of cycles issue). FLUSH of 24 to 48, 4 to 10 entries in shared
// memory, 2 to 8 steps between checks and 12 pending leaves were within 3%
// of each other or worse; 48 registers a thread (10 blocks) spilled and were
// 1.2 to 1.9x slower than 64.
//
// Why the result is the reference walk's although the order and the box
// test are not:
// * Every box that the exact test enters is entered here too. With u = 2^-24,
//   a plane's distance is within 0.006 byte steps (the bytes leave 1/32) and
//   3 u of itself, the exact test's within 2 u (and its far planes are taken
//   6 u too far): SLACK covers both. No term grows with the coordinates, so a
//   small object in a large scene is entered as exactly as by itself.
//   (Widening by 64 u of the largest coordinate, a frame of a 512 k-triangle
//   object of 1 unit above a ground of 10^4 units took 49 ms, of 10^5 units
//   2.4 s; now 7.0 and 7.2.)
// * A closest hit's distance limit T is compared with the entry on the ray's
//   dominant axis alone. The watertight test's distance is a weighted mean of
//   its vertices' distances on that axis, whatever the weights are, so it is
//   at least the box's entry there (but for some u of itself, less than the
//   2e-5 that T leaves): all triangles with t <= T are tested, in whatever
//   order the boxes come. On the other axes no such bound holds: where a
//   triangle's projection is thin against the rounding of its vertices, the
//   weights are noise and the hit lies anywhere in the triangle, also before
//   the ray enters its box. (Culling by the entry on all three axes took 10%
//   less time and could lose such a hit to one behind it. Projections of an
//   area below 1e-30, where products of the test underflow, are not covered.)
// * Any hit: the reference accepts a triangle when its leaf's exact box test
//   passes (a box passes whenever a box inside it does: checked on upload),
//   so an accepted triangle is checked against its leaf's exact box once.
// * Closest hit: T stays 2e-5 above the best distance and the second
//   smallest accepted distance is kept. Let the best hit be at t and the
//   exact entry distance of its leaf be e. The reference walk can miss it
//   only by culling the leaf against another accepted hit in [t, e], or
//   resolve an equal distance by its own order; neither exists when the
//   second distance is above max(t, e) (and e below T).
// A ray whose check fails (an exact tie on a shared edge, a leaf the exact
// test misses) is walked again with the reference's own walk, in place.
#include "kernels.cuh"
#include "walk.cuh"
#include "wavefront.cuh"

namespace oxd {

namespace {

constexpr uint32_t NT = WAVE_TRAVERSE_THREADS;
constexpr unsigned FULL = 0xffffffffu;
constexpr uint32_t LEAF_BIT = 0x80000000u;
constexpr uint32_t NOT_WALKED = 0xfffffffeu;  // for a hit: leave the ray to the reference's walk
constexpr uint32_t LEAFCAP = 8;   // leaves a lane may have pending
constexpr uint32_t SS = 6;        // stack entries a lane keeps in shared memory
constexpr uint32_t FLUSH = 32;    // pending leaves of a warp that start a pass of triangle tests
constexpr uint32_t MIN_RAYS = 4;  // rays of a warp, at least, when they are few
constexpr int STEPS = 4;          // node steps between checks
constexpr float SLACK = 1.0000012f;      // 1 + 20 u, on far planes
// Largest distance of an origin, in scene sizes (a frame of the 512 k-triangle
// object from 3e4 / 6e4 / 1e5 sizes away: 5.3 / 7.2 / 11.2 ms; left to the
// reference's walk from 1.5e5: 6.7).
constexpr float AWAY = 5.0e4f;
constexpr float LIMIT = 1.00002f;        // closest hit: distance limit over the best distance

// One warp's rays and pending work in shared memory.
template <bool EXT>
struct __align__(16) WarpMem {
    float4 o[32];       // origin, distance limit
    float4 shear[32];   // shear.xyz, kx | ky << 2 | kz << 4 | primary << 6
    unsigned long long best[EXT ? 32 : 1];  // closest: distance bits << 32 | slot
    uint32_t second[EXT ? 32 : 1];          // closest: second smallest accepted distance
    uint32_t found[EXT ? 1 : 32];           // any hit: an accepted slot
    uint32_t src[32];             // closest: path slot; any hit: entry of the shadow queue
    uint32_t leaf[LEAFCAP][32];
    uint32_t stack[SS][32];
    float stack_t[EXT ? SS : 1][32];
    uint8_t list[LEAFCAP * 32];   // pending leaves in lane order: lane | index in its column << 5
};

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("{.reg .b64 a, b, c, d;\n\tmov.b64 a, {%2, %3};\n\tmov.b64 b, {%4, %5};\n\tmov.b64 c, {%6, %7};\n\t"
        "fma.rn.f32x2 d, a, b, c;\n\tmov.b64 {%0, %1}, d;}"
        : "=f"(r.x), "=f"(r.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
    return r;
}

__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

struct u8x {
    uint32_t v[8];
};
// One 32-byte read-only load.
__device__ __forceinline__ u8x ld32(const void* p) {
    u8x r;
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]),
          "=r"(r.v[7])
        : "l"(p));
    return r;
}

// What a node step needs of a ray: its origin and reciprocal direction. With m
// the largest coordinate of the scene's box, what a step adds up is at most
// 600 m + |o| times a reciprocal, so reciprocals are cut to keep that finite
// (a zero component has 1e30). The cut only brings planes nearer: a near
// plane stays a lower bound, and a far one is still 0.025 steps of at least
// 2^-40 m away, which must be beyond the scene. False when that does not hold
// (coordinates beyond 1e17), and for origins so far away that SLACK of the
// distance is a good part of the scene: the ray is then left to the
// reference's walk.
struct NodeRay {
    float o[3], inv[3];
};

__device__ __forceinline__ bool node_ray(const Scene& s, const Ray& r, NodeRay& n) {
    const float4 lo = geomv(s, 0), hi = geomv(s, 1);
    const float m = max3(fmaxf(fabsf(lo.x), fabsf(hi.x)), fmaxf(fabsf(lo.y), fabsf(hi.y)),
                         fmaxf(fabsf(lo.z), fabsf(hi.z)));
    const float away = max3(fabsf(r.o.x), fabsf(r.o.y), fabsf(r.o.z)), reach = 600.0f * m + away;
    const float cut = 1.0e37f / reach, main = fabsf(r.shear.z);  // the dominant reciprocal
    const float iv[3] = {r.inv.x, r.inv.y, r.inv.z}, oo[3] = {r.o.x, r.o.y, r.o.z};
#pragma unroll
    for (int a = 0; a < 3; a++) {
        n.o[a] = oo[a];
        n.inv[a] = fminf(fmaxf(iv[a], -cut), cut);
    }
    return main >= 1.0e-9f && reach * main * reach <= 2.0e23f * m && away <= AWAY * m;
}

// Byte k of w as the float 32768 + byte.
__device__ __forceinline__ float plane(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x47000000u, 0x7504u | (uint32_t)k << 4));
}

// The reference's own walk for a ray whose check failed (rare).
__device__ __noinline__ bool reference_walk(const Scene* s, const Ray* r, float t_max, uint32_t path_seed,
                                            uint32_t ray_id, bool primary, bool any, uint32_t skip, Hit* h,
                                            uint32_t* mat, uint32_t* err) {
    Cnt cnt;
    Walk2<64> w;
    Sampler smp{0u, 0u, path_seed};
    if (!walk2_begin<false, 64>(*s, *r, t_max, w, cnt)) return false;
    while (!walk2_step<false, 64>(*s, *r, smp, ray_id, primary, any, skip, w, cnt, err)) {
    }
    *h = w.best;
    *mat = w.best_mat;
    return w.hit_any;
}

__device__ __forceinline__ float comp(f3 v, uint32_t k) { return k == 0u ? v.x : (k == 1u ? v.y : v.z); }

// The scene of the ray from entry `src` (a path slot, or an entry of the
// shadow queue).
template <bool EXT, bool BATCH>
__device__ __forceinline__ const Scene& ray_scene(const WaveArgs& a, uint32_t src) {
    return BATCH ? a.frames[a.st.frame[EXT ? src : a.q.sh_m[src].x]].s : a.s;
}

// Tests one (ray, triangle) pair and records an accepted hit.
template <bool EXT, bool BATCH>
__device__ __forceinline__ void test_pair(const WaveArgs& a, WarpMem<EXT>& M, uint32_t L, uint32_t slot) {
    if (!EXT && *(volatile uint32_t*)&M.found[L] != NONE) return;  // already occluded
    const Scene& s = ray_scene<EXT, BATCH>(a, M.src[L]);
    const float4 ro = M.o[L], rs = M.shear[L];
    const uint32_t kk = __float_as_uint(rs.w);
    const uint64_t tb = tri_base(s, slot);
    if ((uint64_t)slot >= s.slot_count || tb + 3u > s.geom_vec4) {
        atomicOr(a.err, 2u);
        return;
    }
    const float4 q0 = __ldg(s.geom + tb), q1 = __ldg(s.geom + tb + 1), q2 = __ldg(s.geom + tb + 2);
    // intersect() without its barycentrics.
    const uint32_t kx = kk & 3u, ky = (kk >> 2) & 3u, kz = (kk >> 4) & 3u;
    const f3 o = xyz(ro);
    const f3 A = xyz(q0) - o, B = xyz(q1) - o, C = xyz(q2) - o;
    const float akz = comp(A, kz), bkz = comp(B, kz), ckz = comp(C, kz);
    const float ax = comp(A, kx) - rs.x * akz, ay = comp(A, ky) - rs.y * akz;
    const float bx = comp(B, kx) - rs.x * bkz, by = comp(B, ky) - rs.y * bkz;
    const float cx = comp(C, kx) - rs.x * ckz, cy = comp(C, ky) - rs.y * ckz;
    const float uu = cx * by - cy * bx, vv = ax * cy - ay * cx, ww = bx * ay - by * ax;
    if ((uu < 0.0f || vv < 0.0f || ww < 0.0f) && (uu > 0.0f || vv > 0.0f || ww > 0.0f)) return;
    const float det = uu + vv + ww;
    if (det == 0.0f || !finite(det)) return;
    const float rcp = 1.0f / det;
    const float t = (uu * (rs.z * akz) + vv * (rs.z * bkz) + ww * (rs.z * ckz)) * rcp;
    if (!(t >= 0.0f && t <= ro.w)) return;
    const uint32_t src = M.src[L];
    const uint32_t gid = __float_as_uint(q0.w), m = __float_as_uint(q2.w);
    if (!EXT && gid == __float_as_uint(a.q.sh_d[src].w)) return;
    const uint32_t fl = mat_flags(s, m);
    if (EXT && (kk & 64u) && (fl & 4u) == 0u &&
        !(dot(xyz(a.st.dir[src]), cross(xyz(q1) - xyz(q0), xyz(q2) - xyz(q0))) < 0.0f))
        return;  // a primary ray culls back faces
    const uint32_t mode = fl & 3u;
    if (mode != 0u) {
        const float u = vv * rcp, v = ww * rcp;
        uint32_t path_seed, rid;
        if (EXT) {
            const uint4 sd = a.st.seed[src];
            path_seed = sd.z;
            rid = sd.w << 16u;
        } else {
            const uint4 sm = a.q.sh_m[src];
            path_seed = sm.w;
            rid = sm.z;
        }
        if (!alpha_accept(&s, slot, m, gid, 1.0f - u - v, u, v, path_seed, rid, mode)) return;
    }
    if (EXT) {
        // t + 0: a negative zero sorts as zero.
        const unsigned long long key = ((unsigned long long)__float_as_uint(t + 0.0f) << 32) | slot;
        const unsigned long long old = atomicMin(&M.best[L], key);
        const unsigned long long loser = old > key ? old : key;
        if (loser != ~0ull) atomicMin(&M.second[L], (uint32_t)(loser >> 32));
    } else {
        atomicMin(&M.found[L], slot);  // any accepted triangle will do
    }
}

// Tests the triangles of the warp's pending leaves, one (ray, triangle) pair
// per lane. Leaves are taken 32 at a time, one per lane; the lane of pair p
// finds its leaf by counting the leaf starts at or before p.
template <bool EXT, bool BATCH>
__device__ __forceinline__ void flush(const WaveArgs& a, WarpMem<EXT>& M, uint32_t lane, uint32_t leaves) {
    uint32_t incl = leaves;
#pragma unroll
    for (int k = 1; k < 32; k <<= 1) {
        const uint32_t up = __shfl_up_sync(FULL, incl, k);
        if (lane >= (uint32_t)k) incl += up;
    }
    const uint32_t total = __shfl_sync(FULL, incl, 31);
    for (uint32_t k = 0u; k < leaves; k++) M.list[incl - leaves + k] = (uint8_t)(lane | k << 5);
    __syncwarp();
    for (uint32_t at = 0u; at < total; at += 32u) {
        uint32_t ref = 0u, owner = 0u, n = 0u;
        if (at + lane < total) {
            const uint32_t e = M.list[at + lane];
            owner = e & 31u;
            ref = M.leaf[e >> 5][owner];
            n = ((ref >> 27) & 15u) + 1u;
        }
        uint32_t end = n;
#pragma unroll
        for (int k = 1; k < 32; k <<= 1) {
            const uint32_t up = __shfl_up_sync(FULL, end, k);
            if (lane >= (uint32_t)k) end += up;
        }
        const uint32_t start = end - n, pairs = __shfl_sync(FULL, end, 31);
        // Leaf's first slot less its first pair, and its ray.
        const uint32_t first = (ref & 0x07ffffffu) - start;
        for (uint32_t base = 0u; base < pairs; base += 32u) {
            const uint32_t before = __popc(__ballot_sync(FULL, n != 0u && start < base));
            const uint32_t bit = (n != 0u && start - base < 32u) ? 1u << (start - base) : 0u;
            const uint32_t starts = __reduce_or_sync(FULL, bit);
            const uint32_t r = before + __popc(starts & (0xffffffffu >> (31u - lane))) - 1u;
            const uint32_t L = __shfl_sync(FULL, owner, r), f = __shfl_sync(FULL, first, r);
            if (base + lane < pairs) test_pair<EXT, BATCH>(a, M, L, f + base + lane);
            __syncwarp();
        }
    }
}

// The answer of a ray that hits nothing.
template <bool EXT>
__device__ __forceinline__ void nothing_hit(const WaveArgs& a, uint32_t src) {
    if (EXT) {
        a.st.hit[src] = make_uint4(NONE, 0u, 0u, 0u);
    } else {
        const uint4 m = a.q.sh_m[src];
        mark_visible(a.st, a.jobs, m.x, m.y);
    }
}

// Checks the lane's finished ray and stores its answer.
template <bool EXT, bool BATCH>
__device__ __forceinline__ void finish(const WaveArgs& a, WarpMem<EXT>& M, uint32_t lane, float tl) {
    const uint32_t src = M.src[lane];
    const uint32_t tri = EXT ? (uint32_t)M.best[lane] : M.found[lane];
    if (tri == NONE) {
        nothing_hit<EXT>(a, src);
        return;
    }
    const Scene& s = ray_scene<EXT, BATCH>(a, src);
    const float4 o = M.o[lane], d = EXT ? a.st.dir[src] : a.q.sh_d[src];
    const Ray r = make_ray(xyz(o), xyz(d));
    float e = -1.0f;
    if (tri != NOT_WALKED) {
        const uint32_t ln = __ldg(s.leaf_of + tri);
        e = slab(r, geomv(s, 2ull * ln), geomv(s, 2ull * ln + 1u), EXT ? INF : o.w);
    }
    Hit h;
    uint32_t mat;
    if (EXT) {
        bool sure = e >= 0.0f;
        if (sure) {
            const uint64_t tb = tri_base(s, tri);
            const float4 q0 = geomv(s, tb), q1 = geomv(s, tb + 1), q2 = geomv(s, tb + 2);
            sure = intersect(r, q0, q1, q2, INF, &h);
            h.slot = tri;
            mat = __float_as_uint(q2.w);
            // The second distance as a float: a NaN when there is none, so that
            // "not at or below" holds.
            const float t = h.t, sec = __uint_as_float(M.second[lane]);
            sure = sure && (e <= t ? !(sec <= t) : (!(sec <= e) && e < tl));
        }
        bool got = sure;
        if (!sure) {
            const uint4 sd = a.st.seed[src];
            got = reference_walk(&s, &r, INF, sd.z, sd.w << 16u, sd.w == 0u, false, NONE, &h, &mat, a.err);
        }
        if (got) {
            a.st.hit[src] = make_uint4(h.slot, __float_as_uint(h.t), __float_as_uint(h.b.y), __float_as_uint(h.b.z));
            a.st.hmeta[src] = mat | (h.front ? 0x80000000u : 0u);
        } else {
            a.st.hit[src] = make_uint4(NONE, 0u, 0u, 0u);
        }
    } else if (!(e >= 0.0f)) {
        const uint4 m = a.q.sh_m[src];
        if (!reference_walk(&s, &r, o.w, m.w, m.z, false, true, __float_as_uint(d.w), &h, &mat, a.err))
            mark_visible(a.st, a.jobs, m.x, m.y);
    }
}

template <bool EXT, int MINB, int SD, bool BATCH>
__global__ void __launch_bounds__(NT, MINB) wide_walk(const __grid_constant__ WaveArgs a) {
    __shared__ WarpMem<EXT> mem[NT / 32];
    WarpMem<EXT>& M = mem[threadIdx.x >> 5];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t total = *((volatile uint32_t*)&a.ctr[EXT ? 0 : 1]);
    uint32_t* next = &a.ctr[EXT ? 5 : 6];
    // Rays a warp holds at once: all 32 lanes when there are rays for every
    // warp of the grid, else their share. Few rays are bound by the latency of
    // a walk, which the other rays of a warp and their triangles lengthen:
    // Cornell 256 x 256 closest hits 0.33 -> 0.26 ms in 12 launches (1 to 16
    // rays at least: 0.26 to 0.28 ms).
    const uint32_t warps = gridDim.x * (NT / 32u);
    const uint32_t most = min(32u, max(MIN_RAYS, (total + warps - 1u) / warps));
    bool drained = false;
    bool active = false;                 // the lane holds a ray
    uint32_t cur = NONE;                 // next node (NONE: none left)
    uint32_t group = 0u, sp = 0u;        // siblings still to visit, and the groups above them on the stack
    float group_t = 0.0f;                // closest: smallest entry of the group on the dominant axis
    uint32_t leaves = 0u;                // leaves pending
    uint32_t guard = 0u;
    float tl = 0.0f;                     // distance limit
    uint32_t kz = 0u;                    // closest: the ray's dominant axis
    const char* nodes = reinterpret_cast<const char*>(a.s.wide);
    NodeRay nr;
    uint32_t deep[SD];                   // stack entries from SS on
    float deep_t[EXT ? SD : 1];
    for (;;) {
        const bool busy = cur != NONE || leaves != 0u;
        const unsigned act = __ballot_sync(FULL, busy);
        if (act == 0u || (!drained && most - __popc(act) >= a.refill)) {
            if (active && !busy) {
                finish<EXT, BATCH>(a, M, lane, tl);
                active = false;
            }
            if (act == 0u && drained) break;
            bool none_left = false;
            if (!drained && !active && lane < most) {
                uint32_t q = append(next);
                if (q < total) {
                    float4 o, d;
                    uint32_t src;
                    bool primary = false;
                    if (EXT) {
                        src = a.q.ext[q];
                        o = a.st.org[src];
                        d = a.st.dir[src];
                        primary = a.st.seed[src].w == 0u;
                        o.w = INF;
                    } else {
                        src = (a.ray_order & 2u) ? a.q.sh_perm[q] : q;
                        o = a.q.sh_o[src];
                        d = a.q.sh_d[src];
                    }
                    const Scene& s = ray_scene<EXT, BATCH>(a, src);
                    const Ray r = make_ray(xyz(o), xyz(d));
                    if (r.valid && s.bvh4_root != NONE && s.P.env[3] != 0u) {
                        const bool walk = node_ray(s, r, nr);
                        if (BATCH) nodes = reinterpret_cast<const char*>(s.wide);
                        M.o[lane] = o;
                        M.shear[lane] = make_float4(r.shear.x, r.shear.y, r.shear.z,
                                                    __uint_as_float(r.kx | r.ky << 2 | r.kz << 4 |
                                                                    (primary ? 64u : 0u)));
                        M.src[lane] = src;
                        if (EXT) {
                            M.best[lane] = walk ? ~0ull : NOT_WALKED;
                            M.second[lane] = 0xffffffffu;
                        } else {
                            M.found[lane] = walk ? NONE : NOT_WALKED;
                        }
                        tl = o.w;
                        kz = r.kz;
                        sp = group = 0u;
                        if (!EXT) group = s.bvh4_root << 4 | 1u;
                        guard = 4u * STEPS * min(s.bvh4_nodes, 1u << 27) + 64u;
                        cur = walk ? s.bvh4_root : NONE;
                        if (walk && (cur & LEAF_BIT)) {  // a tree of one leaf
                            M.leaf[0][lane] = cur;
                            leaves = 1u;
                            cur = NONE;
                        }
                        active = true;
                    } else {
                        nothing_hit<EXT>(a, src);
                    }
                } else {
                    none_left = true;
                }
            }
            drained = __any_sync(FULL, drained || none_left);
        }
        // Node steps. A tree's nodes are visited at most once each.
        if (guard < (uint32_t)STEPS) {
            if (cur != NONE) atomicOr(a.err, 1u);
            cur = NONE;
        } else {
            guard -= STEPS;
        }
#pragma unroll 1
        for (int step = 0; step < STEPS; step++) {
            if (cur == NONE || leaves > LEAFCAP - 4u) continue;
            if (!EXT) {
                if (!(group & 15u)) {
                    sp--;
                    group = sp < SS ? M.stack[sp][lane] : deep[sp];
                }
                cur = (group >> 4) + (uint32_t)__ffs(group & 15u) - 1u;
                group &= group - 1u;
            }
            const char* nd = nodes + (uint64_t)cur * 64u;
            const u8x v0 = ld32(nd), v1 = ld32(nd + 32);
            float t0[4], t1[4], tx[4], ty[4];
            float td[4];  // closest: entry on the ray's dominant axis
#pragma unroll
            for (int ax = 0; ax < 3; ax++) {
                const float A = __uint_as_float(v0.v[3 + ax]) * nr.inv[ax];
                const float b = (__uint_as_float(v0.v[ax]) - nr.o[ax]) * nr.inv[ax];
                const uint32_t lo = ax < 2 ? v0.v[6 + ax] : v1.v[0], hi = v1.v[1 + ax];
                const bool neg = nr.inv[ax] < 0.0f;
                const uint32_t nw = neg ? hi : lo, fw = neg ? lo : hi;
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const float2 t = fma2(make_float2(plane(nw, k), plane(fw, k)), make_float2(A, A),
                                          make_float2(b, b));
                    if (ax == 0) t0[k] = t.x, t1[k] = t.y;
                    else if (ax == 1) tx[k] = t.x, ty[k] = t.y;
                    else {
                        if (EXT) td[k] = kz == 0u ? t0[k] : (kz == 1u ? tx[k] : t.x);
                        t0[k] = max3(fmaxf(t0[k], 0.0f), tx[k], t.x);
                        t1[k] = min3(EXT ? t1[k] : fminf(t1[k], tl), ty[k], t.y);
                    }
                }
            }
            uint32_t hit = 0u;
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (t0[k] <= t1[k] * SLACK && (!EXT || td[k] <= tl)) hit |= 1u << k;
            const uint32_t inner = hit & v0.v[3], leaf = hit & v0.v[4];  // the low four bits
#pragma unroll
            for (int k = 0; k < 4; k++)
                if (leaf & (1u << k)) M.leaf[leaves++][lane] = v1.v[4 + k];
            if (!EXT) {
                if (inner) {
                    if (group & 15u) {
                        if (sp < SS) M.stack[sp][lane] = group;
                        else deep[sp] = group;
                        sp++;
                    }
                    group = v1.v[4] << 4 | inner;
                }
                if (!(group & 15u) && sp == 0u) cur = NONE;
                continue;
            }
            if (inner) {
                // The nearest inner child is next, its siblings wait as a group.
                uint32_t key[4];
#pragma unroll
                for (int k = 0; k < 4; k++)
                    key[k] = (inner & (1u << k)) ? ((__float_as_uint(t0[k]) & ~3u) | (uint32_t)k) : NONE;
                const uint32_t lo01 = min(key[0], key[1]), lo23 = min(key[2], key[3]);
                const uint32_t nk = min(lo01, lo23) & 3u;
                const uint32_t rest = inner & ~(1u << nk), base = v1.v[4];
                if (rest) {
                    if (group & 15u) {
                        if (sp < SS) {
                            M.stack[sp][lane] = group;
                            M.stack_t[sp][lane] = group_t;
                        } else {
                            deep[sp] = group;
                            deep_t[sp] = group_t;
                        }
                        sp++;
                    }
                    group = base << 4 | rest;
                    group_t = INF;
#pragma unroll
                    for (int k = 0; k < 4; k++) group_t = fminf(group_t, rest & (1u << k) ? td[k] : INF);
                }
                cur = base + nk;
            } else {
                cur = NONE;
                for (;;) {
                    if (!(group & 15u)) {
                        if (sp == 0u) break;
                        sp--;
                        group = sp < SS ? M.stack[sp][lane] : deep[sp];
                        group_t = sp < SS ? M.stack_t[sp][lane] : deep_t[sp];
                    }
                    if (group_t > tl) {
                        group = 0u;
                        continue;
                    }
                    cur = (group >> 4) + (uint32_t)__ffs(group & 15u) - 1u;
                    group &= group - 1u;
                    break;
                }
            }
        }
        // Triangles.
        const uint32_t pending = __reduce_add_sync(FULL, leaves);
        if (pending && (pending >= FLUSH || !__any_sync(FULL, cur != NONE) || __any_sync(FULL, leaves > LEAFCAP - 4u))) {
            flush<EXT, BATCH>(a, M, lane, leaves);
            if (leaves) {
                if (EXT) {
                    const unsigned long long b = M.best[lane];
                    if (b != ~0ull) {
                        tl = __uint_as_float((uint32_t)(b >> 32)) * LIMIT;
                        M.o[lane].w = tl;
                    }
                } else if (M.found[lane] != NONE) {
                    cur = NONE;
                }
            }
            leaves = 0u;
        }
        __syncwarp();
    }
}

template <bool EXT, int SD, bool B>
void* wide_fn(int v) {
    return v == 0 ? (void*)wide_walk<EXT, 6, SD, B> : (void*)wide_walk<EXT, 8, SD, B>;
}

template <int SD, bool B>
void* wide_fn(bool ext, int v) {
    return ext ? wide_fn<true, SD, B>(v) : wide_fn<false, SD, B>(v);
}

}  // namespace

// variant 0: 6 resident blocks per SM; 1 and 2: 8 (10 would leave 48
// registers a thread, see above).
cudaError_t launch_wide_walk(const WaveArgs& a, bool ext, int variant, int sd, int sms, cudaStream_t st) {
    void* fn = a.nframes > 0 && !a.one_frame ? (sd <= 32 ? wide_fn<32, true>(ext, variant) : wide_fn<64, true>(ext, variant))
                             : (sd <= 32 ? wide_fn<32, false>(ext, variant) : wide_fn<64, false>(ext, variant));
    int per_sm = 0;
    cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, NT, 0);
    if (e != cudaSuccess) return e;
    WaveArgs copy = a;
    void* args[] = {&copy};
    cudaLaunchAttribute attr[1];
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(sms * (per_sm > 0 ? per_sm : 1)));
    cfg.blockDim = dim3(NT);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = l2_window(a, a.s.wide, (uint64_t)a.s.bvh4_nodes * 64u, attr);
    return cudaLaunchKernelExC(&cfg, fn, args);
}

}  // namespace oxd
