// The shading work of a bounce in three kernels.
//
// One kernel with texture filtering, the layered BSDF, light sampling and
// path bookkeeping in one body does not fit the instruction cache. So:
//   split_logic  one thread per slot: adds the previous vertex's visible NEE
//                terms in job order, attenuates in a medium, handles misses
//                (environment / ambient), finalises finished paths and
//                regenerates their slots; surface hits go to a shade queue;
//   split_shade  one thread per queued hit: emission, material, BSDF of the
//                vertex (written to a vertex record for split_nee), BSDF
//                sampling and roulette; queues the continuation ray, and
//                lists the vertices by the kind of light they sample;
//   split_nee    the vertices' NEE jobs, one kind of light after the other;
// followed by the extension and shadow traversal kernels. Every path still
// receives its contributions in the reference's order: the vertex's NEE
// terms are added by the next split_logic before anything the next
// continuation ray finds.
#include <cooperative_groups.h>

#include <algorithm>

#include "kernels.cuh"
#include "path.cuh"
#include "shade.cuh"
#include "traverse.cuh"
#include "wavefront.cuh"

namespace cg = cooperative_groups;

namespace oxd {
// Built twice: exactly (the launchers in oxd) and with OXPT_FAST and fast
// math (the tolerance plan's shading; the launchers in oxd::fast).
#ifdef OXPT_FAST
namespace fast {
#endif

namespace {

enum : uint32_t { ST_EMPTY = 0, ST_TRACING = 1, ST_ENDING = 2 };

__device__ __forceinline__ uint32_t append1(uint32_t* ctr) {
    cg::coalesced_group g = cg::coalesced_threads();
    uint32_t base = 0;
    if (g.thread_rank() == 0) base = atomicAdd(ctr, g.size());
    return g.shfl(base, 0) + g.thread_rank();
}
// What split_shade needs of a path (its medium's extinction stays in memory).
__device__ __forceinline__ void load_state(const WaveArgs& a, uint32_t i, PathCore* pc, Sampler* smp) {
    uint4 sd = a.st.seed[i];
    float4 b = a.st.beta[i], r = a.st.rad[i], d = a.st.dir[i], pp = a.st.prev[i];
    smp->pixel_seed = sd.x;
    smp->index = sd.y;
    smp->path_seed = sd.z;
    pc->k = sd.w;
    pc->beta = xyz(b);
    pc->prev_pdf = b.w;
    pc->radiance = xyz(r);
    pc->in_medium = (__float_as_uint(r.w) & 4u) != 0u;
    pc->d = xyz(d);
    pc->prev_pos = xyz(pp);
    pc->sigma = sp(0.0f);
    pc->sigma_set = false;
}

__device__ __forceinline__ void save_rad(const WaveArgs& a, uint32_t i, const PathCore& pc, uint32_t stage) {
    a.st.rad[i] = make_float4(pc.radiance.x, pc.radiance.y, pc.radiance.z,
                              __uint_as_float(stage | (pc.in_medium ? 4u : 0u)));
}

// A path that goes on: only what a bounce changes is written. A path that
// ends needs no more than save_rad.
__device__ __forceinline__ void save_ray(const WaveArgs& a, uint32_t i, const PathCore& pc, f3 o) {
    save_rad(a, i, pc, ST_TRACING);
    a.st.beta[i] = make_float4(pc.beta.x, pc.beta.y, pc.beta.z, pc.prev_pdf);
    a.st.dir[i] = make_float4(pc.d.x, pc.d.y, pc.d.z, 0.0f);
    a.st.org[i] = make_float4(o.x, o.y, o.z, 0.0f);
}

__device__ __forceinline__ Hit load_hit(const WaveArgs& a, uint32_t i, uint32_t* hmat) {
    uint4 hb = a.st.hit[i];
    uint32_t hm = a.st.hmeta[i];
    Hit h;
    h.slot = hb.x;
    h.t = __uint_as_float(hb.y);
    float u = __uint_as_float(hb.z), v = __uint_as_float(hb.w);
    h.b = mk(1.0f - u - v, u, v);
    h.front = (hm >> 31) != 0u;
    *hmat = hm & 0x7fffffffu;
    return h;
}

// Vertex record, 13 float4 fields stored field-major (a warp's loads of one
// field are contiguous).
constexpr uint32_t VREC = 13;

__device__ __forceinline__ void put_vertex(const WaveArgs& a, uint32_t v, const Vertex& x, const PathCore& pc,
                                           uint32_t path_seed) {
    const uint32_t P = a.vcap;
    const Bsdf& b = x.bsdf;
    float4* r = a.q.vrec;
    r[0 * P + v] = make_float4(b.v.x, b.v.y, b.v.z, b.metallic);
    r[1 * P + v] = make_float4(b.n.x, b.n.y, b.n.z, b.alpha);
    r[2 * P + v] = make_float4(b.ng.x, b.ng.y, b.ng.z, b.specular);
    r[3 * P + v] = make_float4(b.ncc.x, b.ncc.y, b.ncc.z, b.transmission);
    r[4 * P + v] = make_float4(b.base.x, b.base.y, b.base.z, b.clearcoat);
    r[5 * P + v] = make_float4(b.f0d.x, b.f0d.y, b.f0d.z, b.cc_alpha);
    r[6 * P + v] = make_float4(b.sheen.x, b.sheen.y, b.sheen.z, b.sheen_rough);
    r[7 * P + v] = make_float4(b.eta_i, b.eta_t, b.sheen_alpha, b.w_cc);
    r[8 * P + v] = make_float4(b.p0, b.p1, b.p2, b.p3);
    r[9 * P + v] = make_float4(b.p4, __uint_as_float(b.thin ? 1u : 0u), __uint_as_float(pc.k), __uint_as_float(path_seed));
    r[10 * P + v] = make_float4(x.p.x, x.p.y, x.p.z, 0.0f);
    r[11 * P + v] = make_float4(pc.beta.x, pc.beta.y, pc.beta.z, 0.0f);
    r[12 * P + v] = x.pl_u;
}

__device__ __forceinline__ void get_vertex(const WaveArgs& a, uint32_t v, Vertex* x, PathCore* pc,
                                           uint32_t* path_seed) {
    const uint32_t P = a.vcap;
    const float4* r = a.q.vrec;
    Bsdf& b = x->bsdf;
    float4 f;
    f = r[0 * P + v]; b.v = xyz(f); b.metallic = f.w;
    f = r[1 * P + v]; b.n = xyz(f); b.alpha = f.w;
    f = r[2 * P + v]; b.ng = xyz(f); b.specular = f.w;
    f = r[3 * P + v]; b.ncc = xyz(f); b.transmission = f.w;
    f = r[4 * P + v]; b.base = xyz(f); b.clearcoat = f.w;
    f = r[5 * P + v]; b.f0d = xyz(f); b.cc_alpha = f.w;
    f = r[6 * P + v]; b.sheen = xyz(f); b.sheen_rough = f.w;
    f = r[7 * P + v]; b.eta_i = f.x; b.eta_t = f.y; b.sheen_alpha = f.z; b.w_cc = f.w;
    f = r[8 * P + v]; b.p0 = f.x; b.p1 = f.y; b.p2 = f.z; b.p3 = f.w;
    f = r[9 * P + v];
    b.p4 = f.x;
    b.thin = __float_as_uint(f.y) != 0u;
    pc->k = __float_as_uint(f.z);
    *path_seed = __float_as_uint(f.w);
    f = r[10 * P + v]; x->p = xyz(f);
    f = r[11 * P + v]; pc->beta = xyz(f);
    x->pl_u = r[12 * P + v];
    x->ng = b.ng;
}

// Batched launches (frames of several scenes in one wavefront): the frame
// of a launch item, and the scene of a slot.
__device__ __forceinline__ uint32_t frame_of1(const WaveArgs& a, unsigned long long item) {
    uint32_t lo = 0u, hi = a.nframes;
    while (hi - lo > 1u) {
        uint32_t mid = (lo + hi) >> 1;
        if (a.frames[mid].base <= item) lo = mid;
        else hi = mid;
    }
    return lo;
}

// What a launch traces: one scene's frame given in its arguments; frames of a
// batch, whose records are in memory; or a batch of one frame, whose scene is
// in the arguments all the same (constant memory; read from a record, every
// field is a load of its own) and whose camera, seed and sample range come
// from the record, so that a captured graph serves the next step.
enum Launch : int { PLAIN = 0, FRAMES = 1, ONE_FRAME = 2 };

template <int M>
__device__ __forceinline__ const Scene& slot_scene(const WaveArgs& a, uint32_t i) {
    return M == FRAMES ? a.frames[a.st.frame[i]].s : a.s;
}

// Shared-memory tables come from the first frame in a batched launch (the
// host checks that every scene holds the same words).
template <int M>
__device__ __forceinline__ const Scene& tables_of(const WaveArgs& a) {
    return M == FRAMES ? a.frames[0].s : a.s;
}

// Radiance-cache inputs of a vertex: position normalised to the scene's
// root box, outgoing direction and shading normal mapped to [0, 1], GGX
// alpha; three float4 (pos.xyz, alpha | dir.xyz, 0 | normal.xyz, 0).
__device__ __forceinline__ void nrc_features(const Scene& s, const Vertex& vx, float4* out) {
    float4 lo = geomv(s, 0), hi = geomv(s, 1);
    f3 ext = mk(fmaxf(hi.x - lo.x, 1e-20f), fmaxf(hi.y - lo.y, 1e-20f), fmaxf(hi.z - lo.z, 1e-20f));
    f3 p = vx.p;
    const Bsdf& b = vx.bsdf;
    out[0] = make_float4(clampf((p.x - lo.x) / ext.x, 0.0f, 1.0f), clampf((p.y - lo.y) / ext.y, 0.0f, 1.0f),
                         clampf((p.z - lo.z) / ext.z, 0.0f, 1.0f), clampf(b.alpha, 0.0f, 1.0f));
    out[1] = make_float4(0.5f * (b.v.x + 1.0f), 0.5f * (b.v.y + 1.0f), 0.5f * (b.v.z + 1.0f), 0.0f);
    out[2] = make_float4(0.5f * (b.n.x + 1.0f), 0.5f * (b.n.y + 1.0f), 0.5f * (b.n.z + 1.0f), 0.0f);
}

// A finished training path: its target is the radiance gathered after the
// recorded vertex, per unit throughput there.
__device__ __forceinline__ void nrc_finish(const WaveArgs& a, uint32_t i, const PathCore& pc) {
    uint32_t ti = a.nrc.s_tidx[i];
    if (ti == NONE) return;
    a.nrc.s_tidx[i] = NONE;
    float4 pre = a.nrc.s_pre[i], b = a.nrc.s_beta[i];
    f3 d = pc.radiance - xyz(pre);
    float t[3] = {d.x, d.y, d.z}, bb[3] = {b.x, b.y, b.z};
    for (int c = 0; c < 3; c++) {
        float v = bb[c] > 0.0f ? t[c] / bb[c] : 0.0f;
        t[c] = finite(v) ? fmaxf(v, 0.0f) : 0.0f;
    }
    a.nrc.t_target[ti] = make_float4(t[0], t[1], t[2], 1.0f);
}

}  // namespace

// What split_logic found at a slot.
enum LogicOutcome : uint32_t { SLOT_SURFACE, SLOT_FREED, SLOT_EMPTY };

// Adds the slot's NEE terms and takes its path past its ray: a surface hit to
// shade, or a finished path, whose result is stored. What every slot reads is
// loaded first, together.
template <int M>
__device__ __forceinline__ uint32_t logic_slot(const WaveArgs& a, uint32_t i) {
    const uint32_t J = a.jobs;
    PathCore pc;
    const float4 rad = a.st.rad[i];
    const uint32_t n = a.st.nee_n[i], vis = a.st.vis ? a.st.vis[i] : 0u;
    const uint4 h = a.st.hit[i];
    const unsigned long long item = a.st.item[i];
    const uint32_t stage = __float_as_uint(rad.w) & 3u;
    if (stage == ST_EMPTY) return SLOT_EMPTY;
    pc.radiance = xyz(rad);
    pc.in_medium = (__float_as_uint(rad.w) & 4u) != 0u;
    if (a.st.vis) {
        // The unoccluded jobs' contributions, in job order.
        uint32_t m = n ? vis : 0u;
        while (m) {
            uint32_t j = __ffs(m) - 1u;
            m &= m - 1u;
            if (j < n) pc.radiance = pc.radiance + xyz(a.st.pend[(uint64_t)i * J + j]);
        }
    } else {
        for (uint32_t j = 0; j < n; j++) {
            float4 pe = a.st.pend[(uint64_t)i * J + j];
            if (pe.w == 2.0f) pc.radiance = pc.radiance + xyz(pe);
        }
    }
    if (n) a.st.nee_n[i] = 0u;
    int r = PATH_DONE;
    if (stage == ST_TRACING) {
        r = PATH_SURFACE;
        if (h.x == NONE || pc.in_medium) {
            const float4 b = a.st.beta[i], d = a.st.dir[i];
            pc.beta = xyz(b);
            pc.prev_pdf = b.w;
            pc.d = xyz(d);
            pc.k = a.st.seed[i].w;
            if (pc.in_medium) pc.sigma = xyz(a.st.sigma[i]);
            Hit hit;
            hit.t = __uint_as_float(h.y);
            r = after_ray(slot_scene<M>(a, i), pc, h.x != NONE, hit);
            if (r == PATH_SURFACE) a.st.beta[i] = make_float4(pc.beta.x, pc.beta.y, pc.beta.z, pc.prev_pdf);
        }
    }
    if (r == PATH_SURFACE) {
        save_rad(a, i, pc, ST_TRACING);
        return SLOT_SURFACE;
    }
    a.out[item] = path_result(pc, r != PATH_UNCOVERED);
    if (a.nrc.on) nrc_finish(a, i, pc);
    return SLOT_FREED;
}

// Starts the path of launch item `item` in slot i.
template <int M>
__device__ __forceinline__ void start_slot(const WaveArgs& a, uint32_t i, unsigned long long item,
                                           const uint4* s_sobol) {
    PathCore pc;
    Sampler smp;
    constexpr bool REC = M != PLAIN;
    uint32_t f = M == FRAMES ? frame_of1(a, item) : 0u;
    const Scene& s = REC ? a.frames[f].s : a.s;
    unsigned long long local = REC ? item - a.frames[f].base : item;
    uint32_t npix = REC ? a.frames[f].npix : a.npix;
    uint32_t y0 = REC ? a.frames[f].y0 : a.y0, first = REC ? a.frames[f].first : a.first;
    uint32_t it = (uint32_t)(local / npix);
    uint32_t q = (uint32_t)(local - (unsigned long long)it * npix);
    uint32_t yy = q / s.P.dims[0];
    f3 o = start_path(s, s_sobol, q - yy * s.P.dims[0], y0 + yy, first + it, &smp, &pc);
    a.st.item[i] = item;
    if (M == FRAMES) a.st.frame[i] = f;
    if (a.nrc.on) {
        a.nrc.s_tidx[i] = NONE;
        a.nrc.s_tail[i] = NONE;
    }
    a.st.seed[i] = make_uint4(smp.pixel_seed, smp.index, smp.path_seed, pc.k);
    save_ray(a, i, pc, o);
}

constexpr uint32_t LOGIC_THREADS = 256u;

// One thread per slot; a block asks for its places in the queues and its new
// items once. Each warp asking for itself made five atomics a warp on one
// 64-byte line the kernel's bound (4.2 M slots: 365 us whether it moved 1.3
// or 0.6 GB).
template <bool COUNT, int M>
__global__ void __launch_bounds__(LOGIC_THREADS, 4) split_logic(const __grid_constant__ WaveArgs a) {
    constexpr uint32_t WARPS = LOGIC_THREADS / 32u;
    __shared__ uint32_t s_dirs[128];
    __shared__ uint4 s_sobol[128];
    __shared__ uint32_t s_surface[WARPS], s_free[WARPS];
    __shared__ uint32_t s_shade_at, s_ext_at;
    __shared__ unsigned long long s_item_at;
    const uint32_t i = blockIdx.x * LOGIC_THREADS + threadIdx.x, lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    if (i == 0u) a.ctr[11] = a.ctr[12] = 0u;  // counted by split_shade
    const uint32_t out = i < a.slots ? logic_slot<M>(a, i) : (uint32_t)SLOT_EMPTY;
    const bool surface = out == SLOT_SURFACE, free_slot = !surface && i < a.slots;
    const unsigned below = (1u << lane) - 1u;
    const unsigned ms = __ballot_sync(0xffffffffu, surface), mf = __ballot_sync(0xffffffffu, free_slot);
    if (lane == 0u) {
        s_surface[warp] = __popc(ms);
        s_free[warp] = __popc(mf);
    }
    __syncthreads();
    uint32_t surfaces = 0u, frees = 0u, my_surface = __popc(ms & below), my_free = __popc(mf & below);
#pragma unroll
    for (uint32_t w = 0; w < WARPS; w++) {
        if (w == warp) {
            my_surface += surfaces;
            my_free += frees;
        }
        surfaces += s_surface[w];
        frees += s_free[w];
    }
    if (threadIdx.x == 0u) {
        uint32_t starts = 0u;
        if (frees) {
            s_item_at = atomicAdd(a.work, (unsigned long long)frees);
            const unsigned long long left = s_item_at < a.total ? a.total - s_item_at : 0ull;
            starts = left < frees ? (uint32_t)left : frees;
            if (starts) s_ext_at = atomicAdd(&a.ctr[0], starts);
        }
        if (surfaces) s_shade_at = atomicAdd(&a.ctr[3], surfaces);
        if (surfaces + starts) atomicAdd(&a.ctr[2], surfaces + starts);
        if (COUNT && starts) atomicAdd(a.counters + C_PATHS, (unsigned long long)starts);
    }
    if (frees) {
        const Scene& s0 = tables_of<M>(a);
        for (uint32_t k = threadIdx.x; k < 128u; k += LOGIC_THREADS) s_dirs[k] = tw(s0, s0.P.offs0[0] + k);
    }
    __syncthreads();
    if (frees) {  // the same for the whole block
        sobol_nibbles(s_dirs, s_sobol);
        __syncthreads();
    }
    if (surface) a.q.shade[s_shade_at + my_surface] = i;
    if (!free_slot) return;
    const unsigned long long item = s_item_at + my_free;
    if (item < a.total) {
        start_slot<M>(a, i, item, s_sobol);
        a.q.ext[s_ext_at + my_free] = i;
    } else if (out != SLOT_EMPTY) {
        a.st.rad[i].w = __uint_as_float(ST_EMPTY);
    }
}

// The radiance cache's part at a vertex; true when the path ends here, the
// cache supplying the rest.
__device__ __forceinline__ bool nrc_vertex(const WaveArgs& a, const Scene& s, uint32_t i, const PathCore& pc,
                                           const Sampler& smp, const Vertex& vx, float t) {
    bool spread_ok = true;
    {
        // Path spread (Mueller et al. 2021): a0 = t^2 / (4 pi |cos|) at the
        // primary vertex, then the sum of sqrt(t^2 / (pdf |cos|)) over bounces.
        const float cosv = fabsf(dot(vx.ng, pc.d));
        float2 sp = pc.k == 0u ? make_float2(0.0f, 0.0f) : a.nrc.s_spread[i];
        if (pc.k == 0u) sp.x = t * t / (4.0f * PI * fmaxf(cosv, 1e-6f));
        else if (pc.prev_pdf > 0.0f && cosv > 0.0f) sp.y += sqrtf(t * t / (pc.prev_pdf * cosv));
        a.nrc.s_spread[i] = sp;
        spread_ok = a.nrc.spread <= 0.0f || sp.y * sp.y > a.nrc.spread * sp.x;
    }
    const uint32_t tail = a.nrc.s_tail[i];
    if (tail == pc.k && (smp.path_seed & a.nrc.train_mask) == 0u) {
        // A training path's suffix ends here, into the cache.
        float4 f[3];
        nrc_features(s, vx, f);
        uint32_t q = atomicAdd(&a.nrc.counts[0], 1u);
        if (q < a.nrc.q_cap) {
            a.nrc.q_in[3 * (size_t)q] = f[0];
            a.nrc.q_in[3 * (size_t)q + 1] = f[1];
            a.nrc.q_in[3 * (size_t)q + 2] = f[2];
            a.nrc.q_beta[q] = make_float4(pc.beta.x, pc.beta.y, pc.beta.z, 0.0f);
            a.nrc.q_item[q] = a.st.item[i];
            uint32_t ti = a.nrc.s_tidx[i];
            if (ti != NONE) {
                float4 b0 = a.nrc.s_beta[i];
                float rx = b0.x > 0.0f ? pc.beta.x / b0.x : 0.0f;
                float ry = b0.y > 0.0f ? pc.beta.y / b0.y : 0.0f;
                float rz = b0.z > 0.0f ? pc.beta.z / b0.z : 0.0f;
                a.nrc.t_tail[ti] = make_uint4(q, __float_as_uint(rx), __float_as_uint(ry), __float_as_uint(rz));
            }
        }
        a.st.nee_n[i] = 0u;
        return true;
    }
    if (pc.k >= a.nrc.query_k && tail == NONE && spread_ok) {
        float4 f[3];
        nrc_features(s, vx, f);
        if ((smp.path_seed & a.nrc.train_mask) != 0u) {
            // A rendering path ends here: the cache supplies the rest.
            uint32_t q = atomicAdd(&a.nrc.counts[0], 1u);
            if (q < a.nrc.q_cap) {
                a.nrc.q_in[3 * (size_t)q] = f[0];
                a.nrc.q_in[3 * (size_t)q + 1] = f[1];
                a.nrc.q_in[3 * (size_t)q + 2] = f[2];
                a.nrc.q_beta[q] = make_float4(pc.beta.x, pc.beta.y, pc.beta.z, 0.0f);
                a.nrc.q_item[q] = a.st.item[i];
            }
            a.st.nee_n[i] = 0u;
            return true;
        }
        a.nrc.s_tail[i] = a.nrc.suffix ? pc.k + a.nrc.suffix : 0xfffffffeu;
        uint32_t ti = atomicAdd(&a.nrc.counts[1], 1u);
        if (ti < a.nrc.t_cap) {
            a.nrc.t_in[3 * (size_t)ti] = f[0];
            a.nrc.t_in[3 * (size_t)ti + 1] = f[1];
            a.nrc.t_in[3 * (size_t)ti + 2] = f[2];
            a.nrc.t_target[ti] = make_float4(0.f, 0.f, 0.f, 0.f);
            a.nrc.t_tail[ti] = make_uint4(NONE, 0u, 0u, 0u);
            a.nrc.s_pre[i] = make_float4(pc.radiance.x, pc.radiance.y, pc.radiance.z, 0.0f);
            a.nrc.s_beta[i] = make_float4(pc.beta.x, pc.beta.y, pc.beta.z, 0.0f);
            a.nrc.s_tidx[i] = ti;
        }
    }
    return false;
}

// Was bound by fetching instructions: of 22 cycles an instruction, 12 waited
// for the next one (ncu, 1080p materials scene with a radiance cache; now half
// a cycle, and load latency, 5.4 of 11.7 cycles, is the bound). So a block
// is 256 threads and stays together: its warps meet before a hit is shaded,
// before the vertex is stored and before the path is continued, and fetch each
// part once (against 128 threads that met once a round, for 8 spp of the
// 1.05 M-triangle frame / of 480 k-triangle boxes: 3.59 to 3.37 / 3.70 to
// 3.34 ms; 512 threads: 3.53 / 3.42).
constexpr uint32_t SHADE_THREADS = 256u;

template <bool COUNT, int MINB, int M>
__global__ void __launch_bounds__(SHADE_THREADS, MINB) split_shade(const __grid_constant__ WaveArgs a) {
    __shared__ uint32_t s_dirs[128];
    __shared__ uint4 s_sobol[128];
    __shared__ float s_sheen[512];
    {
        const Scene& s0 = tables_of<M>(a);
        for (uint32_t i = threadIdx.x; i < 128u; i += blockDim.x) s_dirs[i] = tw(s0, s0.P.offs0[0] + i);
        for (uint32_t i = threadIdx.x; i < 512u; i += blockDim.x) s_sheen[i] = tf(s0, s0.P.offs0[1] + i);
    }
    __syncthreads();
    sobol_nibbles(s_dirs, s_sobol);  // read after the loop's barrier
    const uint32_t n = *((volatile uint32_t*)&a.ctr[3]);
    unsigned long long shaded = 0;
    for (uint32_t q0 = blockIdx.x * blockDim.x; q0 < n; q0 += gridDim.x * blockDim.x) {
        __syncthreads();
        const uint32_t q = q0 + threadIdx.x;
        uint32_t i = 0u;
        PathCore pc;
        Sampler smp;
        Vertex vx;
        bool vertex = false;
        if (q < n) {
            i = a.q.shade[q];
            const Scene& s = slot_scene<M>(a, i);
            load_state(a, i, &pc, &smp);
            uint32_t hmat;
            Hit hit = load_hit(a, i, &hmat);
            const int r = shade_hit<COUNT>(s, M == ONE_FRAME ? a.frames[0].s : s, s_sheen, s_sobol, smp, pc, hit, hmat,
                                           &vx, &shaded);
            vertex = r == PATH_VERTEX && (!a.nrc.on || !nrc_vertex(a, s, i, pc, smp, vx, hit.t));
            if (!vertex) save_rad(a, i, pc, ST_ENDING);
        }
        __syncthreads();
        if (vertex) {
            const Scene& s = slot_scene<M>(a, i);
            uint32_t v = append1(&a.ctr[4]);
            put_vertex(a, v, vx, pc, smp.path_seed);
            a.q.vslot[v] = i;
            const uint32_t jobs = M == FRAMES ? s.P.cfg[2] + 1u : a.jobs;
            a.st.nee_n[i] = jobs;
            if (a.st.vis) a.st.vis[i] = 0u;
            const uint32_t kind = sampled_light(s, vx.pl_u.z);
            if (kind == SAMPLED_ENV) a.q.vlight[append1(&a.ctr[11])] = v;
            else if (kind == SAMPLED_AREA) a.q.vlight[a.vcap - 1u - append1(&a.ctr[12])] = v;
            else if (!a.st.vis) a.st.pend[(uint64_t)i * a.jobs + jobs - 1u] = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        if (!vertex) continue;
        const Scene& s = slot_scene<M>(a, i);
        f3 o;
        if (continue_path(s, s_sheen, s_sobol, smp, pc, vx, &o)) {
            a.st.seed[i].w = pc.k;
            a.st.prev[i] = make_float4(pc.prev_pos.x, pc.prev_pos.y, pc.prev_pos.z, 0.0f);
            if (pc.sigma_set) a.st.sigma[i] = make_float4(pc.sigma.x, pc.sigma.y, pc.sigma.z, 0.0f);
            save_ray(a, i, pc, o);
            a.q.ext[append1(&a.ctr[0])] = i;
        } else {
            save_rad(a, i, pc, ST_ENDING);
        }
    }
    if (COUNT && shaded) atomicAdd(a.counters + C_SHADED, shaded);
}

constexpr uint32_t NEE_THREADS = 256u;
constexpr uint32_t NEE_LIGHTS = 64u;  // punctual lights the vertex-major kernel keeps in shared memory

// Stores NEE job j of `slot`: queues its shadow ray, and its contribution
// (without visibility masks, also that there is none).
__device__ __forceinline__ void put_job(const WaveArgs& a, uint32_t slot, uint32_t j, uint32_t path_seed, bool queued,
                                        const ShadowRay& sr) {
    float4 pe = make_float4(0.f, 0.f, 0.f, 0.f);
    if (queued) {
        pe = make_float4(sr.pending.x, sr.pending.y, sr.pending.z, 1.0f);
        uint32_t q = append1(&a.ctr[1]);
        a.q.sh_o[q] = make_float4(sr.o.x, sr.o.y, sr.o.z, sr.tmax);
        a.q.sh_d[q] = make_float4(sr.d.x, sr.d.y, sr.d.z, __uint_as_float(sr.skip));
        a.q.sh_m[q] = make_uint4(slot, j, sr.rid, path_seed);
    }
    if (queued || !a.st.vis) a.st.pend[(uint64_t)slot * a.jobs + j] = pe;
}

// The vertices' NEE jobs, one kind of light after the other: environment
// samples, emissive-triangle samples (lists made by split_shade, so their
// warps are full), then punctual lights. All warps of the grid then run the
// same few kilobytes of code at a time; with one thread doing every job of a
// vertex in order, 75% of the warps' time went to fetching instructions (ncu,
// 480 k-triangle boxes: 17.6 of 23.5 cycles an instruction, 10.9 of 32 lanes
// active). A block's warps also meet before each round of a phase (punctual
// phase: 480 k-triangle boxes 4.03 to 3.85 ms, 32 spp of a materials scene 2.85
// to 2.74, the 1.05 M-triangle frame 2.71 to 2.75). Punctual lights are taken vertex-major (VMAJOR: one thread loads
// its vertex record once and runs every light in order, so the lanes of a
// warp evaluate the same light) or job-major (one thread per vertex and
// light: batches that mix scenes of different light counts).
template <bool VMAJOR, int MINB, int M>
__global__ void __launch_bounds__(NEE_THREADS, MINB) split_nee(const __grid_constant__ WaveArgs a) {
    constexpr bool BATCH = M == FRAMES;
    __shared__ float s_sheen[512];
    // Punctual lights of a one-scene launch, four 16-byte words each.
    __shared__ float4 s_light[BATCH || !VMAJOR ? 1 : 4 * NEE_LIGHTS];
    {
        const Scene& s0 = tables_of<M>(a);
        for (uint32_t i = threadIdx.x; i < 512u; i += blockDim.x) s_sheen[i] = tf(s0, s0.P.offs0[1] + i);
        if (VMAJOR && !BATCH)
            for (uint32_t i = threadIdx.x; i < 4u * min(a.jobs - 1u, NEE_LIGHTS); i += blockDim.x)
                s_light[i] = tv4(a.s, a.s.P.offs0[3] + 4u * i);
    }
    __syncthreads();
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    const uint32_t nv = *((volatile uint32_t*)&a.ctr[4]);
    const uint32_t n_env = *((volatile uint32_t*)&a.ctr[11]), n_area = *((volatile uint32_t*)&a.ctr[12]);
    Vertex vx;
    PathCore pc;
    uint32_t path_seed;
    ShadowRay sr;
    for (uint32_t k0 = blockIdx.x * blockDim.x; k0 < n_env; k0 += stride) {
        __syncthreads();  // the block's warps fetch the same code together
        const uint32_t k = k0 + threadIdx.x;
        if (k >= n_env) continue;
        const uint32_t v = a.q.vlight[k], slot = a.q.vslot[v];
        const Scene& s = slot_scene<M>(a, slot);
        get_vertex(a, v, &vx, &pc, &path_seed);
        const bool queued = nee_env(s, s_sheen, pc, vx, view_terms(s_sheen, vx.bsdf), &sr);
        put_job(a, slot, s.P.cfg[2], path_seed, queued, sr);
    }
    for (uint32_t k0 = blockIdx.x * blockDim.x; k0 < n_area; k0 += stride) {
        __syncthreads();  // see above
        const uint32_t k = k0 + threadIdx.x;
        if (k >= n_area) continue;
        const uint32_t v = a.q.vlight[a.vcap - 1u - k], slot = a.q.vslot[v];
        const Scene& s = slot_scene<M>(a, slot);
        get_vertex(a, v, &vx, &pc, &path_seed);
        const bool queued = nee_area(s, s_sheen, pc, vx, view_terms(s_sheen, vx.bsdf), &sr);
        put_job(a, slot, s.P.cfg[2], path_seed, queued, sr);
    }
    if (a.jobs == 1u) return;
    if (VMAJOR) {
        for (uint32_t v0 = blockIdx.x * blockDim.x; v0 < nv; v0 += stride) {
            __syncthreads();  // see above
            const uint32_t v = v0 + threadIdx.x;
            if (v >= nv) continue;
            const uint32_t slot = a.q.vslot[v];
            const Scene& s = slot_scene<M>(a, slot);
            const uint32_t np = BATCH ? s.P.cfg[2] : a.jobs - 1u;
            if (BATCH && np == 0u) continue;
            get_vertex(a, v, &vx, &pc, &path_seed);
            const ViewTerms vt = view_terms(s_sheen, vx.bsdf);
#pragma unroll 1
            for (uint32_t j = 0; j < np; j++) {
                LightRec rec;
                if (!BATCH && j < NEE_LIGHTS)
                    rec = {s_light[4u * j], s_light[4u * j + 1u], s_light[4u * j + 2u], s_light[4u * j + 3u]};
                else rec = light_rec(s, j);
                const bool queued = nee_punctual(s, s_sheen, pc, vx, vt, rec, j, &sr);
                put_job(a, slot, j, path_seed, queued, sr);
            }
        }
    } else {
        const uint64_t total = (uint64_t)nv * (a.jobs - 1u);
        for (uint64_t t = first; t < total; t += stride) {
            const uint32_t j = (uint32_t)(t / nv), v = (uint32_t)(t - (uint64_t)j * nv);
            const uint32_t slot = a.q.vslot[v];
            const Scene& s = slot_scene<M>(a, slot);
            if (BATCH && j >= s.P.cfg[2]) continue;  // beyond this scene's punctual lights
            get_vertex(a, v, &vx, &pc, &path_seed);
            const bool queued =
                nee_punctual(s, s_sheen, pc, vx, view_terms(s_sheen, vx.bsdf), light_rec(s, j), j, &sr);
            put_job(a, slot, j, path_seed, queued, sr);
        }
    }
}

// Variants: shade kernel for 2 (0, 1; 128 registers) or 3 (2; 80) blocks per
// SM, 3.37 against 3.26 ms of shading per 8 spp of the 1.05 M-triangle frame,
// 3.34 against 3.71 of 480 k-triangle boxes; the NEE kernel job-major for 2
// (0, 1) or 3 (2) blocks per SM, or vertex-major for 2 (3, 4) or 3 (5).
template <bool C, int M>
static void* shade_fn(int v) {
    return v < 2 ? (void*)split_shade<C, 2, M> : (void*)split_shade<C, 3, M>;
}
template <int M>
static void* nee_fn(int v) {
    if (v < 3) return v < 2 ? (void*)split_nee<false, 2, M> : (void*)split_nee<false, 3, M>;
    return v < 5 ? (void*)split_nee<true, 2, M> : (void*)split_nee<true, 3, M>;
}

// One grid of resident blocks, no more than the slots fill.
static cudaError_t persistent(void* fn, const WaveArgs& a, int sms, cudaStream_t st, unsigned threads) {
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, (int)threads, 0);
    WaveArgs copy = a;
    void* args[] = {&copy};
    unsigned blocks = (unsigned)(sms * (per_sm > 0 ? per_sm : 1));
    return cudaLaunchKernel(fn, dim3(std::min(blocks, (a.slots + threads - 1) / threads)), dim3(threads), args, 0, st);
}

// Batched launches (a.nframes > 0) have no counting build. NEE needs nothing
// of a single frame's record.
static Launch launch_of(const WaveArgs& a) { return !a.nframes ? PLAIN : (a.one_frame ? ONE_FRAME : FRAMES); }

cudaError_t launch_split_logic(const WaveArgs& a, bool count, cudaStream_t st) {
    const unsigned blocks = (a.slots + LOGIC_THREADS - 1u) / LOGIC_THREADS;
    const Launch m = launch_of(a);
    if (m != PLAIN && count) return cudaErrorInvalidValue;
    if (m == FRAMES) split_logic<false, FRAMES><<<blocks, LOGIC_THREADS, 0, st>>>(a);
    else if (m == ONE_FRAME) split_logic<false, ONE_FRAME><<<blocks, LOGIC_THREADS, 0, st>>>(a);
    else if (count) split_logic<true, PLAIN><<<blocks, LOGIC_THREADS, 0, st>>>(a);
    else split_logic<false, PLAIN><<<blocks, LOGIC_THREADS, 0, st>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_split_shade(const WaveArgs& a, bool count, int variant, int sms, cudaStream_t st) {
    variant = variant < 0 ? 0 : (variant > 2 ? 2 : variant);
    const Launch m = launch_of(a);
    if (m != PLAIN && count) return cudaErrorInvalidValue;
    void* fn = m == FRAMES ? shade_fn<false, FRAMES>(variant)
               : m == ONE_FRAME ? shade_fn<false, ONE_FRAME>(variant)
               : count ? shade_fn<true, PLAIN>(variant) : shade_fn<false, PLAIN>(variant);
    return persistent(fn, a, sms, st, SHADE_THREADS);
}

cudaError_t launch_split_nee(const WaveArgs& a, bool count, int variant, int sms, cudaStream_t st) {
    variant = variant < 0 ? 0 : (variant > 5 ? 5 : variant);
    const Launch m = launch_of(a);
    if (m != PLAIN && count) return cudaErrorInvalidValue;
    return persistent(m == FRAMES ? nee_fn<FRAMES>(variant) : nee_fn<PLAIN>(variant), a, sms, st, NEE_THREADS);
}

#ifdef OXPT_FAST
}  // namespace fast
#endif
}  // namespace oxd
