// Wavefront path tracing for sm_100a (Laine, Karras & Aila 2013,
// "Megakernels considered harmful").
//
// The megakernel (trace.cu) interleaves traversal, texture filtering,
// the layered BSDF and light sampling in one divergent loop: its code does
// not fit the instruction cache and a warp's lanes sit at different stages.
// Here a path is a slot of SoA state in HBM and every bounce is the shading
// kernels of wave_split.cu and two traversals:
//   wave_extend  closest-hit traversal of the queued continuation rays;
//   wave_shadow  any-hit traversal of the queued shadow rays
// (this file with the whole stack in local memory, trace_variant 0-2; the
// kernels of wide_walk.cu and wave_walk.cu otherwise). The traversal kernels
// hold nothing but the ray and the stack, so they run at high occupancy with
// coherent code. Each path's radiance receives the same contributions in the
// same order as in the megakernel (emission, the unoccluded NEE terms in job
// order, the next ray's findings), so results are bit-identical; finished
// paths land in the per-launch result buffer that reduce_frame adds to the
// accumulator in sample order.
#include "kernels.cuh"
#include "shade.cuh"
#include "traverse.cuh"
#include "wavefront.cuh"

namespace oxd {

// Traversal kernels: persistent grids over the ray queues, one walk per
// lane. A lane whose ray is finished takes the next queued ray (warp-
// aggregated fetch from a queue head) while the other lanes of its warp
// keep walking, once at least `a.refill` lanes of the warp are idle (1:
// at once; 32: only when the whole warp is idle), so warps are not held
// by their longest ray (Aila & Laine 2009, "Understanding the efficiency
// of ray traversal on GPUs": persistent threads, replacing terminated
// rays). The warp checks for idle lanes every STEPS walk steps. Each walk
// performs the same steps as a single-ray loop.
constexpr unsigned FULL_WARP = 0xffffffffu;
constexpr int STEPS = 4;

template <bool COUNT, int MINB, int SD, bool BATCH>
__global__ void __launch_bounds__(WAVE_TRAVERSE_THREADS, MINB) wave_extend(const __grid_constant__ WaveArgs a) {
    Cnt cnt;
    if (COUNT)
        for (int k = 0; k < C_N; k++) cnt.c[k] = 0;
    const uint32_t n = *((volatile uint32_t*)&a.ctr[0]);
    bool active = false, warp_drained = false;
    uint32_t i = 0u, k = 0u;
    const Scene* sc = &a.s;
    Ray r;
    Sampler smp{0u, 0u, 0u};
    Walk2<SD> w;
    for (;;) {
        const unsigned act = __ballot_sync(FULL_WARP, active);
        if (act == 0u && warp_drained) break;
        if (!warp_drained && 32 - __popc(act) >= (act ? a.refill : 1u)) {
            bool none_left = false;
            if (!active) {
                uint32_t q = append(&a.ctr[5]);
                if (q < n) {
                    i = a.q.ext[q];
                    sc = BATCH ? &a.frames[a.st.frame[i]].s : &a.s;
                    float4 o = a.st.org[i], d = a.st.dir[i];
                    uint4 sd = a.st.seed[i];
                    smp = Sampler{sd.x, sd.y, sd.z};
                    k = sd.w;
                    bump<COUNT>(cnt, C_PATH_RAYS);
                    r = make_ray(xyz(o), xyz(d));
                    if (walk2_begin<COUNT, SD>(*sc, r, INF, w, cnt)) active = true;
                    else a.st.hit[i] = make_uint4(NONE, 0u, 0u, 0u);
                } else {
                    none_left = true;
                }
            }
            warp_drained = __any_sync(FULL_WARP, none_left);
        }
#pragma unroll 1
        for (int st = 0; st < STEPS && active; st++) {
            if (walk2_step<COUNT, SD>(*sc, r, smp, k << 16u, k == 0u, false, NONE, w, cnt, a.err)) {
                active = false;
                if (w.hit_any) {
                    const Hit& h = w.best;
                    a.st.hit[i] = make_uint4(h.slot, __float_as_uint(h.t), __float_as_uint(h.b.y),
                                             __float_as_uint(h.b.z));
                    a.st.hmeta[i] = w.best_mat | (h.front ? 0x80000000u : 0u);
                } else {
                    a.st.hit[i] = make_uint4(NONE, 0u, 0u, 0u);
                }
            }
        }
    }
    if (COUNT)
        for (int c = 0; c < C_N; c++)
            if (cnt.c[c]) atomicAdd(a.counters + c, cnt.c[c]);
}

// FOUR: walk the four-wide tree (same occlusion as the binary walk); a
// batched launch uses it only when every frame's scene has one.
template <int SD, bool FOUR>
struct ShadowWalk {
    Walk2<SD> w;
};
template <int SD>
struct ShadowWalk<SD, true> {
    Walk4<SD> w;
};

template <bool COUNT, int MINB, int SD, bool FOUR, bool BATCH>
__global__ void __launch_bounds__(WAVE_TRAVERSE_THREADS, MINB) wave_shadow(const __grid_constant__ WaveArgs a) {
    Cnt cnt;
    if (COUNT)
        for (int k = 0; k < C_N; k++) cnt.c[k] = 0;
    const uint32_t n = *((volatile uint32_t*)&a.ctr[1]);
    bool active = false, warp_drained = false;
    uint32_t slot = 0u, job = 0u, rid = 0u, skip = NONE;
    const Scene* sc = &a.s;
    Ray r;
    Sampler smp{0u, 0u, 0u};
    ShadowWalk<SD, FOUR> sw;
    for (;;) {
        const unsigned act = __ballot_sync(FULL_WARP, active);
        if (act == 0u && warp_drained) break;
        if (!warp_drained && 32 - __popc(act) >= (act ? a.refill : 1u)) {
            bool none_left = false;
            if (!active) {
                uint32_t q = append(&a.ctr[6]);
                if (q < n) {
                    float4 o = a.q.sh_o[q], d = a.q.sh_d[q];
                    uint4 m = a.q.sh_m[q];
                    slot = m.x;
                    job = m.y;
                    rid = m.z;
                    skip = __float_as_uint(d.w);
                    smp = Sampler{0u, 0u, m.w};
                    sc = BATCH ? &a.frames[a.st.frame[slot]].s : &a.s;
                    bump<COUNT>(cnt, C_SHADOW_RAYS);
                    r = make_ray(xyz(o), xyz(d));
                    bool started;
                    if constexpr (FOUR) started = walk4_begin<SD>(*sc, r, o.w, sw.w);
                    else started = walk2_begin<COUNT, SD>(*sc, r, o.w, sw.w, cnt);
                    if (started) active = true;
                    else mark_visible(a.st, a.jobs, slot, job);  // nothing in the way
                } else {
                    none_left = true;
                }
            }
            warp_drained = __any_sync(FULL_WARP, none_left);
        }
#pragma unroll 1
        for (int st = 0; st < STEPS && active; st++) {
            bool done;
            if constexpr (FOUR) done = walk4_step<COUNT, SD>(*sc, r, smp, rid, false, skip, sw.w, cnt, a.err);
            else done = walk2_step<COUNT, SD>(*sc, r, smp, rid, false, true, skip, sw.w, cnt, a.err);
            if (done) {
                active = false;
                if (!sw.w.hit_any) mark_visible(a.st, a.jobs, slot, job);
            }
        }
    }
    if (COUNT)
        for (int c = 0; c < C_N; c++)
            if (cnt.c[c]) atomicAdd(a.counters + c, cnt.c[c]);
}

// Compiled variants: 6 / 8 / 10 blocks with a 32- or 64-deep stack; batched
// launches have no counting build. The tuner picks one; all give the same
// results.
template <bool C, int SD, bool B>
static void* ext_fn(int v) {
    if (v == 0) return (void*)wave_extend<C, 6, SD, B>;
    if (v == 1) return (void*)wave_extend<C, 8, SD, B>;
    return (void*)wave_extend<C, 10, SD, B>;
}

template <bool C, int SD, bool FOUR, bool B>
static void* shadow_fn(int v) {
    if (v == 0) return (void*)wave_shadow<C, 6, SD, FOUR, B>;
    if (v == 1) return (void*)wave_shadow<C, 8, SD, FOUR, B>;
    return (void*)wave_shadow<C, 10, SD, FOUR, B>;
}

template <bool C, bool B>
static void* trav_kernel_c(bool ext, bool four, int v, int sd) {
    if (ext) return sd <= 32 ? ext_fn<C, 32, B>(v) : ext_fn<C, 64, B>(v);
    if (four) return sd <= 32 ? shadow_fn<C, 32, true, B>(v) : shadow_fn<C, 64, true, B>(v);
    return sd <= 32 ? shadow_fn<C, 32, false, B>(v) : shadow_fn<C, 64, false, B>(v);
}

static void* trav_kernel(bool count, bool batch, bool ext, bool four, int v, int sd) {
    if (batch) return count ? nullptr : trav_kernel_c<false, true>(ext, four, v, sd);
    return count ? trav_kernel_c<true, false>(ext, four, v, sd) : trav_kernel_c<false, false>(ext, four, v, sd);
}

static cudaError_t launch_trav(const WaveArgs& a, bool count, bool ext, bool four, int variant, int sd, int sms,
                               cudaStream_t st) {
    variant = variant < 0 ? 0 : (variant > 2 ? 2 : variant);
    void* fn = trav_kernel(count, a.nframes > 0, ext, four, variant, sd);
    if (!fn) return cudaErrorInvalidValue;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, WAVE_TRAVERSE_THREADS, 0);
    unsigned blocks = (unsigned)(sms * (per_sm > 0 ? per_sm : 1));
    WaveArgs copy = a;
    void* args[] = {&copy};
    return cudaLaunchKernel(fn, dim3(blocks), dim3(WAVE_TRAVERSE_THREADS), args, 0, st);
}

// ctr[10] counts the iterations of the current run (zeroed with the run's
// counters; the per-iteration queue reset clears ctr[0..7] only).
__global__ void wave_continue(cudaGraphConditionalHandle h, uint32_t* ctr, uint32_t cap, uint32_t* err,
                              unsigned long long* tally, uint32_t kernels) {
    uint32_t it = ctr[10] + 1u;
    ctr[10] = it;
    bool more = ctr[2] != 0u;
    if (more && it >= cap) {
        atomicOr(err, 8u);
        more = false;
    }
    tally[0] += kernels;
    tally[1] += 1ull;
    cudaGraphSetConditional(h, more ? 1u : 0u);
}

cudaError_t launch_wave_continue(cudaGraphConditionalHandle h, uint32_t* ctr, uint32_t cap, uint32_t* err,
                                 unsigned long long* tally, uint32_t kernels, cudaStream_t st) {
    wave_continue<<<1, 1, 0, st>>>(h, ctr, cap, err, tally, kernels);
    return cudaGetLastError();
}

cudaError_t launch_wave_extend(const WaveArgs& a, bool count, int variant, int stack, int sms, cudaStream_t st) {
    if (variant >= 3 && !count && a.wide_closest && !a.closest4)
        return launch_wide_walk(a, true, variant - 3, stack, sms, st);
    if (variant >= 3) return launch_walk(a, count, true, a.closest4 != 0u, variant - 3, stack, sms, st);
    return launch_trav(a, count, true, false, variant, stack, sms, st);
}

cudaError_t launch_wave_shadow(const WaveArgs& a, bool count, bool four, int variant, int stack, int sms,
                               cudaStream_t st) {
    if (variant >= 3 && !count && a.wide && four && !a.shadow_post)
        return launch_wide_walk(a, false, variant - 3, stack, sms, st);
    if (variant >= 3) return launch_walk(a, count, false, four, variant - 3, stack, sms, st);
    return launch_trav(a, count, false, four, variant, stack, sms, st);
}

}  // namespace oxd
