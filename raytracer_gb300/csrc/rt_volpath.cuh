// rt_volpath.cuh -- VolPathTracing on the device: the persistent kernel
// (k_volpath, one vol_step pass of the reference's bounce loop per call) and
// the wavefront of five kernels over path queues (k_vw_*).  Textually part of
// rt_api.cu (included there after the PathTracingMIS kernels), which holds
// RenderParams, the queue helpers and the BSDF dispatch these use.
#pragma once

// ---------------------------------------------------------------- VolPathTracing
// Integrator::evalTransmittance (Integrator.cpp:81-133)
// Out-of-line copies of the helpers the VolPath code calls from many sites.
// Inlined, every call site carried its own BVH traversal, tracking loop and
// BSDF switch; the resulting kernel missed the instruction cache on most
// issues.  One out-of-line copy each keeps the hot code small.
__device__ __noinline__ bool vp_trace(const DevScene &S, V3 o, V3 d, float mint, float maxt, Hit &h)
{
    return trace_ray<false>(S, o, d, mint, maxt, h);
}
__device__ __noinline__ Frame vp_frame(const DevScene &S, const Hit &h, V3 o, V3 d) { return hit_frame(S, h, o, d); }
// the frame of a hit that may be shaded, with its texture coordinates when
// the scene has textured BSDFs (a sphere's need the ray that found the hit)
__device__ __noinline__ Frame vp_frame_uv(const DevScene &S, const Hit &h, V3 o, V3 d, V2 &uv)
{
    if (S.has_textured) uv = hit_uv(S, h, o, d);
    return hit_frame(S, h, o, d);
}
__device__ __noinline__ C3 vp_medium_tr(const DevMedium &m, Ray r, Pcg32 &rng, int &limit)
{
    return medium_tr(m, r, rng, limit);
}
__device__ __noinline__ bool vp_medium_sample(const DevMedium &m, Ray r, Pcg32 &rng, float &t, C3 &w, C3 &em, int &limit)
{
    return medium_sample(m, r, rng, t, w, em, limit);
}
__device__ __noinline__ void vp_light_sample(const DevScene &S, int idx, V3 p, V2 u, LightRec &li)
{
    light_sample(S, idx, p, u, li);
}
__device__ __noinline__ float vp_light_pdf(const DevScene &S, int l, V3 p, V3 lp, V3 ln, V3 dir)
{
    return light_pdf(S, l, p, lp, ln, dir);
}

__device__ __noinline__ C3 eval_transmittance(const DevScene &S, Ray ray, int medium, Pcg32 &rng, int &limit)
{
    Ray tr = ray;
    C3 T = cfill(1.f);
    float dist = ray.maxt;
    bool first = true;
    for (int guard = 0; guard < 4096; guard++) {
        Hit h;
        bool inter = vp_trace(S, tr.o, tr.d, tr.mint, tr.maxt, h);
        if (inter && prim_bsdf(S, h.prim) >= 0) return cfill(0.f);
        if (inter) dist -= h.t;
        if (medium >= 0)
            T = T * vp_medium_tr(S.media[medium], make_ray(tr.o, tr.d, first ? tr.mint : 0.f, inter ? h.t : dist), rng, limit);
        first = false;
        if (!inter || iszero(T)) return T;
        V3 np = tr.o + h.t * tr.d;
        Frame f = vp_frame(S, h, tr.o, tr.d);
        tr = make_ray(np, tr.d, RT_EPSILON, dist);
        if (prim_interior(S, h.prim) != prim_exterior(S, h.prim))
            medium = dot(f.n, tr.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
    }
    limit = 1;
    return cfill(0.f);
}

// VolPathTracing::evalTransmittanceFromSampledBSDF (VolPathTracing.cpp:369-424)
__device__ __noinline__ C3 eval_tr_sampled(const DevScene &S, Ray ray, Pcg32 &rng, int medium, Hit &h, Frame &fr, V2 &uv,
                              bool &was, int &newm, int &limit)
{
    Ray tr = ray;
    C3 T = cfill(1.f);
    bool first = true;
    was = false;
    for (int guard = 0; guard < 4096; guard++) {
        Hit nh;
        was = vp_trace(S, tr.o, tr.d, tr.mint, tr.maxt, nh);
        if (was) { h = nh; fr = vp_frame_uv(S, h, tr.o, tr.d, uv); }
        if (medium >= 0)
            T = T * vp_medium_tr(S.media[medium], make_ray(tr.o, tr.d, first ? tr.mint : 0.f, was ? h.t : tr.maxt), rng, limit);
        if (was && prim_bsdf(S, h.prim) >= 0) return T;
        first = false;
        if (!was || iszero(T)) return T;
        V3 np = tr.o + h.t * tr.d;
        tr = make_ray(np, tr.d, RT_EPSILON, tr.maxt);
        if (prim_interior(S, h.prim) != prim_exterior(S, h.prim)) {
            medium = dot(fr.n, tr.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
            newm = medium;
        }
    }
    limit = 1;
    return T;
}

// Integrator::sampleAttenuatedLightDirect (Integrator.cpp:137-172)
__device__ __noinline__ C3 sample_attenuated_light(const DevScene &S, V3 p, Pcg32 &rng, LightRec &li, int medium, int &limit)
{
    C3 value = cfill(0.f);
    if (S.n_lights == 0) return value;
    V2 u = next2d(rng);
    float lw;
    int idx = cdf_sample_reuse(S.light_cdf, S.n_lights + 1, u.x, lw);
    vp_light_sample(S, idx, p, u, li);
    if (li.pdf > 0 && lum(li.intensity) > 0) {
        C3 tr = eval_transmittance(S, make_ray(p, li.to_light, RT_EPSILON, li.distance - RT_EPSILON), medium, rng, limit);
        li.pdf *= lw;
        value = (tr * li.intensity) / li.pdf;
    }
    return value;
}

// VolPathTracing::li (VolPathTracing.cpp:25-367)
// One VolPathTracing path as a resumable state: vol_start traces the camera
// ray, each vol_step runs one pass of the bounce loop of
// VolPathTracing::li (VolPathTracing.cpp:25-367) and returns false once the
// path has finished (its radiance is then in L).  The draws from the path's
// sample stream come in the same order as one uninterrupted loop.
struct VolState {
    C3 L, T;
    V2 uv;            // texture coordinates of h (scenes with textured BSDFs)
    float eta;
    int depth, medium, guard;
    bool emission, was;
    Ray ray;
    Hit h;
    Frame fr;
};

__device__ __forceinline__ void vol_start(const DevScene &S, VolState &st, Ray ray)
{
    st.L = cfill(0.f); st.T = cfill(1.f);
    st.eta = 1.f;
    st.depth = 0;
    st.emission = true;
    st.h.t = RT_MAX_REAL; st.h.u = st.h.v = 0.f; st.h.prim = -1;
    st.fr.p = v3(0, 0, 0); st.fr.n = st.fr.s = st.fr.t = v3(0, 0, 0);
    st.ray = ray;
    Hit nh;
    st.was = vp_trace(S, ray.o, ray.d, ray.mint, ray.maxt, nh);
    st.uv = v2(0.f, 0.f);
    if (st.was) { st.h = nh; st.fr = vp_frame_uv(S, nh, ray.o, ray.d, st.uv); }
    st.medium = S.cam.medium;
    st.guard = 0;
}

__device__ bool vol_step(const DevScene &S, VolState &st, Pcg32 &rng, int max_depth, int min_depth, int &limit)
{
    if (st.depth >= max_depth) return false;
    if (++st.guard > (1 << 16)) { limit = 1; return false; }
    const int env = S.env_light;
    Ray &ray = st.ray;
    Hit &h = st.h;
    Frame &fr = st.fr;
    C3 &L = st.L, &T = st.T;
    bool &was = st.was;
    int &medium = st.medium;
    Hit nh;
    float t = 0.f;
    C3 wm = cfill(0.f), em = cfill(0.f);
    bool scattered = false;
    if (medium >= 0) scattered = vp_medium_sample(S.media[medium], make_ray(ray.o, ray.d, ray.mint, h.t), rng, t, wm, em, limit);
    if (scattered) {
        const DevMedium &M = S.media[medium];
        L = L + T * em;
        T = T * wm;
        fr.p = ray.o + t * ray.d;
        LightRec li;
        li.point = li.to_light = li.normal = v3(0, 0, 0);
        li.intensity = cfill(0.f); li.distance = 0.f; li.pdf = 0.f; li.delta = 0;
        C3 value = sample_attenuated_light(S, fr.p, rng, li, medium, limit);
        if (!iszero(value)) {
            // a delta light's sample takes a zero phase pdf (VolPathTracing.cpp:86)
            float pf = li.delta ? 0.f : phase_eval(M, li.to_light, -ray.d);
            float w = power_heuristic(li.pdf, pf);
            float ev = phase_eval(M, li.to_light, -ray.d);
            L = L + ((T * value) * ev) * w;
        }
        V3 wo; float pfpdf;
        float pfw = phase_sample(M, -ray.d, next2d(rng), wo, pfpdf);
        ray = make_ray(fr.p, wo, 0.f, ray.maxt);
        int newm = -1;
        C3 tr = eval_tr_sampled(S, ray, rng, medium, h, fr, st.uv, was, newm, limit);
        T = T * pfw;
        if (was) {
            int hl = prim_light(S, h.prim);
            if (hl >= 0) {
                C3 Le = area_le(S, hl, -ray.d, fr.n);
                float pl = vp_light_pdf(S, hl, fr.p, li.point, li.normal, li.to_light);
                float w = power_heuristic(pfpdf, pl);
                L = L + ((T * Le) * tr) * w;
            }
        }
    } else {
        if (medium >= 0) {
            L = L + T * em;
            T = T * wm;
        }
        if (!was) {
            if (st.emission && env >= 0) L = L + T * env_le(S.lights[env], ray.d);
            return false;
        }
        int b = prim_bsdf(S, h.prim);
        if (b < 0) {
            // null boundary: pass through without a bounce (no depth, no RR)
            ray = make_ray(fr.p, ray.d, RT_EPSILON, RT_MAX_REAL);
            if (prim_interior(S, h.prim) != prim_exterior(S, h.prim))
                medium = dot(fr.n, ray.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
            was = vp_trace(S, ray.o, ray.d, ray.mint, ray.maxt, nh);
            if (was) { h = nh; fr = vp_frame_uv(S, h, ray.o, ray.d, st.uv); }
            return true;
        }
        // a textured BSDF: a copy with its textures applied at the hit
        const DevBsdf *Bp = &S.bsdfs[b];
        DevBsdf Bl;
        if (Bp->textured) {
            Bl = *Bp;
            tex_apply(S, Bl, st.uv);
            Bp = &Bl;
        }
        const DevBsdf &B = *Bp;
        int hl = prim_light(S, h.prim);
        if (st.emission && hl >= 0) L = L + T * area_le(S, hl, -ray.d, fr.n);
        LightRec li;
        li.point = li.to_light = li.normal = v3(0, 0, 0);
        li.intensity = cfill(0.f); li.distance = 0.f; li.pdf = 0.f; li.delta = 0;
        C3 value = sample_attenuated_light(S, fr.p, rng, li, medium, limit);
        if (!iszero(value)) {
            V3 wi = to_local(fr, li.to_light), wo = to_local(fr, -ray.d);
            float ct = fabsf(wi.z);
            float bp = li.delta ? 0.f : any_bsdf_pdf(B, wi, wo);   // VolPathTracing.cpp:222
            float w = power_heuristic(li.pdf, bp);
            L = L + (((T * value) * any_bsdf_eval(B, wi, wo)) * ct) * w;
        }
        BsdfRec r;
        r.wi = to_local(fr, -ray.d); r.wo = v3(0, 0, 0);
        r.type = BT_ALL; r.rel_eta = 1.f; r.pdf = -1.f;
        V2 bu = next2d(rng);
        C3 f = any_bsdf_sample(B, r, bu, rng.state);
        if (iszero(f)) return false;
        V3 pfrom = fr.p;
        ray = make_ray(fr.p, to_world(fr, r.wo), RT_EPSILON, RT_MAX_REAL);
        if (prim_interior(S, h.prim) != prim_exterior(S, h.prim))
            medium = dot(fr.n, ray.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
        int caught = -1;
        bool isenv = false;
        C3 Le = cfill(0.f);
        int newm = -1;
        C3 tr = eval_tr_sampled(S, ray, rng, medium, h, fr, st.uv, was, newm, limit);
        if (was) {
            int nl = prim_light(S, h.prim);
            if (nl >= 0) { caught = nl; Le = area_le(S, nl, -ray.d, fr.n); }
        } else if (newm < 0) {
            if (env >= 0) { caught = env; isenv = true; Le = env_le(S.lights[env], ray.d); }
        }
        if (caught >= 0) {
            float pl = (r.type & BT_DELTA) ? 0.f : vp_light_pdf(S, caught, pfrom, fr.p, fr.n, ray.d);
            float w = power_heuristic(r.pdf, pl);
            L = L + (((T * Le) * f) * tr) * w;
            if (isenv && medium < 0) return false;
        }
        T = T * f;
        st.eta *= r.rel_eta;
    }
    if (st.depth >= min_depth) {
        float stop = smin(0.95f, cmax(T) * st.eta * st.eta);
        if (next1d(rng) < stop) T = T / stop;
        else return false;
    }
    was = vp_trace(S, ray.o, ray.d, ray.mint, ray.maxt, nh);
    if (was) { h = nh; fr = vp_frame_uv(S, h, ray.o, ray.d, st.uv); }
    st.emission = false;
    st.depth++;
    return true;
}

// Persistent VolPath kernel with per-lane path regeneration: a lane whose
// path finished takes the next path of the batch (warp-aggregated atomic),
// so the lanes of a warp stay busy however long each path runs.
// The kernel waits on memory (grid lookups, traversal) far more than it
// computes: full occupancy (16 blocks of 128 threads per SM, 32 registers,
// the rest spilled to L1-resident local memory) ran it 1.8x faster than the
// 114-register version at 4 blocks per SM.
#ifndef RT_VOLPATH_MINB
#define RT_VOLPATH_MINB 16
#endif
#ifndef RT_VOLPATH_GRID
#define RT_VOLPATH_GRID 32
#endif
__global__ void __launch_bounds__(128, RT_VOLPATH_MINB) k_volpath(RenderParams P, int *work)
{
    const int lane = threadIdx.x & 31;
    int limit = 0;
    VolState st;
    Pcg32 rng;
    rng.state = rng.inc = 0;
    int slot = -1;
    bool active = false, more = true;
    for (;;) {
        const unsigned need = __ballot_sync(0xffffffffu, !active && more);
        if (need) {
            int base = 0;
            const int leader = __ffs(need) - 1;
            if (lane == leader) base = atomicAdd(work, __popc(need));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (!active && more) {
                int q = base + __popc(need & ((1u << lane) - 1));
                if (q < P.n_paths) {
                    slot = q;
                    int flags;
                    rng = path_rng(w_rng(P.W, slot), flags);
                    float4 ro = w_ray_o(P.W, slot), rd = w_ray_d(P.W, slot);
                    vol_start(P.S, st, make_ray(xyz(ro), xyz(rd), ro.w, rd.w));
                    active = true;
                } else {
                    more = false;
                }
            }
        }
        if (!__any_sync(0xffffffffu, active)) break;
        if (active && !vol_step(P.S, st, rng, P.max_depth, P.min_depth, limit)) {
            w_done(P.W, slot, st.L);
            active = false;
        }
    }
    if (limit) atomicOr(P.limit_flag, RT_LIM_VOLPATH);
}

// ---------------------------------------------------------------- VolPathTracing wavefront
// The same bounce loop as vol_step, split at its loops into kernels, each
// over a queue of paths in HBM.  One round runs one vol_step of every live
// path (a bounce, or a null-boundary crossing, which the reference also
// runs as one pass of its loop):
//   k_vw_trace_step [trace queue]  closest hit of a camera ray or a ray behind
//                                  a null boundary (vol_step's last trace is
//                                  kept from the sampled ray's first segment),
//                                  then depth and guard, delta
//                                  tracking through the medium, then either
//                                  the scatter point or the surface
//                                  (emission, null boundary, env miss), and
//                                  the light pick and sample of
//                                  sampleAttenuatedLightDirect
//   k_vw_shadow  [shadow queue]    the light sample's transmittance
//                                  (evalTransmittance: traces through null
//                                  boundaries, ratio tracking in media)
//   k_vw_sample_surface [surface sample queue]  the light sample's MIS
//                                  contribution, the BSDF sample and the new
//                                  ray
//   k_vw_trsamp_finish [trsamp queue]  evalTransmittanceFromSampledBSDF
//                                  along it, then emission MIS of what the
//                                  sampled ray found, throughput, Russian
//                                  roulette
//   k_vw_scatter [medium sample queue]  the same three steps for scatter
//                                  points in media (phase function), in
//                                  one kernel
// Each path's draws come in the order of one uninterrupted vol_step, so a
// path's radiance is the megakernel's.  The hit frame is not stored: it is
// rebuilt from the hit, the origin of the ray segment that found it and the
// path's direction (hit_frame), which is what the megakernel holds.  Queue
// counts live in the round's RoundCounters: trace = closest (queue
// q_closest in even rounds, q_mat[0] in odd ones), shadow = shadow, sample =
// mat[1] (medium vertices) and mat[4] (surface vertices), trsamp = mat[2];
// the next round's trace queue is the next counters' closest.
enum { VF_FIRST = F_FIRST, VF_EMISSION = 2, VF_WAS = 4, VF_SCAT = 8, VF_NULLX = 16, VF_DELTA = 32, VF_NEWM = 64,
       VF_HASVAL = 128, VF_GUARD_SHIFT = 8 };

// Integrator::sampleAttenuatedLightDirect (Integrator.cpp:137-172) up to its
// shadow ray: the light pick and sample.  Returns whether the shadow ray's
// transmittance is needed; li is zero without lights.
__device__ __forceinline__ bool vw_light_pick(const DevScene &S, V3 p, Pcg32 &rng, LightRec &li, float &lw)
{
    li.point = li.to_light = li.normal = v3(0, 0, 0);
    li.intensity = cfill(0.f); li.distance = 0.f; li.pdf = 0.f; li.delta = 0;
    lw = 0.f;
    if (S.n_lights == 0) return false;
    V2 u = next2d(rng);
    int idx = cdf_sample_reuse(S.light_cdf, S.n_lights + 1, u.x, lw);
    light_sample(S, idx, p, u, li);
    return li.pdf > 0 && lum(li.intensity) > 0;
}
__device__ __forceinline__ void vw_store_light(const RenderParams &P, int slot, const LightRec &li, V3 p, float lw)
{
    w_v_p(P.W, slot) = f4(p, lw);
    w_v_li0(P.W, slot) = f4(li.to_light, li.distance);
    w_v_li1(P.W, slot) = f4(li.point, li.pdf);
    w_v_li2(P.W, slot) = f4(li.normal, li.delta ? 1.f : 0.f);
    w_v_val(P.W, slot) = f4c(li.intensity, 0.f);
}

// evalTransmittanceFromSampledBSDF (VolPathTracing.cpp:369-424), as
// eval_tr_sampled, reporting the segment origin of the hit instead of its
// frame, and in h1 and was1 the hit of the ray's first segment: what the
// trace of the same ray at the end of the pass would find
__device__ __forceinline__ C3 vw_tr_sampled(const DevScene &S, Ray ray, Pcg32 &rng, int medium, Hit &h, V3 &seg, bool &was,
                                         Hit &h1, bool &was1, int &newm, int &limit)
{
    Ray tr = ray;
    C3 T = cfill(1.f);
    bool first = true;
    was = false;
    for (int guard = 0; guard < 4096; guard++) {
        Hit nh;
        was = trace_ray<false>(S, tr.o, tr.d, tr.mint, tr.maxt, nh);
        if (was) { h = nh; seg = tr.o; }
        if (first) { h1 = h; was1 = was; }
        if (medium >= 0)
            T = T * medium_tr(S.media[medium], make_ray(tr.o, tr.d, first ? tr.mint : 0.f, was ? h.t : tr.maxt), rng, limit);
        if (was && prim_bsdf(S, h.prim) >= 0) return T;
        first = false;
        if (!was || iszero(T)) return T;
        V3 np = tr.o + h.t * tr.d;
        const V3 seg_o = tr.o;
        tr = make_ray(np, tr.d, RT_EPSILON, tr.maxt);
        if (prim_interior(S, h.prim) != prim_exterior(S, h.prim)) {
            Frame f = hit_frame(S, h, seg_o, tr.d);
            medium = dot(f.n, tr.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
            newm = medium;
        }
    }
    limit = 1;
    return T;
}

__device__ __forceinline__ C3 vw_transmittance(const DevScene &S, Ray ray, int medium, Pcg32 &rng, int &limit)
{
    Ray tr = ray;
    C3 T = cfill(1.f);
    float dist = ray.maxt;
    bool first = true;
    for (int guard = 0; guard < 4096; guard++) {
        Hit h;
        bool inter = trace_ray<false>(S, tr.o, tr.d, tr.mint, tr.maxt, h);
        if (inter && prim_bsdf(S, h.prim) >= 0) return cfill(0.f);
        if (inter) dist -= h.t;
        if (medium >= 0)
            T = T * medium_tr(S.media[medium], make_ray(tr.o, tr.d, first ? tr.mint : 0.f, inter ? h.t : dist), rng, limit);
        first = false;
        if (!inter || iszero(T)) return T;
        V3 np = tr.o + h.t * tr.d;
        Frame f = hit_frame(S, h, tr.o, tr.d);
        tr = make_ray(np, tr.d, RT_EPSILON, dist);
        if (prim_interior(S, h.prim) != prim_exterior(S, h.prim))
            medium = dot(f.n, tr.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
    }
    limit = 1;
    return cfill(0.f);
}

// Each wavefront kernel calls its traversal, tracking, frame and light code
// from one place, so all of it is inline: the calls of the out-of-line copies
// (the vp_ functions, which the persistent kernel shares among many places)
// passed rays, hits and stream states through local memory and waited on
// instruction fetch (7-10 cycles per issue).  128^3 grid-medium frame,
// 512^2 x 128 spp: 61.5 ms with the calls, 51.7 ms inline, 50.4 ms with 6
// blocks per SM (80 registers, hardly any spills) instead of 8.
// resident 128-thread blocks per SM of each wavefront kernel (its launch
// bound and its grid); 5 and 7 for any one of them were within 1 %
#ifndef RT_VW_MINB
#define RT_VW_MINB 6
#endif
#ifndef RT_VW_MINB_STEP
#define RT_VW_MINB_STEP RT_VW_MINB
#endif
#ifndef RT_VW_MINB_SHADOW
#define RT_VW_MINB_SHADOW RT_VW_MINB
#endif
#ifndef RT_VW_MINB_SAMPLE
#define RT_VW_MINB_SAMPLE RT_VW_MINB
#endif
#ifndef RT_VW_MINB_TRSAMP
#define RT_VW_MINB_TRSAMP RT_VW_MINB
#endif
// Each kernel's work on one path is a function of its own (vw_*_path), which
// returns the queues the path goes to (bits, in the order of the kernel's
// queue list); k_vw_tail calls them one after another.
// whole warps run every pass of the loop (VW_LIVE: the lane has a path), so
// that the pushes at its end are the warp's
#define VW_LOOP(COUNT, QUEUE)                                                                      \
    const int n_ = (COUNT);                                                                        \
    const int *qin_ = (QUEUE);                                                                     \
    for (int i_ = blockIdx.x * blockDim.x + threadIdx.x; (i_ & ~31) < n_; i_ += gridDim.x * blockDim.x)
#define VW_LIVE (i_ < n_)

// The trace queue of a round: rounds alternate between two arrays, since
// the kernel that reads round r's queue also appends to round r + 1's.
__device__ __forceinline__ int *vw_trace_queue(const RenderParams &P, int round)
{
    return (round & 1) ? P.W.q_mat[0] : P.W.q_closest;
}

// k_vw_trace_step: the closest hit of the path's ray (the trace that ends
// vol_step, vol_start or a null crossing), then the step over that hit:
// depth and guard, delta tracking through the medium, then the scatter point
// or the surface (emission, null boundary, env miss), and the light pick and
// sample of sampleAttenuatedLightDirect.  The trace's hit, segment origin,
// flags and depth stay in registers for the step; the hit is stored for the
// kernels after it.
// The reference traces a bounce's ray twice (VolPathTracing.cpp:105, :360).
// The first segment of the sampled ray's transmittance is that same ray, with
// the same bounds, and a trace draws no numbers, so the pass's last trace
// takes its hit from there (vw_finish_one stores it); only camera rays and
// the rays behind a null boundary are traced here.  They come first in the
// queue, so few warps mix the two.  128^3 grid-medium frame: 64.4 -> 63.6 ms.
__device__ __forceinline__ unsigned vw_step_path(const RenderParams &P, const DevScene &S, int slot, int &limit)
{
    unsigned want = 0;
    // ---- the trace
    int flags;
    Pcg32 rng = path_rng(w_rng(P.W, slot), flags);
    const float4 ro = w_ray_o(P.W, slot), rd = w_ray_d(P.W, slot);
    float4 tpv = make_float4(1.f, 1.f, 1.f, 1.f), radv = make_float4(0.f, 0.f, 0.f, 0.f);
    if (!(flags & VF_FIRST)) w_load2(P.W.acc, slot, tpv, radv);
    float4 seg;
    Hit h;
    const bool traces = (flags & (VF_FIRST | VF_NULLX)) != 0;
    if (flags & VF_FIRST) {
        h.t = RT_MAX_REAL; h.u = h.v = 0.f; h.prim = -1;
        seg = make_float4(0.f, 0.f, 0.f, __int_as_float(S.cam.medium));
        flags = VF_EMISSION;
    } else {
        const float4 hv = P.W.hit[slot];
        h.t = hv.x; h.u = hv.y; h.v = hv.z; h.prim = __float_as_int(hv.w);
        seg = w_v_seg(P.W, slot);
        if (!(flags & VF_NULLX)) {   // the trace that ends a bounce
            flags &= ~VF_EMISSION;
            radv.w = __int_as_float(__float_as_int(radv.w) + 1);
        }
    }
    if (traces) {
        Hit nh;
        const bool was = trace_ray<false>(S, xyz(ro), xyz(rd), ro.w, rd.w, nh);
        if (was) {
            h = nh;
            seg = make_float4(ro.x, ro.y, ro.z, seg.w);
        }
        flags = (flags & ~(VF_NULLX | VF_WAS)) | (was ? VF_WAS : 0);
        P.W.hit[slot] = make_float4(h.t, h.u, h.v, __int_as_float(h.prim));
    }
    // ---- the step
    C3 L = rgb(radv), T = rgb(tpv);
    const int depth = __float_as_int(radv.w);
    bool push_shadow = false, push_sample = false, push_trace = false;
    int guard = (flags >> VF_GUARD_SHIFT) + 1;
    if (depth >= P.max_depth) {
        w_done(P.W, slot, L);
    } else if (guard > (1 << 16)) {
        limit = 1;
        w_done(P.W, slot, L);
    } else {
        Ray ray = make_ray(xyz(ro), xyz(rd), ro.w, rd.w);
        int medium = __float_as_int(seg.w);
        float t = 0.f;
        C3 wm = cfill(0.f), em = cfill(0.f);
        bool scattered = false;
        if (medium >= 0)
            scattered = medium_sample(S.media[medium], make_ray(ray.o, ray.d, ray.mint, h.t), rng, t, wm, em, limit);
        bool done = false, vertex = false;
        V3 vp = v3(0.f, 0.f, 0.f);
        if (scattered) {
            L = L + T * em;
            T = T * wm;
            vp = ray.o + t * ray.d;
            flags |= VF_SCAT;
            vertex = true;
        } else {
            flags &= ~VF_SCAT;
            if (medium >= 0) {
                L = L + T * em;
                T = T * wm;
            }
            if (!(flags & VF_WAS)) {
                if ((flags & VF_EMISSION) && S.env_light >= 0) L = L + T * env_le(S.lights[S.env_light], ray.d);
                done = true;
            } else {
                Frame fr = hit_frame(S, h, xyz(seg), ray.d);
                if (prim_bsdf(S, h.prim) < 0) {
                    // null boundary: through, without a bounce
                    ray = make_ray(fr.p, ray.d, RT_EPSILON, RT_MAX_REAL);
                    if (prim_interior(S, h.prim) != prim_exterior(S, h.prim))
                        medium = dot(fr.n, ray.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
                    w_ray_o(P.W, slot) = f4(ray.o, ray.mint);
                    w_ray_d(P.W, slot) = f4(ray.d, ray.maxt);
                    flags |= VF_NULLX;
                    push_trace = true;
                } else {
                    int hl = prim_light(S, h.prim);
                    if ((flags & VF_EMISSION) && hl >= 0) L = L + T * area_le(S, hl, -ray.d, fr.n);
                    vp = fr.p;
                    vertex = true;
                }
            }
        }
        if (vertex) {
            LightRec li;
            float lw;
            push_shadow = vw_light_pick(S, vp, rng, li, lw);
            push_sample = !push_shadow;
            vw_store_light(P, slot, li, vp, lw);
            flags &= ~VF_HASVAL;
        }
        if (done) {
            w_done(P.W, slot, L);
        } else {
            w_rad(P.W, slot) = f4c(L, __int_as_float(depth));
            w_tp(P.W, slot) = f4c(T, tpv.w);
            w_v_seg(P.W, slot) = make_float4(seg.x, seg.y, seg.z, __int_as_float(medium));
            w_rng(P.W, slot) = path_rng_pack(rng, (flags & ((1 << VF_GUARD_SHIFT) - 1)) | (guard << VF_GUARD_SHIFT));
        }
    }
    want = push_shadow ? 1u : push_sample ? ((flags & VF_SCAT) ? 2u : 4u) : push_trace ? 8u : 0u;
    return want;
}
__global__ void __launch_bounds__(128, RT_VW_MINB_STEP) k_vw_trace_step(RenderParams P, int round)
{
    round = cur_round(P, round);
    const DevScene &S = P.S;
    RoundCounters *C = &P.W.cnt[round];
    RoundCounters *Cn = &P.W.cnt[round + 1];
    int *next_q = vw_trace_queue(P, round + 1);
    int limit = 0;
    int *const out_q[4] = {P.W.q_shadow, P.W.q_mat[1], P.W.q_mat[4], next_q};
    int *const out_n[4] = {&C->shadow, &C->mat[1], &C->mat[4], &Cn->closest};
    VW_LOOP(C->closest, vw_trace_queue(P, round))
    {
        const int slot = VW_LIVE ? qin_[i_] : 0;
        const unsigned want = VW_LIVE ? vw_step_path(P, S, slot, limit) : 0u;
        q_push(out_q, out_n, slot, want);
    }
    if (limit) atomicOr(P.limit_flag, RT_LIM_VOLPATH);
}

__device__ __forceinline__ unsigned vw_shadow_path(const RenderParams &P, const DevScene &S, int slot, int &limit)
{
    unsigned want = 0;
    int flags;
    Pcg32 rng = path_rng(w_rng(P.W, slot), flags);
    float4 pv = w_v_p(P.W, slot), l0 = w_v_li0(P.W, slot), l1 = w_v_li1(P.W, slot), iv = w_v_val(P.W, slot);
    const int medium = __float_as_int(w_v_seg(P.W, slot).w);
    C3 tr = vw_transmittance(S, make_ray(xyz(pv), xyz(l0), RT_EPSILON, l0.w - RT_EPSILON), medium, rng, limit);
    float pdf = l1.w * pv.w;
    C3 value = (tr * rgb(iv)) / pdf;
    w_v_li1(P.W, slot) = make_float4(l1.x, l1.y, l1.z, pdf);
    w_v_val(P.W, slot) = f4c(value, 0.f);
    w_rng(P.W, slot) = path_rng_pack(rng, flags | VF_HASVAL);
    want = (flags & VF_SCAT) ? 1u : 2u;
    return want;
}
__global__ void __launch_bounds__(128, RT_VW_MINB_SHADOW) k_vw_shadow(RenderParams P, int round)
{
    round = cur_round(P, round);
    const DevScene &S = P.S;
    RoundCounters *C = &P.W.cnt[round];
    int limit = 0;
    int *const out_q[2] = {P.W.q_mat[1], P.W.q_mat[4]};
    int *const out_n[2] = {&C->mat[1], &C->mat[4]};
    VW_LOOP(C->shadow, P.W.q_shadow)
    {
        const int slot = VW_LIVE ? qin_[i_] : 0;
        const unsigned want = VW_LIVE ? vw_shadow_path(P, S, slot, limit) : 0u;
        q_push(out_q, out_n, slot, want);
    }
    if (limit) atomicOr(P.limit_flag, RT_LIM_VOLPATH);
}

// k_vw_sample_surface: the paths whose vertex is on a surface (sample queue
// mat[4]): the light sample's MIS with the BSDF (textures applied), the BSDF
// sample and the new ray.  Scatter points in media (mat[1]) go through
// k_vw_scatter, which continues into the sampled ray's transmittance.
__device__ __forceinline__ unsigned vw_surface_path(const RenderParams &P, const DevScene &S, int slot)
{
    unsigned want = 0;
    int flags;
    Pcg32 rng = path_rng(w_rng(P.W, slot), flags);
    float4 radv = w_rad(P.W, slot), tpv = w_tp(P.W, slot);
    C3 L = rgb(radv), T = rgb(tpv);
    float4 ro = w_ray_o(P.W, slot), rd = w_ray_d(P.W, slot);
    Ray ray = make_ray(xyz(ro), xyz(rd), ro.w, rd.w);
    float4 seg = w_v_seg(P.W, slot);
    int medium = __float_as_int(seg.w);
    const bool hasval = flags & VF_HASVAL;
    C3 value = hasval ? rgb(w_v_val(P.W, slot)) : cfill(0.f);
    bool push = true;
    {
        float4 hv = P.W.hit[slot];
        Hit h; h.t = hv.x; h.u = hv.y; h.v = hv.z; h.prim = __float_as_int(hv.w);
        Frame fr = hit_frame(S, h, xyz(seg), ray.d);
        const DevBsdf *Bp = &S.bsdfs[prim_bsdf(S, h.prim)];
        DevBsdf Bl;
        if (Bp->textured) {
            Bl = *Bp;
            tex_apply(S, Bl, hit_uv(S, h, xyz(seg), ray.d));
            Bp = &Bl;
        }
        const DevBsdf &B = *Bp;
        if (!iszero(value)) {
            V3 to_light = xyz(w_v_li0(P.W, slot));
            float lpdf = w_v_li1(P.W, slot).w;
            V3 wi = to_local(fr, to_light), wo = to_local(fr, -ray.d);
            float ct = fabsf(wi.z);
            float bp = w_v_li2(P.W, slot).w != 0.f ? 0.f : any_bsdf_pdf(B, wi, wo);
            float w = power_heuristic(lpdf, bp);
            L = L + (((T * value) * any_bsdf_eval(B, wi, wo)) * ct) * w;
        }
        BsdfRec r;
        r.wi = to_local(fr, -ray.d); r.wo = v3(0, 0, 0);
        r.type = BT_ALL; r.rel_eta = 1.f; r.pdf = -1.f;
        V2 bu = next2d(rng);
        C3 f = any_bsdf_sample(B, r, bu, rng.state);
        if (iszero(f)) {
            w_done(P.W, slot, L);
            push = false;
        } else {
            ray = make_ray(fr.p, to_world(fr, r.wo), RT_EPSILON, RT_MAX_REAL);
            if (prim_interior(S, h.prim) != prim_exterior(S, h.prim))
                medium = dot(fr.n, ray.d) < 0.f ? prim_interior(S, h.prim) : prim_exterior(S, h.prim);
            w_bs(P.W, slot) = f4c(f, r.pdf);
            tpv.w *= r.rel_eta;   // eta as the end of the pass reads it
            flags = (r.type & BT_DELTA) ? (flags | VF_DELTA) : (flags & ~VF_DELTA);
        }
    }
    if (push) {
        w_tp(P.W, slot) = tpv;
        w_rad(P.W, slot) = f4c(L, radv.w);
        w_ray_o(P.W, slot) = f4(ray.o, ray.mint);
        w_ray_d(P.W, slot) = f4(ray.d, ray.maxt);
        w_v_seg(P.W, slot) = make_float4(seg.x, seg.y, seg.z, __int_as_float(medium));
        w_rng(P.W, slot) = path_rng_pack(rng, flags);
    }
    want = push ? 1u : 0u;
    return want;
}
__global__ void __launch_bounds__(128, RT_VW_MINB_SAMPLE) k_vw_sample_surface(RenderParams P, int round)
{
    round = cur_round(P, round);
    const DevScene &S = P.S;
    RoundCounters *C = &P.W.cnt[round];
    int *const out_q[1] = {P.W.q_mat[2]};
    int *const out_n[1] = {&C->mat[2]};
    VW_LOOP(C->mat[4], P.W.q_mat[4])
    {
        const int slot = VW_LIVE ? qin_[i_] : 0;
        const unsigned want = VW_LIVE ? vw_surface_path(P, S, slot) : 0u;
        q_push(out_q, out_n, slot, want);
    }
}

// The end of a pass once the sampled ray's transmittance is known: emission
// MIS of what the ray found, throughput, Russian roulette
// (VolPathTracing.cpp:300-367).  ro, rd: the sampled ray; h, seg, was,
// flags: what evalTransmittanceFromSampledBSDF reported; L: the radiance with
// this vertex's light-sample MIS; h1, was1, seg1: the first segment's hit and
// its origin, kept for the next pass as its trace.  Returns whether the path goes on (to the
// next round's trace queue, with its sampled ray).
template <bool SCAT>
__device__ __forceinline__ bool vw_finish_one(const RenderParams &P, const DevScene &S, int slot, int flags, Pcg32 rng,
                                              float4 ro, float4 rd, float4 seg, const Hit &h, bool was, const Hit &h1,
                                              bool was1, float4 seg1, C3 tr, C3 L, int depth, float4 tpv, float4 bsv)
{
    C3 T = rgb(tpv);
    float eta = tpv.w;
    const V3 d = xyz(rd);
    const int medium = __float_as_int(seg.w);
    bool done = false;
    if (SCAT) {
        T = T * rgb(bsv);
        if (was) {
            int hl = prim_light(S, h.prim);
            if (hl >= 0) {
                Frame fr = hit_frame(S, h, xyz(seg), d);
                C3 Le = area_le(S, hl, -d, fr.n);
                float pl = light_pdf(S, hl, fr.p, xyz(w_v_li1(P.W, slot)), xyz(w_v_li2(P.W, slot)),
                                        xyz(w_v_li0(P.W, slot)));
                float w = power_heuristic(bsv.w, pl);
                L = L + ((T * Le) * tr) * w;
            }
        }
    } else {
        const C3 f = rgb(bsv);
        int caught = -1;
        bool isenv = false;
        C3 Le = cfill(0.f);
        Frame fr;
        fr.p = fr.n = v3(0, 0, 0);
        if (was) {
            int nl = prim_light(S, h.prim);
            if (nl >= 0) {
                caught = nl;
                fr = hit_frame(S, h, xyz(seg), d);
                Le = area_le(S, nl, -d, fr.n);
            }
        } else if (!(flags & VF_NEWM)) {
            // a miss: the environment (its pdf depends on the direction only)
            if (S.env_light >= 0) { caught = S.env_light; isenv = true; Le = env_le(S.lights[S.env_light], d); }
        }
        if (caught >= 0) {
            float pl = (flags & VF_DELTA) ? 0.f : light_pdf(S, caught, xyz(w_v_p(P.W, slot)), fr.p, fr.n, d);
            float w = power_heuristic(bsv.w, pl);
            L = L + (((T * Le) * f) * tr) * w;
            if (isenv && medium < 0) done = true;
        }
        if (!done) T = T * f;
    }
    if (!done && depth >= P.min_depth) {
        float stop = smin(0.95f, cmax(T) * eta * eta);
        if (next1d(rng) < stop) T = T / stop;
        else done = true;
    }
    if (done) {
        w_done(P.W, slot, L);
    } else {
        w_ray_o(P.W, slot) = ro;
        w_ray_d(P.W, slot) = rd;
        P.W.hit[slot] = make_float4(h1.t, h1.u, h1.v, __int_as_float(h1.prim));
        w_v_seg(P.W, slot) = seg1;
        w_rng(P.W, slot) = path_rng_pack(rng, (flags & ~VF_WAS) | (was1 ? VF_WAS : 0));
        w_rad(P.W, slot) = f4c(L, __int_as_float(depth));
        w_tp(P.W, slot) = f4c(T, eta);
    }
    return !done;
}

// k_vw_trsamp_finish: evalTransmittanceFromSampledBSDF along the ray that
// k_vw_sample_surface sampled at a surface vertex, then vw_finish_one
__device__ __forceinline__ unsigned vw_trsamp_path(const RenderParams &P, const DevScene &S, int slot, int &limit)
{
    unsigned want = 0;
    int flags;
    Pcg32 rng = path_rng(w_rng(P.W, slot), flags);
    const float4 ro = w_ray_o(P.W, slot), rd = w_ray_d(P.W, slot);
    const float4 hv = P.W.hit[slot];
    Hit h; h.t = hv.x; h.u = hv.y; h.v = hv.z; h.prim = __float_as_int(hv.w);
    float4 seg = w_v_seg(P.W, slot);
    V3 so = xyz(seg);
    Hit h1;
    bool was, was1;
    int newm = -1;
    const C3 tr = vw_tr_sampled(S, make_ray(xyz(ro), xyz(rd), ro.w, rd.w), rng, __float_as_int(seg.w), h, so,
                                was, h1, was1, newm, limit);
    flags = (flags & ~VF_NEWM) | (newm >= 0 ? VF_NEWM : 0);
    const float4 seg1 = was1 ? make_float4(ro.x, ro.y, ro.z, seg.w) : seg;
    seg = make_float4(so.x, so.y, so.z, seg.w);
    const float4 radv = w_rad(P.W, slot);
    want = vw_finish_one<false>(P, S, slot, flags, rng, ro, rd, seg, h, was, h1, was1, seg1, tr, rgb(radv), __float_as_int(radv.w),
                         w_tp(P.W, slot), w_bs(P.W, slot))
               ? 1u
               : 0u;
    return want;
}
__global__ void __launch_bounds__(128, RT_VW_MINB_TRSAMP) k_vw_trsamp_finish(RenderParams P, int round)
{
    round = cur_round(P, round);
    const DevScene &S = P.S;
    RoundCounters *C = &P.W.cnt[round];
    RoundCounters *Cn = &P.W.cnt[round + 1];
    int *next_q = vw_trace_queue(P, round + 1);
    int limit = 0;
    int *const out_q[1] = {next_q};
    int *const out_n[1] = {&Cn->closest};
    VW_LOOP(C->mat[2], P.W.q_mat[2])
    {
        const int slot = VW_LIVE ? qin_[i_] : 0;
        const unsigned want = VW_LIVE ? vw_trsamp_path(P, S, slot, limit) : 0u;
        q_push(out_q, out_n, slot, want);
    }
    if (limit) atomicOr(P.limit_flag, RT_LIM_VOLPATH);
}

// k_vw_scatter: a scatter point in a medium (sample queue mat[1]) through the
// rest of its pass in one kernel: the phase sample and the new ray
// (the phase function's), the transmittance along it, then the light
// sample's MIS with the phase function (no draws, so its place after the
// transmittance leaves the path's stream as it was) and vw_finish_one
__device__ __forceinline__ unsigned vw_scatter_path(const RenderParams &P, const DevScene &S, int slot, int &limit)
{
    unsigned want = 0;
    int flags;
    Pcg32 rng = path_rng(w_rng(P.W, slot), flags);
    float4 seg = w_v_seg(P.W, slot);
    const int medium = __float_as_int(seg.w);
    float4 rd = w_ray_d(P.W, slot);
    V3 wo;
    float pfpdf;
    const float pfw = phase_sample(S.media[medium], -xyz(rd), next2d(rng), wo, pfpdf);
    const float4 ro = f4(xyz(w_v_p(P.W, slot)), 0.f);
    rd = f4(wo, rd.w);
    const float4 hv = P.W.hit[slot];
    Hit h; h.t = hv.x; h.u = hv.y; h.v = hv.z; h.prim = __float_as_int(hv.w);
    V3 so = xyz(seg);
    Hit h1;
    bool was, was1;
    int newm = -1;
    const C3 tr = vw_tr_sampled(S, make_ray(xyz(ro), wo, 0.f, rd.w), rng, medium, h, so, was, h1, was1, newm, limit);
    flags = (flags & ~VF_NEWM) | (newm >= 0 ? VF_NEWM : 0);
    const float4 seg1 = was1 ? make_float4(ro.x, ro.y, ro.z, seg.w) : seg;
    seg = make_float4(so.x, so.y, so.z, seg.w);
    // the light sample's MIS at the scatter point
    const float4 radv = w_rad(P.W, slot), tpv = w_tp(P.W, slot);
    C3 L = rgb(radv);
    if (flags & VF_HASVAL) {
        const C3 value = rgb(w_v_val(P.W, slot));
        if (!iszero(value)) {
            const DevMedium &M = S.media[medium];
            const V3 din = xyz(w_ray_d(P.W, slot));
            const V3 to_light = xyz(w_v_li0(P.W, slot));
            const float lpdf = w_v_li1(P.W, slot).w;
            const float pf = w_v_li2(P.W, slot).w != 0.f ? 0.f : phase_eval(M, to_light, -din);
            const float w = power_heuristic(lpdf, pf);
            const float ev = phase_eval(M, to_light, -din);
            L = L + ((rgb(tpv) * value) * ev) * w;
        }
    }
    want = vw_finish_one<true>(P, S, slot, flags, rng, ro, rd, seg, h, was, h1, was1, seg1, tr, L,
                         __float_as_int(radv.w), tpv, f4c(cfill(pfw), pfpdf))
               ? 1u
               : 0u;
    return want;
}
__global__ void __launch_bounds__(128, RT_VW_MINB_TRSAMP) k_vw_scatter(RenderParams P, int round)
{
    round = cur_round(P, round);
    const DevScene &S = P.S;
    RoundCounters *C = &P.W.cnt[round];
    RoundCounters *Cn = &P.W.cnt[round + 1];
    int *next_q = vw_trace_queue(P, round + 1);
    int limit = 0;
    int *const out_q[1] = {next_q};
    int *const out_n[1] = {&Cn->closest};
    VW_LOOP(C->mat[1], P.W.q_mat[1])
    {
        const int slot = VW_LIVE ? qin_[i_] : 0;
        const unsigned want = VW_LIVE ? vw_scatter_path(P, S, slot, limit) : 0u;
        q_push(out_q, out_n, slot, want);
    }
    if (limit) atomicOr(P.limit_flag, RT_LIM_VOLPATH);
}

// Every path of the round's trace queue run to its end by one thread, the
// wavefront's steps one after another with the path's state in memory between
// them.  Taken for a round with at most P.tail_paths paths (tail_begin), where
// a wavefront round is five launches that each wait for their slowest path:
// the rounds that are left cost one launch together.  The films are the
// wavefront's: the steps are.  Grid medium, 133x97 x 9 spp: 3.24 -> 1.78 ms.
// (Two blocks per SM hold RT_VW_TAIL paths; 3 to 8 were 0-10 % slower.)
#ifndef RT_VW_TAIL_MINB
#define RT_VW_TAIL_MINB 2
#endif
__global__ void __launch_bounds__(128, RT_VW_TAIL_MINB) k_vw_tail(RenderParams P, int round)
{
    round = cur_round(P, round);
    const DevScene &S = P.S;
    RoundCounters *C = &P.W.cnt[round];
    const int n = C->closest;
    if (!tail_begin(P, C, n)) return;
    const int *queue = vw_trace_queue(P, round);
    int limit = 0, first, end;
    tail_share(n, first, end);
    for (int i = first; i < end; i += 32) {
        const int slot = queue[i];
        for (;;) {
            const unsigned w = vw_step_path(P, S, slot, limit);
            if (w == 0) break;          // the path has ended
            if (w == 8u) continue;      // a null boundary crossed
            bool scat = w == 2u;
            if (w == 1u) scat = vw_shadow_path(P, S, slot, limit) == 1u;
            if (scat) {
                if (!vw_scatter_path(P, S, slot, limit)) break;
            } else {
                if (!vw_surface_path(P, S, slot)) break;
                if (!vw_trsamp_path(P, S, slot, limit)) break;
            }
        }
    }
    if (limit) atomicOr(P.limit_flag, RT_LIM_VOLPATH);
    tail_end(C);
}
