// rt_kernels.cuh -- wavefront state, kernels and launch helpers shared by
// rt_api.cu.  One batch renders complete reference tiles (block_x x block_y
// pixels, all samples of each pixel), so the film can be reduced per pixel in
// the reference's own summation order without atomics.
#pragma once
#include "rt_device.cuh"

namespace rtgpu {

// path flags
enum { F_FIRST = 1, F_DELTA = 2, F_NEE = 4, F_END = 8 };

#define RT_NBSDF 6        // sorted shading queues (bsdf_queue): types 0-4, then the delta types;
                          // RT_QUEUE_MIXED (rt_device.cuh) is one more: Microfacet, textured BSDFs
                          // where they are not sorted, every BSDF in bounces below the sort threshold
#define RT_QUEUE_FIN 7    // paths whose traced ray missed or hit a surface without a BSDF
#define RT_NQUEUE 8

struct RoundCounters {   // one per wavefront round, zeroed per batch
    int closest, shadow, wc_closest, wc_shadow;
    int mat[RT_NQUEUE];  // paths per shading queue (material-sorted), in the mixed queue, to finish
    int end;             // paths that ended in shading with a light sample pending
    int tail_blocks;     // blocks of the round's tail kernel that have finished
    int pad[2];
};

// Path state.  What a kernel reads or writes together lies together, in
// records of 32 bytes (two float4, one memory sector): the queues hold the
// slots in the order the traversal finished them, so beyond the first bounces
// a warp's accesses scatter, and a lone 16-byte field moves a whole sector for
// half of it (740 bytes of DRAM per shaded vertex against about 310 used).
// Against an array per field: furnished room (1024^2 x 16 spp) 24.3 -> 16.4 ms,
// its shading 15.8 -> 7.9; 1.31M-triangle frame 48.3 -> 43.0 ms, shading 17.7 ->
// 11.9; 128^3 grid-medium frame 48.0 -> 43.0 ms.  (A hit padded to a sector of
// its own was 1-2 % slower than its 16 bytes.)
struct Wave {
    // per path slot
    float4 *ray;       // 2: (origin, mint), (direction, maxt)
    float4 *acc;       // 2: (throughput rgb, eta after the pending sample), (radiance rgb, depth (int bits)); the
                       //    radiance of a path that has ended is what the film sums (w_done).  Not written for a
                       //    camera ray (F_FIRST): throughput 1, eta 1, radiance 0, depth 0
    float4 *smp;       // 2: (pending BSDF sample value rgb, pdf), (stream state, stream increment, flags; path_rng)
    float4 *hit;       // t, u, v, prim (int bits)
    float4 *sh;        // 2: light sample's shadow ray (direction, maxt; it starts at the ray's origin with its mint),
                       //    (pending contribution rgb, occluded (int bits, written by the any-hit trace))
    uint8_t *splat;    // film footprint code of the sample
    uint8_t *pix_irregular;  // per batch pixel: some sample splats off its pixel
    // queues of the current round
    int *q_closest, *q_shadow;
    int *q_mat[RT_NQUEUE];  // shading queues (bsdf_queue), the unsorted one (RT_QUEUE_MIXED) and the
                            // paths to finish (RT_QUEUE_FIN), filled by the closest-hit trace
    int *q_end;        // paths whose BSDF sample was zero, light sample pending
    // ray reordering (optional): per-ray keys, the reordered queue, key counts
    unsigned *sort_keys;
    int *sort_tmp;
    unsigned *sort_hist;
    RoundCounters *cnt;
    int *sid;          // multi-scene batches: scene-table index of the path's job
    int capacity;
    int max_rounds;
    // VolPathTracing wavefront (allocated only for it, vw_capacity paths)
    float4 *v_light;   // 2: (vertex position, light-selection weight), (direction to the sampled light, distance)
    float4 *v_point;   // 2: (point on the light, pdf), (normal at the point, delta light)
    float4 *v_val;     // 2: (light sample intensity, then its attenuated value), (origin of the ray segment that
                       //    found `hit` (its direction is the path's), medium)
    int vw_capacity;
};
__device__ __forceinline__ float4 &w_ray_o(const Wave &W, int s) { return W.ray[2 * (size_t)s]; }
__device__ __forceinline__ float4 &w_ray_d(const Wave &W, int s) { return W.ray[2 * (size_t)s + 1]; }
__device__ __forceinline__ float4 &w_tp(const Wave &W, int s) { return W.acc[2 * (size_t)s]; }
__device__ __forceinline__ float4 &w_rad(const Wave &W, int s) { return W.acc[2 * (size_t)s + 1]; }
// both halves of a slot's record in one 32-byte access
__device__ __forceinline__ void w_load2(const float4 *rec, int s, float4 &a, float4 &b)
{
    const float4 *p = rec + 2 * (size_t)s;
    asm volatile("ld.global.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
                 : "l"(p)
                 : "memory");
}
__device__ __forceinline__ void w_store2(float4 *rec, int s, float4 a, float4 b)
{
    float4 *p = rec + 2 * (size_t)s;
    asm volatile("st.global.v8.f32 [%8], {%0, %1, %2, %3, %4, %5, %6, %7};"
                 :
                 : "f"(a.x), "f"(a.y), "f"(a.z), "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w), "l"(p)
                 : "memory");
}
// a path's end: its whole record, so that the sector need not be read for it
__device__ __forceinline__ void w_done(const Wave &W, int s, C3 L)
{
    w_store2(W.acc, s, make_float4(0.f, 0.f, 0.f, 0.f), make_float4(L.r, L.g, L.b, 0.f));
}
__device__ __forceinline__ float4 &w_bs(const Wave &W, int s) { return W.smp[2 * (size_t)s]; }
__device__ __forceinline__ float4 &w_rng(const Wave &W, int s) { return W.smp[2 * (size_t)s + 1]; }
__device__ __forceinline__ float4 &w_sh_d(const Wave &W, int s) { return W.sh[2 * (size_t)s]; }
__device__ __forceinline__ float4 &w_nee(const Wave &W, int s) { return W.sh[2 * (size_t)s + 1]; }
__device__ __forceinline__ void w_set_occluded(const Wave &W, int s, bool o) { w_nee(W, s).w = __int_as_float(o ? 1 : 0); }
__device__ __forceinline__ float4 &w_v_p(const Wave &W, int s) { return W.v_light[2 * (size_t)s]; }
__device__ __forceinline__ float4 &w_v_li0(const Wave &W, int s) { return W.v_light[2 * (size_t)s + 1]; }
__device__ __forceinline__ float4 &w_v_li1(const Wave &W, int s) { return W.v_point[2 * (size_t)s]; }
__device__ __forceinline__ float4 &w_v_li2(const Wave &W, int s) { return W.v_point[2 * (size_t)s + 1]; }
__device__ __forceinline__ float4 &w_v_val(const Wave &W, int s) { return W.v_val[2 * (size_t)s]; }
__device__ __forceinline__ float4 &w_v_seg(const Wave &W, int s) { return W.v_val[2 * (size_t)s + 1]; }
// A path's stream and flags in 16 bytes: the state, the increment's low word,
// the flags (31 bits) with the increment's bit 32 on top (an increment is
// twice a 32-bit sample index plus one).
__device__ __forceinline__ float4 path_rng_pack(const Pcg32 &r, int flags)
{
    return make_float4(__uint_as_float((unsigned)r.state), __uint_as_float((unsigned)(r.state >> 32)),
                       __uint_as_float((unsigned)r.inc),
                       __uint_as_float(((unsigned)flags & 0x7fffffffu) | ((unsigned)(r.inc >> 32) << 31)));
}
__device__ __forceinline__ Pcg32 path_rng(float4 v, int &flags)
{
    const unsigned w = __float_as_uint(v.w);
    Pcg32 r;
    r.state = (uint64_t)__float_as_uint(v.x) | (uint64_t)__float_as_uint(v.y) << 32;
    r.inc = (uint64_t)__float_as_uint(v.z) | (uint64_t)(w >> 31) << 32;
    flags = (int)(w & 0x7fffffffu);
    return r;
}

// One work item of a multi-scene batch (rt_internal_render_multi): whole
// tiles of one job with every sample of their pixels.  The batch's path
// slots are the items' slots one after another; within an item, slot
// path0 + q * spp + s is sample s of the item's pixel q, as in a
// single-scene batch.
struct MultiItem {
    int job;             // scene-table index
    int path0;           // first path slot of the item
    int pix0;            // first batch pixel of the item (film threads, pix_irregular)
    int npix;            // pixels of the item's tiles
    int spp, sample_begin;
    int g0;              // first entry of the item's tiles in its job's tile order
    int width;           // film width of the job
    int accumulate;      // add to the film instead of writing it
    int pad;
    const int4 *tileorder;   // the job's tile-order table
    float4 *film;            // the job's film (device memory)
    uint64_t seed;
};

// batch geometry: tiles [tile0, tile0 + ntiles) of the reference job grid
struct Batch {
    int tile0, ntiles;      // tiles in raster order of the job grid
    int tiles_x;            // job grid width in tiles
    int bx, by;             // block size
    int npix;               // pixels in the batch
    int spp, sample_begin;
    int n_paths;            // npix * spp
    int *pix_of;            // batch pixel -> image pixel (y * W + x)
    int *tile_of;           // batch pixel -> (local x | local y << 16)
};

}  // namespace rtgpu
