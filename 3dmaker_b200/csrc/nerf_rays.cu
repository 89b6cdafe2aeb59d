// Rays: slab test against the outermost cascade, the walk over the cascaded occupancy pyramid, exclusive scan of the
// per-ray sample counts and the compaction of the samples of a ray range into the field kernels' input.
//
// Replaces compute_ray_aabb_inv_kernel (modules/NeRF/otherKernels.cu:91-154), march_rays_dda_calc_hits,
// custom_exclusive_sum, find_cutoff_ray_kernel / find_cutoff_ray_from_kernel and march_rays_dda_offset
// (modules/NeRF/processRays.cu:486-549, 626-929) and the host orchestration processRaysHitLinear /
// processRaysHitData / processRaysHitPositions (processRays.cu:931-1173).
//
// The sample list (counts, offsets, ray ids, t, contracted positions, all in ray order) is the reference's, bit for
// bit; how it is produced is not:
//   * ONE walk per ray.  The reference walks every ray twice per batch (count, then emit) and, when training, walks
//     all remaining rays of the chunk again for every optimizer step.  Here the walk stores the sample distances of a
//     ray in that ray's row of a scratch matrix [ray][1024] (HBM is plentiful: 4 KB per ray) together with the count;
//     a batch is then cut out of the rows by a warp-per-ray copy that also evaluates the contracted positions.
//   * Where to cut is decided by the host from the scanned offsets, read back once per walk instead of once (the
//     reference: three times) per batch.
//   * A probe order that skips the pyramid descent inside solid regions (see walk_ray).
// The two-pass entry points (count / scan / cutoff / emit) remain for callers that want the reference's sequence.
#include <atomic>
#include <cmath>

#include "common.cuh"

namespace nb {

extern std::atomic<uint64_t> g_launch_count;

constexpr uint32_t MAX_HITS = 1024;  // per-ray sample cap, modules/NeRF/InstantNerf.h:24
constexpr int MAX_MIP_LEVELS = 8;
// Hard bound on the advances of one ray.  A ray crosses at most 3 x 128 finest voxels per cascade plus its 1024 samples;
// 65536 is far beyond any walk that makes progress and only ends one that does not.
constexpr uint32_t MAX_WALK_ADVANCES = 1u << 16;

struct Scene {
    uint3 res;
    float3 aabb_min, aabb_max;
    int num_cascades, levels, spv;
    uint32_t level_offset[MAX_MIP_LEVELS];  // first cell of every pyramid level inside a cascade
    uint32_t pyramid_cells;                 // cells of one cascade's whole pyramid
    int nested;                             // every level halves the one below exactly (resolution divisible by 2^(levels-1))
};

static Scene make_scene(const nb_scene_desc* d) {
    Scene s;
    s.res = make_uint3(d->grid_res[0], d->grid_res[1], d->grid_res[2]);
    s.aabb_min = make_float3(d->aabb_min[0], d->aabb_min[1], d->aabb_min[2]);
    s.aabb_max = make_float3(d->aabb_max[0], d->aabb_max[1], d->aabb_max[2]);
    s.num_cascades = d->num_cascades; s.levels = d->mip_levels; s.spv = d->samples_per_voxel;
    uint32_t off = 0;
    uint3 r = s.res;
    for (int l = 0; l < MAX_MIP_LEVELS; l++) {
        s.level_offset[l] = off;
        if (l < s.levels) { off += r.x * r.y * r.z; r.x >>= 1; r.y >>= 1; r.z >>= 1; }
    }
    s.pyramid_cells = off;
    const uint32_t m = (1u << (s.levels - 1)) - 1u;
    s.nested = ((s.res.x & m) == 0 && (s.res.y & m) == 0 && (s.res.z & m) == 0) ? 1 : 0;
    return s;
}

struct Slab {
    float3 inv;
    float near, far;
};

__device__ __forceinline__ Slab slab_test(float3 o3, float3 d3, float3 aabb_min, float3 aabb_max, int num_cascades) {
    const float scale = exp2f((float)(num_cascades - 1));
    const float lo[3] = {aabb_min.x * scale, aabb_min.y * scale, aabb_min.z * scale};
    const float hi[3] = {aabb_max.x * scale, aabb_max.y * scale, aabb_max.z * scale};
    const float o[3] = {o3.x, o3.y, o3.z};
    float d[3] = {d3.x, d3.y, d3.z};
    float inv[3];
    float t_enter = -INFINITY, t_exit = INFINITY;
#pragma unroll
    for (int a = 0; a < 3; a++) {
        if (fabsf(d[a]) < 1e-8f) d[a] = 1e-8f;
        inv[a] = 1.0f / d[a];
        const float ta = (lo[a] - o[a]) * inv[a], tb = (hi[a] - o[a]) * inv[a];
        t_enter = fmaxf(t_enter, fminf(ta, tb));
        t_exit = fminf(t_exit, fmaxf(ta, tb));
    }
    const bool miss = t_enter > t_exit || t_exit < 0.0f;
    return Slab{make_float3(inv[0], inv[1], inv[2]), miss ? 0.0f : fmaxf(t_enter, 0.0f), miss ? 0.0f : t_exit};
}

__global__ void __launch_bounds__(256) ray_aabb_kernel(const uint32_t num_rays, const float3* __restrict__ rays_o,
                                                       const float3* __restrict__ rays_d, const float3 aabb_min, const float3 aabb_max,
                                                       const int num_cascades, float3* __restrict__ rays_d_inv,
                                                       float* __restrict__ nears, float* __restrict__ fars) {
    after_previous();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= num_rays) return;
    const Slab s = slab_test(rays_o[i], rays_d[i], aabb_min, aabb_max, num_cascades);
    rays_d_inv[i] = s.inv;
    nears[i] = s.near;
    fars[i] = s.far;
}

// Which cascade a point belongs to: ceil(log2(largest |p| / box half-extent ratio)), modules/NeRF/processRays.cu:11-19.
__device__ __forceinline__ int get_cascade(float3 pos, float3 aabb_min, float3 aabb_max, int num_cascades) {
    const float rx = fmaxf(pos.x / aabb_max.x, pos.x / aabb_min.x);
    const float ry = fmaxf(pos.y / aabb_max.y, pos.y / aabb_min.y);
    const float rz = fmaxf(pos.z / aabb_max.z, pos.z / aabb_min.z);
    const float max_scale = fmaxf(rx, fmaxf(ry, rz));
    if (max_scale <= 1.0f) return 0;
    return max(0, min((int)ceilf(log2f(max_scale)), num_cascades - 1));
}

// The voxel of pyramid level `level` that holds the point at relative position `rel` of its cascade box: is it
// occupied, and at which ray distance does the ray leave it.
struct Probe {
    bool occupied;
    float exit_t;
};

struct RayConst {
    float3 o, d_inv;
    float3 ahead;  // 1 where the ray moves towards +axis, else 0: selects the far face of a voxel
};

__device__ __forceinline__ Probe probe_level(const Scene& sc, const RayConst& rc, const uint8_t* __restrict__ bits, int level, uint32_t cascade_base,
                                             float3 box_min, float3 box_extent, float3 rel) {
    const uint32_t rx = sc.res.x >> level, ry = sc.res.y >> level, rz = sc.res.z >> level;
    const float sx = box_extent.x / rx, sy = box_extent.y / ry, sz = box_extent.z / rz;  // voxel size
    const int vx = max(0, min((int)floorf(rel.x * rx), (int)rx - 1));
    const int vy = max(0, min((int)floorf(rel.y * ry), (int)ry - 1));
    const int vz = max(0, min((int)floorf(rel.z * rz), (int)rz - 1));
    const uint32_t cell = cascade_base + sc.level_offset[level] + vz * (rx * ry) + vy * rx + vx;
    Probe p;
    p.occupied = (bits[cell >> 3] >> (cell & 7u)) & 1u;
    const float fx = box_min.x + (vx + rc.ahead.x) * sx, fy = box_min.y + (vy + rc.ahead.y) * sy, fz = box_min.z + (vz + rc.ahead.z) * sz;
    p.exit_t = fminf(fminf((fx - rc.o.x) * rc.d_inv.x, (fy - rc.o.y) * rc.d_inv.y), (fz - rc.o.z) * rc.d_inv.z);
    return p;
}

// One ray through the occupancy pyramid.  sink(k, t) receives sample k at ray distance t; returns the sample count.
//
// The reference (march_rays_dda_calc_hits / _offset) restarts every advance at the coarsest level and descends while
// the voxel is occupied; it then either samples the occupied finest voxel or jumps to the exit of the first empty
// voxel it met.  Because a parent bit is the OR of its children, "first empty level from the top" is the same level
// whichever order the levels are looked at, so inside solid regions - where the last advance ended in an occupied
// finest voxel and the next one most likely does too - the finest level is probed first and the descent is skipped.
// That needs parent and child voxels to nest exactly (sc.nested); otherwise the reference's order is kept.
template <class Sink>
__device__ __forceinline__ uint32_t walk_ray(const Scene& sc, float3 o, float3 d, float3 d_inv, float t_begin, float t_end,
                                             const uint8_t* __restrict__ bits, Sink&& sink) {
    const float3 extent = make_float3(sc.aabb_max.x - sc.aabb_min.x, sc.aabb_max.y - sc.aabb_min.y, sc.aabb_max.z - sc.aabb_min.z);
    RayConst rc;
    rc.o = o; rc.d_inv = d_inv;
    rc.ahead = make_float3(d.x >= 0.0f ? 1.0f : 0.0f, d.y >= 0.0f ? 1.0f : 0.0f, d.z >= 0.0f ? 1.0f : 0.0f);
    const int top = sc.levels - 1;
    uint32_t count = 0;
    float t = t_begin;
    bool in_solid = false;
    uint32_t advances = 0;
    while (t < t_end && count < MAX_HITS && advances++ < MAX_WALK_ADVANCES) {
        const float3 pos = make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
        const int cascade = get_cascade(pos, sc.aabb_min, sc.aabb_max, sc.num_cascades);
        const float cs = exp2f((float)cascade);
        const float3 box_min = make_float3(sc.aabb_min.x * cs, sc.aabb_min.y * cs, sc.aabb_min.z * cs);
        const float3 box_extent = make_float3(extent.x * cs, extent.y * cs, extent.z * cs);
        const float3 rel = make_float3((pos.x - box_min.x) / box_extent.x, (pos.y - box_min.y) / box_extent.y, (pos.z - box_min.z) / box_extent.z);
        const uint32_t cascade_base = cascade * sc.pyramid_cells;
        Probe p;
        if (in_solid && sc.nested) {
            p = probe_level(sc, rc, bits, 0, cascade_base, box_min, box_extent, rel);
            if (!p.occupied) {
                for (int l = top; l > 0; l--) {
                    const Probe q = probe_level(sc, rc, bits, l, cascade_base, box_min, box_extent, rel);
                    if (!q.occupied) { p = q; break; }
                }
            }
        } else {
            for (int l = top;; l--) {
                p = probe_level(sc, rc, bits, l, cascade_base, box_min, box_extent, rel);
                if (!p.occupied || l == 0) break;
            }
        }
        in_solid = p.occupied;
        if (p.occupied) {
            // samples_per_voxel points at the centres of equal sub-spans of [t, exit)
            const int K = sc.spv;
            const float span = p.exit_t - t;
            for (int k = 0; k < K && count < MAX_HITS; ++k) {
                sink(count, t + (k + 0.5f) / (float)K * span);
                count++;
            }
        }
        // The reference advances with exactly this expression (processRays.cu:235,733,925).  From t = 256 on the 1e-5 is
        // below half an ulp and is rounded away, and a voxel face computed a rounding error behind t (or an exit of -inf
        // from a -0.0 direction component) then leaves t where it was: the reference's loop would never end.  Where the
        // expression makes progress its value is kept bit for bit; where it does not, t moves to the next float.
        const float next = fmaxf(t + 1e-5f, p.exit_t + 1e-6f);
        t = next > t ? next : nextafterf(t, INFINITY);
    }
    return count;
}

struct CountOnly {
    __device__ __forceinline__ void operator()(uint32_t, float) const {}
};
struct RowSink {
    float* row;
    __device__ __forceinline__ void operator()(uint32_t k, float t) const { row[k] = t; }
};
// Writes a sample straight into the compacted arrays (the two-pass entry point).
struct CompactSink {
    const Scene* sc;
    float3 o, d;
    uint32_t ray_id, base;
    float* t_out;
    uint32_t* ray_out;
    float4* pos_out;
    __device__ __forceinline__ void operator()(uint32_t k, float t) const {
        const uint32_t w = base + k;
        t_out[w] = t;
        ray_out[w] = ray_id;
        const float3 p = contract_pos(make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z), sc->aabb_min, sc->aabb_max);
        st_cs_v4(&pos_out[w], make_uint4(__float_as_uint(p.x), __float_as_uint(p.y), __float_as_uint(p.z), 0u));
    }
};

struct RayArrays {
    const float3* o;
    const float3* d;
    const float3* d_inv;
    const float* nears;
    const float* fars;
};

__global__ void __launch_bounds__(256) march_count_kernel(const __grid_constant__ Scene sc, const uint32_t num_rays, RayArrays r,
                                                          const uint8_t* __restrict__ bits, uint32_t* __restrict__ num_steps) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= num_rays) return;
    num_steps[i] = walk_ray(sc, r.o[i], r.d[i], r.d_inv[i], r.nears[i], r.fars[i], bits, CountOnly{});
}

// The single walk: sample distances of ray i into rows[i * row_stride ...], count into num_steps[i].
__global__ void __launch_bounds__(256) march_fill_kernel(const __grid_constant__ Scene sc, const uint32_t num_rays, RayArrays r,
                                                         const uint8_t* __restrict__ bits, uint32_t* __restrict__ num_steps,
                                                         float* __restrict__ rows, uint32_t row_stride) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= num_rays) return;
    num_steps[i] = walk_ray(sc, r.o[i], r.d[i], r.d_inv[i], r.nears[i], r.fars[i], bits, RowSink{rows + (size_t)i * row_stride});
}

// ---- the single walk, split at the voxels of one pyramid level -----------------------------------------
// A walk is a chain of dependent steps (170 advances for a ray through the middle of a 128^3 grid), and a warp of one-ray
// threads waits for its longest ray.  But a step depends on the ones before it through t alone, and a ray leaves a coarse
// voxel at a distance that the coarse voxel's own faces give: the walk can be cut there.
//   1. One lane per ray steps over the voxels of level `split` (8 finest voxels wide; empty regions in larger steps) and
//      queues the occupied ones as items: where the ray enters, and where this coarse step says that it goes on.
//   2. The warp takes 32 items at a time, whatever rays they belong to, and walks each through its finer voxels until it
//      is in another coarse voxel, 22 advances at most, keeping the samples in shared memory.
//   3. An item that starts where its predecessor ended is what the sequential walk would have produced.  Predecessors end
//      elsewhere when the last finest voxel is crossed in less than the minimum advance (1e-5, about one item in a
//      thousand): the item is then walked again from the true distance, so that the list is the sequential one bit for bit.
//   4. The samples are appended to the rows of their rays.
// A warp takes `rays_per_warp` rays: few when there are few rays, so that more lanes share each ray's items.
// Bound by instruction latency: 16 warps an SM issue every other cycle.  Against one thread per ray (the walk, us): 14400 rays
// of a preview 162 -> 44, 20011 training rays 93 -> 44, 65536 157 -> 88, 131072 rays through three cascades 500 -> 519 (there
// the rays alone fill the chip; slab test and scan, now in fewer launches, make up for it).
// Measured and not better: 12 blocks an SM at 80 registers, 16 at 64 (+50 %), 4 warps a block, a descent of the levels in
// place of the three loads (+15 %).
constexpr int SPLIT_WARPS = 2, SPLIT_BLOCKS = 8;   // warps of a block, blocks of an SM: 16 warps, 91 registers a thread
constexpr uint32_t FLOOR_BITS = 0x4b000000u;   // the float 2^23
constexpr uint32_t ITEM_SAMPLES = 24, ITEM_PITCH = ITEM_SAMPLES + 1, QUEUE = 64;

struct SplitScene {
    Scene sc;
    int split;                 // pyramid level of the items
    // powers of two, see exact_reciprocals
    float3 voxel;              // finest voxel of the innermost cascade
    float3 per_voxel;          // 1 / voxel
    float3 inv_max, inv_min;
    uint32_t cell_bias[MAX_MIP_LEVELS];   // level_offset minus what FLOOR_BITS in the coordinates adds to a cell number
};

// Boxes and resolutions that are powers of two on every axis (unit and half boxes, 64 / 128 / 256 grids): every division of
// the walk is then exact, and so is the multiplication by the reciprocal that replaces it.
static bool power_of_two(float x) { int e; return x != 0.0f && std::isfinite(x) && std::fabs(std::frexp(x, &e)) == 0.5f && e > -60 && e < 60; }
static bool exact_reciprocals(const Scene& s) {
    const float3 e = make_float3(s.aabb_max.x - s.aabb_min.x, s.aabb_max.y - s.aabb_min.y, s.aabb_max.z - s.aabb_min.z);
    for (float x : {e.x, e.y, e.z, s.aabb_max.x, s.aabb_max.y, s.aabb_max.z, s.aabb_min.x, s.aabb_min.y, s.aabb_min.z,
                    (float)s.res.x, (float)s.res.y, (float)s.res.z})
        if (!power_of_two(x)) return false;
    return s.num_cascades <= 32;
}
static SplitScene make_split_scene(const Scene& s) {
    SplitScene p;
    p.sc = s;
    p.split = s.levels - 1 < 3 ? s.levels - 1 : 3;
    const float3 e = make_float3(s.aabb_max.x - s.aabb_min.x, s.aabb_max.y - s.aabb_min.y, s.aabb_max.z - s.aabb_min.z);
    p.voxel = make_float3(e.x / (float)s.res.x, e.y / (float)s.res.y, e.z / (float)s.res.z);
    p.per_voxel = make_float3(1.0f / p.voxel.x, 1.0f / p.voxel.y, 1.0f / p.voxel.z);
    for (int l = 0; l < MAX_MIP_LEVELS; l++) {
        const uint32_t rx = s.res.x >> l, ry = s.res.y >> l;
        p.cell_bias[l] = s.level_offset[l] - FLOOR_BITS * (rx * ry + rx + 1u);
    }
    p.inv_max = make_float3(1.0f / s.aabb_max.x, 1.0f / s.aabb_max.y, 1.0f / s.aabb_max.z);
    p.inv_min = make_float3(1.0f / s.aabb_min.x, 1.0f / s.aabb_min.y, 1.0f / s.aabb_min.z);
    return p;
}
// Where the split walk is used: voxels nest exactly, an item is at least four finest voxels wide (else there is nothing to
// share) and one sample per voxel (else an item's samples do not fit its slots).
static bool can_split(const Scene& s) { return s.nested && s.levels >= 3 && s.spv == 1; }

// Where a point of the ray lies: cells of the pyramid around it and the distances at which the ray leaves them.  The
// expressions are walk_ray's, and so are the bits that come out.
template <bool EXACT>
struct Place;

template <>
struct Place<false> {
    float scale;        // size of this cascade's box against the innermost one's: a power of two
    uint32_t base;      // first cell of the cascade's pyramid
    int x, y, z;        // finest voxel

    __device__ __forceinline__ Place(const SplitScene& p, float3 o, float3 d, float t) {
        const Scene& sc = p.sc;
        const float3 pos = make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
        const int cascade = get_cascade(pos, sc.aabb_min, sc.aabb_max, sc.num_cascades);
        scale = exp2f((float)cascade);
        base = cascade * sc.pyramid_cells;
        const float3 e = make_float3(sc.aabb_max.x - sc.aabb_min.x, sc.aabb_max.y - sc.aabb_min.y, sc.aabb_max.z - sc.aabb_min.z);
        const float3 rel = make_float3((pos.x - sc.aabb_min.x * scale) / (e.x * scale), (pos.y - sc.aabb_min.y * scale) / (e.y * scale),
                                       (pos.z - sc.aabb_min.z * scale) / (e.z * scale));
        x = max(0, min((int)floorf(rel.x * sc.res.x), (int)sc.res.x - 1));
        y = max(0, min((int)floorf(rel.y * sc.res.y), (int)sc.res.y - 1));
        z = max(0, min((int)floorf(rel.z * sc.res.z), (int)sc.res.z - 1));
    }
    __device__ __forceinline__ uint32_t cell(const SplitScene& p, int level) const {
        const uint32_t rx = p.sc.res.x >> level, ry = p.sc.res.y >> level;
        return base + p.sc.level_offset[level] + (z >> level) * (rx * ry) + (y >> level) * rx + (x >> level);
    }
    __device__ __forceinline__ float leave(const SplitScene& p, const RayConst& rc, int level) const {
        const Scene& sc = p.sc;
        const float3 e = make_float3(sc.aabb_max.x - sc.aabb_min.x, sc.aabb_max.y - sc.aabb_min.y, sc.aabb_max.z - sc.aabb_min.z);
        const float3 s = make_float3(e.x * scale / (sc.res.x >> level), e.y * scale / (sc.res.y >> level), e.z * scale / (sc.res.z >> level));
        const float fx = __fmaf_rn((x >> level) + rc.ahead.x, s.x, sc.aabb_min.x * scale), fy = __fmaf_rn((y >> level) + rc.ahead.y, s.y, sc.aabb_min.y * scale),
                    fz = __fmaf_rn((z >> level) + rc.ahead.z, s.z, sc.aabb_min.z * scale);
        return fminf(fminf((fx - rc.o.x) * rc.d_inv.x, (fy - rc.o.y) * rc.d_inv.y), (fz - rc.o.z) * rc.d_inv.z);
    }
};

// Powers of two: every division is exact, and so are the multiplications by reciprocals and the scalings that replace it.
// Floors come out of an addition rounded down (2^23 + v, the integer in the low bits) instead of the conversion unit.
template <>
struct Place<true> {
    float scale;
    uint32_t base;
    float x, y, z;      // in finest voxels, inside the box

    __device__ __forceinline__ Place(const SplitScene& p, float3 o, float3 d, float t) {
        const Scene& sc = p.sc;
        const float3 pos = make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z);
        float3 k = p.per_voxel;
        scale = 1.0f; base = 0u;
        if (sc.num_cascades > 1) {
            const float m = fmaxf(fmaxf(fmaxf(pos.x * p.inv_max.x, pos.x * p.inv_min.x), fmaxf(pos.y * p.inv_max.y, pos.y * p.inv_min.y)),
                                  fmaxf(pos.z * p.inv_max.z, pos.z * p.inv_min.z));
            if (m > 1.0f) {
                const int cascade = max(0, min((int)ceilf(log2f(m)), sc.num_cascades - 1));
                scale = __uint_as_float((127u + cascade) << 23);
                base = cascade * sc.pyramid_cells;
                const float back = __uint_as_float((127u - cascade) << 23);
                k = make_float3(k.x * back, k.y * back, k.z * back);
            }
        }
        x = fmaxf(0.0f, fminf((pos.x - sc.aabb_min.x * scale) * k.x, (float)(sc.res.x - 1)));
        y = fmaxf(0.0f, fminf((pos.y - sc.aabb_min.y * scale) * k.y, (float)(sc.res.y - 1)));
        z = fmaxf(0.0f, fminf((pos.z - sc.aabb_min.z * scale) * k.z, (float)(sc.res.z - 1)));
    }
    static __device__ __forceinline__ float down(float v, int level) { return __fmaf_rd(v, __uint_as_float((127u - level) << 23), 8388608.0f); }
    __device__ __forceinline__ uint32_t cell(const SplitScene& p, int level) const {
        const uint32_t rx = p.sc.res.x >> level, ry = p.sc.res.y >> level;
        return base + p.cell_bias[level] + __float_as_uint(down(z, level)) * (rx * ry) + __float_as_uint(down(y, level)) * rx +
               __float_as_uint(down(x, level));
    }
    __device__ __forceinline__ float leave(const SplitScene& p, const RayConst& rc, int level) const {
        const Scene& sc = p.sc;
        const float k = scale * __uint_as_float((127u + level) << 23);
        const float fx = sc.aabb_min.x * scale + (down(x, level) + (rc.ahead.x - 8388608.0f)) * (p.voxel.x * k),
                    fy = sc.aabb_min.y * scale + (down(y, level) + (rc.ahead.y - 8388608.0f)) * (p.voxel.y * k),
                    fz = sc.aabb_min.z * scale + (down(z, level) + (rc.ahead.z - 8388608.0f)) * (p.voxel.z * k);
        return fminf(fminf((fx - rc.o.x) * rc.d_inv.x, (fy - rc.o.y) * rc.d_inv.y), (fz - rc.o.z) * rc.d_inv.z);
    }
};

__device__ __forceinline__ bool occupied_bit(const uint8_t* __restrict__ bits, uint32_t cell) { return (bits[cell >> 3] >> (cell & 7u)) & 1u; }
__device__ __forceinline__ float advance_past(float t, float exit_t) {   // see walk_ray
    const float next = fmaxf(t + 1e-5f, exit_t + 1e-6f);
    return next > t ? next : nextafterf(t, INFINITY);
}

// One step of the coarse walk from t: past the first empty voxel on the way down to level `split`, or, when the voxel of
// that level is occupied (returns true), past it.
template <bool EXACT>
__device__ __forceinline__ bool coarse_step(const SplitScene& p, const RayConst& rc, float3 d, const uint8_t* __restrict__ bits, float t, float& next) {
    const Place<EXACT> at(p, rc.o, d, t);
    int l = p.sc.levels - 1;
    bool occupied = occupied_bit(bits, at.cell(p, l));
    while (occupied && l > p.split) occupied = occupied_bit(bits, at.cell(p, --l));
    next = advance_past(t, at.leave(p, rc, l));
    return occupied;
}
// From t on to the next occupied voxel of level `split`: the distance at which its walk starts (t_end or more: there is none).
template <bool EXACT>
__device__ __noinline__ float coarse_chain(const SplitScene& p, RayConst rc, float3 d, const uint8_t* __restrict__ bits, float t, float t_end) {
    float next;
    for (uint32_t k = 0; t < t_end && k < MAX_WALK_ADVANCES; k++) {
        if (coarse_step<EXACT>(p, rc, d, bits, t, next)) return t;
        t = next;
    }
    return t_end;
}

// The part of the walk that starts at t, inside one coarse voxel.  Returns the number of samples; t becomes the distance
// from which the walk goes on (also when the item's slots are full: the rest is then an item of its own).
template <bool EXACT>
__device__ __forceinline__ uint32_t walk_item(const SplitScene& p, const RayConst& rc, float3 d, const uint8_t* __restrict__ bits, float& t, float t_end,
                                              float* samples) {
    uint32_t count = 0, coarse = 0;
    for (uint32_t k = 0; t < t_end && count < ITEM_SAMPLES && k < 64u; k++) {
        const Place<EXACT> at(p, rc.o, d, t);
        const uint32_t c = at.cell(p, p.split);
        if (k == 0) coarse = c;
        else if (c != coarse) break;
        // the levels between are looked at together: three loads in flight instead of a descent of dependent ones
        const bool b0 = occupied_bit(bits, at.cell(p, 0)), b1 = occupied_bit(bits, at.cell(p, 1));
        const bool b2 = p.split <= 2 || occupied_bit(bits, at.cell(p, 2));
        const float exit_t = at.leave(p, rc, !b2 ? 2 : (!b1 ? 1 : 0));
        if (b0) samples[count++] = t + 0.5f * (exit_t - t);
        t = advance_past(t, exit_t);
    }
    return count;
}

struct SplitWarp {
    float4 ray[32][3];            // o, far; d, where the coarse walk stands; 1 / d
    float end[32], expected[32];  // per ray: where its last item ended and where the coarse step had put that
    uint32_t count[32];
    float q_start[QUEUE], q_next[QUEUE];
    uint32_t q_ray[QUEUE];
    float samples[32 * ITEM_PITCH];

    __device__ __forceinline__ void load(uint32_t k, RayConst& rc, float3& d, float& far, float& t) const {
        const float4 a = ray[k][0], b = ray[k][1], c = ray[k][2];
        rc.o = make_float3(a.x, a.y, a.z); far = a.w;
        d = make_float3(b.x, b.y, b.z); t = b.w;
        rc.d_inv = make_float3(c.x, c.y, c.z);
        rc.ahead = make_float3(d.x >= 0.0f ? 1.0f : 0.0f, d.y >= 0.0f ? 1.0f : 0.0f, d.z >= 0.0f ? 1.0f : 0.0f);
    }
};

template <bool EXACT>
__global__ void __launch_bounds__(SPLIT_WARPS * 32, SPLIT_BLOCKS) march_split_kernel(const __grid_constant__ SplitScene p, const uint32_t num_rays, RayArrays r,
                                                                       const uint32_t rays_per_warp, const uint8_t* __restrict__ bits,
                                                                       uint32_t* __restrict__ num_steps, float* __restrict__ rows) {
    after_previous();
    constexpr uint32_t FULL = 0xffffffffu;
    extern __shared__ float4 s_split[];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    SplitWarp& w = reinterpret_cast<SplitWarp*>(s_split)[warp];
    const uint32_t first = (blockIdx.x * SPLIT_WARPS + warp) * rays_per_warp;
    if (first >= num_rays) return;
    const uint32_t i = first + lane;

    const bool owner = lane < rays_per_warp && i < num_rays;
    bool active = false;
    if (owner) {
        const float3 o = r.o[i], d = r.d[i];
        Slab s;
        if (r.nears != nullptr) s = Slab{r.d_inv[i], r.nears[i], r.fars[i]};
        else s = slab_test(o, d, p.sc.aabb_min, p.sc.aabb_max, p.sc.num_cascades);
        w.ray[lane][0] = make_float4(o.x, o.y, o.z, s.far);
        w.ray[lane][1] = make_float4(d.x, d.y, d.z, s.near);
        w.ray[lane][2] = make_float4(s.inv.x, s.inv.y, s.inv.z, 0.f);
        active = s.near < s.far;
    }
    w.end[lane] = 0.0f; w.expected[lane] = 0.0f; w.count[lane] = 0u;
    uint32_t head = 0, tail = 0, steps = 0;
    __syncwarp();

    for (;;) {
        {
            // the rays of the coarse walk live in shared memory between its turns: their registers are the items' then
            RayConst rc;
            float3 d;
            float t_end, t;
            w.load(lane & (rays_per_warp - 1), rc, d, t_end, t);
            while (tail - head < 32u && __any_sync(FULL, active)) {
                float next = 0.0f;
                const bool push = active && coarse_step<EXACT>(p, rc, d, bits, t, next);
                const uint32_t pushed = __ballot_sync(FULL, push);
                if (push) {
                    const uint32_t slot = (tail + __popc(pushed & ((1u << lane) - 1u))) % QUEUE;
                    w.q_start[slot] = t; w.q_next[slot] = next; w.q_ray[slot] = lane;
                }
                tail += __popc(pushed);
                if (active) { t = next; active = t < t_end && ++steps < MAX_WALK_ADVANCES; }
            }
            if (owner) w.ray[lane][1].w = t;
        }
        __syncwarp();
        const uint32_t items = min(32u, tail - head);
        if (items == 0) break;
        const bool mine = lane < items;
        const uint32_t slot = (head + lane) % QUEUE;
        head += items;
        const uint32_t ray = mine ? w.q_ray[slot] : 32u + lane;   // lanes without an item are groups of their own
        const uint32_t group = __match_any_sync(FULL, ray), before = group & ((1u << lane) - 1u);
        const int prev = before ? 31 - __clz(before) : -1;
        RayConst ic{};
        float3 id{};
        float far = 0.0f, queued = 0.0f, go_on = 0.0f, start = 0.0f, end = 0.0f;
        float* samples = w.samples + lane * ITEM_PITCH;
        uint32_t n = 0;
        if (mine) {
            float unused;
            w.load(ray, ic, id, far, unused);
            queued = w.q_start[slot]; go_on = w.q_next[slot];
            start = queued;
            if (prev < 0 && w.end[ray] != w.expected[ray]) start = coarse_chain<EXACT>(p, ic, id, bits, w.end[ray], far);
            end = start;
            n = walk_item<EXACT>(p, ic, id, bits, end, far, samples);
        }
        // each pass settles at least one more item of every ray, in the rays' order
        for (int pass = 0; pass < 32; pass++) {
            const float prev_end = __shfl_sync(FULL, end, prev & 31), prev_go_on = __shfl_sync(FULL, go_on, prev & 31);
            float want = start;
            if (prev >= 0) want = prev_end == prev_go_on ? queued : coarse_chain<EXACT>(p, ic, id, bits, prev_end, far);
            const bool again = want != start;
            if (!__any_sync(FULL, again)) break;
            if (again) {
                start = end = want;
                n = walk_item<EXACT>(p, ic, id, bits, end, far, samples);
            }
        }
        // samples of the ray's items up to and including this one, by pointer jumping along the ray's lanes
        uint32_t upto = n;
        int link = prev;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            const uint32_t v = __shfl_sync(FULL, upto, link & 31);
            const int further = __shfl_sync(FULL, link, link & 31);
            if (link >= 0) { upto += v; link = further; }
        }
        uint32_t at = 0;
        if (mine) {
            at = w.count[ray] + upto - n;
            float* row = rows + (size_t)(first + ray) * MAX_HITS;
            for (uint32_t k = 0; k < n; k++)
                if (at + k < MAX_HITS) row[at + k] = samples[k];
        }
        __syncwarp();
        if (mine && (group >> lane) == 1u) { w.count[ray] = at + n; w.end[ray] = end; w.expected[ray] = go_on; }   // the ray's last item here
        __syncwarp();
    }
    if (owner) {
        uint32_t count = w.count[lane];
        const float end = w.end[lane];
        if (end != w.expected[lane] && end < w.ray[lane][0].w && count < MAX_HITS) {
            // the last item ended late: whatever is still ahead was not in the queue
            float* row = rows + (size_t)i * MAX_HITS;
            const uint32_t base = count;
            RayConst rc;
            float3 d;
            float t_end, unused;
            w.load(lane, rc, d, t_end, unused);
            count += walk_ray(p.sc, rc.o, d, rc.d_inv, end, t_end, bits, [&](uint32_t k, float s) { if (base + k < MAX_HITS) row[base + k] = s; });
        }
        num_steps[i] = min(count, MAX_HITS);
    }
}


// plan[0] = one past the last ray of the batch (absolute index), plan[2] = first sample of the batch.
// Rays [rays_done, plan[0]) are walked; ray ids are written relative to rays_done.
__global__ void __launch_bounds__(256) march_emit_kernel(const __grid_constant__ Scene sc, const uint32_t num_rays, const uint32_t rays_done,
                                                         RayArrays r, const uint8_t* __restrict__ bits, const uint32_t* __restrict__ ray_offsets,
                                                         const uint32_t* __restrict__ plan, float* __restrict__ t_out,
                                                         uint32_t* __restrict__ ray_idx_out, float4* __restrict__ pos_out) {
    after_previous();
    uint32_t local = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t i = local + rays_done;
    uint32_t end = min(plan[0], num_rays);
    if (i >= end) return;
    CompactSink s{&sc, r.o[i], r.d[i], local, ray_offsets[i] - plan[2], t_out, ray_idx_out, pos_out};
    walk_ray(sc, s.o, s.d, r.d_inv[i], r.nears[i], r.fars[i], bits, s);
}

// Cuts rays [ray_begin, ray_begin + ray_count) out of the scratch rows: one warp per ray, lane k copies sample k and
// evaluates its contracted position; ray ids are relative to ray_begin, samples land at offsets[ray] - sample_base.
__global__ void __launch_bounds__(256) march_compact_kernel(const float3 aabb_min, const float3 aabb_max, const float3* __restrict__ rays_o,
                                                            const float3* __restrict__ rays_d, uint32_t ray_begin, uint32_t ray_count,
                                                            const uint32_t* __restrict__ num_steps, const uint32_t* __restrict__ offsets,
                                                            uint32_t sample_base, const float* __restrict__ rows, uint32_t row_stride,
                                                            float* __restrict__ t_out, uint32_t* __restrict__ ray_idx_out,
                                                            float4* __restrict__ pos_out) {
    after_previous();
    const uint32_t local = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t lane = threadIdx.x & 31;
    if (local >= ray_count) return;
    const uint32_t i = ray_begin + local;
    const uint32_t count = num_steps[i];
    if (count == 0) return;
    const uint32_t dst = offsets[i] - sample_base;
    const float3 o = rays_o[i], d = rays_d[i];
    const float* row = rows + (size_t)i * row_stride;
    for (uint32_t k = lane; k < count; k += 32) {
        const float t = row[k];
        t_out[dst + k] = t;
        ray_idx_out[dst + k] = local;
        const float3 p = contract_pos(make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z), aabb_min, aabb_max);
        st_cs_v4(&pos_out[dst + k], make_uint4(__float_as_uint(p.x), __float_as_uint(p.y), __float_as_uint(p.z), 0u));
    }
}

// The order in which the field kernel takes a batch's samples: ray after ray or, where 32 consecutive rays are so close to one another
// that their samples at equal place share the cells of most grid levels (rays_close), all first samples, all second ones and so on
// (2^20 samples of a 1920-pixel frame: 219 -> 196 us).  A warp per 32 rays.
__global__ void __launch_bounds__(256) march_order_kernel(const float3 aabb_min, const float3 aabb_max, const float3* __restrict__ rays_o,
                                                          const float3* __restrict__ rays_d, uint32_t ray_begin, uint32_t ray_count,
                                                          const uint32_t* __restrict__ num_steps, const uint32_t* __restrict__ offsets,
                                                          uint32_t sample_base, uint32_t* __restrict__ order) {
    after_previous();
    constexpr uint32_t FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31, local = (((blockIdx.x * blockDim.x + threadIdx.x) >> 5) << 5) + lane;
    if (local - lane >= ray_count) return;
    const bool mine = local < ray_count;
    const uint32_t i = ray_begin + min(local, ray_count - 1);
    const uint32_t count = mine ? num_steps[i] : 0u, off = offsets[i] - sample_base;   // read for lanes with samples only
    if (rays_close<32>(rays_o[i], rays_d[i], aabb_min, aabb_max, lane)) {
        uint32_t at = __shfl_sync(FULL, off, 0);
        for (uint32_t k = 0;; k++) {
            const uint32_t has = __ballot_sync(FULL, k < count);
            if (has == 0) break;
            if (k < count) order[at + __popc(has & ((1u << lane) - 1u))] = off + k;
            at += __popc(has);
        }
    } else {
        for (uint32_t j = 0; j < 32; j++) {
            const uint32_t c = __shfl_sync(FULL, count, j), first = __shfl_sync(FULL, off, j);
            for (uint32_t k = lane; k < c; k += 32) order[first + k] = first + k;
        }
    }
}

// One round of front-to-back rendering: samples [round_begin, round_begin + round_width) of every ray of
// [ray_begin, ray_begin + ray_count) that is still visible (transmittance at least 1e-4 after the rounds before) and
// has that many samples.  A block plans 256 rays (count per ray, scan, ONE atomic on the round's counter for the
// block's sample range) and its threads then copy the samples out of the rows.  Sample ranges of different blocks
// land in arrival order; a ray's own samples are contiguous and in order, which is all compositing needs.  order (nullable) lists the samples for the field kernel: by place along
// the ray within groups of eight close rays (see march_order_kernel), else ray after ray.
__global__ void __launch_bounds__(256) round_emit_kernel(const float3 aabb_min, const float3 aabb_max, const float3* __restrict__ rays_o,
                                                         const float3* __restrict__ rays_d, uint32_t ray_begin, uint32_t ray_count,
                                                         const uint32_t* __restrict__ num_steps, const float* __restrict__ transmittance,
                                                         uint32_t round_begin, uint32_t round_width, const float* __restrict__ rows,
                                                         uint32_t row_stride, uint32_t capacity, uint32_t* __restrict__ counter,
                                                         unsigned long long* __restrict__ emitted_total, uint32_t* __restrict__ round_off, uint32_t* __restrict__ ray_idx_out,
                                                         float4* __restrict__ pos_out,
                                                         uint32_t* __restrict__ order) {
    after_previous();
    __shared__ uint32_t s_warp[8], s_off[257], s_base;
    __shared__ bool s_close[32];
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t local = blockIdx.x * 256 + threadIdx.x;
    uint32_t c = 0;
    if (local < ray_count) {
        const uint32_t i = ray_begin + local;
        const uint32_t n = num_steps[i];
        const bool visible = round_begin == 0 || transmittance[i] >= 1e-4f;
        if (visible && n > round_begin) c = min(n - round_begin, round_width);
    }
    uint32_t incl = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8; w++) {
        const uint32_t v = s_warp[w];
        if (w < warp) before += v;
        total += v;
    }
    if (threadIdx.x == 0) {
        s_base = total ? atomicAdd(counter, total) : 0u;
        if (total && emitted_total != nullptr) atomicAdd(emitted_total, (unsigned long long)total);
    }
    s_off[threadIdx.x] = before + incl - c;
    if (order != nullptr) {
        const uint32_t i = ray_begin + min(local, ray_count - 1);
        const bool close = rays_close<8>(rays_o[i], rays_d[i], aabb_min, aabb_max, lane);
        if ((lane & 7) == 0) s_close[threadIdx.x >> 3] = close;
    }
    if (threadIdx.x == 255) s_off[256] = total;
    __syncthreads();
    const uint32_t base = s_base;
    if (c > 0) round_off[ray_begin + local] = base + before + incl - c;
    if (base + total > capacity) return;   // cannot happen when the caller's bound holds; never write past the arrays
    copy_round_out<256, 256, 4>(s_off, s_close, base, total, ray_begin + blockIdx.x * 256, round_begin, rays_o, rays_d, aabb_min, aabb_max, rows, row_stride, ray_idx_out,
                             pos_out, order);
}

// ---- exclusive scan + cutoff --------------------------------------------------------------------------
constexpr int SCAN_BLOCK = 1024;

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t val, uint32_t* warp_sums, uint32_t& block_total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = val;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = warp_sums[lane];
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t n = __shfl_up_sync(0xffffffffu, wi, o);
            if (lane >= o) wi += n;
        }
        warp_sums[lane] = wi - w;  // exclusive prefix of the warps
        if (lane == 31) warp_sums[32] = wi;
    }
    __syncthreads();
    block_total = warp_sums[32];
    return incl - val + warp_sums[warp];
}

__global__ void __launch_bounds__(SCAN_BLOCK) scan_blocks_kernel(const uint32_t* __restrict__ in, uint32_t* __restrict__ out,
                                                                 uint32_t* __restrict__ block_sums, uint32_t n) {
    after_previous();
    __shared__ uint32_t warp_sums[33];
    uint32_t gid = blockIdx.x * SCAN_BLOCK + threadIdx.x;
    uint32_t v = gid < n ? in[gid] : 0u;
    uint32_t total;
    uint32_t ex = block_exclusive_scan(v, warp_sums, total);
    if (gid < n) out[gid] = ex;
    if (threadIdx.x == 0) block_sums[blockIdx.x] = total;
}

// One block: exclusive scan of the block sums in place, and the plan's initial state.
__global__ void __launch_bounds__(SCAN_BLOCK) scan_block_sums_kernel(uint32_t* __restrict__ block_sums, uint32_t num_blocks,
                                                                     uint32_t* __restrict__ plan, uint32_t rays_done) {
    after_previous();
    __shared__ uint32_t warp_sums[33];
    uint32_t v = threadIdx.x < num_blocks ? block_sums[threadIdx.x] : 0u;
    uint32_t total;
    uint32_t ex = block_exclusive_scan(v, warp_sums, total);
    if (threadIdx.x < num_blocks) block_sums[threadIdx.x] = ex;
    if (threadIdx.x == 0) {
        plan[0] = rays_done; plan[1] = 0u; plan[2] = 0u; plan[3] = total;
    }
}

// Adds the block prefixes and marks the cutoff: the last ray whose inclusive sample count (from the batch's
// first ray) still fits the budget.  Inclusive counts never decrease, so exactly one ray is that boundary.
__global__ void __launch_bounds__(SCAN_BLOCK) scan_finish_kernel(uint32_t* __restrict__ offsets, const uint32_t* __restrict__ num_steps,
                                                                 const uint32_t* __restrict__ block_sums, uint32_t n,
                                                                 uint32_t batch_size, uint32_t* __restrict__ plan) {
    after_previous();
    uint32_t gid = blockIdx.x * SCAN_BLOCK + threadIdx.x;
    if (gid >= n) return;
    uint32_t off = offsets[gid] + block_sums[blockIdx.x];
    offsets[gid] = off;
    uint32_t steps = num_steps[gid];
    uint32_t incl = off + steps;  // base is 0: the scan starts at ray 0
    if (incl <= batch_size) {
        bool boundary = true;
        if (gid + 1 < n) {
            // next ray's inclusive count = incl + its own count
            if (incl + num_steps[gid + 1] <= batch_size) boundary = false;
        }
        if (boundary) { plan[0] = gid + 1; plan[1] = incl; }
    }
}

// Adds the prefix of the blocks before this one (at most 1023 sums, added up by every block itself: one launch less than
// scanning them) and writes the total behind the last offset; host, when given, is a mapped copy of the offsets.
__global__ void __launch_bounds__(SCAN_BLOCK) scan_offsets_kernel(uint32_t* __restrict__ offsets, const uint32_t* __restrict__ num_steps,
                                                                  const uint32_t* __restrict__ block_sums, uint32_t n, uint32_t* __restrict__ host) {
    after_previous();
    __shared__ uint32_t warp_sums[33];
    uint32_t prefix;
    block_exclusive_scan(threadIdx.x < blockIdx.x ? block_sums[threadIdx.x] : 0u, warp_sums, prefix);
    const uint32_t gid = blockIdx.x * SCAN_BLOCK + threadIdx.x;
    if (gid >= n) return;
    const uint32_t off = offsets[gid] + prefix;
    offsets[gid] = off;
    if (host != nullptr) host[gid] = off;
    if (gid == n - 1) {
        const uint32_t total = off + num_steps[gid];
        offsets[n] = total;
        if (host != nullptr) host[n] = total;
    }
}

__global__ void plan_init_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ num_steps, uint32_t n,
                                 uint32_t rays_done, uint32_t* __restrict__ plan) {
    after_previous();
    plan[0] = rays_done; plan[1] = 0u;
    plan[2] = rays_done < n ? offsets[rays_done] : 0u;
    plan[3] = n > 0 ? offsets[n - 1] + num_steps[n - 1] : 0u;
}

// find_cutoff_ray_from_kernel, modules/NeRF/processRays.cu:771-799
__global__ void __launch_bounds__(256) cutoff_from_kernel(const uint32_t* __restrict__ offsets, const uint32_t* __restrict__ num_steps,
                                                          uint32_t n, uint32_t batch_size, uint32_t rays_done, uint32_t* __restrict__ plan) {
    after_previous();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x + rays_done;
    if (i >= n) return;
    const uint32_t base = offsets[rays_done];
    uint32_t incl = offsets[i] + num_steps[i] - base;
    if (incl <= batch_size) {
        bool boundary = true;
        if (i < n - 1 && offsets[i + 1] + num_steps[i + 1] - base <= batch_size) boundary = false;
        if (boundary) { plan[0] = i + 1; plan[1] = incl; }
    }
}

}  // namespace nb

using namespace nb;

static int check_scene(const nb_scene_desc* s, const char* who) {
    if (!s) return nb_set_error(NB_ERR_INVALID, who);
    if (s->num_cascades < 1 || s->mip_levels < 1 || s->mip_levels > MAX_MIP_LEVELS || s->samples_per_voxel < 1)
        return nb_set_error(NB_ERR_INVALID, "scene: cascades >= 1, 1 <= mip levels <= 8, samples per voxel >= 1 required");
    for (int a = 0; a < 3; a++)
        if (s->grid_res[a] == 0 || (s->grid_res[a] >> (s->mip_levels - 1)) == 0)
            return nb_set_error(NB_ERR_INVALID, "scene: grid resolution too small for the mip levels");
    return NB_OK;
}

extern "C" int nb_ray_aabb(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, int64_t num_rays, float* d_rays_d_inv,
                           float* d_nears, float* d_fars, void* stream) {
    int rc = check_scene(scene, "nb_ray_aabb: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_rays_d_inv || !d_nears || !d_fars || num_rays < 0 || num_rays > 0x7fffffff)
        return nb_set_error(NB_ERR_INVALID, "nb_ray_aabb: null pointer or bad ray count");
    if (num_rays == 0) return NB_OK;
    Scene sc = make_scene(scene);
    launch_after(ray_aabb_kernel, (unsigned)((num_rays + 255) / 256), 256, 0, (cudaStream_t)stream, 
        (uint32_t)num_rays, (const float3*)d_rays_o, (const float3*)d_rays_d, sc.aabb_min, sc.aabb_max, sc.num_cascades, (float3*)d_rays_d_inv,
        d_nears, d_fars);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_march_count(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, const float* d_rays_d_inv,
                              const float* d_nears, const float* d_fars, const uint8_t* d_bitfield, int64_t num_rays,
                              uint32_t* d_num_steps, void* stream) {
    int rc = check_scene(scene, "nb_march_count: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_rays_d_inv || !d_nears || !d_fars || !d_bitfield || !d_num_steps || num_rays < 0 || num_rays > 0x7fffffff)
        return nb_set_error(NB_ERR_INVALID, "nb_march_count: null pointer or bad ray count");
    if (num_rays == 0) return NB_OK;
    Scene sc = make_scene(scene);
    RayArrays r{(const float3*)d_rays_o, (const float3*)d_rays_d, (const float3*)d_rays_d_inv, d_nears, d_fars};
    launch_after(march_count_kernel, (unsigned)((num_rays + 255) / 256), 256, 0, (cudaStream_t)stream, sc, (uint32_t)num_rays, r, d_bitfield, d_num_steps);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_march_scan(const uint32_t* d_num_steps, uint32_t* d_ray_offsets, uint32_t* d_block_sums, int64_t num_rays,
                             uint32_t batch_size, uint32_t* d_plan, void* stream) {
    if (!d_num_steps || !d_ray_offsets || !d_block_sums || !d_plan || num_rays < 0)
        return nb_set_error(NB_ERR_INVALID, "nb_march_scan: null pointer or negative ray count");
    if (num_rays > (int64_t)SCAN_BLOCK * SCAN_BLOCK)
        return nb_set_error(NB_ERR_LIMIT, "nb_march_scan: at most 1048576 rays per chunk");
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t n = (uint32_t)num_rays;
    uint32_t blocks = (n + SCAN_BLOCK - 1) / SCAN_BLOCK;
    if (n > 0) launch_after(scan_blocks_kernel, blocks, SCAN_BLOCK, 0, st, d_num_steps, d_ray_offsets, d_block_sums, n);
    launch_after(scan_block_sums_kernel, 1, SCAN_BLOCK, 0, st, d_block_sums, blocks, d_plan, 0u);
    if (n > 0) launch_after(scan_finish_kernel, blocks, SCAN_BLOCK, 0, st, d_ray_offsets, d_num_steps, d_block_sums, n, batch_size, d_plan);
    NB_CHECK_LAUNCH();
    g_launch_count += (n > 0 ? 3 : 1);
    return NB_OK;
}

extern "C" int nb_march_cutoff(const uint32_t* d_num_steps, const uint32_t* d_ray_offsets, int64_t num_rays, uint32_t rays_done,
                               uint32_t batch_size, uint32_t* d_plan, void* stream) {
    if (!d_num_steps || !d_ray_offsets || !d_plan || num_rays < 0 || num_rays > 0x7fffffff || (int64_t)rays_done > num_rays)
        return nb_set_error(NB_ERR_INVALID, "nb_march_cutoff: null pointer or bad ray range");
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t n = (uint32_t)num_rays;
    launch_after(plan_init_kernel, 1, 1, 0, st, d_ray_offsets, d_num_steps, n, rays_done, d_plan);
    uint32_t left = n - rays_done;
    if (left > 0) launch_after(cutoff_from_kernel, (left + 255) / 256, 256, 0, st, d_ray_offsets, d_num_steps, n, batch_size, rays_done, d_plan);
    NB_CHECK_LAUNCH();
    g_launch_count += (left > 0 ? 2 : 1);
    return NB_OK;
}

extern "C" int nb_march_emit(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, const float* d_rays_d_inv,
                             const float* d_nears, const float* d_fars, const uint8_t* d_bitfield, int64_t num_rays, uint32_t rays_done,
                             int64_t max_rays_in_batch, const uint32_t* d_ray_offsets, const uint32_t* d_plan, float* d_t_out,
                             uint32_t* d_ray_idx_out, float* d_pos4_out, void* stream) {
    int rc = check_scene(scene, "nb_march_emit: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_rays_d_inv || !d_nears || !d_fars || !d_bitfield || !d_ray_offsets || !d_plan || !d_t_out ||
        !d_ray_idx_out || !d_pos4_out || num_rays < 0 || num_rays > 0x7fffffff || (int64_t)rays_done > num_rays || max_rays_in_batch < 0)
        return nb_set_error(NB_ERR_INVALID, "nb_march_emit: null pointer or bad ray range");
    if (reinterpret_cast<uintptr_t>(d_pos4_out) & 15u) return nb_set_error(NB_ERR_INVALID, "nb_march_emit: positions must be 16-byte aligned");
    int64_t span = num_rays - rays_done;
    if (max_rays_in_batch < span) span = max_rays_in_batch;
    if (span == 0) return NB_OK;
    Scene sc = make_scene(scene);
    RayArrays r{(const float3*)d_rays_o, (const float3*)d_rays_d, (const float3*)d_rays_d_inv, d_nears, d_fars};
    launch_after(march_emit_kernel, (unsigned)((span + 255) / 256), 256, 0, (cudaStream_t)stream, sc, (uint32_t)num_rays, rays_done, r, d_bitfield, d_ray_offsets,
                                                                                         d_plan, d_t_out, d_ray_idx_out, (float4*)d_pos4_out);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_march_row_stride(void) { return (int)MAX_HITS; }

// Rays of a warp: as many as leave every SM its SPLIT_WARPS * SPLIT_BLOCKS warps, at least 2.  Fewer rays than that (28 warps
// per SM asked for) cost 15-20 %: the coarse walk of a warp then has idle lanes without adding warps in flight.
static uint32_t split_rays_per_warp(uint32_t n) {
    uint32_t k = 32;
    while (k > 2 && (n + k - 1) / k < (uint32_t)nb_num_sms() * SPLIT_WARPS * SPLIT_BLOCKS) k >>= 1;
    return k;
}

// The walk and the scan of its counts.  r.nears == nullptr: the slab test is part of the walk (split walks only).
static int launch_walk(const Scene& sc, const RayArrays& r, uint32_t n, const uint8_t* bits, uint32_t* num_steps, float* rows, uint32_t* offsets,
                       uint32_t* block_sums, uint32_t* host_offsets, cudaStream_t st) {
    if (can_split(sc)) {
        const SplitScene p = make_split_scene(sc);
        const uint32_t per_warp = split_rays_per_warp(n), per_block = per_warp * SPLIT_WARPS;
        constexpr int smem = (int)sizeof(SplitWarp) * SPLIT_WARPS;
        static_assert(smem <= 48 * 1024, "no opt-in needed");
        const auto kernel = exact_reciprocals(sc) ? march_split_kernel<true> : march_split_kernel<false>;
        launch_after(kernel, (n + per_block - 1) / per_block, SPLIT_WARPS * 32, smem, st, p, n, r, per_warp, bits, num_steps, rows);
    } else {
        launch_after(march_fill_kernel, (n + 255) / 256, 256, 0, st, sc, n, r, bits, num_steps, rows, MAX_HITS);
    }
    const uint32_t blocks = (n + SCAN_BLOCK - 1) / SCAN_BLOCK;
    launch_after(scan_blocks_kernel, blocks, SCAN_BLOCK, 0, st, num_steps, offsets, block_sums, n);
    launch_after(scan_offsets_kernel, blocks, SCAN_BLOCK, 0, st, offsets, num_steps, block_sums, n, host_offsets);
    NB_CHECK_LAUNCH();
    g_launch_count += 3;
    return NB_OK;
}

extern "C" int nb_march_fill(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, const float* d_rays_d_inv,
                             const float* d_nears, const float* d_fars, const uint8_t* d_bitfield, int64_t num_rays, uint32_t* d_num_steps,
                             float* d_t_rows, uint32_t* d_ray_offsets, uint32_t* d_block_sums, void* stream) {
    int rc = check_scene(scene, "nb_march_fill: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_rays_d_inv || !d_nears || !d_fars || !d_bitfield || !d_num_steps || !d_t_rows || !d_ray_offsets ||
        !d_block_sums || num_rays < 0)
        return nb_set_error(NB_ERR_INVALID, "nb_march_fill: null pointer or negative ray count");
    if (num_rays > (int64_t)SCAN_BLOCK * SCAN_BLOCK) return nb_set_error(NB_ERR_LIMIT, "nb_march_fill: at most 1048576 rays per call");
    if (num_rays == 0) return nb_zero_async(d_ray_offsets, sizeof(uint32_t), stream);
    const RayArrays r{(const float3*)d_rays_o, (const float3*)d_rays_d, (const float3*)d_rays_d_inv, d_nears, d_fars};
    return launch_walk(make_scene(scene), r, (uint32_t)num_rays, d_bitfield, d_num_steps, d_t_rows, d_ray_offsets, d_block_sums, nullptr,
                       (cudaStream_t)stream);
}

extern "C" int nb_march_walk(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, float* d_rays_d_inv, float* d_nears,
                             float* d_fars, const uint8_t* d_bitfield, int64_t num_rays, uint32_t* d_num_steps, float* d_t_rows,
                             uint32_t* d_ray_offsets, uint32_t* d_block_sums, uint32_t* h_ray_offsets, void* stream) {
    int rc = check_scene(scene, "nb_march_walk: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_rays_d_inv || !d_nears || !d_fars || !d_bitfield || !d_num_steps || !d_t_rows || !d_ray_offsets ||
        !d_block_sums || !h_ray_offsets || num_rays < 0)
        return nb_set_error(NB_ERR_INVALID, "nb_march_walk: null pointer or negative ray count");
    if (num_rays == 0 || num_rays > (int64_t)SCAN_BLOCK * SCAN_BLOCK)
        return nb_set_error(NB_ERR_LIMIT, "nb_march_walk: 1 to 1048576 rays per call");
    const Scene sc = make_scene(scene);
    RayArrays r{(const float3*)d_rays_o, (const float3*)d_rays_d, nullptr, nullptr, nullptr};
    if (!can_split(sc)) {
        rc = nb_ray_aabb(scene, d_rays_o, d_rays_d, num_rays, d_rays_d_inv, d_nears, d_fars, stream);
        if (rc) return rc;
        r.d_inv = (const float3*)d_rays_d_inv; r.nears = d_nears; r.fars = d_fars;
    }
    return launch_walk(sc, r, (uint32_t)num_rays, d_bitfield, d_num_steps, d_t_rows, d_ray_offsets, d_block_sums, h_ray_offsets, (cudaStream_t)stream);
}

extern "C" int nb_march_compact(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, uint32_t ray_begin,
                                uint32_t ray_count, const uint32_t* d_num_steps, const uint32_t* d_ray_offsets, uint32_t sample_base,
                                const float* d_t_rows, float* d_t_out, uint32_t* d_ray_idx_out, float* d_pos4_out, void* stream) {
    int rc = check_scene(scene, "nb_march_compact: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_num_steps || !d_ray_offsets || !d_t_rows || !d_t_out || !d_ray_idx_out || !d_pos4_out)
        return nb_set_error(NB_ERR_INVALID, "nb_march_compact: null pointer");
    if (reinterpret_cast<uintptr_t>(d_pos4_out) & 15u) return nb_set_error(NB_ERR_INVALID, "nb_march_compact: positions must be 16-byte aligned");
    if (ray_count == 0) return NB_OK;
    Scene sc = make_scene(scene);
    const uint64_t threads = (uint64_t)ray_count * 32;
    launch_after(march_compact_kernel, (unsigned)((threads + 255) / 256), 256, 0, (cudaStream_t)stream, 
        sc.aabb_min, sc.aabb_max, (const float3*)d_rays_o, (const float3*)d_rays_d, ray_begin, ray_count, d_num_steps, d_ray_offsets, sample_base,
        d_t_rows, MAX_HITS, d_t_out, d_ray_idx_out, (float4*)d_pos4_out);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_march_order(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, uint32_t ray_begin, uint32_t ray_count,
                              const uint32_t* d_num_steps, const uint32_t* d_ray_offsets, uint32_t sample_base, uint32_t* d_order, void* stream) {
    int rc = check_scene(scene, "nb_march_order: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_num_steps || !d_ray_offsets || !d_order) return nb_set_error(NB_ERR_INVALID, "nb_march_order: null pointer");
    if (ray_count == 0) return NB_OK;
    const Scene sc = make_scene(scene);
    launch_after(march_order_kernel, (ray_count + 255) / 256, 256, 0, (cudaStream_t)stream, sc.aabb_min, sc.aabb_max, (const float3*)d_rays_o,
                 (const float3*)d_rays_d, ray_begin, ray_count, d_num_steps, d_ray_offsets, sample_base, d_order);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_march_round_emit_order(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, uint32_t ray_begin,
                                   uint32_t ray_count, const uint32_t* d_num_steps, const float* d_transmittance, uint32_t round_begin,
                                   uint32_t round_width, const float* d_t_rows, uint32_t capacity, uint32_t* d_counter,
                                   uint64_t* d_emitted_total, uint32_t* d_round_offsets, uint32_t* d_ray_idx_out, float* d_pos4_out,
                                   uint32_t* d_order, void* stream) {
    int rc = check_scene(scene, "nb_march_round_emit: null scene");
    if (rc) return rc;
    if (!d_rays_o || !d_rays_d || !d_num_steps || !d_t_rows || !d_counter || !d_round_offsets || !d_ray_idx_out || !d_pos4_out ||
        (round_begin > 0 && !d_transmittance))
        return nb_set_error(NB_ERR_INVALID, "nb_march_round_emit: null pointer");
    if (round_width == 0 || round_begin >= (uint32_t)MAX_HITS)
        return nb_set_error(NB_ERR_INVALID, "nb_march_round_emit: the round must lie inside a row");
    if (reinterpret_cast<uintptr_t>(d_pos4_out) & 15u)
        return nb_set_error(NB_ERR_INVALID, "nb_march_round_emit: positions must be 16-byte aligned");
    if (ray_count == 0) return NB_OK;
    Scene sc = make_scene(scene);
    launch_after(round_emit_kernel, (ray_count + 255) / 256, 256, 0, (cudaStream_t)stream, 
        sc.aabb_min, sc.aabb_max, (const float3*)d_rays_o, (const float3*)d_rays_d, ray_begin, ray_count, d_num_steps, d_transmittance, round_begin,
        round_width, d_t_rows, MAX_HITS, capacity, d_counter, (unsigned long long*)d_emitted_total, d_round_offsets, d_ray_idx_out,
        (float4*)d_pos4_out, d_order);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_march_round_emit(const nb_scene_desc* scene, const float* d_rays_o, const float* d_rays_d, uint32_t ray_begin,
                                   uint32_t ray_count, const uint32_t* d_num_steps, const float* d_transmittance, uint32_t round_begin,
                                   uint32_t round_width, const float* d_t_rows, uint32_t capacity, uint32_t* d_counter,
                                   uint64_t* d_emitted_total, uint32_t* d_round_offsets, uint32_t* d_ray_idx_out, float* d_pos4_out,
                                   void* stream) {
    return nb_march_round_emit_order(scene, d_rays_o, d_rays_d, ray_begin, ray_count, d_num_steps, d_transmittance, round_begin, round_width, d_t_rows, capacity,
                                     d_counter, d_emitted_total, d_round_offsets, d_ray_idx_out, d_pos4_out, nullptr, stream);
}
