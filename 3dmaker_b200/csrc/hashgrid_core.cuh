// Device pieces of the multiresolution hash grid shared by the stand-alone and the fused kernels: level geometry,
// corner indices and weights of one (point, level), the fixed-order trilinear blend and the CTA-wide encode of a
// 128-point tile into shared memory.  Arithmetic follows modules/TinyMLP/networkFusionHashtable.cu:62-70,111-222.
#pragma once

#include <atomic>

#include "mlp_core.cuh"

namespace nb {

extern std::atomic<int> g_pair_ops;   // nb_set_tuning("pair_ops", ...)
extern std::atomic<int> g_run_merge;  // nb_set_tuning("scatter_run_merge", ...)
extern std::atomic<int> g_grad_table_half;        // nb_set_tuning("grad_table_half", ...)
extern std::atomic<int> g_grad_table_scale_log2;  // nb_set_tuning("grad_table_scale_log2", ...)
inline float grad_table_scale() { return g_grad_table_half.load() ? (float)(1u << g_grad_table_scale_log2.load()) : 1.0f; }

struct GridParams {
    int L, T, dls;
    int ls;        // entries between the starts of consecutive levels in the table and its gradient: T for a whole grid,
                   // ranks * T for the view of the levels one rank owns (level_view)
    int run_merge; // > 0: the gradient scatter sums runs of consecutive samples in one cell before reducing, in warps that
                   // have at most this many runs (merging costs about 300 instructions per warp and level)
    int pair_ops;  // non-zero: where one lane handles all corners, x-neighbours that share an aligned slot pair move as one access
    int grad_half; // non-zero: the table gradient is one __half2 per entry (4 bytes), every contribution multiplied by
    float grad_scale;  // grad_scale before it is rounded to fp16; zero: two floats per entry, unscaled
    float scales[NB_MAX_LEVELS];   // forward (encode) resolutions
    float sscales[NB_MAX_LEVELS];  // resolutions of the gradient scatter
};

inline GridParams make_params(const nb_grid_desc* d) {
    GridParams p;
    p.L = d->num_levels; p.T = d->table_size; p.ls = d->table_size; p.dls = d->dense_level_start; p.pair_ops = g_pair_ops.load(); p.run_merge = g_run_merge.load();
    p.grad_half = g_grad_table_half.load() != 0; p.grad_scale = grad_table_scale();
    for (int i = 0; i < NB_MAX_LEVELS; i++) { p.scales[i] = d->scales[i]; p.sscales[i] = d->scatter_scales[i]; }
    return p;
}

// The grid as the owner of levels rank, rank + ranks, rank + 2 ranks, ... sees it: those levels renumbered 0, 1, ...,
// resolutions picked accordingly, consecutive levels ranks * T entries apart.  Pointers into the table or its gradient
// that go with this view start at level `rank` (first_level_offset entries into the array).  Dense levels stay a prefix
// because resolutions grow with the level.
inline GridParams level_view(const GridParams& whole, int rank, int ranks) {
    GridParams p = whole;
    p.L = whole.L / ranks;
    p.ls = whole.T * ranks;
    p.dls = 0;
    for (int k = 0; k < p.L; k++) {
        const int l = rank + k * ranks;
        p.scales[k] = whole.scales[l]; p.sscales[k] = whole.sscales[l];
        if (l < whole.dls) p.dls = k + 1;
    }
    return p;
}

__device__ __forceinline__ uint32_t hash_coords(int cx, int cy, int cz, int T) {
    return ((static_cast<uint32_t>(cx) * 1U) ^ (static_cast<uint32_t>(cy) * 2654435761U) ^
            (static_cast<uint32_t>(cz) * 805459861U)) & static_cast<uint32_t>(T - 1);
}
__device__ __forceinline__ uint32_t dense_index(int cx, int cy, int cz, int N_l) {
    return cx + cy * (N_l + 1) + cz * (N_l + 1) * (N_l + 1);
}

struct Corners {
    uint32_t idx[8];  // entry index inside the level (pairs of features), corner order 000,100,010,110,001,101,011,111
    float wx1, wy1, wz1;
    uint32_t cell;    // the low corner (x0 | y0 << 10 | z0 << 20) when the level has fewer than 1024 cells per axis, else ~0
};

// BWD_CLAMP = false: low corner clamped to [0, N_l] (forward); true: to [0, N_l - 1] (backward).
template <bool BWD_CLAMP>
__device__ __forceinline__ void corners_of(float px, float py, float pz, float scale, bool dense, int T, Corners& c) {
    int N_l = __float2int_rd(scale);
    float x_l = px * scale, y_l = py * scale, z_l = pz * scale;
    int x0 = __float2int_rd(x_l), y0 = __float2int_rd(y_l), z0 = __float2int_rd(z_l);
    const int hi = BWD_CLAMP ? N_l - 1 : N_l;
    x0 = max(0, min(x0, hi)); y0 = max(0, min(y0, hi)); z0 = max(0, min(z0, hi));
    int x1 = min(x0 + 1, N_l), y1 = min(y0 + 1, N_l), z1 = min(z0 + 1, N_l);
    c.cell = (N_l < 1024) ? ((uint32_t)x0 | ((uint32_t)y0 << 10) | ((uint32_t)z0 << 20)) : 0xffffffffu;
    c.wx1 = 1.0f - x_l + floorf(x_l);
    c.wy1 = 1.0f - y_l + floorf(y_l);
    c.wz1 = 1.0f - z_l + floorf(z_l);
    if (dense) {
        c.idx[0] = dense_index(x0, y0, z0, N_l); c.idx[1] = dense_index(x1, y0, z0, N_l);
        c.idx[2] = dense_index(x0, y1, z0, N_l); c.idx[3] = dense_index(x1, y1, z0, N_l);
        c.idx[4] = dense_index(x0, y0, z1, N_l); c.idx[5] = dense_index(x1, y0, z1, N_l);
        c.idx[6] = dense_index(x0, y1, z1, N_l); c.idx[7] = dense_index(x1, y1, z1, N_l);
    } else {
        c.idx[0] = hash_coords(x0, y0, z0, T); c.idx[1] = hash_coords(x1, y0, z0, T);
        c.idx[2] = hash_coords(x0, y1, z0, T); c.idx[3] = hash_coords(x1, y1, z0, T);
        c.idx[4] = hash_coords(x0, y0, z1, T); c.idx[5] = hash_coords(x1, y0, z1, T);
        c.idx[6] = hash_coords(x0, y1, z1, T); c.idx[7] = hash_coords(x1, y1, z1, T);
    }
}

__device__ __forceinline__ void corner_weights(const Corners& c, float (&w)[8]) {
    const float wx1 = c.wx1, wy1 = c.wy1, wz1 = c.wz1;
    w[0] = wx1 * wy1 * wz1;                   w[1] = (1 - wx1) * wy1 * wz1;
    w[2] = wx1 * (1 - wy1) * wz1;             w[3] = (1 - wx1) * (1 - wy1) * wz1;
    w[4] = wx1 * wy1 * (1 - wz1);             w[5] = (1 - wx1) * wy1 * (1 - wz1);
    w[6] = wx1 * (1 - wy1) * (1 - wz1);       w[7] = (1 - wx1) * (1 - wy1) * (1 - wz1);
}

// The 8 corner entries (feature pairs) of one level.  Corners 2j and 2j+1 differ in x only; whenever their indices
// differ in the lowest bit only (every even x0 on a hashed level, since the x prime is 1; every even low index on a
// dense level) both sit in one aligned 8-byte slot pair and are fetched with one load.
__device__ __forceinline__ void gather_corners(const uint32_t* __restrict__ tl, const Corners& c, bool pair_ops, uint32_t (&f)[8]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t a = c.idx[2 * j], b = c.idx[2 * j + 1];
        if (pair_ops && ((a ^ b) == 1u)) {
            uint2 v = __ldg(reinterpret_cast<const uint2*>(tl + (a & ~1u)));
            const bool a_hi = (a & 1u) != 0;
            f[2 * j] = a_hi ? v.y : v.x;
            f[2 * j + 1] = a_hi ? v.x : v.y;
        } else {
            f[2 * j] = __ldg(tl + a);
            f[2 * j + 1] = __ldg(tl + b);
        }
    }
}

// Fixed-order blend of the reference (networkFusionHashtable.cu:185-201), both features.
__device__ __forceinline__ uint32_t blend(const uint32_t (&f)[8], const float (&w)[8]) {
    float2 v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = unpack_half2(f[k]);
    float rx = v[7].x * w[7], ry = v[7].y * w[7];
#pragma unroll
    for (int k = 6; k >= 0; k--) {
        rx = __fmaf_rn(v[k].x, w[k], rx);
        ry = __fmaf_rn(v[k].y, w[k], ry);
    }
    return pack_half2(rx, ry);
}

// ---- lane pairs --------------------------------------------------------------------------------------------------------
// Two neighbouring lanes gather together.  Corners 2j and 2j + 1 of a cell differ in x only, and x enters the index without
// a factor (prime 1 on hashed levels, stride 1 on dense ones), so both entries lie in one 128-byte line 31 times out of 32.
// What bounds the gathers is the rate of lines a warp's load asks the L2 for, one per clock and SM (282 G/s measured, for one
// lane or several lanes per line alike), so lane 0 of a pair loads the x0 corners and lane 1 the x1 corners of one sample
// IN THE SAME INSTRUCTION, first of the even lane's sample, then of the odd lane's, and the pair swaps what belongs to the
// other: 4 lines per sample and level instead of about 4.9 (an 8-byte load where the two entries share an aligned
// slot, two loads where not), and no divergent branch.  12 hashed levels of 2^20 samples: 0.219 -> 0.187 ms.  Plain loads:
// L1::no_allocate and L1::evict_first on the hashed levels, meant to keep the coarse ones in L1, give the table away in L2 too
// and cost 0.41 and 0.50 ms where this takes 0.34 (the forward at 2^20 samples).
struct PairPos {
    float ax, ay, az, bx, by, bz;   // even and odd lane's sample, clamped to the unit cube: index arithmetic
    float px, py, pz;               // this lane's own sample as it came: interpolation weights
    bool plain;                     // every sample of the warp lies in the unit cube
};

// ALL lanes of the warp must call; a lane without a sample passes any position.
__device__ __forceinline__ void pair_positions(float px, float py, float pz, int odd, PairPos& q) {
    q.px = px; q.py = py; q.pz = pz;
    // floor(clamp(p) * scale) is clamp(floor(p * scale)) for the clamps of corners_of: floor(1 * scale) = N_l
    const float cx = fminf(fmaxf(px, 0.0f), 1.0f), cy = fminf(fmaxf(py, 0.0f), 1.0f), cz = fminf(fmaxf(pz, 0.0f), 1.0f);
    q.plain = __all_sync(0xffffffffu, cx == px && cy == py && cz == pz);
    const float ox = __shfl_xor_sync(0xffffffffu, cx, 1), oy = __shfl_xor_sync(0xffffffffu, cy, 1), oz = __shfl_xor_sync(0xffffffffu, cz, 1);
    q.ax = odd ? ox : cx; q.ay = odd ? oy : cy; q.az = odd ? oz : cz;
    q.bx = odd ? cx : ox; q.by = odd ? cy : oy; q.bz = odd ? cz : oz;
}

// floor of 0 <= v < 2^22 without the conversion unit: rounding v + 2^23 towards minus infinity leaves the integer in the low
// bits of the sum, FLOOR_BITS above it.  Levels finer than that (scale >= 2^22) take the conversion, brought to the same form.
constexpr uint32_t FLOOR_BITS = 0x4b000000u;
__device__ __forceinline__ uint32_t floor_bits(float v, bool small) {
    return small ? __float_as_uint(__fadd_rd(v, 8388608.0f)) : static_cast<uint32_t>(__float2int_rd(v)) + FLOOR_BITS;
}

// Two fp32 values per register pair and instruction: the floors of a pair's two samples, the weights and sums of two levels.
// Where neighbouring samples share lines the encoding is bound by its instructions (a 1080p frame's forward launches 200 -> 188
// us each, a preview's 155 -> 141); scattered samples, bound by their lines, do not notice (306 and 310 us at 2^20).
struct F2 { unsigned long long v; };
__device__ __forceinline__ F2 f2(float a, float b) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ float2 parts(F2 a) { float2 r; asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v)); return r; }
__device__ __forceinline__ F2 mul(F2 a, F2 b) { F2 r; asm("mul.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 add(F2 a, F2 b) { F2 r; asm("add.rn.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 add_down(F2 a, F2 b) { F2 r; asm("add.rm.ftz.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 fma(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.ftz.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
__device__ __forceinline__ F2 one_minus(F2 a) { return fma(a, f2(-1.0f, -1.0f), f2(1.0f, 1.0f)); }

// Byte offsets inside a level of the four (y, z) corners of one sample on the lane's x side, and their loads; bx, by, bz are the
// floor_bits of its corner.  The hash is taken on coordinates times four (XOR and the mask commute with the shift), so the offset
// needs no address arithmetic.
__device__ __forceinline__ void pair_gather(const uint32_t* __restrict__ tl, uint32_t bx, uint32_t by, uint32_t bz, int N_l, bool dense, uint32_t mask4,
                                            int odd, uint32_t (&f)[4]) {
    const uint32_t x = min(static_cast<int>(bx + (odd - FLOOR_BITS)), N_l);   // the low corner is at most N_l
    const uint32_t y1 = min(static_cast<int>(by + (1u - FLOOR_BITS)), N_l), z1 = min(static_cast<int>(bz + (1u - FLOOR_BITS)), N_l);
    uint32_t o[4];
    if (dense) {
        const uint32_t w = 4u * (N_l + 1), wh = w * (N_l + 1);
        const uint32_t r0 = (by - FLOOR_BITS) * w + 4u * x, r1 = y1 * w + 4u * x, s0 = (bz - FLOOR_BITS) * wh, s1 = z1 * wh;
        o[0] = r0 + s0; o[1] = r1 + s0; o[2] = r0 + s1; o[3] = r1 + s1;
    } else {
        constexpr uint32_t PY = 4u * 2654435761U, PZ = 4u * 805459861U;
        const uint32_t hy0 = by * PY - FLOOR_BITS * PY, hy1 = y1 * PY, hz0 = bz * PZ - FLOOR_BITS * PZ, hz1 = z1 * PZ;
        const uint32_t ux = (4u * x) & mask4;
        o[0] = ((hy0 ^ hz0) & mask4) ^ ux; o[1] = ((hy1 ^ hz0) & mask4) ^ ux;
        o[2] = ((hy0 ^ hz1) & mask4) ^ ux; o[3] = ((hy1 ^ hz1) & mask4) ^ ux;
    }
    const char* base = reinterpret_cast<const char*>(tl);
#pragma unroll
    for (int j = 0; j < 4; j++) f[j] = __ldg(reinterpret_cast<const uint32_t*>(base + o[j]));
}

// Issues the 8 loads of one level: fa = even lane's sample, fb = odd lane's.
__device__ __forceinline__ void pair_gather_level(const uint32_t* __restrict__ tl, float scale, const PairPos& q, bool dense, int T, int odd,
                                                  uint32_t (&fa)[4], uint32_t (&fb)[4]) {
    const int N_l = __float2int_rd(scale);
    const uint32_t mask4 = 4u * static_cast<uint32_t>(T - 1);
    const F2 s = f2(scale, scale), vx = mul(f2(q.ax, q.bx), s), vy = mul(f2(q.ay, q.by), s), vz = mul(f2(q.az, q.bz), s);
    float2 x, y, z;
    if (scale < 4194304.0f) {
        const F2 magic = f2(8388608.0f, 8388608.0f);
        x = parts(add_down(vx, magic)); y = parts(add_down(vy, magic)); z = parts(add_down(vz, magic));
    } else {
        x = parts(vx); y = parts(vy); z = parts(vz);
        float* const c[6] = {&x.x, &x.y, &y.x, &y.y, &z.x, &z.y};
#pragma unroll
        for (int i = 0; i < 6; i++) *c[i] = __uint_as_float(floor_bits(*c[i], false));
    }
    pair_gather(tl, __float_as_uint(x.x), __float_as_uint(y.x), __float_as_uint(z.x), N_l, dense, mask4, odd, fa);
    pair_gather(tl, __float_as_uint(x.y), __float_as_uint(y.y), __float_as_uint(z.y), N_l, dense, mask4, odd, fb);
}

// corner_weights and blend of two levels for the lane's own sample, the same operations in the same order: fa, fb = the 8 corner
// entries on the level of the first halves and on that of the second; xl, yl, zl = the scaled position, fx, fy, fz its floors.
__device__ __forceinline__ uint2 blend_at(const uint32_t (&fa)[8], const uint32_t (&fb)[8], F2 xl, F2 yl, F2 zl, F2 fx, F2 fy, F2 fz) {
    const F2 wx1 = add(one_minus(xl), fx), wy1 = add(one_minus(yl), fy), wz1 = add(one_minus(zl), fz);
    const F2 wx0 = one_minus(wx1), wy0 = one_minus(wy1), wz0 = one_minus(wz1);
    const F2 w11 = mul(wx1, wy1), w01 = mul(wx0, wy1), w10 = mul(wx1, wy0), w00 = mul(wx0, wy0);
    const F2 w[8] = {mul(w11, wz1), mul(w01, wz1), mul(w10, wz1), mul(w00, wz1), mul(w11, wz0), mul(w01, wz0), mul(w10, wz0), mul(w00, wz0)};
    F2 rx, ry;
#pragma unroll
    for (int k = 7; k >= 0; k--) {
        const float2 a = unpack_half2(fa[k]), b = unpack_half2(fb[k]);
        rx = k == 7 ? mul(f2(a.x, b.x), w[k]) : fma(f2(a.x, b.x), w[k], rx);
        ry = k == 7 ? mul(f2(a.y, b.y), w[k]) : fma(f2(a.y, b.y), w[k], ry);
    }
    const float2 x = parts(rx), y = parts(ry);
    return make_uint2(pack_half2(x.x, y.x), pack_half2(x.y, y.y));
}
__device__ __forceinline__ uint2 blend_two(const uint32_t (&fa)[8], const uint32_t (&fb)[8], const PairPos& q, float2 scale) {
    const F2 s = f2(scale.x, scale.y), xl = mul(f2(q.px, q.px), s), yl = mul(f2(q.py, q.py), s), zl = mul(f2(q.pz, q.pz), s);
    F2 fx, fy, fz;
    if (q.plain && fmaxf(scale.x, scale.y) < 4194304.0f) {
        const F2 magic = f2(8388608.0f, 8388608.0f), back = f2(-8388608.0f, -8388608.0f);
        fx = add(add_down(xl, magic), back); fy = add(add_down(yl, magic), back); fz = add(add_down(zl, magic), back);
    } else {
        const float2 x = parts(xl), y = parts(yl), z = parts(zl);
        fx = f2(floorf(x.x), floorf(x.y)); fy = f2(floorf(y.x), floorf(y.y)); fz = f2(floorf(z.x), floorf(z.y));
    }
    return blend_at(fa, fb, xl, yl, zl, fx, fy, fz);
}

// Swaps the pair's corners: f = the 8 corners of the lane's own sample.
__device__ __forceinline__ void pair_swap(const uint32_t (&fa)[4], const uint32_t (&fb)[4], int odd, uint32_t (&f)[8]) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
        const uint32_t other = __shfl_xor_sync(0xffffffffu, odd ? fa[j] : fb[j], 1);
        f[2 * j] = odd ? other : fa[j];      // x0 corner
        f[2 * j + 1] = odd ? fb[j] : other;  // x1 corner
    }
}

// Levels la and lb of the lane's own sample; 16 gathers in flight.
__device__ __forceinline__ uint2 pair_encode_two(const GridParams& gp, const uint32_t* __restrict__ table2, int la, int lb, const PairPos& q, int odd) {
    const float2 scale = make_float2(gp.scales[la], gp.scales[lb]);
    uint32_t a[2][4], b[2][4], fa[8], fb[8];
    pair_gather_level(table2 + (size_t)la * gp.ls, scale.x, q, la < gp.dls, gp.T, odd, a[0], a[1]);
    pair_gather_level(table2 + (size_t)lb * gp.ls, scale.y, q, lb < gp.dls, gp.T, odd, b[0], b[1]);
    pair_swap(a[0], a[1], odd, fa);
    pair_swap(b[0], b[1], odd, fb);
    return blend_two(fa, fb, q, scale);
}

// The 8 corners of the lane's own sample on one level; bx, by, bz are the floor_bits of its corner.
__device__ __forceinline__ void own_gather(const uint32_t* __restrict__ tl, uint32_t bx, uint32_t by, uint32_t bz, int N_l, bool dense, uint32_t mask4,
                                           uint32_t (&f)[8]) {
    const uint32_t x1 = min(static_cast<int>(bx + (1u - FLOOR_BITS)), N_l), y1 = min(static_cast<int>(by + (1u - FLOOR_BITS)), N_l),
                   z1 = min(static_cast<int>(bz + (1u - FLOOR_BITS)), N_l);
    uint32_t o[8];
    if (dense) {
        const uint32_t w = 4u * (N_l + 1), wh = w * (N_l + 1);
        const uint32_t r0 = (by - FLOOR_BITS) * w, r1 = y1 * w, s0 = (bz - FLOOR_BITS) * wh, s1 = z1 * wh, x0 = 4u * (bx - FLOOR_BITS), xx = 4u * x1;
        const uint32_t yz[4] = {r0 + s0, r1 + s0, r0 + s1, r1 + s1};
#pragma unroll
        for (int j = 0; j < 4; j++) { o[2 * j] = yz[j] + x0; o[2 * j + 1] = yz[j] + xx; }
    } else {
        constexpr uint32_t PY = 4u * 2654435761U, PZ = 4u * 805459861U;
        const uint32_t hy0 = by * PY - FLOOR_BITS * PY, hy1 = y1 * PY, hz0 = bz * PZ - FLOOR_BITS * PZ, hz1 = z1 * PZ;
        const uint32_t x0 = (4u * (bx - FLOOR_BITS)) & mask4, xx = (4u * x1) & mask4;
        const uint32_t yz[4] = {(hy0 ^ hz0) & mask4, (hy1 ^ hz0) & mask4, (hy0 ^ hz1) & mask4, (hy1 ^ hz1) & mask4};
#pragma unroll
        for (int j = 0; j < 4; j++) { o[2 * j] = yz[j] ^ x0; o[2 * j + 1] = yz[j] ^ xx; }
    }
    const char* base = reinterpret_cast<const char*>(tl);
#pragma unroll
    for (int j = 0; j < 8; j++) f[j] = __ldg(reinterpret_cast<const uint32_t*>(base + o[j]));
}

// pair_encode_two with each lane gathering for itself: a fifth fewer instructions - no swaps, floors shared by index and weights -, more
// lines where the lanes of a warp are far apart.  1920x1080 frame with close samples side by side 21.4 -> 19.6 ms; rays of 2^18 training
// samples 63.7 -> 67, and a choice per level in one kernel costs the other callers 2 to 4 % for the second loop.
__device__ __forceinline__ uint2 own_encode_two(const GridParams& gp, const uint32_t* __restrict__ table2, int la, int lb, const PairPos& q, int odd) {
    const float2 scale = make_float2(gp.scales[la], gp.scales[lb]);
    if (!q.plain || fmaxf(scale.x, scale.y) >= 4194304.0f) return pair_encode_two(gp, table2, la, lb, q, odd);   // the same for the warp
    const F2 s = f2(scale.x, scale.y), xl = mul(f2(q.px, q.px), s), yl = mul(f2(q.py, q.py), s), zl = mul(f2(q.pz, q.pz), s);
    const F2 magic = f2(8388608.0f, 8388608.0f), back = f2(-8388608.0f, -8388608.0f);
    const F2 tx = add_down(xl, magic), ty = add_down(yl, magic), tz = add_down(zl, magic);
    const float2 x = parts(tx), y = parts(ty), z = parts(tz);
    const uint32_t mask4 = 4u * static_cast<uint32_t>(gp.T - 1);
    uint32_t fa[8], fb[8];
    own_gather(table2 + (size_t)la * gp.ls, __float_as_uint(x.x), __float_as_uint(y.x), __float_as_uint(z.x), __float2int_rd(scale.x), la < gp.dls, mask4, fa);
    own_gather(table2 + (size_t)lb * gp.ls, __float_as_uint(x.y), __float_as_uint(y.y), __float_as_uint(z.y), __float2int_rd(scale.y), lb < gp.dls, mask4, fb);
    return blend_at(fa, fb, xl, yl, zl, add(tx, back), add(ty, back), add(tz, back));
}

// One level of the lane's own sample from a copy of the level's dense grid in shared memory (32 banks serve random entries
// about three times as fast as L1 does, and they leave the lines of the other levels alone).
__device__ __forceinline__ void staged_level(const uint32_t* __restrict__ s, float scale, const PairPos& q, int odd, uint32_t (&f)[8]) {
    const int N_l = __float2int_rd(scale), w = N_l + 1, wh = w * w;
    const int x0 = floor_bits(__fmul_rn(odd ? q.bx : q.ax, scale), true) - FLOOR_BITS, y0 = floor_bits(__fmul_rn(odd ? q.by : q.ay, scale), true) - FLOOR_BITS,
              z0 = floor_bits(__fmul_rn(odd ? q.bz : q.az, scale), true) - FLOOR_BITS;
    const int x1 = min(x0 + 1, N_l), r0 = y0 * w, r1 = min(y0 + 1, N_l) * w, s0 = z0 * wh, s1 = min(z0 + 1, N_l) * wh;
    const int o[8] = {x0 + r0 + s0, x1 + r0 + s0, x0 + r1 + s0, x1 + r1 + s0, x0 + r0 + s1, x1 + r0 + s1, x0 + r1 + s1, x1 + r1 + s1};
#pragma unroll
    for (int k = 0; k < 8; k++) f[k] = s[o[k]];
}

// Encodes the CTA's 128 points into the shared tile: tile[r][2l .. 2l+1].  Thread = (row, every other level), so that both
// halves of the CTA get coarse and fine levels; two levels at a time keep 16 gathers in flight per thread.
template <int TILE_STRIDE>
__device__ __forceinline__ void encode_tile(const GridParams& gp, const float* __restrict__ pos4, const uint32_t* __restrict__ table2,
                                            int64_t row_base, int64_t n, __half* tile, int tid) {
    const int r = tid & (TILE_ROWS - 1), hsel = tid >> 7, odd = tid & 1;
    const int64_t row = row_base + r;
    const bool has = row < n;
    float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
    if (has) p = ld_nc_f4(pos4 + row * 4);
    PairPos q;
    pair_positions(p.x, p.y, p.z, odd, q);
    uint32_t* dst = reinterpret_cast<uint32_t*>(&tile[r * TILE_STRIDE]);
    for (int la = hsel; la < gp.L; la += 4) {
        const int lb = la + 2;
        const bool has_b = lb < gp.L;
        const uint2 e = pair_encode_two(gp, table2, la, has_b ? lb : la, q, odd);
        dst[la] = has ? e.x : 0u;
        if (has_b) dst[lb] = has ? e.y : 0u;
    }
}

// ---- gradient scatter ----------------------------------------------------------------------------------------------------
// Adds the gradient of one level of the warp's 32 samples to the table gradient: 8 corner entries per sample.  Backward clamp
// and scatter resolution as hashTableScatter_Backward (networkFusionBackwardHashtable.cu:797-900).
//
// Lane pairs again: what the L2 charges for is a reduction request per 32-byte sector (185 to 215 G/s for 4, 8 and 16 bytes in
// it alike), and the requests of a warp's instruction that fall into one sector travel as one.  Lane 0 of a pair adds to the x0
// corners and lane 1 to the x1 corners of the same sample in the same instruction: the two 8-byte entries share a sector three
// times out of four, 1.25 requests per corner pair instead of 1.5 with a 16-byte reduction where they share an aligned
// slot.  12 hashed levels of 2^20 scattered samples: 0.354 -> 0.289 ms.
//
// Samples that arrive in ray order stay inside one cell of the coarser levels for many consecutive samples.  Lanes that follow
// each other in the same cell form a run; while the warp has few runs their contributions are summed across the run with
// shuffles and only the run's first lane issues reductions (the reference merges equal addresses inside a warp on its dense
// levels for the same reason, networkFusionBackwardHashtable.cu:843-887).  Finer levels have more runs: the first level
// with too many ends the looking for this warp's samples.
struct ScatterState {
    float px, py, pz;               // this lane's sample
    float ax, ay, az, bx, by, bz;   // the even and the odd lane's sample
    bool plain;                     // every sample of the warp lies in the unit cube
    bool merging;
};

// ALL 32 LANES MUST CALL; lanes without a sample pass any position.
__device__ __forceinline__ void scatter_begin_warp(const GridParams& gp, float px, float py, float pz, int lane, ScatterState& st) {
    const bool odd = lane & 1;
    st.px = px; st.py = py; st.pz = pz;
    const float ox = __shfl_xor_sync(0xffffffffu, px, 1), oy = __shfl_xor_sync(0xffffffffu, py, 1), oz = __shfl_xor_sync(0xffffffffu, pz, 1);
    st.ax = odd ? ox : px; st.ay = odd ? oy : py; st.az = odd ? oz : pz;
    st.bx = odd ? px : ox; st.by = odd ? py : oy; st.bz = odd ? pz : oz;
    st.plain = __all_sync(0xffffffffu, px >= 0.0f && px <= 1.0f && py >= 0.0f && py <= 1.0f && pz >= 0.0f && pz <= 1.0f);
    st.merging = gp.run_merge > 0;
}

// One coordinate: low corner and the weight of it.
__device__ __forceinline__ void scatter_axis(float v, bool small, int hi, int& c0, float& w1) {
    float fl;
    if (small) {
        const float s = __fadd_rd(v, 8388608.0f);   // floor_bits
        c0 = min(__float_as_int(s) - static_cast<int>(FLOOR_BITS), hi);
        fl = s - 8388608.0f;
    } else {
        c0 = max(0, min(__float2int_rd(v), hi));
        fl = floorf(v);
    }
    w1 = __fadd_rn(__fsub_rn(1.0f, v), fl);
}

// The four (y, z) corners of one sample on the lane's x side.
template <bool GRAD_HALF>
__device__ __forceinline__ void scatter_side(const GridParams& gp, float x, float y, float z, float scale, bool small, bool dense, float2 g, bool odd,
                                             void* __restrict__ base) {
    const int N_l = __float2int_rd(scale);
    int x0, y0, z0;
    float wx1, wy1, wz1;
    scatter_axis(__fmul_rn(x, scale), small, N_l - 1, x0, wx1);
    scatter_axis(__fmul_rn(y, scale), small, N_l - 1, y0, wy1);
    scatter_axis(__fmul_rn(z, scale), small, N_l - 1, z0, wz1);
    const float wx = odd ? 1.0f - wx1 : wx1, wy0 = 1.0f - wy1, wz0 = 1.0f - wz1;
    const float wxy1 = wx * wy1, wxy0 = wx * wy0;
    const float w[4] = {wxy1 * wz1, wxy0 * wz1, wxy1 * wz0, wxy0 * wz0};
    const uint32_t ux = static_cast<uint32_t>(x0) + (odd ? 1u : 0u), uy = static_cast<uint32_t>(y0), uz = static_cast<uint32_t>(z0);
    uint32_t e[4];
    if (dense) {
        const uint32_t w1 = static_cast<uint32_t>(N_l) + 1u, i0 = (uz * w1 + uy) * w1 + ux;
        e[0] = i0; e[1] = i0 + w1; e[2] = i0 + w1 * w1; e[3] = e[2] + w1;
    } else {
        const uint32_t m = static_cast<uint32_t>(gp.T - 1);
        const uint32_t hy0 = uy * 2654435761U, hy1 = hy0 + 2654435761U, hz0 = uz * 805459861U, hz1 = hz0 + 805459861U;
        e[0] = (ux ^ hy0 ^ hz0) & m; e[1] = (ux ^ hy1 ^ hz0) & m; e[2] = (ux ^ hy0 ^ hz1) & m; e[3] = (ux ^ hy1 ^ hz1) & m;
    }
#pragma unroll
    for (int j = 0; j < 4; j++) {
        if constexpr (GRAD_HALF) red_add_h2(reinterpret_cast<uint32_t*>(base) + e[j], pack_half2(g.x * w[j] * gp.grad_scale, g.y * w[j] * gp.grad_scale));
        else red_add_v2(reinterpret_cast<float*>(base) + 2 * static_cast<size_t>(e[j]), g.x * w[j], g.y * w[j]);
    }
}

// Sums the 16 contributions of lanes that form a run (equal `run`) into the run's first lane.
__device__ __forceinline__ void sum_runs(float (&v)[16], unsigned heads, int lane) {
    const int run = __popc(heads & (0xffffffffu >> (31 - lane)));  // index of this lane's run
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int other = __shfl_down_sync(0xffffffffu, run, o);
        const bool same = (lane + o < 32) && other == run;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const float n = __shfl_down_sync(0xffffffffu, v[k], o);
            if (same) v[k] += n;
        }
    }
}

// Lanes that start a run of samples in one cell; inactive lanes and levels too fine for a cell key never join one.
__device__ __forceinline__ unsigned run_heads(const Corners& c, bool active, int lane) {
    const uint32_t key = (active && c.cell != 0xffffffffu) ? c.cell : (0xc0000000u | (uint32_t)lane);
    const uint32_t below = __shfl_up_sync(0xffffffffu, key, 1);
    return __ballot_sync(0xffffffffu, lane == 0 || key != below);
}

// v[2k], v[2k + 1] = the two features' contributions to corner k.
__device__ __forceinline__ void corner_contributions(const Corners& c, float2 g, float (&v)[16]) {
    float w[8];
    corner_weights(c, w);
#pragma unroll
    for (int k = 0; k < 8; k++) { v[2 * k] = g.x * w[k]; v[2 * k + 1] = g.y * w[k]; }
}

// packed = this lane's gradient pair on the level (two halves; 0 for a lane without a sample).  Levels in ascending order.
// base = where the level's gradient starts.  GRAD_HALF is a compile-time choice (kernels exist in both forms and the launchers pick by
// gp.grad_half).
template <bool GRAD_HALF>
__device__ __forceinline__ void scatter_level_at(const GridParams& gp, int level, ScatterState& st, uint32_t packed, void* __restrict__ base, int lane) {
    const float scale = gp.sscales[level];
    const bool dense = level < gp.dls;
    if (st.merging) {
        const float2 g = unpack_half2(packed);
        const bool active = g.x != 0.f || g.y != 0.f;
        Corners c;
        corners_of<true>(st.px, st.py, st.pz, scale, dense, gp.T, c);
        const unsigned heads = run_heads(c, active, lane);
        if (__popc(heads) <= gp.run_merge) {
            float v[16];
            corner_contributions(c, g, v);
            sum_runs(v, heads, lane);
            if (((heads >> lane) & 1u) && active) {
                // one lane has all 8 corners: x-neighbours in one aligned slot pair as one 16-byte (8-byte) reduction
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const uint32_t a = c.idx[2 * j], b = c.idx[2 * j + 1];
                    const bool pair = gp.pair_ops != 0 && (a ^ b) == 1u, a_hi = (a & 1u) != 0;
                    if constexpr (GRAD_HALF) {
                        const float s = gp.grad_scale;
                        const uint32_t va = pack_half2(v[4 * j] * s, v[4 * j + 1] * s), vb = pack_half2(v[4 * j + 2] * s, v[4 * j + 3] * s);
                        uint32_t* t = reinterpret_cast<uint32_t*>(base);
                        if (pair) red_add_h2x2(t + (a & ~1u), a_hi ? vb : va, a_hi ? va : vb);
                        else { red_add_h2(t + a, va); red_add_h2(t + b, vb); }
                    } else {
                        float* t = reinterpret_cast<float*>(base);
                        if (pair)
                            red_add_v4(t + (size_t)(a & ~1u) * 2, a_hi ? v[4 * j + 2] : v[4 * j], a_hi ? v[4 * j + 3] : v[4 * j + 1],
                                       a_hi ? v[4 * j] : v[4 * j + 2], a_hi ? v[4 * j + 1] : v[4 * j + 3]);
                        else { red_add_v2(t + (size_t)a * 2, v[4 * j], v[4 * j + 1]); red_add_v2(t + (size_t)b * 2, v[4 * j + 2], v[4 * j + 3]); }
                    }
                }
            }
            return;
        }
        st.merging = false;
    }
    const bool odd = lane & 1, small = st.plain && scale < 4194304.0f;
    const uint32_t theirs = __shfl_xor_sync(0xffffffffu, packed, 1);
    const float2 ga = unpack_half2(odd ? theirs : packed), gb = unpack_half2(odd ? packed : theirs);
    if (ga.x != 0.f || ga.y != 0.f) scatter_side<GRAD_HALF>(gp, st.ax, st.ay, st.az, scale, small, dense, ga, odd, base);
    if (gb.x != 0.f || gb.y != 0.f) scatter_side<GRAD_HALF>(gp, st.bx, st.by, st.bz, scale, small, dense, gb, odd, base);
}

// ... into the table's gradient.
template <bool GRAD_HALF = false>
__device__ __forceinline__ void scatter_level_warp(const GridParams& gp, int level, ScatterState& st, uint32_t packed, float* __restrict__ grads,
                                                   int lane) {
    scatter_level_at<GRAD_HALF>(gp, level, st, packed,
                                GRAD_HALF ? (void*)(reinterpret_cast<uint32_t*>(grads) + (size_t)level * gp.ls) : (void*)(grads + (size_t)level * gp.ls * 2), lane);
}

// ---- coarse levels from shared memory ------------------------------------------------------------------------------
// When the samples a CTA works on lie close together, the corners they touch on a coarse level form a small box of the
// level's grid.  The CTA then copies that box into shared memory once (forward) or accumulates into it and adds it to the
// table gradient once (backward) instead of going to L2 eight times per sample and level.  Which levels are staged is
// decided per group of tiles from the bounding box of the group's positions: levels 0, 1, ... as long as their boxes fit
// the capacity.  Works for any sample order; nb_sample_order makes the boxes small.
struct StagePlan {
    int count;                                  // levels [0, count) are staged
    int ox[NB_MAX_LEVELS], oy[NB_MAX_LEVELS], oz[NB_MAX_LEVELS];   // lowest corner of the box, in corner coordinates
    int w[NB_MAX_LEVELS], wh[NB_MAX_LEVELS], whd[NB_MAX_LEVELS];   // extent in x, x * y, x * y * z (= entries)
    int h[NB_MAX_LEVELS], d[NB_MAX_LEVELS];                        // extent in y and z
    int base[NB_MAX_LEVELS];                    // first entry of the level in the staging array
};

// Low / high corner coordinates and interpolation weights of a point on one level (the arithmetic of corners_of).
struct CornerBox {
    int x0, y0, z0, x1, y1, z1, N_l;
    float wx1, wy1, wz1;
};

template <bool BWD_CLAMP>
__device__ __forceinline__ void corner_box(float px, float py, float pz, float scale, CornerBox& b) {
    const int N_l = __float2int_rd(scale);
    const float x_l = px * scale, y_l = py * scale, z_l = pz * scale;
    const int hi = BWD_CLAMP ? N_l - 1 : N_l;
    b.N_l = N_l;
    b.x0 = max(0, min(__float2int_rd(x_l), hi)); b.y0 = max(0, min(__float2int_rd(y_l), hi)); b.z0 = max(0, min(__float2int_rd(z_l), hi));
    b.x1 = min(b.x0 + 1, N_l); b.y1 = min(b.y0 + 1, N_l); b.z1 = min(b.z0 + 1, N_l);
    b.wx1 = 1.0f - x_l + floorf(x_l);
    b.wy1 = 1.0f - y_l + floorf(y_l);
    b.wz1 = 1.0f - z_l + floorf(z_l);
}

// Entry index of corner (x, y, z) inside its level.
__device__ __forceinline__ uint32_t level_index(int x, int y, int z, int N_l, bool dense, int T) {
    return dense ? dense_index(x, y, z, N_l) : hash_coords(x, y, z, T);
}

__device__ __forceinline__ void corners_from_box(const CornerBox& b, bool dense, int T, Corners& c) {
    c.wx1 = b.wx1; c.wy1 = b.wy1; c.wz1 = b.wz1;
    c.cell = (b.N_l < 1024) ? ((uint32_t)b.x0 | ((uint32_t)b.y0 << 10) | ((uint32_t)b.z0 << 20)) : 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 8; k++) c.idx[k] = level_index((k & 1) ? b.x1 : b.x0, (k & 2) ? b.y1 : b.y0, (k & 4) ? b.z1 : b.z0, b.N_l, dense, T);
}

// True when all 8 corners of the point lie inside the staged box of the level; loc[k] = their places in the staging array.
__device__ __forceinline__ bool staged_corners(const StagePlan& pl, int level, const CornerBox& b, int (&loc)[8]) {
    const int lx0 = b.x0 - pl.ox[level], ly0 = b.y0 - pl.oy[level], lz0 = b.z0 - pl.oz[level];
    const int lx1 = b.x1 - pl.ox[level], ly1 = b.y1 - pl.oy[level], lz1 = b.z1 - pl.oz[level];
    const int w = pl.w[level], wh = pl.wh[level], h = pl.h[level], d = pl.d[level];
    if (lx0 < 0 || ly0 < 0 || lz0 < 0 || lx1 >= w || ly1 >= h || lz1 >= d) return false;
#pragma unroll
    for (int k = 0; k < 8; k++) loc[k] = pl.base[level] + ((k & 1) ? lx1 : lx0) + ((k & 2) ? ly1 : ly0) * w + ((k & 4) ? lz1 : lz0) * wh;
    return true;
}

// Block-wide: bounding box of the positions of rows [row_first, row_first + rows) (through perm when given), then the
// staging plan of levels 0, 1, ... while their boxes fit `capacity` entries.  s_box: 6 floats of shared memory.
// All THREADS threads of the group must call (tid = 0 .. THREADS - 1, whole warps); `barrier()` synchronises exactly
// them; ends with a barrier.  BWD_CLAMP selects the backward's clamp and resolutions.
template <bool BWD_CLAMP, int THREADS, class Barrier>
__device__ __forceinline__ void plan_stage(const GridParams& gp, const float* __restrict__ pos4, const uint32_t* __restrict__ perm,
                                           int64_t row_first, int rows, int64_t n, int capacity, int max_levels, float* s_box, StagePlan& pl,
                                           int tid, Barrier&& barrier) {
    float lo[3] = {INFINITY, INFINITY, INFINITY}, hi[3] = {-INFINITY, -INFINITY, -INFINITY};
    for (int r = tid; r < rows; r += THREADS) {
        const int64_t row = row_first + r;
        if (row < n) {
            const int64_t s = perm ? (int64_t)perm[row] : row;
            const float4 p = ld_nc_f4(pos4 + s * 4);
            lo[0] = fminf(lo[0], p.x); lo[1] = fminf(lo[1], p.y); lo[2] = fminf(lo[2], p.z);
            hi[0] = fmaxf(hi[0], p.x); hi[1] = fmaxf(hi[1], p.y); hi[2] = fmaxf(hi[2], p.z);
        }
    }
#pragma unroll
    for (int a = 0; a < 3; a++)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo[a] = fminf(lo[a], __shfl_xor_sync(0xffffffffu, lo[a], o));
            hi[a] = fmaxf(hi[a], __shfl_xor_sync(0xffffffffu, hi[a], o));
        }
    if (tid < 6) s_box[tid] = tid < 3 ? INFINITY : -INFINITY;
    barrier();
    if ((tid & 31) == 0) {
        // float min / max through the integer atomics: order-preserving for non-negative values, and a box that comes out
        // too large (negative or non-finite coordinates) only means fewer levels are staged
#pragma unroll
        for (int a = 0; a < 3; a++) {
            atomicMin(reinterpret_cast<int*>(&s_box[a]), __float_as_int(fmaxf(lo[a], 0.0f)));
            atomicMax(reinterpret_cast<int*>(&s_box[3 + a]), __float_as_int(fmaxf(hi[a], 0.0f)));
        }
    }
    barrier();
    if (tid < gp.L && tid < max_levels) {
        const int l = tid;
        const float scale = BWD_CLAMP ? gp.sscales[l] : gp.scales[l];
        CornerBox a, b;
        corner_box<BWD_CLAMP>(s_box[0], s_box[1], s_box[2], scale, a);
        corner_box<BWD_CLAMP>(s_box[3], s_box[4], s_box[5], scale, b);
        pl.ox[l] = a.x0; pl.oy[l] = a.y0; pl.oz[l] = a.z0;
        const int w = b.x1 - a.x0 + 1, h = b.y1 - a.y0 + 1, d = b.z1 - a.z0 + 1;
        const bool sane = w > 0 && h > 0 && d > 0 && w <= 1024 && h <= 1024 && d <= 1024;
        pl.w[l] = sane ? w : 1; pl.wh[l] = sane ? w * h : 1; pl.h[l] = sane ? h : 1; pl.d[l] = sane ? d : 1;
        pl.whd[l] = (sane && (int64_t)w * h * d <= capacity) ? w * h * d : capacity + 1;
    }
    barrier();
    if (tid == 0) {
        int used = 0, count = 0;
        const int top = min(gp.L, max_levels);
        while (count < top && used + pl.whd[count] <= capacity) { pl.base[count] = used; used += pl.whd[count]; count++; }
        pl.count = count;
    }
    barrier();
}

// Host side of the stand-alone scatter (hashgrid.cu): levels [level_begin, level_end) from a gradient matrix whose
// rows are denc_stride halves apart.  scatter_shared_levels = how many leading levels of a launch over n samples go
// through the shared-memory accumulation kernel.
int scatter_shared_levels(const GridParams& gp, int64_t n);
int scatter_launch(const GridParams& gp, const float* d_pos4, const __half* d_denc, int denc_stride, int64_t n, float* d_table_grads,
                   int level_begin, int level_end, cudaStream_t st);
// The same for the owner of some levels of a level-partitioned grid (level_partition.cu): `view` = level_view of the
// grid, samples of all ranks from the gathered position slots, gradients from the received pieces.
int scatter_launch_pieces(const GridParams& view, const float* d_pos_all, const uint32_t* d_pieces, int ranks, int own, int64_t cap,
                          float* d_table_grads_view, cudaStream_t st);

// Coalesced write of the encoded tile (128 x 2L halves) to global memory.
template <int TILE_STRIDE>
__device__ __forceinline__ void store_enc_tile(const __half* tile, __half* __restrict__ enc_out, int L, int64_t row_base, int64_t n,
                                               int tid) {
    const int cpr = (2 * L) / 8;
    for (int c = tid; c < TILE_ROWS * cpr; c += CTA_THREADS) {
        int r = c / cpr, c8 = c % cpr;
        if (row_base + r < n) {
            uint4 v = *reinterpret_cast<const uint4*>(&tile[r * TILE_STRIDE + c8 * 8]);
            st_cs_v4(&enc_out[(row_base + r) * (2 * L) + c8 * 8], v);
        }
    }
}

}  // namespace nb
