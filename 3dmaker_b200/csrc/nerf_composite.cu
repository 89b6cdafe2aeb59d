// Front-to-back volume compositing (inference and training variants), the distortion loss terms and the
// per-sample loss gradients.
//
// Replaces render_rays_kernel and render_rays_distortion_kernel (modules/NeRF/compositing.cu:5-213, launcher
// launchVolumeRendering :215-279) and compute_color_grad (modules/NeRF/otherKernels.cu:303-409).
//
// The reference gives every ray to one thread that walks the ray's samples in a loop: neighbouring lanes read
// addresses a whole ray apart and the loop is a chain of dependent loads, exponentials and multiplies.  Here a WARP
// owns a ray and lane k owns sample k of the current 32-sample window, so loads are contiguous and everything that
// the reference carries from sample to sample - transmittance, accumulated colour, the distortion loss's prefix
// sums, the suffix terms of the gradients - becomes a warp scan with a carry between windows:
//     T_i      = prod_{j<i} (1 - alpha_j)                       exclusive product scan
//     W_<i     = sum_{j<i} w_j ,  WM_<i = sum_{j<i} w_j m_j      exclusive sum scans (distortion loss)
//     C_<=i    = sum_{j<=i} w_j c_j , G_<=i = sum_{j<=i} w_j g_j   inclusive sum scans (gradient suffix terms)
// The formulas are the reference's; sums are associated differently, so results agree to fp32 rounding, not bitwise.
// Colour buffers carry a row stride so the colour network's padded output and gradient are used in place (the
// reference un-pads to [n][3] and pads back with two extra kernels, TinyMLP.cu:276-284,361-367).
#include <atomic>

#include "common.cuh"

namespace nb {

extern std::atomic<uint64_t> g_launch_count;

constexpr unsigned FULL = 0xffffffffu;

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(FULL, v, o);
    return v;
}
__device__ __forceinline__ float warp_incl_sum(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float n = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v += n;
    }
    return v;
}
__device__ __forceinline__ float warp_incl_prod(float v, int lane) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        float n = __shfl_up_sync(FULL, v, o);
        if (lane >= o) v *= n;
    }
    return v;
}
// value of the lane below (identity for lane 0): turns an inclusive scan into an exclusive one
__device__ __forceinline__ float from_lane_below(float incl, int lane, float identity) {
    float n = __shfl_up_sync(FULL, incl, 1);
    return lane == 0 ? identity : n;
}

// Sample i of a ray with `count` samples starting at `first`: distance, distance of the next sample, interval clamped
// at zero.  The last sample has no successor and gets a 1e-3 interval: as the literal where NOMINAL_LAST (the
// inference and gradient kernels of the reference), as (t + 1e-3) - t otherwise (its training kernel) - the two differ
// in the last bits and each kernel keeps its own form.
struct Interval {
    float t, t_next, dt;
};
template <bool NOMINAL_LAST>
__device__ __forceinline__ Interval load_interval(const float* __restrict__ t_sorted, uint32_t first, uint32_t i, uint32_t count) {
    Interval v;
    v.t = t_sorted[first + i];
    v.t_next = (i + 1 < count) ? t_sorted[first + i + 1] : v.t + 1e-3f;
    v.dt = (NOMINAL_LAST && i + 1 >= count) ? 1e-3f : v.t_next - v.t;
    if (v.dt < 0.0f) { v.dt = 0.0f; v.t_next = v.t; }
    return v;
}

// ---------------------------------------------------------------------------------------------------------
// inference: colour and depth of a ray, stopping once the transmittance has dropped below 1e-4
// ---------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) composite_infer_kernel(const uint32_t num_rays, const uint32_t sample_base,
                                                              const uint32_t* __restrict__ ray_offsets, const uint32_t* __restrict__ num_steps,
                                                              const float* __restrict__ t_sorted, const float* __restrict__ sigma_in,
                                                              const float* __restrict__ rgb_in, const int rgb_stride,
                                                              const float* __restrict__ rgb_true, float* __restrict__ final_rgb,
                                                              float* __restrict__ final_depth, float* __restrict__ phi_out, float3 bg) {
    after_previous();
    const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= num_rays) return;
    const uint32_t first = ray_offsets[r] - sample_base;
    const uint32_t count = num_steps[r];
    float T = 1.0f;  // transmittance in front of the current window
    float cr = 0.f, cg = 0.f, cb = 0.f, depth = 0.f;
    for (uint32_t w0 = 0; w0 < count; w0 += 32) {
        const uint32_t i = w0 + lane;
        const bool valid = i < count;
        float alpha = 0.f, t = 0.f;
        if (valid) {
            Interval iv = load_interval<true>(t_sorted, first, i, count);
            t = iv.t;
            alpha = 1.0f - expf(-sigma_in[first + i] * iv.dt);
        }
        const float incl = warp_incl_prod(1.0f - alpha, lane);
        const float T_before = T * from_lane_below(incl, lane, 1.0f);
        // the reference leaves its loop after the first sample that takes T below 1e-4: sample i counts exactly when
        // the transmittance in front of it is still at least 1e-4
        const bool live = valid && T_before >= 1e-4f;
        if (live) {
            const float w = alpha * T_before;
            const float* c = rgb_in + (size_t)(first + i) * rgb_stride;
            cr += w * c[0]; cg += w * c[1]; cb += w * c[2];
            depth += w * t;
        }
        const unsigned live_mask = __ballot_sync(FULL, live);
        const int last = 31 - __clz((int)live_mask);            // live_mask != 0: lane 0 of a window is live or the loop ended
        const float T_after_last = __shfl_sync(FULL, T * incl, last);
        T = T_after_last;
        if (live_mask != __ballot_sync(FULL, valid) || T < 1e-4f) break;
    }
    cr = warp_sum(cr); cg = warp_sum(cg); cb = warp_sum(cb); depth = warp_sum(depth);
    if (lane == 0) {
        cr += T * bg.x; cg += T * bg.y; cb += T * bg.z;
        final_rgb[r * 3 + 0] = cr; final_rgb[r * 3 + 1] = cg; final_rgb[r * 3 + 2] = cb;
        if (final_depth != nullptr) final_depth[r] = depth;
        if (rgb_true != nullptr && phi_out != nullptr) {
            phi_out[r * 3 + 0] = 2.0f * (cr - rgb_true[r * 3 + 0]);
            phi_out[r * 3 + 1] = 2.0f * (cg - rgb_true[r * 3 + 1]);
            phi_out[r * 3 + 2] = 2.0f * (cb - rgb_true[r * 3 + 2]);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// inference in rounds: the same front-to-back sum, cut into rounds of samples so that rays whose transmittance has
// dropped below 1e-4 are not evaluated any further (the samples the reference's loop never reaches contribute
// nothing to it either).  State per ray between rounds: transmittance and (r, g, b, depth) composited so far.
// ---------------------------------------------------------------------------------------------------------
// When next_width > 0 the kernel also copies out the NEXT round (samples [round_begin + round_width, ... + next_width)) of
// the rays that are still visible after this one: a block's rays take one range of the next round's counter, and its threads copy their
// samples as round_emit_kernel does in a launch of its own.
// Bound by latency: a ray is a chain of loads, exponentials, scans and sums.  A block looks at ROUND_RAYS rays, lists those that this round
// was planned with and lets LANES lanes take one after the other of them: 16 in rounds of 16 samples, where a warp per ray left half
// of its lanes idle.  65536 rays, with the copy-out (us): first round 42 -> 20,
// second 34 -> 20, one of 32 samples 21 -> 18, one without rays 10 -> 4.  Two windows of 16 lanes in rounds of 32 would associate the products
// differently.
constexpr uint32_t ROUND_RAYS = 32, ROUND_THREADS = 256;

template <int LANES>
__global__ void __launch_bounds__(ROUND_THREADS) composite_round_kernel(
    const uint32_t ray_begin, const uint32_t ray_count, const uint32_t* __restrict__ num_steps, uint32_t* __restrict__ round_off,
    const float* __restrict__ rows, const uint32_t row_stride, const uint32_t round_begin, const uint32_t round_width, const float* __restrict__ sigma_in,
    const float* __restrict__ rgb_in, const int rgb_stride, float* __restrict__ transmittance, float4* __restrict__ composited,
    float* __restrict__ final_rgb, float* __restrict__ final_depth, float3 bg, const uint32_t next_width, const float3 aabb_min, const float3 aabb_max,
    const float3* __restrict__ rays_o, const float3* __restrict__ rays_d, const uint32_t capacity, uint32_t* __restrict__ next_counter,
    unsigned long long* __restrict__ emitted_total, uint32_t* __restrict__ ray_idx_out, float4* __restrict__ pos_out, uint32_t* __restrict__ order) {
    after_previous();
    static_assert(ROUND_RAYS == 32, "a lane of the first warp per ray");
    __shared__ uint32_t s_n[ROUND_RAYS], s_first[ROUND_RAYS], s_next[ROUND_RAYS], s_off[ROUND_RAYS + 1], s_base;
    __shared__ float s_T[ROUND_RAYS];
    __shared__ uint8_t s_list[ROUND_RAYS];
    __shared__ bool s_close[ROUND_RAYS / 8];
    __shared__ int s_active;
    const uint32_t first_ray = ray_begin + blockIdx.x * ROUND_RAYS;
    if (threadIdx.x < ROUND_RAYS) {
        const uint32_t local = blockIdx.x * ROUND_RAYS + threadIdx.x, r = ray_begin + local;
        uint32_t n = 0u, first = 0u;
        float T = 0.0f;
        if (local < ray_count) {
            n = num_steps[r];
            T = round_begin == 0 ? 1.0f : transmittance[r];
            first = round_off[r];
        }
        const bool active = T >= 1e-4f && n > round_begin;  // the predicate this round was planned with
        if (local < ray_count && !active && round_begin == 0) {
            final_rgb[r * 3 + 0] = bg.x; final_rgb[r * 3 + 1] = bg.y; final_rgb[r * 3 + 2] = bg.z;
            if (final_depth != nullptr) final_depth[r] = 0.0f;
        }
        s_n[threadIdx.x] = n; s_first[threadIdx.x] = first; s_T[threadIdx.x] = T; s_next[threadIdx.x] = 0u;
        const unsigned all = __ballot_sync(FULL, active);
        if (active) s_list[__popc(all & ((1u << threadIdx.x) - 1u))] = (uint8_t)threadIdx.x;
        if (threadIdx.x == 0) s_active = __popc(all);
    }
    __syncthreads();
    const int active = s_active;
    if (active == 0) return;
    const int lane = threadIdx.x % LANES;
    const unsigned group = LANES == 32 ? FULL : ((1u << (LANES & 31)) - 1u) << (threadIdx.x & 31 & ~(LANES - 1));   // lanes of this ray's group
    auto sum = [&](float v) {
#pragma unroll
        for (int o = LANES / 2; o > 0; o >>= 1) v += __shfl_xor_sync(group, v, o);
        return v;
    };
    const uint32_t next_begin = round_begin + round_width;
    for (int k = threadIdx.x / LANES; k < active; k += ROUND_THREADS / LANES) {
        const uint32_t j = s_list[k], r = first_ray + j, n = s_n[j], first = s_first[j];
        const float* row = rows + (size_t)r * row_stride;
        float T = s_T[j];
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        if (round_begin > 0) acc = composited[r];
        const uint32_t count = min(n - round_begin, round_width);
        float cr = 0.f, cg = 0.f, cb = 0.f, depth = 0.f;
        for (uint32_t w0 = 0; w0 < count; w0 += LANES) {
            const uint32_t i = w0 + lane;
            const bool valid = i < count;
            float alpha = 0.f, t = 0.f, c[3] = {0.f, 0.f, 0.f};
            if (valid) {
                const uint32_t at = round_begin + i;  // index of the sample in its ray
                t = row[at];
                float dt = (at + 1 < n) ? row[at + 1] - t : 1e-3f;
                if (dt < 0.0f) dt = 0.0f;
                const float* rgb = rgb_in + (size_t)(first + i) * rgb_stride;
                c[0] = rgb[0]; c[1] = rgb[1]; c[2] = rgb[2];
                alpha = 1.0f - expf(-sigma_in[first + i] * dt);
            }
            float incl = 1.0f - alpha;
#pragma unroll
            for (int o = 1; o < LANES; o <<= 1) {
                const float below = __shfl_up_sync(group, incl, o, LANES);
                if (lane >= o) incl *= below;
            }
            const float before = __shfl_up_sync(group, incl, 1, LANES);
            const float T_before = T * (lane == 0 ? 1.0f : before);
            const bool live = valid && T_before >= 1e-4f;
            if (live) {
                const float w = alpha * T_before;
                cr += w * c[0]; cg += w * c[1]; cb += w * c[2];
                depth += w * t;
            }
            const unsigned live_mask = __ballot_sync(group, live);
            const int last = 31 - __clz((int)live_mask);
            T = __shfl_sync(group, T * incl, last & (LANES - 1), LANES);
            if (live_mask != __ballot_sync(group, valid) || T < 1e-4f) break;
        }
        cr = sum(cr); cg = sum(cg); cb = sum(cb); depth = sum(depth);
        if (lane == 0) {
            acc.x += cr; acc.y += cg; acc.z += cb; acc.w += depth;
            composited[r] = acc;
            transmittance[r] = T;
            final_rgb[r * 3 + 0] = acc.x + T * bg.x; final_rgb[r * 3 + 1] = acc.y + T * bg.y; final_rgb[r * 3 + 2] = acc.z + T * bg.z;
            if (final_depth != nullptr) final_depth[r] = acc.w;
            if (T >= 1e-4f && n > next_begin) s_next[j] = min(n - next_begin, next_width);
        }
    }
    if (next_width == 0) return;  // the same for the whole grid
    __syncthreads();
    if (threadIdx.x < ROUND_RAYS) {
        const uint32_t i = min(first_ray + threadIdx.x, ray_begin + ray_count - 1), c = s_next[threadIdx.x];
        uint32_t upto = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t below = __shfl_up_sync(FULL, upto, o);
            if ((int)threadIdx.x >= o) upto += below;
        }
        s_off[threadIdx.x] = upto - c;
        uint32_t base = 0u;
        if (threadIdx.x == 31) {
            s_off[ROUND_RAYS] = upto;
            s_base = base = upto ? atomicAdd(next_counter, upto) : 0u;
            if (upto && emitted_total != nullptr) atomicAdd(emitted_total, (unsigned long long)upto);
        }
        base = __shfl_sync(FULL, base, 31);
        if (c > 0) round_off[first_ray + threadIdx.x] = base + upto - c;
        if (order != nullptr) {
            const bool close = rays_close<8>(rays_o[i], rays_d[i], aabb_min, aabb_max, threadIdx.x);
            if ((threadIdx.x & 7) == 0) s_close[threadIdx.x >> 3] = close;
        }
    }
    __syncthreads();
    const uint32_t total = s_off[ROUND_RAYS], base = s_base;
    if (base + total > capacity) return;  // cannot happen when the caller's bound holds; never write past the arrays
    copy_round_out<ROUND_RAYS, ROUND_THREADS, 1>(s_off, s_close, base, total, first_ray, next_begin, rays_o, rays_d, aabb_min, aabb_max, rows, row_stride, ray_idx_out,
                                              pos_out, order);
}

// ---------------------------------------------------------------------------------------------------------
// training: colour, depth, dL/dw of the distortion (and depth-prior) loss per sample, sum_i w_i dL/dw_i per ray; the gradients of
// colour and loss behind them
// ---------------------------------------------------------------------------------------------------------

// Sums of eight values over the warp's lanes in 9 exchanges instead of 40, by the tree of warp_sum: lane 16 a + 8 b + 4 c + d ends with
// the sum of value 4 a + 2 b + c.
__device__ __forceinline__ float warp_sums8(const float (&v)[8], int lane) {
    float a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = ((lane & 16) ? v[4 + i] : v[i]) + __shfl_xor_sync(FULL, (lane & 16) ? v[i] : v[4 + i], 16);
#pragma unroll
    for (int i = 0; i < 2; i++) b[i] = ((lane & 8) ? a[2 + i] : a[i]) + __shfl_xor_sync(FULL, (lane & 8) ? a[i] : a[2 + i], 8);
    float s = ((lane & 4) ? b[1] : b[0]) + __shfl_xor_sync(FULL, (lane & 4) ? b[0] : b[1], 4);
    s += __shfl_xor_sync(FULL, s, 2);
    s += __shfl_xor_sync(FULL, s, 1);
    return s;
}
__device__ __forceinline__ float from_sums8(float s, int k) { return __shfl_sync(FULL, s, ((k >> 2) & 1) * 16 + ((k >> 1) & 1) * 8 + (k & 1) * 4); }

// What a ray's colour and weight loss hand to its samples' gradients.
struct RayLoss {
    float phi_r, phi_g, phi_b, fin_r, fin_g, fin_b, wg_total, scale;
};
// Everything of a ray up to the current window.
struct LossCarry {
    float T = 1.0f, r = 0.f, g = 0.f, b = 0.f, wg = 0.f;
};

// One window of the gradient pass; dt of the last sample is the nominal one, logit the raw density output, g = dL/dw of the sample.
template <bool GRAD8>
__device__ __forceinline__ void loss_window(const RayLoss& ray, LossCarry& at, bool valid, size_t sample, float dt, float logit, float c_r, float c_g,
                                            float c_b, float g, float density_bias, __half* __restrict__ color_grad, float* __restrict__ dsigma_out, int lane) {
    float alpha = 0.f, sigma = 0.f;
    if (valid) {
        sigma = expf(fminf(logit - density_bias, 8.0f));
        alpha = 1.0f - expf(-sigma * dt);
    }
    const float incl = warp_incl_prod(1.0f - alpha, lane);
    const float T_before = at.T * from_lane_below(incl, lane, 1.0f);
    const float w = T_before * alpha;
    // colour composited up to and including this sample, and the same for w g
    const float cum_r = at.r + warp_incl_sum(w * c_r, lane), cum_g = at.g + warp_incl_sum(w * c_g, lane);
    const float cum_b = at.b + warp_incl_sum(w * c_b, lane), cum_wg = at.wg + warp_incl_sum(w * g, lane);
    if (valid) {
        const float scale = ray.scale;
        float gr = ray.phi_r * w * c_r * (1.0f - c_r) * scale, gg = ray.phi_g * w * c_g * (1.0f - c_g) * scale, gb = ray.phi_b * w * c_b * (1.0f - c_b) * scale;
        gr = fmaxf(-65504.0f, fminf(65504.0f, gr)); gg = fmaxf(-65504.0f, fminf(65504.0f, gg)); gb = fmaxf(-65504.0f, fminf(65504.0f, gb));
        if (gr != gr || gg != gg || gb != gb) { gr = 0.0f; gg = 0.0f; gb = 0.0f; }
        if (GRAD8) {
            *reinterpret_cast<uint4*>(color_grad + sample * 8) = make_uint4(pack_half2(gr, gg), pack_half2(gb, 0.0f), 0u, 0u);
        } else {
            __half* o = color_grad + sample * 3;
            o[0] = __float2half(gr); o[1] = __float2half(gg); o[2] = __float2half(gb);
        }
        // d/d sigma_i of the colour loss: this sample's own term minus everything composited behind it
        const float keep = T_before * (1.0f - alpha);
        const float ds_r = keep * c_r - (ray.fin_r - cum_r), ds_g = keep * c_g - (ray.fin_g - cum_g), ds_b = keep * c_b - (ray.fin_b - cum_b);
        float d = dt * (ds_r * ray.phi_r + ds_g * ray.phi_g + ds_b * ray.phi_b);
        // ... and of the distortion / depth loss through the weights
        d += dt * (g * keep - (ray.wg_total - cum_wg));
        d = d * sigma * scale;
        d = fmaxf(-65504.0f, fminf(65504.0f, d));
        if (d != d) d = 0.0f;
        dsigma_out[sample] = d;
    }
    at.T *= __shfl_sync(FULL, incl, 31);
    at.r = __shfl_sync(FULL, cum_r, 31); at.g = __shfl_sync(FULL, cum_g, 31);
    at.b = __shfl_sync(FULL, cum_b, 31); at.wg = __shfl_sync(FULL, cum_wg, 31);
}

// Outputs of the gradient pass when it follows in the same kernel; rgb_copy (nullable): a second place for the rays' colours.
struct LossOut {
    const float* logit0;
    int logit_stride;
    __half* color_grad;   // rows of 8
    float* dsigma;
    float loss_scale, density_bias;
    uint32_t total_rays;
    float* rgb_copy;
};

__device__ __forceinline__ float disparity_warp(float t, float t_near, float inv_g_range) {
    return (1.0f - t_near / fmaxf(t, 1e-4f)) * inv_g_range;
}

// GRAD: the gradient pass follows at once, on values still in registers for rays of one window; 2^18 samples of 9400 rays 11.6 + 7.9 us in
// two launches, a training call of seven steps 1998 -> 1963 us.  Bound by the latency of a warp's scans and exponentials.
// Blocks of four warps: rays differ in length, and a block's place is free only when its longest ray is done.  2^18 samples of 10600 rays
// 19.7 us with eight warps a block, 17.5 with four, 17.7 with two, 21.4 with one (32 blocks an SM); 2^21 samples 63 -> 58.  At 42
// registers instead of 48 it is 19.6, and with 16 lanes a ray and two samples a lane 23: a warp then waits for the longer of two rays.
// Loads are not what the long rays wait for: their later windows fetched into L1 at the start give 17.4 to 17.5.
constexpr int TRAIN_THREADS = 128, TRAIN_BLOCKS = 10;
template <bool GRAD>
__global__ void __launch_bounds__(TRAIN_THREADS, TRAIN_BLOCKS) composite_train_kernel(
    const uint32_t num_rays, const uint32_t sample_base, const uint32_t* __restrict__ ray_offsets, const uint32_t* __restrict__ num_steps,
    const float* __restrict__ t_sorted, const float* __restrict__ sigma_in, const float* __restrict__ depth_prior,
    const float* __restrict__ sigma_prior_in, const float* __restrict__ rgb_in, const int rgb_stride, const float* __restrict__ rgb_true,
    float* __restrict__ final_rgb, float* __restrict__ final_depth, float* __restrict__ phi_out, float* __restrict__ dw_out,
    float* __restrict__ weight_sum, float lambda_dist, float lambda_depth, float3 bg, const LossOut loss) {
    after_previous();
    const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= num_rays) return;
    const uint32_t first = ray_offsets[r] - sample_base;
    const uint32_t count = num_steps[r];
    const float d_prior = depth_prior ? depth_prior[r] : -1.0f;
    const float s_prior = sigma_prior_in ? sigma_prior_in[r] : -1.0f;
    const float depth_lambda = (d_prior >= 0) ? lambda_depth : 0.0f;
    // normalised disparity s(t) = (1 - t_near / t) / g_far over the ray's own sample range
    const float t_near = (count > 0) ? fmaxf(t_sorted[first], 1e-4f) : 1.0f;
    const float t_far = (count > 0) ? t_sorted[first + count - 1] : 1.0f;
    const float g_far = 1.0f - t_near / fmaxf(t_far, t_near + 1e-4f);
    const float inv_g = (g_far > 1e-6f) ? (1.0f / g_far) : 0.0f;

    // A window's samples: a ray of at most 32 loads them once for all passes.
    const bool one_window = count <= 32;
    float t = 0.f, t_next = 0.f, dt = 0.f, sigma = 0.f, c_r = 0.f, c_g = 0.f, c_b = 0.f, logit = 0.f;
    auto load = [&](uint32_t i, bool colour) {
        const Interval iv = load_interval<false>(t_sorted, first, i, count);
        t = iv.t; t_next = iv.t_next; dt = iv.dt;
        if (colour) {
            const float* c = rgb_in + (size_t)(first + i) * rgb_stride;
            c_r = c[0]; c_g = c[1]; c_b = c[2];
            if (GRAD) logit = loss.logit0[(size_t)(first + i) * loss.logit_stride];
        }
    };

    // pass 1: weights (staged in dw_out), colour, depth, W = sum w, WM = sum w m, depth-prior normaliser
    float T = 1.0f;
    float sums[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // colour, depth, W, WM, DN
    float w_keep = 0.f;  // this lane's weight when the ray fits one window (the common case): pass 2 skips the re-read
    for (uint32_t w0 = 0; w0 < count; w0 += 32) {
        const uint32_t i = w0 + lane;
        const bool valid = i < count;
        float alpha = 0.f, m = 0.f, dterm = 0.f;
        if (valid) {
            load(i, true);
            sigma = sigma_in[first + i];
            m = 0.5f * (disparity_warp(t, t_near, inv_g) + disparity_warp(t_next, t_near, inv_g));
            alpha = 1.0f - expf(-sigma * dt);
            const float tx = (t - d_prior) / s_prior;
            dterm = expf(-0.5f * tx * tx) * dt;
        }
        const float incl = warp_incl_prod(1.0f - alpha, lane);
        const float w = alpha * (T * from_lane_below(incl, lane, 1.0f));
        if (valid) {
            sums[0] += w * c_r; sums[1] += w * c_g; sums[2] += w * c_b;
            sums[3] += w * t; sums[4] += w; sums[5] += w * m; sums[6] += dterm;
            if (!one_window) dw_out[first + i] = w;
        }
        w_keep = w;
        T *= __shfl_sync(FULL, incl, 31);
    }
    const float summed = warp_sums8(sums, lane);
    float cr = from_sums8(summed, 0), cg = from_sums8(summed, 1), cb = from_sums8(summed, 2);
    const float depth = from_sums8(summed, 3), W = from_sums8(summed, 4), WM = from_sums8(summed, 5), DN = from_sums8(summed, 6);
    const float depth_norm = 1.0f / fmaxf(DN, 1e-8f);

    // pass 2: dL/dw_i = lambda (2 (m_i (2 W_<i - W) + (WM - 2 WM_<i)) + (2/3) w_i ds_i) + depth term
    float W_lt = 0.f, WM_lt = 0.f, wg = 0.f, g_keep = 0.f;
    const float two_thirds = 2.0f / 3;
    for (uint32_t w0 = 0; w0 < count; w0 += 32) {
        const uint32_t i = w0 + lane;
        const bool valid = i < count;
        float w = 0.f, m = 0.f, ds = 0.f, dloss = 0.f;
        if (valid) {
            if (!one_window) load(i, false);
            const float s = disparity_warp(t, t_near, inv_g), s_next = disparity_warp(t_next, t_near, inv_g);
            m = 0.5f * (s + s_next);
            ds = fmaxf(s_next - s, 0.0f);
            w = one_window ? w_keep : dw_out[first + i];
            const float tx = (t - d_prior) / s_prior;
            dloss = -(expf(-0.5f * tx * tx) * dt * depth_norm) * (1.0f / fmaxf(w, 1e-6));
        }
        const float w_incl = warp_incl_sum(w, lane), wm_incl = warp_incl_sum(w * m, lane);
        const float w_before = W_lt + (w_incl - w), wm_before = WM_lt + (wm_incl - w * m);
        if (valid) {
            const float bilinear = m * (2 * w_before - W) + (WM - 2 * wm_before);
            g_keep = lambda_dist * (2 * bilinear + two_thirds * w * ds) + depth_lambda * dloss;
            dw_out[first + i] = g_keep;
            wg += w * g_keep;
        }
        W_lt += __shfl_sync(FULL, w_incl, 31);
        WM_lt += __shfl_sync(FULL, wm_incl, 31);
    }
    wg = warp_sum(wg);
    cr += T * bg.x; cg += T * bg.y; cb += T * bg.z;
    RayLoss ray{};
    if (rgb_true != nullptr) {
        ray.phi_r = 2.0f * (cr - rgb_true[r * 3 + 0]);
        ray.phi_g = 2.0f * (cg - rgb_true[r * 3 + 1]);
        ray.phi_b = 2.0f * (cb - rgb_true[r * 3 + 2]);
    }
    if (lane == 0) {
        weight_sum[r] = wg;
        final_rgb[r * 3 + 0] = cr; final_rgb[r * 3 + 1] = cg; final_rgb[r * 3 + 2] = cb;
        if (GRAD && loss.rgb_copy != nullptr) { loss.rgb_copy[r * 3 + 0] = cr; loss.rgb_copy[r * 3 + 1] = cg; loss.rgb_copy[r * 3 + 2] = cb; }
        if (final_depth != nullptr) final_depth[r] = depth;
        if (rgb_true != nullptr && phi_out != nullptr) { phi_out[r * 3 + 0] = ray.phi_r; phi_out[r * 3 + 1] = ray.phi_g; phi_out[r * 3 + 2] = ray.phi_b; }
    }
    if constexpr (GRAD) {
        ray.fin_r = cr; ray.fin_g = cg; ray.fin_b = cb; ray.wg_total = wg;
        ray.scale = loss.loss_scale * (1.0f / (float)loss.total_rays);
        LossCarry at;
        for (uint32_t w0 = 0; w0 < count; w0 += 32) {
            const uint32_t i = w0 + lane;
            const bool valid = i < count;
            if (valid && !one_window) {
                load(i, true);
                g_keep = dw_out[first + i];
            }
            if (!valid) { c_r = c_g = c_b = g_keep = 0.f; }
            loss_window<true>(ray, at, valid, first + i, i + 1 >= count ? 1e-3f : dt, logit, c_r, c_g, c_b, g_keep, loss.density_bias, loss.color_grad,
                              loss.dsigma, lane);
        }
    }
}

// ---------------------------------------------------------------------------------------------------------
// loss gradients per sample: dL/d(colour pre-activation) in fp16 and dL/d(logit 0) through sigma
// ---------------------------------------------------------------------------------------------------------
// GRAD8: the gradient row is 8 halves wide (16-byte store, channels 3..7 zero); otherwise 3 halves.
template <bool GRAD8>
__global__ void __launch_bounds__(256) loss_grad_kernel(const uint32_t num_rays, const uint32_t sample_base, const uint32_t* __restrict__ num_steps,
                                                        const uint32_t* __restrict__ ray_offsets, const float* __restrict__ t_sorted,
                                                        const float* __restrict__ logit0, const int logit_stride,
                                                        const float* __restrict__ rgb_in, const int rgb_stride, const float* __restrict__ phi_in,
                                                        const float* __restrict__ final_rgb, const float* __restrict__ dw_in,
                                                        const float* __restrict__ weight_sum, __half* __restrict__ color_grad,
                                                        float* __restrict__ dsigma_out, float loss_scale, const float density_bias,
                                                        const uint32_t total_rays) {
    after_previous();
    const uint32_t r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (r >= num_rays) return;
    const uint32_t first = ray_offsets[r] - sample_base;
    const uint32_t count = num_steps[r];
    const RayLoss ray{phi_in[r * 3], phi_in[r * 3 + 1], phi_in[r * 3 + 2], final_rgb[r * 3], final_rgb[r * 3 + 1], final_rgb[r * 3 + 2], weight_sum[r],
                      loss_scale * (1.0f / (float)total_rays)};
    LossCarry at;   // everything up to the current window
    for (uint32_t w0 = 0; w0 < count; w0 += 32) {
        const uint32_t i = w0 + lane;
        const bool valid = i < count;
        float dt = 0.f, logit = 0.f, c_r = 0.f, c_g = 0.f, c_b = 0.f, g = 0.f;
        if (valid) {
            dt = load_interval<true>(t_sorted, first, i, count).dt;
            logit = logit0[(size_t)(first + i) * logit_stride];
            const float* c = rgb_in + (size_t)(first + i) * rgb_stride;
            c_r = c[0]; c_g = c[1]; c_b = c[2];
            g = dw_in[first + i];
        }
        loss_window<GRAD8>(ray, at, valid, first + i, dt, logit, c_r, c_g, c_b, g, density_bias, color_grad, dsigma_out, lane);
    }
}

}  // namespace nb

using namespace nb;

static unsigned warp_grid(int64_t rays) { return (unsigned)((rays * 32 + 255) / 256); }
static unsigned train_grid(int64_t rays) { return (unsigned)((rays * 32 + TRAIN_THREADS - 1) / TRAIN_THREADS); }

extern "C" int nb_composite_infer(int64_t num_rays, uint32_t base, uint32_t rays_done, const uint32_t* d_ray_offsets,
                                  const uint32_t* d_num_steps, const float* d_t_sorted, const float* d_sigma, const float* d_rgb,
                                  int rgb_stride, const float* d_rgb_true, float* d_final_rgb, float* d_final_depth, float* d_phi,
                                  const float* bg_color3, void* stream) {
    if (!d_ray_offsets || !d_num_steps || !d_t_sorted || !d_sigma || !d_rgb || !d_final_rgb || !bg_color3 || num_rays < 0 ||
        num_rays > 0x3ffffff || rgb_stride < 3)
        return nb_set_error(NB_ERR_INVALID, "nb_composite_infer: null pointer, bad ray count or rgb stride < 3");
    if (num_rays == 0) return NB_OK;
    // a plain launch: frames are composited on two streams, and blocks waiting on the chip would be in the other's way (1080p 22.3 ->
    // 22.6 ms)
    composite_infer_kernel<<<warp_grid(num_rays), 256, 0, (cudaStream_t)stream>>>((uint32_t)num_rays, base, d_ray_offsets + rays_done, d_num_steps, d_t_sorted, d_sigma, d_rgb, rgb_stride, d_rgb_true, d_final_rgb,
        d_final_depth, d_phi, make_float3(bg_color3[0], bg_color3[1], bg_color3[2]));
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_composite_train(int64_t num_rays, uint32_t sample_base, const uint32_t* d_ray_offsets, const uint32_t* d_num_steps,
                                  const float* d_t_sorted, const float* d_sigma, const float* d_depth_prior, const float* d_sigma_prior,
                                  const float* d_rgb, int rgb_stride, const float* d_rgb_true, float* d_final_rgb, float* d_final_depth,
                                  float* d_phi, float* d_dw_out, float* d_weight_sum, float lambda_dist, float lambda_depth,
                                  const float* bg_color3, void* stream) {
    if (!d_ray_offsets || !d_num_steps || !d_t_sorted || !d_sigma || !d_rgb || !d_final_rgb || !d_dw_out || !d_weight_sum || !bg_color3 ||
        num_rays < 0 || num_rays > 0x3ffffff || rgb_stride < 3)
        return nb_set_error(NB_ERR_INVALID, "nb_composite_train: null pointer, bad ray count or rgb stride < 3");
    if (num_rays == 0) return NB_OK;
    launch_after(composite_train_kernel<false>, train_grid(num_rays), TRAIN_THREADS, 0, (cudaStream_t)stream, 
        (uint32_t)num_rays, sample_base, d_ray_offsets, d_num_steps, d_t_sorted, d_sigma, d_depth_prior, d_sigma_prior, d_rgb, rgb_stride,
        d_rgb_true, d_final_rgb, d_final_depth, d_phi, d_dw_out, d_weight_sum, lambda_dist, lambda_depth,
        make_float3(bg_color3[0], bg_color3[1], bg_color3[2]), LossOut{});
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_composite_train_grad(int64_t num_rays, uint32_t sample_base, const uint32_t* d_ray_offsets, const uint32_t* d_num_steps,
                                       const float* d_t_sorted, const float* d_sigma, const float* d_depth_prior, const float* d_sigma_prior,
                                       const float* d_rgb, int rgb_stride, const float* d_rgb_true, float* d_final_rgb, float* d_rgb_copy,
                                       float* d_final_depth, float* d_phi, float* d_dw_out, float* d_weight_sum, float lambda_dist, float lambda_depth,
                                       const float* bg_color3, const float* d_logit0, int logit_stride, void* d_color_grad_h, float* d_tmp_dsigma,
                                       float loss_scale, float density_bias, uint32_t total_rays_batch, void* stream) {
    if (!d_ray_offsets || !d_num_steps || !d_t_sorted || !d_sigma || !d_rgb || !d_rgb_true || !d_final_rgb || !d_dw_out || !d_weight_sum || !bg_color3 ||
        !d_logit0 || logit_stride < 1 || !d_color_grad_h || !d_tmp_dsigma || num_rays < 0 || num_rays > 0x3ffffff || rgb_stride < 3 || total_rays_batch == 0)
        return nb_set_error(NB_ERR_INVALID, "nb_composite_train_grad: null pointer, bad ray count or stride");
    if (reinterpret_cast<uintptr_t>(d_color_grad_h) & 15u)
        return nb_set_error(NB_ERR_INVALID, "nb_composite_train_grad: gradient rows must be 16-byte aligned");
    if (num_rays == 0) return NB_OK;
    const LossOut loss{d_logit0, logit_stride, (__half*)d_color_grad_h, d_tmp_dsigma, loss_scale, density_bias, total_rays_batch, d_rgb_copy};
    launch_after(composite_train_kernel<true>, train_grid(num_rays), TRAIN_THREADS, 0, (cudaStream_t)stream, (uint32_t)num_rays, sample_base, d_ray_offsets, d_num_steps,
                 d_t_sorted, d_sigma, d_depth_prior, d_sigma_prior, d_rgb, rgb_stride, d_rgb_true, d_final_rgb, d_final_depth, d_phi, d_dw_out, d_weight_sum,
                 lambda_dist, lambda_depth, make_float3(bg_color3[0], bg_color3[1], bg_color3[2]), loss);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_color_grad(int64_t num_rays, uint32_t sample_base, const uint32_t* d_num_steps, const uint32_t* d_ray_offsets,
                             const float* d_t_sorted, const float* d_logit0, int logit_stride, const float* d_color_out, int color_stride,
                             const float* d_phi, const float* d_final_rgb, const float* d_dw_out, const float* d_weight_sum,
                             void* d_color_grad_h, int grad_stride, float* d_tmp_dsigma, float loss_scale, float density_bias,
                             uint32_t total_rays_batch, void* stream) {
    if (!d_num_steps || !d_ray_offsets || !d_t_sorted || !d_logit0 || logit_stride < 1 || !d_color_out || !d_phi || !d_final_rgb || !d_dw_out ||
        !d_weight_sum || !d_color_grad_h || !d_tmp_dsigma || num_rays < 0 || num_rays > 0x3ffffff || color_stride < 3)
        return nb_set_error(NB_ERR_INVALID, "nb_color_grad: null pointer, bad ray count or colour stride < 3");
    if (grad_stride != 3 && grad_stride != 8) return nb_set_error(NB_ERR_UNSUPPORTED, "nb_color_grad: gradient row stride must be 3 or 8 halves");
    if (grad_stride == 8 && (reinterpret_cast<uintptr_t>(d_color_grad_h) & 15u))
        return nb_set_error(NB_ERR_INVALID, "nb_color_grad: 8-wide gradient rows must be 16-byte aligned");
    if (total_rays_batch == 0) return nb_set_error(NB_ERR_INVALID, "nb_color_grad: total_rays_batch must be positive");
    if (num_rays == 0) return NB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    if (grad_stride == 8)
        launch_after(loss_grad_kernel<true>, warp_grid(num_rays), 256, 0, st, (uint32_t)num_rays, sample_base, d_num_steps, d_ray_offsets, d_t_sorted, d_logit0,
                                                                    logit_stride, d_color_out, color_stride, d_phi, d_final_rgb, d_dw_out,
                                                                    d_weight_sum, (__half*)d_color_grad_h, d_tmp_dsigma, loss_scale, density_bias,
                                                                    total_rays_batch);
    else
        launch_after(loss_grad_kernel<false>, warp_grid(num_rays), 256, 0, st, (uint32_t)num_rays, sample_base, d_num_steps, d_ray_offsets, d_t_sorted, d_logit0,
                                                                     logit_stride, d_color_out, color_stride, d_phi, d_final_rgb, d_dw_out,
                                                                     d_weight_sum, (__half*)d_color_grad_h, d_tmp_dsigma, loss_scale, density_bias,
                                                                     total_rays_batch);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_composite_round_order(uint32_t ray_begin, uint32_t ray_count, const uint32_t* d_num_steps, uint32_t* d_round_offsets,
                                  const float* d_t_rows, uint32_t round_begin, uint32_t round_width, const float* d_sigma, const float* d_rgb,
                                  int rgb_stride, float* d_transmittance, float* d_composited4, float* d_final_rgb, float* d_final_depth,
                                  const float* bg_color3, uint32_t next_width, const nb_scene_desc* scene, const float* d_rays_o,
                                  const float* d_rays_d, uint32_t capacity, uint32_t* d_next_counter, uint64_t* d_emitted_total,
                                  uint32_t* d_ray_idx_out, float* d_pos4_out, uint32_t* d_order, void* stream) {
    if (!d_num_steps || !d_round_offsets || !d_t_rows || !d_sigma || !d_rgb || !d_transmittance || !d_composited4 || !d_final_rgb ||
        !bg_color3 || rgb_stride < 3 || round_width == 0)
        return nb_set_error(NB_ERR_INVALID, "nb_composite_round: null pointer, empty round or rgb stride < 3");
    if (reinterpret_cast<uintptr_t>(d_composited4) & 15u)
        return nb_set_error(NB_ERR_INVALID, "nb_composite_round: the composited state must be 16-byte aligned");
    if (ray_count > 0x3ffffffu) return nb_set_error(NB_ERR_INVALID, "nb_composite_round: too many rays");
    float3 lo = make_float3(0.f, 0.f, 0.f), hi = make_float3(1.f, 1.f, 1.f);
    if (next_width > 0) {
        if (!scene || !d_rays_o || !d_rays_d || !d_next_counter || !d_ray_idx_out || !d_pos4_out)
            return nb_set_error(NB_ERR_INVALID, "nb_composite_round: the next round's copy-out needs the scene, the rays, a counter and the sample arrays");
        if (reinterpret_cast<uintptr_t>(d_pos4_out) & 15u)
            return nb_set_error(NB_ERR_INVALID, "nb_composite_round: positions must be 16-byte aligned");
        if ((uint64_t)round_begin + round_width >= (uint64_t)nb_march_row_stride())
            return nb_set_error(NB_ERR_INVALID, "nb_composite_round: the next round must lie inside a row");
        lo = make_float3(scene->aabb_min[0], scene->aabb_min[1], scene->aabb_min[2]);
        hi = make_float3(scene->aabb_max[0], scene->aabb_max[1], scene->aabb_max[2]);
    }
    if (ray_count == 0) return NB_OK;
    launch_after(round_width <= 16 ? composite_round_kernel<16> : composite_round_kernel<32>, (ray_count + ROUND_RAYS - 1) / ROUND_RAYS, ROUND_THREADS, 0,
                 (cudaStream_t)stream, ray_begin, ray_count, d_num_steps, d_round_offsets, d_t_rows, (uint32_t)nb_march_row_stride(), round_begin, round_width,
                 d_sigma, d_rgb, rgb_stride, d_transmittance, (float4*)d_composited4, d_final_rgb, d_final_depth, make_float3(bg_color3[0], bg_color3[1], bg_color3[2]),
                 next_width, lo, hi, (const float3*)d_rays_o, (const float3*)d_rays_d, capacity, d_next_counter, (unsigned long long*)d_emitted_total,
                 d_ray_idx_out, (float4*)d_pos4_out, d_order);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

extern "C" int nb_composite_round(uint32_t ray_begin, uint32_t ray_count, const uint32_t* d_num_steps, uint32_t* d_round_offsets,
                                  const float* d_t_rows, uint32_t round_begin, uint32_t round_width, const float* d_sigma, const float* d_rgb,
                                  int rgb_stride, float* d_transmittance, float* d_composited4, float* d_final_rgb, float* d_final_depth,
                                  const float* bg_color3, uint32_t next_width, const nb_scene_desc* scene, const float* d_rays_o,
                                  const float* d_rays_d, uint32_t capacity, uint32_t* d_next_counter, uint64_t* d_emitted_total,
                                  uint32_t* d_ray_idx_out, float* d_pos4_out, void* stream) {
    return nb_composite_round_order(ray_begin, ray_count, d_num_steps, d_round_offsets, d_t_rows, round_begin, round_width, d_sigma, d_rgb, rgb_stride,
                                    d_transmittance, d_composited4, d_final_rgb, d_final_depth, bg_color3, next_width, scene, d_rays_o, d_rays_d, capacity,
                                    d_next_counter, d_emitted_total, d_ray_idx_out, d_pos4_out, nullptr, stream);
}
