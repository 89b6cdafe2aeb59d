// Shared device helpers for the sm_100a kernels: status codes, PTX wrappers (mma.sync, ldmatrix,
// cp.async, vector reductions) and fp16 packing.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <utility>
#include <stdint.h>

#include "../../include/nerf_b200.h"

#define NB_CHECK_LAUNCH()                                   \
    do {                                                    \
        cudaError_t e_ = cudaGetLastError();                \
        if (e_ != cudaSuccess) return nb_set_cuda_error(e_); \
    } while (0)

#define NB_CUDA(call)                                        \
    do {                                                     \
        cudaError_t e_ = (call);                             \
        if (e_ != cudaSuccess) return nb_set_cuda_error(e_); \
    } while (0)

int nb_set_cuda_error(cudaError_t e);
int nb_set_error(int code, const char* msg);
int nb_num_sms();

namespace nb {

__device__ __forceinline__ uint32_t pack_half2(float lo, float hi) {
    __half2 h = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&h);
}

__device__ __forceinline__ float2 unpack_half2(uint32_t v) {
    return __half22float2(*reinterpret_cast<__half2*>(&v));
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// D(16x8,f32) += A(16x16,f16,row) * B(16x8,f16,col)
__device__ __forceinline__ void mma_16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldmatrix_x4_trans(uint32_t (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldmatrix_x2(uint32_t& r0, uint32_t& r1, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];\n" : "=r"(r0), "=r"(r1) : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldmatrix_x2_trans(uint32_t& r0, uint32_t& r1, const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                 : "=r"(r0), "=r"(r1)
                 : "r"(smem_u32(p)));
}

// 16-byte asynchronous global->shared copy; src_bytes = 0 zero-fills the destination.
__device__ __forceinline__ void cp_async16(void* smem, const void* gmem, bool valid) {
    int src = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(smem)), "l"(gmem), "r"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Two-wide fp32 reduction to global memory (one L2 atomic for a feature pair).
__device__ __forceinline__ void red_add_v2(float* addr, float a, float b) {
    asm volatile("red.global.add.v2.f32 [%0], {%1, %2};\n" ::"l"(addr), "f"(a), "f"(b) : "memory");
}
// Four-wide: two adjacent feature pairs (16-byte aligned address).
__device__ __forceinline__ void red_add_v4(float* addr, float a, float b, float c, float d) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(addr), "f"(a), "f"(b), "f"(c), "f"(d) : "memory");
}
// fp16 pair reductions (the half-precision gradient table): one entry, or two entries in an aligned 8-byte slot pair.
__device__ __forceinline__ void red_add_h2(uint32_t* addr, uint32_t v) {
    asm volatile("red.global.add.noftz.f16x2 [%0], %1;\n" ::"l"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ void red_add_h2x2(uint32_t* addr, uint32_t lo, uint32_t hi) {
    asm volatile("red.global.add.noftz.v2.f16x2 [%0], {%1, %2};\n" ::"l"(addr), "r"(lo), "r"(hi) : "memory");
}
__device__ __forceinline__ void red_add(float* addr, float a) {
    asm volatile("red.global.add.f32 [%0], %1;\n" ::"l"(addr), "f"(a) : "memory");
}

__device__ __forceinline__ void st_cs_v4(void* addr, uint4 v) {
    asm volatile("st.global.cs.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"l"(addr), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
}

__device__ __forceinline__ float4 ld_nc_f4(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ uint4 ld_nc_v4(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// ---- launches that overlap the end of the kernel before them --------------------------------------------------------------
// A launch costs the device one to two microseconds between the last block of one kernel and the first of the next.  Kernels
// started with launch_after may be set up, and their blocks wait on the chip, while the kernel before them in the stream still
// runs; after_previous(), their first statement, waits until everything before them in the stream has finished and its writes are
// visible, then lets the kernel behind them come up.  In that order: a kernel must not be set up - which is when an SM drops its
// stale L1 lines - while one before its predecessor still fetches them.  No kernel may touch global memory before it.
// Kernels that live on L1 (gathers, streams) say so with launch_after_with_l1: blocks that come up early otherwise find the SM's division
// into L1 and shared memory as the kernel before had it, and behind one that takes nearly all of it as shared memory they run without
// L1 (forward of 2^21 samples at T = 2^22 0.56 -> 1.3 ms, optimizer 0.39 -> 0.43).
// Training calls of 2^16 rays 2096 -> 1998 us, with L1 named 1965 -> 1934; with default options 223 -> 209, 201 -> 197; frames in rounds
// 11.34 -> 11.21 ms, plain network steps 156 -> 152.5, grid network steps 162.5 -> 157.
__device__ __forceinline__ void after_previous() {
    asm volatile("griddepcontrol.wait;\n\tgriddepcontrol.launch_dependents;\n" ::: "memory");
}
template <class... P, class... A>
inline void launch_after_as(int smem_percent, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
    attr[1].val.sharedMemCarveout = smem_percent < 0 ? 0 : smem_percent;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid; cfg.blockDim = block; cfg.dynamicSmemBytes = smem; cfg.stream = stream;
    cfg.attrs = attr; cfg.numAttrs = smem_percent < 0 ? 1 : 2;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);   // an error is what NB_CHECK_LAUNCH finds
}
template <class... P, class... A>
inline void launch_after(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    launch_after_as(-1, kernel, grid, block, smem, stream, std::forward<A>(args)...);
}
// ... for kernels that live on L1 and whose blocks need `smem` bytes of shared memory an SM all together.
template <class... P, class... A>
inline void launch_after_with_l1(size_t smem_per_sm, void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t stream, A&&... args) {
    launch_after_as((int)((smem_per_sm * 100 + 228 * 1024 - 1) / (228 * 1024)), kernel, grid, block, smem, stream, std::forward<A>(args)...);
}

// ---- mbarriers with bounded waits ---------------------------------------------------------------------------------------
constexpr uint64_t WAIT_LIMIT_NS = 1000000000ull;   // one second: the longest any wait inside a kernel lasts

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
    return t;
}
__device__ __forceinline__ bool mbar_test(uint32_t bar_addr, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(ok) : "r"(bar_addr), "r"(parity) : "memory");
    return ok != 0;
}
// Waits for the phase with the given parity, for at most limit_ns nanoseconds of the global timer (false when the time
// ran out, or when *give_up - a flag another warp of the CTA raises - became non-zero).  limit_ns == 0 does not wait at
// all: one non-blocking test decides.  That setting exists for the test of the give-up path.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns, volatile int* give_up = nullptr) {
    const uint32_t a = smem_u32(bar);
    if (mbar_test(a, parity)) return true;
    if (limit_ns == 0) return false;
    // the timer is looked at once in 256 failed polls (a poll itself waits a while in hardware): the common case, a
    // barrier that completes within a few polls, never reads it
    uint64_t t0 = 0;
    for (uint32_t polls = 1;; polls++) {
        uint32_t ok;
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                     : "=r"(ok) : "r"(a), "r"(parity) : "memory");
        if (ok) return true;
        if (give_up != nullptr && *give_up != 0) return false;
        if ((polls & 255u) == 0u) {
            const uint64_t now = global_ns();
            if (t0 == 0) t0 = now;
            else if (now - t0 > limit_ns) return false;
        }
    }
}

__device__ __forceinline__ float contract_axis(float v) {
    return fabsf(v) <= 1.0f ? v : (2.0f - 1.0f / fabsf(v)) * copysignf(1.0f, v);
}

// World position -> the unit cube the hash grid is defined on: [-1, 1] of the inner box maps linearly, everything
// outside is folded into (1, 2) per axis, then (c + 2) / 4.  modules/NeRF/processRays.cu:21-46.
__device__ __forceinline__ float3 contract_pos(float3 pos, float3 aabb_min, float3 aabb_max) {
    const float ex = aabb_max.x - aabb_min.x, ey = aabb_max.y - aabb_min.y, ez = aabb_max.z - aabb_min.z;
    const float rx = (pos.x - aabb_min.x) / ex, ry = (pos.y - aabb_min.y) / ey, rz = (pos.z - aabb_min.z) / ez;
    const float cx = contract_axis(rx * 2.0f - 1.0f), cy = contract_axis(ry * 2.0f - 1.0f), cz = contract_axis(rz * 2.0f - 1.0f);
    return make_float3(fmaxf(0.0f, fminf((cx + 2.0f) * 0.25f, 1.0f)), fmaxf(0.0f, fminf((cy + 2.0f) * 0.25f, 1.0f)),
                       fmaxf(0.0f, fminf((cz + 2.0f) * 0.25f, 1.0f)));
}


// Are the GROUP rays of this lane's group of lanes (GROUP consecutive ones) so close that their samples at equal place share cells?
// Closer than 1 / 400 of the direction from ray to ray, and of the box in origin: pixels farther apart gain nothing from depth
// order.  All lanes of the warp call; a lane without a ray passes the last one's.
template <int GROUP>
__device__ __forceinline__ bool rays_close(float3 o, float3 d, float3 aabb_min, float3 aabb_max, int lane) {
    auto step = [&](float v) { return v - __shfl_up_sync(0xffffffffu, v, 1, GROUP); };   // the group's first lane keeps its own value: 0
    const float dx = step(d.x), dy = step(d.y), dz = step(d.z), ox = step(o.x), oy = step(o.y), oz = step(o.z);
    const float extent = fmaxf(aabb_max.x - aabb_min.x, fmaxf(aabb_max.y - aabb_min.y, aabb_max.z - aabb_min.z));
    constexpr float CLOSE2 = 1.0f / (400.0f * 400.0f);
    const bool near = dx * dx + dy * dy + dz * dz < CLOSE2 && ox * ox + oy * oy + oz * oz < CLOSE2 * extent * extent;
    constexpr uint32_t ALL = 0xffffffffu >> (32 - GROUP);
    return ((__ballot_sync(0xffffffffu, near) >> (lane & (32 - GROUP))) & ALL) == ALL;
}

// Copies the next round's `total` samples of a block's RAYS rays out: s_off has the block's samples before each ray and in all (RAYS + 1
// entries), base is where they start.  A thread takes every THREADS-th sample and looks its ray up: the loads of different samples are
// independent (a warp that took one ray after the other spent 25 us on a launch of 16 samples per ray, one after the other's latencies).
// order (nullable) lists the samples by place along the ray within groups of eight rays that s_close has, else ray after ray.
template <uint32_t RAYS, uint32_t THREADS, int UNROLL>
__device__ __forceinline__ void copy_round_out(const uint32_t* s_off, const bool* s_close, uint32_t base, uint32_t total, uint32_t first_ray,
                                               uint32_t round_begin, const float3* __restrict__ rays_o, const float3* __restrict__ rays_d, float3 aabb_min, float3 aabb_max,
                                               const float* __restrict__ rows, uint32_t row_stride, uint32_t* __restrict__ ray_idx_out,
                                               float4* __restrict__ pos_out, uint32_t* __restrict__ order) {
#pragma unroll UNROLL
    for (uint32_t s = threadIdx.x; s < total; s += THREADS) {
        uint32_t j = 0;   // the last ray whose samples start at or before s: rays without samples start where the next one does
#pragma unroll
        for (uint32_t step = RAYS / 2; step > 0; step >>= 1) j += s_off[j + step] <= s ? step : 0u;
        const uint32_t i = first_ray + j, k = s - s_off[j];
        const float3 o = rays_o[i], d = rays_d[i];
        const float t = rows[(size_t)i * row_stride + round_begin + k];
        ray_idx_out[base + s] = i;
        if (order != nullptr) {
            const uint32_t g = j & ~7u;
            uint32_t place = s;
            if (s_close[j >> 3]) {
                place = s_off[g];
#pragma unroll
                for (uint32_t m = 0; m < 8; m++) place += min(s_off[g + m + 1] - s_off[g + m], m < (j & 7u) ? k + 1 : k);
            }
            order[base + place] = base + s;
        }
        const float3 p = contract_pos(make_float3(o.x + t * d.x, o.y + t * d.y, o.z + t * d.z), aabb_min, aabb_max);
        st_cs_v4(&pos_out[base + s], make_uint4(__float_as_uint(p.x), __float_as_uint(p.y), __float_as_uint(p.z), 0u));
    }
}

}  // namespace nb
