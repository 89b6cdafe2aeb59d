// Backward of a plain MLP with hidden width 64 on the 5th-generation tensor cores: dW, db and optionally dX.
//
// Same contract and fp16 rounding points as mlp_backward_kernel (mlp.cu), which remains for the other widths: there every
// operand fragment passes the load/store pipe, a layer's tile is fetched when the layer before is done with its buffer, and
// the chain load - products - mask repeats per layer with nothing underneath.  Here
//   * activations and gradients are core-matrix tiles in shared memory that tcgen05.mma reads directly, K-major for
//     dA = dZ W and, the same bytes viewed MN-major, for dW = dZ^T A (a reduction over the rows; where dZ is narrower than
//     64 columns the transpose A^T dZ); a product with eight columns of ones gives db, the same one where there is room for
//     them behind every activation;
//   * the masked gradient of a layer overwrites the activation that masked it, so a layer's buffers fall free one by one
//     and the next tile's are fetched into them (SETS == 1), or a whole second set is in flight where it fits (SETS == 2);
//   * all weight gradients stay in tensor memory for the life of the CTA, one per SM, and are added to global memory once;
//   * GROUPS row groups of 256 threads (two threads per row) work on a tile each, so that one's epilogue runs under the
//     other's products.  ONE warp issues everything, taking the groups in turn: the accumulators are shared, and MMAs
//     are ordered among themselves only when one thread issues them.
// Every wait is bounded in time; a CTA whose wait runs out adds nothing, raises the error flag and leaves after its MMAs.
// The chain of a tile - hand-over, products, tensor-memory load, mask - binds, and memory: past the first 2^16 rows it moves
// 3.7 TB/s.  dA is committed before dW so that its epilogue starts under dW's products.  Against the register kernel, caches cold (us):
// 64-64-64-64-64 at 2^18 rows 152 -> 82, 64-64-64 70 -> 54, 32-64-64-8 74 -> 55, 32-64-16 42 -> 38; at 1000 rows the two are equal.
// Issued by a whole warp instead of by one thread, which cost 46 cycles an MMA, and one arrival per warp where every thread had
// arrived (2^18 rows, caches warm): 82 -> 72, 55 -> 53, 52.5 -> 49.
#include <atomic>

#include "field_backward_tc.cuh"
#include "mlp_backward_tc.cuh"
#include "tensor_memory.cuh"

namespace nb {

extern std::atomic<uint64_t> g_launch_count;

namespace tc {

constexpr int MLP_H = 64, GROUPS = 2, GROUP_THREADS = 2 * ROWS, MLP_THREADS = GROUPS * GROUP_THREADS + 32;

template <int K0_, int OUT_, int NL_>
struct MlpTc {
    static constexpr int K0 = K0_, OUT = OUT_, NL = NL_, H = MLP_H;
    static_assert(NL >= 2 && (K0 == 32 || K0 == 64) && (OUT == 8 || OUT == 16 || OUT == 64), "shapes of this kernel");
    static constexpr int ZC = OUT < 16 ? 16 : OUT;      // columns of the output gradient's tile
    __host__ __device__ static constexpr int in_dim(int l) { return l == 0 ? K0 : H; }
    __host__ __device__ static constexpr int out_dim(int l) { return l == NL - 1 ? OUT : H; }
    __host__ __device__ static constexpr int z_cols(int l) { return l == NL - 1 ? ZC : H; }
    __host__ __device__ static constexpr int w_off(int l) { int o = 0; for (int i = 0; i < l; i++) o += in_dim(i) * out_dim(i); return o; }
    // buffer b < NL: input activation of layer b and ones, later the gradient of layer b - 1's output; buffer NL: output gradient
    __host__ __device__ static constexpr int cols(int b) { return b == NL ? ZC : in_dim(b); }
    // Ones behind the activations save a product per layer (32-64-64-8 at 2^18 rows: 59 -> 55 us), but with four 64-wide layers
    // it is 82 -> 93 us.
    static constexpr bool ONES_BEHIND = NL < 4;
    __host__ __device__ static constexpr int pitch(int b) { return b == NL ? ZC : in_dim(b) + (ONES_BEHIND ? 8 : 0); }
    __host__ __device__ static constexpr uint32_t buf_off(int b) { uint32_t o = 0; for (int i = 0; i < b; i++) o += tile_bytes(ROWS, pitch(i)); return o; }
    static constexpr uint32_t SET_BYTES = buf_off(NL + 1);
    // shared memory: weights [z_cols][in_dim] per layer, ones, buffer sets
    __host__ __device__ static constexpr uint32_t sw_off(int l) { uint32_t o = 0; for (int i = 0; i < l; i++) o += tile_bytes(z_cols(i), in_dim(i)); return o; }
    static constexpr uint32_t OFF_ONES = sw_off(NL), OFF_SETS = OFF_ONES + (ONES_BEHIND ? 0u : tile_bytes(ROWS, 8));
    static constexpr int SETS = OFF_SETS + 2 * GROUPS * SET_BYTES <= 226 * 1024 ? 2 : 1;
    static constexpr uint32_t SMEM = OFF_SETS + SETS * GROUPS * SET_BYTES;
    static_assert(SMEM <= 226 * 1024, "one CTA per SM");
    // tensor memory columns
    __host__ __device__ static constexpr bool transposed(int l) { return out_dim(l) != 64; }
    __host__ __device__ static constexpr uint32_t dw_cols(int l) { return transposed(l) ? ZC : in_dim(l) + 8; }   // db behind dW
    __host__ __device__ static constexpr uint32_t col_dw(int l) { uint32_t o = 64 * GROUPS; for (int i = 0; i < l; i++) o += dw_cols(i); return o; }
    static constexpr uint32_t COLS = col_dw(NL), TMEM = COLS <= 256 ? 256 : 512;
    static_assert(COLS <= 512 && ZC % 16 == 0, "tensor memory");
};

struct MlpArgs {
    const __half *dL, *W, *act0, *acts;
    int64_t n;
    float *dW, *db;
    __half* dX;          // nullable
    int dx_wide;         // rows of dX start on 32-byte boundaries
    int* error_flag;
};

// 16-byte chunks of rows [row0, row0 + 128) of src[n][VALID] into a tile of COLS columns; rows past n and columns past VALID are zero.
// Eight lanes take eight rows of one chunk column: shared-memory writes without conflicts, 64-byte runs of global memory.
template <int COLS, int VALID, int PITCH>
__device__ __forceinline__ void load_tile(unsigned char* tile, const __half* __restrict__ src, int64_t row0, int64_t n, int t) {
    constexpr int CPR = COLS / 8, PER = CPR < 4 ? CPR : 4, ROWS_PER_WARP = 32 / PER, PARTS = CPR / PER, TASKS = ROWS / ROWS_PER_WARP * PARTS;
    const int warp = t >> 5, lane = t & 31;
#pragma unroll
    for (int k = 0; k < TASKS / (GROUP_THREADS / 32); k++) {
        const int task = warp + k * (GROUP_THREADS / 32);
        const int r = (task / PARTS) * ROWS_PER_WARP + (lane & 7) + 8 * (lane / (8 * PER)), c8 = (task % PARTS) * PER + (lane >> 3) % PER;
        const bool valid = row0 + r < n && c8 * 8 < VALID;
        cp_async16(tile + core_off(r, c8 * 8, PITCH), valid ? src + (row0 + r) * VALID + c8 * 8 : src, valid);
    }
}

template <class S, int B>
__device__ __forceinline__ void load_buffer(unsigned char* set, const MlpArgs& a, int64_t row0, int t) {
    if constexpr (B == S::NL) load_tile<S::ZC, S::OUT, S::ZC>(set + S::buf_off(B), a.dL, row0, a.n, t);
    else if constexpr (B == 0) load_tile<S::K0, S::K0, S::pitch(B)>(set + S::buf_off(B), a.act0, row0, a.n, t);
    else load_tile<S::H, S::H, S::pitch(B)>(set + S::buf_off(B), a.acts + (int64_t)(B - 1) * a.n * S::H, row0, a.n, t);
}
template <class S, int B>
__device__ __forceinline__ void load_buffers_down(unsigned char* set, const MlpArgs& a, int64_t row0, int t) {
    load_buffer<S, B>(set, a, row0, t);
    if constexpr (B > 0) load_buffers_down<S, B - 1>(set, a, row0, t);
}
template <class S, int L>
__device__ __forceinline__ void stage_mlp_weights(unsigned char* smem, const __half* __restrict__ W, int tid) {
    if constexpr (L < S::NL) {
        constexpr int K = S::in_dim(L), R = S::z_cols(L), CPR = K / 8;
        for (int c = tid; c < R * CPR; c += MLP_THREADS) {
            const int r = c / CPR, c8 = c % CPR;
            const bool valid = r < S::out_dim(L);
            cp_async16(smem + S::sw_off(L) + core_off(r, c8 * 8, K), valid ? W + S::w_off(L) + r * K + c8 * 8 : W, valid);
        }
        stage_mlp_weights<S, L + 1>(smem, W, tid);
    }
}

__device__ __forceinline__ void st_global_v8(void* p, const uint32_t (&v)[8]) {
    asm volatile("st.global.v8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};\n" ::"l"(p), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]),
                 "r"(v[7]) : "memory");
}

// A CTA's waits share this: the first that runs out ends all of them.
struct MlpSync {
    uint64_t ready[GROUPS];   // a group's tiles for the next stage are in place
    uint64_t done[GROUPS];    // its dA is there
    uint64_t used[GROUPS];    // its buffers have been read
    uint64_t drain;
    uint32_t tmem_base;
    volatile int abort;
};

// The MMAs of layer L's backward for one tile.
template <class S, int L, bool WRITE_DX>
__device__ __forceinline__ void issue_layer(uint32_t lead, MlpSync& sync, uint32_t tmem, uint32_t sbase, uint32_t set, int group, bool accumulate) {
    const uint32_t z = set + S::buf_off(L + 1), x = set + S::buf_off(L);
    constexpr int K = S::in_dim(L), ZC = S::z_cols(L), ZP = S::pitch(L + 1), XP = S::pitch(L);
    if constexpr (L > 0 || WRITE_DX) gemm_dinput(lead, tmem + 64 * group, z, ZP, ZC, sbase + S::sw_off(L), K, K);
    umma_commit(lead, &sync.done[group]);
    if constexpr (S::transposed(L)) gemm_outer(lead, tmem + S::col_dw(L), x, XP, z, ZP, ZC, accumulate);
    else gemm_outer(lead, tmem + S::col_dw(L), z, ZP, x, XP, S::ONES_BEHIND ? K + 8 : K, accumulate);
    if constexpr (!S::transposed(L) && !S::ONES_BEHIND) gemm_outer(lead, tmem + S::col_dw(L) + K, z, ZP, sbase + S::OFF_ONES, 8, 8, accumulate);
    umma_commit(lead, &sync.used[group]);
}

// Stages NL-1 .. 0 of one tile, from a row group's side.  Returns false when a wait ran out.
template <class S, int L, bool WRITE_DX>
__device__ __forceinline__ bool group_stages(const MlpArgs& a, unsigned char* set, MlpSync& sync, int group, int t, uint32_t tmem, uint32_t& phase,
                                             int64_t tile, int64_t next_tile, int64_t ntiles, float& db_out) {
    const int lane = t & 31, r = t & (ROWS - 1), h = t >> 7;
    const uint32_t work = tmem + ((uint32_t)(((t >> 5) & 3) * 32) << 16) + 64 * group;
    if constexpr (S::SETS == 1 && L > 0) asm volatile("cp.async.wait_group 2;\n" ::: "memory");
    if constexpr (S::SETS == 2 && L == S::NL - 1) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    proxy_fence();
    tc_fence_before();
    __syncwarp();
    if (lane == 0) mbar_arrive(&sync.ready[group]);
    if constexpr (L == S::NL - 1 && S::OUT < 64) {
        // bias gradient of a narrow output layer: column sums of its gradient, under the products
        if (8 * h < S::OUT) {
            const int64_t row = tile * ROWS + r;
            const uint4 q = row < a.n ? ld_nc_v4(a.dL + row * S::OUT + 8 * h) : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
            float g8[8];
#pragma unroll
            for (int i = 0; i < 4; i++) { const float2 f = unpack_half2(w[i]); g8[2 * i] = f.x; g8[2 * i + 1] = f.y; }
            db_out += column_sums8(g8, lane);
        }
    }
    auto await = [&](uint64_t* bar) {
        if (__all_sync(0xffffffffu, mbar_wait(bar, phase & 1, WAIT_LIMIT_NS, &sync.abort))) return true;
        sync.abort = 1;
        return false;
    };
    if (!await(&sync.done[group])) return false;
    tc_fence_after();
    // what the other products of this layer read stays until they are through
    auto buffers_free = [&]() {
        if (!await(&sync.used[group])) return false;
        phase++;
        if constexpr (S::SETS == 1) {
            // the gradient just consumed was the last user of its buffer
            if (next_tile < ntiles) load_buffer<S, L + 1>(set, a, next_tile * ROWS, t);
            if constexpr (L == 0)
                if (next_tile < ntiles) load_buffer<S, 0>(set, a, next_tile * ROWS, t);
            cp_async_commit();
        }
        return true;
    };
    if constexpr (L > 0) {
        float v[32];
        uint4 masked[4];
        tmem_ld32(work + 32 * h, v);
        uint4* p[4];
#pragma unroll
        for (int c = 0; c < 4; c++) {
            p[c] = reinterpret_cast<uint4*>(set + S::buf_off(L) + core_off(r, (4 * h + c) * 8, S::pitch(L)));
            masked[c] = masked_chunk(v + 8 * c, *p[c]);
        }
        if (!buffers_free()) return false;
#pragma unroll
        for (int c = 0; c < 4; c++) *p[c] = masked[c];
        return group_stages<S, L - 1, WRITE_DX>(a, set, sync, group, t, tmem, phase, tile, next_tile, ntiles, db_out);
    } else {
        if constexpr (WRITE_DX) {
            constexpr int HALF = S::K0 / 2;   // columns of this thread
            float v[HALF];
            if constexpr (HALF == 32) tmem_ld32(work + 32 * h, v);
            else tmem_ld16(work + 16 * h, v);
            const int64_t row = tile * ROWS + r;
            if (row < a.n) {
                __half* dst = a.dX + row * S::K0 + HALF * h;
#pragma unroll
                for (int q = 0; q < HALF / 16; q++) {
                    uint32_t o[8];
#pragma unroll
                    for (int i = 0; i < 8; i++) o[i] = pack_half2(v[16 * q + 2 * i], v[16 * q + 2 * i + 1]);
                    if (a.dx_wide) st_global_v8(dst + 16 * q, o);
                    else {
                        *reinterpret_cast<uint4*>(dst + 16 * q) = make_uint4(o[0], o[1], o[2], o[3]);
                        *reinterpret_cast<uint4*>(dst + 16 * q + 8) = make_uint4(o[4], o[5], o[6], o[7]);
                    }
                }
            }
        }
        return buffers_free();
    }
}

// ... and from the issuing warp's side: the groups in turn.
template <class S, int L, bool WRITE_DX>
__device__ __forceinline__ bool issue_stages(uint32_t lead, uint32_t sbase, MlpSync& sync, uint32_t tmem, int64_t it, int64_t ntiles) {
    for (int g = 0; g < GROUPS; g++) {
        if ((it * GROUPS + g) * gridDim.x + blockIdx.x >= ntiles) continue;
        const uint32_t stage = (uint32_t)it * S::NL + (S::NL - 1 - L);
        if (!__all_sync(0xffffffffu, mbar_wait(&sync.ready[g], stage & 1, WAIT_LIMIT_NS, &sync.abort))) { sync.abort = 1; return false; }
        tc_fence_after();
        const uint32_t set = sbase + S::OFF_SETS + (g * S::SETS + (S::SETS == 2 ? (uint32_t)it & 1u : 0u)) * S::SET_BYTES;
        issue_layer<S, L, WRITE_DX>(lead, sync, tmem, sbase, set, g, it > 0 || g > 0);
    }
    if constexpr (L > 0) return issue_stages<S, L - 1, WRITE_DX>(lead, sbase, sync, tmem, it, ntiles);
    return true;
}

// Accumulators to global memory.  Row m of a 64-row accumulator sits in lane m % 16 of lane quarter m / 16; the warps of a quarter
// take 32 columns in turn.
template <class S, int L>
__device__ __forceinline__ void flush_layers(const MlpArgs& a, uint32_t lanes, int turn, int lane, int m) {
    if constexpr (L < S::NL) {
        constexpr int TURNS = GROUPS * 2, K = S::in_dim(L);
        float* dW = a.dW + S::w_off(L);
        constexpr int b_off = L * S::H;
        if constexpr (S::transposed(L)) {
            if (turn == L % TURNS) {
                float v[16];
                tmem_ld16(lanes + S::col_dw(L), v);
                if (lane < 16)
#pragma unroll
                    for (int o = 0; o < S::OUT; o++) red_add(dW + o * K + m, v[o]);
            }
        } else {
#pragma unroll
            for (int c = 0; c < K / 32; c++)
                if (turn == (2 * L + c) % TURNS) {
                    float v[32];
                    tmem_ld32(lanes + S::col_dw(L) + 32 * c, v);
                    if (lane < 16)
#pragma unroll
                        for (int q = 0; q < 8; q++) red_add_v4(dW + m * K + 32 * c + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                }
            if (turn == (2 * L + 2) % TURNS) {
                float v[8];
                tmem_ld8(lanes + S::col_dw(L) + K, v);
                if (lane < 16) red_add(a.db + b_off + m, v[0]);
            }
        }
        flush_layers<S, L + 1>(a, lanes, turn, lane, m);
    }
}

template <class S, bool WRITE_DX>
__global__ void __launch_bounds__(MLP_THREADS, 1) mlp_backward_tc_kernel(const MlpArgs a) {
    after_previous();
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) MlpSync sync;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t sbase = smem_u32(smem);
    const int64_t ntiles = (a.n + ROWS - 1) / ROWS;
    const int group = tid / GROUP_THREADS, t = tid % GROUP_THREADS;   // group == GROUPS: the issuing warp
    auto tile_of = [&](int64_t it) { return (it * GROUPS + group) * gridDim.x + blockIdx.x; };
    unsigned char* sets = smem + S::OFF_SETS + group * S::SETS * S::SET_BYTES;

    stage_mlp_weights<S, 0>(smem, a.W, tid);
    const uint32_t one2 = pack_half2(1.0f, 1.0f);
    const uint4 ones = make_uint4(one2, one2, one2, one2);
    if constexpr (!S::ONES_BEHIND) {
        if (tid < ROWS) *reinterpret_cast<uint4*>(smem + S::OFF_ONES + core_off(tid, 0, 8)) = ones;
    } else if (group < GROUPS) {
        static_assert(!S::ONES_BEHIND || S::SETS == 2, "a thread of a row for each set");
#pragma unroll
        for (int b = 0; b < S::NL; b++)
            *reinterpret_cast<uint4*>(sets + (t >> 7) * S::SET_BYTES + S::buf_off(b) + core_off(t & (ROWS - 1), S::in_dim(b), S::pitch(b))) = ones;
    }
    cp_async_commit();
    // the first tile: with one set in the order, and the commit groups, in which its stages will ask for the buffers
    if (group < GROUPS) {
        const bool any = tile_of(0) < ntiles;
        if constexpr (S::SETS == 2) {
            if (any) load_buffers_down<S, S::NL>(sets, a, tile_of(0) * ROWS, t);
            cp_async_commit();
        } else {
            static_assert(S::SETS == 2 || S::NL == 4, "the waits of one set count the groups of four layers");
            if (any) load_buffer<S, 4>(sets, a, tile_of(0) * ROWS, t);
            cp_async_commit();
            if (any) load_buffer<S, 3>(sets, a, tile_of(0) * ROWS, t);
            cp_async_commit();
            if (any) load_buffer<S, 2>(sets, a, tile_of(0) * ROWS, t);
            cp_async_commit();
            if (any) { load_buffer<S, 1>(sets, a, tile_of(0) * ROWS, t); load_buffer<S, 0>(sets, a, tile_of(0) * ROWS, t); }
            cp_async_commit();
        }
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&sync.tmem_base)), "r"(S::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        for (int g = 0; g < GROUPS; g++) { mbar_init(&sync.ready[g], GROUP_THREADS / 32); mbar_init(&sync.done[g], 1u); mbar_init(&sync.used[g], 1u); }
        mbar_init(&sync.drain, 1u);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        sync.abort = 0;
    }
    // the weights: everything but this thread's last group(s)
    if constexpr (S::SETS == 2) asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    else asm volatile("cp.async.wait_group 4;\n" ::: "memory");
    if (group == GROUPS) cp_async_wait_all();
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = sync.tmem_base;
    float db_out = 0.f;

    if (group < GROUPS) {
        uint32_t phase = 0;
        for (int64_t it = 0; tile_of(it) < ntiles; it++) {
            unsigned char* set = sets;
            if constexpr (S::SETS == 2) {
                set += (it & 1) * S::SET_BYTES;
                if (tile_of(it + 1) < ntiles) load_buffers_down<S, S::NL>(sets + (~it & 1) * S::SET_BYTES, a, tile_of(it + 1) * ROWS, t);
                cp_async_commit();
            }
            if (!group_stages<S, S::NL - 1, WRITE_DX>(a, set, sync, group, t, tmem, phase, tile_of(it), tile_of(it + 1), ntiles, db_out)) break;
        }
        cp_async_wait_all();
    } else {
        const uint32_t lead = elected_lane();
        for (int64_t it = 0; it * GROUPS * gridDim.x + blockIdx.x < ntiles; it++)
            if (!issue_stages<S, S::NL - 1, WRITE_DX>(lead, sbase, sync, tmem, it, ntiles)) break;
        // nothing of this CTA's may still write tensor memory when it is read or handed back
        umma_commit(lead, &sync.drain);
        if (!mbar_wait(&sync.drain, 0, WAIT_LIMIT_NS)) sync.abort = 1;
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (sync.abort == 0) {
        if (group < GROUPS) {
            flush_layers<S, 0>(a, tmem + ((uint32_t)((warp & 3) * 32) << 16), warp >> 2, lane, 16 * (warp & 3) + lane);
            if constexpr (S::OUT < 64)
                if (8 * (t >> 7) < S::OUT && (lane & 3) == 0) red_add(a.db + (S::NL - 1) * S::H + 8 * (t >> 7) + column_of_lane(lane), db_out);
        }
    } else if (tid == 0) {
        atomicExch_system(a.error_flag, 1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(S::TMEM) : "memory");
}

}  // namespace tc

template <class S>
static int launch_tc(tc::MlpArgs a, cudaStream_t st) {
    a.error_flag = wait_error_flag();
    if (a.error_flag == nullptr) return nb_set_error(NB_ERR_CUDA, "nb_mlp_backward: no mapped host memory for the error flag");
    auto kern = a.dX != nullptr ? tc::mlp_backward_tc_kernel<S, true> : tc::mlp_backward_tc_kernel<S, false>;
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM));
    const int64_t ntiles = (a.n + tc::ROWS - 1) / tc::ROWS;
    const int64_t grid = ntiles < nb_num_sms() ? ntiles : nb_num_sms();
    launch_after(kern, (unsigned)grid, tc::MLP_THREADS, S::SMEM, st, a);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

int launch_mlp_backward_tc(const nb_mlp_desc* d, const void* dL, const void* W, const void* act0, const void* acts, int64_t n, float* dW, float* db,
                           void* dX, cudaStream_t st) {
    const tc::MlpArgs a{(const __half*)dL, (const __half*)W, (const __half*)act0, (const __half*)acts, n, dW, db, (__half*)dX,
                        (reinterpret_cast<uintptr_t>(dX) & 31u) == 0, nullptr};
#define X(K0, OUT, NL) \
    if (d->input_dim == K0 && d->output_dim == OUT && d->num_layers == NL) return launch_tc<tc::MlpTc<K0, OUT, NL>>(a, st);
    NB_MLP_TC_SHAPES(X)
#undef X
    return nb_set_error(NB_ERR_UNSUPPORTED, "nb_mlp_backward: no tensor-memory kernel for this shape");
}

}  // namespace nb
