// Backward pass of the whole field on the 5th-generation tensor cores: tcgen05.mma with accumulators in tensor memory.
//
// Same contract and same fp16 rounding points as field_backward_kernel (field_fused.cu).  What changes is where the
// GEMM operands and accumulators live.  The mma.sync formulation pulls every operand fragment through the load/store
// pipe (ldmatrix) and keeps the weight-gradient accumulators in 40 registers per thread; measured, that operand traffic
// is half of the kernel's L1TEX time - the pipe the gradient scatter's reductions also need.  Here
//   * every activation / gradient tile sits in shared memory in the tensor core's own core-matrix layout (8 rows x 16
//     bytes per core, no swizzle) and is read by the MMA unit directly, as a K-major operand in the layer GEMMs and, the
//     same bytes viewed MN-major, as an operand of the weight-gradient GEMMs (dW = dZ^T x A, a reduction over the rows);
//   * the weight-gradient accumulators of all five layers, and the bias gradients of the three wide layers (a GEMM with a
//     tile of ones), stay in tensor memory for the lifetime of the persistent CTA and are added to global memory once;
//   * two threads share a sample row, half of the columns each: they read it from tensor memory, apply bias / ReLU / mask,
//     round to fp16 and write their half of the next operand tile's row; after the last layer each holds 16 of the sample's 32
//     encoding gradients in registers and hands them to the scatter warps through shared memory.
//
// Warps 0-7 (two threads per row) run the epilogues of the chain of layer GEMMs above; that chain is a sequence of dependent
// stages, each waiting on the tensor core, so its warps are mostly asleep.  Warp 12 issues the MMAs: it waits until the chain warps
// have written a stage's operands, issues the product they wait for, then the stage's weight-gradient products, which run under
// the epilogue.  Warps 8-11 do nothing but the gradient scatter: they receive a tile's encoding gradients through a
// double-buffered shared-memory hand-over and issue its reductions while the chain is already on the next tile.  The scatter's
// index arithmetic and its L1TEX traffic thus run underneath the tensor-core chain instead of after it.
//
// What bounds the chain: a stage of a tile is about 450 cycles of epilogue, 200 of handing over (proxy fence, barrier) and 250 to 500 from
// there to the result, of which the products are 50 to 200; two tiles an SM are in flight, and their operands take a third of the
// shared memory's bandwidth.  Cycles a tile, one CTA on its SM / two: 13150 / 16900 with one thread of warp 0 issuing everything and the
// stage waiting for all of it, 11700 / 15300 with warp 0 as a whole issuing and the result committed first, 9900 / 14600 with
// a warp of its own (2^18 rows without scatter 84 -> 78 us).
// Beside these, 2^20 rows of rays (us): samples and rays looked up two stages before what they address, without scatter 242 -> 236, with
// list and scatter 302 as before; one arrival per warp instead of per thread, with list and scatter 309 -> 302, without 233 -> 236.
// Every wait - MMA barrier, hand-over full / empty - is bounded in TIME (the global timer, one second); a CTA whose wait
// runs out drops its accumulated weight gradients, raises an error flag in mapped host memory that the next
// nb_field_backward call (and nb_field_backward_tc_status) reports, waits for its MMAs in flight and leaves.
#include <atomic>
#include <type_traits>

#include "hashgrid_core.cuh"
#include "field_backward_tc.cuh"
#include "field_core.cuh"
#include "tensor_memory.cuh"

namespace nb {

extern std::atomic<uint64_t> g_launch_count;

namespace tc {

constexpr int CHAIN_WARPS = 8, CHAIN_THREADS = CHAIN_WARPS * 32;   // warps 0-7: GEMM chain, two threads per row
constexpr int SCATTER_WARPS = ROWS / 32;                           // warps 8-11: gradient scatter, a thread per row
constexpr int THREADS = CHAIN_THREADS + ROWS + 32;                 // warp 12: issues the MMAs

// ---- shared-memory map (bytes) ---------------------------------------------------------------------------------
static_assert(ROWS == ROWS_OF_TILE, "field_backward_tc.cuh");
constexpr uint32_t OFF_WD0 = 0;                                   // [64][32]
constexpr uint32_t OFF_WD1 = OFF_WD0 + tile_bytes(64, 32);        // [16][64]
constexpr uint32_t OFF_WC0 = OFF_WD1 + tile_bytes(16, 64);        // [64][32]
constexpr uint32_t OFF_WC1 = OFF_WC0 + tile_bytes(64, 32);        // [64][64]
constexpr uint32_t OFF_WC2 = OFF_WC1 + tile_bytes(64, 64);        // [16][64], rows 8..15 zero
constexpr uint32_t OFF_ONES = OFF_WC2 + tile_bytes(16, 64);       // [128][8] of 1.0
constexpr uint32_t OFF_E = OFF_ONES + tile_bytes(ROWS, 8);        // encoding            [128][32]
constexpr uint32_t OFF_CI = OFF_E + tile_bytes(ROWS, 32);         // colour input        [128][32]
constexpr uint32_t OFF_A = OFF_CI + tile_bytes(ROWS, 32);         // density hidden, later its gradient  [128][64]
constexpr uint32_t OFF_B = OFF_A + tile_bytes(ROWS, 64);          // colour hidden 1, later its gradient [128][64]
constexpr uint32_t OFF_C = OFF_B + tile_bytes(ROWS, 64);          // colour hidden 2, later its gradient [128][64]
constexpr uint32_t OFF_Z = OFF_C + tile_bytes(ROWS, 64);          // 16-wide gradients: colour output, then density output [128][16]
constexpr uint32_t OFF_BIAS = OFF_Z + tile_bytes(ROWS, 16);       // fp32 biases: density 64 + 16, colour 64 + 64 + 8
constexpr uint32_t OFF_X = OFF_BIAS + (64 + 16 + 64 + 64 + 8) * 4;   // hand-over: 2 buffers x [16 levels][128 rows] fp16 pairs
constexpr uint32_t SMEM_BYTES = OFF_X + 2 * 16 * ROWS * 4;   // 107 KB: two CTAs per SM (measured: at 111 KB only one is resident)

// ---- tensor-memory map (32-bit columns) ----------------------------------------------------------------------
constexpr uint32_t COL_WORK = 0;      // result of the current layer GEMM, up to 64 columns, 128 lanes
constexpr uint32_t COL_DWC1 = 64;     // dW colour 1   [64 out][64 in]   (64-row accumulators use lanes 0-15 of each warp's 32)
constexpr uint32_t COL_DWC0 = 128;    // dW colour 0   [64 out][32 in]
constexpr uint32_t COL_DWD0 = 160;    // dW density 0  [64 out][32 in]
constexpr uint32_t COL_DWC2T = 192;   // dW colour 2, transposed  [64 in][16 out]
constexpr uint32_t COL_DWD1T = 208;   // dW density 1, transposed [64 in][16 out]
constexpr uint32_t COL_DBC1 = 224;    // db colour 1 in column 0 of [64 out][8]
constexpr uint32_t COL_DBC0 = 232;
constexpr uint32_t COL_DBD0 = 240;
constexpr uint32_t TMEM_COLS = 256;   // two CTAs per SM share the 512 columns

__device__ __forceinline__ float clamp_logit(float v) {
    v = fmaxf(-64.0f, fminf(64.0f, v));
    return (v != v) ? 0.0f : v;
}
__device__ __forceinline__ float clamp_half_range(float v) {
    v = fmaxf(-65504.0f, fminf(65504.0f, v));
    return (v != v) ? 0.0f : v;
}

// All chain threads: do any of them pass true?
__device__ __forceinline__ bool any_of_chain(bool mine) {
    uint32_t any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\tbar.red.or.pred p, 1, %2, q;\n\tselp.u32 %0, 1, 0, p;\n\t}\n"
                 : "=r"(any) : "r"((uint32_t)mine), "n"(CHAIN_THREADS) : "memory");
    return any != 0;
}

template <bool GRAD_HALF, int COLOR_LAYERS>
__global__ void __launch_bounds__(THREADS, 2) field_backward_tc_kernel(const __grid_constant__ GridParams gp, const BackwardArgs a) {
    after_previous();
    static_assert(COLOR_LAYERS == 2 || COLOR_LAYERS == 3, "colour 32-64-8 or 32-64-64-8");
    // With two colour layers tile C holds their only hidden activation and the stages of the middle layer fall away.
    constexpr uint32_t OFF_H1 = COLOR_LAYERS == 3 ? OFF_B : OFF_C;                  // colour hidden 1, later its gradient
    constexpr int W_OUT = 64 * 32 + (COLOR_LAYERS == 3 ? 64 * 64 : 0);              // colour output layer in the weights
    constexpr int B_OUT = COLOR_LAYERS == 3 ? 128 : 64;                             // ... and in the biases
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t ready;        // the chain warps have written the stage's operands and read the last result
    __shared__ __align__(8) uint64_t done;         // the stage's result is in tensor memory
    __shared__ __align__(8) uint64_t used;         // the stage's weight-gradient products have read their operands
    __shared__ __align__(8) uint64_t drain;        // every MMA of the CTA is through
    __shared__ __align__(8) uint64_t x_full[2];    // hand-over buffer written by the 256 chain threads
    __shared__ __align__(8) uint64_t x_empty[2];   // ... read by the 128 scatter threads
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_flag_s;
    volatile int* abort_flag = &abort_flag_s;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;   // the shuffle tells the compiler that warp is the warp's
    const uint32_t sbase = smem_u32(smem);
    float* sBias = reinterpret_cast<float*>(smem + OFF_BIAS);
    const float* bD0 = sBias, *bD1 = sBias + 64, *bC0 = sBias + 80, *bC1 = sBias + 144;

    // ---- one-time set-up (all threads): weights and the ones tile in core-matrix order, biases, tensor memory, barriers
    auto stage_weights = [&](uint32_t off, const __half* W, int rows_valid, int rows, int cols) {
        const int cpr = cols >> 3;
        for (int c = tid; c < rows * cpr; c += THREADS) {
            const int r = c / cpr, c8 = c % cpr;
            cp_async16(smem + off + core_off(r, c8 * 8, cols), r < rows_valid ? (const void*)(W + r * cols + c8 * 8) : (const void*)W, r < rows_valid);
        }
    };
    stage_weights(OFF_WD0, a.Wd, 64, 64, 32);
    stage_weights(OFF_WD1, a.Wd + 64 * 32, 16, 16, 64);
    stage_weights(OFF_WC0, a.Wc, 64, 64, 32);
    if constexpr (COLOR_LAYERS == 3) stage_weights(OFF_WC1, a.Wc + 64 * 32, 64, 64, 64);
    stage_weights(OFF_WC2, a.Wc + W_OUT, 8, 16, 64);
    cp_async_commit();
    for (int i = tid; i < 80; i += THREADS) sBias[i] = a.bd[i];
    for (int i = tid; i < B_OUT; i += THREADS) sBias[80 + i] = a.bc[i];   // the output layer's are not needed
    if (tid < ROWS) {
        const uint32_t one2 = pack_half2(1.0f, 1.0f);
        *reinterpret_cast<uint4*>(smem + OFF_ONES + core_off(tid, 0, 8)) = make_uint4(one2, one2, one2, one2);
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_base_s)), "r"(TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    if (tid == 0) {
        mbar_init(&ready, (uint32_t)CHAIN_WARPS);
        mbar_init(&done, 1u);
        mbar_init(&used, 1u);
        mbar_init(&drain, 1u);
#pragma unroll
        for (int b = 0; b < 2; b++) {
            mbar_init(&x_full[b], (uint32_t)CHAIN_THREADS);
            mbar_init(&x_empty[b], (uint32_t)ROWS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        abort_flag_s = 0;
    }
    cp_async_wait_all();
    proxy_fence();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    const int64_t n = a.count != nullptr ? min((int64_t)__ldg(a.count), a.n) : a.n;
    const int64_t ntiles = (n + ROWS - 1) / ROWS;
    bool ok = true;

    if (warp == CHAIN_WARPS + SCATTER_WARPS) {
        // ================= issuing warp: all its lanes walk through, the elected one acts =================================
        // A stage's result is committed before the weight-gradient products of the same stage, which run under its epilogue; `used`
        // is committed where that epilogue, or the next tile's stage 0, overwrites what they read.
        const uint32_t lead = elected_lane();
        uint32_t phase = 0;
        auto next_stage = [&]() {
            if (!ok) return false;
            ok = __all_sync(0xffffffffu, mbar_wait(&ready, phase & 1, WAIT_LIMIT_NS, abort_flag));
            phase++;
            tc_fence_after();
            return ok;
        };
        bool add = false;   // the weight gradients have a sum to add to
        for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, add = true) {
            if (next_stage()) { gemm_layer(lead, tmem + COL_WORK, sbase + OFF_E, sbase + OFF_WD0, 32, 64); umma_commit(lead, &done); }
            if (next_stage()) { gemm_layer(lead, tmem + COL_WORK, sbase + OFF_A, sbase + OFF_WD1, 64, 16); umma_commit(lead, &done); }
            if (next_stage()) { gemm_layer(lead, tmem + COL_WORK, sbase + OFF_CI, sbase + OFF_WC0, 32, 64); umma_commit(lead, &done); }
            if constexpr (COLOR_LAYERS == 3)
                if (next_stage()) { gemm_layer(lead, tmem + COL_WORK, sbase + OFF_B, sbase + OFF_WC1, 64, 64); umma_commit(lead, &done); }
            if (next_stage()) {
                gemm_dinput(lead, tmem + COL_WORK, sbase + OFF_Z, 16, 16, sbase + OFF_WC2, 64, 64);
                umma_commit(lead, &done);
                gemm_outer(lead, tmem + COL_DWC2T, sbase + OFF_C, 64, sbase + OFF_Z, 16, 16, add);
                umma_commit(lead, &used);
            }
            if constexpr (COLOR_LAYERS == 3)
                if (next_stage()) {
                    gemm_dinput(lead, tmem + COL_WORK, sbase + OFF_C, 64, 64, sbase + OFF_WC1, 64, 64);
                    umma_commit(lead, &done);
                    gemm_outer(lead, tmem + COL_DWC1, sbase + OFF_C, 64, sbase + OFF_B, 64, 64, add);
                    umma_commit(lead, &used);
                    gemm_outer(lead, tmem + COL_DBC1, sbase + OFF_C, 64, sbase + OFF_ONES, 8, 8, add);
                }
            if (next_stage()) {
                gemm_dinput(lead, tmem + COL_WORK, sbase + OFF_H1, 64, 64, sbase + OFF_WC0, 32, 16);
                umma_commit(lead, &done);
                gemm_outer(lead, tmem + COL_DWC0, sbase + OFF_H1, 64, sbase + OFF_CI, 32, 32, add);
                gemm_outer(lead, tmem + COL_DBC0, sbase + OFF_H1, 64, sbase + OFF_ONES, 8, 8, add);
            }
            if (next_stage()) {
                gemm_dinput(lead, tmem + COL_WORK, sbase + OFF_Z, 16, 16, sbase + OFF_WD1, 64, 64);
                umma_commit(lead, &done);
                gemm_outer(lead, tmem + COL_DWD1T, sbase + OFF_A, 64, sbase + OFF_Z, 16, 16, add);
                umma_commit(lead, &used);
            }
            if (next_stage()) {
                gemm_dinput(lead, tmem + COL_WORK, sbase + OFF_A, 64, 64, sbase + OFF_WD0, 32, 32);
                umma_commit(lead, &done);
                gemm_outer(lead, tmem + COL_DWD0, sbase + OFF_A, 64, sbase + OFF_E, 32, 32, add);
                umma_commit(lead, &used);
                gemm_outer(lead, tmem + COL_DBD0, sbase + OFF_A, 64, sbase + OFF_ONES, 8, 8, add);
            }
        }
        // nothing of this CTA's may still write tensor memory when it is read or handed back, however the loop ended
        umma_commit(lead, &drain);
        if (!mbar_wait(&drain, 0, WAIT_LIMIT_NS)) ok = false;
    } else if (warp >= CHAIN_WARPS) {
        // ================= scatter warpgroup: thread = row of the tile handed over =====================================
        if (a.table_grads != nullptr) {
            const int r = tid - CHAIN_THREADS;
            int it = 0;
            for (int64_t tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x, it++) {
                const int buf = it & 1, use = it >> 1;
                const int64_t row = tile * ROWS + r;
                const bool has = row < n;
                float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
                if (has) p = ld_nc_f4(a.pos4 + (a.perm ? (int64_t)a.perm[row] : row) * 4);
                ScatterState ss;
                scatter_begin_warp(gp, p.x, p.y, p.z, lane, ss);
                const bool got = __all_sync(0xffffffffu, mbar_wait(&x_full[buf], use & 1, WAIT_LIMIT_NS, abort_flag));
                if (!got) { ok = false; break; }   // the chain gave up (or never came): leave, every wait here is bounded
                const uint32_t* x = reinterpret_cast<const uint32_t*>(smem + OFF_X) + buf * 16 * ROWS + r;
                // a warp is 32 consecutive rows working on one level at a time
#pragma unroll 1
                for (int l = a.scatter_begin; l < 16; l++) {
                    void* base = GRAD_HALF ? (void*)(reinterpret_cast<uint32_t*>(a.table_grads) + (size_t)l * gp.ls) : (void*)(a.table_grads + (size_t)l * gp.ls * 2);
                    if (!GRAD_HALF && l < a.coarse.levels)
                        base = a.coarse.copies + 2 * ((size_t)(blockIdx.x % a.coarse.count) * a.coarse.entries + (l > 0 ? a.coarse.first : 0));
                    scatter_level_at<GRAD_HALF>(gp, l, ss, has ? x[l * ROWS] : 0u, base, lane);
                }
                mbar_arrive(&x_empty[buf]);
            }
        }
    } else {
        // ================= chain warpgroups: row = tensor-memory lane, half of the columns each ===========================
        const int rt = tid & (ROWS - 1), h = tid >> 7;                                // row of the tile; which half of a result's columns
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);        // this warp's 32 lanes
        uint32_t phase = 0, used_phase = 0;
        int it = 0;
        float db_c2 = 0.f, db_d1 = 0.f;   // partial bias gradients of one output column per lane (see column_sums8)

        // The next stage's operands are written and the last result is read: visible to the tensor core, and said once a warp.
        auto hand_over = [&]() {
            proxy_fence();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&ready);
        };
        // Waits for the stage's result.  A warp whose wait runs out says so and goes on with whatever there is - every access stays
        // where it would have been - until its tile's end, where it leaves; nothing of it is kept.
        auto await = [&]() {
            if (!mbar_wait(&done, phase & 1, a.wait_ns, abort_flag)) *abort_flag = 1;
            __syncwarp();
            phase++;
            tc_fence_after();
        };
        // ... for the weight-gradient products behind it: what those read is overwritten next
        auto await_used = [&]() {
            if (!mbar_wait(&used, used_phase & 1, a.wait_ns, abort_flag)) *abort_flag = 1;
            __syncwarp();
            used_phase++;
        };
        // this thread's 32 columns of the result + bias, ReLU, fp16 -> the same columns of a 64-wide tile
        auto relu_stage = [&](uint32_t dst, const float* bias) {
            float v[32];
            tmem_ld32(lane_base + COL_WORK + 32 * h, v);
#pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int k = 8 * c + 2 * i;
                    add_f2(v[k], v[k + 1], *reinterpret_cast<const float2*>(bias + 32 * h + k));
                    o[i] = relu_half2(v[k], v[k + 1]);
                }
                *reinterpret_cast<uint4*>(smem + dst + core_off(rt, (4 * h + c) * 8, 64)) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        };
        // ... fp16, zeroed where the activation in the tile is not positive, written over the activation once the products that
        // read it are through
        auto mask_stage = [&](uint32_t dst) {
            float v[32];
            tmem_ld32(lane_base + COL_WORK + 32 * h, v);
            uint4 masked[4];
#pragma unroll
            for (int c = 0; c < 4; c++)
                masked[c] = masked_chunk(v + 8 * c, *reinterpret_cast<const uint4*>(smem + dst + core_off(rt, (4 * h + c) * 8, 64)));
            await_used();
#pragma unroll
            for (int c = 0; c < 4; c++) *reinterpret_cast<uint4*>(smem + dst + core_off(rt, (4 * h + c) * 8, 64)) = masked[c];
        };
        // The next tile's sample of this thread's row and its ray, and the samples whose encoding it fetches, which the addresses of its
        // inputs depend on: asked for two stages before them.  Rows past n take the last one's.
        auto e_row = [&](int i) { return (tid + CHAIN_THREADS * i) >> 2; };
        uint32_t pre_smp = 0, pre_ray = 0, pre_enc[2];
        auto fetch_index = [&](int64_t tile) {
            const int64_t last = min(tile * ROWS + rt, n - 1);
            pre_smp = a.perm ? a.perm[last] : (uint32_t)last;
            pre_ray = a.ray_idx ? a.ray_idx[pre_smp + a.ray_idx_offset] : pre_smp;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int64_t r = min(tile * ROWS + e_row(i), n - 1);
                pre_enc[i] = a.perm && !a.enc_by_row ? a.perm[r] : (uint32_t)r;
            }
        };
        // The next tile's inputs travel to registers while this tile's last stages run: two chunks of the encoding, the colour
        // gradient row, the direction.  Rows past n become zeros where they are used: a choice beside the load would wait for it there.
        uint4 pre_e[2], pre_z = make_uint4(0u, 0u, 0u, 0u);
        float pre_d[3];
        auto fetch = [&]() {
#pragma unroll
            for (int i = 0; i < 2; i++) pre_e[i] = ld_nc_v4(a.enc + (size_t)pre_enc[i] * 32 + (tid & 3) * 8);
            if (h == 0) pre_z = ld_nc_v4(a.dcolor + (size_t)pre_smp * 8);
            const float* dp = a.dirs3 + 3 * (size_t)pre_ray;
            pre_d[0] = dp[0]; pre_d[1] = dp[1]; pre_d[2] = dp[2];
        };
        if ((int64_t)blockIdx.x < ntiles) { fetch_index(blockIdx.x); fetch(); }

        for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x, it++) {
            const int64_t row = tile * ROWS + rt;
            const bool has = row < n;
            // ---- stage 0: encoding tile (zero rows past n) -----------------------------------------------------------------------
            if (it > 0) await_used();
#pragma unroll
            for (int i = 0; i < 2; i++)
                *reinterpret_cast<uint4*>(smem + OFF_E + core_off(e_row(i), (tid & 3) * 8, 32)) =
                    tile * ROWS + e_row(i) < n ? pre_e[i] : make_uint4(0u, 0u, 0u, 0u);
            if (!has) pre_z = make_uint4(0u, 0u, 0u, 0u);
            hand_over();

            // ---- stage 1: density hidden = relu(E Wd0^T + b) -> tile A; meanwhile the colour gradient (columns 8..15 zero) and the SH
            //      half of the colour input ------------------------------------------------------------------------------------------
            *reinterpret_cast<uint4*>(smem + OFF_Z + core_off(rt, 8 * h, 16)) = pre_z;
            {
                float sh[16];
                sh16(pre_d[0], pre_d[1], pre_d[2], sh);
                if (h == 0) store_chunk(smem + OFF_CI, rt, 2, 32, sh);
                else store_chunk(smem + OFF_CI, rt, 3, 32, sh + 8);
            }
            await();
            relu_stage(OFF_A, bD0);
            hand_over();

            // ---- stage 2: 16 logits = A Wd1^T + b; clamp; with the SH -> colour input tile ---------------------------------
            // bias gradient of the colour output layer: column sums of this tile's colour gradient (8 valid columns)
            if (h == 0) {
                const uint32_t w[4] = {pre_z.x, pre_z.y, pre_z.z, pre_z.w};
                float g8[8];
#pragma unroll
                for (int i = 0; i < 4; i++) { const float2 f = unpack_half2(w[i]); g8[2 * i] = f.x; g8[2 * i + 1] = f.y; }
                db_c2 += column_sums8(g8, lane);
            }
            await();
            {
                float v[8];
                tmem_ld8(lane_base + COL_WORK + 8 * h, v);
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = clamp_logit(v[i] + bD1[8 * h + i]);
                store_chunk(smem + OFF_CI, rt, h, 32, v);
            }
            hand_over();

            // ---- stage 3: colour hidden 1 = relu(CI Wc0^T + b) -> tile B (C) --------------------------------------------------
            await();
            relu_stage(OFF_H1, bC0);
            hand_over();

            // ---- stage 4: colour hidden 2 = relu(B Wc1^T + b) -> tile C ------------------------------------------------------
            if constexpr (COLOR_LAYERS == 3) {
                await();
                relu_stage(OFF_C, bC1);
                hand_over();
            }

            // ---- stage 5: colour output layer backward: dA = Z Wc2 ; dW^T += C^T Z ; dA masked by C > 0 -> tile C (in place) ----
            if (tile + gridDim.x < ntiles) fetch_index(tile + gridDim.x);
            await();
            mask_stage(OFF_C);
            hand_over();

            // ---- stage 6: colour layer 1 backward: dA = C Wc1 ; dW1 += C^T B ; dA masked by B > 0 -> tile B --------------------
            if constexpr (COLOR_LAYERS == 3) {
                await();
                mask_stage(OFF_B);
                hand_over();
            }

            // ---- stage 7: colour layer 0 backward: gradient of the 16 density outputs ; dW0 += B^T CI ; db0 += B^T 1 ----------
            // the sample of this row, its dL/dsigma, and the next tile's inputs: their latency lies under the MMAs
            const int64_t smp = has ? (a.perm ? (int64_t)a.perm[row] : row) : 0;
            const float ds = (h == 0 && has && a.dsigma != nullptr) ? a.dsigma[smp] : 0.f;
            if (tile + gridDim.x < ntiles) fetch();
            await();
            float g8[8];
            {
                float v[8];
                tmem_ld8(lane_base + COL_WORK + 8 * h, v);
                // compute_density_grad (modules/NeRF/otherKernels.cu:497-562): fp16 gradient, + dL/dsigma on logit 0, clamp, NaN -> 0
#pragma unroll
                for (int i = 0; i < 8; i++) v[i] = clamp_half_range(__half2float(__float2half_rn(v[i])) + (i == 0 ? ds : 0.f));
                store_chunk(smem + OFF_Z, rt, h, 16, v);
#pragma unroll
                for (int i = 0; i < 8; i++) g8[i] = __half2float(__float2half_rn(v[i]));
            }
            hand_over();

            // ---- stage 8: density layer 1 backward: dA = Z Wd1 ; dW1^T += A^T Z ; dA masked by A > 0 -> tile A ------------------
            // bias gradient of the density output layer: column sums of the fp16 values just written
            db_d1 += column_sums8(g8, lane);
            await();
            mask_stage(OFF_A);
            hand_over();

            // ---- stage 9: density layer 0 backward: dL/d(encoding) = A Wd0 ; dW0 += A^T E ; db0 += A^T 1 -------------------------
            await();
            {
                float v[16];
                tmem_ld16(lane_base + COL_WORK + 16 * h, v);
                uint32_t pk[8];  // half of the sample's 16 feature-pair gradients, fp16 as the reference rounds them
#pragma unroll
                for (int l = 0; l < 8; l++) pk[l] = pack_half2(v[2 * l], v[2 * l + 1]);
                if (has && a.denc_cols > 16 * h && *abort_flag == 0) {
                    uint2* dst = reinterpret_cast<uint2*>(a.denc + smp * a.denc_cols + 16 * h);
#pragma unroll
                    for (int q = 0; q < 4; q++)
                        if (16 * h + 4 * q < a.denc_cols) dst[q] = make_uint2(pk[2 * q], pk[2 * q + 1]);
                }
                if (a.table_grads != nullptr && *abort_flag == 0) {
                    // hand the tile's gradients to the scatter warps: buffer `it & 1`, free again once they have read it
                    const int buf = it & 1, use = it >> 1;
                    bool free_now = true;
                    if (use > 0) free_now = mbar_wait(&x_empty[buf], (use - 1) & 1, a.wait_ns);
                    if (free_now) {
                        uint32_t* x = reinterpret_cast<uint32_t*>(smem + OFF_X) + (buf * 16 + 8 * h) * ROWS + rt;
#pragma unroll
                        for (int l = 0; l < 8; l++) x[l * ROWS] = pk[l];
                        mbar_arrive(&x_full[buf]);
                    } else {
                        *abort_flag = 1;
                    }
                }
            }
            // The next tile's stage 0 overwrites E once this stage's products have read it; whatever else is written before a wait was
            // read by products that have been waited for.
            if (__any_sync(0xffffffffu, *abort_flag != 0)) break;
        }
        if ((int64_t)blockIdx.x < ntiles) {
            // the accumulators are complete; one warp that gave up is enough to drop them
            if (!mbar_wait(&drain, 0, a.wait_ns, abort_flag)) *abort_flag = 1;
            __syncwarp();
            tc_fence_after();
            if (any_of_chain(*abort_flag != 0)) ok = false;
        }

        // ---- flush: accumulators of this CTA -> global (fp32 reductions), once ---------------------------------------------
        if (ok && (int64_t)blockIdx.x < ntiles) {
            // a 64-row accumulator keeps row m in lane (m % 16) of warp (m / 16): lanes 0..15 of every warp hold rows; the two
            // warps of a lane quarter share the accumulators out
            const int m = 16 * (warp & 3) + lane;
            const bool holds = lane < 16;
            float v[32];
            if constexpr (COLOR_LAYERS == 3) {
                tmem_ld32(lane_base + COL_DWC1 + 32 * h, v);   // colour layer 1: [64 out][64 in]
                if (holds)
#pragma unroll
                    for (int q = 0; q < 8; q++) red_add_v4(a.dWc + 64 * 32 + m * 64 + 32 * h + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
            }
            if (h == 0) {
                tmem_ld32(lane_base + COL_DWC0, v);  // colour layer 0: [64 out][32 in]
                if (holds)
#pragma unroll
                    for (int q = 0; q < 8; q++) red_add_v4(a.dWc + m * 32 + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                tmem_ld32(lane_base + COL_DBC1, v);  // columns 0, 8, 16: bias gradients of colour 1, colour 0, density 0
                if (holds) {
                    if constexpr (COLOR_LAYERS == 3) red_add(a.dbc + 64 + m, v[0]);
                    red_add(a.dbc + m, v[8]);
                    red_add(a.dbd + m, v[16]);
                }
                if ((lane & 3) == 0) red_add(a.dbc + B_OUT + column_of_lane(lane), db_c2);
            } else {
                tmem_ld32(lane_base + COL_DWD0, v);  // density layer 0: [64 out][32 in]
                if (holds)
#pragma unroll
                    for (int q = 0; q < 8; q++) red_add_v4(a.dWd + m * 32 + 4 * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
                tmem_ld32(lane_base + COL_DWC2T, v);  // columns 0-15: colour output layer transposed [64 in][16 out], 16-31: density layer 1 transposed
                if (holds) {
#pragma unroll
                    for (int o = 0; o < 8; o++) red_add(a.dWc + W_OUT + o * 64 + m, v[o]);
#pragma unroll
                    for (int o = 0; o < 16; o++) red_add(a.dWd + 64 * 32 + o * 64 + m, v[16 + o]);
                }
            }
            if ((lane & 3) == 0) red_add(a.dbd + 64 + 8 * h + column_of_lane(lane), db_d1);
        }
    }
    if (!ok && lane == 0 && a.error_flag != nullptr) atomicExch_system(a.error_flag, 1);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
}

// ---- samples that matter -------------------------------------------------------------------------------------------------
// A sample whose colour gradient is zero in fp16 and whose density gradient rounds to zero in it (at most 2^-25) adds nothing to any
// gradient: every product of its row is a product with zero (one with an activation that has overflowed to infinity would be NaN).  Of a training step's samples - behind a surface, in empty
// space - that is four to seven in ten.  The backward goes through the others' list: (count, samples).
constexpr int LIVE_THREADS = 256, LIVE_PER_THREAD = 4;

__global__ void clear_count_kernel(uint32_t* count) {
    after_previous();
    *count = 0u;
}

// The samples of a block keep their order, which a ray's runs of samples in one cell live on.
__global__ void __launch_bounds__(LIVE_THREADS) live_rows_kernel(const __half* __restrict__ dcolor, const float* __restrict__ dsigma, int64_t n,
                                                                 uint32_t* count, uint32_t* rows) {
    after_previous();
    constexpr int WARPS = LIVE_THREADS / 32, PARTS = LIVE_PER_THREAD * WARPS;
    static_assert(PARTS == 32, "a lane per part");
    __shared__ uint32_t start[PARTS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t first = (int64_t)blockIdx.x * (LIVE_THREADS * LIVE_PER_THREAD) + threadIdx.x;
    uint4 z[LIVE_PER_THREAD];
    float ds[LIVE_PER_THREAD];
#pragma unroll
    for (int k = 0; k < LIVE_PER_THREAD; k++) {
        const int64_t i = first + k * LIVE_THREADS;
        z[k] = i < n ? ld_nc_v4(dcolor + i * 8) : make_uint4(0u, 0u, 0u, 0u);
        ds[k] = i < n ? __ldg(dsigma + i) : 0.f;
    }
    unsigned live[LIVE_PER_THREAD];
#pragma unroll
    for (int k = 0; k < LIVE_PER_THREAD; k++) {
        // what is no number is not zero
        live[k] = __ballot_sync(0xffffffffu, ((z[k].x | z[k].y | z[k].z | z[k].w) & 0x7fff7fffu) != 0u || !(fabsf(ds[k]) <= 1.0f / 33554432.0f));
        if (lane == 0) start[k * WARPS + warp] = __popc(live[k]);
    }
    __syncthreads();
    if (warp == 0) {
        const uint32_t mine = start[lane];
        uint32_t upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t below = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += below;
        }
        uint32_t base = 0u;
        if (lane == 31 && upto > 0u) base = atomicAdd(count, upto);
        base = __shfl_sync(0xffffffffu, base, 31);
        start[lane] = base + upto - mine;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < LIVE_PER_THREAD; k++)
        if ((live[k] >> lane) & 1u) rows[start[k * WARPS + warp] + __popc(live[k] & ((1u << lane) - 1u))] = (uint32_t)(first + k * LIVE_THREADS);
}

__global__ void __launch_bounds__(256) clear_copies_kernel(float2* copies, int count) {
    after_previous();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i < count) copies[i] = make_float2(0.f, 0.f);
}

// The copies' sums into the table's gradient.
__global__ void __launch_bounds__(256) add_copies_kernel(const CoarseCopies c, float* table_grads, int level_stride) {
    after_previous();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= c.entries) return;
    const float2* from = reinterpret_cast<const float2*>(c.copies) + i;
    float x = 0.f, y = 0.f;
#pragma unroll 8
    for (int k = 0; k < c.count; k++) {
        const float2 v = from[(size_t)k * c.entries];
        x += v.x; y += v.y;
    }
    const int64_t entry = i < c.first ? i : (int64_t)level_stride + (i - c.first);
    if (x != 0.f || y != 0.f) red_add_v2(table_grads + 2 * entry, x, y);
}

}  // namespace tc
}  // namespace nb

namespace nb {

std::atomic<int> g_backward_tc{2};        // nb_set_tuning("backward_tc", ...)
std::atomic<int> g_backward_tc_wait_us{1000000};   // nb_set_tuning("backward_tc_wait_us", ...): the chain's wait limit

// The error flag lives in mapped, portable host memory: the kernel raises it with a system-scope atomic, the host
// reads it without a CUDA call.  One flag per process, allocated on the first launch.
static std::atomic<int*> g_tc_error_flag{nullptr};

int* wait_error_flag() {
    int* p = g_tc_error_flag.load(std::memory_order_acquire);
    if (p != nullptr) return p;
    int* fresh = nullptr;
    if (cudaHostAlloc((void**)&fresh, 64, cudaHostAllocPortable | cudaHostAllocMapped) != cudaSuccess || fresh == nullptr) return nullptr;
    *fresh = 0;
    int* expected = nullptr;
    if (!g_tc_error_flag.compare_exchange_strong(expected, fresh)) { cudaFreeHost(fresh); return expected; }
    return fresh;
}

// Non-zero when a wait of the tensor-memory backward kernel has run out since the flag was last cleared.
int field_backward_tc_failed() {
    int* p = g_tc_error_flag.load(std::memory_order_acquire);
    return p != nullptr && *reinterpret_cast<volatile int*>(p) != 0;
}

tc::CoarseCopies coarse_copies(const GridParams& gp, void* at, int64_t room) {
    tc::CoarseCopies c{};
    if (gp.dls < tc::COARSE_LEVELS || at == nullptr || gp.grad_half) return c;
    int64_t entries[tc::COARSE_LEVELS];
    for (int l = 0; l < tc::COARSE_LEVELS; l++) {
        const int64_t w = (int64_t)gp.sscales[l] + 1;
        entries[l] = (w * w * w + 1) / 2 * 2;   // every copy of a level starts on 16 bytes: x neighbours are reduced as one where a run's sums are
    }
    const int64_t all = entries[0] + entries[1];
    const int64_t fit = room / (all * 8);
    if (fit < tc::COARSE_COPIES_MIN) return c;
    c.count = (int)(fit < tc::COARSE_COPIES_MAX ? fit : tc::COARSE_COPIES_MAX);
    c.copies = (float*)at; c.levels = tc::COARSE_LEVELS; c.first = (int)entries[0]; c.entries = (int)all;
    return c;
}

// Host side: launched by nb_field_backward when the tensor-memory path is selected.
int launch_field_backward_tc(const GridParams& gp, const tc::BackwardArgs& args_in, cudaStream_t st) {
    tc::BackwardArgs args = args_in;
    args.error_flag = wait_error_flag();
    if (args.error_flag == nullptr) return nb_set_error(NB_ERR_CUDA, "field backward: no mapped host memory for the error flag");
    const int wait_us = g_backward_tc_wait_us.load();
    args.wait_ns = wait_us <= 0 ? 0ull : (uint64_t)wait_us * 1000ull;
    auto kern = args.color_layers == 3 ? (gp.grad_half ? tc::field_backward_tc_kernel<true, 3> : tc::field_backward_tc_kernel<false, 3>)
                                       : (gp.grad_half ? tc::field_backward_tc_kernel<true, 2> : tc::field_backward_tc_kernel<false, 2>);
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc::SMEM_BYTES));
    const int64_t ntiles = (args.n + tc::ROWS - 1) / tc::ROWS;
    // Two CTAs per SM: 107 KB of shared memory, 72 registers x 416 threads (59904 of 65536; 80 registers would leave room for one) and 256
    // tensor-memory columns each.  The grid is sized by that count, not by cudaOccupancyMaxActiveBlocksPerMultiprocessor, which answers 1
    // for this kernel although two CTAs are resident (2^20 samples with their scatter: 0.35 ms with 296 CTAs, 0.50 ms with 148).
    int64_t grid = (int64_t)nb_num_sms() * 2;
    if (grid > ntiles) grid = ntiles;
    if (args.live != nullptr) {
        constexpr int PER_BLOCK = tc::LIVE_THREADS * tc::LIVE_PER_THREAD;
        launch_after(tc::clear_count_kernel, 1, 1, 0, st, args.live);
        NB_CHECK_LAUNCH();
        launch_after(tc::live_rows_kernel, (unsigned)((args.n + PER_BLOCK - 1) / PER_BLOCK), tc::LIVE_THREADS, 0, st, args.dcolor, args.dsigma, args.n,
                     args.live, args.live + 1);
        NB_CHECK_LAUNCH();
        g_launch_count += 2;
        args.count = args.live;
        args.perm = args.live + 1;
    }
    const int copies = args.coarse.levels > 0 ? args.coarse.entries * args.coarse.count : 0;
    if (copies > 0) {
        launch_after(tc::clear_copies_kernel, (unsigned)((copies + 255) / 256), 256, 0, st, (float2*)args.coarse.copies, copies);
        NB_CHECK_LAUNCH();
        g_launch_count++;
    }
    launch_after(kern, (unsigned)grid, tc::THREADS, tc::SMEM_BYTES, st, gp, args);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    if (copies > 0) {
        launch_after(tc::add_copies_kernel, (unsigned)((args.coarse.entries + 255) / 256), 256, 0, st, args.coarse, args.table_grads, gp.ls);
        NB_CHECK_LAUNCH();
        g_launch_count++;
    }
    return NB_OK;
}

}  // namespace nb

// NB_OK when no wait of the tensor-memory backward kernel has run out since the last call; otherwise NB_ERR_CUDA, and
// the flag is cleared.  Synchronises the device first, so that it speaks for every launch enqueued so far.
extern "C" int nb_field_backward_tc_status(void) {
    NB_CUDA(cudaDeviceSynchronize());
    if (nb::field_backward_tc_failed()) {
        *reinterpret_cast<volatile int*>(nb::g_tc_error_flag.load()) = 0;
        return nb_set_error(NB_ERR_CUDA, "field backward (tensor memory): a bounded wait inside the kernel ran out; the gradients of that launch are incomplete");
    }
    return NB_OK;
}
