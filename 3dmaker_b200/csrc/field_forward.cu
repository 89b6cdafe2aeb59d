// The field's forward pass: positions -> hash encode -> density MLP -> clamp + SH -> colour MLP -> (sigma, logit, rgb),
// optionally with the MSE loss and its gradient in the epilogue, in one launch.
//
// Replaces TinyMLPHashGrid::forward -> compute_SH_gather -> TinyMLP::forward (modules/NeRF/InstantNerf.cu:436-459) and,
// with the loss, launchMSELossGrad (modules/TinyMLP/optimizerKernel.cu:169-224).  Same fp16 rounding points and the same
// order of every sum as the kernel-by-kernel sequence.
//
// What bounds it: the rate of 128-byte lines the gathers ask the L2 for, about one per clock and SM (see the lane pairs in
// hashgrid_core.cuh): 60.7 M of them for 2^20 scattered samples are 0.215 ms of its 0.304.  A WARP takes 32 samples from positions
// to colours by itself - encode, then two 16-row tensor-core tiles per weight fragment - and goes on to its next 32, without a
// barrier between the phases of different warps; weights are staged once per CTA.  2^20 samples, T = 2^19: 0.366 -> 0.304 ms
// (0.385 -> 0.322 with the loss) against a CTA-wide 128-row tile with the plain gathers; 0.252 without the networks.
// Shared memory is spent sparingly: what it takes is missing in L1, which holds the lines in flight - with 28 KB of L1 left the
// same kernel takes 0.47 ms at T = 2^19 and 1.25 ms instead of 0.51 at T = 2^22, where lines come from HBM.  The first two dense
// levels are copied to shared memory for their random reads only where a line's latency is the L2's.
// Tried and not faster, all between 0.30 and 0.33 ms: warps that only gather feeding warps that only run the networks through
// mbarriers (weights in shared memory or resident in registers), the networks of one tile cut into pieces between the gathers of
// the next, double-buffered gathers, 12 to 32 warps.
#include <algorithm>
#include <atomic>

#include "field_core.cuh"

namespace nb {

extern std::atomic<uint64_t> g_launch_count;

namespace fwd {

constexpr int WARPS = 16, THREADS = WARPS * 32;   // 128 registers each
constexpr int SHARERS = 4;                  // warps that share a tile when tiles are few
constexpr int ROWS = 32;                    // samples of a tile
constexpr int TILE = ROWS * (32 + 16);      // halves of a tile: [32][32] encoding, then [32][16] SH
constexpr int STAGE_CAP = 80 * 1024;        // bytes of dense levels in shared memory

// Halves from the start of a tile to 8-half chunk c of row r.  Rows of 64 and 32 bytes without padding - shared memory is taken
// from L1, which holds the lines in flight - with the chunks of a row exchanged so that ldmatrix meets no bank twice.
__device__ __forceinline__ int enc_chunk(int r, int c) { return r * 32 + ((c ^ (r >> 1)) & 3) * 8; }
__device__ __forceinline__ int sh_chunk(int r, int c) { return ROWS * 32 + r * 16 + ((c ^ (r >> 2)) & 1) * 8; }

struct Outputs {
    __half* enc;      // nullable
    float* sigma;     // nullable
    float* logit;     // nullable
    float* rgb;
    int rgb_stride;
};

struct Work {
    int staged;       // leading dense levels in shared memory (even)
};

template <class DS, class CS>
constexpr size_t smem_bytes() {
    return (size_t)(DS::SW_TOTAL + CS::SW_TOTAL) * 2 + (size_t)(DS::B_TOTAL + CS::B_TOTAL) * 4 + (size_t)WARPS * TILE * 2;
}

// Waits for the warps of a slot: the warp itself, or the SHARERS warps of group `group`.
template <bool SHARED>
__device__ __forceinline__ void slot_sync(int group) {
    if constexpr (SHARED) asm volatile("bar.sync %0, %1;\n" ::"r"(1 + group), "n"(SHARERS * 32) : "memory");
    else __syncwarp();
}

// The leading dense levels into shared memory (the caller waits).
template <int COUNT>
__device__ __forceinline__ void stage_levels(const GridParams& gp, const uint32_t* __restrict__ table2, uint32_t* s_stage, int staged, int tid) {
    uint32_t base = 0;
    for (int l = 0; l < staged; l++) {
        const int w = __float2int_rd(gp.scales[l]) + 1, quads = (w * w * w + 3) >> 2;   // the table's level is longer than its dense grid
        for (int i = tid; i < quads; i += COUNT) cp_async16(s_stage + base + 4 * i, table2 + (size_t)l * gp.ls + 4 * i, true);
        base += 4 * quads;
    }
}

// Levels [begin, end) of this lane's sample into its row of the tile, two at a time (16 gathers in flight per lane).
template <bool OWN>
__device__ __forceinline__ void encode_row(const GridParams& gp, const uint32_t* __restrict__ table2, const uint32_t* s_stage, int staged, int begin,
                                           int end, const PairPos& q, bool has, int odd, __half* tile, int r) {
    uint32_t base = 0;   // first entry of the next staged level
#pragma unroll 1
    for (int l = begin; l < staged; l += 2) {
        const float2 scale = make_float2(gp.scales[l], gp.scales[l + 1]);
        uint32_t fa[8], fb[8];
        const int wa = __float2int_rd(scale.x) + 1, wb = __float2int_rd(scale.y) + 1;
        staged_level(s_stage + base, scale.x, q, odd, fa);
        base += (wa * wa * wa + 3) & ~3;
        staged_level(s_stage + base, scale.y, q, odd, fb);
        base += (wb * wb * wb + 3) & ~3;
        const uint2 e = blend_two(fa, fb, q, scale);
        *reinterpret_cast<uint2*>(tile + enc_chunk(r, l >> 2) + 2 * (l & 3)) = has ? e : make_uint2(0u, 0u);
    }
#pragma unroll 1
    for (int l = max(begin, staged); l < end; l += 2) {
        const uint2 e = OWN ? own_encode_two(gp, table2, l, l + 1, q, odd) : pair_encode_two(gp, table2, l, l + 1, q, odd);
        *reinterpret_cast<uint2*>(tile + enc_chunk(r, l >> 2) + 2 * (l & 3)) = has ? e : make_uint2(0u, 0u);
    }
}

// ... taken from the pieces the levels' owners delivered.
__device__ __forceinline__ void pieces_row(const FieldPiecesIO& pio, int64_t i, int begin, int end, bool has, __half* tile, int r) {
    const int own = 16 / pio.ranks;
    for (int l0 = begin; l0 < end; l0 += 4) {
        uint32_t e[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const int l = l0 + k;
            e[k] = has ? __ldg(pio.pieces + ((int64_t)(l % pio.ranks) * own + l / pio.ranks) * pio.cap + i) : 0u;
        }
        *reinterpret_cast<uint4*>(tile + enc_chunk(r, l0 >> 2)) = make_uint4(e[0], e[1], e[2], e[3]);
    }
}

// 16 columns (block q) of a ReLU layer on `in`, consumed at once as k chunk q of the narrow layer behind it.
template <int K, int H, int NT, int MT>
__device__ __forceinline__ void hidden_into(const uint32_t (&in)[MT][K / 16][4], const __half* w0, const float* b0, const __half* w1, int q, int lane,
                                            float (&acc)[NT][MT][4]) {
    float c[2][MT][4];
    tile_accumulate<K, 2, MT>(in, w0, b0, 16 * q, lane, c);
    uint32_t b[NT][2];
#pragma unroll
    for (int j = 0; j < NT; j++) ldmatrix_x2(b[j][0], b[j][1], &w1[(8 * j + (lane & 7)) * (H + 8) + 16 * q + ((lane >> 3) & 1) * 8]);
#pragma unroll
    for (int m = 0; m < MT; m++) {
        const uint32_t h[4] = {relu_half2(c[0][m][0], c[0][m][1]), relu_half2(c[0][m][2], c[0][m][3]), relu_half2(c[1][m][0], c[1][m][1]),
                               relu_half2(c[1][m][2], c[1][m][3])};
#pragma unroll
        for (int j = 0; j < NT; j++) mma_16816(acc[j][m], h, b[j][0], b[j][1]);
    }
}
template <int NT, int MT>
__device__ __forceinline__ void add_bias(const float* b, int lane, float (&acc)[NT][MT][4]) {
#pragma unroll
    for (int j = 0; j < NT; j++) {
        const float2 bb = *reinterpret_cast<const float2*>(&b[8 * j + 2 * (lane & 3)]);
#pragma unroll
        for (int m = 0; m < MT; m++) { add_f2(acc[j][m][0], acc[j][m][1], bb); add_f2(acc[j][m][2], acc[j][m][3], bb); }
    }
}

struct NetWeights {
    const __half *Wd, *Wc;   // shared memory
    const float *bd, *bc;
};

// Both networks for MT * 16 rows of a tile from row r0 on; the tile is that of `left` samples from row0 on.
template <class DS, class CS, bool WITH_LOSS, bool ORDERED, int MT>
__device__ __forceinline__ void networks(const NetWeights& w, const FieldIO& io, const Outputs& out, const FieldLossIO& lio, const __half* tile, int r0,
                                         int64_t row0, uint32_t sample, int left, int lane, float& sq) {
    constexpr int H = DS::H;
    const int g = lane >> 2, t = lane & 3, col = 2 * t, lq = lane >> 3, lr = lane & 7;
    // where the results of row r go: by row, or by the sample that lane r of the tile holds
    auto place = [&](int r) -> int64_t {
        if constexpr (ORDERED) return __shfl_sync(0xffffffffu, sample, r);
        else return row0 + r;
    };
    uint32_t target[MT][2];
    if constexpr (WITH_LOSS) {
        // targets early: they arrive while the networks run
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = r0 + m * 16 + g + 8 * h;
                target[m][h] = r < left ? __ldg(reinterpret_cast<const uint32_t*>(lio.target + row0 * 8 + (r * 8 + col))) : 0u;
            }
    }
    uint32_t a[MT][2][4];
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int kc = 0; kc < 2; kc++) ldmatrix_x4(a[m][kc], tile + enc_chunk(r0 + m * 16 + lr + (lq & 1) * 8, 2 * kc + (lq >> 1)));
    {
        float acc[2][MT][4] = {};
#pragma unroll
        for (int q = 0; q < H / 16; q++) hidden_into<32, H, 2, MT>(a, w.Wd + DS::sw_off(0), w.bd + DS::b_off(0), w.Wd + DS::sw_off(1), q, lane, acc);
        add_bias<2, MT>(w.bd + DS::b_off(1), lane, acc);
#pragma unroll
        for (int m = 0; m < MT; m++) {
            // the colour network's input: clamped logits, SH
            a[m][0][0] = pack_half2(sanitize_logit_f(acc[0][m][0]), sanitize_logit_f(acc[0][m][1]));
            a[m][0][1] = pack_half2(sanitize_logit_f(acc[0][m][2]), sanitize_logit_f(acc[0][m][3]));
            a[m][0][2] = pack_half2(sanitize_logit_f(acc[1][m][0]), sanitize_logit_f(acc[1][m][1]));
            a[m][0][3] = pack_half2(sanitize_logit_f(acc[1][m][2]), sanitize_logit_f(acc[1][m][3]));
            ldmatrix_x4(a[m][1], tile + sh_chunk(r0 + m * 16 + lr + (lq & 1) * 8, lq >> 1));
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = r0 + m * 16 + g + 8 * h;
                const int64_t at = place(r);
                const float raw = acc[0][m][2 * h];
                if (t == 0 && r < left) {
                    if (out.logit) out.logit[at] = raw;
                    if (out.sigma) out.sigma[at] = expf(fminf(sanitize_logit_f(raw) - io.density_bias, 8.0f));
                }
            }
        }
    }
    float fin[1][MT][4] = {};
    if constexpr (CS::NL == 3) {
        uint32_t h1[MT][H / 16][4];
        tile_hidden<32, H, MT>(a, w.Wc + CS::sw_off(0), w.bc + CS::b_off(0), lane, h1);
#pragma unroll
        for (int q = 0; q < H / 16; q++) hidden_into<H, H, 1, MT>(h1, w.Wc + CS::sw_off(1), w.bc + CS::b_off(1), w.Wc + CS::sw_off(2), q, lane, fin);
    } else {
#pragma unroll
        for (int q = 0; q < H / 16; q++) hidden_into<32, H, 1, MT>(a, w.Wc + CS::sw_off(0), w.bc + CS::b_off(0), w.Wc + CS::sw_off(1), q, lane, fin);
    }
    add_bias<1, MT>(w.bc + CS::b_off(CS::NL - 1), lane, fin);
#pragma unroll
    for (int m = 0; m < MT; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = r0 + m * 16 + g + 8 * h;
            const int64_t at = place(r);
            if (r >= left) continue;
            const float px = 1.0f / (1.0f + expf(-fin[0][m][2 * h])), py = 1.0f / (1.0f + expf(-fin[0][m][2 * h + 1]));
            if (col < out.rgb_stride) *reinterpret_cast<float2*>(out.rgb + at * out.rgb_stride + col) = make_float2(px, py);
            if constexpr (WITH_LOSS) {
                // the arithmetic of mse_loss_grad_kernel (optim.cu) on the colour still in registers
                const float2 tg = unpack_half2(target[m][h]);
                const float dxv = (col < 3) ? (px - tg.x) : 0.0f;
                const float dyv = (col + 1 < 3) ? (py - tg.y) : 0.0f;
                sq += (dxv * dxv) + (dyv * dyv);
                float gx = dxv * lio.grad_scale, gy = dyv * lio.grad_scale;
                gx *= px * (1.0f - px);
                gy *= py * (1.0f - py);
                *reinterpret_cast<__half2*>(lio.grad + row0 * 8 + (r * 8 + col)) = __floats2half2_rn(gx, gy);
            }
        }
}

template <class DS, class CS, bool WITH_LOSS, bool FROM_PIECES, bool ORDERED, bool SHARED>
__global__ void __launch_bounds__(THREADS, 1) field_forward_kernel(const __grid_constant__ GridParams gp, FieldIO io, const Outputs out, const Work work,
                                                                   const FieldLossIO lio, const FieldPiecesIO pio) {
    after_previous();
    static_assert(DS::K0 == 32 && DS::NL == 2 && DS::OUT == 16 && CS::K0 == 32 && CS::OUT == 8 && (CS::NL == 2 || CS::NL == 3), "field shapes");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* sWd = reinterpret_cast<__half*>(smem_raw);
    __half* sWc = sWd + DS::SW_TOTAL;
    float* sBd = reinterpret_cast<float*>(sWc + CS::SW_TOTAL);
    float* sBc = sBd + DS::B_TOTAL;
    __half* tiles = reinterpret_cast<__half*>(sBc + CS::B_TOTAL);
    uint32_t* s_stage = reinterpret_cast<uint32_t*>(tiles + WARPS * TILE);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, odd = lane & 1;

    const int64_t n_max = io.n;
    if (io.count != nullptr) {
        // the launch covers an upper bound of the samples; a kernel before this one left the count
        const int64_t counted = (int64_t)__ldg(io.count);
        if (counted < io.n) io.n = counted;
    }
    const int64_t ntiles = (io.n + ROWS - 1) / ROWS;
    // consecutive tiles for a CTA: neighbouring samples meet in one SM's L1
    const int64_t chunk = (ntiles + gridDim.x - 1) / gridDim.x, first = (int64_t)blockIdx.x * chunk, last = min(ntiles, first + chunk);
    if (first >= last) return;
    load_weights_to_smem<DS, THREADS>(io.Wd, io.bd, sWd, sBd, tid);
    load_weights_to_smem<CS, THREADS>(io.Wc, io.bc, sWc, sBc, tid);
    if constexpr (!FROM_PIECES) {
        stage_levels<THREADS>(gp, io.table2, s_stage, work.staged, tid);
    }
    cp_async_commit();
    // Every thread meets the barrier below once: before its first tile where levels are staged, else between its first tile's
    // encoding and networks, so that the weights arrive under the first gathers.
    bool staged_in = false;
    auto weights_ready = [&]() {
        if (staged_in) return;
        cp_async_wait_all();
        __syncthreads();
        staged_in = true;
    };
    if (!SHARED && work.staged > 0) weights_ready();

    // A slot is a warp, or SHARERS warps that share a tile: a quarter of the levels each, then half of the rows for two of them.
    constexpr int step = SHARED ? SHARERS : 1;
    const int part = warp % step, group = warp / step;
    const int begin = SHARED ? 4 * part : 0, end = SHARED ? begin + 4 : 16;
    const NetWeights w{sWd, sWc, sBd, sBc};
    __half* tile = tiles + group * TILE;
    float sq = 0.f;   // WITH_LOSS: this thread's share of the squared differences
    for (int64_t wt = first + group; wt < last; wt += WARPS / step) {
        const int64_t row0 = wt * ROWS, mine = row0 + lane;
        const int left = (int)min(io.n - row0, (int64_t)ROWS);
        const bool has = lane < left;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        int64_t sample = mine;
        if (ORDERED && has) sample = min((int64_t)__ldg(io.order + mine), n_max - 1);   // never past the arrays, whatever the order says
        if (!FROM_PIECES && has) p = ld_nc_f4(io.pos4 + sample * 4);
        float dx, dy, dz;
        {
            const int64_t i = has ? sample : io.n - 1;
            const float* dp = io.dirs3 + 3 * (io.ray_idx ? (int64_t)io.ray_idx[i + io.ray_idx_offset] : i);
            dx = dp[0]; dy = dp[1]; dz = dp[2];
        }
        if constexpr (FROM_PIECES) {
            pieces_row(pio, mine, begin, end, has, tile, lane);
        } else {
            PairPos q;
            pair_positions(p.x, p.y, p.z, odd, q);
            encode_row<ORDERED>(gp, io.table2, s_stage, SHARED ? 0 : work.staged, begin, end, q, has, odd, tile, lane);
        }
        if (begin == 0) {
            float sh[16];
            sh16(dx, dy, dz, sh);
            *reinterpret_cast<uint4*>(tile + sh_chunk(lane, 0)) =
                make_uint4(pack_half2(sh[0], sh[1]), pack_half2(sh[2], sh[3]), pack_half2(sh[4], sh[5]), pack_half2(sh[6], sh[7]));
            *reinterpret_cast<uint4*>(tile + sh_chunk(lane, 1)) =
                make_uint4(pack_half2(sh[8], sh[9]), pack_half2(sh[10], sh[11]), pack_half2(sh[12], sh[13]), pack_half2(sh[14], sh[15]));
        }
        if (SHARED && out.enc != nullptr && has)
            st_cs_v4(out.enc + mine * 32 + 2 * begin, *reinterpret_cast<const uint4*>(tile + enc_chunk(lane, begin >> 2)));
        weights_ready();
        slot_sync<SHARED>(group);
        if constexpr (SHARED) {
            if (part < 2) networks<DS, CS, WITH_LOSS, ORDERED, 1>(w, io, out, lio, tile, 16 * part, row0, (uint32_t)sample, left, lane, sq);
        } else {
            if (out.enc != nullptr) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const int c = lane + 32 * i, r = c >> 2, c8 = c & 3;
                    if (r < left) st_cs_v4(out.enc + row0 * 32 + 8 * c, *reinterpret_cast<const uint4*>(tile + enc_chunk(r, c8)));
                }
            }
            networks<DS, CS, WITH_LOSS, ORDERED, 2>(w, io, out, lio, tile, 0, row0, (uint32_t)sample, left, lane, sq);
        }
        slot_sync<SHARED>(group);   // the tile is free again
    }
    weights_ready();   // a warp without a tile
    if constexpr (WITH_LOSS) {
        // one addition per CTA to the total; the tiles are free by now, their first words carry the warps' sums
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
        __syncthreads();
        float* warp_sums = reinterpret_cast<float*>(tiles);
        if (lane == 0) warp_sums[warp] = sq;
        __syncthreads();
        if (tid == 0 && lio.total != nullptr) {
            float total = 0.f;
            for (int k = 0; k < WARPS; k++) total += warp_sums[k];
            atomicAdd(lio.total, total);
        }
    }
}

// ---- density of occupancy samples -------------------------------------------------------------------------------------------
// The same path up to the density, of which only the first output matters, and then the largest density per cell (a sample's cell
// is its fourth component): what nb_grid_mlp_forward and nb_occ_update_tmp_grid do with rows of 16 floats between them.
// Against the two kernels, of which the first took a CTA per 128 samples (us): 2^21 samples cell by cell 323 -> 275 at T = 2^19 and
// 352 -> 319 at 2^22, 2^20 in random cells 291 -> 242 and 377 -> 320.  16 to 32 warps, and each lane gathering for itself where
// the samples come cell by cell, lie within 10 us of that.
struct CellIO {
    const float* pos4;
    const uint32_t* table2;
    const __half* Wd;
    const float* bd;
    int64_t n;
    float density_bias;
    float* cells;
};

constexpr int CELL_WARPS = 20, CELL_THREADS = CELL_WARPS * 32;
constexpr int CELL_TILE = ROWS * 32;   // halves of a tile

template <class DS>
constexpr size_t cell_smem_bytes() { return (size_t)DS::SW_TOTAL * 2 + (size_t)DS::B_TOTAL * 4 + (size_t)CELL_WARPS * CELL_TILE * 2; }

template <class DS>
__global__ void __launch_bounds__(CELL_THREADS, 1) cell_density_kernel(const __grid_constant__ GridParams gp, const CellIO io, const Work work) {
    after_previous();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __half* sWd = reinterpret_cast<__half*>(smem_raw);
    float* sBd = reinterpret_cast<float*>(sWd + DS::SW_TOTAL);
    __half* tiles = reinterpret_cast<__half*>(sBd + DS::B_TOTAL);
    uint32_t* s_stage = reinterpret_cast<uint32_t*>(tiles + CELL_WARPS * CELL_TILE);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, odd = lane & 1, g = lane >> 2, t = lane & 3, lq = lane >> 3, lr = lane & 7;
    const int64_t ntiles = (io.n + ROWS - 1) / ROWS;
    const int64_t chunk = (ntiles + gridDim.x - 1) / gridDim.x, first = (int64_t)blockIdx.x * chunk, last = min(ntiles, first + chunk);
    if (first >= last) return;
    load_weights_to_smem<DS, CELL_THREADS>(io.Wd, io.bd, sWd, sBd, tid);
    stage_levels<CELL_THREADS>(gp, io.table2, s_stage, work.staged, tid);
    cp_async_commit();
    cp_async_wait_all();
    __syncthreads();
    __half* tile = tiles + warp * CELL_TILE;
    for (int64_t wt = first + warp; wt < last; wt += CELL_WARPS) {
        const int64_t mine = wt * ROWS + lane;
        const bool has = mine < io.n;
        float4 p = make_float4(0.f, 0.f, 0.f, 0.f);
        if (has) p = ld_nc_f4(io.pos4 + mine * 4);
        PairPos q;
        pair_positions(p.x, p.y, p.z, odd, q);
        encode_row<false>(gp, io.table2, s_stage, work.staged, 0, 16, q, has, odd, tile, lane);
        __syncwarp();
        uint32_t a[2][2][4];
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int kc = 0; kc < 2; kc++) ldmatrix_x4(a[m][kc], tile + enc_chunk(m * 16 + lr + (lq & 1) * 8, 2 * kc + (lq >> 1)));
        float acc[2][2][4] = {};
#pragma unroll
        for (int k = 0; k < DS::H / 16; k++) hidden_into<32, DS::H, 2, 2>(a, sWd + DS::sw_off(0), sBd + DS::b_off(0), sWd + DS::sw_off(1), k, lane, acc);
        add_bias<2, 2>(sBd + DS::b_off(1), lane, acc);
#pragma unroll
        for (int m = 0; m < 2; m++)
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int r = m * 16 + g + 8 * h;
                const int cell = __shfl_sync(0xffffffffu, __float_as_int(p.w), r);
                const float sigma = expf(fminf(acc[0][m][2 * h] - io.density_bias, 8.0f));
                // never negative: an integer maximum of the bits orders it
                if (t == 0 && wt * ROWS + r < io.n) atomicMax(reinterpret_cast<int*>(io.cells) + cell, __float_as_int(sigma));
            }
        __syncwarp();   // the tile is free again
    }
}

}  // namespace fwd

// Leading dense levels in shared memory, two at a time, as many as fit: not for tables beyond the L2 (see the top of the
// file), and not where copying them would cost about as much as gathering them.  16-byte copies need the alignment.
// Returns their bytes.
static size_t plan_staged_levels(const GridParams& gp, const uint32_t* table2, int64_t tiles_per_cta, fwd::Work& work) {
    size_t stage = 0;
    if (tiles_per_cta < 3 * fwd::WARPS || (int64_t)gp.L * gp.T * 4 > (64 << 20) || (reinterpret_cast<uintptr_t>(table2) & 15u) != 0 || gp.T % 4 != 0) return 0;
    while (work.staged + 2 <= gp.dls && gp.scales[work.staged + 1] < 64.0f) {
        size_t bytes = 0;
        for (int l = work.staged; l < work.staged + 2; l++) {
            const size_t w = (size_t)gp.scales[l] + 1;
            bytes += (w * w * w + 3) / 4 * 16;
        }
        if (stage + bytes > (size_t)fwd::STAGE_CAP) break;
        stage += bytes;
        work.staged += 2;
    }
    return stage;
}

int launch_cell_density(const GridParams& gp, const float* pos4, const void* table_h, const void* Wd_h, const float* bd, int64_t n, float density_bias, float* cells,
                        cudaStream_t st) {
    const fwd::CellIO io{pos4, (const uint32_t*)table_h, (const __half*)Wd_h, bd, n, density_bias, cells};
    const int64_t ntiles = (n + fwd::ROWS - 1) / fwd::ROWS, grid = std::min<int64_t>(ntiles, nb_num_sms());
    fwd::Work work{};
    const size_t stage = plan_staged_levels(gp, io.table2, (ntiles + grid - 1) / grid, work), smem = fwd::cell_smem_bytes<DensityNet>();
    auto kern = fwd::cell_density_kernel<DensityNet>;
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem + fwd::STAGE_CAP)));
    launch_after_with_l1(smem + stage + 1024, kern, (unsigned)grid, fwd::CELL_THREADS, smem + stage, st, gp, io, work);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

template <class CS, bool WITH_LOSS, bool FROM_PIECES, bool ORDERED = false>
static int launch_forward_as(const GridParams& gp, const FieldIO& io, const fwd::Outputs& out, const FieldLossIO& lio, const FieldPiecesIO& pio,
                             cudaStream_t st) {
    const int64_t ntiles = (io.n + fwd::ROWS - 1) / fwd::ROWS;
    const int64_t grid = std::min<int64_t>(ntiles, nb_num_sms());
    fwd::Work work{};
    const int64_t chunk = (ntiles + grid - 1) / grid;
    // Few tiles: SHARERS warps share one, which divides the latency of its gathers.  A round of shared tiles takes about 0.35
    // of a round of whole ones and does a quarter of it, so it pays while rounding up to whole rounds is what counts.
    const int64_t whole = fwd::WARPS, quarter = fwd::WARPS / fwd::SHARERS;
    const bool shared = 7 * ((chunk + quarter - 1) / quarter) < 20 * ((chunk + whole - 1) / whole);
    const size_t stage = !FROM_PIECES && !shared && io.count == nullptr ? plan_staged_levels(gp, io.table2, chunk, work) : 0;
    const size_t smem = fwd::smem_bytes<DensityNet, CS>();
    auto kern = shared ? fwd::field_forward_kernel<DensityNet, CS, WITH_LOSS, FROM_PIECES, ORDERED, true> : fwd::field_forward_kernel<DensityNet, CS, WITH_LOSS, FROM_PIECES, ORDERED, false>;
    // always the cap: the attribute belongs to the function, and launches of other host threads may stage more
    NB_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(smem + fwd::STAGE_CAP)));
    // The gathers want L1: the launch names the shared memory it needs (see launch_after_with_l1).  In rounds the kernels between
    // have that division already.  Depth-ordered frames come in batches on two streams, where blocks that wait on the chip are in the
    // other stream's way.
    if (shared || io.count != nullptr) launch_after(kern, (unsigned)grid, fwd::THREADS, smem + stage, st, gp, io, out, work, lio, pio);
    else if (!ORDERED) launch_after_with_l1(smem + stage + 1024, kern, (unsigned)grid, fwd::THREADS, smem + stage, st, gp, io, out, work, lio, pio);
    else kern<<<(unsigned)grid, fwd::THREADS, smem + stage, st>>>(gp, io, out, work, lio, pio);
    NB_CHECK_LAUNCH();
    g_launch_count++;
    return NB_OK;
}

template <class CS>
static int launch_forward_color(const GridParams& gp, const FieldIO& io, const fwd::Outputs& out, const FieldLossIO* loss, const FieldPiecesIO* pieces,
                                cudaStream_t st) {
    if (loss != nullptr) return launch_forward_as<CS, true, false>(gp, io, out, *loss, FieldPiecesIO{}, st);
    if (pieces != nullptr) return launch_forward_as<CS, false, true>(gp, io, out, FieldLossIO{}, *pieces, st);
    if (io.order != nullptr) return launch_forward_as<CS, false, false, true>(gp, io, out, FieldLossIO{}, FieldPiecesIO{}, st);
    return launch_forward_as<CS, false, false>(gp, io, out, FieldLossIO{}, FieldPiecesIO{}, st);
}

int launch_field_forward(const GridParams& gp, const FieldIO& io, int color_layers, void* d_enc_save_h, float* d_sigma, float* d_logit0, float* d_rgb,
                         int rgb_stride, const FieldLossIO* loss, const FieldPiecesIO* pieces, cudaStream_t st) {
    const fwd::Outputs out{(__half*)d_enc_save_h, d_sigma, d_logit0, d_rgb, rgb_stride};
    return color_layers == 3 ? launch_forward_color<ColorNet>(gp, io, out, loss, pieces, st) : launch_forward_color<ColorNet2>(gp, io, out, loss, pieces, st);
}

}  // namespace nb
