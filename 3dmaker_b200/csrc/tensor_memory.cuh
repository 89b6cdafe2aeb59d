// tcgen05 building blocks shared by the kernels that keep operands in core-matrix tiles and accumulators in tensor memory:
// descriptors, MMA issue, tensor-memory loads, GEMMs over 128-row tiles and the row helpers of their epilogues.
#pragma once

#include "common.cuh"

namespace nb {
namespace tc {

constexpr int ROWS = 128;      // rows of a tile = tensor-memory lanes

// A tile is [rows][cols] fp16 in the tensor core's core-matrix order (8 rows x 16 bytes per core, no swizzle).
__host__ __device__ constexpr uint32_t tile_bytes(int rows, int cols) { return (uint32_t)rows * cols * 2; }
// byte offset of element (row, col) in a tile with `cols` columns: cores of one 8-row block are contiguous
__host__ __device__ constexpr uint32_t core_off(int row, int col, int cols) {
    return (uint32_t)(row >> 3) * (cols >> 3) * 128 + (uint32_t)(col >> 3) * 128 + (uint32_t)(row & 7) * 16 + (uint32_t)(col & 7) * 2;
}

// ---- PTX wrappers -----------------------------------------------------------------------------------------------
// shared-memory matrix descriptor: no swizzle; lbo = byte step between cores along K, sbo = along M/N (K-major), or
// lbo = along K, sbo = along M/N for MN-major as well - what differs between the two views is which storage step is K
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3fffu) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) | ((uint64_t)((sbo >> 4) & 0x3fffu) << 32) | ((uint64_t)1 << 46);
}
// instruction descriptor: fp16 operands, fp32 accumulate
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, int a_mn_major, int b_mn_major) {
    return (1u << 4) | ((uint32_t)a_mn_major << 15) | ((uint32_t)b_mn_major << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// The lane of a warp that issues its MMAs and commits.  All lanes of a converged warp call.
__device__ __forceinline__ uint32_t elected_lane() {
    uint32_t lead;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}\n" : "=r"(lead));
    return lead;
}
// MMAs are issued by WHOLE WARPS, of which the lane with lead != 0 does it: descriptors are then the same for the warp and live in
// uniform registers.  Issued from inside `if (thread == 0)` every one of them is carried over from ordinary registers: 46 cycles per MMA
// whatever its size, against 20 to 39 (M 64, N 8 to M 128, N 64), where what its operands take of shared memory's 128 bytes per clock
// begins to show (18 to 48 cycles).
__device__ __forceinline__ void umma_f16(uint32_t lead, uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %4, 0;\n\tsetp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d), "l"(da), "l"(db), "r"(idesc), "r"((uint32_t)accumulate), "r"(lead)
        : "memory");
}
__device__ __forceinline__ void umma_commit(uint32_t lead, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}\n" ::"r"(smem_u32(bar)), "r"(lead) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// 32 consecutive columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]),
          "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]),
          "=r"(r[31])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; i++) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]),
          "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; i++) v[i] = __uint_as_float(r[i]);
}

// ---- GEMM issue helpers (a whole warp calls) ------------------------------------------------------------------------------
// D[128][N] (+)= X[128][K] x W[N][K]^T : both operands K-major tiles with K columns
__device__ __forceinline__ void gemm_layer(uint32_t lead, uint32_t tmem_d, uint32_t x_addr, uint32_t w_addr, int K, int N) {
    const uint32_t idesc = instr_desc(ROWS, N, 0, 0);
    const uint32_t sbo = (uint32_t)(K >> 3) * 128;
#pragma unroll
    for (int k = 0; k < K; k += 16)
        umma_f16(lead, tmem_d, smem_desc(x_addr + (k >> 3) * 128, 128, sbo), smem_desc(w_addr + (k >> 3) * 128, 128, sbo), idesc, k > 0);
}
// D[128][N] = dZ[128][zcols(first KO)] x W[KO][wcols] restricted to the first N input columns: dZ K-major, W viewed MN-major
__device__ __forceinline__ void gemm_dinput(uint32_t lead, uint32_t tmem_d, uint32_t dz_addr, int zcols, int KO, uint32_t w_addr, int wcols, int N) {
    const uint32_t idesc = instr_desc(ROWS, N, 0, 1);
    const uint32_t dz_sbo = (uint32_t)(zcols >> 3) * 128, w_lbo = (uint32_t)(wcols >> 3) * 128;
#pragma unroll
    for (int k = 0; k < KO; k += 16)
        umma_f16(lead, tmem_d, smem_desc(dz_addr + (k >> 3) * 128, 128, dz_sbo), smem_desc(w_addr + (k >> 3) * w_lbo, w_lbo, 128), idesc, k > 0);
}
// D[64][N] += P[128][pcols(first 64)]^T x Q[128][qcols(first N)] : a reduction over the 128 rows, both operands MN-major
__device__ __forceinline__ void gemm_outer(uint32_t lead, uint32_t tmem_d, uint32_t p_addr, int pcols, uint32_t q_addr, int qcols, int N, bool accumulate) {
    const uint32_t idesc = instr_desc(64, N, 1, 1);
    const uint32_t p_lbo = (uint32_t)(pcols >> 3) * 128, q_lbo = (uint32_t)(qcols >> 3) * 128;
#pragma unroll
    for (int r = 0; r < ROWS; r += 16)
        umma_f16(lead, tmem_d, smem_desc(p_addr + (r >> 3) * p_lbo, p_lbo, 128), smem_desc(q_addr + (r >> 3) * q_lbo, q_lbo, 128), idesc, accumulate || r > 0);
}

// ---- row helpers (thread = row) -------------------------------------------------------------------------------------
// 8 fp32 -> 8 fp16 -> the 16-byte chunk (row, c8) of a tile with `cols` columns
__device__ __forceinline__ void store_chunk(unsigned char* tile, int row, int c8, int cols, const float* v) {
    uint4 q = make_uint4(pack_half2(v[0], v[1]), pack_half2(v[2], v[3]), pack_half2(v[4], v[5]), pack_half2(v[6], v[7]));
    *reinterpret_cast<uint4*>(tile + core_off(row, c8 * 8, cols)) = q;
}
// gradient chunk rounded to fp16, entries whose activation (same chunk of the layer's input tile) is not positive zeroed
__device__ __forceinline__ uint4 masked_chunk(const float* g, uint4 act) {
    const uint32_t a[4] = {act.x, act.y, act.z, act.w};
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; i++) o[i] = pack_half2(g[2 * i], g[2 * i + 1]) & __hgt2_mask(*reinterpret_cast<const __half2*>(&a[i]), __half2half2(__ushort_as_half(0)));
    return make_uint4(o[0], o[1], o[2], o[3]);
}

// Sums of 8 columns over the warp's 32 rows in 9 exchanges: halves of the columns change places until a lane has one; lane L ends
// with the whole sum of column column_of_lane(L).
__device__ __forceinline__ int column_of_lane(int lane) { return ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1); }
__device__ __forceinline__ float column_sums8(const float (&g)[8], int lane) {
    float a[4], b[2];
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = ((lane & 16) ? g[4 + i] : g[i]) + __shfl_xor_sync(0xffffffffu, (lane & 16) ? g[i] : g[4 + i], 16);
#pragma unroll
    for (int i = 0; i < 2; i++) b[i] = ((lane & 8) ? a[2 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, (lane & 8) ? a[i] : a[2 + i], 8);
    float s = ((lane & 4) ? b[1] : b[0]) + __shfl_xor_sync(0xffffffffu, (lane & 4) ? b[0] : b[1], 4);
    s += __shfl_xor_sync(0xffffffffu, s, 2);
    s += __shfl_xor_sync(0xffffffffu, s, 1);
    return s;
}

}  // namespace tc
}  // namespace nb
