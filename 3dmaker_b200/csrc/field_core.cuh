// What the kernels of the whole field (field_forward.cu, field_fused.cu, field_backward_tc.cu) share: their inputs, the
// spherical harmonics of a ray's direction (nerf_glue.cu takes them from here too) and the colour network's input.
#pragma once

#include "field_backward_tc.cuh"
#include "hashgrid_core.cuh"

namespace nb {

// The 16 SH coefficients of a direction (bands 0..3, constants of modules/NeRF/otherKernels.cu:182-200).
__device__ __forceinline__ void sh16(float x, float y, float z, float (&sh)[16]) {
    const float x2 = x * x, y2 = y * y, z2 = z * z;
    sh[0] = 0.28209479f;
    sh[1] = -0.48860251f * y;
    sh[2] = 0.48860251f * z;
    sh[3] = -0.48860251f * x;
    sh[4] = 1.09254843f * x * y;
    sh[5] = -1.09254843f * y * z;
    sh[6] = 0.31539156f * (3.0f * z2 - 1.0f);
    sh[7] = -1.09254843f * x * z;
    sh[8] = 0.54627421f * (x2 - y2);
    sh[9] = -0.59004359f * y * (3.0f * x2 - y2);
    sh[10] = 2.89061144f * x * y * z;
    sh[11] = -0.45704580f * y * (5.0f * z2 - 1.0f);
    sh[12] = 0.37317633f * z * (5.0f * z2 - 3.0f);
    sh[13] = -0.45704580f * x * (5.0f * z2 - 1.0f);
    sh[14] = 1.44530572f * z * (x2 - y2);
    sh[15] = -0.59004359f * x * (x2 - 3.0f * y2);
}

__device__ __forceinline__ float sanitize_logit_f(float v) {
    v = fmaxf(-64.0f, fminf(64.0f, v));
    return (v != v) ? 0.0f : v;
}

// The four SH coefficients that lane column-pair t needs: indices 2t, 2t+1 (lo) and 8+2t, 9+2t (hi).
__device__ __forceinline__ void sh_quad(float x, float y, float z, int t, float& lo0, float& lo1, float& hi0, float& hi1) {
    float sh[16];
    sh16(x, y, z, sh);
    lo0 = t == 0 ? sh[0] : (t == 1 ? sh[2] : (t == 2 ? sh[4] : sh[6]));
    lo1 = t == 0 ? sh[1] : (t == 1 ? sh[3] : (t == 2 ? sh[5] : sh[7]));
    hi0 = t == 0 ? sh[8] : (t == 1 ? sh[10] : (t == 2 ? sh[12] : sh[14]));
    hi1 = t == 0 ? sh[9] : (t == 1 ? sh[11] : (t == 2 ? sh[13] : sh[15]));
}

struct FieldIO {
    const float* pos4;        // [n] float4
    const uint32_t* table2;   // fp16 feature pairs
    const float* dirs3;       // float3 per ray
    const uint32_t* ray_idx;  // sample -> ray (nullable: sample i uses direction i)
    int64_t ray_idx_offset;
    const __half* Wd; const float* bd;  // density network
    const __half* Wc; const float* bc;  // colour network
    int64_t n;
    float density_bias;
    const uint32_t* count;  // nullable: sample count known only on the device (at most n)
    const uint32_t* order;    // nullable (inference): place k of the kernel's order is sample order[k]; outputs stay by sample
};

// Colour-network input fragments of the warp's 16 rows from the density output fragments (16 logits) and the
// ray directions: k chunk 0 = clamped logits, k chunk 1 = SH.  Also hands back sigma / raw logit of the rows
// (valid in lanes with t == 0).
// perm (nullable): row r of the tile order is sample perm[r].
__device__ __forceinline__ void build_color_input(const float (&dout)[2][4], const FieldIO& io, int64_t row0, int lane, uint32_t (&a)[2][4],
                                                  float& raw0, float& raw1, const uint32_t* __restrict__ perm = nullptr) {
    const int g = lane >> 2, t = lane & 3;
    raw0 = dout[0][0]; raw1 = dout[0][2];  // column 0 of rows g and g+8 (lanes with t == 0)
    a[0][0] = pack_half2(sanitize_logit_f(dout[0][0]), sanitize_logit_f(dout[0][1]));
    a[0][1] = pack_half2(sanitize_logit_f(dout[0][2]), sanitize_logit_f(dout[0][3]));
    a[0][2] = pack_half2(sanitize_logit_f(dout[1][0]), sanitize_logit_f(dout[1][1]));
    a[0][3] = pack_half2(sanitize_logit_f(dout[1][2]), sanitize_logit_f(dout[1][3]));
    float lo0, lo1, hi0, hi1;
#pragma unroll
    for (int h = 0; h < 2; h++) {
        int64_t r = row0 + g + 8 * h;
        if (r >= io.n) r = io.n - 1;
        if (perm != nullptr) r = (int64_t)perm[r];
        int64_t ray = io.ray_idx ? (int64_t)io.ray_idx[r + io.ray_idx_offset] : r;
        const float* dp = io.dirs3 + 3 * ray;
        sh_quad(dp[0], dp[1], dp[2], t, lo0, lo1, hi0, hi1);
        a[1][h] = pack_half2(lo0, lo1);
        a[1][2 + h] = pack_half2(hi0, hi1);
    }
}

// MSE loss against per-sample target colours, taken in the forward's epilogue (the arithmetic of mse_loss_grad_kernel,
// optim.cu, on the colour the kernel has in registers): grad[n][8] fp16 = dL/d(colour pre-activation) x loss scale,
// total += sum of squared differences.
struct FieldLossIO {
    const __half* target;   // [n][8] fp16, columns >= 3 ignored
    __half* grad;           // [n][8] fp16
    float* total;           // nullable
    float grad_scale;       // 2 / (n * 3) * loss scale
};

// The encoding of this rank's samples as the level owners delivered it (level_partition.cu): piece q holds the levels
// q, q + ranks, ... of every sample, level-major, `cap` samples per level.
struct FieldPiecesIO {
    const uint32_t* pieces;
    int ranks;
    int64_t cap;
};

using DensityNet = MlpShape<32, 64, 16, 2>;
using ColorNet = MlpShape<32, 64, 8, 3>;
using ColorNet2 = MlpShape<32, 64, 8, 2>;   // NerfOptions' default

// Host side of the forward kernel (field_forward.cu): loss and pieces are null where the launch has none.
int launch_field_forward(const GridParams& gp, const FieldIO& io, int color_layers, void* d_enc_save_h, float* d_sigma, float* d_logit0, float* d_rgb, int rgb_stride,
                         const FieldLossIO* loss, const FieldPiecesIO* pieces, cudaStream_t st);
int launch_cell_density(const GridParams& gp, const float* pos4, const void* table_h, const void* Wd_h, const float* bd, int64_t n, float density_bias, float* cells,
                        cudaStream_t st);

}  // namespace nb
