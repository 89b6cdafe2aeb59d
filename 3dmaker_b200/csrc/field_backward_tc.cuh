// Argument block and launcher of the tensor-memory (tcgen05) backward kernel of the field, shared between
// field_backward_tc.cu (the kernel) and field_fused.cu (the nb_field_backward entry point that selects it).
#pragma once

#include <atomic>

#include "hashgrid_core.cuh"

namespace nb {
namespace tc {

// Copies of the leading dense levels' gradients, side by side: entries of level 0, then of level 1.  Large scattered batches queue up at
// their few entries (the L2 executes 79 G/s adds to 2^12 entries, 152 to 2^15, 200 to many); accumulated per CTA in shared memory by a kernel of
// their own they took 52 to 78 us of a step on 2^20 samples, the longer the more gradients have not rounded to zero.  Scattered with the
// other levels into copies they hide under the chain where it is the longer one: step 697 -> 675 us with a quarter of the gradients
// non-zero, 844 -> 824 with all; 2^19 samples 432 -> 420, 200000 263 -> 258.  2^16 samples take 160 without copies, 166 with.  A CTA reduces into copy
// blockIdx % count, so that the adds to their few entries do not queue up in the L2.
constexpr int COARSE_COPIES_MIN = 4, COARSE_COPIES_MAX = 16, COARSE_LEVELS = 2;
struct CoarseCopies {
    float* copies;
    int count;
    int levels;               // 0, or COARSE_LEVELS
    int first, entries;       // entries of level 0, of both; even
};

constexpr int ROWS_OF_TILE = 128;

struct BackwardArgs {
    // inputs
    const __half* enc;        // [n][32]
    const __half* dcolor;     // [n][8]
    const float* dsigma;      // [n], nullable
    const float* dirs3;
    const uint32_t* ray_idx;  // nullable
    int64_t ray_idx_offset;
    const __half *Wd, *Wc;    // density [64][32] [16][64]; colour [64][32] [64][64] [8][64]
    const float *bd, *bc;
    int color_layers;         // 3, or 2: without the [64][64] layer
    int64_t n;
    // outputs
    float *dWd, *dbd, *dWc, *dbc;
    __half* denc;             // leading denc_cols columns, rows denc_cols halves apart
    int denc_cols;
    const float* pos4;        // scatter
    float* table_grads;
    int scatter_begin;
    CoarseCopies coarse;      // levels [0, coarse.levels) are scattered into these; scatter_begin is 0 then
    const uint32_t* perm;     // nullable: row r of the tile order is sample perm[r] (everything is by sample, but enc in row order where enc_by_row)
    bool enc_by_row;
    uint32_t* live;           // nullable: room for a list of samples and its length, 4 (n + 1) bytes; the launcher fills it and sets perm and count
    const uint32_t* count;    // nullable: rows there are, at most n
    int* error_flag;          // mapped host memory; set when a wait ran out
    uint64_t wait_ns;         // limit of the chain's waits (0: give up at once when a barrier is not ready - test only)
};

}  // namespace tc

// Samples from which those with a gradient are listed: two tiles for every CTA, of which there are two an SM.  With one tile each the CTAs run
// side by side and fewer rows save nothing.  Backward of rays' samples at T = 2^19 (us), taken as they lie / by the list, which itself takes
// 4 to 8, by share of the samples that have a gradient:
//     75776 samples: all 64.5 / 71.7, six in ten 54.2 / 57.3, four in ten 51.2 / 46.1       100000: 67.7 / 75, 60.5 / 56.4, 57.3 / 50.1
//     2^18:          all 130 / 135, nine in ten 126 / 128, six in ten 116 / 96              2^20:   453 / 464, nine in ten 436 / 420, 381 / 293
// The share is not known before the list is made.  A sphere trained from random weights, steps of 2^18 samples, whole steps (us) without the list /
// with it: 288 / 290 after 70 steps (98 in 100 samples have a gradient), 292 / 291 after 360, 287 / 279 after 840 (eight in ten), 282 / 252 after 1600.
// Steps of a scene that is known: 2^18 samples, six in ten, 88 without the list and 61 with it; 160000, half, 43 and 28.5; 2^21, three in ten, 559 and 254.
inline int64_t live_list_min() { return (int64_t)2 * 2 * nb_num_sms() * tc::ROWS_OF_TILE; }
extern std::atomic<int> g_backward_tc;
extern std::atomic<int> g_backward_tc_wait_us;
extern std::atomic<int> g_forward_staged;
extern std::atomic<int> g_forward_stage_levels;
extern std::atomic<int> g_forward_persistent;
int field_backward_tc_failed();
int* wait_error_flag();   // mapped host memory that a kernel of the field raises when one of its bounded waits has run out
int launch_field_backward_tc(const GridParams& gp, const tc::BackwardArgs& args, cudaStream_t st);
// The copies of a grid whose first two levels are dense, in `room` bytes at `at`; levels == 0 where they do not fit.
tc::CoarseCopies coarse_copies(const GridParams& gp, void* at, int64_t room);

}  // namespace nb
