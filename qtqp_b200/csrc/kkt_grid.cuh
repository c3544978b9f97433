// The whole-GPU form of the dense KKT plugin backend (kkt_plugin.cu), for n
// from kKktGridN on: the phases of the large dense solve (large_ipm.cuh), one
// cooperative launch per call.
#pragma once

#include "dense_ipm.cuh"
#include "large_ipm.cuh"

namespace qtqp {

// Below this the single-block form is used.  One factorisation, three solves
// and three products through the host interface with m = 2n take, in us, with
// one block / the whole GPU: n = 40 389 / 466, 64 403 / 462, 96 548 / 481, 124
// 686 / 515; above, where the single block's factor no longer fits its
// registers, 300 13400 / 640 (factorisation 240, solve 40, product 20).
constexpr int kKktGridN = 80;
constexpr int kKktGridMaxN = kLB * kLargeBlocks;  // one 128-row block of the factor per CTA

// The sizes that have a grid form, and whether a call takes it: where the
// current device holds fewer than its 148 blocks at once, the single block does.
__host__ __device__ inline bool kkt_grid_form(int n) {
  return n >= kKktGridN && n <= kKktGridMaxN;
}
__host__ __device__ inline bool kkt_grid_route(int n, int resident_blocks) {
  return kkt_grid_form(n) && resident_blocks >= kLargeBlocks;
}
// Blocks of the grid form's kernels that the current device holds at once, and 0
// without cooperative launches.
int kkt_grid_resident();

// The factor in the workspace (its header, an int32).
constexpr int kKktFactor32 = 32, kKktFactor64 = 64, kKktFactorGrid = 65;

// Bytes of the grid form's part of the workspace (256-byte aligned start).
size_t kkt_grid_bytes(int n, int m);
// ws: the workspace, whose header and single-block layout (A, P and the vectors,
// `header` bytes in) both forms share; gws: the grid form's part.  kkt_grid_solve
// also solves with a single block's factor (FP32, or made where the grid did not
// fit), by that form.  A factorisation starts from a clean barrier and clean slots,
// whatever an earlier call left; *info is -1 when one of its waits gave up.  A solve
// whose waits gave up gives NaN.
int kkt_grid_factorize(int n, int m, const double* diag, char* ws, size_t header, char* gws,
                       int* info, cudaStream_t stream);
int kkt_grid_solve(int n, int m, const double* rhs, double* out, char* ws, size_t header,
                   char* gws, cudaStream_t stream);
int kkt_grid_matvec(int n, int m, const double* x, double* out, char* ws, size_t header,
                    char* gws, cudaStream_t stream);

}  // namespace qtqp
