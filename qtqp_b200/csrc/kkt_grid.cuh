// The whole-GPU form of the dense KKT plugin backend (kkt_plugin.cu), for n
// from kKktGridN on: the phases of the large dense solve (large_ipm.cuh), one
// cooperative launch per call.
#pragma once

#include "dense_ipm.cuh"

namespace qtqp {

// Below this the single-block form is used.  One factorisation, three solves
// and three products through the host interface with m = 2n take, in us, with
// one block / the whole GPU: n = 40 421 / 494, 64 434 / 483, 96 638 / 492, 124
// 740 / 553; above, where the single block's factor no longer fits its
// registers, 300 14200 / 897 (factorisation 472, solve 48, product 20).
constexpr int kKktGridN = 80;
constexpr int kKktGridMaxN = 128 * 148;  // one 128-row block of the factor per CTA

__host__ __device__ inline bool kkt_grid_form(int n) {
  return n >= kKktGridN && n <= kKktGridMaxN;
}

// Bytes of the grid form's part of the workspace (256-byte aligned start).
size_t kkt_grid_bytes(int n, int m);
// ws: the workspace, whose header (an int32: the factor's precision, 32 or 64)
// and single-block layout (A, P and the vectors, `header` bytes in) both forms
// share; gws: the grid form's part.  An FP32 factor is always the single
// block's: kkt_grid_solve then runs that form.  A factorisation starts from a clean
// barrier and clean slots, whatever an earlier call left; *info is -1 when one of
// its waits gave up.  A solve whose waits gave up gives NaN.
int kkt_grid_factorize(int n, int m, const double* diag, char* ws, size_t header, char* gws,
                       int* info, cudaStream_t stream);
int kkt_grid_solve(int n, int m, const double* rhs, double* out, char* ws, size_t header,
                   char* gws, cudaStream_t stream);
int kkt_grid_matvec(int n, int m, const double* x, double* out, char* ws, size_t header,
                    char* gws, cudaStream_t stream);

}  // namespace qtqp
