// Device-resident interior-point solve of one dense QP by one thread block.
//
// Algorithm: the homogeneous-embedding Mehrotra predictor-corrector of
// google-deepmind/qtqp v0.0.5, src/qtqp/__init__.py:351-614, with the KKT layer
// of src/qtqp/direct.py:112-311 and the Gram/Cholesky backend of
// src/qtqp/solvers_dense.py:25-145.  Every scalar decision (IR convergence and
// stall, tau root selection and fallback, ratio test, termination precedence)
// follows the reference; only the summation order of reductions differs.
//
// Work distribution inside the block ("ownership"): every per-element vector
// lives in the N-space [0, n+m) with the x-part at [0, n) and the y/s-part at
// [n, n+m); element k is always handled by thread k % NT.  Elementwise phases
// therefore need no barrier between them; a barrier is only needed before a
// phase that reads other threads' elements (matrix-vector products, the
// triangular solves) and is folded into the block reductions where possible.
#pragma once

#include <math.h>

#include <type_traits>

#include "common.cuh"

namespace qtqp {

// ----------------------------------------------------------------------------
// Per-instance memory layout (shared by host planning and device code).
// ----------------------------------------------------------------------------
enum VecId : int {
  kQ = 0,    // q = [c_eq; b_eq]
  kXY,       // iterate [x; y]
  kKQ,       // K^{-1} q (warm-started across iterations)
  kKQ0,      // warm start of K^{-1} q kept for an FP64 redo (mixed precision)
  kXYP,      // predictor K^{-1} r, then [x_p; y_p]
  kXYC,      // corrector K^{-1} r, then [x_c; y_c]
  kRHS,      // KKT right-hand side with the dual block negated
  kRES,      // IR residual
  kTMP,      // solve scratch (FP64 Gram right-hand side / solution)
  kREG,      // regularised KKT diagonal (dual block negative)
  kCORR,     // reg - true diagonal
  kDE,       // [e; d] accumulated Ruiz scalings
  kPI,       // [diag(P_eq); 1/Ry]
  kPW,       // [P_eq K^{-1}q_x; 1/sqrt(Ry)]
  kRS,       // [P_eq K^{-1}r_x; s]
  kXD,       // [P_eq x; d_s]
  kCT,       // [FP32 scratch (2n floats); Mehrotra correction / warm-start rows]
  kW,        // triangular-solve scratch (FP64)
  kNumVec
};

__host__ __device__ inline int odd_ld(int n) { return (n & 1) ? n : n + 1; }
__host__ __device__ inline size_t round16(size_t b) { return (b + 15) & ~size_t(15); }

// Panel buffer (PB): the tile Cholesky's two panels of (n+3)/4 tiles of
// 4 x 4, each tile padded to 17 elements so that lanes reading different
// tiles hit different banks; outside the factorisation, the staged column
// sums of dense_products (up to 8 warps x n).
__host__ __device__ inline size_t panel_buf_elems(int n) {
  return size_t(34) * ((n + 3) >> 2) + size_t(2) * n;
}

struct InstLayout {
  int lda, ldp, ldg, np;  // leading dims (doubles) and padded vector length
  size_t a_bytes, p_bytes, g_bytes, v_bytes;  // v_bytes: vectors + panel buffer
  int ap_smem, gv_smem;   // 1 when that region lives in shared memory
  size_t smem_bytes, global_bytes;
};

// Places G + vectors (and A + P when they also fit) in `smem_cap` bytes of
// shared memory; everything else goes to the instance's global workspace.
__host__ __device__ inline InstLayout plan_layout(int n, int m, size_t smem_cap) {
  InstLayout L;
  L.lda = odd_ld(n);
  L.ldp = odd_ld(n);
  L.ldg = odd_ld(n);
  L.np = (max(n + m, n + 4) + 1) & ~1;  // >= n + 4: pivot broadcast scalars
  L.a_bytes = round16(size_t(m) * L.lda * 8);
  L.p_bytes = round16(size_t(n) * L.ldp * 8);
  L.g_bytes = round16(size_t(n) * L.ldg * 8);
  L.v_bytes = round16((size_t(kNumVec) * L.np + panel_buf_elems(n)) * 8);
  const size_t gv = L.g_bytes + L.v_bytes, ap = L.a_bytes + L.p_bytes;
  L.gv_smem = gv <= smem_cap;
  L.ap_smem = L.gv_smem && (gv + ap <= smem_cap);
  L.smem_bytes = (L.gv_smem ? gv : 0) + (L.ap_smem ? ap : 0);
  L.global_bytes = (L.gv_smem ? 0 : gv) + (L.ap_smem ? 0 : ap);
  return L;
}

// Global workspace of one banded instance: vectors, the band factor (n x
// (bw+1)), working copies of the A (CSR and CSC) and P value arrays, and the
// rows of the Gram product's column groups (band_gram_groups).
struct BandLayout {
  int np;
  size_t v_bytes, l_bytes, val_bytes, row_bytes, total;
};
__host__ __device__ inline BandLayout plan_band_layout(int n, int m, int bw, int nnz_a,
                                                       int nnz_p) {
  BandLayout L;
  L.np = (max(n + m, n + 4) + 1) & ~1;
  L.v_bytes = round16(size_t(kNumVec) * L.np * 8);
  L.l_bytes = round16(size_t(n) * (bw + 1) * 8);
  L.val_bytes = round16((2 * size_t(nnz_a) + size_t(nnz_p)) * 8);
  L.row_bytes = round16((size_t(nnz_a) + size_t(n) / 8 + 2) * sizeof(int));
  L.total = L.v_bytes + L.l_bytes + L.val_bytes + L.row_bytes;
  return L;
}

// Shared-memory window of the banded factorisation / solves: bands up to
// kBandWinMaxBw use it (a panel has one row per thread of a 256-thread block,
// a step of the solves one per thread of its first 128).
constexpr int kBandWinMaxBw = 126;
// The blocked band solves: kBandSolveBlk columns per step; the rows that a step
// updates are spread over band_solve_owners(bw) threads (>= bw, a power of two).
constexpr int kBandSolveBlk = 8;
__host__ __device__ inline int band_solve_owners(int bw) {
  return bw <= 32 ? 32 : bw <= 64 ? 64 : 128;
}
// Their shared-memory elements: a ring of staged steps (the rows' factor entries,
// pitch kBandSolveBlk + 1, and the 8 x 8 diagonal block), a step's right-hand
// side and results, each twice, and the known values behind the last column.
constexpr int kBandSolveStages = 8;
__host__ __device__ inline size_t band_solve_stage(int bw) {
  return size_t(kBandSolveBlk + 1) * band_solve_owners(bw) + kBandSolveBlk * kBandSolveBlk;
}
__host__ __device__ inline size_t band_solve_elems(int bw) {
  return kBandSolveStages * band_solve_stage(bw) + 4 * kBandSolveBlk + 128;
}
// The Gram product of the banded format: a warp forms kGramCols columns from
// four dense rows of their entries in shared memory.  The pitch is 4 (mod 16)
// doubles, so that a half-warp's fragment loads hit 16 different banks.
constexpr int kGramCols = 8;
__host__ __device__ inline int gram_pitch(int bw) {
  const int w = (bw + 7 + 8) / 8 * 8;  // whole 8-column tiles
  return w + (4 - w % 16 + 16) % 16;
}
__host__ __device__ inline size_t gram_warp_elems(int bw) { return 4 * size_t(gram_pitch(bw)); }
constexpr int kBandPanel = 8;  // columns per panel of the blocked band Cholesky
// Shared memory of the blocked band Cholesky (band_chol_panel_range): the
// circular (bw + kBandPanel)^2 window, the panel rows, two stages of entering
// rows and the list of the window's lower 16 x 16 tiles.
__host__ __device__ inline size_t band_panel_bytes(int bw) {
  const size_t B = size_t(bw) + kBandPanel, nt16 = (size_t(bw) + 15) / 16;
  return (B * B + B * (kBandPanel + 1) + 2 * kBandPanel * (size_t(bw) + 1)) * sizeof(double) +
         nt16 * (nt16 + 1) / 2 * sizeof(uint16_t);
}
// The shared memory a band needs in a block of nt threads: the Cholesky, the
// solves, the Gram rows of every warp.
__host__ __device__ inline size_t band_win_bytes(int bw, int nt) {
  size_t e = band_panel_bytes(bw);
  const size_t cols = size_t(nt / 32) * gram_warp_elems(bw) * sizeof(double);
  const size_t solve = band_solve_elems(bw) * sizeof(double);
  if (cols > e) e = cols;
  if (solve > e) e = solve;
  return (e + 15) & ~size_t(15);
}

// Fields of one qtqp_iter_stats record.
enum StatField : int {
  kStIter = 0, kStCtx, kStBty, kStPcost, kStDcost, kStPres, kStDres, kStGap,
  kStPinfeas, kStDinfeas, kStDinfeasA, kStDinfeasP, kStMu, kStSigma,
  kStAlpha, kStTau, kStNormX, kStNormY, kStStatus, kStTime, kStPrel, kStDrel,
  kStCompl, kStNormS, kStMaxSy, kStMinSy, kStStdSy, kStMaxSoy, kStMinSoy,
  kStMeanSoy, kStStdSoy,
  kStLin0 = 31,  // three blocks of kLinFields: q, predictor, corrector
};
enum LinField : int {
  kLinSolves = 0, kLinFinalRes, kLinRhsNorm, kLinTol, kLinStatus, kLinTau,
  kLinPrec, kLinFields
};
// kLinStatus: 0 non-converged, 1 converged, 2 stalled.  kLinTau: -1 none,
// 0 quadratic, 1 linearised.  kLinPrec: 32 or 64 (factor precision used).

struct IrOutcome {
  int solves;
  int status;  // 0 non-converged, 1 converged, 2 stalled
  double final_res, rhs_norm, tol;
  bool nan;
};

// Copies of the instance's fields as local constants.  Phase functions are
// not inlined, so `this` points at a stack object; reading fields through it
// inside loops would be a local-memory load after every store that might
// alias it.  Each phase therefore starts with QTQP_LOCALS.
#define QTQP_LOCALS                                                             \
  const int tid = this->tid, n = this->n, m = this->m, z = this->z, N = this->N; \
  const int lda = this->lda, ldp = this->ldp, ldg = this->ldg;                   \
  double* const A = this->A;                                                     \
  double* const P = this->P;                                                     \
  double* const G = this->G;                                                     \
  const bool has_p = this->has_p;                                                \
  (void)tid; (void)n; (void)m; (void)z; (void)N; (void)lda; (void)ldp; (void)ldg; \
  (void)A; (void)P; (void)G; (void)has_p

// Independent partial sums per lane of a block's row dots (rowdot) outside
// the per-block dense format, which sets its own by block size (rowdot).
#ifndef QTQP_ROWDOT_UNROLL
#define QTQP_ROWDOT_UNROLL 4
#endif

// Storage formats of A, P and the KKT factor.
enum MatFormat : int {
  kFmtDense = 0,  // dense A (m x n), dense P, dense Gram G / Cholesky factor
  kFmtBand = 1,   // sparse A (CSR + CSC), sparse P (CSR), banded Gram / factor
  kFmtLarge = 2,  // one large dense QP on the whole GPU (grid mode, NT > 1024):
                  // dense A / P in global memory, blocked Gram + Cholesky
  kFmtSparse = 3, // one sparse QP on the whole GPU (grid mode): A and P as in
                  // kFmtBand, a supernodal Cholesky of the Gram matrix
};

// ----------------------------------------------------------------------------
// The solver state of one instance, replicated in every thread of the block.
// FMT selects the matrix backend; the interior-point logic is shared.
// ----------------------------------------------------------------------------
// Large-format phases (large_ipm.cuh), called from the Ipm dispatch points.
template <typename T, class S>
__device__ int large_factorize(S& s);
template <class S>
__device__ __noinline__ void large_equilibrate(S& s);
template <typename T, class S>
__device__ __noinline__ void large_chol_solve(S& s, T* v, T* w);
template <class S, class RowEpi, class ColEpi>
__device__ void large_products(S& s, const double* vx, const double* vy, const double* vs,
                               const double* vp, RowEpi row_epi, ColEpi col_epi);
// Partitioned banded factorisation / solve of grid mode (band_grid.cuh).
template <typename T, class S>
__device__ int bandp_factorize(S& s);
template <typename T, class S>
__device__ __noinline__ void bandp_solve(S& s, T* v, T* w);
// Supernodal factorisation / solve of grid mode (sparse_grid.cuh).
struct SnFactor;
template <typename T, class S>
__device__ int sparse_factorize(S& s);
template <typename T, class S>
__device__ void sparse_solve(S& s, T* v, T* w);

template <int NT, int FMT = kFmtDense>
struct Ipm {
  // Sparse A and P (CSR / CSC) with a banded or supernodal Gram factor.
  static constexpr bool kSparseA = FMT == kFmtBand || FMT == kFmtSparse;
  int tid;
  int n, m, z, N;
  bool has_p;
  // Original (presolved, unequilibrated) data in global memory: row-major,
  // or column-major (the value order of a dense CSC matrix) when colmajor.
  const double* A0;
  const double* P0;
  bool colmajor = false;
  const double* b0;
  const double* c0;
  // Working data.
  double* A;  // m x lda equilibrated A
  double* P;  // n x ldp equilibrated P with a zero diagonal (P_off)
  double* G;  // n x ldg Gram matrix / Cholesky factor (FP64, or FP32 alias)
  double* V;  // kNumVec vectors of np doubles
  double* PB;  // panel buffer of tile_cholesky (panel_buf_elems(n) elements)
  int lda, ldp, ldg, np;
  double* red;
  int phase;
  // Options.
  const qtqp_options* o;
  // Banded backend (FMT == kFmtBand): A as CSR (ip, ix) and CSC (jp, jx),
  // P as CSR (pp, px) holding both triangles; the working (equilibrated)
  // values av / at / pv; the factor in lower band storage by columns,
  // Lb[j * (bw + 1) + (i - j)] = L_ij for j <= i <= j + bw.
  const int* ip;
  const int* ix;
  const int* jp;
  const int* jx;
  const int* pp;
  const int* px;
  const double* av0;
  const double* at0;
  const double* pv0;
  double* av;
  double* at;
  double* pv;
  double* Lb;
  int bw, nnz_a, nnz_p;
  int* grow;  // band_gram_groups
  int* gcnt;
  // Shared-memory window of the banded factorisation and solves (null: the
  // band is too wide for it and the global-memory variants run).
  double* bwin;
  size_t bwin_bytes;
  // Banded backend in grid mode: the number of partitions of the columns,
  // the partitions' spikes, the separator blocks and the separator vectors.
  int nparts;
  double* bp_wl;
  double* bp_sep;
  double* bp_vec;
  // Supernodal factor of grid mode (FMT == kFmtSparse).
  const SnFactor* sn;

  // Grid mode (NT > 1024, FMT == kFmtLarge): the group is a cooperative grid
  // of NT / kGridBT blocks; barriers and reductions go through gctl.
  GridCtl* gctl;
  // Large format: padded sizes (multiples of 128 / 32), the factor in FP64
  // (g64) or FP32 (g32), both npad x npad row-major (lower triangle), the
  // split TF32 operands X = (diag(1/sqrt(Ry)) A)^T
  // (xhi / xlo, npad x mpad), their tensor maps, the CTA's shared-memory
  // arena (tensor-core ring / staging tiles), its TMEM accumulator and the
  // per-thread pipeline counters of the tensor-core ring.
  int npad, mpad;
  int* linfo;  // factorisation status shared by the grid
  double* g64;
  float* g32l;
  double* sinv;  // sub-block inverses of the current panel step
  double* gpart;    // parts of split Gram tiles (GramSplit)
  double* colpart;  // per-block column sums of large_products (gridDim x npad)
  float* xhi;
  float* xlo;
  const void* map_hi;
  const void* map_lo;
  unsigned char* arena;
  uint32_t tmem;
  uint32_t tc_load, tc_mma, tc_tiles;
  uint32_t tri_gen;   // whole-GPU triangular solves so far (their slots' tags)
  GridSlot* tri_slot; // and the slots, one per row

  __device__ __forceinline__ void sync() const {
    if constexpr (NT > 1024) {
      grid_sync(gctl);
    } else {
      group_sync<NT>();
    }
  }
  template <int NS, int NM>
  __device__ __forceinline__ void reduce(double (&sums)[NS > 0 ? NS : 1],
                                         double (&maxs)[NM > 0 ? NM : 1]) {
    if constexpr (NT > 1024) {
      grid_reduce<kGridBT, NS, NM>(sums, maxs, red, gctl, phase);
    } else {
      block_reduce<NT, NS, NM, kSumT>(sums, maxs, red, phase);
    }
  }
  // The threads that add up the terms of a sum over a vector: all, but in a
  // banded block the first 128, whatever its size (one term order, and so one
  // result, for every block size: the iterates of an infeasible QP diverge along
  // a ray, which amplifies a change of rounding by 1e6 and more).
  static constexpr int kSumT = FMT == kFmtBand && NT <= 1024 ? 128 : NT;
  __device__ __forceinline__ int sum_own(int lo) const {  // first index >= lo of this thread
    if constexpr (kSumT == NT) {
      return own(lo);
    } else {
      return tid < kSumT ? lo + ((tid - lo) & (kSumT - 1)) : 0x7fffffff - kSumT;
    }
  }

  __device__ __forceinline__ double* vec(int id) const { return V + size_t(id) * np; }
  // First index >= lo owned by this thread (k % NT == tid).  NT is a power of
  // two except for the large grid (one CTA per SM of a B200: 148 x 256).
  __device__ __forceinline__ int own(int lo) const {
    if constexpr ((NT & (NT - 1)) == 0) {
      return lo + ((tid - lo) & (NT - 1));
    } else {
      const int d = (tid - lo) % NT;
      return lo + (d < 0 ? d + NT : d);
    }
  }
  __device__ __forceinline__ float* g32() const { return reinterpret_cast<float*>(G); }

  // log2 of the lanes cooperating on one dot product when K outputs share the
  // block: the largest power of two S <= 32 with K S <= NT (1 when K > NT).
  __device__ __forceinline__ int lanes_log2(int K) const {
    if constexpr ((NT & (NT - 1)) == 0) {  // no division: a call costs 350 cycles less
      return max(0, min(5, 31 - __clz(NT) - (K > 1 ? 32 - __clz(K - 1) : 0)));
    } else {
      return K >= NT ? 0 : min(5, 31 - __clz(NT / K));
    }
  }

  // out_k = sum_{i < len} body(k, i) for k < K, S = 2^lanes_log2(K) lanes per
  // output.  The S lanes of an output are strided across the warp (lane =
  // s * (32/S) + g) so that neighbouring lanes work on neighbouring outputs;
  // their partial sums are combined with xor shuffles, and lane s == 0 calls
  // epi(k, sum).  NACC independent sums per output.  No barrier inside.
  template <int NACC, bool MAXOP = false, int FORCE_S = 0, typename AccT = double,
            typename Body, typename Epi>
  __device__ __forceinline__ void rowdot(int K, int len, Body body, Epi epi) const {
    static_assert(FORCE_S == 0 || FORCE_S == 32, "a warp per output or the automatic split");
    const int ls = FORCE_S > 0 ? 5 : lanes_log2(K);
    const int S = 1 << ls, per_warp = 32 >> ls;
    const int tid = this->tid;
    const int lane = tid & 31, warp = tid >> 5;
    const int s = lane >> (5 - ls), g = lane & (per_warp - 1);
    const int per_pass = (NT / 32) * per_warp;
    for (int k0 = 0; k0 < K; k0 += per_pass) {
      const int k = k0 + warp * per_warp + g;
      AccT acc[NACC];
#pragma unroll
      for (int a = 0; a < NACC; ++a) acc[a] = AccT(0);
      if (k < K) {
        // U independent partial sums per lane keep U loads (and U FMA
        // chains) in flight: grid mode streams A and P from HBM; a block's
        // loads come from shared memory or L2.  The per-block dense format
        // keeps its loops short (one or two sums): its QPs are small, and
        // several blocks per SM run different phases of the IPM, whose code
        // then competes for the instruction cache (measured per block size:
        // 2-14 % faster at n = 16..64 than four sums).
        constexpr int U = NT > 1024                           ? 16
                          : (FMT == kFmtDense && NT <= 128)   ? 1
                          : FMT == kFmtDense                  ? 2
                                                              : QTQP_ROWDOT_UNROLL;
        AccT part[U][NACC];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
          for (int a = 0; a < NACC; ++a) part[u][a] = AccT(0);
        int i = s;
        if constexpr (FMT == kFmtDense) {
          // Eight loads in flight, in straight-line code and the order of the
          // loop below: n > 64, whose A may come from L2 (n = 96, m = 193, one QP:
          // 4.1 ms, 5.6 with one or two in flight).
          for (; i + 7 * S < len; i += 8 * S) {
#pragma unroll
            for (int u = 0; u < 8; ++u) body(k, i + u * S, part[u % U]);
          }
        }
        for (; i + (U - 1) * S < len; i += U * S) {
#pragma unroll
          for (int u = 0; u < U; ++u) body(k, i + u * S, part[u]);
        }
        for (; i < len; i += S) body(k, i, part[0]);
#pragma unroll
        for (int a = 0; a < NACC; ++a) {
          AccT t = part[0][a];
#pragma unroll
          for (int u = 1; u < U; ++u) t = MAXOP ? fmax(t, part[u][a]) : t + part[u][a];
          acc[a] = t;
        }
      }
#pragma unroll 1
      for (int off = 16; off >= per_warp; off >>= 1) {
#pragma unroll
        for (int a = 0; a < NACC; ++a) {
          const AccT o = __shfl_xor_sync(0xffffffffu, acc[a], off);
          acc[a] = MAXOP ? fmax(acc[a], o) : acc[a] + o;
        }
      }
      if (k < K && s == 0) epi(k, acc);
    }
  }
  // Lanes per output of a row dot (body reads element (k, j)): a whole warp
  // per output in grid mode (coalesced rows), the automatic split otherwise.
  static constexpr int kRowS = NT > 1024 ? 32 : 0;
  __device__ __forceinline__ float* t32() const { return reinterpret_cast<float*>(vec(kCT)); }

  // --------------------------------------------------------------------------
  // Binding of memory regions.
  // --------------------------------------------------------------------------
  __device__ void bind(int n_, int m_, char* smem, char* gmem, size_t smem_cap) {
    tid = threadIdx.x;
    n = n_;
    m = m_;
    N = n + m;
    const InstLayout L = plan_layout(n, m, smem_cap);
    lda = L.lda;
    ldp = L.ldp;
    ldg = L.ldg;
    np = L.np;
    char* gv = L.gv_smem ? smem : gmem;
    G = reinterpret_cast<double*>(gv);
    V = reinterpret_cast<double*>(gv + L.g_bytes);
    PB = V + size_t(kNumVec) * np;
    char* ap = L.ap_smem ? smem + L.g_bytes + L.v_bytes
                         : gmem + (L.gv_smem ? 0 : L.g_bytes + L.v_bytes);
    A = reinterpret_cast<double*>(ap);
    P = reinterpret_cast<double*>(ap + L.a_bytes);
  }

  // --------------------------------------------------------------------------
  // Ruiz equilibration (src/qtqp/__init__.py:616-663), done in place on the
  // working copies, bit-compatible with the reference: the nonzero a_ij is
  // multiplied by (d_i * e_j), the clip bounds are [1e-3, 1e3].
  // --------------------------------------------------------------------------
  QTQP_PHASE void load_and_equilibrate(bool equilibrate, double& nb, double& nc) {
    if constexpr (kSparseA) {
      band_load_and_equilibrate(equilibrate, nb, nc);
      return;
    }
    QTQP_LOCALS;
    double* de = vec(kDE);
    double* sc = vec(kTMP);  // per-sweep [e_i; d_i]
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int NW = NT / 32;
    if (colmajor) {  // coalesced column reads; odd lda/ldp keep the stores conflict-free
      for (int j = warp; j < n; j += NW)
        for (int i = lane; i < m; i += 32) A[i * lda + j] = A0[size_t(j) * m + i];
      for (int j = warp; j < n; j += NW)
        for (int i = lane; i < n; i += 32) P[i * ldp + j] = has_p ? P0[size_t(j) * n + i] : 0.0;
    } else {
      for (int i = warp; i < m; i += NW)
        for (int j = lane; j < n; j += 32) A[i * lda + j] = A0[size_t(i) * n + j];
      for (int i = warp; i < n; i += NW)
        for (int j = lane; j < n; j += 32) P[i * ldp + j] = has_p ? P0[size_t(i) * n + j] : 0.0;
    }
    for (int k = tid; k < N; k += NT) de[k] = 1.0;
    sync();
    if constexpr (FMT == kFmtLarge) {
      if (equilibrate) large_equilibrate(*this);
    } else if (equilibrate) {
      const double* Ap = A;
      const double* Pp = P;
      const int la = lda, lp = ldp, mm = m, nn = n;
      const int plen = has_p ? n : 0;
      auto scale_of = [](double mx) {
        if (mx == 0.0) mx = 1.0;
        return fmin(fmax(1.0 / sqrt(mx), 1e-3), 1e3);
      };
      for (int sweep = 0; sweep < 10; ++sweep) {
        // Column maxima over A and P, row maxima over A.
        rowdot<1, true>(n, m + plen,
                        [&](int k, int i, double* acc) {
                          const double v = i < mm ? Ap[i * la + k] : Pp[(i - mm) * lp + k];
                          acc[0] = fmax(acc[0], fabs(v));
                        },
                        [&](int k, double* acc) { sc[k] = scale_of(acc[0]); });
        rowdot<1, true>(m, n,
                        [&](int k, int j, double* acc) {
                          acc[0] = fmax(acc[0], fabs(Ap[k * la + j]));
                        },
                        [&](int k, double* acc) { sc[nn + k] = scale_of(acc[0]); });
        sync();
        for (int i = warp; i < m; i += NW) {
          const double di = sc[n + i];
          for (int j = lane; j < n; j += 32) A[i * lda + j] *= di * sc[j];
        }
        if (has_p) {
          for (int i = warp; i < n; i += NW) {
            const double ei = sc[i];
            for (int j = lane; j < n; j += 32) P[i * ldp + j] *= ei * sc[j];
          }
        }
        for (int k = tid; k < N; k += NT) de[k] *= sc[k];
        sync();
      }
    }
    double* q = vec(kQ);
    double* pi = vec(kPI);
    double mx[2] = {0.0, 0.0};
    double dummy[1] = {0.0};
    for (int k = tid; k < N; k += NT) {
      if (k < n) {
        q[k] = c0[k] * de[k];
        pi[k] = P[k * ldp + k];  // diag(P_eq); P keeps only its off-diagonal
        P[k * ldp + k] = 0.0;
        mx[1] = nanmax(mx[1], fabs(c0[k]));
      } else {
        q[k] = b0[k - n] * de[k];
        mx[0] = nanmax(mx[0], fabs(b0[k - n]));
      }
    }
    reduce<0, 2>(dummy, mx);
    nb = mx[0];
    nc = mx[1];
    sync();
  }

  // --------------------------------------------------------------------------
  // DirectKktSolver.update (direct.py:183-216): true and regularised diagonal,
  // the backend's update_diag (solvers_dense.py:95-97) and the derived
  // 1/Ry and 1/sqrt(Ry) used by factorize/solve (solvers_dense.py:103, 132).
  // Owner-wise; the caller synchronises before factorising.
  // --------------------------------------------------------------------------
  __device__ void kkt_diag(double mu, double min_reg) {
    QTQP_LOCALS;
    const double* xy = vec(kXY);
    const double* s = vec(kRS);
    const double* pi = vec(kPI);
    double* reg = vec(kREG);
    double* corr = vec(kCORR);
    double* piw = vec(kPI);
    double* pw = vec(kPW);
    for (int k = tid; k < N; k += NT) {
      double t;
      if (k < n) {
        t = pi[k];
        t += mu;
      } else if (k < n + z) {
        t = mu;
      } else {
        t = s[k] / xy[k] + mu;
      }
      double r = fmax(t, min_reg);
      if (k >= n) {
        t = -t;
        r = -r;
        const double ry = -r;
        piw[k] = 1.0 / ry;
        pw[k] = 1.0 / sqrt(ry);
      }
      reg[k] = r;
      corr[k] = r - t;
    }
  }

  // Same for an externally supplied diagonal (the plugin's update_diag).
  __device__ void kkt_diag_given(const double* diag) {
    QTQP_LOCALS;
    double* reg = vec(kREG);
    double* piw = vec(kPI);
    double* pw = vec(kPW);
    for (int k = tid; k < N; k += NT) {
      const double r = diag[k];
      reg[k] = r;
      if (k >= n) {
        const double ry = -r;
        piw[k] = 1.0 / ry;
        pw[k] = 1.0 / sqrt(ry);
      }
    }
  }

  // --------------------------------------------------------------------------
  // factorize (solvers_dense.py:99-116): G = P_off + diag(Rx) + A_s^T A_s with
  // A_s = diag(1/sqrt(Ry)) A, a relative diagonal jitter, then Cholesky.
  // Returns 0 or the 1-based index of the first non-positive pivot.
  // Small n: the register-tiled path; otherwise Gram into memory + cholesky.
  // --------------------------------------------------------------------------
  template <typename T>
  QTQP_PHASE int factorize() {
    if constexpr (kSparseA) {
      return band_factorize<T>();
    } else if constexpr (FMT == kFmtLarge) {
      return large_factorize<T>(*this);
    } else {
      const int nb = (n + 3) >> 2;
      if (nb * (nb + 1) / 2 <= 2 * NT) return factorize_regs<T>();
      return factorize_mem<T>();
    }
  }

  // Register-tiled factorisation: each thread owns TPT (1 or 2) 4x4 tiles of
  // the lower triangle of G (tile t = tid + q NT, q < TPT); the Gram product
  // fills them (the FP64 one on the FP64 tensor cores through g, see
  // gram_dmma; the FP32 one on the registers), then tile_cholesky factors
  // them in place.  The finished L is written to G for the solves.
  template <typename T>
  __device__ int factorize_regs() {
    const int nb = (n + 3) >> 2;
    if (nb * (nb + 1) / 2 <= NT) return factorize_tiles<T, 1>();
    return factorize_tiles<T, 2>();
  }

  template <typename T, int TPT>
  __device__ int factorize_tiles() {
    QTQP_LOCALS;
    QTQP_TIC();
    T* g = reinterpret_cast<T*>(G);
    const double* reg = vec(kREG);
    const double* wsc = vec(kPW);
    const int nb = (n + 3) >> 2;
    const int tiles = nb * (nb + 1) / 2;
    bool mine[TPT];
    int bi[TPT], bj[TPT];
    T acc[TPT][4][4];
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
      const int t = tid + q * NT;
      mine[q] = t < tiles;
      bi[q] = bj[q] = 0;
      if (mine[q]) {
        int b = int((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
        while (b * (b + 1) / 2 > t) --b;
        while ((b + 1) * (b + 2) / 2 <= t) ++b;
        bi[q] = b;
        bj[q] = t - b * (b + 1) / 2;
      }
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[q][a][b] = T(0);
    }
    if constexpr (sizeof(T) == 8) {
      // FP64 Gram on the FP64 tensor cores: each warp forms 16 x 16 lower
      // blocks of A^T diag(1/Ry) A with mma.sync m8n8k4 (DMMA) over 4-row
      // slices of A, writes them to g, and each thread then reads its tiles.
      gram_dmma(g);
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        if (!mine[q]) continue;
        const int i0 = bi[q] * 4, j0 = bj[q] * 4;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int i = i0 + a, j = j0 + b;
            if (i < n && j <= i) acc[q][a][b] = g[i * ldg + j];
          }
      }
    } else {
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        if (!mine[q]) continue;
        const int i0 = bi[q] * 4, j0 = bj[q] * 4;
        for (int r = 0; r < m; ++r) {
          const double w = wsc[n + r];
          const double* row = A + r * lda;
          T ai[4], aj[4];
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            ai[a] = (i0 + a < n) ? T(row[i0 + a] * w) : T(0);
            aj[a] = (j0 + a < n) ? T(row[j0 + a] * w) : T(0);
          }
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[q][a][b] = fma(ai[a], aj[b], acc[q][a][b]);
        }
      }
    }
    double dmax[1] = {0.0};
    double dummy[1] = {0.0};
#pragma unroll
    for (int q = 0; q < TPT; ++q) {
      if (!mine[q]) continue;
      const int i0 = bi[q] * 4, j0 = bj[q] * 4;
#pragma unroll
      for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int i = i0 + a, j = j0 + b;
          if (i < n && j <= i) {
            double base = P[i * ldp + j];
            if (i == j) base += reg[i];
            acc[q][a][b] = T(base) + acc[q][a][b];
            if (i == j) dmax[0] = nanmax(dmax[0], double(acc[q][a][b]));
          }
        }
      }
    }
    reduce<0, 1>(dummy, dmax);
    const double jit = (sizeof(T) == 8 ? 1e-14 : 2.384185791015625e-07) * dmax[0];
#pragma unroll
    for (int q = 0; q < TPT; ++q)
#pragma unroll
      for (int a = 0; a < 4; ++a)
        if (mine[q] && bi[q] == bj[q] && bi[q] * 4 + a < n)
          acc[q][a][a] = T(double(acc[q][a][a]) + jit);
    QTQP_TOC(kPhGram);
    QTQP_RETIC();
    const int info = tile_cholesky<T, TPT>(acc, mine, bi, bj, g);
    QTQP_TOC(kPhChol);
    return info;
  }

  // Lower 16 x 16 blocks of the FP64 Gram A^T diag(1/Ry) A into g (entries
  // i >= j, i, j < n), one warp per block, on the FP64 tensor cores: for each
  // 4-row slice of A, lane l holds a = A[r + l%4][I + l/4] / Ry and
  // b = A[r + l%4][J + l/4] (dmma_8x8x4's fragment layout) of the block's two
  // row and column halves, rows past m and columns past n are zero.  Ends with
  // a barrier.
  __device__ __forceinline__ void gram_dmma(double* g) {
    QTQP_LOCALS;
    const double* iry = vec(kPI) + n;  // 1 / Ry
    const int lane = tid & 31, warp = tid >> 5;
    const int lr = lane & 3, lc = lane >> 2;
    const int n16 = (n + 15) >> 4;
    const int nblk = n16 * (n16 + 1) / 2;
#pragma unroll 1
    for (int t = warp; t < nblk; t += NT / 32) {
      int bi = 0;
      while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
      const int bj = t - bi * (bi + 1) / 2;
      int ci[2], cj[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        ci[h] = bi * 16 + 8 * h + lc;
        cj[h] = bj * 16 + 8 * h + lc;
      }
      double d[2][2][2];
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 2; ++q) d[h][q][0] = d[h][q][1] = 0.0;
      // Two slices per step, their loads issued first (A may come from L2
      // when it does not fit on chip); the products accumulate in row order.
#pragma unroll 1
      for (int r = 0; r < m; r += 8) {
        double a[2][2], b[2][2];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
          const int rr = r + 4 * u + lr;
          const bool in = rr < m;
          const double* row = A + rr * lda;
          const double w = in ? iry[rr] : 0.0;
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            a[u][h] = in && ci[h] < n ? row[ci[h]] * w : 0.0;
            b[u][h] = in && cj[h] < n ? row[cj[h]] : 0.0;
          }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 2; ++q) dmma_8x8x4(d[h][q], a[u][h], b[u][q]);
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const int i = ci[h], j = bj * 16 + 8 * q + 2 * lr;
          if (i < n) {
            if (j <= i) g[i * ldg + j] = d[h][q][0];
            if (j + 1 <= i) g[i * ldg + j + 1] = d[h][q][1];
          }
        }
    }
    sync();
  }

  // Right-looking Cholesky of the register tiles of factorize_tiles in
  // 4-column panels, one barrier per panel.  Panel k's off-diagonal tiles
  // L_{i,k} = G_{i,k} L_kk^{-T} are published in the double-buffered panel
  // buffer PB; every tile right of panel k is then updated by the rank-4
  // product L_{i,k} L_{j,k}^T.  The 4 x 4 diagonal factor L_kk is formed by
  // each thread that owns a tile of panel k from the diagonal tile, which its
  // owner publishes in g (its own, not yet written, region of the factor) one
  // panel ahead, before its last update; each of them applies that update
  // itself in the owner's order, so all copies agree to the bit.  A
  // non-positive pivot is recorded in shared memory and stops every thread
  // after the panel's barrier.  The diagonal of the result keeps 1 / l_jj,
  // and every 32 x 32 diagonal block of L is inverted in place afterwards
  // (see chol_solve).  Returns 0 or the 1-based index of the first
  // non-positive pivot.
  template <typename T, int TPT>
  __device__ int tile_cholesky(T (&acc)[TPT][4][4], const bool (&mine)[TPT],
                               const int (&bi)[TPT], const int (&bj)[TPT], T* g) {
    QTQP_LOCALS;
    const int nb = (n + 3) >> 2;
    // Panel t's tiles (L values; exactly zero in rows and columns beyond n)
    // live in pb[t & 1] at 17 elements per tile.
    T* const pb0 = reinterpret_cast<T*>(PB);
    const int pstride = 17 * nb;
    // Lower entries of a diagonal tile into g (its own region).
    auto put_diag = [&](int t) {
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        if (!mine[q] || bi[q] != t || bj[q] != t) continue;
        const int i0 = bi[q] * 4, j0 = bj[q] * 4;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b)
            if (b <= a && i0 + a < n) g[(i0 + a) * ldg + j0 + b] = acc[q][a][b];
      }
    };
    // The factor of diagonal tile t: D (as published, one update short when
    // t > 0) minus the rows of panel t-1, then the 4 x 4 Cholesky.  ld keeps
    // 1 / l on its diagonal.  Returns 0 or the failing 1-based column.
    auto diag_factor = [&](int t, T (&ld)[4][4]) -> int {
      T d[4][4];
      const int r0 = t * 4;
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b)
          d[a][b] = (b <= a && r0 + a < n) ? g[(r0 + a) * ldg + r0 + b] : T(0);
      if (t > 0) {  // the owner's last update, in the owner's order
        const T* pr = pb0 + ((t - 1) & 1) * pstride + t * 17;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          T l[4];
#pragma unroll
          for (int a = 0; a < 4; ++a) l[a] = pr[a * 4 + c];
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) d[a][b] = fma(-l[a], l[b], d[a][b]);
        }
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int a = 0; a < 4; ++a) ld[a][c] = T(0);
        if (r0 + c >= n) continue;
        const T piv = d[c][c];
        if (!(piv > T(0))) return r0 + c + 1;
        const T il = rsqrt(piv);
        ld[c][c] = il;
#pragma unroll
        for (int a = c + 1; a < 4; ++a) ld[a][c] = d[a][c] * il;
#pragma unroll
        for (int a = c + 1; a < 4; ++a)
#pragma unroll
          for (int b = c + 1; b <= a; ++b) d[a][b] = fma(-ld[a][c], ld[b][c], d[a][b]);
      }
      return 0;
    };
    // Tile q of panel t (already updated by panels < t) becomes
    // L_{i,t} = tile L_tt^{-T}, published in the panel buffer; the diagonal
    // tile becomes L_tt itself.
    auto finish_panel = [&](int q, int t, const T (&ld)[4][4]) {
      if (bi[q] == t) {
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int c = 0; c < 4; ++c) acc[q][a][c] = ld[a][c];
        return;
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          T x = acc[q][a][c];
#pragma unroll
          for (int e = 0; e < c; ++e) x = fma(-acc[q][a][e], ld[c][e], x);
          acc[q][a][c] = x * ld[c][c];  // ld[c][c] = 1 / l_cc (0 beyond n)
        }
      }
      T* dst = pb0 + (t & 1) * pstride + bi[q] * 17;
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = 0; c < 4; ++c) dst[a * 4 + c] = acc[q][a][c];
    };
    // Panel t for the tiles of this thread that belong to it.
    auto do_panel = [&](int t, int* s_info) {
      bool need = false;
#pragma unroll
      for (int q = 0; q < TPT; ++q) need = need || (mine[q] && bj[q] == t);
      if (!need) return;
      T ld[4][4];
      const int f = diag_factor(t, ld);
      if (f != 0) {
        s_info[t & 1] = f;
        return;
      }
#pragma unroll
      for (int q = 0; q < TPT; ++q)
        if (mine[q] && bj[q] == t) finish_panel(q, t, ld);
    };
    // A failure is noted in the slot of the panel's parity, which the next
    // panel does not write, so every thread reads the same value after the
    // barrier.
    __shared__ int s_info[2];
    if (tid < 2) s_info[tid] = 0;
    put_diag(0);
    put_diag(1);
    sync();
    do_panel(0, s_info);
    sync();
    int info = s_info[0];
    for (int kb = 0; info == 0 && kb + 1 < nb; ++kb) {
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        if (!mine[q] || bj[q] <= kb) continue;
        // rank-4 update with panel kb, one column at a time
        const T* pi = pb0 + (kb & 1) * pstride + bi[q] * 17;
        const T* pj = pb0 + (kb & 1) * pstride + bj[q] * 17;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          T li[4], lj[4];
#pragma unroll
          for (int a = 0; a < 4; ++a) {
            li[a] = pi[a * 4 + c];
            lj[a] = pj[a * 4 + c];
          }
#pragma unroll
          for (int a = 0; a < 4; ++a)
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[q][a][b] = fma(-li[a], lj[b], acc[q][a][b]);
        }
      }
      do_panel(kb + 1, s_info);
      if (kb + 2 < nb) put_diag(kb + 2);
      sync();
      info = s_info[(kb + 1) & 1];
    }
    if (info == 0) {
#pragma unroll
      for (int q = 0; q < TPT; ++q) {
        if (!mine[q]) continue;
        const int i0 = bi[q] * 4, j0 = bj[q] * 4;
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) {
            const int i = i0 + a, j = j0 + b;
            if (i < n && j <= i) g[i * ldg + j] = acc[q][a][b];
          }
      }
    }
    sync();
    if (info == 0) invert_diag_blocks<T>(g);
    return info;
  }

  template <typename T>
  __device__ int factorize_mem() {
    QTQP_LOCALS;
    QTQP_TIC();
    T* g = reinterpret_cast<T*>(G);
    const double* reg = vec(kREG);
    const double* wsc = vec(kPW);
    const int nb = (n + 3) >> 2;
    const int tiles = nb * (nb + 1) / 2;
    double dmax[1] = {0.0};
    double dummy[1] = {0.0};
    for (int t = tid; t < tiles; t += NT) {
      int bi = int((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
      while (bi * (bi + 1) / 2 > t) --bi;
      while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
      const int bj = t - bi * (bi + 1) / 2;
      const int i0 = bi * 4, j0 = bj * 4;
      T acc[4][4];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) acc[a][b] = T(0);
      for (int r = 0; r < m; ++r) {
        const double w = wsc[n + r];
        const double* row = A + r * lda;
        T ai[4], aj[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
          ai[a] = (i0 + a < n) ? T(row[i0 + a] * w) : T(0);
          aj[a] = (j0 + a < n) ? T(row[j0 + a] * w) : T(0);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int b = 0; b < 4; ++b) acc[a][b] = fma(ai[a], aj[b], acc[a][b]);
      }
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const int i = i0 + a;
        if (i >= n) continue;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
          const int j = j0 + b;
          if (j > i) continue;
          double base = P[i * ldp + j];
          if (i == j) base += reg[i];
          const T v = T(base) + acc[a][b];
          g[i * ldg + j] = v;
          if (i == j) dmax[0] = nanmax(dmax[0], double(v));
        }
      }
    }
    reduce<0, 1>(dummy, dmax);
    // FP64: the reference's 1e-14 relative jitter (solvers_dense.py:112).
    // FP32: the same idea at FP32 resolution (2^-22 relative).
    const double jit = (sizeof(T) == 8 ? 1e-14 : 2.384185791015625e-07) * dmax[0];
    for (int k = tid; k < n; k += NT) g[k * ldg + k] = T(double(g[k * ldg + k]) + jit);
    sync();
    QTQP_TOC(kPhGram);
    QTQP_RETIC();
    const int info = cholesky<T>(g);
    QTQP_TOC(kPhChol);
    return info;
  }

  // Right-looking Cholesky of the lower triangle, two barriers per column;
  // afterwards every 32x32 diagonal block of L is replaced by its inverse so
  // that the triangular solves are block-parallel (see chol_solve).
  //
  // One barrier per column: phase k updates the trailing matrix with the
  // still-unscaled column k (a_ij -= a_ik a_jk / d_k) and, independently,
  // finishes column k-1 (l_ik = a_ik / sqrt(d_{k-1}), l_kk = sqrt(d_{k-1})),
  // which phase k does not read.
  template <typename T>
  QTQP_PHASE int cholesky(T* g) {
    QTQP_LOCALS;
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int NW = NT / 32;
    T il_prev = T(1);  // 1 / sqrt(d) of the previous pivot
    for (int k = 0; k <= n; ++k) {
      if (k > 0) {  // finish column k-1
        const T inv = il_prev;
        for (int i = k + tid; i < n; i += NT) g[i * ldg + k - 1] *= inv;
        if (tid == NT - 1) g[(k - 1) * ldg + k - 1] = inv;  // diagonal keeps 1/l_kk
      }
      if (k == n) break;
      const T d = g[k * ldg + k];
      if (!(d > T(0))) {
        sync();
        return k + 1;
      }
      // One reciprocal square root per pivot, no divisions on this chain:
      // 1 / l_kk = rsqrt(d), 1 / d = (1 / l_kk)^2.
      const T il = rsqrt(d);
      const T inv_d = il * il;
      for (int j = k + 1 + warp; j < n; j += NW) {
        const T t = g[j * ldg + k] * inv_d;
        for (int i = j + lane; i < n; i += 32) g[i * ldg + j] = fma(-g[i * ldg + k], t, g[i * ldg + j]);
      }
      il_prev = il;
      sync();
    }
    sync();
    invert_diag_blocks<T>(g);
    return 0;
  }

  // In-place inverse of each 32x32 lower-triangular diagonal block of L (the
  // last one smaller), whose diagonal holds 1 / L_jj already, by doubling:
  // with the s x s diagonal blocks inverted, the block below each pair's first
  // becomes X21 = -X22 (L21 X11), s = 1, 2, 4, 8, 16.  The transpose of T = L21
  // X11 is formed in the unused upper triangle, L21's mirror image.  Two barriers per level,
  // dots of at most s products: 3k cycles for n = 24 (column by column, 31
  // dependent steps with shuffles, 17k).
  template <typename T>
  QTQP_PHASE void invert_diag_blocks(T* g) {
    QTQP_LOCALS;
    QTQP_TIC();
    const int nblk = (n + 31) >> 5;
#pragma unroll 1
    for (int ls = 0; ls < 5; ++ls) {
      const int s = 1 << ls;
#pragma unroll 1
      for (int half = 0; half < 2; ++half) {
#pragma unroll 1
        for (int e = tid; e < nblk << (4 + ls); e += NT) {
          // Element (i, j) of pair p of 32-block b.
          const int j = e & (s - 1), i = (e >> ls) & (s - 1);
          const int p = (e >> (2 * ls)) & ((16 >> ls) - 1), b = e >> (4 + ls);
          const int r0 = b * 32 + p * 2 * s;  // the pair's first row
          if (r0 + s + i >= n) continue;
          T* row = g + (r0 + s + i) * ldg + r0;   // row i of [L21 X22]
          T* up = g + (r0 + j) * ldg + r0 + s;    // T_kj at up[k]
          T a0 = T(0), a1 = T(0);
          if (half == 0) {  // T_ij = sum_{k >= j} L21_ik X11_kj
            const T* x = g + r0 * ldg + r0 + j;
            int k = j;
            for (; k + 1 < s; k += 2) {
              a0 = fma(row[k], x[k * ldg], a0);
              a1 = fma(row[k + 1], x[(k + 1) * ldg], a1);
            }
            if (k < s) a0 = fma(row[k], x[k * ldg], a0);
            up[i] = a0 + a1;
          } else {  // X21_ij = -sum_{k <= i} X22_ik T_kj
            int k = 0;
            for (; k < i; k += 2) {
              a0 = fma(row[s + k], up[k], a0);
              a1 = fma(row[s + k + 1], up[k + 1], a1);
            }
            if (k == i) a0 = fma(row[s + k], up[k], a0);
            row[j] = -(a0 + a1);
          }
        }
        sync();
      }
    }
    QTQP_TOC(kPhInv);
  }

  // Solves L L^T v = v in place with the block-inverted factor: forward
  // z_b = X_bb (v_b - sum_{c<b} L_bc z_c), backward x_b = X_bb^T (z_b -
  // sum_{c>b} L_cb^T x_c), two barriers per 32-block; w is n scratch entries.
  // Each phase is a set of dots with several lanes each (block_mv), so no
  // thread walks a 32-long chain alone.
  template <typename T>
  QTQP_PHASE void chol_solve(const T* g, T* v, T* w) {
    if constexpr (FMT == kFmtLarge) {
      large_chol_solve<T>(*this, v, w);
      return;
    }
    QTQP_LOCALS;
    const int nblk = (n + 31) >> 5;
#pragma unroll 1
    for (int blk = 0; blk < nblk; ++blk) {
      const int kb = blk * 32, bs = min(32, n - kb), rest = n - kb - bs;
      const T* gb = g + kb * ldg + kb;
      block_mv<T>(gb, ldg, 1, bs, bs, 1, v + kb, w + kb, false);
      if (rest > 0) block_mv<T>(gb + bs * ldg, ldg, 1, rest, bs, 0, w + kb, v + kb + bs, true);
    }
#pragma unroll 1
    for (int blk = nblk - 1; blk >= 0; --blk) {
      const int kb = blk * 32, bs = min(32, n - kb);
      const T* gb = g + kb * ldg + kb;
      block_mv<T>(gb, 1, ldg, bs, bs, 2, w + kb, v + kb, false);
      if (kb > 0) block_mv<T>(g + kb * ldg, 1, ldg, kb, bs, 0, v + kb, w, true);
    }
  }

  // out_k = sum_i M[k sk + i si] v_i (sub: out_k -= it) for k < K over i < len
  // (tri 0), i <= k (tri 1) or i >= k (tri 2), several lanes per output as in
  // rowdot, then a barrier.  One short copy for every step of a triangular
  // solve, for the instruction cache.
  template <typename T>
  QTQP_PHASE void block_mv(const T* M, int sk, int si, int K, int len, int tri, const T* v, T* out,
                           bool sub) {
    const int ls = lanes_log2(K), S = 1 << ls, per_warp = 32 >> ls;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int sl = lane >> (5 - ls), gl = lane & (per_warp - 1);
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += (NT / 32) * per_warp) {
      const int k = k0 + warp * per_warp + gl;
      const T* Mk = M + k * sk;
      const int i1 = tri == 1 ? min(len, k + 1) : len;
      T a0 = T(0), a1 = T(0);
      if (k < K) {
        int i = sl;
        if (tri == 2) i += (k - sl + S - 1) >> ls << ls;  // the first i >= k of this lane
        if (tri == 2 && i < sl) i = sl;
#pragma unroll 1
        for (; i + S < i1; i += 2 * S) {
          a0 = fma(Mk[i * si], v[i], a0);
          a1 = fma(Mk[(i + S) * si], v[i + S], a1);
        }
        if (i < i1) a0 = fma(Mk[i * si], v[i], a0);
      }
      a0 += a1;
#pragma unroll 1
      for (int off = 16; off >= per_warp; off >>= 1) a0 += __shfl_xor_sync(0xffffffffu, a0, off);
      if (k < K && sl == 0) out[k] = sub ? out[k] - a0 : a0;
    }
    sync();
  }

  // --------------------------------------------------------------------------
  // Backend solve (solvers_dense.py:130-142): out (+)= K_reg^{-1} r.
  // Entry: r complete (barrier passed).  Exit: out written (barrier needed
  // before other threads read it).
  // --------------------------------------------------------------------------
  QTQP_PHASE void kkt_solve(const double* r, double* out, bool accumulate, bool fp64) {
    if constexpr (kSparseA) {
      band_kkt_solve(r, out, accumulate, fp64);
      return;
    }
    QTQP_LOCALS;
    QTQP_TIC();
    const double* iry = vec(kPI);
    double* tmp = vec(kTMP);
    float* t32 = this->t32();
    const double* Ap = A;
    const int ld = lda, nn = n;
    // g = r_x + A^T (r_y / Ry)
    auto put_g = [&](int k, double g) {
      if (fp64) {
        tmp[k] = g;
      } else {
        t32[k] = float(g);
      }
    };
    // (In grid mode a lane group per column streams A with many loads in
    // flight; a row pass with per-block column sums measured slower here,
    // where no row dot rides along.)
    {
      QTQP_TIC();
      if constexpr (FMT == kFmtLarge) {
        large_products(*this, nullptr, r + n, iry + n, nullptr, [](int, double) {},
                       [&](int k, double cs) { put_g(k, r[k] + cs); });
      } else if (fused_ok()) {
        dense_products(nullptr, r + n, iry + n, nullptr, nullptr);
        sync();
        for (int k = tid; k < n; k += NT) put_g(k, r[k] + fused_colsum(k));
      } else {
        rowdot<1>(n, m,
                  [&](int k, int i, double* acc) {
                    acc[0] = fma(Ap[i * ld + k], iry[nn + i] * r[nn + i], acc[0]);
                  },
                  [&](int k, double* acc) { put_g(k, r[k] + acc[0]); });
      }
      sync();
      QTQP_TOC(kPhSolveCols);
    }
    {
      QTQP_TIC();
      if (fp64) {
        chol_solve<double>(G, tmp, vec(kW));
      } else {
        chol_solve<float>(g32(), t32, t32 + n);
      }
      QTQP_TOC(kPhTri);
    }
    for (int k = tid; k < n; k += NT) {
      const double val = fp64 ? tmp[k] : double(t32[k]);
      out[k] = accumulate ? out[k] + val : val;
      if (fused_ok() && !fp64) tmp[k] = val;
    }
    // y = (A x - r_y) / Ry
    if (fused_ok()) {
      QTQP_TIC();
      if (!fp64) sync();  // the converted x
      dense_products(tmp, nullptr, nullptr, nullptr, tmp + n);
      sync();
      for (int k = own(n); k < N; k += NT) {
        const double val = iry[k] * (tmp[k] - r[k]);
        out[k] = accumulate ? out[k] + val : val;
      }
      QTQP_TOC(kPhSolveRows);
    } else {
      QTQP_TIC();
      rowdot<1, false, kRowS>(m, n,
                [&](int k, int j, double* acc) {
                  const double xj = fp64 ? tmp[j] : double(t32[j]);
                  acc[0] = fma(Ap[k * ld + j], xj, acc[0]);
                },
                [&](int k, double* acc) {
                  const double val = iry[nn + k] * (acc[0] - r[nn + k]);
                  out[nn + k] = accumulate ? out[nn + k] + val : val;
                });
      QTQP_TOC(kPhSolveRows);
    }
    QTQP_TOC(kPhSolve);
  }

  // The products of a dense block for n <= 64, each from one coalesced pass
  // over A (and P): with wy, the column sums c_k = sum_{i<m} A_ik wy_i (ws_i)
  // + sum_{i<n} P_ik wp_i (k < n; wy, ws, wp may be null), staged per warp in
  // the panel buffer PB (PB[w * n + k]; fused_colsum adds the warps' rows after
  // a barrier); with vx, the row products (A vx)_i into rows_out[i].  A warp
  // takes 4, 8 or 16 rows at a time, lane l columns l and l + 32 (n <= 32: eight
  // rows, column l), their loads issued first; the row sums are reduced across the
  // warp, the first steps sending half of the values to the partner lane and
  // keeping the other half.  Ends without a barrier.
  //
  // What bounds these small solves is instruction fetch: code that an
  // iteration runs once through costs about 0.4 cycles per byte whatever it
  // does (one n = 24 QP alone on an SM spent 5.7k cycles per residual), loops
  // whose body stays in the nearest instruction cache next to nothing.  So one
  // short loop, in one copy, serves the residual, both products of a KKT
  // solve, the tau equations and the termination test.
  static constexpr bool kFused = FMT == kFmtDense && NT <= 1024;
  __device__ __forceinline__ bool fused_ok() const { return kFused && n <= 64; }
  QTQP_PHASE void dense_products(const double* vx, const double* wy, const double* ws,
                                 const double* wp, double* rows_out) const {
    QTQP_LOCALS;
    constexpr int NW = NT / 32;
    const int lane = tid & 31, warp = tid >> 5;
    const int c0 = lane, c1 = lane + 32;
    const bool ok0 = c0 < n, ok1 = c1 < n;
    double cs0 = 0.0, cs1 = 0.0;
    if (n <= 32) {
      // One column per lane, eight rows at a time: half the rounds of latency of
      // the two-column loop below, which left lone small QPs slower than row dots
      // (n = 16, m = 33, one QP in us: row dots 632, two columns 652, this 600).
      if (vx != nullptr || wy != nullptr) {
        const double x0 = ok0 && vx != nullptr ? vx[c0] : 0.0;
        const int rsel = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
#pragma unroll 1
        for (int base = warp * 8; base < m; base += NW * 8) {
          double t[8];
#pragma unroll
          for (int r = 0; r < 8; ++r) t[r] = base + r < m && ok0 ? A[(base + r) * lda + c0] : 0.0;
          if (wy != nullptr) {
#pragma unroll
            for (int r = 0; r < 8; ++r) {
              const int i = min(base + r, m - 1);  // rows from m on hold zeros
              cs0 = fma(t[r], ws != nullptr ? ws[i] * wy[i] : wy[i], cs0);
            }
          }
          if (vx != nullptr) {
#pragma unroll
            for (int r = 0; r < 8; ++r) t[r] *= x0;
#pragma unroll
            for (int half = 4, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
              const bool hi = (lane & bit) != 0;
#pragma unroll
              for (int j = 0; j < half; ++j) {
                const double send = hi ? t[j] : t[j + half];
                const double keep = hi ? t[j + half] : t[j];
                t[j] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
              }
            }
#pragma unroll
            for (int bit = 2; bit >= 1; bit >>= 1) t[0] += __shfl_xor_sync(0xffffffffu, t[0], bit);
            if ((lane & 3) == 0 && base + rsel < m) rows_out[base + rsel] = t[0];
          }
        }
      }
      if (wp != nullptr) {
#pragma unroll 1
        for (int i0 = warp; i0 < n; i0 += 8 * NW) {
          double p0[8];
#pragma unroll
          for (int u = 0; u < 8; ++u)
            p0[u] = i0 + u * NW < n && ok0 ? P[(i0 + u * NW) * ldp + c0] : 0.0;
#pragma unroll
          for (int u = 0; u < 8; ++u) cs0 = fma(p0[u], wp[min(i0 + u * NW, n - 1)], cs0);
        }
      }
    } else {
      // RB rows per warp and round: few rows are short code, many rows few rounds of
      // latency.  100 QPs with n = 48..50, m = 2n on four warps, mixed precision, in
      // ms: 4 rows a round 3.07, 8 rows 2.98, 16 rows 2.78; n = 44: 2.72, 2.56, 2.66;
      // n = 34: 4 rows 2.37 (1000 QPs of n = 8..40 lost 7 % with 16 rows for all).
      auto rows_of_a = [&](auto rb) {
        constexpr int RB = decltype(rb)::value;
        const double x0 = ok0 && vx != nullptr ? vx[c0] : 0.0;
        const double x1 = ok1 && vx != nullptr ? vx[c1] : 0.0;
        // The row a lane ends with: its top bits, after log2(RB) halving steps.
        int rsel = 0;
#pragma unroll
        for (int half = RB / 2, bit = 16; half >= 1; half >>= 1, bit >>= 1)
          rsel += (lane & bit) != 0 ? half : 0;
#pragma unroll 1
        for (int base = warp * RB; base < m; base += NW * RB) {
          double t[RB], a1[RB];
#pragma unroll
          for (int r = 0; r < RB; ++r) {
            const double* row = A + (base + r) * lda;
            const bool in = base + r < m;
            t[r] = in && ok0 ? row[c0] : 0.0;
            a1[r] = in && ok1 ? row[c1] : 0.0;
          }
          if (wy != nullptr) {
#pragma unroll
            for (int r = 0; r < RB; ++r) {
              const int i = min(base + r, m - 1);  // rows from m on hold zeros
              const double w = ws != nullptr ? ws[i] * wy[i] : wy[i];
              cs0 = fma(t[r], w, cs0);
              cs1 = fma(a1[r], w, cs1);
            }
          }
          if (vx != nullptr) {
#pragma unroll
            for (int r = 0; r < RB; ++r) t[r] = fma(t[r], x0, a1[r] * x1);
#pragma unroll
            for (int half = RB / 2, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
              const bool hi = (lane & bit) != 0;
#pragma unroll
              for (int j = 0; j < half; ++j) {
                const double send = hi ? t[j] : t[j + half];
                const double keep = hi ? t[j + half] : t[j];
                t[j] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
              }
            }
#pragma unroll
            for (int bit = 16 / RB; bit >= 1; bit >>= 1)
              t[0] += __shfl_xor_sync(0xffffffffu, t[0], bit);
            if ((lane & (32 / RB - 1)) == 0 && base + rsel < m) rows_out[base + rsel] = t[0];
          }
        }
      };
      if (vx != nullptr || wy != nullptr) {
        if (m > 24 * NW) {
          rows_of_a(std::integral_constant<int, 16>());
        } else if (m > 20 * NW) {
          rows_of_a(std::integral_constant<int, 8>());
        } else {
          rows_of_a(std::integral_constant<int, 4>());
        }
      }
      if (wp != nullptr) {
#pragma unroll 1
        for (int i0 = warp; i0 < n; i0 += 4 * NW) {
          double p0[4], p1[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const int i = i0 + u * NW;
            const double* row = P + i * ldp;
            p0[u] = i < n && ok0 ? row[c0] : 0.0;
            p1[u] = i < n && ok1 ? row[c1] : 0.0;
          }
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const double w = wp[min(i0 + u * NW, n - 1)];
            cs0 = fma(p0[u], w, cs0);
            cs1 = fma(p1[u], w, cs1);
          }
        }
      }
    }
    if (wy != nullptr || wp != nullptr) {
      double* stage = PB + warp * n;
      if (ok0) stage[c0] = cs0;
      if (ok1) stage[c1] = cs1;
    }
  }
  // Column sum k of dense_products (after a barrier).
  __device__ __forceinline__ double fused_colsum(int k) const {
    constexpr int NW = NT / 32;
    double t = 0.0;
#pragma unroll
    for (int w = 0; w < NW; ++w) t += PB[w * n + k];
    return t;
  }

  // res = krhs - K_reg v + corr o v (direct.py:256, 266 with the matvec of
  // solvers_dense.py:118-128).  Reads all of v; returns this thread's partial
  // max |res| and NaN flag of v (combined by the caller's reduction).
  QTQP_PHASE void kkt_residual(const double* v, const double* krhs, double* res, double& mres,
                               double& vnan) const {
    if constexpr (kSparseA) {
      band_kkt_residual(v, krhs, res, mres, vnan);
      return;
    }
    QTQP_LOCALS;
    if (fused_ok()) {
      const double* reg = vec(kREG);
      const double* corr = vec(kCORR);
      dense_products(v, v + n, nullptr, has_p ? v : nullptr, res + n);
      sync();
      for (int k = tid; k < N; k += NT) {
        const double kv = k < n ? fused_colsum(k) + reg[k] * v[k] : res[k] - (-reg[k]) * v[k];
        const double rk = krhs[k] - kv + corr[k] * v[k];
        res[k] = rk;
        mres = nanmax(mres, fabs(rk));
        vnan = fmax(vnan, (v[k] != v[k]) ? 1.0 : 0.0);
      }
      return;
    }
    const double* reg = vec(kREG);
    const double* corr = vec(kCORR);
    if constexpr (FMT == kFmtLarge) {
      // One pass over A (and P): row dots A v_x and column sums
      // A^T v_y + P v_x (large_ipm.cuh); the column epilogue runs after a
      // grid barrier, in the thread that owns column k.
      const int nn = n;
      large_products(*this, v, v + n, nullptr, has_p ? v : nullptr,
                     [&](int i, double ax) {
                       const int kk = nn + i;
                       const double kv = ax - (-reg[kk]) * v[kk];
                       const double rk = krhs[kk] - kv + corr[kk] * v[kk];
                       res[kk] = rk;
                       mres = nanmax(mres, fabs(rk));
                       vnan = fmax(vnan, (v[kk] != v[kk]) ? 1.0 : 0.0);
                     },
                     [&](int k, double cs) {
                       const double kv = cs + reg[k] * v[k];
                       const double rk = krhs[k] - kv + corr[k] * v[k];
                       res[k] = rk;
                       mres = nanmax(mres, fabs(rk));
                       vnan = fmax(vnan, (v[k] != v[k]) ? 1.0 : 0.0);
                     });
      return;
    }
    const double* Ap = A;
    const double* Pp = P;
    const int la = lda, lp = ldp, nn = n, mm = m;
    const int plen = has_p ? n : 0;
    rowdot<2>(n, m + plen,
              [&](int k, int i, double* acc) {
                if (i < mm) {
                  acc[1] = fma(Ap[i * la + k], v[nn + i], acc[1]);
                } else {
                  acc[0] = fma(Pp[(i - mm) * lp + k], v[i - mm], acc[0]);
                }
              },
              [&](int k, double* acc) {
                double t = acc[0];
                t += reg[k] * v[k];
                const double kv = t + acc[1];
                const double rk = krhs[k] - kv + corr[k] * v[k];
                res[k] = rk;
                mres = nanmax(mres, fabs(rk));
                vnan = fmax(vnan, (v[k] != v[k]) ? 1.0 : 0.0);
              });
    rowdot<1, false, kRowS>(m, n,
              [&](int k, int j, double* acc) { acc[0] = fma(Ap[k * la + j], v[j], acc[0]); },
              [&](int k, double* acc) {
                const int kk = nn + k;
                const double kv = acc[0] - (-reg[kk]) * v[kk];
                const double rk = krhs[kk] - kv + corr[kk] * v[kk];
                res[kk] = rk;
                mres = nanmax(mres, fabs(rk));
                vnan = fmax(vnan, (v[kk] != v[kk]) ? 1.0 : 0.0);
              });
  }

  // K_reg x (solvers_dense.py:118-128), written to out.
  __device__ void kkt_matvec(const double* v, double* out) const {
    QTQP_LOCALS;
    const double* reg = vec(kREG);
    const double* Ap = A;
    const double* Pp = P;
    const int la = lda, lp = ldp, nn = n, mm = m;
    rowdot<2>(n, m + n,
              [&](int k, int i, double* acc) {
                if (i < mm) {
                  acc[1] = fma(Ap[i * la + k], v[nn + i], acc[1]);
                } else {
                  acc[0] = fma(Pp[(i - mm) * lp + k], v[i - mm], acc[0]);
                }
              },
              [&](int k, double* acc) {
                double t = acc[0];
                t += reg[k] * v[k];
                out[k] = t + acc[1];
              });
    rowdot<1>(m, n,
              [&](int k, int j, double* acc) { acc[0] = fma(Ap[k * la + j], v[j], acc[0]); },
              [&](int k, double* acc) { out[nn + k] = acc[0] - (-reg[nn + k]) * v[nn + k]; });
  }

  // The KKT right-hand side of a solve into vec(kRHS): krhs[k] = rhs_k(k),
  // negated on the dual block (k >= n), owner-wise (k % NT == tid).
  template <typename RhsF>
  __device__ __forceinline__ void set_rhs(RhsF rhs_k) {
    double* krhs = vec(kRHS);
    for (int k = tid; k < N; k += NT) {
      const double r = rhs_k(k);
      krhs[k] = k >= n ? -r : r;
    }
  }

  // --------------------------------------------------------------------------
  // DirectKktSolver.solve (direct.py:218-307).  The right-hand side is in
  // vec(kRHS) (set_rhs, written owner-wise by this thread); `sol` holds the
  // warm start and receives the solution.  Entry: sol complete (barrier
  // passed).  One copy of this function serves every solve of an iteration,
  // which keeps the per-iteration code small for the instruction cache.
  // --------------------------------------------------------------------------
  QTQP_PHASE IrOutcome ir_solve(double* sol, bool fp64) {
    const qtqp_options& op = *o;
    const double* krhs = vec(kRHS);
    double* res = vec(kRES);
    double dummy[1] = {0.0};
    IrOutcome out;
    {
      double mx[3] = {0.0, 0.0, 0.0};  // |rhs|, |res|, nan(sol)
      for (int k = tid; k < N; k += NT) mx[0] = nanmax(mx[0], fabs(krhs[k]));
      sync();
      QTQP_TIC();
      kkt_residual(sol, krhs, res, mx[1], mx[2]);
      // The reduction's barrier also orders every thread's res writes before
      // the solve that reads them.
      reduce<0, 3>(dummy, mx);
      if constexpr (NT <= 1024) {
        if (NT / 32 == 1) sync();  // a one-warp reduction has no barrier
      } else {
        sync();
      }
      QTQP_TOC(kPhResidual);
      out.rhs_norm = mx[0];
      out.final_res = mx[1];
    }
    out.tol = op.linear_solver_atol + op.linear_solver_rtol * out.rhs_norm;
    out.status = 0;
    out.solves = 0;
    out.nan = false;
    double rn = out.final_res;
    for (int it = 1; it <= op.max_iterative_refinement_steps; ++it) {
      out.solves = it;
      const double prev = rn;
      kkt_solve(res, sol, true, fp64);
      sync();
      QTQP_TIC();
      double mx[2] = {0.0, 0.0};
      kkt_residual(sol, krhs, res, mx[0], mx[1]);
      reduce<0, 2>(dummy, mx);  // its barrier orders the res writes (as above)
      if constexpr (NT <= 1024) {
        if (NT / 32 == 1) sync();
      } else {
        sync();
      }
      QTQP_TOC(kPhResidual);
      rn = mx[0];
      out.nan = mx[1] > 0.0;
      if (rn < out.tol) {
        out.status = 1;
        break;
      }
      if (rn >= prev) {
        out.status = 2;
        break;
      }
    }
    out.final_res = rn;
    return out;
  }

  // IR with the mixed-precision policy: an FP32 factor whose refinement does
  // not converge is replaced by an FP64 factor (kept for the rest of the
  // solve) and the refinement is redone from the same warm start, so the
  // outcome is the one the plain FP64 path would produce.
  // `warm` is the warm start (a vector that the solve leaves unchanged); the
  // right-hand side is set once and kept in vec(kRHS) for the second try.
  template <typename RhsF>
  __device__ IrOutcome ir_solve_policy(RhsF rhs_k, const double* warm, double* sol, bool& fp64,
                                       int& n32, int& n64, int& err) {
    set_rhs(rhs_k);
    for (int k = tid; k < N; k += NT) sol[k] = warm[k];
    sync();
    IrOutcome r = ir_solve(sol, fp64);
    if (!fp64 && r.status != 1) {
      fp64 = true;
      ++n64;
      const int info = factorize<double>();
      if (info != 0) {
        err = QTQP_ERR_NOT_SPD;
        return r;
      }
      for (int k = tid; k < N; k += NT) sol[k] = warm[k];
      sync();
      r = ir_solve(sol, fp64);
    }
    return r;
  }

  // --------------------------------------------------------------------------
  // tau+ of the homogeneous embedding: the quadratic root
  // (__init__.py:759-817) or, when the KKT solve was not accurate or the
  // quadratic fails, the linearised update (__init__.py:819-857).
  // `kr` is K^{-1} r (complete).  Per-iteration constants come in `it`.
  // --------------------------------------------------------------------------
  struct IterConsts {
    double kqq;    // K^{-1}q . q
    double kqpkq;  // (K^{-1}q)_x . P (K^{-1}q)_x
    double qz;     // q_x . x + q_y . y
    double xpx;    // x . P x
    double pxkq;   // P x . (K^{-1}q)_x
  };

  QTQP_PHASE double tau_step(const double* kr, const IrOutcome& irr, double mu, double mu_t,
                             double r_tau, double tau, double tau_anchor, const IterConsts& ic,
                             int& method) {
    QTQP_LOCALS;
    const double* q = vec(kQ);
    const double* kq = vec(kKQ);
    const double* pkq = vec(kPW);
    const double* px = vec(kXD);
    const double* pi = vec(kPI);
    double* pkr = vec(kRS);
    double sm[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // kr.q, kr.Pkq, kq.Pkr, kr.Pkr, Px.kr
    double dummy[1] = {0.0};
    for (int k = sum_own(0); k < N; k += kSumT) sm[0] = fma(kr[k], q[k], sm[0]);
    if (has_p) {
      auto add = [&](int k, double t) {
        sm[1] = fma(kr[k], pkq[k], sm[1]);
        sm[2] = fma(kq[k], t, sm[2]);
        sm[3] = fma(kr[k], t, sm[3]);
        sm[4] = fma(px[k], kr[k], sm[4]);
      };
      auto epi = [&](int k, double poff) {
        const double t = fma(pi[k], kr[k], poff);
        pkr[k] = t;
        if constexpr (kSumT == NT) add(k, t);
      };
      if constexpr (kSparseA) {
        for (int k = tid; k < n; k += NT) epi(k, band_poff_row(kr, k));
        if constexpr (kSumT != NT) {
          sync();
          for (int k = sum_own(0); k < n; k += kSumT) add(k, pkr[k]);
        }
      } else if (fused_ok()) {
        dense_products(nullptr, nullptr, nullptr, kr, nullptr);
        sync();
        for (int k = tid; k < n; k += NT) epi(k, fused_colsum(k));
      } else {
        const double* Pp = P;
        const int lp = ldp;
        rowdot<1>(n, n,
                  [&](int k, int j, double* acc) { acc[0] = fma(Pp[j * lp + k], kr[j], acc[0]); },
                  [&](int k, double* acc) { epi(k, acc[0]); });
      }
    }
    reduce<5, 0>(sm, dummy);
    const bool accurate = irr.status == 1 || irr.final_res < 1e-7;
    if (o->tau_mode == 0 && accurate) {
      double ta = mu + ic.kqq;
      double tb = -r_tau - sm[0];
      double tc = -mu_t;
      if (has_p) {
        ta -= ic.kqpkq;
        tb += sm[1] + sm[2];
        tc -= sm[3];
      }
      double root = 0.0;
      bool ok = true;
      if (fabs(ta) < kEps) {
        if (fabs(tb) < kEps) {
          ok = false;
        } else {
          root = -tc / tb;
          ok = isfinite(root) && !(root < -1e-10);
        }
      } else {
        double disc = tb * tb - 4.0 * ta * tc;
        if (disc < -1e-9) {
          ok = false;
        } else {
          disc = fmax(0.0, disc);
          if (tb > 0.0) {
            root = tc / (-0.5 * (tb + sqrt(disc)));
          } else {
            root = (-0.5 * (tb - sqrt(disc))) / ta;
          }
          ok = isfinite(root) && !(root < -1e-10);
        }
      }
      if (ok) {
        method = 0;
        return fmax(0.0, root);
      }
    }
    method = 1;
    const double q_rz = sm[0] - tau * ic.kqq - ic.qz;
    const double px_rz = (has_p ? sm[4] : 0.0) - tau * ic.pxkq - ic.xpx;
    const double g = mu * tau * tau + (mu_t - mu) * tau_anchor * tau - tau * ic.qz - mu_t - ic.xpx;
    const double num = g - tau * q_rz - 2.0 * px_rz;
    const double den =
        2.0 * mu * tau + (mu_t - mu) * tau_anchor - ic.qz + tau * ic.kqq + 2.0 * ic.pxkq;
    const double root = tau + (fabs(den) < 1e-16 ? 0.0 : -num / den);
    if (!isfinite(root)) return tau;
    return fmin(fmax(root, 0.1 * tau), 10.0 * tau);
  }

  // Ratio test (__init__.py:671-680, 882-886) over the inequality block for
  // the step (dy, ds) given owner-wise by `dir(k, dy, ds)`.
  template <typename DirF>
  __device__ double step_to_boundary(DirF dir) {
    QTQP_LOCALS;
    const double* xy = vec(kXY);
    const double* s = vec(kRS);
    double mx[1] = {-1.0};  // max of -alpha candidates == -(min alpha)
    double dummy[1] = {0.0};
    for (int k = own(n + z); k < N; k += NT) {
      double dy, ds;
      dir(k, dy, ds);
      if (ds < -kEps) mx[0] = fmax(mx[0], -(-s[k] / ds));
      if (dy < -kEps) mx[0] = fmax(mx[0], -(-xy[k] / dy));
    }
    reduce<0, 1>(dummy, mx);
    return fmin(1.0, -mx[0]);
  }

  // --------------------------------------------------------------------------
  // _check_termination (__init__.py:888-1008) on the unequilibrated iterate,
  // computed from the equilibrated products: A_o x_o = (A_eq x)/d,
  // A_o^T y_o = (A_eq^T y)/e, P_o x_o = (P_eq x)/e.
  // --------------------------------------------------------------------------
  QTQP_PHASE int termination(double tau, double nb, double nc, double* st, bool collect) {
    QTQP_LOCALS;
    const qtqp_options& op = *o;
    const double* xy = vec(kXY);
    const double* s = vec(kRS);
    const double* de = vec(kDE);
    const double* pi = vec(kPI);
    const double inv_tau = 1.0 / fmax(tau, kEps);
    // sums: ctx, bty, xpx ; maxes: pres, dres, |aty|, |px|, |ax+s|, |ax|, |s|, |x|, |y|
    double sm[3] = {0.0, 0.0, 0.0};
    double mx[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    const double* Ap = A;
    const double* Pp = P;
    const int la = lda, lp = ldp, nn = n, mm = m;
    const int plen = has_p ? n : 0;
    const bool hp = has_p;
    const double* b0p = b0;
    const double* c0p = c0;
    double* const xy_o = vec(kRES);
    double* const px_o = vec(kTMP);
    auto epi_x = [&](int k, double aty_raw, double poff) {
      const double aty = aty_raw / de[k];
      const double px = hp ? fma(pi[k], xy[k], poff) / de[k] : 0.0;
      const double xo = de[k] * xy[k];
      if constexpr (kSumT == NT) {
        sm[0] = fma(c0p[k], xo, sm[0]);
        sm[2] = fma(xo, px, sm[2]);
      } else {  // summed below (the residual and the solve's scratch are free here)
        xy_o[k] = xo;
        px_o[k] = px;
      }
      mx[1] = nanmax(mx[1], fabs((px + aty) * inv_tau + c0p[k]));
      mx[2] = nanmax(mx[2], fabs(aty));
      mx[3] = nanmax(mx[3], fabs(px));
      mx[7] = nanmax(mx[7], fabs(xo));
    };
    auto epi_y = [&](int k, double ax_raw) {
      const int kk = nn + k;
      const double ax = ax_raw / de[kk];
      const double yo = de[kk] * xy[kk];
      const double so = s[kk] / de[kk];
      const double bo = b0p[k];
      if constexpr (kSumT == NT) {
        sm[1] = fma(bo, yo, sm[1]);
      } else {
        xy_o[kk] = yo;
      }
      mx[0] = nanmax(mx[0], fabs((ax + so) * inv_tau - bo));
      mx[4] = nanmax(mx[4], fabs(ax + so));
      mx[5] = nanmax(mx[5], fabs(ax));
      mx[6] = nanmax(mx[6], fabs(so));
      mx[8] = nanmax(mx[8], fabs(yo));
    };
    if constexpr (kSparseA) {
      for (int k = tid; k < n; k += NT) epi_x(k, band_at_col(xy, k), band_poff_row(xy, k));
      for (int k = tid; k < m; k += NT) epi_y(k, band_a_row(xy, k));
      if constexpr (kSumT != NT) {
        sync();
        for (int k = sum_own(0); k < n; k += kSumT) {
          sm[0] = fma(c0p[k], xy_o[k], sm[0]);
          sm[2] = fma(xy_o[k], px_o[k], sm[2]);
        }
        for (int k = sum_own(0); k < m; k += kSumT) sm[1] = fma(b0p[k], xy_o[nn + k], sm[1]);
      }
    } else if (fused_ok()) {
      // P x, then A^T y and A x in one pass over A (the residual's vector is
      // free here).
      double* pxs = vec(kRES);
      double* axs = vec(kRES) + n;
      if (hp) {
        dense_products(nullptr, nullptr, nullptr, xy, nullptr);
        sync();
        for (int k = tid; k < n; k += NT) pxs[k] = fused_colsum(k);
        sync();
      }
      dense_products(xy, xy + nn, nullptr, nullptr, axs);
      sync();
      for (int k = tid; k < n; k += NT) epi_x(k, fused_colsum(k), hp ? pxs[k] : 0.0);
      for (int k = own(n) - n; k < m; k += NT) epi_y(k, axs[k]);
    } else {
      rowdot<2>(n, m + plen,
                [&](int k, int i, double* acc) {
                  if (i < mm) {
                    acc[0] = fma(Ap[i * la + k], xy[nn + i], acc[0]);
                  } else {
                    acc[1] = fma(Pp[(i - mm) * lp + k], xy[i - mm], acc[1]);
                  }
                },
                [&](int k, double* acc) { epi_x(k, acc[0], acc[1]); });
      rowdot<1, false, kRowS>(m, n, [&](int k, int j, double* acc) { acc[0] = fma(Ap[k * la + j], xy[j], acc[0]); },
                [&](int k, double* acc) { epi_y(k, acc[0]); });
    }
    reduce<3, 9>(sm, mx);
    const double ctx = sm[0], bty = sm[1], xpx = has_p ? sm[2] : 0.0;
    const double pcost = (ctx + 0.5 * xpx * inv_tau) * inv_tau;
    const double dcost = (-bty - 0.5 * xpx * inv_tau) * inv_tau;
    const double pres = mx[0], dres = mx[1];
    const double gap = fabs((ctx + bty + xpx * inv_tau) * inv_tau);
    const double norm_aty = mx[2], norm_px = mx[3];
    const double dinf_a = mx[4] / (fabs(ctx) + kEps);
    const double dinf_p = norm_px / (fabs(ctx) + kEps);
    const double dinf = fmax(dinf_a, dinf_p);
    const double pinf = norm_aty / (fabs(bty) + kEps);
    const double prel = fmax(fmax(mx[5] * inv_tau, mx[6] * inv_tau), nb);
    const double drel = fmax(fmax(norm_px * inv_tau, norm_aty * inv_tau), nc);
    const double nx = mx[7], ny = mx[8];
    int status;
    if (gap < op.atol + op.rtol * fmin(fabs(pcost), fabs(dcost)) &&
        pres < op.atol + op.rtol * prel && dres < op.atol + op.rtol * drel) {
      status = QTQP_STATUS_SOLVED;
    } else if (ctx < -kEps && dinf < op.atol_infeas + op.rtol_infeas * nx / fabs(ctx)) {
      status = QTQP_STATUS_UNBOUNDED;
    } else if (bty < -kEps && pinf < op.atol_infeas + op.rtol_infeas * ny / fabs(bty)) {
      status = QTQP_STATUS_INFEASIBLE;
    } else {
      status = QTQP_STATUS_UNFINISHED;
    }
    if (st != nullptr && tid == 0) {
      st[kStCtx] = ctx;
      st[kStBty] = bty;
      st[kStPcost] = pcost;
      st[kStDcost] = dcost;
      st[kStPres] = pres;
      st[kStDres] = dres;
      st[kStGap] = gap;
      st[kStPinfeas] = pinf;
      st[kStDinfeas] = dinf;
      st[kStDinfeasA] = dinf_a;
      st[kStDinfeasP] = dinf_p;
      st[kStNormX] = nx;
      st[kStNormY] = ny;
      st[kStStatus] = status;
      st[kStPrel] = prel;
      st[kStDrel] = drel;
    }
    if (collect && st != nullptr) {
      // collect_stats extras (__init__.py:992-1007): complementarity, norm_s
      // and the per-inequality statistics of s*y and s/y.
      double a[5] = {0, 0, 0, 0, 0};  // y.s, sum sy, sum s/y
      double b[5] = {0, 0, -INFINITY, 0, 0};  // max sy, max -sy, max soy, max -soy
      b[0] = -INFINITY;
      b[1] = -INFINITY;
      b[3] = -INFINITY;
      for (int k = sum_own(n); k < N; k += kSumT) {
        const double yo = de[k] * xy[k], so = s[k] / de[k];
        a[0] = fma(yo, so, a[0]);
        if (k >= n + z) {
          const double sy = so * yo, soy = so / fmax(kEps, yo);
          a[1] += sy;
          a[2] += soy;
          b[0] = fmax(b[0], sy);
          b[1] = fmax(b[1], -sy);
          b[2] = fmax(b[2], soy);
          b[3] = fmax(b[3], -soy);
        }
      }
      reduce<5, 5>(a, b);
      const int cnt = m - z;
      const double mean_sy = a[1] / cnt, mean_soy = a[2] / cnt;
      double v[2] = {0, 0};
      double dummy[1] = {0};
      for (int k = sum_own(n + z); k < N; k += kSumT) {
        const double yo = de[k] * xy[k], so = s[k] / de[k];
        const double sy = so * yo, soy = so / fmax(kEps, yo);
        v[0] += (sy - mean_sy) * (sy - mean_sy);
        v[1] += (soy - mean_soy) * (soy - mean_soy);
      }
      reduce<2, 0>(v, dummy);
      if (tid == 0) {
        st[kStCompl] = fabs(a[0] * inv_tau * inv_tau);
        st[kStNormS] = mx[6];
        st[kStMaxSy] = b[0];
        st[kStMinSy] = -b[1];
        st[kStStdSy] = sqrt(v[0] / cnt);
        st[kStMaxSoy] = b[2];
        st[kStMinSoy] = -b[3];
        st[kStMeanSoy] = mean_soy;
        st[kStStdSoy] = sqrt(v[1] / cnt);
      }
    }
    last_pcost = pcost;
    last_dcost = dcost;
    last_pres = pres;
    last_dres = dres;
    last_gap = gap;
    return status;
  }
  double last_pcost = 0, last_dcost = 0, last_pres = 0, last_dres = 0, last_gap = 0;

  __device__ void write_lin_stats(double* st, int block, const IrOutcome& r, int tau_method,
                                  bool fp64) const {
    if (st == nullptr || tid != 0) return;
    double* b = st + kStLin0 + block * kLinFields;
    b[kLinSolves] = r.solves;
    b[kLinFinalRes] = r.final_res;
    b[kLinRhsNorm] = r.rhs_norm;
    b[kLinTol] = r.tol;
    b[kLinStatus] = r.status;
    b[kLinTau] = tau_method;
    b[kLinPrec] = fp64 ? 64 : 32;
  }

  // out[n + i] = (A v)_i (equilibrated A).  Exit: needs a barrier before
  // other threads read out.
  __device__ void a_times(const double* v, double* out) const {
    if constexpr (kSparseA) {
      for (int k = own(n); k < N; k += NT) out[k] = band_a_row(v, k - n);
    } else {
      const double* Ap = A;
      const int la = lda, nn = n;
      rowdot<1, false, kRowS>(m, n, [&](int k, int j, double* acc) { acc[0] = fma(Ap[k * la + j], v[j], acc[0]); },
                [&](int k, double* acc) { out[nn + k] = acc[0]; });
    }
  }

  // --------------------------------------------------------------------------
  // Learned warm start (no reference counterpart).  Given a predicted point
  // (wx, wy) in the original scaling and a predicted active set (act[i] for
  // the inequality rows), solve the KKT system of the equality QP
  //   min 1/2 x'Px + c'x  s.t.  a_i x = b_i for i < z or i active
  // (free rows carry a huge D, i.e. y_i = 0) by the IPM's own regularised
  // factorisation and FP64 refinement; then y_i = 0 on free rows and
  // s = b - A x.  Each solution is projected onto the cone (y[z:] >= 0,
  // s[z:] >= 0) and accepted only if the plain termination test reports
  // SOLVED for it at tau = 1.  Up to options.warm_corrections primal-dual
  // active-set corrections may follow a rejected solution (tight rows whose
  // dual came out negative leave, free rows whose slack came out negative
  // enter, and the reduced system is solved again) while the set changes;
  // 0 keeps exactly one reduced solve.  On false the caller runs the plain
  // method from its usual starting point.
  // --------------------------------------------------------------------------
  __device__ bool warm_try(const double* wx, const double* wy, const unsigned char* act,
                           double nb, double nc, bool& fp64, int& n32, int& n64, int& nsolves) {
    const qtqp_options& op = *o;
    double* xy = vec(kXY);
    double* s = vec(kRS);
    double* xyc = vec(kXYC);
    double* reg = vec(kREG);
    double* corr = vec(kCORR);
    double* pi = vec(kPI);
    double* pw = vec(kPW);
    double* tight = vec(kCT);  // at [n, N): 1.0 where the row is held tight
    const double* de = vec(kDE);
    const double* q = vec(kQ);
    const double dmin = fmax(op.min_static_regularization, 1e-10);
    const double big = 1e10;
    for (int k = tid; k < N; k += NT) {
      if (k < n) {
        xy[k] = wx[k] / de[k];
      } else {
        const int i = k - n;
        tight[k] = (i < z || act[i] != 0) ? 1.0 : 0.0;
        xy[k] = wy[i] / de[k];
      }
    }
    double dummy[1] = {0.0};
    const int rounds = 1 + max(0, min(op.warm_corrections, 64));
    for (int round = 0; round < rounds; ++round) {
      for (int k = tid; k < N; k += NT) {
        if (k < n) {
          const double t = pi[k];
          const double r = fmax(t, op.min_static_regularization);
          reg[k] = r;
          corr[k] = r - t;
        } else {
          const bool tk = tight[k] != 0.0;
          const double t = -(tk ? 0.0 : big), r = -(tk ? dmin : big);
          reg[k] = r;
          corr[k] = r - t;
          pi[k] = 1.0 / (-r);
          pw[k] = 1.0 / sqrt(-r);
        }
      }
      sync();
      int info;
      if (fp64) {
        ++n64;
        info = factorize<double>();
      } else {
        ++n32;
        info = factorize<float>();
        if (info != 0) {
          fp64 = true;
          ++n64;
          info = factorize<double>();
        }
      }
      if (info != 0) return false;  // not an error of the problem: fall back
      int err = 0;
      IrOutcome r = ir_solve_policy([&](int k) { return -q[k]; }, xy,
                                    xyc, fp64, n32, n64, err);
      nsolves += r.solves;
      if (err || r.nan) return false;
      a_times(xyc, s);  // s[n + i] = (A x)_i
      sync();
      double v[1] = {0.0};  // 1 when a row changes
      for (int k = tid; k < N; k += NT) {
        if (k < n) {
          xy[k] = xyc[k];
          continue;
        }
        const int i = k - n;
        const double sk = q[k] - s[k];
        if (i < z) {
          xy[k] = xyc[k];
          s[k] = 0.0;
        } else if (tight[k] != 0.0) {
          xy[k] = fmax(xyc[k], 0.0);
          if (xyc[k] < 0.0) {
            tight[k] = 0.0;
            v[0] = 1.0;
          }
          s[k] = fmax(sk, 0.0);
        } else {
          xy[k] = 0.0;
          if (sk < 0.0) {
            tight[k] = 1.0;
            v[0] = 1.0;
          }
          s[k] = fmax(sk, 0.0);
        }
      }
      reduce<0, 1>(dummy, v);
      // The plain test evaluates the projected point: clipped duals and slacks
      // show up in its residuals.
      if (termination(1.0, nb, nc, nullptr, false) == QTQP_STATUS_SOLVED) return true;
      if (!(v[0] > 0.0)) return false;  // the set is stable yet not acceptable
      sync();
    }
    return false;
  }

  // --------------------------------------------------------------------------
  // The whole solve (QTQP._solve_impl, __init__.py:429-614).  warm_*: the
  // learned warm start of this instance (x and y in the original scaling,
  // active-row mask), or null for the plain method.
  // --------------------------------------------------------------------------
  // start_*: a starting point in the original scaling (y, s positive on the
  // inequality rows) that replaces the cold start (no reference counterpart:
  // a re-solve started from an earlier solution), or null.
  __device__ void solve(qtqp_result* result, double* stats, double* x_out, double* y_out,
                        double* s_out, const double* warm_x = nullptr,
                        const double* warm_y = nullptr,
                        const unsigned char* warm_act = nullptr,
                        const double* start_x = nullptr, const double* start_y = nullptr,
                        const double* start_s = nullptr) {
    const qtqp_options& op = *o;
    const uint64_t t_start = globaltimer_ns();
    double nb, nc;
    {
      QTQP_TIC();
      load_and_equilibrate(op.equilibrate != 0, nb, nc);
      QTQP_TOC(kPhLoad);
    }
    int w32 = 0, w64 = 0, wsolves = 0;  // work of a rejected warm start counts too
    if (warm_act != nullptr) {
      // FP64 factor: the reduced system is as ill-conditioned as the last
      // interior-point iterations, where an FP32 factor is refused anyway.
      bool fp64w = true;
      const bool ok = warm_try(warm_x, warm_y, warm_act, nb, nc, fp64w, w32, w64, wsolves);
      sync();
      if (ok) {
        finish(QTQP_STATUS_SOLVED, 1.0, x_out, y_out, s_out);
        if (tid == 0) {
          result->status = QTQP_STATUS_SOLVED;
          result->iterations = 0;
          result->error = 0;
          result->fp32_factorizations = w32;
          result->fp64_factorizations = w64;
          result->ir_solves = wsolves;
          result->warm_started = 1;
          result->tau = 1.0;
          result->pcost = last_pcost;
          result->dcost = last_dcost;
          result->pres = last_pres;
          result->dres = last_dres;
          result->gap = last_gap;
        }
        return;
      }
    }
    double* xy = vec(kXY);
    double* s = vec(kRS);
    double* kq = vec(kKQ);
    double* kq0 = vec(kKQ0);
    double* xyp = vec(kXYP);
    double* xyc = vec(kXYC);
    double* ds = vec(kXD);  // d_s at [n, N)
    double* ct = vec(kCT);  // Mehrotra correction at [n, N)
    const double* q = vec(kQ);
    const double* de = vec(kDE);
    // Starting point.  A learned warm start that was not accepted starts the
    // method from its prediction when options.warm_shift > 0: x = x_hat,
    // y = y_hat on the equality rows, y = max(y_hat, 0) + shift and
    // s = max(b - A x_hat, 0) + shift on the inequality rows.  A given
    // start_* point is taken as it is.  Both are equilibrated like the cold
    // start (x/e, y/d, s*d).
    const bool from_pred = warm_act != nullptr && op.warm_shift > 0.0;
    const bool from_start = start_x != nullptr;
    if (from_pred || from_start) {
      const double sh = from_pred ? op.warm_shift : 0.0;
      const double* px0 = from_start ? start_x : warm_x;
      for (int k = tid; k < n; k += NT) xy[k] = px0[k] / de[k];
      sync();
      if (!from_start) {
        a_times(xy, s);  // s[n + i] = (A_eq x)_i = d_i (A x_hat)_i
        sync();
      }
      for (int k = own(n); k < N; k += NT) {
        const int i = k - n;
        const double yi = from_start ? start_y[i] : warm_y[i];
        if (i < z) {
          xy[k] = yi / de[k];
          s[k] = 0.0;
        } else if (from_start) {
          xy[k] = yi / de[k];
          s[k] = start_s[i] * de[k];
        } else {
          const double slack = fmax((q[k] - s[k]) / de[k], 0.0);  // b - A x_hat
          xy[k] = (fmax(yi, 0.0) + sh) / de[k];
          s[k] = (slack + sh) * de[k];
        }
      }
    }
    // _init_variables (__init__.py:299-307): x = 0, y[z:] = s[z:] = 1, then
    // equilibrated (x/e, y/d, s*d); K^{-1} q starts at zero.
    for (int k = tid; k < N; k += NT) {
      kq[k] = 0.0;
      if (from_pred || from_start) {
      } else if (k < n) {
        xy[k] = 0.0 / de[k];
      } else if (k < n + z) {
        xy[k] = 0.0;
        s[k] = 0.0;
      } else {
        xy[k] = 1.0 / de[k];
        s[k] = 1.0 * de[k];
      }
      ds[k] = 0.0;
      ct[k] = 0.0;
    }
    sync();
    double tau = 1.0, alpha = 0.0, sigma = 0.0, mu = 0.0;
    bool fp64 = op.precision == QTQP_PREC_FP64;
    int n32 = w32, n64 = w64, nsolves = wsolves, err = 0;
    int status = QTQP_STATUS_UNFINISHED;
    int it = 0, taken = 0;
    const double cnt = double(m - z);
    double dummy[1] = {0.0};
    for (it = 0; it < op.max_iter; ++it) {
      double* st = (stats != nullptr) ? stats + size_t(it) * QTQP_STATS_DOUBLES : nullptr;
      // _normalize (__init__.py:859-880) and mu (:477).
      {
        QTQP_TIC();
        double sm[2] = {0.0, 0.0};
        for (int k = sum_own(0); k < N; k += kSumT) {
          sm[0] = fma(xy[k], xy[k], sm[0]);
          if (k >= n) sm[1] = fma(xy[k], s[k], sm[1]);
        }
        reduce<2, 0>(sm, dummy);
        const double scale = sqrt(double(m - z + 1)) / fmax(kEps, sqrt(sm[0] + tau * tau));
        for (int k = tid; k < N; k += NT) {
          xy[k] *= scale;
          if (k >= n) s[k] *= scale;
        }
        tau *= scale;
        mu = (sm[1] * scale * scale) / cnt;
        QTQP_TOC(kPhNormalize);
      }
      // DirectKktSolver.update (direct.py:183-216).
      kkt_diag(mu, op.min_static_regularization);
      sync();
      {
        int info;
        if (fp64) {
          ++n64;
          info = factorize<double>();
        } else {
          ++n32;
          info = factorize<float>();
          if (info != 0) {  // FP32 pivot failure: refactor in FP64 for good
            fp64 = true;
            ++n64;
            info = factorize<double>();
          }
        }
        if (info != 0) {
          err = QTQP_ERR_NOT_SPD;
          break;
        }
      }
      // kinv_q = K^{-1} q, warm-started (__init__.py:484).
      for (int k = tid; k < N; k += NT) kq0[k] = kq[k];
      IrOutcome rq = ir_solve_policy([&](int k) { return q[k]; }, kq0,
                                     kq, fp64, n32, n64, err);
      nsolves += rq.solves;
      if (err) break;
      if (rq.nan) {
        err = QTQP_ERR_NAN;
        break;
      }
      write_lin_stats(st, 0, rq, -1, fp64);
      // Per-iteration constants of the tau equations: P K^{-1}q, P x and dots.
      IterConsts ic;
      {
        double* pkq = vec(kPW);
        double* px = vec(kXD);
        const double* pi = vec(kPI);
        double sm[5] = {0, 0, 0, 0, 0};
        for (int k = sum_own(0); k < N; k += kSumT) {
          sm[0] = fma(kq[k], q[k], sm[0]);
          sm[2] = fma(q[k], xy[k], sm[2]);
        }
        if (has_p) {
          auto add = [&](int k, double a, double b) {
            sm[1] = fma(kq[k], a, sm[1]);
            sm[3] = fma(xy[k], b, sm[3]);
            sm[4] = fma(b, kq[k], sm[4]);
          };
          auto epi = [&](int k, double pq, double pxk) {
            const double a = fma(pi[k], kq[k], pq);
            const double b = fma(pi[k], xy[k], pxk);
            pkq[k] = a;
            px[k] = b;
            if constexpr (kSumT == NT) add(k, a, b);
          };
          if constexpr (kSparseA) {
            for (int k = tid; k < n; k += NT) epi(k, band_poff_row(kq, k), band_poff_row(xy, k));
            if constexpr (kSumT != NT) {
              sync();
              for (int k = sum_own(0); k < n; k += kSumT) add(k, pkq[k], px[k]);
            }
          } else if (fused_ok()) {
            dense_products(nullptr, nullptr, nullptr, kq, nullptr);
            sync();
            for (int k = tid; k < n; k += NT) pkq[k] = fused_colsum(k);
            sync();
            dense_products(nullptr, nullptr, nullptr, xy, nullptr);
            sync();
            for (int k = tid; k < n; k += NT) epi(k, pkq[k], fused_colsum(k));
          } else {
            const double* Pp = P;
            const int lp = ldp;
            rowdot<2>(n, n,
                      [&](int k, int j, double* acc) {
                        const double pjk = Pp[j * lp + k];
                        acc[0] = fma(pjk, kq[j], acc[0]);
                        acc[1] = fma(pjk, xy[j], acc[1]);
                      },
                      [&](int k, double* acc) { epi(k, acc[0], acc[1]); });
          }
        }
        reduce<5, 0>(sm, dummy);
        ic.kqq = sm[0];
        ic.kqpkq = sm[1];
        ic.qz = sm[2];
        ic.xpx = has_p ? sm[3] : 0.0;
        ic.pxkq = has_p ? sm[4] : 0.0;
      }
      // ---- Predictor (__init__.py:489-516) -------------------------------
      const double mu_c = mu;
      auto rhs_pred = [&](int k) {
        double r = (mu_c - 0.0) * xy[k];
        if (k >= n + z) r += s[k];
        return r;
      };
      IrOutcome rp = ir_solve_policy(rhs_pred, xy, xyp, fp64, n32,
                                     n64, err);
      nsolves += rp.solves;
      if (err) break;
      if (rp.nan) {
        err = QTQP_ERR_NAN;
        break;
      }
      int tm_p = 0;
      double tau_p;
      {
        QTQP_TIC();
        tau_p = tau_step(xyp, rp, mu, 0.0, mu * tau, tau, tau, ic, tm_p);
        QTQP_TOC(kPhTau);
      }
      write_lin_stats(st, 1, rp, tm_p, fp64);
      for (int k = tid; k < N; k += NT) {
        xyp[k] -= kq[k] * tau_p;  // [x_p; y_p]
        if (k >= n + z) ds[k] = -xyp[k] * s[k] / xy[k];
      }
      const double alpha_p = step_to_boundary([&](int k, double& dy, double& dsk) {
        dy = xyp[k] - xy[k];
        dsk = ds[k];
      });
      // _compute_sigma (__init__.py:682-706).
      {
        double sm[3] = {0, 0, 0};
        const double dtp = tau_p - tau;
        for (int k = sum_own(0); k < N; k += kSumT) {
          const double va = xy[k] + alpha_p * (xyp[k] - xy[k]);
          if (k < n) {
            sm[0] = fma(va, va, sm[0]);
          } else {
            sm[1] = fma(va, va, sm[1]);
            const double sa = s[k] + alpha_p * ds[k];
            sm[2] = fma(va, sa, sm[2]);
          }
        }
        reduce<3, 0>(sm, dummy);
        const double ta = tau + alpha_p * dtp;
        const double nrm2 = sm[0] + sm[1] + ta * ta;
        const double scale_sq = double(m - z + 1) / fmax(kEps * kEps, nrm2);
        const double mu_aff = scale_sq * sm[2] / cnt;
        const double sb = mu_aff / fmax(kEps, mu);
        sigma = fmin(fmax(sb * sb * sb, 0.0), 1.0);
      }
      // Mehrotra correction (__init__.py:528).
      for (int k = own(n + z); k < N; k += NT) {
        const double dyp = xyp[k] - xy[k];
        ct[k] = -ds[k] * dyp / xy[k];
      }
      // ---- Corrector (__init__.py:529-543) -------------------------------
      const double mu_t = sigma * mu;
      auto rhs_corr = [&](int k) {
        double r = (mu_c - mu_t) * xyp[k];
        if (k >= n + z) {
          if (mu_t != 0.0) r += mu_t / xy[k];
          r += s[k];
          r += ct[k];
        }
        return r;
      };
      sync();  // x_p, y_p complete before the corrector reads them
      IrOutcome rc = ir_solve_policy(rhs_corr, xyp, xyc, fp64, n32,
                                     n64, err);
      nsolves += rc.solves;
      if (err) break;
      if (rc.nan) {
        err = QTQP_ERR_NAN;
        break;
      }
      int tm_c = 0;
      const double tau_c =
          tau_step(xyc, rc, mu, mu_t, (mu - mu_t) * tau_p, tau, tau_p, ic, tm_c);
      write_lin_stats(st, 2, rc, tm_c, fp64);
      for (int k = tid; k < N; k += NT) {
        xyc[k] -= kq[k] * tau_c;  // [x_c; y_c]
        if (k >= n + z) ds[k] = mu_t / xy[k] + ct[k] - xyc[k] * s[k] / xy[k];
      }
      alpha = step_to_boundary([&](int k, double& dy, double& dsk) {
        dy = xyc[k] - xy[k];
        dsk = ds[k];
      });
      // ---- Update (__init__.py:556-565) --------------------------------
      {
        const double stp = op.step_size_scale * alpha;
        for (int k = tid; k < N; k += NT) {
          xy[k] += stp * (xyc[k] - xy[k]);
          if (k >= n) s[k] += stp * ds[k];
          if (k >= n + z) {
            xy[k] = fmax(xy[k], 1e-30);
            s[k] = fmax(s[k], 1e-30);
          }
        }
        tau += stp * (tau_c - tau);
        tau = fmax(tau, 1e-30);
      }
      sync();
      {
        QTQP_TIC();
        status = termination(tau, nb, nc, st, op.collect_stats != 0);
        QTQP_TOC(kPhTerm);
      }
      taken = it + 1;
      if (st != nullptr && tid == 0) {
        st[kStIter] = it;
        st[kStMu] = mu;
        st[kStSigma] = sigma;
        st[kStAlpha] = alpha;
        st[kStTau] = tau;
        st[kStTime] = double(globaltimer_ns() - t_start) * 1e-9;
      }
      if (status != QTQP_STATUS_UNFINISHED) break;
    }
    if (err == 0 && status == QTQP_STATUS_UNFINISHED && taken == op.max_iter) {
      status = QTQP_STATUS_HIT_MAX_ITER;
      if (stats != nullptr && tid == 0)
        stats[size_t(taken - 1) * QTQP_STATS_DOUBLES + kStStatus] = status;
    }
    sync();
    finish(status, tau, x_out, y_out, s_out);
    if (tid == 0) {
      result->status = err ? QTQP_STATUS_FAILED : status;
      result->iterations = taken;
      result->error = err;
      result->fp32_factorizations = n32;
      result->fp64_factorizations = n64;
      result->ir_solves = nsolves;
      result->warm_started = 0;
      result->tau = tau;
      result->pcost = last_pcost;
      result->dcost = last_dcost;
      result->pres = last_pres;
      result->dres = last_dres;
      result->gap = last_gap;
    }
  }

  // Unequilibrate and scale by status (__init__.py:580-614).
  QTQP_PHASE void finish(int status, double tau, double* x_out, double* y_out, double* s_out) {
    QTQP_LOCALS;
    const double* xy = vec(kXY);
    const double* s = vec(kRS);
    const double* de = vec(kDE);
    const double nan = __longlong_as_double(0x7ff8000000000000ll);
    double sm[2] = {0.0, 0.0};  // b_o . y_o, c_o . x_o
    double dummy[1] = {0.0};
    if (status == QTQP_STATUS_INFEASIBLE || status == QTQP_STATUS_UNBOUNDED) {
      for (int k = sum_own(0); k < N; k += kSumT) {
        if (k < n) {
          sm[1] = fma(c0[k], de[k] * xy[k], sm[1]);
        } else {
          sm[0] = fma(b0[k - n], de[k] * xy[k], sm[0]);
        }
      }
      reduce<2, 0>(sm, dummy);
    }
    for (int k = tid; k < N; k += NT) {
      if (k < n) {
        const double xo = de[k] * xy[k];
        double v;
        if (status == QTQP_STATUS_INFEASIBLE) {
          v = nan;
        } else if (status == QTQP_STATUS_UNBOUNDED) {
          v = xo / fabs(sm[1]);
        } else {
          v = xo / tau;
        }
        x_out[k] = v;
      } else {
        const double yo = de[k] * xy[k], so = s[k] / de[k];
        double vy, vs;
        if (status == QTQP_STATUS_INFEASIBLE) {
          vy = yo / fabs(sm[0]);
          vs = nan;
        } else if (status == QTQP_STATUS_UNBOUNDED) {
          vy = nan;
          vs = so / fabs(sm[1]);
        } else {
          vy = yo / tau;
          vs = so / tau;
        }
        y_out[k - n] = vy;
        s_out[k - n] = vs;
      }
    }
  }
  // ==========================================================================
  // Banded backend (FMT == kFmtBand): sparse A and P, and the Gram matrix
  // G = P_off + diag(Rx) + A^T diag(1/Ry) A of half-bandwidth bw (e.g. the
  // block-tridiagonal Gram of a stage-ordered MPC problem).  Everything lives
  // in the instance's global workspace slot.
  // ==========================================================================
  __device__ void bind_band(int n_, int m_, int bw_, int nnz_a_, int nnz_p_, char* gmem) {
    tid = threadIdx.x;
    n = n_;
    m = m_;
    N = n + m;
    bw = bw_;
    nnz_a = nnz_a_;
    nnz_p = nnz_p_;
    const BandLayout L = plan_band_layout(n, m, bw, nnz_a, nnz_p);
    np = L.np;
    V = reinterpret_cast<double*>(gmem);
    Lb = reinterpret_cast<double*>(gmem + L.v_bytes);
    G = Lb;
    av = reinterpret_cast<double*>(gmem + L.v_bytes + L.l_bytes);
    at = av + nnz_a;
    pv = at + nnz_a;
    grow = reinterpret_cast<int*>(gmem + L.v_bytes + L.l_bytes + L.val_bytes);
    gcnt = grow + nnz_a;
    A = P = nullptr;
    lda = ldp = ldg = 0;
  }

#define QTQP_BAND_LOCALS                                                        \
  const int tid = this->tid, n = this->n, m = this->m, N = this->N;             \
  const int bw = this->bw, ldl = this->bw + 1;                                  \
  const int* const ip = this->ip;                                               \
  const int* const ix = this->ix;                                               \
  const int* const jp = this->jp;                                               \
  const int* const jx = this->jx;                                               \
  const int* const pp = this->pp;                                               \
  const int* const px = this->px;                                               \
  double* const av = this->av;                                                  \
  double* const at = this->at;                                                  \
  double* const pv = this->pv;                                                  \
  const bool has_p = this->has_p;                                               \
  (void)tid; (void)n; (void)m; (void)N; (void)bw; (void)ldl; (void)ip; (void)ix; \
  (void)jp; (void)jx; (void)pp; (void)px; (void)av; (void)at; (void)pv; (void)has_p

  // Ruiz equilibration on the CSR (A), CSC (A) and CSR (P) value arrays, with
  // the reference's arithmetic: a_ij *= (d_i * e_j), p_ij *= (e_i * e_j).
  __device__ void band_load_and_equilibrate(bool equilibrate, double& nb, double& nc) {
    QTQP_BAND_LOCALS;
    double* de = vec(kDE);
    double* sc = vec(kTMP);
    for (int q = tid; q < nnz_a; q += NT) {
      av[q] = av0[q];
      at[q] = at0[q];
    }
    for (int q = tid; q < nnz_p; q += NT) pv[q] = has_p ? pv0[q] : 0.0;
    for (int k = tid; k < N; k += NT) de[k] = 1.0;
    if constexpr (FMT == kFmtBand) {
      if (bwin != nullptr) band_gram_groups();
    }
    sync();
    if constexpr (FMT == kFmtBand) {
      if (bwin != nullptr) band_gram_duplicates();
    }
    auto scale_of = [](double mx) {
      if (mx == 0.0) mx = 1.0;
      return fmin(fmax(1.0 / sqrt(mx), 1e-3), 1e3);
    };
    if (equilibrate) {
      for (int sweep = 0; sweep < 10; ++sweep) {
        for (int k = tid; k < N; k += NT) {
          double mx = 0.0;
          if (k < n) {
            for (int q = jp[k]; q < jp[k + 1]; ++q) mx = fmax(mx, fabs(at[q]));
            if (has_p)
              for (int q = pp[k]; q < pp[k + 1]; ++q) mx = fmax(mx, fabs(pv[q]));
          } else {
            for (int q = ip[k - n]; q < ip[k - n + 1]; ++q) mx = fmax(mx, fabs(av[q]));
          }
          sc[k] = scale_of(mx);
        }
        sync();
        for (int r = tid; r < m; r += NT) {
          const double dr = sc[n + r];
          for (int q = ip[r]; q < ip[r + 1]; ++q) av[q] *= dr * sc[ix[q]];
        }
        for (int j = tid; j < n; j += NT) {
          const double ej = sc[j];
          for (int q = jp[j]; q < jp[j + 1]; ++q) at[q] *= sc[n + jx[q]] * ej;
        }
        if (has_p) {
          for (int i = tid; i < n; i += NT) {
            const double ei = sc[i];
            for (int q = pp[i]; q < pp[i + 1]; ++q) pv[q] *= ei * sc[px[q]];
          }
        }
        for (int k = tid; k < N; k += NT) de[k] *= sc[k];
        sync();
      }
    }
    double* q = vec(kQ);
    double* pi = vec(kPI);
    double mx[2] = {0.0, 0.0};
    double dummy[1] = {0.0};
    for (int k = tid; k < N; k += NT) {
      if (k < n) {
        q[k] = c0[k] * de[k];
        double d = 0.0;
        if (has_p) {
          for (int qq = pp[k]; qq < pp[k + 1]; ++qq) {
            if (px[qq] == k) {  // diag(P_eq); pv keeps only the off-diagonal
              d = pv[qq];
              pv[qq] = 0.0;
            }
          }
        }
        pi[k] = d;
        mx[1] = nanmax(mx[1], fabs(c0[k]));
      } else {
        q[k] = b0[k - n] * de[k];
        mx[0] = nanmax(mx[0], fabs(b0[k - n]));
      }
    }
    reduce<0, 2>(dummy, mx);
    nb = mx[0];
    nc = mx[1];
    sync();
  }

  // sum_{q0 <= q < q1} val[q] v[voff + idx[q]]: indices and values are
  // loaded 8 at a time, then the 8 gathers, so that several loads are in
  // flight per thread (these sparse dots are latency-bound).
  __device__ __forceinline__ static double sparse_dot(const int* idx, const double* val,
                                                      const double* v, int voff, int q0, int q1) {
    double t0 = 0.0, t1 = 0.0;
    int q = q0;
    for (; q + 8 <= q1; q += 8) {
      int ii[8];
      double aa[8], xx[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        ii[e] = idx[q + e];
        aa[e] = val[q + e];
      }
#pragma unroll
      for (int e = 0; e < 8; ++e) xx[e] = v[voff + ii[e]];
#pragma unroll
      for (int e = 0; e < 8; e += 2) {
        t0 = fma(aa[e], xx[e], t0);
        t1 = fma(aa[e + 1], xx[e + 1], t1);
      }
    }
    for (; q < q1; ++q) t0 = fma(val[q], v[voff + idx[q]], t0);
    return t0 + t1;
  }
  // sum_{q0 <= q < q1} val[q] (scale[idx[q]] v[idx[q]]) (scale null: without it),
  // loaded the same way and added up in the order of the entries.
  template <typename V>
  __device__ __forceinline__ static double sparse_dot_ordered(const int* idx, const double* val,
                                                              const V* v, const double* scale,
                                                              int q0, int q1) {
    double t = 0.0;
    int q = q0;
    for (; q + 8 <= q1; q += 8) {
      int ii[8];
      double aa[8], xx[8];
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        ii[e] = idx[q + e];
        aa[e] = val[q + e];
      }
#pragma unroll
      for (int e = 0; e < 8; ++e)
        xx[e] = scale != nullptr ? scale[ii[e]] * double(v[ii[e]]) : double(v[ii[e]]);
#pragma unroll
      for (int e = 0; e < 8; ++e) t = fma(aa[e], xx[e], t);
    }
    for (; q < q1; ++q)
      t = fma(val[q], scale != nullptr ? scale[idx[q]] * double(v[idx[q]]) : double(v[idx[q]]), t);
    return t;
  }
  // (P_off v)_k for the owner of row k (P symmetric, so row k = column k).
  __device__ __forceinline__ double band_poff_row(const double* v, int k) const {
    return has_p ? sparse_dot(px, pv, v, 0, pp[k], pp[k + 1]) : 0.0;
  }
  // (A^T y)_k with y at v[n + i].
  __device__ __forceinline__ double band_at_col(const double* v, int k) const {
    return sparse_dot(jx, at, v, n, jp[k], jp[k + 1]);
  }
  // (A x)_i.
  __device__ __forceinline__ double band_a_row(const double* v, int i) const {
    return sparse_dot(ix, av, v, 0, ip[i], ip[i + 1]);
  }

  // The rows of A that meet each group of kGramCols columns, once per solve:
  // grow[jp[8 g] ..) holds the rows of group g (gcnt[g] of them) in ascending
  // order.  A warp per group marks the rows of the group's CSC entries in a bit
  // map in shared memory (the rows between the first and the last, a window of
  // them at a time) and lists the marked ones, so nothing depends on how the
  // entries are ordered or whether some are stored twice.
  __device__ void band_gram_groups() {
    QTQP_BAND_LOCALS;
    constexpr int kWarps = (NT > 1024 ? kGridBT : NT) / 32;
    const int lane = threadIdx.x & 31;
    const int words = min(1024, int(bwin_bytes / (kWarps * sizeof(unsigned int))));
    unsigned int* bits = reinterpret_cast<unsigned int*>(bwin) + (threadIdx.x >> 5) * words;
    const int ng = (n + kGramCols - 1) / kGramCols;
    for (int g = tid >> 5; g < ng; g += NT / 32) {
      const int j0 = g * kGramCols, q0 = jp[j0], q1 = jp[min(n, j0 + kGramCols)];
      int lo = m, hi = -1;
      for (int q = q0 + lane; q < q1; q += 32) {
        lo = min(lo, jx[q]);
        hi = max(hi, jx[q]);
      }
      lo = __reduce_min_sync(0xffffffffu, lo);
      hi = __reduce_max_sync(0xffffffffu, hi);
      int at_row = q0;  // where the next row goes
      for (int base = lo; base <= hi; base += 32 * words) {
        const int nw = min(words, ((hi - base) >> 5) + 1);
        for (int w = lane; w < nw; w += 32) bits[w] = 0;
        __syncwarp();
        for (int q = q0 + lane; q < q1; q += 32) {
          const int r = jx[q] - base;
          if (r >= 0 && (r >> 5) < nw) atomicOr(bits + (r >> 5), 1u << (r & 31));
        }
        __syncwarp();
        for (int w0 = 0; w0 < nw; w0 += 32) {
          unsigned int u = w0 + lane < nw ? bits[w0 + lane] : 0u;
          const int own_rows = __popc(u);
          int upto = own_rows;  // rows of the lanes up to this one
          for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += x;
          }
          for (int p = at_row + upto - own_rows; u != 0; u &= u - 1, ++p)
            grow[p] = base + 32 * (w0 + lane) + __ffs(u) - 1;
          at_row += __shfl_sync(0xffffffffu, upto, 31);
        }
        __syncwarp();
      }
      if (lane == 0) gcnt[g] = at_row - q0;
    }
    if (tid == 0) gcnt[ng] = 0;
  }
  // Whether some row's columns are not strictly ascending, so that an entry may
  // be stored twice, in gcnt[number of groups]; after a barrier that follows
  // band_gram_groups.
  __device__ void band_gram_duplicates() {
    QTQP_BAND_LOCALS;
    for (int q = 1 + tid; q < nnz_a; q += NT) {
      if (ix[q] > ix[q - 1]) continue;
      int lo = 0, hi = m;  // the row of entry q: the last i with ip[i] <= q
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ip[mid] <= q) {
          lo = mid;
        } else {
          hi = mid;
        }
      }
      if (ip[lo] < q) gcnt[(n + kGramCols - 1) / kGramCols] = 1;  // q - 1 is in the same row
    }
  }

  // The Gram matrix G = P_off + diag(Rx) + A^T diag(1/Ry) A in column band
  // storage (Lb) plus the relative diagonal jitter of the dense backend.  A
  // warp per group of 8 columns: the rows that meet the group are taken four
  // at a time, their entries at columns j0 .. j0 + bw + 7 scattered (scaled
  // by 1/sqrt(Ry)) into four dense rows of shared memory, and G[j0 .. j0 + 8,
  // j0 ..] += the product of their first 8 columns with all of them: FP64
  // tensor-core steps (DMMA m8n8k4) into (bw + 14) / 8 accumulators, which
  // stay in registers.  T = 50 MPC QP (2000 rows of 61 entries, half-bandwidth
  // 99): 5.5 ms per factorisation with a thread per column, 2.7 ms with a warp
  // per column accumulating in shared memory (a row's every visit by a column
  // cost some 60 instructions; a group of 8 columns now shares one visit).
  // buf: the block's scratch, gram_warp_elems(bw) entries per warp.
  // dup: rows may store an entry twice; their values are added up.
  // A tensor-core step adds its four products one after the other, and the rows
  // come in ascending order: every entry of G is the plain sum over the rows.
  template <typename T, int NT8>
  __device__ __forceinline__ void band_gram_group(int g, T* buf, bool dup, double& dmax) const {
    QTQP_BAND_LOCALS;
    const double* wsc = vec(kPW);
    const double* reg = vec(kREG);
    const int lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3;
    const int pitch = gram_pitch(bw), width = min(bw + kGramCols, pitch);
    const int j0 = g * kGramCols, cnt = gcnt[g];
    const int* rows = grow + jp[j0];
    const int nt = (bw + 7 + 8) >> 3;  // 8-column tiles from j0 to j0 + bw + 7
    T acc[NT8][2];
#pragma unroll
    for (int t = 0; t < NT8; ++t) acc[t][0] = acc[t][1] = T(0);
    const int rr = lane >> 3, sub = lane & 7;  // this lane's row of the four, its share of it
    int rn = rr < cnt ? rows[rr] : -1;
    for (int c0 = 0; c0 < cnt; c0 += 4) {
      const int r = rn;
      rn = c0 + 4 + rr < cnt ? rows[c0 + 4 + rr] : -1;
      for (int e = lane; e < 4 * pitch; e += 32) buf[e] = T(0);
      __syncwarp();
      if (r >= 0) {
        const double w = wsc[n + r];
        const int e1 = ip[r + 1];
        T* row = buf + rr * pitch;
        int e = ip[r] + sub;
        if (dup) {
          for (; e < e1; e += 8) {
            const int i = ix[e] - j0;
            if (i >= 0 && i < width) atomicAdd(row + i, T(av[e] * w));
          }
        }
        for (; e + 24 < e1; e += 32) {  // four loads in flight
          int ii[4];
          double aa[4];
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            ii[u] = ix[e + 8 * u] - j0;
            aa[u] = av[e + 8 * u];
          }
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (ii[u] >= 0 && ii[u] < width) row[ii[u]] = T(aa[u] * w);
        }
        for (; e < e1; e += 8) {
          const int i = ix[e] - j0;
          const double x = av[e];
          if (i >= 0 && i < width) row[i] = T(x * w);
        }
      }
      __syncwarp();
      if constexpr (sizeof(T) == 8) {
        const T* br = buf + tg * pitch + gi;
        const double a = br[0];
#pragma unroll
        for (int t = 0; t < NT8; ++t)
          if (t < nt) dmma_8x8x4(acc[t], a, br[8 * t]);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const T* br = buf + k * pitch;
          const T a = br[gi];
#pragma unroll
          for (int t = 0; t < NT8; ++t) {
            if (t < nt) {
              acc[t][0] = fma(a, br[8 * t + 2 * tg], acc[t][0]);
              acc[t][1] = fma(a, br[8 * t + 2 * tg + 1], acc[t][1]);
            }
          }
        }
      }
      __syncwarp();
    }
    // Lane (gi, tg) holds G[j0 + gi][j0 + 8 t + 2 tg + e].
    const int j = j0 + gi;
    T* col = reinterpret_cast<T*>(Lb) + size_t(j) * ldl;
    if (j < n) {
#pragma unroll
      for (int t = 0; t < NT8; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int d = 8 * t + 2 * tg + e - gi;
          if (d >= 0 && d <= bw) col[d] = d == 0 ? T(reg[j]) + acc[t][e] : acc[t][e];
        }
    }
    __syncwarp();
    if (j < n && has_p && tg == 0) {
      const int q1 = pp[j + 1];
      for (int q = pp[j]; q < q1; q += 4) {
        int dd[4];
        double x[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          dd[u] = q + u < q1 ? px[q + u] - j : 0;
          x[u] = q + u < q1 ? pv[q + u] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (dd[u] > 0 && dd[u] <= bw) col[dd[u]] = T(x[u]) + col[dd[u]];
      }
    }
    if (j < n && tg == 0) dmax = nanmax(dmax, double(col[0]));
    __syncwarp();
  }

  template <typename T>
  __device__ void band_gram(T* buf) {
    const int ldl = bw + 1;
    T* L = reinterpret_cast<T*>(Lb);
    T* wbuf = buf + size_t(threadIdx.x >> 5) * gram_warp_elems(bw);
    double dmax[1] = {0.0};
    double dummy[1] = {0.0};
    const int ng = (n + kGramCols - 1) / kGramCols;
    const bool dup = gcnt[ng] != 0;
    for (int g = tid >> 5; g < ng; g += NT / 32) {
      if (bw <= 32) {
        band_gram_group<T, 6>(g, wbuf, dup, dmax[0]);
      } else {
        band_gram_group<T, 17>(g, wbuf, dup, dmax[0]);
      }
    }
    static_assert((kBandWinMaxBw + 7 + 8) / 8 <= 17 && (32 + 7 + 8) / 8 <= 6, "tiles");
    reduce<0, 1>(dummy, dmax);
    const double jit = (sizeof(T) == 8 ? 1e-14 : 2.384185791015625e-07) * dmax[0];
    for (int j = tid; j < n; j += NT) L[size_t(j) * ldl] = T(double(L[size_t(j) * ldl]) + jit);
    sync();
  }

  // Gram matrix in column band storage, then Cholesky.  With the shared-
  // memory window (bw <= kBandWinMaxBw) the blocked factorisation
  // (band_chol_panel_range); otherwise the global-memory variant below runs.  In
  // grid mode the partitioned factorisation runs (band_grid.cuh).
  template <typename T>
  __device__ int band_factorize() {
    if constexpr (FMT == kFmtSparse) {
      return sparse_factorize<T>(*this);
    } else if constexpr (NT > 1024) {
      return bandp_factorize<T>(*this);
    } else {
      if (bwin == nullptr) return band_factorize_global<T>();
      QTQP_TIC();
      band_gram<T>(reinterpret_cast<T*>(bwin));
      QTQP_TOC(kPhGram);
      QTQP_RETIC();
      const int info = band_chol_panel_range<T, NT>(tid, 0, n, n, nullptr, 0);
      QTQP_TOC(kPhChol);
      return info;
    }
  }

  // Band Cholesky with the active part of the band in shared memory, over
  // the principal submatrix of rows / columns [lo, lo + nsub) of which the
  // first ne columns are eliminated (ne == nsub: the whole factorisation), by
  // the BT threads of a block (lt: this thread's index), BT >= kBandPanel +
  // bw.  The diagonal of the factor keeps 1 / l_kk.  tail (when ne < nsub):
  // the lower triangle of the trailing (nsub-ne)^2 block after the
  // elimination (the Schur complement of the eliminated columns), row-major
  // with leading dimension ldt.  Columns before lo are not part of the
  // submatrix.  Returns 0 or the 1-based global column of the first
  // non-positive pivot.
  //
  // kBandPanel-column panels; the window is circular with period B = bw +
  // kBandPanel (lower triangle, row-major).  Per panel, two barriers:
  //  * every thread that holds a row of the panel (kBandPanel + bw rows)
  //    factors the panel's 8 x 8 diagonal block for itself, in registers, and
  //    solves its own row with it as it goes, so no barrier lies on the chain
  //    from column to column (eight barriers and publishes per panel before);
  //    the finished columns go to global memory and to the panel buffer;
  //  * the rank-8 update of the window's lower bw x bw part, by 16 x 16 tiles,
  //    a warp per tile, on the FP64 tensor cores (DMMA).
  //    The kBandPanel rows that enter the window, copied from the Gram matrix
  //    (cp.async) since the panel before, are stored, and the columns left of
  //    their band zeroed.
  template <typename T, int BT>
  __device__ int band_chol_panel_range(int lt, int lo, int nsub, int ne, T* tail, int ldt) {
    constexpr int KP = kBandPanel, PP = KP + 1;
    const int bw = this->bw, ldl = bw + 1, B = bw + KP;
    T* L = reinterpret_cast<T*>(Lb) + size_t(lo) * ldl;
    T* W = reinterpret_cast<T*>(bwin);
    T* Pn = W + B * B;
    T* En = Pn + B * PP;  // two stages of the rows that enter the window
    uint16_t* tiles = reinterpret_cast<uint16_t*>(En + 2 * KP * (bw + 1));
    __shared__ int s_bad;
    const int nt16 = (bw + 15) >> 4, ntiles = nt16 * (nt16 + 1) / 2;
    const int lane = lt & 31, warp = lt >> 5, gi = lane >> 2, tg = lane & 3;
    for (int a = lt; a < nt16; a += BT)
      for (int b = 0; b <= a; ++b) tiles[a * (a + 1) / 2 + b] = uint16_t(a | (b << 8));
    for (int e = lt; e < B * B; e += BT) {
      const int i = e / B, j = e - i * B;
      W[e] = (j <= i && i - j <= bw && i < nsub) ? L[size_t(j) * ldl + (i - j)] : T(0);
    }
    if (lt == 0) s_bad = 0;
    group_sync<BT>();
    int bad = 0;
    constexpr int MAXPRE = (KP * 128 + BT - 1) / BT;  // entering entries per thread (bw < 128)
    int pre_e[MAXPRE], pre_d[MAXPRE];
#pragma unroll
    for (int q = 0; q < MAXPRE; ++q) {
      pre_e[q] = (lt + BT * q) / (bw + 1);
      pre_d[q] = (lt + BT * q) % (bw + 1);
    }
    // Rows kk + B .. kk + B + 7 enter after the panel of column kk: their band
    // entries (row r, column r - bw + d), each stored later by the thread that
    // copies it.
    auto issue_rows = [&](int kk) {
#pragma unroll
      for (int q = 0; q < MAXPRE; ++q) {
        const int e = pre_e[q], d = pre_d[q], r = kk + B + e;
        if (e < KP && kk < ne && r < nsub)
          cp_async_elem(En + ((kk / KP) & 1) * KP * (bw + 1) + lt + BT * q,
                        L + size_t(r - bw + d) * ldl + (bw - d), true);
      }
      cp_async_commit();
    };
    issue_rows(0);
    int sk = 0;  // k mod B
    for (int k = 0; k < ne; k += KP, sk = sk + KP >= B ? sk + KP - B : sk + KP) {
      const int pw = min(KP, ne - k);
      const int nr = min(pw + bw, nsub - k);
      auto sl = [&](int x) {  // slot of index k + x, 0 <= x < 2 B
        int t = sk + x;
        t = t >= B ? t - B : t;
        return t >= B ? t - B : t;
      };
      issue_rows(k + KP);
      if (lt < nr) {
        // The diagonal block (the same in every thread) and this thread's row.
        T dg[KP][KP], v[KP];
        int sc[KP];
#pragma unroll
        for (int c = 0; c < KP; ++c) sc[c] = sl(c);
        const T* wr = W + sl(lt) * B;
#pragma unroll
        for (int a = 0; a < KP; ++a) {
#pragma unroll
          for (int c = 0; c <= a; ++c) dg[a][c] = a < pw ? W[sc[a] * B + sc[c]] : T(0);
          v[a] = (a < pw && a <= lt) ? wr[sc[a]] : T(0);
        }
        // Columns from pw on (the last panel) have a zero diagonal block and
        // are not used.  A non-positive pivot is only noted: the panel then
        // runs to its end on whatever follows, and nothing of it is kept.
        int f = 0;
#pragma unroll
        for (int c = 0; c < KP; ++c) {
          const T piv = dg[c][c];
          f = f == 0 && c < pw && !(piv > T(0)) ? k + c + 1 : f;
          const T il = rsqrt(piv);
          const T lic = v[c] * il;
          v[c] = lt == c ? il : lic;  // the factor keeps 1 / l_cc
#pragma unroll
          for (int a = c + 1; a < KP; ++a) dg[a][c] *= il;
#pragma unroll
          for (int a = c + 1; a < KP; ++a) {
            v[a] = fma(-lic, dg[a][c], v[a]);
#pragma unroll
            for (int b = c + 1; b <= a; ++b) dg[a][b] = fma(-dg[a][c], dg[b][c], dg[a][b]);
          }
        }
        if (pw < KP) {  // zero columns for the rank-8 update
#pragma unroll
          for (int c = 0; c < KP; ++c)
            if (c >= pw) v[c] = T(0);
        }
        if (f != 0) {
          if (lt == 0) s_bad = f;
        } else {
#pragma unroll
          for (int c = 0; c < KP; ++c)
            if (c < pw && c <= lt && lt - c <= bw) L[size_t(k + c) * ldl + (lt - c)] = v[c];
          if (lt >= pw) {
#pragma unroll
            for (int c = 0; c < KP; ++c) Pn[lt * PP + c] = v[c];
          }
        }
      }
      group_sync<BT>();
      bad = s_bad;
      if (bad) break;
      // Trailing update of the window: rows / columns k + pw .. k + pw + bw - 1.
      const int span = min(bw, nsub - k - pw);  // of which these exist
      for (int t = warp; t < ntiles; t += BT / 32) {
        const int pr = tiles[t];
        const int ta = (pr & 0xff) * 16, tb = (pr >> 8) * 16;
        if (ta >= span) continue;
        T acc[2][2][2];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y) acc[x][y][0] = acc[x][y][1] = T(0);
        if constexpr (sizeof(T) == 8) {
          double fa[2][2], fb[2][2];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const int a = ta + 8 * x + gi, b = tb + 8 * x + gi;
            const T* ra = Pn + (pw + min(a, span - 1)) * PP + tg;
            const T* rb = Pn + (pw + min(b, span - 1)) * PP + tg;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              fa[x][h] = a < span ? ra[4 * h] : 0.0;
              fb[x][h] = b < span ? rb[4 * h] : 0.0;
            }
          }
#pragma unroll
          for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
              for (int y = 0; y < 2; ++y) dmma_8x8x4(acc[x][y], fa[x][h], fb[y][h]);
        } else {
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            const T* ra = Pn + (pw + min(ta + 8 * x + gi, span - 1)) * PP;
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
              for (int e = 0; e < 2; ++e) {
                const T* rb = Pn + (pw + min(tb + 8 * y + 2 * tg + e, span - 1)) * PP;
#pragma unroll
                for (int c = 0; c < KP; ++c) acc[x][y][e] = fma(ra[c], rb[c], acc[x][y][e]);
              }
          }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
          const int a = ta + 8 * x + gi;
          if (a >= span) continue;
          T* wr = W + sl(pw + a) * B;
#pragma unroll
          for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const int b = tb + 8 * y + 2 * tg + e;
              if (b <= a) wr[sl(pw + b)] -= acc[x][y][e];
            }
        }
      }
      // Entering rows: band entries, and zeros left of the band.
      cp_async_wait<1>();  // this panel's; the next one's may be in flight
#pragma unroll
      for (int q = 0; q < MAXPRE; ++q) {
        const int e = pre_e[q], d = pre_d[q], r = k + B + e;
        if (e < pw && r < nsub)
          W[sl(B + e) * B + sl(KP + e + d)] = En[((k / KP) & 1) * KP * (bw + 1) + lt + BT * q];
      }
      for (int f = lt; f < pw * (KP - 1); f += BT) {
        const int e = f / (KP - 1), t = f - e * (KP - 1);
        const int r = k + B + e, j = k + pw + t;  // columns k+pw .. r-bw-1
        if (r < nsub && j < r - bw) W[sl(B + e) * B + sl(pw + t)] = T(0);
      }
      group_sync<BT>();
    }
    cp_async_wait<0>();
    if (tail != nullptr && bad == 0) {
      const int t = nsub - ne;
      for (int e = lt; e < t * t; e += BT) {
        const int i = e / t, j = e - i * t;
        if (j <= i) tail[size_t(i) * ldt + j] = W[((ne + i) % B) * B + (ne + j) % B];
      }
    }
    group_sync<BT>();
    return bad == 0 ? 0 : lo + bad;
  }

  // Global-memory variant (wide bands): Gram in column band storage, then
  // Cholesky with one barrier per column (the unscaled column k updates the
  // trailing band and column k-1 is finished in the same phase).
  template <typename T>
  __device__ int band_factorize_global() {
    QTQP_BAND_LOCALS;
    QTQP_TIC();
    T* L = reinterpret_cast<T*>(Lb);
    const double* reg = vec(kREG);
    const double* wsc = vec(kPW);
    double dmax[1] = {0.0};
    double dummy[1] = {0.0};
    for (int j = tid; j < n; j += NT) {
      T* col = L + size_t(j) * ldl;
      for (int d = 0; d <= bw; ++d) col[d] = T(0);
      for (int q = jp[j]; q < jp[j + 1]; ++q) {
        const int r = jx[q];
        const double w = wsc[n + r];
        const T arj = T(at[q] * w);
        for (int q2 = ip[r]; q2 < ip[r + 1]; ++q2) {
          const int i = ix[q2];
          if (i >= j && i - j <= bw) col[i - j] = fma(arj, T(av[q2] * w), col[i - j]);
        }
      }
      if (has_p) {
        for (int q = pp[j]; q < pp[j + 1]; ++q) {
          const int i = px[q];
          if (i > j && i - j <= bw) col[i - j] = T(pv[q]) + col[i - j];
        }
      }
      col[0] = T(reg[j]) + col[0];
      dmax[0] = nanmax(dmax[0], double(col[0]));
    }
    reduce<0, 1>(dummy, dmax);
    const double jit = (sizeof(T) == 8 ? 1e-14 : 2.384185791015625e-07) * dmax[0];
    for (int j = tid; j < n; j += NT) L[size_t(j) * ldl] = T(double(L[size_t(j) * ldl]) + jit);
    sync();
    QTQP_TOC(kPhGram);
    QTQP_RETIC();
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int NW = NT / 32;
    T il_prev = T(1);
    int info = 0;
    for (int k = 0; k <= n; ++k) {
      if (k > 0) {  // finish column k-1
        T* ck = L + size_t(k - 1) * ldl;
        const T il = il_prev;
        const int rows = min(bw, n - k);
        for (int d = 1 + tid; d <= rows; d += NT) ck[d] *= il;
        if (tid == NT - 1) ck[0] = il;
      }
      if (k == n) break;
      const T* ck = L + size_t(k) * ldl;
      const T d = ck[0];
      if (!(d > T(0))) {
        info = k + 1;
        break;
      }
      const T il = rsqrt(d), inv_d = il * il;
      const int last = min(n - 1, k + bw);
      for (int j = k + 1 + warp; j <= last; j += NW) {
        const T t = ck[j - k] * inv_d;
        T* cj = L + size_t(j) * ldl;
        for (int i = j + lane; i <= last; i += 32) cj[i - j] = fma(-ck[i - k], t, cj[i - j]);
      }
      il_prev = il;
      sync();
    }
    sync();
    QTQP_TOC(kPhChol);
    return info;
  }

  // Solves L L^T v = v (column band storage, reciprocal diagonal): forward
  // into w, backward into v.  With the shared-memory window the blocked
  // solves below run (the whole group); without it one warp walks the
  // columns in global memory.  In grid mode the partitioned solve runs
  // (band_grid.cuh).
  template <typename T>
  __device__ void band_chol_solve(T* v, T* w) {
    if constexpr (FMT == kFmtSparse) {
      sparse_solve<T>(*this, v, w);
    } else if constexpr (NT > 1024) {
      bandp_solve<T>(*this, v, w);
    } else {
      if (bwin == nullptr) {
        band_chol_solve_global<T>(v, w);
        return;
      }
      band_fwd_blocked<T, NT>(v, w, 0, n, n, tid);
      band_bwd_blocked<T, NT>(v, w, 0, n, n, tid);
    }
  }

  // Blocked band triangular solves over the columns [lo, lo + ne), called by all
  // BT >= 256 threads of the group (lt: this thread's index).  Forward: z_k =
  // (v_k - sum_c l_kc z_c) / l_kk into w, the rows [lo + ne, R) of v receiving
  // their updates.  Backward: x_k = (w_k - sum_d l_{k+d,k} x_{k+d}) / l_kk for k
  // in [lo, hi) into v, the rows [hi, R) holding known values of x in v (the
  // separator that follows a partition).
  //
  // Plain substitution in steps of 8 columns, every term added by itself: the
  // forward's in the order of the columns, the backward's step by step from the
  // last column, the known values first, within a step in ascending order.  The first W =
  // band_solve_owners(bw) threads run the steps, each with one of the rows that a
  // step updates in a register; every one of them solves the step's 8 x 8 diagonal
  // block for itself from eight right-hand-side values in shared memory, applies
  // the result to its row, and publishes the row when it enters the next diagonal
  // block.  The next W threads copy (cp.async) the factor's entries of the steps
  // ahead into a ring of eight stages; one barrier over both lies between two
  // steps, and the other threads wait at the end.
  //
  // Bound by the fetch of a step's instructions and its chain: 890 cycles per step
  // forward and 1010 backward at half-bandwidth 99 with 148 blocks at work, 760 and
  // 700 without the copies.  (Kept short on purpose: with the copies in the owners'
  // threads 2800 and 1900; one thread solving each diagonal block, then a barrier
  // and the rows, then another: about 1600.)
  template <typename T>
  __device__ __forceinline__ static void band_pair(const T* p, T& a, T& b) {
    using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
    const V t = *reinterpret_cast<const V*>(p);
    a = t.x;
    b = t.y;
  }
  template <typename T>
  __device__ __forceinline__ static void band_pair_put(T* p, T a, T b) {
    using V = typename std::conditional<sizeof(T) == 8, double2, float2>::type;
    V t;
    t.x = a;
    t.y = b;
    *reinterpret_cast<V*>(p) = t;
  }
  __device__ __forceinline__ static void band_step_sync(int threads) {
    asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory");
  }

  template <typename T, int BT>
  __device__ void band_fwd_blocked(T* v, T* w, int lo, int ne, int R, int lt) {
    constexpr int KB = kBandSolveBlk, NS = kBandSolveStages;
    static_assert(BT >= 256 && (NS & (NS - 1)) == 0, "owners and copiers; ring");
    const int bw = this->bw, ldl = bw + 1, hi = lo + ne, nb = (ne + KB - 1) / KB;
    const int W = band_solve_owners(bw), SS = int(band_solve_stage(bw));
    const T* L = reinterpret_cast<const T*>(Lb);
    T* ring = reinterpret_cast<T*>(bwin);
    T* rhs = ring + NS * SS;
    T* done = rhs + 2 * KB;  // the last step's results, to w a step later
    if (lt >= W && lt < 2 * W) {
      // Step b: columns k0 = lo + 8 b ..; copier and owner ct have row k0 + 8 + d
      // with d = (ct - 8 (b + 1)) mod W.  Rows from hi on are updated, not solved
      // (columns from hi on are zero).
      const int ct = lt - W;
      auto issue = [&](int b) {
        if (b < nb) {
          T* st = ring + (b & (NS - 1)) * SS;
          const int k0 = lo + b * KB, d = (ct - KB * (b + 1)) & (W - 1);
          const T* src = L + size_t(k0) * ldl + KB + d;  // column k0 + c: src[c bw]
          const int c0 = k0 + KB + d < R ? KB + d - bw : KB;
          const int c1 = min(KB, hi - k0);
#pragma unroll
          for (int c = 0; c < KB; ++c) {
            const bool ok = c >= c0 && c < c1;
            cp_async_elem(st + c * W + ct, ok ? src + c * bw : L, ok);
          }
#pragma unroll 1
          for (int e = ct; e < KB * KB; e += W) {
            const int c = e >> 3, dd = e & 7;
            const bool ok = c + dd < KB && dd <= bw && c < c1 && k0 + c + dd < R;
            cp_async_elem(st + KB * W + e, ok ? L + size_t(k0 + c) * ldl + dd : L, ok);
          }
        }
        cp_async_commit();
      };
#pragma unroll 1
      for (int b = 0; b + 1 < NS; ++b) issue(b);
#pragma unroll 1
      for (int b = 0; b < nb; ++b) {
        // Step b's entries have landed; after the barrier every owner is done with
        // step b - 1, whose stage is filled again.
        cp_async_wait<NS - 2>();
        band_step_sync(2 * W);
        issue(b + NS - 1);
      }
      cp_async_wait<0>();
    } else if (lt < W) {
      int row = lo + lt;
      T t = row < R ? v[row] : T(0), tn = row + W < R ? v[row + W] : T(0);
      if (lt < KB) {
        rhs[lt] = t;
        row += W;
        t = tn;
        tn = row + W < R ? v[row + W] : T(0);
      }
#pragma unroll 1
      for (int b = 0; b < nb; ++b) {
        band_step_sync(2 * W);
        const int k0 = lo + b * KB, pw = hi - k0;
        const T* st = ring + (b & (NS - 1)) * SS;
        if (b > 0 && lt < KB) w[k0 - KB + lt] = done[((b - 1) & 1) * KB + lt];
        T dg[KB][KB], z[KB], l[KB];
        const T* rp = rhs + (b & 1) * KB;
        const T* blk = st + KB * W;
#pragma unroll
        for (int c = 0; c < KB; c += 2) band_pair(rp + c, z[c], z[c + 1]);
#pragma unroll
        for (int c = 0; c < KB; ++c)
#pragma unroll
          for (int d = 0; d < KB - c; d += 2) band_pair(blk + KB * c + d, dg[c][d], dg[c][d + 1]);
#pragma unroll
        for (int c = 0; c < KB; ++c) l[c] = st[c * W + lt];
#pragma unroll
        for (int c = 0; c < KB; ++c) {
          if (c < pw) z[c] *= dg[c][0];
#pragma unroll
          for (int j = c + 1; j < KB; ++j) z[j] = fma(-dg[c][j - c], z[c], z[j]);
        }
#pragma unroll
        for (int c = 0; c < KB; ++c) t = fma(-l[c], z[c], t);
        if (lt == 0) {
#pragma unroll
          for (int c = 0; c < KB; c += 2) band_pair_put(done + (b & 1) * KB + c, z[c], z[c + 1]);
        }
        const int d = (lt - KB * (b + 1)) & (W - 1);
        if (d < KB && b + 1 < nb) {  // the row enters the next diagonal block
          rhs[((b + 1) & 1) * KB + d] = t;
          row += W;
          t = tn;
          tn = row + W < R ? v[row + W] : T(0);
        }
      }
      if (row >= hi && row < R) v[row] = t;
    }
    group_sync<BT>();
    if (lt < KB && nb > 0) {
      const int k = lo + (nb - 1) * KB + lt;
      if (k < R) (k < hi ? w : v)[k] = done[((nb - 1) & 1) * KB + lt];
    }
    group_sync<BT>();
  }

  template <typename T, int BT>
  __device__ void band_bwd_blocked(T* v, T* w, int lo, int hi, int R, int lt) {
    constexpr int KB = kBandSolveBlk, NS = kBandSolveStages, LP = KB + 1;
    const int bw = this->bw, ldl = bw + 1;
    const int nb = (hi - lo + KB - 1) / KB;
    const int W = band_solve_owners(bw), SS = int(band_solve_stage(bw));
    const T* L = reinterpret_cast<const T*>(Lb);
    T* ring = reinterpret_cast<T*>(bwin);
    T* rhs = ring + NS * SS;
    T* done = rhs + 2 * KB;
    T* known = done + 2 * KB;
    if (R > hi) {
      for (int r = hi + lt; r < R; r += BT) known[r - hi] = v[r];
      group_sync<BT>();
    }
    if (lt >= W && lt < 2 * W) {
      // Step b: rows kb = hi - 8 (b + 1) ..; owner ct has row kb - 1 - d with d =
      // (ct - 8 (b + 1)) mod W, whose entries L(kb + q, row) are contiguous in the
      // band: eight neighbouring copiers copy one row's.
      const int ct = lt - W;
      auto issue = [&](int b) {
        if (b < nb) {
          T* st = ring + (b & (NS - 1)) * SS;
          const int kb = hi - KB * (b + 1), q = ct & (KB - 1);
#pragma unroll
          for (int u = 0; u < KB; ++u) {
            const int d = (ct + u * W) >> 3, i = kb - 1 - d;
            const bool ok = q + 1 + d <= bw && i >= lo;
            cp_async_elem(st + ((d + KB * (b + 1)) & (W - 1)) * LP + q,
                          ok ? L + size_t(i) * ldl + (q + 1 + d) : L, ok);
          }
#pragma unroll 1
          for (int e = ct; e < KB * KB; e += W) {
            const int c = e >> 3, dd = e & 7;
            const bool ok = c + dd < KB && dd <= bw && kb + c >= lo;
            cp_async_elem(st + LP * W + e, ok ? L + size_t(kb + c) * ldl + dd : L, ok);
          }
        }
        cp_async_commit();
      };
#pragma unroll 1
      for (int b = 0; b + 1 < NS; ++b) issue(b);
#pragma unroll 1
      for (int b = 0; b < nb; ++b) {
        cp_async_wait<NS - 2>();
        band_step_sync(2 * W);
        issue(b + NS - 1);
      }
      cp_async_wait<0>();
    } else if (lt < W) {
      auto value = [&](int r) { return r >= lo ? w[r] : T(0); };
      int row = hi - 1 - lt;
      T t = value(row), tn = value(row - W);
      // The known values that reach this row, eight entries in flight.
      const int reach = row >= lo ? min(R, row + bw + 1) - hi : 0;
      const T* Lr = L + size_t(max(row, lo)) * ldl + (hi - row);
#pragma unroll 1
      for (int r = 0; r < reach; r += 8) {
        T l[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) l[u] = r + u < reach ? Lr[r + u] : T(0);
#pragma unroll
        for (int u = 0; u < 8; ++u)
          if (r + u < reach) t = fma(-l[u], known[r + u], t);
      }
      if (lt < KB) {
        rhs[KB - 1 - lt] = t;
        row -= W;
        t = tn;
        tn = value(row - W);
      }
#pragma unroll 1
      for (int b = 0; b < nb; ++b) {
        band_step_sync(2 * W);
        const int kb = hi - KB * (b + 1);
        const T* st = ring + (b & (NS - 1)) * SS;
        if (b > 0 && lt < KB) v[kb + KB + lt] = done[((b - 1) & 1) * KB + lt];
        T dg[KB][KB], x[KB], l[KB];
        const T* rp = rhs + (b & 1) * KB;
        const T* blk = st + LP * W;
#pragma unroll
        for (int c = 0; c < KB; c += 2) band_pair(rp + c, x[c], x[c + 1]);
#pragma unroll
        for (int q = 0; q < KB; ++q) l[q] = st[lt * LP + q];
#pragma unroll
        for (int c = 0; c < KB; ++c)
#pragma unroll
          for (int d = 0; d < KB - c; d += 2) band_pair(blk + KB * c + d, dg[c][d], dg[c][d + 1]);
#pragma unroll
        for (int c = KB - 1; c >= 0; --c) {
          T s = x[c];
#pragma unroll
          for (int j = c + 1; j < KB; ++j) s = fma(-dg[c][j - c], x[j], s);
          x[c] = s * dg[c][0];
        }
        if (lt == 0) {
#pragma unroll
          for (int c = 0; c < KB; c += 2) band_pair_put(done + (b & 1) * KB + c, x[c], x[c + 1]);
        }
#pragma unroll
        for (int q = 0; q < KB; ++q) t = fma(-l[q], x[q], t);
        const int d = (lt - KB * (b + 1)) & (W - 1);
        if (d < KB && b + 1 < nb) {
          rhs[((b + 1) & 1) * KB + KB - 1 - d] = t;
          row -= W;
          t = tn;
          tn = value(row - W);
        }
      }
    }
    group_sync<BT>();
    if (lt < KB && nb > 0) {
      const int k = hi - KB * nb + lt;
      if (k >= lo) v[k] = done[((nb - 1) & 1) * KB + lt];
    }
    group_sync<BT>();
  }

  template <typename T>
  __device__ void band_chol_solve_global(T* v, T* w) {
    QTQP_BAND_LOCALS;
    const T* L = reinterpret_cast<const T*>(Lb);
    if (tid < 32) {
      const int lane = tid;
      for (int k = 0; k < n; ++k) {
        const T* ck = L + size_t(k) * ldl;
        const T zk = v[k] * ck[0];
        const int rows = min(bw, n - 1 - k);
        for (int d = 1 + lane; d <= rows; d += 32) v[k + d] = fma(-ck[d], zk, v[k + d]);
        if (lane == 0) w[k] = zk;
        __syncwarp();
      }
      for (int k = n - 1; k >= 0; --k) {
        const T xk = w[k] * L[size_t(k) * ldl];
        const int rows = min(bw, k);
        for (int d = 1 + lane; d <= rows; d += 32) {
          const int i = k - d;
          w[i] = fma(-L[size_t(i) * ldl + d], xk, w[i]);
        }
        if (lane == 0) v[k] = xk;
        __syncwarp();
      }
    }
    sync();
  }

  __device__ void band_kkt_solve(const double* r, double* out, bool accumulate, bool fp64) {
    QTQP_BAND_LOCALS;
    QTQP_TIC();
    const double* iry = vec(kPI);
    double* tmp = vec(kTMP);
    float* t32 = this->t32();
    for (int j = tid; j < n; j += NT) {
      const double g = r[j] + sparse_dot_ordered(jx, at, r + n, iry + n, jp[j], jp[j + 1]);
      if (fp64) {
        tmp[j] = g;
      } else {
        t32[j] = float(g);
      }
    }
    sync();
    QTQP_TOC(kPhSolveCols);
    {
      QTQP_TIC();
      if (fp64) {
        band_chol_solve<double>(tmp, vec(kW));
      } else {
        band_chol_solve<float>(t32, t32 + n);
      }
      QTQP_TOC(kPhTri);
    }
    for (int k = tid; k < N; k += NT) {
      double val;
      if (k < n) {
        val = fp64 ? tmp[k] : double(t32[k]);
      } else {
        const int i = k - n;
        const double ax = fp64 ? sparse_dot_ordered(ix, av, tmp, nullptr, ip[i], ip[i + 1])
                               : sparse_dot_ordered(ix, av, t32, nullptr, ip[i], ip[i + 1]);
        val = iry[k] * (ax - r[k]);
      }
      out[k] = accumulate ? out[k] + val : val;
    }
    QTQP_TOC(kPhSolve);
  }

  __device__ void band_kkt_residual(const double* v, const double* krhs, double* res,
                                    double& mres, double& vnan) const {
    QTQP_BAND_LOCALS;
    const double* reg = vec(kREG);
    const double* corr = vec(kCORR);
    for (int k = tid; k < N; k += NT) {
      double kv;
      if (k < n) {
        double t = band_poff_row(v, k);
        t += reg[k] * v[k];
        kv = t + band_at_col(v, k);
      } else {
        kv = band_a_row(v, k - n) - (-reg[k]) * v[k];
      }
      const double rk = krhs[k] - kv + corr[k] * v[k];
      res[k] = rk;
      mres = nanmax(mres, fabs(rk));
      vnan = fmax(vnan, (v[k] != v[k]) ? 1.0 : 0.0);
    }
  }
};

template <int NT>
using DenseIpm = Ipm<NT, kFmtDense>;

}  // namespace qtqp
