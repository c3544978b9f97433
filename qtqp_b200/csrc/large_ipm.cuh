// Large-format phases of the device IPM (FMT == kFmtLarge): one large dense QP
// solved by a cooperative grid of kLargeBlocks blocks.  The interior-point
// logic is the shared Ipm code; here are the KKT factorisation and the
// triangular solves, blocked for the whole GPU:
//
//   Gram      G = P_off + diag(Rx) + A^T diag(1/Ry) A  (solvers_dense.py:99-116)
//             FP32 factor: X = (diag(1/sqrt(Ry)) A)^T split into TF32 hi + lo,
//             lower 128 x 128 tiles of X X^T on tcgen05 (three TF32 products,
//             FP32 accumulation in TMEM).  FP64 factor: lower 128 x 128 tiles
//             on the FP64 tensor cores (DMMA, mma.sync m8n8k4).
//   Cholesky  right-looking with 128-wide panels: the diagonal block by one
//             CTA in shared memory, the panel eight rows per warp (both DMMA),
//             the trailing update in 128 x 128 tiles (DMMA in FP64, 8 x 8
//             register tiles in FP32); then the inverse of every diagonal block.
//   Solves    block forward / backward substitution with the inverted
//             diagonal blocks; CTA j owns block row j and polls the value
//             slots of the blocks it needs, one grid barrier per solve.
//
// Padding: the factor is npad x npad (npad = n rounded up to 128) with an
// identity on the padded diagonal; X is npad x mpad with zero padding.
#pragma once

#include "dense_ipm.cuh"
#include "tc_common.cuh"

namespace qtqp {

constexpr int kLB = 128;                          // panel / diagonal block size
constexpr int kLargeBlocks = 148;                 // CTAs of the cooperative grid: one per SM
constexpr int kLargeNT = kLargeBlocks * kGridBT;  // 37888 threads
constexpr int kTcStages = 3;
constexpr uint32_t kTcTileBytes = kLB * 32 * 4;        // 128 rows x 32 FP32
constexpr uint32_t kTcStageBytes = 4 * kTcTileBytes;   // A hi, B hi, A lo, B lo
constexpr size_t kArenaBytes = kTcStages * kTcStageBytes;  // 192 KB
constexpr size_t kLargeSmem = 1024 + kArenaBytes + 256;    // + alignment + barriers

__host__ __device__ inline int round_up(int v, int q) { return (v + q - 1) / q * q; }

constexpr int kPitch = kLB + 1;   // shared-memory pitch of a staged 128 x 128 block
constexpr int kSubPitch = 36;     // pitch of a staged 32 x 32 block
// Pitch of a 128 x 128 block whose rows feed the FP64 tensor cores: 4 (mod 16),
// so that a half-warp's fragment (4 rows x 4 columns) hits 16 banks, as does
// kSubPitch.
constexpr int kMmaPitch = kLB + 4;

// The split of the FP64 Gram matrix over the CTAs: the lower 128 x 128 tiles,
// row by row, times their slices of kGramKS rows of A are one sequence of
// units, of which CTA c < ctas takes [unit0(c), unit0(c + 1)).  Whole tiles go
// straight to G; a part of a tile goes to the CTA's slot 2 c (its first tile) or
// 2 c + 1 (its last), and large_finish_gram adds a tile's parts in order.
// Whole tiles only would leave the last wave nearly empty (n = 4096: 528 tiles
// = 3.6 waves of 148) or most CTAs idle (n = 1000: 36 tiles).
constexpr int kGramKS = 32;
constexpr int kGramMinUnits = 4;  // slices per CTA at least, else fewer CTAs
struct GramSplit {
  int slices, ctas;
  long long units;
  __host__ __device__ GramSplit(int npad, int m) {
    const int nt = npad / kLB;
    const long long tiles = (long long)nt * (nt + 1) / 2;
    slices = m > kGramKS ? (m + kGramKS - 1) / kGramKS : 1;
    units = tiles * slices;
    const long long want = units / kGramMinUnits > tiles ? units / kGramMinUnits : tiles;
    ctas = want < kLargeBlocks ? int(want) : kLargeBlocks;
  }
  __host__ __device__ size_t slot_bytes() const { return size_t(2) * ctas * kLB * kLB * 8; }
  __device__ long long unit0(int c) const { return c * units / ctas; }
  __device__ int owner(long long u) const { return int(((u + 1) * ctas - 1) / units); }
};

// Global workspace of a large solve.
struct LargeLayout {
  int n, m, npad, mpad, nblk, np;
  size_t ctl_off, tri_off, info_off, v_off, a_off, p_off, g64_off, g32_off, sinv_off, xhi_off, xlo_off,
      cp_off, gpart_off, total;
};
__host__ __device__ inline LargeLayout plan_large_layout(int n, int m) {
  LargeLayout L;
  L.n = n;
  L.m = m;
  L.npad = round_up(n, kLB);
  L.mpad = round_up(m, 32);
  L.nblk = L.npad / kLB;
  L.np = (max(n + m, n + 4) + 1) & ~1;
  auto al = [](size_t b) { return (b + 1023) & ~size_t(1023); };
  size_t off = 0;
  L.ctl_off = off;
  off += al(sizeof(GridCtl));
  L.tri_off = off;  // slots of the triangular solves; zeroed with the control block
  off += al(size_t(L.npad) * sizeof(GridSlot));
  L.info_off = off;
  off += al(16);
  L.v_off = off;
  off += al(size_t(kNumVec) * L.np * 8);
  L.a_off = off;
  off += al(size_t(m) * n * 8);
  L.p_off = off;
  off += al(size_t(n) * n * 8);
  L.g64_off = off;
  off += al(size_t(L.npad) * L.npad * 8);
  L.g32_off = off;
  off += al(size_t(L.npad) * L.npad * 4);
  L.sinv_off = off;
  off += al(4 * 32 * kSubPitch * 8);               // sub-block inverses of one step
  L.xhi_off = off;
  off += al(size_t(L.npad) * L.mpad * 4);
  L.xlo_off = off;
  off += al(size_t(L.npad) * L.mpad * 4);
  L.cp_off = off;  // per-block column sums of large_products
  off += al(size_t(kLargeBlocks) * L.npad * 8);
  L.gpart_off = off;  // parts of split Gram tiles
  off += al(GramSplit(L.npad, m).slot_bytes());
  L.total = off;
  return L;
}

// Ruiz equilibration of the working copies (the sweeps of load_and_equilibrate,
// bit for bit: maxima have no rounding, and every entry takes the same products
// d_i e_j).  One pass over the rows of [A; P] per sweep applies the last sweep's
// scales and takes the next one's row and column maxima; each block has a
// contiguous band of rows, nw warps share a row (512 columns each) and the
// block's other warps take other rows.
// Bound by HBM (a pass reads and writes both matrices; 1.3 ms for n = 4096, m =
// 8192 at the copy rate).  Three separate passes per sweep, the column one strided,
// made the whole solve 7 ms longer there (144.5 ms, now 137.5).
template <class S>
__device__ __noinline__ void large_equilibrate(S& s) {
  constexpr int kTile = 4096, kChunk = 1024, kCpl = 16;
  const int n = s.n, m = s.m, tid = s.tid, N = s.N;
  double* sc = s.vec(kTMP);   // the last sweep's [e; d]
  double* rmx = s.vec(kREG);  // the rows' maxima (not in use yet)
  double* de = s.vec(kDE);
  unsigned long long* ckey = reinterpret_cast<unsigned long long*>(s.arena);  // kTile
  unsigned long long* rkey = ckey + kTile;                                     // kChunk
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int total = m + (s.has_p ? n : 0), per = (total + gridDim.x - 1) / gridDim.x;
  const int i0 = min(total, int(blockIdx.x) * per), i1 = min(total, i0 + per);
  int nw = 1;
  while (nw < kGridBT / 32 && nw * 32 * kCpl < n) nw *= 2;
  const int groups = kGridBT / 32 / nw, grp = warp / nw, wc = warp % nw;
  double* part = s.colpart + size_t(blockIdx.x) * s.npad;
  for (int sweep = 0; sweep <= 10; ++sweep) {
    for (int j = threadIdx.x; i0 >= i1 && j < n; j += kGridBT) part[j] = 0.0;
    for (int c0 = i0; c0 < i1; c0 += kChunk) {
      const int ce = min(i1, c0 + kChunk);
      for (int k = threadIdx.x; k < kChunk; k += kGridBT) rkey[k] = 0;
      for (int t0 = 0; t0 < n; t0 += kTile) {
        for (int k = threadIdx.x; k < kTile; k += kGridBT) ckey[k] = 0;
        __syncthreads();
        const int j0 = t0 + wc * 32 * kCpl + lane;
        double e[kCpl], cm[kCpl];
#pragma unroll
        for (int q = 0; q < kCpl; ++q) {
          e[q] = sweep > 0 && j0 + 32 * q < n ? sc[j0 + 32 * q] : 1.0;
          cm[q] = 0.0;
        }
        for (int i = c0 + grp; i < ce; i += groups) {
          double* row = (i < m ? s.A + size_t(i) * s.lda : s.P + size_t(i - m) * s.ldp) + j0;
          const double d = sweep == 0 ? 1.0 : i < m ? sc[n + i] : sc[i - m];
          double v[kCpl], mx = 0.0;
#pragma unroll
          for (int q = 0; q < kCpl; ++q) v[q] = j0 + 32 * q < n ? row[32 * q] : 0.0;
#pragma unroll
          for (int q = 0; q < kCpl; ++q) {
            if (sweep > 0) {
              v[q] *= d * e[q];
              if (j0 + 32 * q < n) row[32 * q] = v[q];
            }
            const double av = fabs(v[q]);
            cm[q] = fmax(cm[q], av);
            mx = fmax(mx, av);
          }
          if (i < m && sweep < 10) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            if (lane == 0) atomicMax(rkey + (i - c0), (unsigned long long)__double_as_longlong(mx));
          }
        }
        if (sweep < 10) {
#pragma unroll
          for (int q = 0; q < kCpl; ++q)
            if (j0 + 32 * q < n)
              atomicMax(ckey + (j0 + 32 * q - t0), (unsigned long long)__double_as_longlong(cm[q]));
        }
        __syncthreads();
        for (int k = threadIdx.x; sweep < 10 && k < kTile && t0 + k < n; k += kGridBT) {
          const double v = __longlong_as_double(ckey[k]);
          part[t0 + k] = c0 == i0 ? v : fmax(part[t0 + k], v);
        }
        __syncthreads();
      }
      for (int k = threadIdx.x; sweep < 10 && k < kChunk && c0 + k < min(ce, m); k += kGridBT)
        rmx[c0 + k] = __longlong_as_double(rkey[k]);
      __syncthreads();
    }
    s.sync();
    if (sweep == 10) break;
    for (int k = tid; k < N; k += kLargeNT) {
      double mx = 0.0;
      if (k < n) {
#pragma unroll 4
        for (int b = 0; b < int(gridDim.x); ++b) mx = fmax(mx, s.colpart[size_t(b) * s.npad + k]);
      } else {
        mx = rmx[k - n];
      }
      if (mx == 0.0) mx = 1.0;
      sc[k] = fmin(fmax(1.0 / sqrt(mx), 1e-3), 1e3);
      de[k] *= sc[k];
    }
    s.sync();
  }
}

// ---------------------------------------------------------------------------
// One pass over the rows of A (and P) for the products a KKT residual needs
// together: the row dots (A vx)_i, passed to row_epi(i, value) by one thread
// each (none when vx is null), and the column sums c_k = sum_i A_ik vy_i
// vs_i (vs null: 1) + sum_i P_ik vp_i (when vp is given; P is symmetric, so
// that is (P vp)_k), passed to col_epi(k, c_k) by the thread k % NT after a
// grid barrier.  The rows of the stacked matrix
// [A; P] are cut into one contiguous band per block, and each band into
// chunks of kPrRows rows; within a tile of kPrTile columns each warp takes
// kPrCpl x 32 consecutive columns (lane l: columns l + 32 t), so every row is
// read once, coalesced, with kPrCpl loads in flight per lane, and each lane
// keeps its columns' sums in registers over the chunk.  The row dots of a
// chunk are combined over warps and tiles in shared memory; the blocks'
// column sums go to global memory and are added in block order.  Every sum
// runs in a fixed order, so the results are the same on every run.
// ---------------------------------------------------------------------------
constexpr int kPrCpl = 16;                         // columns per lane in a tile
constexpr int kPrTile = (kGridBT / 32) * 32 * kPrCpl;  // 4096 columns
constexpr int kPrRows = 256;                       // rows per chunk (rowpart in smem)
// The products' shared memory starts behind the diagonal-block inverse (128
// x 129 doubles) and the partial sums (128) that large_chol_solve keeps
// resident in the arena from the factorisation on.
constexpr size_t kPrSmemOff = (size_t(kLB) * (kLB + 1) + kLB) * sizeof(double);
static_assert(kPrSmemOff + (size_t(kPrRows) * (kGridBT / 32) + kPrTile) * sizeof(double) <=
                  kArenaBytes, "the products' shared memory exceeds the arena");

template <class S, class RowEpi, class ColEpi>
__device__ void large_products(S& s, const double* vx, const double* vy, const double* vs,
                               const double* vp, RowEpi row_epi, ColEpi col_epi) {
  constexpr int NW = kGridBT / 32;
  const int n = s.n, m = s.m, lda = s.lda, ldp = s.ldp;
  const double* A = s.A;
  const double* P = s.P;
  const int G = gridDim.x, b = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rows = m + (vp != nullptr ? n : 0);
  const int band = (rows + G - 1) / G;
  const int r0 = min(rows, b * band), r1 = min(rows, r0 + band);
  double* rowpart = reinterpret_cast<double*>(s.arena + kPrSmemOff);  // kPrRows x NW
  double* xs = rowpart + kPrRows * NW;                    // vx of one tile
  double* part = s.colpart + size_t(b) * s.npad;
  for (int k = threadIdx.x; k < n; k += blockDim.x) part[k] = 0.0;
  __syncthreads();
  for (int c0 = r0; c0 < r1; c0 += kPrRows) {
    const int c1 = min(r1, c0 + kPrRows);
    for (int e = threadIdx.x; e < (c1 - c0) * NW; e += blockDim.x) rowpart[e] = 0.0;
    for (int t0 = 0; t0 < n; t0 += kPrTile) {
      if (vx != nullptr)
        for (int k = threadIdx.x; k < kPrTile; k += blockDim.x)
          xs[k] = t0 + k < n ? vx[t0 + k] : 0.0;
      __syncthreads();
      const int cb = t0 + warp * 32 * kPrCpl + lane;  // this lane's first column
      double acc[kPrCpl];
#pragma unroll
      for (int t = 0; t < kPrCpl; ++t) acc[t] = 0.0;
      auto row_of = [&](int i) {
        return i < m ? A + size_t(i) * lda : P + size_t(i - m) * ldp;
      };
      auto weight_of = [&](int i) {
        return i < m ? (vs != nullptr ? vy[i] * vs[i] : vy[i]) : vp[i - m];
      };
      // The row dot of row i from its loaded values (the same branch for the
      // whole warp).
      auto row_dot = [&](int i, const double (&a)[kPrCpl]) {
        if (i < m && vx != nullptr) {
          double d = 0.0;
#pragma unroll
          for (int t = 0; t < kPrCpl; ++t) d = fma(a[t], xs[cb - t0 + 32 * t], d);
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) d += __shfl_xor_sync(0xffffffffu, d, o);
          if (lane == 0) rowpart[(i - c0) * NW + warp] += d;
        }
      };
      // Two rows per step, all of their loads issued before the first use
      // (2 x kPrCpl loads in flight per lane); the column sums still add row
      // i before row i + 1.
      int i = c0;
      for (; i + 1 < c1; i += 2) {
        const double* M0 = row_of(i);
        const double* M1 = row_of(i + 1);
        double a0[kPrCpl], a1[kPrCpl];
#pragma unroll
        for (int t = 0; t < kPrCpl; ++t) {
          const bool in = cb + 32 * t < n;
          a0[t] = in ? M0[cb + 32 * t] : 0.0;
          a1[t] = in ? M1[cb + 32 * t] : 0.0;
        }
        const double w0 = weight_of(i), w1 = weight_of(i + 1);
#pragma unroll
        for (int t = 0; t < kPrCpl; ++t) acc[t] = fma(a1[t], w1, fma(a0[t], w0, acc[t]));
        row_dot(i, a0);
        row_dot(i + 1, a1);
      }
      if (i < c1) {
        const double* M0 = row_of(i);
        double a0[kPrCpl];
#pragma unroll
        for (int t = 0; t < kPrCpl; ++t) a0[t] = cb + 32 * t < n ? M0[cb + 32 * t] : 0.0;
        const double w0 = weight_of(i);
#pragma unroll
        for (int t = 0; t < kPrCpl; ++t) acc[t] = fma(a0[t], w0, acc[t]);
        row_dot(i, a0);
      }
#pragma unroll
      for (int t = 0; t < kPrCpl; ++t)
        if (cb + 32 * t < n) part[cb + 32 * t] += acc[t];
      __syncthreads();
    }
    for (int i = c0 + threadIdx.x; i < c1 && vx != nullptr; i += blockDim.x) {
      if (i >= m) continue;
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < NW; ++w) v += rowpart[(i - c0) * NW + w];
      row_epi(i, v);
    }
    __syncthreads();
  }
  s.sync();
  for (int k = s.tid; k < n; k += kLargeNT) {
    double v = 0.0;
    for (int bb = 0; bb < G; ++bb) v += s.colpart[size_t(bb) * s.npad + k];
    col_epi(k, v);
  }
}

// ---------------------------------------------------------------------------
// Gram of the FP32 factor on tcgen05.
// ---------------------------------------------------------------------------
// X = (diag(w) A)^T split into TF32 hi + lo (w = 1/sqrt(Ry) at vec(kPW)[n+i]),
// by 32 x 32 tiles transposed through shared memory.
template <class S>
__device__ void large_scale_split(S& s) {
  const int n = s.n, m = s.m, npad = s.npad, mpad = s.mpad;
  const double* A = s.A;
  const double* w = s.vec(kPW) + n;
  float* t = reinterpret_cast<float*>(s.arena);  // 32 x 33
  const int tr = threadIdx.x >> 5, tc = threadIdx.x & 31;  // 8 rows per pass
  const int tiles_i = mpad / 32, tiles_j = npad / 32;
  for (int t_id = blockIdx.x; t_id < tiles_i * tiles_j; t_id += gridDim.x) {
    const int i0 = (t_id % tiles_i) * 32, j0 = (t_id / tiles_i) * 32;
    for (int r = tr; r < 32; r += 8) {  // rows i of A, columns j coalesced
      const int i = i0 + r, j = j0 + tc;
      t[r * 33 + tc] = (i < m && j < n) ? float(A[size_t(i) * n + j] * w[i]) : 0.0f;
    }
    __syncthreads();
    for (int r = tr; r < 32; r += 8) {  // rows j of X, columns i coalesced
      const float v = t[tc * 33 + r];
      uint32_t h;
      asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(v));
      const size_t o = size_t(j0 + r) * mpad + i0 + tc;
      s.xhi[o] = __uint_as_float(h);
      s.xlo[o] = v - __uint_as_float(h);
    }
    __syncthreads();
  }
}

// Lower 128 x 128 tiles of X X^T (three TF32 products) into g32.  Warp 0
// lane 0 loads (TMA, 3-stage ring), warp 1 lane 0 issues the MMAs, all
// eight warps drain TMEM (warp w: lanes 32 (w % 4), columns 64 (w / 4)).
// The ring counters continue across tiles and calls (s.tc_load / s.tc_mma /
// s.tc_tiles are per-thread copies; each role advances its own).
template <class S>
__device__ void large_gram_tc(S& s) {
  const int npad = s.npad, k_tiles = s.mpad / 32, nt = npad / kLB;
  uint8_t* ring = s.arena;
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + kArenaBytes);
  uint64_t* full = bars;
  uint64_t* empty = bars + kTcStages;
  uint64_t* done = bars + 2 * kTcStages;
  int* failed = reinterpret_cast<int*>(done + 1);
  const CUtensorMap* mh = static_cast<const CUtensorMap*>(s.map_hi);
  const CUtensorMap* ml = static_cast<const CUtensorMap*>(s.map_lo);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t idesc = tc::idesc_f32acc(kLB, kLB, false);
  const int tiles = nt * (nt + 1) / 2;
  for (int t = blockIdx.x; t < tiles; t += gridDim.x) {
    int ti = 0;
    while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
    const int tj = t - ti * (ti + 1) / 2;
    if (warp == 0 && lane == 0) {
      for (int kt = 0; kt < k_tiles; ++kt) {
        const uint32_t g = s.tc_load++;
        const int st = int(g % kTcStages);
        const uint32_t use = g / kTcStages;
        if (use > 0 && !tc::mbar_wait(&empty[st], (use - 1) & 1)) {
          s.tc_load--;  // stage g was not issued
          atomicExch(failed, 1);
          break;
        }
        uint8_t* sb = ring + st * kTcStageBytes;
        tc::mbar_arrive_expect_tx(&full[st], kTcStageBytes);
        tc::tma_load_2d(sb, mh, kt * 32, ti * kLB, &full[st]);
        tc::tma_load_2d(sb + kTcTileBytes, mh, kt * 32, tj * kLB, &full[st]);
        tc::tma_load_2d(sb + 2 * kTcTileBytes, ml, kt * 32, ti * kLB, &full[st]);
        tc::tma_load_2d(sb + 3 * kTcTileBytes, ml, kt * 32, tj * kLB, &full[st]);
      }
    } else if (warp == 1 && lane == 0) {
      for (int kt = 0; kt < k_tiles; ++kt) {
        const uint32_t g = s.tc_mma++;
        const int st = int(g % kTcStages);
        const uint32_t use = g / kTcStages;
        if (!tc::mbar_wait(&full[st], use & 1)) {
          s.tc_mma--;  // stage g was not consumed
          atomicExch(failed, 1);
          break;
        }
        tc::fence_after_sync();
        const uint32_t a_hi = tc::smem_u32(ring + st * kTcStageBytes);
        const uint32_t b_hi = a_hi + kTcTileBytes, a_lo = a_hi + 2 * kTcTileBytes,
                       b_lo = a_hi + 3 * kTcTileBytes;
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          const uint32_t off = kk * 32;
          tc::mma_tf32(s.tmem, tc::desc_kmajor_sw128(a_hi + off), tc::desc_kmajor_sw128(b_hi + off),
                       idesc, (kt | kk) != 0);
          tc::mma_tf32(s.tmem, tc::desc_kmajor_sw128(a_hi + off), tc::desc_kmajor_sw128(b_lo + off),
                       idesc, 1);
          tc::mma_tf32(s.tmem, tc::desc_kmajor_sw128(a_lo + off), tc::desc_kmajor_sw128(b_hi + off),
                       idesc, 1);
        }
        tc::mma_commit(&empty[st]);
      }
      tc::mma_commit(done);
    }
    __syncwarp();
    if (!tc::mbar_wait(done, s.tc_tiles & 1)) atomicExch(failed, 1);
    s.tc_tiles++;
    tc::fence_after_sync();
    if (warp == 1 && lane == 0) failed[1] = int(s.tc_mma);  // stages consumed so far
    __syncthreads();
    if (*failed != 0) {
      // A bounded wait gave up: stop issuing tiles.  Before the CTA moves on,
      // the producer waits (again bounded) for the stages it issued that the
      // MMA issuer never consumed, so that no bulk copy still targets the
      // ring when the arena is reused.
      if (warp == 0 && lane == 0) {
        for (uint32_t g = uint32_t(failed[1]); g < s.tc_load; ++g)
          if (!tc::mbar_wait(&full[g % kTcStages], (g / kTcStages) & 1)) break;
      }
      __syncthreads();
      break;
    }
    {
      const int q = warp & 3, half = warp >> 2;
      const int row = ti * kLB + q * 32 + lane;
      float* grow = s.g32l + size_t(row) * npad + size_t(tj) * kLB + half * 64;
#pragma unroll 1
      for (int c0 = 0; c0 < 64; c0 += 32) {
        float v[32];
        tc::tmem_ld32(s.tmem + (uint32_t(q * 32) << 16) + uint32_t(half * 64 + c0), v);
#pragma unroll
        for (int e = 0; e < 32; e += 4)
          *reinterpret_cast<float4*>(grow + c0 + e) = make_float4(v[e], v[e + 1], v[e + 2], v[e + 3]);
      }
    }
    tc::fence_before_sync();
    __syncthreads();  // TMEM free for the next tile's MMAs
  }
  if (threadIdx.x == 0 && *failed) grid_fail(s.gctl);
}

// Row and column of lower tile t (row by row).
__device__ __forceinline__ void lower_tile(int t, int& ti, int& tj) {
  ti = int((sqrtf(8.0f * float(t) + 1.0f) - 1.0f) * 0.5f);
  while (ti * (ti + 1) / 2 > t) --ti;
  while ((ti + 1) * (ti + 2) / 2 <= t) ++ti;
  tj = t - ti * (ti + 1) / 2;
}

// G_lower = A^T diag(1/Ry) A in FP64 on the FP64 tensor cores (DMMA,
// mma.sync m8n8k4): slices of 32 rows of A (both column panels) and their
// weights staged by cp.async into two buffers, with a row pitch of 132 so that
// each half-warp's fragment loads hit 16 different banks; warp w computes the
// 64 x 32 block (w / 4, w % 4) of the tile with 8 x 4 accumulators of 8 x 8.
// Rows and columns beyond m, n are zero-filled.  Rows of A that start on 16
// bytes (even lda) are copied 16 bytes at a time.
// Bound by the FP64 tensor cores (36.7 TFLOP/s alone).  n = 4096, m = 8192, rate
// within a tile: 26.5 TFLOP/s with 8-byte copies, slices of 16 rows, two barriers
// each and the weights on the longer fragment; 29.1 with 16-byte copies, 30.6
// with one barrier and the weights on the shorter one, 31.2 with slices of 32
// rows.  (Row copies by the TMA unit: 31.0, so the copies no longer matter.)
template <int VEC, class S>
__device__ __noinline__ void large_gram_dmma(S& s) {
  const int n = s.n, m = s.m, npad = s.npad, lda = s.lda;
  const double* A = s.A;
  const double* iry = s.vec(kPI) + n;  // 1 / Ry
  constexpr int KS = kGramKS;
  constexpr int LP = kLB + 4;          // staged row pitch
  constexpr int SL = 2 * KS * LP + KS; // doubles per buffer
  static_assert(2 * SL * sizeof(double) <= kArenaBytes, "Gram buffers exceed the arena");
  double* smem = reinterpret_cast<double*>(s.arena);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int gi = lane >> 2, tg = lane & 3;
  const int wr = warp >> 2, wc = warp & 3;
  const GramSplit P(npad, m);
  if (int(blockIdx.x) >= P.ctas) return;
  auto issue = [&](int r0, int i0, int j0, int buf) {
    double* sa = smem + buf * SL;
    double* sb = sa + KS * LP;
    double* sw = sb + KS * LP;
    constexpr int kPer = kLB / VEC;  // copies per row and panel
#pragma unroll
    for (int q = 0; q < KS * kPer / kGridBT; ++q) {
      const int e = threadIdx.x + q * kGridBT, r = e / kPer, c = e % kPer * VEC, i = r0 + r;
      const bool ok = i < m;
      if constexpr (VEC == 2) {
        const int ba = ok ? max(0, min(16, 8 * (n - i0 - c))) : 0;
        const int bb = ok ? max(0, min(16, 8 * (n - j0 - c))) : 0;
        cp_async16z(sa + r * LP + c, A + (ba ? size_t(i) * lda + i0 + c : 0), ba);
        cp_async16z(sb + r * LP + c, A + (bb ? size_t(i) * lda + j0 + c : 0), bb);
      } else {
        cp_async8(sa + r * LP + c, A + (ok && i0 + c < n ? size_t(i) * lda + i0 + c : 0),
                  ok && i0 + c < n);
        cp_async8(sb + r * LP + c, A + (ok && j0 + c < n ? size_t(i) * lda + j0 + c : 0),
                  ok && j0 + c < n);
      }
    }
    if (threadIdx.x < KS) {
      const int i = r0 + threadIdx.x;
      cp_async8(sw + threadIdx.x, iry + (i < m ? i : 0), i < m);
    }
    cp_async_commit();
  };
  const long long u0 = P.unit0(blockIdx.x), u1 = P.unit0(blockIdx.x + 1);
  for (long long u = u0; u < u1;) {
    const int t = int(u / P.slices), qa = int(u - (long long)t * P.slices);
    const int qb = int(min((long long)P.slices, qa + (u1 - u)));
    int ti, tj;
    lower_tile(t, ti, tj);
    const int i0 = ti * kLB, j0 = tj * kLB;
    double acc[8][4][2];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
    issue(qa * KS, i0, j0, 0);
    int buf = 0;
    for (int q = qa; q < qb; ++q) {
      // Slice q has landed, and every warp is done with slice q - 1, whose
      // buffer takes slice q + 1.
      cp_async_wait<0>();
      __syncthreads();
      if (q + 1 < qb) issue((q + 1) * KS, i0, j0, buf ^ 1);
      const double* sa = smem + buf * SL + wr * 64 + gi;
      const double* sb = smem + buf * SL + KS * LP + wc * 32 + gi;
      const double* sw = smem + buf * SL + 2 * KS * LP;
#pragma unroll
      for (int k0 = 0; k0 < KS; k0 += 4) {
        const int r = k0 + tg;
        const double w = sw[r];
        double a[8], b[4];
#pragma unroll
        for (int mi = 0; mi < 8; ++mi) a[mi] = sa[r * LP + mi * 8];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) b[ni] = sb[r * LP + ni * 8] * w;
#pragma unroll
        for (int mi = 0; mi < 8; ++mi)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni) dmma_8x8x4(acc[mi][ni], a[mi], b[ni]);
      }
      buf ^= 1;
    }
    __syncthreads();
    const bool whole = qb - qa == P.slices;
    double* out = whole ? s.g64 + size_t(i0) * npad + j0
                        : s.gpart + (size_t(2) * blockIdx.x + (u == u0 ? 0 : 1)) * kLB * kLB;
    const size_t ldo = whole ? npad : kLB;
#pragma unroll
    for (int mi = 0; mi < 8; ++mi)
#pragma unroll
      for (int ni = 0; ni < 4; ++ni)
        *reinterpret_cast<double2*>(out + (wr * 64 + mi * 8 + gi) * ldo + wc * 32 + ni * 8 + 2 * tg) =
            make_double2(acc[mi][ni][0], acc[mi][ni][1]);
    u += qb - qa;
  }
}

// G += P_off + diag(Rx) on the lower triangle (FP64: of the sums of the tiles'
// parts, see GramSplit), identity padding, then the relative diagonal jitter
// (1e-14 in FP64 as solvers_dense.py:112; 2^-22 at FP32 resolution).
template <typename T, class S>
__device__ void large_finish_gram(S& s, T* g) {
  const int n = s.n, npad = s.npad, tid = s.tid;
  const double* P = s.P;
  const double* reg = s.vec(kREG);
  double dmax[1] = {0.0};
  double dummy[1] = {0.0};
  const GramSplit sp(npad, s.m);
  const int nt = npad / kLB, tiles = nt * (nt + 1) / 2;
  constexpr int kRows = 16;  // rows of a work item, two per warp
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int it = blockIdx.x; it < tiles * (kLB / kRows); it += gridDim.x) {
    const int t = it / (kLB / kRows);
    int ti, tj;
    lower_tile(t, ti, tj);
    const int row0 = it % (kLB / kRows) * kRows + 2 * warp;
    // This lane's entries q: row row0 + q / 4, column lane + 32 (q % 4) of the tile.
    T* gt = g + (size_t(ti) * kLB + row0) * npad + tj * kLB + lane;
    T sum[8];
    int c0 = 0, c1 = 0;
    if constexpr (sizeof(T) == 8) {
      c0 = sp.owner((long long)t * sp.slices);
      c1 = sp.owner((long long)(t + 1) * sp.slices - 1);
    }
    if (c0 == c1) {
#pragma unroll
      for (int q = 0; q < 8; ++q) sum[q] = gt[size_t(q >> 2) * npad + 32 * (q & 3)];
    } else if constexpr (sizeof(T) == 8) {
#pragma unroll
      for (int q = 0; q < 8; ++q) sum[q] = 0.0;
      for (int k = c0; k <= c1; ++k) {
        const bool first = sp.unit0(k) >= (long long)t * sp.slices;
        const double* part =
            s.gpart + ((size_t(2) * k + (first ? 0 : 1)) * kLB + row0) * kLB + lane;
#pragma unroll
        for (int q = 0; q < 8; ++q) sum[q] += part[(q >> 2) * kLB + 32 * (q & 3)];
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int i = ti * kLB + row0 + (q >> 2), j = tj * kLB + lane + 32 * (q & 3);
      if (j > i) continue;
      T* ge = gt + size_t(q >> 2) * npad + 32 * (q & 3);
      if (i >= n || j >= n) {
        *ge = (i == j) ? T(1) : T(0);
        continue;
      }
      double base = P[size_t(i) * s.ldp + j];
      if (i == j) base += reg[i];
      const T v = T(base) + sum[q];
      *ge = v;
      if (i == j) dmax[0] = nanmax(dmax[0], double(v));
    }
  }
  s.template reduce<0, 1>(dummy, dmax);
  const double jit = (sizeof(T) == 8 ? 1e-14 : 2.384185791015625e-07) * dmax[0];
  for (int k = tid; k < n; k += kLargeNT) g[size_t(k) * npad + k] = T(double(g[size_t(k) * npad + k]) + jit);
  s.sync();
}

// ---------------------------------------------------------------------------
// Blocked Cholesky of the lower triangle of g (npad x npad), then the
// inverses of the diagonal blocks, each resident in the shared memory of the
// CTA that owns the block in the solves.
// Returns 0 or the 1-based index of the first non-positive pivot (uniform
// over the grid).
//
// Step k (panel width 128):
//   (a) one CTA factors the diagonal block in shared memory and inverts its four
//       32 x 32 diagonal sub-blocks (cta_chol128); from the second step on it
//       does so during the trailing update of the step before, on the block it
//       has updated itself (cta_diag_update);
//   (b) every warp takes eight panel rows and solves x L_kk^T = g_i with the
//       sub-block inverses (warp_panel_rows);
//   (c) the lower 128 x 128 tiles right of the panel get g_ij -= L_ik L_jk^T
//       (trailing_tiles).
// (a) and (b) run on the FP64 tensor cores whatever T is, so the FP32 factor's
// diagonal blocks and panels are rounded once.
// ---------------------------------------------------------------------------
// 128 x 128 block of g at (r0, c0) into dst[r * kPitch + c], eight loads in
// flight per thread.
template <typename T>
__device__ __forceinline__ void stage_block(T* dst, const T* g, size_t ld, int r0, int c0) {
  for (int base = threadIdx.x; base < kLB * kLB; base += 8 * kGridBT) {
    T v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = base + q * kGridBT, r = e >> 7, c = e & 127;
      v[q] = g[size_t(r0 + r) * ld + c0 + c];
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = base + q * kGridBT;
      dst[(e >> 7) * kPitch + (e & 127)] = v[q];
    }
  }
}

// Two consecutive values of T as doubles, and back.
__device__ __forceinline__ void load_pair(double (&v)[2], const double* p) {
  const double2 t = *reinterpret_cast<const double2*>(p);
  v[0] = t.x;
  v[1] = t.y;
}
__device__ __forceinline__ void load_pair(double (&v)[2], const float* p) {
  const float2 t = *reinterpret_cast<const float2*>(p);
  v[0] = t.x;
  v[1] = t.y;
}
__device__ __forceinline__ void store_pair(double* p, const double (&v)[2]) {
  *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
}
__device__ __forceinline__ void store_pair(float* p, const double (&v)[2]) {
  *reinterpret_cast<float2*>(p) = make_float2(float(v[0]), float(v[1]));
}

// The 128 x 128 block of g (leading dimension ld) at (r0, c0) as doubles into
// dst (pitch kMmaPitch).
template <typename T>
__device__ __forceinline__ void stage_mma(double* dst, const T* g, size_t ld, int r0, int c0) {
  if constexpr (sizeof(T) == 8) {
#pragma unroll 8
    for (int q = 0; q < kLB * kLB / 2 / kGridBT; ++q) {
      const int e = threadIdx.x + q * kGridBT, r = e >> 6, c = 2 * (e & 63);
      cp_async16(dst + r * kMmaPitch + c, g + size_t(r0 + r) * ld + c0 + c);
    }
    cp_async_commit();
    cp_async_wait<0>();
  } else {
#pragma unroll 1
    for (int base = 0; base < kLB * kLB / 2; base += 8 * kGridBT) {
      double v[8][2];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int e = base + threadIdx.x + q * kGridBT;
        load_pair(v[q], g + size_t(r0 + (e >> 6)) * ld + c0 + 2 * (e & 63));
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int e = base + threadIdx.x + q * kGridBT;
        store_pair(dst + (e >> 6) * kMmaPitch + 2 * (e & 63), v[q]);
      }
    }
  }
  __syncthreads();
}

// sm = (the diagonal block of g at row b0) - L L^T, lower part, with L the 128
// rows b0 .. of the panel at column k0 (pitch kMmaPitch; the strict upper part
// of sm is undefined).  The block's 20 lower 16 x 32 units go to the eight
// warps, five per pair that shares a tensor core, with L staged whole.
// Bound by the SM's FP64 tensor cores: 29000 cycles, against 70000 for a square
// tile through the trailing update's loop, written back and staged again (and
// that on the chain of the factorisation).
template <typename T>
__device__ __noinline__ void cta_diag_update(double* sm, const T* g, size_t ld, int b0, int k0) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3;
  stage_mma(sm, g, ld, b0, k0);
  // Unit u: 16 rows at 16 ui, 32 columns at 32 uj (2 uj <= ui + 1).
  int ui[3], uj[3];
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    const int u = warp + 8 * q;
    // Units of the row pair p (rows 32 p ..): 2 (p + 1), starting at p (p + 1).
    int p = 0;
    while (p < 3 && (p + 1) * (p + 2) <= u) ++p;
    const int e = u - p * (p + 1);
    ui[q] = 2 * p + (e > p ? 1 : 0);
    uj[q] = e > p ? e - p - 1 : e;
  }
  double acc[3][2][4][2];
#pragma unroll
  for (int q = 0; q < 3; ++q)
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[q][a][b][0] = acc[q][a][b][1] = 0.0;
  const bool third = warp < 4;
#pragma unroll 2
  for (int k = 0; k < kLB; k += 4) {
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      if (q == 2 && !third) continue;
      const double* ra = sm + (16 * ui[q] + gi) * kMmaPitch + k + tg;
      const double* rb = sm + (32 * uj[q] + gi) * kMmaPitch + k + tg;
      double a[2], b[4];
#pragma unroll
      for (int x = 0; x < 2; ++x) a[x] = ra[x * 8 * kMmaPitch];
#pragma unroll
      for (int x = 0; x < 4; ++x) b[x] = rb[x * 8 * kMmaPitch];
#pragma unroll
      for (int x = 0; x < 2; ++x)
#pragma unroll
        for (int y = 0; y < 4; ++y) dmma_8x8x4(acc[q][x][y], a[x], b[y]);
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    if (q == 2 && !third) continue;
#pragma unroll
    for (int x = 0; x < 2; ++x)
#pragma unroll
      for (int y = 0; y < 4; ++y) {
        const int r = 16 * ui[q] + 8 * x + gi, c = 32 * uj[q] + 8 * y + 2 * tg;
        double v[2];
        load_pair(v, g + size_t(b0 + r) * ld + b0 + c);
        v[0] -= acc[q][x][y][0];
        v[1] -= acc[q][x][y][1];
        store_pair(sm + r * kMmaPitch + c, v);
      }
  }
  __syncthreads();
}

// C -= A B^T for one 8 x 8 tile and inner length 8, all in shared memory with
// pitch kMmaPitch, the calling warp; valid: whether to store (uniform).
__device__ __forceinline__ void warp_tile8(double* C, const double* A, const double* B, bool valid) {
  const int lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3;
  double* out = C + gi * kMmaPitch + 2 * tg;
  double acc[2];
  load_pair(acc, out);
#pragma unroll
  for (int h = 0; h < 8; h += 4)
    dmma_8x8x4(acc, -A[gi * kMmaPitch + h + tg], B[gi * kMmaPitch + h + tg]);
  if (valid) store_pair(out, acc);
}

// Panel p (columns 8 p ..) of the 32 x 32 block D: lane l has row l.  Returns
// the updated index of the first bad pivot (0: none).
__device__ __forceinline__ int warp_chol_panel(double* D, double* rd, int p, int bad) {
  const int lane = threadIdx.x & 31, c0 = 8 * p;
  double* row = D + lane * kMmaPitch + c0;
  double a[8];
#pragma unroll
  for (int c = 0; c < 8; c += 2) {
    double v[2];
    load_pair(v, row + c);
    a[c] = lane >= c0 ? v[0] : 0.0;
    a[c + 1] = lane >= c0 ? v[1] : 0.0;
  }
  double d = __shfl_sync(0xffffffffu, a[0], c0);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double r = rsqrt(d);
    if (bad == 0 && !(d > 0.0)) bad = c0 + k + 1;
    const double l = lane >= c0 + k ? a[k] * r : 0.0;
    a[k] = l;
    if (lane == c0 + k) rd[lane] = r;
    // The next pivot's lane needs only its own l.
    if (k < 7) d = __shfl_sync(0xffffffffu, fma(-l, l, a[(k + 1) & 7]), c0 + k + 1);
#pragma unroll
    for (int j = k + 1; j < 8; ++j) a[j] = fma(-l, __shfl_sync(0xffffffffu, l, c0 + j), a[j]);
  }
  if (lane >= c0) {  // zero above the diagonal
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      const double v[2] = {a[c], a[c + 1]};
      store_pair(row + c, v);
    }
  }
  return bad;
}

// Rows 8 p .. 8 p + 7 of X = inv(L) (pitch kSubPitch) of the 32 x 32 block L
// (pitch kMmaPitch), the calling warp: X_pp by substitution, X_pc = -X_pp t_c
// with t_c = sum_{c<=q<p} L_pq X_qc from warp_inv_sums.
__device__ __forceinline__ void warp_inv_rows(const double* L, const double* rd, double* X, int p,
                                              const double (&t)[3][2]) {
  const int lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3, c0 = 8 * p;
#pragma unroll
  for (int c = 0; c < 3; ++c)
    if (c < p) store_pair(X + (c0 + gi) * kSubPitch + 8 * c + 2 * tg, t[c]);
  double w[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) w[i] = i == (lane & 7) ? 1.0 : 0.0;
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    w[k] *= rd[c0 + k];
#pragma unroll
    for (int i = k + 1; i < 8; ++i) w[i] = fma(-L[(c0 + i) * kMmaPitch + c0 + k], w[k], w[i]);
  }
  if (lane < 8) {
#pragma unroll
    for (int i = 0; i < 8; ++i) X[(c0 + i) * kSubPitch + c0 + lane] = w[i];
  }
  __syncwarp();
  if (p == 0) return;
  double av[2], bv[3][2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    av[h] = -X[(c0 + gi) * kSubPitch + c0 + 4 * h + tg];
#pragma unroll
    for (int c = 0; c < 3; ++c) bv[c][h] = X[(c0 + 4 * h + tg) * kSubPitch + 8 * c + gi];
  }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    double x[2] = {0.0, 0.0};
#pragma unroll
    for (int h = 0; h < 2; ++h) dmma_8x8x4(x, av[h], bv[c][h]);
    if (c < p) store_pair(X + (c0 + gi) * kSubPitch + 8 * c + 2 * tg, x);
  }
  __syncwarp();
}
__device__ __forceinline__ void warp_inv_sums(const double* L, const double* X, int p,
                                              double (&t)[3][2]) {
  const int lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3;
#pragma unroll
  for (int c = 0; c < 3; ++c) t[c][0] = t[c][1] = 0.0;
#pragma unroll 1
  for (int q = 0; q < p; ++q)
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
      const double a = L[(8 * p + gi) * kMmaPitch + 8 * q + h + tg];
#pragma unroll
      for (int c = 0; c < 3; ++c)  // X is zero above its diagonal: q < c adds nothing
        dmma_8x8x4(t[c], a, X[(8 * q + h + tg) * kSubPitch + 8 * c + gi]);
    }
}
__device__ __forceinline__ void pair_barrier() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

// Cholesky of the 128 x 128 block in shared memory (lower, pitch kMmaPitch) by
// the CTA, and the inverses of its four 32 x 32 diagonal sub-blocks into inv
// (pitch kSubPitch, zero above the diagonal).  Per sub-block b:
//   * warp 0 factors it in panels of eight columns, lane l with row l's eight
//     values in registers: per column one chain of pivot shuffle, reciprocal
//     square root, scaling and the update of the next pivot, the other updates
//     beside it; then the next panel's update (FP64 tensor cores);
//   * warp 1 follows a panel behind (named barrier 1): the update of the columns
//     after the next panel, and the panel's rows of the inverse;
//   * warps 2 - 7 meanwhile apply the previous sub-block's products to the rest
//     of the block, all but the sub-block in work;
//   * then all warps multiply the rows below by the inverse's transpose and
//     update the next sub-block (FP64 tensor cores).
// rd: 32 doubles, sflag: one slot.  Returns 0 or the 1-based index of the first
// non-positive pivot.
// The chain over the columns bounds it: 42000 cycles in all with the code in the
// instruction cache.  Register tiles of 4 x 4 over the whole block with a barrier
// per four columns took 75000 cycles, and the inverses, a column per lane from
// shared memory, another 18000.  A block is factored once per step by another SM
// each time, so the code is short on purpose: with the 32 columns unrolled (43700
// cycles when cached) a step of the factorisation took 65 us, so it takes 50 us.
__device__ __noinline__ static int cta_chol128(double* sm, double* inv, double* rd, volatile int* sflag) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3;
  if (threadIdx.x == 0) *sflag = 0;
#pragma unroll 1
  for (int b = 0; b < 4; ++b) {
    const int o = 32 * b;
    double* D = sm + o * kMmaPitch + o;
    if (warp == 0) {
      int bad = 0;
#pragma unroll 1
      for (int p = 0; p < 4; ++p) {
        bad = warp_chol_panel(D, rd, p, bad);
        pair_barrier();
        if (p == 3) break;
        // Column tile p + 1.
        const double* P = D + 8 * p;
#pragma unroll
        for (int x = 1; x < 4; ++x) {
          const int i = min(p + x, 3), j = min(p + 1, 3);
          warp_tile8(D + 8 * i * kMmaPitch + 8 * j, P + 8 * i * kMmaPitch, P + 8 * j * kMmaPitch,
                     p + x < 4);
        }
        __syncwarp();
      }
      if (bad != 0 && lane == 0) *sflag = o + bad;
    } else if (warp == 1) {
      double* X = inv + b * 32 * kSubPitch;
      const double zero[2] = {0.0, 0.0};
      for (int e = lane; e < 32 * 16; e += 32) store_pair(X + (e >> 4) * kSubPitch + 2 * (e & 15), zero);
      __syncwarp();
      double sums[3][2];
#pragma unroll 1
      for (int p = 0; p < 4; ++p) {
        warp_inv_sums(D, X, p, sums);
        pair_barrier();
        // The column tiles after p + 1.
        const double* P = D + 8 * p;
        if (p < 2) {
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const int x = q == 0 ? 2 : 3, y = q == 2 ? 3 : 2;
            const int i = min(p + x, 3), j = min(p + y, 3);
            warp_tile8(D + 8 * i * kMmaPitch + 8 * j, P + 8 * i * kMmaPitch,
                       P + 8 * j * kMmaPitch, p + x < 4);
          }
        }
        warp_inv_rows(D, rd, X, p, sums);
      }
    } else if (b > 0) {
      // The products of sub-block column b - 1 for the lower 16 x 16 units of
      // rows and columns >= o, without the sub-block at o itself (units 0 - 2).
      const int units = (8 - 2 * b) * (9 - 2 * b) / 2;
      for (int u = 3 + warp - 2; u < units; u += 6) {
        int p = 0;
        while ((p + 1) * (p + 2) / 2 <= u) ++p;
        const int r0 = o + 16 * p, c0 = o + 16 * (u - p * (p + 1) / 2);
        const double* ra = sm + (r0 + gi) * kMmaPitch + o - 32 + tg;
        const double* rb = sm + (c0 + gi) * kMmaPitch + o - 32 + tg;
        double acc[2][2][2];
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              acc[x][y][e] = sm[(r0 + 8 * x + gi) * kMmaPitch + c0 + 8 * y + 2 * tg + e];
#pragma unroll
        for (int k = 0; k < 32; k += 4) {
          double av[2], bv[2];
#pragma unroll
          for (int x = 0; x < 2; ++x) {
            av[x] = -ra[x * 8 * kMmaPitch + k];
            bv[x] = rb[x * 8 * kMmaPitch + k];
          }
#pragma unroll
          for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) dmma_8x8x4(acc[x][y], av[x], bv[y]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
          for (int y = 0; y < 2; ++y)
            store_pair(sm + (r0 + 8 * x + gi) * kMmaPitch + c0 + 8 * y + 2 * tg, acc[x][y]);
      }
    }
    __syncthreads();
    const int bad = *sflag;
    if (bad != 0 || b == 3) return bad;
    // The rows below: L_ib = A_ib inv(L_bb)^T, eight rows at a time per warp
    // (in place: a warp reads its rows' fragments before it writes them).
    const double* X = inv + b * 32 * kSubPitch + gi * kSubPitch + tg;
    double xf[4][8];  // its fragments: zero right of the diagonal
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int k = 0; k < 2 * y + 2; ++k) xf[y][k] = X[8 * y * kSubPitch + 4 * k];
#pragma unroll 1
    for (int r = o + 32 + 8 * warp; r < kLB; r += 64) {
      double* row = sm + (r + gi) * kMmaPitch + o;
      double av[8], acc[4][2];
#pragma unroll
      for (int k = 0; k < 8; ++k) av[k] = row[4 * k + tg];
#pragma unroll
      for (int y = 0; y < 4; ++y) acc[y][0] = acc[y][1] = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int y = 0; y < 4; ++y)
          if (k < 2 * y + 2) dmma_8x8x4(acc[y], av[k], xf[y][k]);
      __syncwarp();
#pragma unroll
      for (int y = 0; y < 4; ++y) store_pair(row + 8 * y + 2 * tg, acc[y]);
    }
    __syncthreads();
    // The next sub-block's update: its ten lower 8 x 8 tiles.
    {
      double f[2][2][8], acc[2][2][2];
      double* out[2];
#pragma unroll
      for (int q = 0; q < 2; ++q) {  // tiles warp and, for two warps, warp + 8
        const int t = min(warp + 8 * q, 9);
        const int p = t < 1 ? 0 : t < 3 ? 1 : t < 6 ? 2 : 3;
        const int r0 = o + 32 + 8 * p, c0 = o + 32 + 8 * (t - p * (p + 1) / 2);
        out[q] = sm + (r0 + gi) * kMmaPitch + c0 + 2 * tg;
        load_pair(acc[q][0], out[q]);
        acc[q][1][0] = acc[q][1][1] = 0.0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          f[q][0][k] = -sm[(r0 + gi) * kMmaPitch + o + 4 * k + tg];
          f[q][1][k] = sm[(c0 + gi) * kMmaPitch + o + 4 * k + tg];
        }
        if (warp > 1) break;
      }
#pragma unroll
      for (int q = 0; q < 2; ++q) {
#pragma unroll
        for (int k = 0; k < 8; ++k) dmma_8x8x4(acc[q][k & 1], f[q][0][k], f[q][1][k]);
        acc[q][0][0] += acc[q][1][0];
        acc[q][0][1] += acc[q][1][1];
        store_pair(out[q], acc[q][0]);
        if (warp > 1) break;
      }
    }
    __syncthreads();
  }
  return 0;
}

// Eight rows of the panel at column k0 of g (leading dimension ld) from row r
// on, the calling warp: x L_kk^T = g_row for each row, 32 columns at a time
// (x_q = (g_q - sum_{p<q} x_p L_qp^T) inv(L_qq)^T) on the FP64 tensor cores.
// lkk: L_kk (pitch kMmaPitch), inv: the inverses of its diagonal sub-blocks.
template <typename T>
__device__ __forceinline__ void warp_panel_rows(T* g, size_t ld, int r, int k0, const double* lkk,
                                                const double* inv) {
  const int lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3;
  T* row = g + size_t(r + gi) * ld + k0 + 2 * tg;
  double v[4][4][2];  // the 8 x 128 values in accumulator layout
#pragma unroll
  for (int q = 0; q < 4; ++q)
#pragma unroll
    for (int y = 0; y < 4; ++y) load_pair(v[q][y], row + 32 * q + 8 * y);
  // Accumulator layout (row gi, columns 8 y + 2 tg + e) to the fragment of step
  // k (row gi, column 4 k + tg).
  auto fragment = [&](const double (&c)[4][2], int k) {
    const int src = 4 * gi + 2 * (k & 1) + (tg >> 1);
    const double e0 = __shfl_sync(0xffffffffu, c[k >> 1][0], src);
    const double e1 = __shfl_sync(0xffffffffu, c[k >> 1][1], src);
    return (tg & 1) ? e1 : e0;
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    double x[4][2];
#pragma unroll
    for (int y = 0; y < 4; ++y) x[y][0] = x[y][1] = 0.0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const double f = fragment(v[q], k);
#pragma unroll
      for (int y = 0; y < 4; ++y)
        if (4 * k < 8 * y + 8)
          dmma_8x8x4(x[y], f, inv[q * 32 * kSubPitch + (8 * y + gi) * kSubPitch + 4 * k + tg]);
    }
#pragma unroll
    for (int y = 0; y < 4; ++y) store_pair(row + 32 * q + 8 * y, x[y]);
    if (q < 3) {
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const double f = -fragment(x, k);
#pragma unroll
        for (int q2 = q + 1; q2 < 4; ++q2)
#pragma unroll
          for (int y = 0; y < 4; ++y)
            dmma_8x8x4(v[q2][y], f, lkk[(32 * q2 + 8 * y + gi) * kMmaPitch + 32 * q + 4 * k + tg]);
      }
    }
  }
}

// Inverses of the four 32 x 32 diagonal sub-blocks of the factored block sm
// (pitch kPitch) into inv[q] (pitch kSubPitch, zero above the diagonal), a warp
// each, lane c with column c in registers; then a barrier.
__device__ __noinline__ static void cta_sub_inverses(const double* sm, double* inv) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp < 4) {
    const double* L = sm + 32 * warp * (kPitch + 1);
    const double rl = 1.0 / L[lane * kPitch + lane];
    double w[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) w[i] = i == lane ? 1.0 : 0.0;
#pragma unroll
    for (int k = 0; k < 32; ++k) {
      const double x = w[k] * __shfl_sync(0xffffffffu, rl, k);
      w[k] = x;
#pragma unroll
      for (int i = k + 1; i < 32; ++i) w[i] = fma(-L[i * kPitch + k], x, w[i]);
    }
    double* X = inv + warp * 32 * kSubPitch + lane;
#pragma unroll
    for (int i = 0; i < 32; ++i) X[i * kSubPitch] = w[i];
  }
  __syncthreads();
}

// C = s A B for 32-row, 32-column blocks in shared memory (leading dimensions
// pa, pb, pc; inner length K, a multiple of 4) on the FP64 tensor cores, the
// CTA's eight warps two 8 x 8 tiles each, then a barrier.
__device__ __forceinline__ void cta_gemm32(double* C, int pc, const double* A, int pa,
                                           const double* B, int pb, int K, double scale) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gi = lane >> 2, tg = lane & 3;
  const int r0 = (warp >> 1) * 8, c0 = (warp & 1) * 16;
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    const double a = A[(r0 + gi) * pa + k + tg];
    const double b0 = B[(k + tg) * pb + c0 + gi], b1 = B[(k + tg) * pb + c0 + 8 + gi];
    dmma_8x8x4(acc[0], a, b0);
    dmma_8x8x4(acc[1], a, b1);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int e = 0; e < 2; ++e) C[(r0 + gi) * pc + c0 + 8 * h + 2 * tg + e] = scale * acc[h][e];
  __syncthreads();
}

// In place, the inverse of the factored 128 x 128 block sm (lower, pitch
// kPitch) from the inverses of its 32 x 32 diagonal blocks: block column by
// block column, X_ij = -X_ii sum_{j<=k<i} L_ik X_kj (block column j of L is
// not needed by the later ones).  tmp: 32 x kSubPitch.
__device__ __noinline__ static void cta_inverse128(double* sm, const double* inv, double* tmp) {
  for (int j = 0; j < 4; ++j) {
    for (int i = j + 1; i < 4; ++i) {
      // X_jj for k = j, then the rows j + 1 .. i - 1 of this block column.
      cta_gemm32(tmp, kSubPitch, sm + 32 * i * kPitch + 32 * j, kPitch,
                    inv + j * 32 * kSubPitch, kSubPitch, 32, 1.0);
      if (i > j + 1) {
        // The rest of the sum into the block's own place, then both added.
        cta_gemm32(sm + 32 * i * kPitch + 32 * j, kPitch,
                      sm + 32 * i * kPitch + 32 * (j + 1), kPitch,
                      sm + 32 * (j + 1) * kPitch + 32 * j, kPitch, 32 * (i - j - 1), 1.0);
        for (int e = threadIdx.x; e < 1024; e += kGridBT)
          tmp[(e >> 5) * kSubPitch + (e & 31)] +=
              sm[(32 * i + (e >> 5)) * kPitch + 32 * j + (e & 31)];
        __syncthreads();
      }
      cta_gemm32(sm + 32 * i * kPitch + 32 * j, kPitch, inv + i * 32 * kSubPitch, kSubPitch,
                    tmp, kSubPitch, 32, -1.0);
    }
    // X_jj: rows of L_jj are not needed any more (the columns to its right
    // do not touch block column j).
    for (int e = threadIdx.x; e < 1024; e += kGridBT)
      sm[(32 * j + (e >> 5)) * kPitch + 32 * j + (e & 31)] =
          inv[j * 32 * kSubPitch + (e >> 5) * kSubPitch + (e & 31)];
    __syncthreads();
  }
}

// Trailing update g_ij -= L_ik L_jk^T of the lower 128 x 128 tiles t0, t0 +
// step, ... < tiles of the block at (base, base), with the panel at column k0.
// FP64: on the FP64 tensor cores, warp w on the 64 x 32 block (w / 4, w % 4) of
// the tile; slices of 32 panel columns staged row by row (pitch kSubPitch, 16-byte
// copies), two buffers and one barrier per slice; the next tile's first slice
// is in flight during this one's last.  The upper parts of the diagonal tiles
// are written too; nothing reads them.
// n = 4096: the trailing steps with their lookahead take 24.8 ms in 13
// factorisations, 31.2 with transposed 8-byte copies, slices of 16 columns and
// two barriers each.
__device__ __noinline__ static void trailing_tiles(double* sm, double* g, int npad, int base,
                                                   int k0, int t0, int tiles, int step) {
  constexpr int KS = 32, SL = 2 * kLB * kSubPitch;
  static_assert(2 * SL * sizeof(double) <= kArenaBytes, "trailing buffers exceed the arena");
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gi = lane >> 2, tg = lane & 3;
  const int wr = warp >> 2, wc = warp & 3;
  if (t0 >= tiles) return;
  auto issue = [&](int t, int s, int buf) {
    int ti, tj;
    lower_tile(t, ti, tj);
    double* pa = sm + buf * SL;
    double* pb = pa + kLB * kSubPitch;
    const double* ga = g + size_t(base + ti * kLB) * npad + k0 + s * KS;
    const double* gb = g + size_t(base + tj * kLB) * npad + k0 + s * KS;
#pragma unroll
    for (int q = 0; q < kLB * KS / 2 / kGridBT; ++q) {
      const int e = threadIdx.x + q * kGridBT, r = e >> 4, c = 2 * (e & 15);
      cp_async16(pa + r * kSubPitch + c, ga + size_t(r) * npad + c);
      cp_async16(pb + r * kSubPitch + c, gb + size_t(r) * npad + c);
    }
    cp_async_commit();
  };
  issue(t0, 0, 0);
  int buf = 0;
  for (int t = t0; t < tiles; t += step) {
    double acc[8][4][2];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll 1
    for (int s = 0; s < kLB / KS; ++s) {
      cp_async_wait<0>();
      __syncthreads();
      if (s + 1 < kLB / KS) {
        issue(t, s + 1, buf ^ 1);
      } else if (t + step < tiles) {
        issue(t + step, 0, buf ^ 1);
      }
      const double* pa = sm + buf * SL + (wr * 64 + gi) * kSubPitch + tg;
      const double* pb = sm + buf * SL + (kLB + wc * 32 + gi) * kSubPitch + tg;
#pragma unroll
      for (int k = 0; k < KS; k += 4) {
        double a[8], b[4];
#pragma unroll
        for (int mi = 0; mi < 8; ++mi) a[mi] = pa[mi * 8 * kSubPitch + k];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) b[ni] = pb[ni * 8 * kSubPitch + k];
#pragma unroll
        for (int mi = 0; mi < 8; ++mi)
#pragma unroll
          for (int ni = 0; ni < 4; ++ni) dmma_8x8x4(acc[mi][ni], a[mi], b[ni]);
      }
      buf ^= 1;
    }
    int ti, tj;
    lower_tile(t, ti, tj);
    double* out = g + size_t(base + ti * kLB + wr * 64 + gi) * npad + base + tj * kLB + wc * 32 +
                  2 * tg;
#pragma unroll
    for (int m0 = 0; m0 < 8; m0 += 2) {
      double v[2][4][2];
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
          load_pair(v[mi][ni], out + size_t(8 * (m0 + mi)) * npad + 8 * ni);
#pragma unroll
      for (int mi = 0; mi < 2; ++mi)
#pragma unroll
        for (int ni = 0; ni < 4; ++ni) {
          v[mi][ni][0] -= acc[m0 + mi][ni][0];
          v[mi][ni][1] -= acc[m0 + mi][ni][1];
          store_pair(out + size_t(8 * (m0 + mi)) * npad + 8 * ni, v[mi][ni]);
        }
    }
  }
}

// FP32: 8 x 8 outputs per thread, slices of 16 panel columns, transposed.
__device__ __noinline__ static void trailing_tiles(float* sm, float* g, int npad, int base, int k0,
                                                   int t0, int tiles, int step) {
  constexpr int KS = 16;
  constexpr int SP = kLB + 1;      // slice pitch
  constexpr int SL = 2 * KS * SP;  // elements per buffer
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  auto issue = [&](int kk0, int i0, int j0, int buf) {
    float* pa = sm + buf * SL;
    float* pb = pa + KS * SP;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = threadIdx.x + q * kGridBT, r = e >> 4, kk = e & 15;
      cp_async4(pa + kk * SP + r, g + size_t(i0 + r) * npad + k0 + kk0 + kk);
      cp_async4(pb + kk * SP + r, g + size_t(j0 + r) * npad + k0 + kk0 + kk);
    }
    cp_async_commit();
  };
  for (int t = t0; t < tiles; t += step) {
    int ti, tj;
    lower_tile(t, ti, tj);
    const int i0 = base + ti * kLB, j0 = base + tj * kLB;
    float acc[8][8];
#pragma unroll
    for (int a = 0; a < 8; ++a)
#pragma unroll
      for (int b = 0; b < 8; ++b) acc[a][b] = 0.0f;
    issue(0, i0, j0, 0);
    int buf = 0;
    for (int kk0 = 0; kk0 < kLB; kk0 += KS) {
      if (kk0 + KS < kLB) {
        issue(kk0 + KS, i0, j0, buf ^ 1);
        cp_async_wait<1>();
      } else {
        cp_async_wait<0>();
      }
      __syncthreads();
      const float* pa = sm + buf * SL;
      const float* pb = pa + KS * SP;
#pragma unroll 2
      for (int kk = 0; kk < KS; ++kk) {
        float av[8], bv[8];
#pragma unroll
        for (int a = 0; a < 8; ++a) {
          av[a] = pa[kk * SP + ty + 16 * a];
          bv[a] = pb[kk * SP + tx + 16 * a];
        }
#pragma unroll
        for (int a = 0; a < 8; ++a)
#pragma unroll
          for (int b = 0; b < 8; ++b) acc[a][b] = fma(av[a], bv[b], acc[a][b]);
      }
      __syncthreads();
      buf ^= 1;
    }
#pragma unroll
    for (int a = 0; a < 8; ++a) {
      const int i = i0 + ty + 16 * a;
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const int j = j0 + tx + 16 * b;
        if (j <= i) g[size_t(i) * npad + j] -= acc[a][b];
      }
    }
  }
}

template <typename T, class S>
__device__ int large_cholesky(S& s, T* g) {
  const int npad = s.npad, nblk = npad / kLB;
  int* info = s.linfo;
  T* sm = reinterpret_cast<T*>(s.arena);      // the trailing update's slices
  // The diagonal block and the panel rows are computed in FP64 whatever T is.
  double* blk = reinterpret_cast<double*>(s.arena);  // 128 x 128 block
  double* sinv = blk + kLB * kMmaPitch;              // 4 sub-block inverses
  double* rdiag = sinv + 4 * 32 * kSubPitch;
  double* tmp32 = rdiag + 32;                        // 32 x kSubPitch
  volatile int* sflag = reinterpret_cast<volatile int*>(tmp32 + 32 * kSubPitch);
  static_assert((size_t(kLB) * kMmaPitch + 5 * 32 * kSubPitch + 32) * sizeof(double) + 16 <=
                    kArenaBytes, "the factorisation's shared memory");
  double* ginv = s.sinv;  // the same inverses in global memory
  const int warp = threadIdx.x >> 5;
  if (s.tid == 0) *info = 0;
  s.sync();
  QTQP_TIC();
  // (a) Factor the diagonal block at column k0, in blk (the calling CTA), then
  // to g, and the four 32 x 32 sub-block inverses to global memory for the
  // panel step.
  auto factor_diag = [&](int k0) {
    const int bad = cta_chol128(blk, sinv, rdiag, sflag);
    if (bad) {
      if (threadIdx.x == 0) atomicCAS(info, 0, k0 + bad);
    } else {
      for (int e = threadIdx.x; e < 4 * 32 * kSubPitch; e += kGridBT) ginv[e] = sinv[e];
      for (int e = threadIdx.x; e < kLB * kLB; e += kGridBT) {
        const int r = e >> 7, c = e & 127;
        if (c <= r) g[size_t(k0 + r) * npad + k0 + c] = T(blk[r * kMmaPitch + c]);
      }
    }
    __syncthreads();
  };
  for (int k = 0; k < nblk; ++k) {
    const int k0 = k * kLB;
    QTQP_RETIC();
    // (a) diagonal block: only for the first one; every later one is
    // factored during the previous step's trailing update (lookahead).
    if (k == 0 && blockIdx.x == 0) {
      stage_mma(blk, g, npad, 0, 0);
      factor_diag(0);
    }
    if (k == 0) s.sync();
    QTQP_TOC(kPhLgDiag);
    QTQP_RETIC();
    if (*reinterpret_cast<volatile int*>(info) != 0) break;
    const int rest = npad - k0 - kLB;
    if (rest == 0) break;
    // (b) panel rows, eight per warp, spread over the CTAs before the warps.
    if (int(blockIdx.x) * 8 < rest) {
      stage_mma(blk, g, npad, k0, k0);
      for (int e = threadIdx.x; e < 4 * 32 * kSubPitch; e += kGridBT) sinv[e] = ginv[e];
      __syncthreads();
      for (int t = blockIdx.x + warp * gridDim.x; 8 * t < rest; t += gridDim.x * (kGridBT / 32))
        warp_panel_rows<T>(g, npad, k0 + kLB + 8 * t, k0, blk, sinv);
    }
    s.sync();
    QTQP_TOC(kPhLgPanel);
    QTQP_RETIC();
    // (c) trailing update.  Lookahead: the CTA that owns the next diagonal block
    // (tile 0) updates it and factors it at once; the other tiles go round robin
    // over the others.
    {
      const int nt = rest / kLB, tiles = nt * (nt + 1) / 2, base = k0 + kLB;
      const int G = int(gridDim.x), owner = (k + 1) % G, me = int(blockIdx.x);
      if (me == owner) {
        cta_diag_update<T>(blk, g, npad, base, k0);
        factor_diag(base);
      } else {
        trailing_tiles(sm, g, npad, base, k0, 1 + (me - owner - 1 + G) % G, tiles, G - 1);
      }
    }
    s.sync();
    QTQP_TOC(kPhLgTrail);
  }
  const int rc = *reinterpret_cast<volatile int*>(info);
  if (rc != 0) return rc;
  QTQP_RETIC();
  // Each CTA inverts the diagonal block it owns in the solves and keeps it
  // resident in shared memory until the next factorisation.
  if (int(blockIdx.x) < nblk) {
    const int b0 = int(blockIdx.x) * kLB;
    // L (pitch kPitch) and its four diagonal sub-blocks' inverses.
    for (int e = threadIdx.x; e < kLB * kLB; e += kGridBT) {
      const int r = e >> 7, c = e & 127;
      blk[r * kPitch + c] = c <= r ? double(g[size_t(b0 + r) * npad + b0 + c]) : 0.0;
    }
    __syncthreads();
    cta_sub_inverses(blk, sinv);
    cta_inverse128(blk, sinv, tmp32);
    if constexpr (sizeof(T) == 4) {  // to T in place, 16 rows at a time
      for (int r0 = 0; r0 < kLB; r0 += 16) {
        T v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int e = threadIdx.x + q * kGridBT;
          v[q] = T(blk[(r0 + (e >> 7)) * kPitch + (e & 127)]);
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int e = threadIdx.x + q * kGridBT;
          sm[(r0 + (e >> 7)) * kPitch + (e & 127)] = v[q];
        }
        __syncthreads();
      }
    }
  }
  QTQP_TOC(kPhLgInv);
  return 0;
}

template <typename T, class S>
__device__ int large_factorize(S& s) {
  QTQP_TIC();
  int info;
  if constexpr (sizeof(T) == 4) {
    large_scale_split(s);
    s.sync();
    large_gram_tc(s);
    s.sync();
    large_finish_gram<float>(s, s.g32l);
    QTQP_TOC(kPhGram);
    QTQP_RETIC();
    info = large_cholesky<float>(s, s.g32l);
  } else {
    if (s.lda % 2 == 0) {
      large_gram_dmma<2>(s);
    } else {
      large_gram_dmma<1>(s);
    }
    s.sync();
    large_finish_gram<double>(s, s.g64);
    QTQP_TOC(kPhGram);
    QTQP_RETIC();
    info = large_cholesky<double>(s, s.g64);
  }
  QTQP_TOC(kPhChol);
  return info;
}

// ---------------------------------------------------------------------------
// L L^T v = v in place (v, w: n entries of T; w is scratch), block by block
// with slots instead of grid barriers.  CTA j (j < nb) owns block row j and
// keeps inv(L_jj) resident in shared memory since the factorisation.
//   Forward:  z_j = inv(L_jj) (v_j - sum_{c<j} L_jc z_c), into w and the
//             block's slots.  CTA j adds L_jc z_c as soon as the slots hold
//             z_c, in the order c = 0, 1, ..., so only the last product
//             L_{j,j-1} z_{j-1} and the diagonal step lie on the chain from one
//             block to the next; L_{j,j-1} waits in registers.
//   Backward: x_j = inv(L_jj)^T (z_j - sum_{c>j} L_cj^T x_c) into v and the
//             slots, the same way from c = nb-1 down, with L_{j+1,j} in registers.
// Every sum runs in a fixed order (c ascending or descending, then the
// lanes' and warps' partials in a fixed tree), so results do not depend on
// timing.  Tags: 2t - 1 (forward) and 2t (backward) for the t-th solve; a block
// overwrites its z with its x only after every later block has published its
// own x, and so has read that z.  One grid barrier at the end.
// The chain of 2 nb steps bounds it: 3.0 us per step at n = 4096 and 2.4 us at
// n = 1000 in FP32; 6.0 and 5.0 us when a block published by fences and a flag
// that one warp polled for the CTA, and the chain's block came from L2 (128 KB).
// ---------------------------------------------------------------------------
template <typename T, class S>
__device__ __noinline__ void large_chol_solve(S& s, T* v, T* w) {
  const int n = s.n, npad = s.npad;
  const int nb = (n + kLB - 1) / kLB;
  const T* g = sizeof(T) == 4 ? reinterpret_cast<const T*>(s.g32l)
                              : reinterpret_cast<const T*>(s.g64);
  constexpr int WPB = kGridBT / 32;
  static_assert(WPB * 16 == kLB, "one warp per 16 rows of a block");
  // Shared memory: inv(L_bb) (pitch kPitch), then the block's right-hand side
  // (kLB) and the warps' column partials of the backward step (WPB x kLB).
  const T* rinv = reinterpret_cast<const T*>(s.arena);
  T* red = reinterpret_cast<T*>(s.arena) + kLB * kPitch;
  T* cpart = red + kLB;
  static_assert((size_t(kLB) * kPitch + kLB) * sizeof(double) <= kPrSmemOff,
                "large_products would overwrite the resident inverse");
  static_assert((size_t(kLB) * kPitch + kLB + WPB * kLB) * sizeof(double) <= kArenaBytes,
                "the solve's shared memory exceeds the arena");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int j = blockIdx.x;
  s.tri_gen += 1;
  const unsigned long long tag_fwd = 2ull * s.tri_gen - 1, tag_bwd = 2ull * s.tri_gen;
  GridCtl* gc = s.gctl;
  GridSlot* slots = s.tri_slot;
  QTQP_TIC();
  if (j < nb) {
    const int b0 = j * kLB, bs = min(kLB, n - b0);
    const int r0 = 16 * warp;  // this warp's 16 rows of the block
    const T* lrow = g + size_t(b0 + r0) * npad + lane;
    // Rows beyond n are padding inside g (npad rows): read, never used.
    // (The first block reads its own: a conditional load puts the array into
    // local memory.)
    T near[16][4];
#pragma unroll
    for (int r = 0; r < 16; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        near[r][q] = lrow[size_t(r) * npad + max(j - 1, 0) * kLB + 32 * q];
    // Forward: lane partials of rows r0 + r over columns lane + 32 q.
    T acc[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) acc[r] = T(0);
    double z[4];
    for (int c = 0; c < j - 1; ++c) {
      const T* lr = lrow + c * kLB;
      T far[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) far[r][q] = lr[size_t(r) * npad + 32 * q];
      slots_wait<4>(gc, slots + c * kLB + lane, 32, tag_fwd, z);
#pragma unroll
      for (int r = 0; r < 16; ++r) {
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[r] = fma(far[r & 3][q], T(z[q]), acc[r]);
        if (r < 12) {
#pragma unroll
          for (int q = 0; q < 4; ++q) far[r & 3][q] = lr[size_t(r + 4) * npad + 32 * q];
        }
      }
    }
    if (j > 0) {
      slots_wait<4>(gc, slots + (j - 1) * kLB + lane, 32, tag_fwd, z);
#pragma unroll
      for (int r = 0; r < 16; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[r] = fma(near[r][q], T(z[q]), acc[r]);
    }
    // Sum the 16 rows over the warp: each exchange step sends half of the
    // values to the partner lane and keeps the other half, so lane l ends with
    // row rsel(l) (lanes l and l ^ 1 hold the same row).
#pragma unroll
    for (int half = 8, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
      const bool up = (lane & bit) != 0;
#pragma unroll
      for (int q = 0; q < half; ++q) {
        const T send = up ? acc[q] : acc[q + half];
        const T keep = up ? acc[q + half] : acc[q];
        acc[q] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
      }
    }
    acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
    const int rsel = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 +
                     ((lane >> 1) & 1);
    if ((lane & 1) == 0 && r0 + rsel < bs) red[r0 + rsel] = v[b0 + r0 + rsel] - acc[0];
    __syncthreads();
    {
      // z_r = sum_{c <= r} inv(L_jj)_rc u_c by two threads per row: the
      // half-warp h of warp w takes rows 16 w .. 16 w + 15 and the columns
      // c = h (mod 2) (distinct banks across the half-warp, u_c broadcast).
      const int r = r0 + (lane & 15), h = lane >> 4;
      const T* ir = rinv + r * kPitch;
      T a0 = T(0), a1 = T(0), a2 = T(0), a3 = T(0);
      if (r < bs) {
        int c = h;
        for (; c + 6 <= r; c += 8) {
          a0 = fma(ir[c + 0], red[c + 0], a0);
          a1 = fma(ir[c + 2], red[c + 2], a1);
          a2 = fma(ir[c + 4], red[c + 4], a2);
          a3 = fma(ir[c + 6], red[c + 6], a3);
        }
        for (; c <= r; c += 2) a0 = fma(ir[c], red[c], a0);
      }
      T zr = (a0 + a1) + (a2 + a3);
      zr += __shfl_xor_sync(0xffffffffu, zr, 16);
      if (h == 0) {
        if (r >= bs) zr = T(0);
        slot_store(slots + b0 + r, double(zr), tag_fwd);
        if (r < bs) w[b0 + r] = zr;
      }
    }
  }
  QTQP_TOC(kPhLgFwd);
  QTQP_RETIC();
  if (j < nb) {
    const int b0 = j * kLB, bs = min(kLB, n - b0);
    const int r0 = 16 * warp;
    const T* lcol = g + size_t(r0) * npad + b0 + lane;
    T near[16][4];
#pragma unroll
    for (int r = 0; r < 16; ++r)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        near[r][q] = lcol[size_t(min(j + 1, nb - 1) * kLB + r) * npad + 32 * q];
    // Backward: lane partials of columns lane + 32 q of block j over this
    // warp's 16 rows of every later block (lane l holds x of row l % 16).
    // The last block's rows beyond n have x = 0 in their slots.
    T acc[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = T(0);
    double x[1];
    for (int c = nb - 1; c > j + 1; --c) {
      const T* lc = lcol + size_t(c) * kLB * npad;
      T far[4][4];
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) far[r][q] = lc[size_t(r) * npad + 32 * q];
      slots_wait<1>(gc, slots + c * kLB + r0 + (lane & 15), 0, tag_bwd, x);
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const T xi = __shfl_sync(0xffffffffu, T(x[0]), r);
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = fma(far[r & 3][q], xi, acc[q]);
        if (r < 12) {
#pragma unroll
          for (int q = 0; q < 4; ++q) far[r & 3][q] = lc[size_t(r + 4) * npad + 32 * q];
        }
      }
    }
    if (j + 1 < nb) {
      slots_wait<1>(gc, slots + (j + 1) * kLB + r0 + (lane & 15), 0, tag_bwd, x);
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const T xi = __shfl_sync(0xffffffffu, T(x[0]), r);
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = fma(near[r][q], xi, acc[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) cpart[warp * kLB + lane + 32 * q] = acc[q];
    __syncthreads();
    if (int(threadIdx.x) < bs) {
      const int k = threadIdx.x;
      T t = T(0);
#pragma unroll
      for (int q = 0; q < WPB; ++q) t += cpart[q * kLB + k];
      red[k] = w[b0 + k] - t;  // w_j: this CTA's forward result
    }
    __syncthreads();
    {
      // x_r = sum_{c >= r} inv(L_jj)_cr u_c, two threads per row as forward
      // (half-warp h: the columns c >= r with c = r + h (mod 2)).
      const int r = r0 + (lane & 15), h = lane >> 4;
      T a0 = T(0), a1 = T(0), a2 = T(0), a3 = T(0);
      if (r < bs) {
        int c = r + h;
        for (; c + 6 < bs; c += 8) {
          a0 = fma(rinv[(c + 0) * kPitch + r], red[c + 0], a0);
          a1 = fma(rinv[(c + 2) * kPitch + r], red[c + 2], a1);
          a2 = fma(rinv[(c + 4) * kPitch + r], red[c + 4], a2);
          a3 = fma(rinv[(c + 6) * kPitch + r], red[c + 6], a3);
        }
        for (; c < bs; c += 2) a0 = fma(rinv[c * kPitch + r], red[c], a0);
      }
      T xr = (a0 + a1) + (a2 + a3);
      xr += __shfl_xor_sync(0xffffffffu, xr, 16);
      if (h == 0) {
        if (r >= bs) xr = T(0);
        slot_store(slots + b0 + r, double(xr), tag_bwd);
        if (r < bs) v[b0 + r] = xr;
      }
    }
  }
  s.sync();
  // The KKT backend (no options) has no result record to report a wait that
  // gave up: its solution becomes NaN.
  if (s.o == nullptr && __syncthreads_or(*reinterpret_cast<volatile int*>(&gc->err) != 0)) {
    for (int k = threadIdx.x; k < n; k += blockDim.x) v[k] = T(NAN);
    __syncthreads();
  }
  QTQP_TOC(kPhLgBwd);
}

}  // namespace qtqp
