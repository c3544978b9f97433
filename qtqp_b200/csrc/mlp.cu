// Kernels of the warm-start MLP (no reference counterpart): a tiled FP32 GEMM
// with fused bias and ReLU, the ReLU backward mask, column sums (bias
// gradients), the MSE gradient with its loss, the hinge term on the sign of
// the inequality outputs, Adam, and the decoder that
// turns network outputs into per-instance warm starts for the banded solver.
#include <cooperative_groups.h>

#include <algorithm>
#include <cmath>

#include "common.cuh"

namespace qtqp {

constexpr int kTile = 64;          // C tile is kTile x kTile
constexpr int kTk = 16;            // K slice staged in shared memory
constexpr int kGemmThreads = 256;  // 16 x 16 threads, 4 x 4 outputs each
constexpr int kGemmPitch = kTile + 4;  // float4-aligned rows, 2-way store conflicts at most
constexpr int kGemmMaxSplit = 16;  // CTAs of one cluster sharing a tile's K

// C = alpha op(A) op(B) + beta C (+ bias[col]) (ReLU), and what a training
// step does to C or op(B) while they are at hand:
//   mask:   C_ij = 0 where !(mask_ij > 0) (the ReLU backward), laid out like C;
//   colsum: the column sums of op(B) (the bias gradient when B is dY);
//   dy:     dy_ij = dscale (C_ij - target_ij), *loss += sum (C - target)^2.
struct GemmArgs {
  int M, N, K;
  float alpha;
  const float* a;
  int lda;
  const float* b;
  int ldb;
  float beta;
  float* c;
  int ldc;
  const float* bias;
  int relu;
  const float* mask;
  float* colsum;
  const float* target;
  float* dy;
  float dscale;
  double* loss;
};

// op(A)(r, k) is A[r * lda + k], or A[k * lda + r] when TA; op(B)(k, c) is
// B[k * ldb + c], or B[c * ldb + k] when TB.  Both operand slices are staged
// k-major in two shared-memory buffers; the next slice's loads are in flight
// (registers) while the current one is multiplied, one barrier per slice.
//
// The gridDim.z CTAs of a cluster share one tile: each takes a contiguous
// part of the K slices, and the partial tiles are summed over distributed
// shared memory in part order (no workspace, no atomics, the same sum on
// every run).  Without the split a weight-sized product with a long K (dH =
// dY W^T of a 256-wide layer under 11000 outputs: 16 tiles, 688 slices) ran on
// 16 of 148 SMs and took about half of the step.
template <bool TA, bool TB>
__global__ void __launch_bounds__(kGemmThreads) gemm_kernel(const GemmArgs g) {
  namespace cg = cooperative_groups;
  __shared__ __align__(16) float sm[2 * 2 * kTk * kGemmPitch];
  static_assert(2 * 2 * kTk * kGemmPitch >= kTile * kTile + kTile, "partial tile + column sums");
  __shared__ double lpart[kGemmThreads / 32];
  const int tid = threadIdx.x;
  const int tx = tid & 15, ty = tid >> 4;
  const int row0 = blockIdx.y * kTile, col0 = blockIdx.x * kTile;
  const int parts = gridDim.z, part = blockIdx.z;
  const int ns = (g.K + kTk - 1) / kTk;
  const int q0 = int(int64_t(ns) * part / parts), q1 = int(int64_t(ns) * (part + 1) / parts);
  const bool sums = g.colsum != nullptr && blockIdx.y == 0;
  float* const as = sm;
  float* const bs = sm + 2 * kTk * kGemmPitch;
  // Element t of this thread in a slice: (row ar + t dr, k ka + t dk) of
  // op(A), (column bc + t dc, k kb + t dk2) of op(B); the fast index is the
  // contiguous one, so a warp reads whole 64- or 128-byte pieces.
  constexpr int E = kTile * kTk / kGemmThreads;
  constexpr int adr = TA ? 0 : kGemmThreads / kTk, adk = TA ? kGemmThreads / kTile : 0;
  constexpr int bdc = TB ? kGemmThreads / kTk : 0, bdk = TB ? 0 : kGemmThreads / kTile;
  const int ar = TA ? (tid & 63) : (tid >> 4), ka = TA ? (tid >> 6) : (tid & 15);
  const int bc = TB ? (tid >> 4) : (tid & 63), kb = TB ? (tid & 15) : (tid >> 6);
  const float* pa = g.a + (TA ? size_t(q0 * kTk + ka) * g.lda + row0 + ar
                              : size_t(row0 + ar) * g.lda + q0 * kTk + ka);
  const float* pb = g.b + (TB ? size_t(col0 + bc) * g.ldb + q0 * kTk + kb
                              : size_t(q0 * kTk + kb) * g.ldb + col0 + bc);
  const size_t astep = TA ? size_t(adk) * g.lda : size_t(adr) * g.lda;
  const size_t bstep = TB ? size_t(bdc) * g.ldb : size_t(bdk) * g.ldb;
  float ra[E], rb[E];
  auto fetch = [&](int q) {
    const int k0 = q * kTk;
#pragma unroll
    for (int t = 0; t < E; ++t) {
      const bool va = row0 + ar + t * adr < g.M && k0 + ka + t * adk < g.K;
      ra[t] = va ? pa[t * astep] : 0.0f;
      const bool vb = col0 + bc + t * bdc < g.N && k0 + kb + t * bdk < g.K;
      rb[t] = vb ? pb[t * bstep] : 0.0f;
    }
    pa += TA ? size_t(kTk) * g.lda : size_t(kTk);
    pb += TB ? size_t(kTk) : size_t(kTk) * g.ldb;
  };
  auto put = [&](int buf) {
    float* a0 = as + (buf * kTk + ka) * kGemmPitch + ar;
    float* b0 = bs + (buf * kTk + kb) * kGemmPitch + bc;
#pragma unroll
    for (int t = 0; t < E; ++t) {
      a0[t * (adk * kGemmPitch + adr)] = ra[t];
      b0[t * (bdk * kGemmPitch + bdc)] = rb[t];
    }
  };
  float acc[4][4];
  float csum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
  if (q0 < q1) {
    fetch(q0);
    put(0);
  }
  __syncthreads();
  for (int q = q0; q < q1; ++q) {
    const int buf = (q - q0) & 1;
    if (q + 1 < q1) fetch(q + 1);
    const float* sa = as + buf * kTk * kGemmPitch + ty * 4;
    const float* sb = bs + buf * kTk * kGemmPitch + tx * 4;
#pragma unroll
    for (int kk = 0; kk < kTk; ++kk) {
      const float4 a0 = *reinterpret_cast<const float4*>(sa + kk * kGemmPitch);
      const float4 bv = *reinterpret_cast<const float4*>(sb + kk * kGemmPitch);
      const float av[4] = {a0.x, a0.y, a0.z, a0.w};
      const float br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], br[j], acc[i][j]);
      if (sums) {
#pragma unroll
        for (int j = 0; j < 4; ++j) csum[j] += br[j];
      }
    }
    // The other buffer's readers passed the barrier that ended slice q - 1.
    if (q + 1 < q1) put(buf ^ 1);
    __syncthreads();
  }
  // The partial tile (and column sums) into shared memory, summed over the
  // cluster, then the epilogue row by row (coalesced stores).
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(&sm[(ty * 4 + i) * kTile + tx * 4]) =
        make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  if (sums && ty == 0) {
#pragma unroll
    for (int j = 0; j < 4; ++j) sm[kTile * kTile + tx * 4 + j] = csum[j];
  }
  if (parts > 1) {
    cg::this_cluster().sync();
  } else {
    __syncthreads();
  }
  auto total = [&](int idx) {
    if (parts == 1) return sm[idx];
    float v = 0.0f;
    for (int p = 0; p < parts; ++p) v += cg::this_cluster().map_shared_rank(sm, p)[idx];
    return v;
  };
  const int rows = kTile / parts;  // parts is a power of two, at most 16
  double lacc = 0.0;
  for (int e = tid; e < rows * kTile; e += kGemmThreads) {
    const int rl = part * rows + (e >> 6), cl = e & 63;
    const int r = row0 + rl, cc = col0 + cl;
    if (r >= g.M || cc >= g.N) continue;
    const size_t o = size_t(r) * g.ldc + cc;
    float v = g.alpha * total(rl * kTile + cl);
    if (g.beta != 0.0f) v = fmaf(g.beta, g.c[o], v);
    if (g.bias != nullptr) v += g.bias[cc];
    if (g.relu) v = fmaxf(v, 0.0f);
    if (g.mask != nullptr && !(g.mask[o] > 0.0f)) v = 0.0f;
    g.c[o] = v;
    if (g.dy != nullptr) {
      const float d = v - g.target[o];
      g.dy[o] = g.dscale * d;
      lacc += double(d) * double(d);
    }
  }
  if (sums && part == 0 && tid < kTile && col0 + tid < g.N)
    g.colsum[col0 + tid] = total(kTile * kTile + tid);
  if (g.dy != nullptr) {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) lacc += __shfl_xor_sync(0xffffffffu, lacc, off);
    if ((tid & 31) == 0) lpart[tid >> 5] = lacc;
    __syncthreads();
    if (tid == 0) {
      for (int w = 1; w < kGemmThreads / 32; ++w) lacc += lpart[w];
      atomicAdd(g.loss, lacc);
    }
  }
  if (parts > 1) cg::this_cluster().sync();  // peers may still read this CTA's partial
}

// The CTAs that share a tile's K: enough to give every SM about two, each
// with at least four slices.  The training step of a 32-256-256-11000 network
// at batch 256 (forward_loss + backward, 8 launches) takes 275 us against
// 1539 us with one CTA per tile and separate passes for the error, the masks
// and the bias gradients (14 launches); its 4.4 GFLOP take 60 us at the FP32
// peak.  The three 11000-wide products take 60-92 us each, bound by the
// issue slots of the 4 x 4 tiles (FMA pipe half busy); 8 x 4 tiles with 128
// threads measured 292 us for the step, a four-stage cp.async ring 280 us.
static int gemm_split(int M, int N, int K) {
  const int tiles = ((M + kTile - 1) / kTile) * ((N + kTile - 1) / kTile);
  const int slices = (K + kTk - 1) / kTk;
  int s = 1;
  while (s < kGemmMaxSplit && 2 * s * tiles <= 2 * 148 && slices >= 4 * 2 * s) s *= 2;
  return s;
}

template <bool TA, bool TB>
static int launch_gemm_as(const GemmArgs& g, cudaStream_t stream) {
  const int split = gemm_split(g.M, g.N, g.K);
  if (split > 8) {  // beyond the portable cluster size
    const int rc = cuda_check(
        cudaFuncSetAttribute(gemm_kernel<TA, TB>, cudaFuncAttributeNonPortableClusterSizeAllowed,
                             1),
        "cudaFuncSetAttribute(gemm_kernel)");
    if (rc) return rc;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((g.N + kTile - 1) / kTile, (g.M + kTile - 1) / kTile, split);
  cfg.blockDim = dim3(kGemmThreads);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 1;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = split;
  cfg.attrs = at;
  cfg.numAttrs = split > 1 ? 1 : 0;
  return cuda_check(cudaLaunchKernelEx(&cfg, gemm_kernel<TA, TB>, g), "gemm_kernel launch");
}

static int launch_gemm(const GemmArgs& g, bool ta, bool tb, cudaStream_t stream) {
  if (g.M == 0 || g.N == 0) return QTQP_OK;
  if (ta) return tb ? launch_gemm_as<true, true>(g, stream) : launch_gemm_as<true, false>(g, stream);
  return tb ? launch_gemm_as<false, true>(g, stream) : launch_gemm_as<false, false>(g, stream);
}

__global__ void relu_grad_kernel(float* __restrict__ dh, const float* __restrict__ h,
                                 int64_t count) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count;
       i += int64_t(gridDim.x) * blockDim.x)
    if (!(h[i] > 0.0f)) dh[i] = 0.0f;
}

// One thread per column; consecutive threads read consecutive columns.
__global__ void colsum_kernel(const float* __restrict__ d, int rows, int cols,
                              float* __restrict__ db) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= cols) return;
  float t = 0.0f;
  for (int i = 0; i < rows; ++i) t += d[size_t(i) * cols + j];
  db[j] = t;
}

// dy = 2 (y - t) / count; the squared errors are summed per block in FP64
// and added to *loss (zeroed by the caller's memset on the same stream).
__global__ void mse_grad_kernel(const float* __restrict__ y, const float* __restrict__ t,
                                int64_t count, float* __restrict__ dy, double* loss) {
  __shared__ double part[32];
  double acc = 0.0;
  const float scale = 2.0f / float(count);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count;
       i += int64_t(gridDim.x) * blockDim.x) {
    const float e = y[i] - t[i];
    dy[i] = scale * e;
    acc += double(e) * double(e);
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) part[warp] = acc;
  __syncthreads();
  if (warp == 0) {
    acc = lane < int(blockDim.x >> 5) ? part[lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) atomicAdd(loss, acc);
  }
}

// Hinge on the sign of the inequality outputs, added to dy after the MSE
// gradient: for columns [col0, cols) of a rows x cols output, with the
// column's decision point zero[j] (the standardised value of y_i - s_i = 0)
// and the target's side sign = +1 (t > zero) or -1,
//   loss += weight * mean relu(margin - sign (y - zero))  (as a sum, see below),
//   dy   += -weight * sign * [margin - sign (y - zero) > 0] / (rows (cols - col0)).
__global__ void hinge_grad_kernel(const float* __restrict__ y, const float* __restrict__ t,
                                  int rows, int cols, int col0, const float* __restrict__ zero,
                                  float weight, float margin, float* __restrict__ dy,
                                  double* loss) {
  __shared__ double part[32];
  const int w = cols - col0;
  const int64_t total = int64_t(rows) * w;
  const float inv = 1.0f / float(total);
  double acc = 0.0;
  for (int64_t e = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; e < total;
       e += int64_t(gridDim.x) * blockDim.x) {
    const int r = int(e / w), j = col0 + int(e % w);
    const size_t i = size_t(r) * cols + j;
    const float z0 = zero[j - col0];
    const float sg = t[i] > z0 ? 1.0f : -1.0f;
    const float h = margin - sg * (y[i] - z0);
    if (h > 0.0f) {
      dy[i] -= weight * sg * inv;
      acc += double(h);
    }
  }
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) part[warp] = acc;
  __syncthreads();
  if (warp == 0) {
    acc = lane < int(blockDim.x >> 5) ? part[lane] : 0.0;
    for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    // *loss holds a sum over all rows x cols outputs (the MSE kernel's sum of
    // squares); scaled so that loss / (rows cols) = mse + weight mean(h).
    if (lane == 0)
      atomicAdd(loss, double(weight) * acc * (double(rows) * cols / double(total)));
  }
}

__global__ void adam_kernel(float* __restrict__ p, const float* __restrict__ g,
                            float* __restrict__ m, float* __restrict__ v, int64_t count, float lr,
                            float b1, float b2, float eps, float c1, float c2) {
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < count;
       i += int64_t(gridDim.x) * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

// v = pred * scale + shift per coordinate.  x = v[0:n], y_eq = v[n:n+z];
// inequality row i carries v_i = y_i - s_i, decoded as y_i = max(v_i, 0) and
// active[i] = (v_i > threshold).
__global__ void decode_kernel(const float* __restrict__ pred, const double* __restrict__ scale,
                              const double* __restrict__ shift, int n, int m, int z, int count,
                              double threshold, double* __restrict__ x_out,
                              double* __restrict__ y_out, unsigned char* __restrict__ active) {
  const int N = n + m;
  const size_t total = size_t(count) * N;
  for (size_t e = blockIdx.x * size_t(blockDim.x) + threadIdx.x; e < total;
       e += size_t(gridDim.x) * blockDim.x) {
    const int inst = int(e / N), k = int(e % N);
    const double v = double(pred[e]) * scale[k] + shift[k];
    if (k < n) {
      x_out[size_t(inst) * n + k] = v;
    } else {
      const int i = k - n;
      y_out[size_t(inst) * m + i] = (i < z) ? v : fmax(v, 0.0);
      active[size_t(inst) * m + i] = (i < z || v > threshold) ? 1 : 0;
    }
  }
}

static int grid_for(size_t count) {
  return int(std::max<size_t>(1, std::min<size_t>((count + 255) / 256, 148 * 16)));
}

}  // namespace qtqp

using namespace qtqp;

extern "C" int qtqp_mlp_gemm(int32_t M, int32_t N, int32_t K, float alpha, const float* d_a,
                             int32_t lda, int32_t trans_a, const float* d_b, int32_t ldb,
                             int32_t trans_b, float beta, float* d_c, int32_t ldc,
                             const float* d_bias, int32_t relu, void* stream) {
  if (M < 0 || N < 0 || K < 0 || d_a == nullptr || d_b == nullptr || d_c == nullptr ||
      ldc < N || lda < (trans_a ? M : K) || ldb < (trans_b ? K : N))
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_gemm: bad sizes, leading dimensions or pointers");
  GemmArgs g = {};
  g.M = M;
  g.N = N;
  g.K = K;
  g.alpha = alpha;
  g.a = d_a;
  g.lda = lda;
  g.b = d_b;
  g.ldb = ldb;
  g.beta = beta;
  g.c = d_c;
  g.ldc = ldc;
  g.bias = d_bias;
  g.relu = relu;
  return launch_gemm(g, trans_a != 0, trans_b != 0, static_cast<cudaStream_t>(stream));
}

// The network of one training step: the layer sizes dim -> hidden -> hidden
// -> out and a batch of rows.
static int step_args(const qtqp_mlp_step* s, const char* who) {
  if (s == nullptr || s->batch < 1 || s->dim < 1 || s->hidden < 1 || s->out < 1)
    return fail(QTQP_ERR_BAD_ARG, std::string(who) + ": null step or sizes below 1");
  for (const void* p : {(const void*)s->x, (const void*)s->target, (const void*)s->w1,
                        (const void*)s->b1, (const void*)s->w2, (const void*)s->b2,
                        (const void*)s->w3, (const void*)s->b3, (const void*)s->h1,
                        (const void*)s->h2, (const void*)s->y, (const void*)s->dy,
                        (const void*)s->dh1, (const void*)s->dh2, (const void*)s->g1,
                        (const void*)s->gb1, (const void*)s->g2, (const void*)s->gb2,
                        (const void*)s->g3, (const void*)s->gb3, (const void*)s->loss})
    if (p == nullptr) return fail(QTQP_ERR_BAD_ARG, std::string(who) + ": null pointer");
  return QTQP_OK;
}

static GemmArgs gemm_of(int M, int N, int K, const float* a, int lda, const float* b, int ldb,
                        float* c) {
  GemmArgs g = {};
  g.M = M;
  g.N = N;
  g.K = K;
  g.alpha = 1.0f;
  g.a = a;
  g.lda = lda;
  g.b = b;
  g.ldb = ldb;
  g.c = c;
  g.ldc = N;
  return g;
}

// Forward pass with the squared error and its gradient formed in the last
// product's epilogue: three launches (the error and gradient were a fourth
// pass over y and the target).
extern "C" int qtqp_mlp_forward_loss(const qtqp_mlp_step* s, void* stream) {
  int rc = step_args(s, "qtqp_mlp_forward_loss");
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  rc = cuda_check(cudaMemsetAsync(s->loss, 0, sizeof(double), st), "cudaMemsetAsync");
  if (rc) return rc;
  const int B = s->batch, H = s->hidden;
  GemmArgs g = gemm_of(B, H, s->dim, s->x, s->dim, s->w1, H, s->h1);
  g.bias = s->b1;
  g.relu = 1;
  if ((rc = launch_gemm(g, false, false, st))) return rc;
  g = gemm_of(B, H, H, s->h1, H, s->w2, H, s->h2);
  g.bias = s->b2;
  g.relu = 1;
  if ((rc = launch_gemm(g, false, false, st))) return rc;
  g = gemm_of(B, s->out, H, s->h2, H, s->w3, s->out, s->y);
  g.bias = s->b3;
  g.target = s->target;
  g.dy = s->dy;
  g.dscale = 2.0f / float(int64_t(B) * s->out);
  g.loss = s->loss;
  return launch_gemm(g, false, false, st);
}

// Backward pass from dy: five launches.  The weight gradients' products also
// give the bias gradients (the column sums of their right operand), and the
// hidden gradients' products apply the ReLU mask as they store.
extern "C" int qtqp_mlp_backward(const qtqp_mlp_step* s, void* stream) {
  int rc = step_args(s, "qtqp_mlp_backward");
  if (rc) return rc;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int B = s->batch, H = s->hidden, out = s->out;
  GemmArgs g = gemm_of(H, out, B, s->h2, H, s->dy, out, s->g3);  // dW3 = H2^T dY
  g.colsum = s->gb3;
  if ((rc = launch_gemm(g, true, false, st))) return rc;
  g = gemm_of(B, H, out, s->dy, out, s->w3, out, s->dh2);  // dH2 = dY W3^T
  g.mask = s->h2;
  if ((rc = launch_gemm(g, false, true, st))) return rc;
  g = gemm_of(H, H, B, s->h1, H, s->dh2, H, s->g2);  // dW2 = H1^T dH2
  g.colsum = s->gb2;
  if ((rc = launch_gemm(g, true, false, st))) return rc;
  g = gemm_of(B, H, H, s->dh2, H, s->w2, H, s->dh1);  // dH1 = dH2 W2^T
  g.mask = s->h1;
  if ((rc = launch_gemm(g, false, true, st))) return rc;
  g = gemm_of(s->dim, H, B, s->x, s->dim, s->dh1, H, s->g1);  // dW1 = X^T dH1
  g.colsum = s->gb1;
  return launch_gemm(g, true, false, st);
}

extern "C" int qtqp_mlp_relu_grad(float* d_dh, const float* d_h, int64_t count, void* stream) {
  if (count < 0 || (count > 0 && (d_dh == nullptr || d_h == nullptr)))
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_relu_grad: bad arguments");
  if (count == 0) return QTQP_OK;
  relu_grad_kernel<<<grid_for(count), 256, 0, static_cast<cudaStream_t>(stream)>>>(d_dh, d_h,
                                                                                   count);
  return cuda_check(cudaGetLastError(), "relu_grad_kernel launch");
}

extern "C" int qtqp_mlp_colsum(const float* d_d, int32_t rows, int32_t cols, float* d_db,
                               void* stream) {
  if (rows < 0 || cols < 0 || (cols > 0 && (d_d == nullptr || d_db == nullptr)))
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_colsum: bad arguments");
  if (cols == 0) return QTQP_OK;
  colsum_kernel<<<(cols + 255) / 256, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_d, rows,
                                                                                   cols, d_db);
  return cuda_check(cudaGetLastError(), "colsum_kernel launch");
}

extern "C" int qtqp_mlp_mse_grad(const float* d_y, const float* d_t, int64_t count, float* d_dy,
                                 double* d_loss, void* stream) {
  if (count < 1 || d_y == nullptr || d_t == nullptr || d_dy == nullptr || d_loss == nullptr)
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_mse_grad: bad arguments");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  int rc = cuda_check(cudaMemsetAsync(d_loss, 0, sizeof(double), st), "cudaMemsetAsync");
  if (rc) return rc;
  mse_grad_kernel<<<grid_for(count), 256, 0, st>>>(d_y, d_t, count, d_dy, d_loss);
  return cuda_check(cudaGetLastError(), "mse_grad_kernel launch");
}

extern "C" int qtqp_mlp_adam(float* d_p, const float* d_g, float* d_m, float* d_v, int64_t count,
                             float lr, float beta1, float beta2, float eps, int32_t step,
                             void* stream) {
  if (count < 0 || step < 1 || d_p == nullptr || d_g == nullptr || d_m == nullptr ||
      d_v == nullptr)
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_adam: bad arguments");
  if (count == 0) return QTQP_OK;
  const float c1 = 1.0f - float(std::pow(double(beta1), double(step)));
  const float c2 = 1.0f - float(std::pow(double(beta2), double(step)));
  adam_kernel<<<grid_for(count), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      d_p, d_g, d_m, d_v, count, lr, beta1, beta2, eps, c1, c2);
  return cuda_check(cudaGetLastError(), "adam_kernel launch");
}

extern "C" int qtqp_mlp_decode(const float* d_pred, const double* d_scale, const double* d_shift,
                               int32_t n, int32_t m, int32_t z, int32_t count, double threshold,
                               double* d_x, double* d_y, unsigned char* d_active, void* stream) {
  if (n < 1 || m < 1 || z < 0 || z > m || count < 0)
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_decode: bad sizes");
  if (count == 0) return QTQP_OK;
  if (d_pred == nullptr || d_scale == nullptr || d_shift == nullptr || d_x == nullptr ||
      d_y == nullptr || d_active == nullptr)
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_decode: null pointer");
  decode_kernel<<<grid_for(size_t(count) * (n + m)), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      d_pred, d_scale, d_shift, n, m, z, count, threshold, d_x, d_y, d_active);
  return cuda_check(cudaGetLastError(), "decode_kernel launch");
}

extern "C" int qtqp_mlp_hinge_grad(const float* d_y, const float* d_t, int32_t rows,
                                   int32_t cols, int32_t col0, const float* d_zero, float weight,
                                   float margin, float* d_dy, double* d_loss, void* stream) {
  if (rows < 1 || cols < 1 || col0 < 0 || col0 >= cols || d_y == nullptr || d_t == nullptr ||
      d_zero == nullptr || d_dy == nullptr || d_loss == nullptr)
    return fail(QTQP_ERR_BAD_ARG, "qtqp_mlp_hinge_grad: bad arguments");
  hinge_grad_kernel<<<grid_for(size_t(rows) * (cols - col0)), 256, 0,
                      static_cast<cudaStream_t>(stream)>>>(d_y, d_t, rows, cols, col0, d_zero,
                                                            weight, margin, d_dy, d_loss);
  return cuda_check(cudaGetLastError(), "hinge_grad_kernel launch");
}
