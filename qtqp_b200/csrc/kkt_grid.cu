// See kkt_grid.cuh.  The factor, the inverses of its diagonal blocks and the
// slots' generation live in the workspace between the calls; a solve's CTAs
// bring the inverse of their block back into shared memory first.
#include "kkt_grid.cuh"

#include <algorithm>

namespace qtqp {

struct KktGridLayout {
  int npad, nblk;
  size_t tri_off, gen_off, info_off, g_off, inv_off, sinv_off, cp_off, gpart_off, total;
};
static __host__ __device__ inline KktGridLayout plan_kkt_grid(int n, int m) {
  KktGridLayout L;
  L.npad = round_up(n, kLB);
  L.nblk = L.npad / kLB;
  auto al = [](size_t b) { return (b + 255) & ~size_t(255); };
  size_t off = al(sizeof(GridCtl));  // the barrier and the slots come first
  L.tri_off = off;
  off += al(size_t(L.npad) * sizeof(GridSlot));
  L.gen_off = off;
  L.info_off = off + 16;
  off += 256;
  L.g_off = off;
  off += al(size_t(L.npad) * L.npad * 8);
  L.inv_off = off;
  off += al(size_t(L.nblk) * kLB * kLB * 8);
  L.sinv_off = off;
  off += al(size_t(4) * 32 * kSubPitch * 8);
  L.cp_off = off;
  off += al(size_t(kLargeBlocks) * L.npad * 8);
  L.gpart_off = off;
  off += al(GramSplit(L.npad, m).slot_bytes());
  L.total = off;
  return L;
}

size_t kkt_grid_bytes(int n, int m) {
  return plan_kkt_grid(n, m).total;
}

using KktGridIpm = Ipm<kLargeNT, kFmtLarge>;

__device__ inline void kkt_grid_bind(KktGridIpm& s, int n, int m, char* ws, char* gws,
                                     unsigned char* arena, double* red) {
  const InstLayout I = plan_layout(n, m, 0);
  const KktGridLayout L = plan_kkt_grid(n, m);
  s.tid = blockIdx.x * blockDim.x + threadIdx.x;
  s.n = n;
  s.m = m;
  s.N = n + m;
  s.z = 0;
  s.has_p = true;
  s.lda = I.lda;
  s.ldp = I.ldp;
  s.ldg = L.npad;
  s.np = I.np;
  s.V = reinterpret_cast<double*>(ws + I.g_bytes);
  s.A = reinterpret_cast<double*>(ws + I.g_bytes + I.v_bytes);
  s.P = reinterpret_cast<double*>(ws + I.g_bytes + I.v_bytes + I.a_bytes);
  s.gctl = reinterpret_cast<GridCtl*>(gws);
  s.linfo = reinterpret_cast<int*>(gws + L.info_off);
  s.npad = L.npad;
  s.mpad = 0;
  s.g64 = reinterpret_cast<double*>(gws + L.g_off);
  s.G = s.g64;
  s.g32l = nullptr;
  s.sinv = reinterpret_cast<double*>(gws + L.sinv_off);
  s.gpart = reinterpret_cast<double*>(gws + L.gpart_off);
  s.colpart = reinterpret_cast<double*>(gws + L.cp_off);
  s.arena = arena;
  s.tri_gen = *reinterpret_cast<const uint32_t*>(gws + L.gen_off);
  s.tri_slot = reinterpret_cast<GridSlot*>(gws + L.tri_off);
  s.red = red;
  s.phase = 0;
  s.o = nullptr;
}

__global__ void __launch_bounds__(kGridBT, 1)
    kkt_grid_factorize_kernel(int n, int m, const double* diag, char* ws, size_t header, char* gws,
                              int* info) {
  __shared__ double red[2 * (kGridBT / 32) * kRedMax];
  extern __shared__ __align__(16) unsigned char arena[];
  KktGridIpm s;
  kkt_grid_bind(s, n, m, ws + header, gws, arena, red);
  const KktGridLayout L = plan_kkt_grid(n, m);
  s.kkt_diag_given(diag);
  s.sync();
  const int rc = s.template factorize<double>();
  if (rc == 0 && int(blockIdx.x) < L.nblk) {  // the block's inverse, for the solves
    const double* inv = reinterpret_cast<const double*>(arena);
    double* dst = reinterpret_cast<double*>(gws + L.inv_off) + size_t(blockIdx.x) * kLB * kLB;
    for (int e = threadIdx.x; e < kLB * kLB; e += kGridBT)
      dst[e] = inv[(e >> 7) * kPitch + (e & 127)];
  }
  if (s.tid == 0) {
    // A wait that gave up leaves no usable factor.
    const bool gave_up = *reinterpret_cast<volatile int*>(&s.gctl->err) != 0;
    *info = gave_up ? -1 : rc;
    *reinterpret_cast<int*>(ws) = kKktFactorGrid;
  }
}

__global__ void __launch_bounds__(kGridBT, 1)
    kkt_grid_solve_kernel(int n, int m, const double* rhs, double* out, char* ws, size_t header,
                          char* gws) {
  __shared__ double red[2 * (kGridBT / 32) * kRedMax];
  extern __shared__ __align__(16) unsigned char arena[];
  const int factor = *reinterpret_cast<const int*>(ws);
  if (factor != kKktFactorGrid) {  // the single block's
    if (blockIdx.x != 0) return;
    DenseIpm<kGridBT> d;
    d.bind(n, m, nullptr, ws + header, 0);
    d.z = 0;
    d.has_p = true;
    d.red = red;
    d.phase = 0;
    d.o = nullptr;
    d.kkt_solve(rhs, out, false, factor != kKktFactor32);
    return;
  }
  KktGridIpm s;
  kkt_grid_bind(s, n, m, ws + header, gws, arena, red);
  const KktGridLayout L = plan_kkt_grid(n, m);
  if (int(blockIdx.x) < L.nblk)
    stage_block(reinterpret_cast<double*>(arena),
                reinterpret_cast<const double*>(gws + L.inv_off) + size_t(blockIdx.x) * kLB * kLB,
                kLB, 0, 0);
  __syncthreads();
  s.kkt_solve(rhs, out, false, true);
  // Every block has passed the solve's barriers, so it has read the old value.
  if (s.tid == 0) *reinterpret_cast<uint32_t*>(gws + L.gen_off) = s.tri_gen;
}

__global__ void __launch_bounds__(kGridBT)
    kkt_grid_matvec_kernel(int n, int m, const double* x, double* out, char* ws, size_t header,
                           char* gws) {
  KktGridIpm s;
  kkt_grid_bind(s, n, m, ws + header, gws, nullptr, nullptr);
  s.kkt_matvec(x, out);
}

// (kkt_grid_resident, which every call asks first, has set the kernels' shared
// memory.)
static int coop_launch(const void* kern, void** args, cudaStream_t stream, const char* what) {
  return cuda_check(cudaLaunchCooperativeKernel(kern, dim3(kLargeBlocks), dim3(kGridBT), args,
                                                kArenaBytes, stream),
                    what);
}

int kkt_grid_resident() {
  int dev = 0, sms = 0, coop = 0, a = 0, b = 0;
  for (const void* kern : {reinterpret_cast<const void*>(kkt_grid_factorize_kernel),
                           reinterpret_cast<const void*>(kkt_grid_solve_kernel)})
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kArenaBytes)) !=
        cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&a, kkt_grid_factorize_kernel, kGridBT,
                                                    kArenaBytes) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kkt_grid_solve_kernel, kGridBT,
                                                    kArenaBytes) != cudaSuccess) {
    cudaGetLastError();
    return 0;
  }
  return coop ? sms * std::min(a, b) : 0;
}

int kkt_grid_factorize(int n, int m, const double* diag, char* ws, size_t header, char* gws,
                       int* info, cudaStream_t stream) {
  int rc = cuda_check(cudaMemsetAsync(gws, 0, plan_kkt_grid(n, m).g_off, stream),
                      "cudaMemsetAsync");
  if (rc) return rc;
  void* args[] = {&n, &m, &diag, &ws, &header, &gws, &info};
  return coop_launch(reinterpret_cast<const void*>(kkt_grid_factorize_kernel), args, stream,
                     "kkt_grid_factorize_kernel launch");
}

int kkt_grid_solve(int n, int m, const double* rhs, double* out, char* ws, size_t header,
                   char* gws, cudaStream_t stream) {
  void* args[] = {&n, &m, &rhs, &out, &ws, &header, &gws};
  return coop_launch(reinterpret_cast<const void*>(kkt_grid_solve_kernel), args, stream,
                     "kkt_grid_solve_kernel launch");
}

int kkt_grid_matvec(int n, int m, const double* x, double* out, char* ws, size_t header,
                    char* gws, cudaStream_t stream) {
  kkt_grid_matvec_kernel<<<kLargeBlocks, kGridBT, 0, stream>>>(n, m, x, out, ws, header, gws);
  return cuda_check(cudaGetLastError(), "kkt_grid_matvec_kernel launch");
}

}  // namespace qtqp
