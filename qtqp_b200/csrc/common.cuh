// Shared device helpers: block-wide fused reductions and error bookkeeping.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cstdio>
#include <string>

#include "qtqp_cuda.h"

namespace qtqp {

constexpr double kEps = 1e-15;  // src/qtqp/__init__.py:51

void set_last_error(const std::string& msg);
int fail(int code, const std::string& msg);
int cuda_check(cudaError_t err, const char* what);

// Propagates NaN like numpy's max (np.linalg.norm(.., inf) of a vector with
// a NaN is NaN); fmax would drop it.
__device__ __forceinline__ double nanmax(double a, double b) {
  return (a != a || b != b) ? __longlong_as_double(0x7ff8000000000000ll) : fmax(a, b);
}

// A double as a signed integer of the same order, and back: the block
// reductions take their maxima in integers (a compare and a select; the NaN
// test and FP64 maximum of nanmax cost three times as much).  A NaN without
// its sign bit, which is what fabs and nanmax give, is above every number.
__device__ __forceinline__ long long max_key(double v) {
  const long long i = __double_as_longlong(v);
  return i ^ ((i >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double from_max_key(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}

// The IPM's heavy phases are compiled as separate device functions: each then
// gets its own register allocation, which keeps the long solve loop's live
// state from spilling into the phases' inner loops.
#define QTQP_PHASE __device__ __noinline__

// Largest number of values one fused reduction may carry.
constexpr int kRedMax = 16;

// Block-wide reduction of NS sums and NM maxima in one barrier.  Every thread
// receives the results.  `red` is shared scratch of 2 * (NT/32) * kRedMax
// doubles; `phase` alternates between its two halves so that consecutive
// reductions need a single __syncthreads each (a thread can only reach the
// reduction after next once every thread has finished reading this one,
// because the next reduction's barrier separates them).
// ST < NT: only the first ST threads carry sums (the others' are zero or stale
// and are not read); their warps' sums are added one after the other, so the
// result depends on ST alone and not on the block's size.
template <int NT, int NS, int NM, int ST = NT>
__device__ __forceinline__ void block_reduce(double (&sums)[NS > 0 ? NS : 1],
                                             double (&maxs)[NM > 0 ? NM : 1],
                                             double* red, int& phase) {
  static_assert(NS + NM <= kRedMax, "too many reduction slots");
  constexpr int NW = NT / 32;
  // The loops over shuffle distances and warps stay rolled (the values of
  // one step unrolled): every reduction of the IPM is inlined at its call
  // site, and fully unrolled they made up much of the per-iteration code
  // that competes for the instruction cache.  The order of the operations
  // is the same either way.
  long long keys[NM > 0 ? NM : 1];
#pragma unroll
  for (int k = 0; k < NM; ++k) keys[k] = max_key(maxs[k]);
#pragma unroll 1
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int k = 0; k < NS; ++k) sums[k] += __shfl_xor_sync(0xffffffffu, sums[k], off);
#pragma unroll
    for (int k = 0; k < NM; ++k) keys[k] = max(keys[k], __shfl_xor_sync(0xffffffffu, keys[k], off));
  }
  if constexpr (NW > 1) {
    double* buf = red + phase * (NW * kRedMax);
    phase ^= 1;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0) {
#pragma unroll
      for (int k = 0; k < NS; ++k) buf[warp * kRedMax + k] = sums[k];
#pragma unroll
      for (int k = 0; k < NM; ++k) buf[warp * kRedMax + NS + k] = __longlong_as_double(keys[k]);
    }
    __syncthreads();
    // Lane l starts from warp l % NW's values; log2(NW) shuffles combine them.
    const double* mine = buf + (lane & (NW - 1)) * kRedMax;
    if constexpr (ST < NT) {
#pragma unroll
      for (int k = 0; k < NS; ++k) {
        sums[k] = 0.0;
        for (int w = 0; w < ST / 32; ++w) sums[k] += buf[w * kRedMax + k];
      }
    } else {
#pragma unroll
      for (int k = 0; k < NS; ++k) sums[k] = mine[k];
    }
#pragma unroll
    for (int k = 0; k < NM; ++k) keys[k] = __double_as_longlong(mine[NS + k]);
#pragma unroll 1
    for (int off = NW / 2; off > 0; off >>= 1) {
      if constexpr (ST == NT) {
#pragma unroll
        for (int k = 0; k < NS; ++k) sums[k] += __shfl_xor_sync(0xffffffffu, sums[k], off);
      }
#pragma unroll
      for (int k = 0; k < NM; ++k)
        keys[k] = max(keys[k], __shfl_xor_sync(0xffffffffu, keys[k], off));
    }
  }
#pragma unroll
  for (int k = 0; k < NM; ++k) maxs[k] = from_max_key(keys[k]);
}

// A barrier for the whole group (one thread block).
template <int NT>
__device__ __forceinline__ void group_sync() {
  if constexpr (NT == 32) {
    __syncwarp();
  } else {
    __syncthreads();
  }
}

// ----------------------------------------------------------------------------
// Grid-wide barrier and reductions of a cooperative launch (every block
// resident), for one large QP solved by the whole GPU.  The barrier is one
// 64-bit counter in global memory: every block adds 1 with release semantics
// and polls the same word with acquire loads; block 0 adds 2^31 - (blocks -
// 1) instead, so bit 31 flips when the last block has arrived.  A wait that
// exceeds kGridWaitLimit polls sets the sticky `err` flag and the counter's
// top bit, after which every barrier returns at once (the solve then finishes
// its bounded loops and reports the error).
// (148 blocks: 1.9 us per barrier.  An arrival counter with a separate
// generation word, fences and polls spaced by 64 ns took 3.5 us, that pair
// without the spacing 2.5 us, a flag per block polled by a warp 4.0-6.5 us.)
// ----------------------------------------------------------------------------
constexpr int kGridMaxBlocks = 256;
constexpr int kGridBT = 256;  // threads per block of a grid-mode solve
// Supernodal factorisation: the widest supernode (its diagonal block stays in
// shared memory) and the rows of a top-level supernode per work item.  Both
// the host symbolic stage and the device phases use them.
constexpr int kSnMaxWidth = 64;
constexpr int kSnSlabRows = 64;
constexpr int kSnDenseMax = 4096;  // most columns of the dense part above the subtrees
constexpr uint32_t kGridWaitLimit = 1u << 25;

struct GridCtl {
  unsigned long long arrive;  // grid_sync's counter; kGridErrBit: a wait gave up
  int err;                    // 1: a barrier or slot wait gave up
  int pad;
  double part[2][kGridMaxBlocks][kRedMax];  // per-block partials (double-buffered)
};

constexpr unsigned long long kGridErrBit = 1ull << 63;

__device__ __forceinline__ void grid_fail(GridCtl* g) {
  atomicExch(&g->err, 1);
  atomicOr(&g->arrive, kGridErrBit);
}

__device__ __forceinline__ void grid_sync(GridCtl* g, uint32_t limit = kGridWaitLimit) {
  __syncthreads();
  if (threadIdx.x == 0) {
    const unsigned long long add = blockIdx.x == 0 ? (1ull << 31) - (gridDim.x - 1) : 1ull;
    unsigned long long old, v;
    asm volatile("atom.add.release.gpu.global.u64 %0, [%1], %2;"
                 : "=l"(old)
                 : "l"(&g->arrive), "l"(add)
                 : "memory");
    if (!(old & kGridErrBit)) {
      for (uint32_t it = 0;; ++it) {
        asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(&g->arrive) : "memory");
        if (((old ^ v) & (1ull << 31)) != 0 || (v & kGridErrBit) != 0) break;
        if (it >= limit) {
          grid_fail(g);
          break;
        }
      }
    }
  }
  __syncthreads();
}

// Point-to-point hand-off between the blocks of a cooperative grid: a 16-byte
// slot per value, the value with the tag of the step that wrote it, stored and
// loaded as one 128-bit access.  So the value itself is what a consumer polls;
// no fence, flag or barrier lies between the two blocks.  Tags only grow and the
// slots start at zero, so a slot is never reset.
struct alignas(16) GridSlot {
  unsigned long long bits, tag;
};
__device__ __forceinline__ void slot_store(GridSlot* p, double v, unsigned long long tag) {
  asm volatile(
      "{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
      "l"(__double_as_longlong(v)), "l"(tag)
      : "memory");
}
__device__ __forceinline__ GridSlot slot_load(const GridSlot* p) {
  GridSlot r;
  asm volatile(
      "{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
      : "=l"(r.bits), "=l"(r.tag)
      : "l"(p)
      : "memory");
  return r;
}

// Called by one whole warp: the values of slots p[0], p[stride], ... (K per
// lane), once all of the warp's carry `tag` (bounded wait).  A wait that exceeds
// `limit` polls sets the sticky err flag, after which every later wait returns
// soon, with whatever is there (the solve runs to its end and reports it).
template <int K>
__device__ __forceinline__ void slots_wait(GridCtl* g, const GridSlot* p, int stride,
                                           unsigned long long tag, double (&out)[K],
                                           uint32_t limit = kGridWaitLimit) {
  for (uint32_t it = 0;; ++it) {
    bool ok = true;
    GridSlot r[K];
#pragma unroll
    for (int k = 0; k < K; ++k) r[k] = slot_load(p + k * stride);
#pragma unroll
    for (int k = 0; k < K; ++k) {
      ok = ok && r[k].tag == tag;
      out[k] = __longlong_as_double(r[k].bits);
    }
    if (__all_sync(0xffffffffu, ok)) return;
    const int lane = threadIdx.x & 31;
    if ((it & 15) == 15) {  // each look at the error is another L2 round trip
      int err = lane == 0 ? *reinterpret_cast<volatile int*>(&g->err) : 0;
      if (__shfl_sync(0xffffffffu, err, 0)) return;
    }
    if (it >= limit) {
      if (lane == 0) grid_fail(g);
      return;
    }
  }
}

// NS sums and NM maxima over every thread of the grid; all threads receive
// the same values (the partials are combined in one fixed order in every
// block, so control flow that depends on them agrees across blocks).  `red`
// is shared scratch of 2 * (blockDim.x / 32) * kRedMax doubles; `phase`
// alternates the global partial buffers (see block_reduce).
template <int BT, int NS, int NM>
__device__ __forceinline__ void grid_reduce(double (&sums)[NS > 0 ? NS : 1],
                                            double (&maxs)[NM > 0 ? NM : 1], double* red,
                                            GridCtl* g, int& phase) {
  static_assert(NS + NM <= kRedMax, "too many reduction slots");
  constexpr int NW = BT / 32;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
    for (int k = 0; k < NS; ++k) sums[k] += __shfl_xor_sync(0xffffffffu, sums[k], off);
#pragma unroll
    for (int k = 0; k < NM; ++k)
      maxs[k] = nanmax(maxs[k], __shfl_xor_sync(0xffffffffu, maxs[k], off));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double* wbuf = red;                // NW x kRedMax warp partials
  double* res = red + NW * kRedMax;  // kRedMax results
  if (lane == 0) {
#pragma unroll
    for (int k = 0; k < NS; ++k) wbuf[warp * kRedMax + k] = sums[k];
#pragma unroll
    for (int k = 0; k < NM; ++k) wbuf[warp * kRedMax + NS + k] = maxs[k];
  }
  __syncthreads();
  double* part = &g->part[phase][0][0];
  phase ^= 1;
  // Value k: thread k over the block's warps, after the barrier warp k (mod
  // NW) over the blocks, each in one fixed order.
  if (threadIdx.x < NS + NM) {
    const int k = threadIdx.x;
    double acc = k < NS ? 0.0 : wbuf[k];
    for (int w = k < NS ? 0 : 1; w < NW; ++w) {
      const double v = wbuf[w * kRedMax + k];
      acc = k < NS ? acc + v : nanmax(acc, v);
    }
    part[blockIdx.x * kRedMax + k] = acc;
  }
  grid_sync(g);
  const int nb = gridDim.x;
  for (int k = warp; k < NS + NM; k += NW) {
    constexpr int Q = kGridMaxBlocks / 32;
    double v[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q)
      v[q] = lane + 32 * q < nb ? part[(lane + 32 * q) * kRedMax + k] : 0.0;
    double acc = 0.0;
    if (k < NS) {
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (lane + 32 * q < nb) acc += v[q];
      for (int off = 16; off > 0; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    } else {
      acc = part[k];  // block 0's partial starts every lane
#pragma unroll
      for (int q = 0; q < Q; ++q)
        if (lane + 32 * q < nb) acc = nanmax(acc, v[q]);
      for (int off = 16; off > 0; off >>= 1)
        acc = nanmax(acc, __shfl_xor_sync(0xffffffffu, acc, off));
    }
    if (lane == 0) res[k] = acc;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < NS; ++k) sums[k] = res[k];
#pragma unroll
  for (int k = 0; k < NM; ++k) maxs[k] = res[NS + k];
}

// Asynchronous global -> shared copies (cp.async): 8 bytes (zero-filled
// when !valid) or 4 bytes; commit a group; wait until at most N groups of
// this thread are in flight.
__device__ __forceinline__ void cp_async8(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(valid ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() {
  asm volatile("cp.async.commit_group;" ::: "memory");
}
__device__ __forceinline__ void cp_async4z(void* dst, const void* src, bool valid) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(valid ? 4 : 0)
               : "memory");
}
// 16 bytes, both addresses 16-byte aligned.
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src)
               : "memory");
}
// The same with the first `bytes` (0, 8 or 16) read and the rest zero-filled.
__device__ __forceinline__ void cp_async16z(void* dst, const void* src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "r"(bytes)
               : "memory");
}
// Element copy of T (double or float), zero-filled when !valid.
template <typename T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src, bool valid) {
  if constexpr (sizeof(T) == 8) {
    cp_async8(dst, src, valid);
  } else {
    cp_async4z(dst, src, valid);
  }
}
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src)
               : "memory");
}
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}


// One FP64 tensor-core step d += a b (mma.sync m8n8k4, row.col; tcgen05 has
// no FP64 kind): lane l holds a = A[l/4][l%4], b = B[l%4][l/4] and the
// accumulator entries (l/4, 2 (l%4)) and (l/4, 2 (l%4) + 1).
__device__ __forceinline__ void dmma_8x8x4(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__device__ __forceinline__ uint64_t globaltimer_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// Optional per-phase cycle counters for profiling builds (-DQTQP_PHASE_TIMERS):
// thread 0 of each block adds the SM cycles spent in a phase to
// g_phase_cycles[phase].  Default builds compile these to nothing.
enum Phase : int {
  kPhLoad = 0, kPhNormalize, kPhGram, kPhChol, kPhSolve, kPhResidual, kPhTau, kPhStep,
  kPhTerm, kPhOther,
  // Sub-phases of the large (grid-mode) factorisation and solves.
  kPhLgDiag, kPhLgPanel, kPhLgTrail, kPhLgInv, kPhLgFwd, kPhLgBwd,
  // Sub-phases of the partitioned banded factorisation and solves.
  kPhBpInterior, kPhBpChain, kPhBpFwd, kPhBpChains, kPhBpBwd,
  // Steps of one reduction level (per participating block).
  kPhBpCrStage, kPhBpCrSweep, kPhBpCrGemm, kPhBpCrGather,
  // Sub-phases of the supernodal factorisation and solves (subtrees / top levels).
  kPhSnSub, kPhSnTop, kPhSnFwdSub, kPhSnFwdTop, kPhSnBwdTop, kPhSnBwdSub,
  kPhSnTopUpd, kPhSnTopDiag, kPhSnTopPanel,
  // Sub-phases of the dense KKT solve: the column sums A^T (r_y / Ry) and the
  // row products A x around the triangular solves.
  kPhSolveCols, kPhSolveRows,
  // Sub-phases of the per-block dense format: the inverse of the factor's
  // 32 x 32 diagonal blocks and the triangular solves of a KKT solve.
  kPhInv, kPhTri, kNumPhases
};
#ifdef QTQP_PHASE_TIMERS
extern __device__ unsigned long long g_phase_cycles[kNumPhases];
#define QTQP_TIC() long long qtqp_t0_ = clock64()
#define QTQP_RETIC() qtqp_t0_ = clock64()
#define QTQP_TOC(ph)                                                                   \
  do {                                                                                 \
    if (threadIdx.x == 0)                                                              \
      atomicAdd(&qtqp::g_phase_cycles[ph], (unsigned long long)(clock64() - qtqp_t0_)); \
  } while (0)
#else
#define QTQP_TIC() \
  do {             \
  } while (0)
#define QTQP_RETIC() \
  do {               \
  } while (0)
#define QTQP_TOC(ph) \
  do {               \
  } while (0)
#endif

}  // namespace qtqp
