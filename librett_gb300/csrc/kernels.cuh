// Device kernels of the transpose engine (sm_103a).
//
// LibreTT counterparts (src/kernel.cpp): transposeTiled (:48-170),
// transposePacked (:175-296), transposePackedSplit (:304-444) and
// transposeTiledCopy (:453-545), plus the cudaMemcpyAsync used for Trivial
// (:1014-1026).  Here one persistent tile kernel covers Tiled, Packed and
// PackedSplit: the planner's tile (an extent per fused rank) decides which of
// them a launch behaves like.  All data moves as raw 4/8/16-byte words.
#pragma once

#include <cuda_runtime.h>
#include <cstdint>

#include "launch.h"
#include "plan.h"

namespace lt {

template <int ES> struct Word;
template <> struct Word<4> { using T = unsigned int; };
template <> struct Word<8> { using T = uint2; };
template <> struct Word<16> { using T = uint4; };

__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
  return (uint32_t)(((unsigned long long)n * f.mul) >> f.shift);
}

// Programmatic dependent launch: a kernel launched by launchDependent may
// start while the stream's previous kernel is still draining, so its launch
// latency and address decode overlap that kernel's tail.  It must call
// dependencyWait before its first access to global memory (which returns when
// every earlier kernel has completed and its writes are visible; at once for
// an ordinary launch) and calls dependencyRelease first, which lets its own
// successor do the same as soon as all its CTAs run.  Loads that the compiler
// may treat as invariant (const __restrict__ pointers) can be moved above the
// wait, so such kernels load through ldGlobal.  A non-coherent load
// (ld.global.nc, __ldg) is defined for memory that nobody writes while the
// kernel runs; the predecessors still write these inputs then, so they are read by
// ordinary loads only.  Tables fixed before the launch may be read either way.
__device__ __forceinline__ void dependencyRelease() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
}

__device__ __forceinline__ void dependencyWait() {
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

template <int BYTES>
__device__ __forceinline__ typename Word<BYTES>::T ldGlobal(const void* p) {
  typename Word<BYTES>::T v;
  if constexpr (BYTES == 4)
    asm volatile("ld.global.b32 %0, [%1];\n" : "=r"(v) : "l"(p) : "memory");
  else if constexpr (BYTES == 8)
    asm volatile("ld.global.v2.b32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "l"(p) : "memory");
  else
    asm volatile("ld.global.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
  return v;
}

// Launches fn with programmatic stream serialization; as an ordinary launch
// while s is being captured, so a caller's graph keeps its plain edges.
template <typename... Params, typename... Args>
cudaError_t launchDependent(void (*fn)(Params...), unsigned grid, unsigned threads, size_t smem,
                            cudaStream_t s, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute attr = {};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone) {
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
  }
  cudaLaunchKernelEx(&cfg, fn, Params(args)...);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// Trivial: contiguous copy in units of US bytes.  Each CTA copies one block
// of COPY_THREADS * COPY_UNROLL units (four independent loads per thread,
// issued before the stores) and exits; no grid-stride loop, so the block
// scheduler streams blocks through the SMs in address order.
// ---------------------------------------------------------------------------
constexpr int COPY_UNROLL = 4;

template <int US>
__global__ void __launch_bounds__(COPY_THREADS)
copyKernel(const typename Word<US>::T* __restrict__ in, typename Word<US>::T* __restrict__ out,
           long long n) {
  using T = typename Word<US>::T;
  const long long base = (long long)blockIdx.x * (COPY_THREADS * COPY_UNROLL) + threadIdx.x;
  T v[COPY_UNROLL];
  dependencyRelease();
  dependencyWait();
#pragma unroll
  for (int u = 0; u < COPY_UNROLL; ++u)
    if (base + u * COPY_THREADS < n) v[u] = ldGlobal<US>(in + base + u * COPY_THREADS);
#pragma unroll
  for (int u = 0; u < COPY_UNROLL; ++u)
    if (base + u * COPY_THREADS < n) out[base + u * COPY_THREADS] = v[u];
}

// ---------------------------------------------------------------------------
// TiledCopy: input rank 0 is also output rank 0, so the tensor is a set of
// contiguous rows (dim[0] elements) that move to new row positions.  Work
// item = 32 units of one row.  Each CTA takes ROW_ITEMS_PER_CTA consecutive
// items (four per warp, loads issued before stores) and exits.
// ---------------------------------------------------------------------------
constexpr int ROW_ITEMS_PER_WARP = 4;
constexpr int ROW_ITEMS_PER_CTA = (ROW_THREADS / 32) * ROW_ITEMS_PER_WARP;

template <int US>
__global__ void __launch_bounds__(ROW_THREADS)
rowCopyKernel(const __grid_constant__ RowParams p, const typename Word<US>::T* __restrict__ in,
              typename Word<US>::T* __restrict__ out) {
  using T = typename Word<US>::T;
  const int lane = threadIdx.x & 31;
  const uint32_t first =
      blockIdx.x * ROW_ITEMS_PER_CTA + (threadIdx.x >> 5) * ROW_ITEMS_PER_WARP;
  T v[ROW_ITEMS_PER_WARP];
  long long src[ROW_ITEMS_PER_WARP], dst[ROW_ITEMS_PER_WARP];
  bool ok[ROW_ITEMS_PER_WARP];
  dependencyRelease();
#pragma unroll
  for (int u = 0; u < ROW_ITEMS_PER_WARP; ++u) {
    const uint32_t item = first + u;
    ok[u] = false;
    if (item < p.numItems) {
      const uint32_t row = fdiv(item, p.chunkDiv);
      const int col = (int)(item - row * p.chunkDiv.d) * 32 + lane;
      uint32_t rem = row;
      long long bi = 0, bo = 0;
      for (int g = 0; g < p.nR; ++g) {
        const uint32_t q = fdiv(rem, p.rDiv[g]);
        const uint32_t c = rem - q * p.rDiv[g].d;
        rem = q;
        bi += (long long)c * p.rSin[g];
        bo += (long long)c * p.rSout[g];
      }
      if (col < p.rowUnits) {
        ok[u] = true;
        src[u] = bi + col;
        dst[u] = bo + col;
      }
    }
  }
  dependencyWait();
#pragma unroll
  for (int u = 0; u < ROW_ITEMS_PER_WARP; ++u)
    if (ok[u]) v[u] = ldGlobal<US>(in + src[u]);
#pragma unroll
  for (int u = 0; u < ROW_ITEMS_PER_WARP; ++u)
    if (ok[u]) out[dst[u]] = v[u];
}

// Launch helpers (defined in the per-element-size translation units).
cudaError_t launchTile4(const PlanDesc& pd, const DeviceTables* dt, const void* in, void* out,
                        cudaStream_t s, int numSMs, int* grid);
cudaError_t launchTile8(const PlanDesc& pd, const DeviceTables* dt, const void* in, void* out,
                        cudaStream_t s, int numSMs, int* grid);
cudaError_t launchTile16(const PlanDesc& pd, const DeviceTables* dt, const void* in, void* out,
                         cudaStream_t s, int numSMs, int* grid);

}  // namespace lt
