// Training and batch-inference kernels of the plan-selection MLP
// (NFEAT -> 128 -> 128 -> 128 -> 1, ReLU), exposed through the C-ABI on
// device pointers so that a driver (Python or C++) can run the training
// loop while every forward, backward, loss and optimiser step runs in these
// kernels.
//
// A training step is a chain of small dependent products (1,024 rows: 0.2
// GFLOP), so its time is latency: launches, and the serial sum of each output.
// The forward pass is one launch and the backward pass two:
//   mlpForwardKernel   a CTA takes R rows through all layers; the weights
//                      (152 KB) are copied to shared memory at the start, each
//                      layer waits for its own;
//   mlpBackwardRows    a CTA takes R rows back through layers 3 and 2 (the
//                      gradients of their inputs, D2 and D1);
//   mlpWeightGrads     a cluster of 8 CTAs per 32 x 64 tile of a weight
//                      gradient, each summing an eighth of the rows, combined
//                      through distributed shared memory in a fixed order.
// A layer-by-layer version (a 64 x 64-tiled SGEMM, bias, mask and column-sum
// kernels, 22 launches) took 721 us for a step of 1,024 rows, most of it in the
// weight gradients, whose four CTAs each summed all rows one after the other;
// this takes 28.8 us (28.5 to 31.1 from run to run), of which forward 8.1 and
// backward 15.7.
//
// Everything is float32 on the FMA units: an output's products are added in
// input order, one fused multiply-add each, as a plain loop would.  The tensor
// cores have no float32 product, and at 0.2 GFLOP they would save nothing.
//
// Parameter layout (also used by the host inference in select.cpp): W1
// [128][NFEAT], b1 [128], W2 [128][128], b2, W3 [128][128], b3, W4 [1][128],
// b4 [1]; weights row-major [out][in].
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <type_traits>

#include "tile_kernel.cuh"
#include "librett.h"
#include "librett_c.h"
#include "plans.h"
#include "select.h"

namespace lt {
namespace {

namespace cg = cooperative_groups;

// Kernel arguments carry no __restrict__: a load that the compiler may take for
// invariant could be moved above dependencyWait.

constexpr int H = MLP_HIDDEN;
constexpr int MLP_THREADS = 256;
static_assert(H == 128, "thread layout");
constexpr int LD = H + 4;           // padded row of 128 in shared memory (16-byte aligned,
                                    // rows 33 16-byte units apart: no bank conflict)
constexpr int XLD = (NFEAT + 3) / 4 * 4;

__device__ __forceinline__ void copyAsync4(float* dst, const float* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

__device__ __forceinline__ void copyAsync16(float* dst, const float* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

__device__ __forceinline__ void copyCommit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

template <int N>
__device__ __forceinline__ void copyWait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Weights come by bulk copies that complete on an mbarrier (16 bytes per thread
// and cp.async moved 25 bytes a cycle into an SM), where the parameters are
// 16-byte aligned.  The waits are bounded like the transpose kernels': when a
// copy does not arrive in time, the CTA writes NaN for all of its results, waits
// once more (bounded) for its copies in flight, and returns.
struct Arrival {
  unsigned long long bar;
};

// Test hook: bytes armed beyond what the copies bring, per wait (zeros in every
// other launch).
struct ExtraBytes {
  int wait[3];
};

__device__ __forceinline__ uint32_t sharedAddr(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}

// Called by one thread: one arrival, `bytes` to come.
__device__ __forceinline__ void expect(Arrival& a, uint32_t bytes) {
  mbarArriveExpectTx(sharedAddr(&a.bar), bytes);
}

__device__ __forceinline__ void bulkFloats(float* dst, const float* src, int n, Arrival& a) {
  bulkLoad(sharedAddr(dst), src, (uint32_t)(n * 4), sharedAddr(&a.bar));
}

__device__ __forceinline__ bool arrived(Arrival& a) {
  return mbarWaitBounded(sharedAddr(&a.bar), 0, BULK_WAIT_NS);
}

// The bounded wait of a CTA that gives up: its copies write its shared memory.
__device__ __forceinline__ void outlast(Arrival& a) {
  mbarWaitBounded(sharedAddr(&a.bar), 0, BULK_WAIT_NS);
}

// NaN for n floats at p, by the CTA.
__device__ __forceinline__ void fillNaN(float* p, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = nanf("");
}

// rows x cols of src (row stride sld) into dst (row stride dld) by cp.async, in
// 16-byte units when vec (cols, sld and dld multiples of 4, src 16-byte aligned).
__device__ __forceinline__ void copyRows(float* dst, int dld, const float* src, int sld, int rows,
                                         int cols, bool vec) {
  const int per = vec ? 4 : 1, units = cols / per;
  // one division per thread: (r, c) then advances by blockDim.x units
  int r = (int)threadIdx.x / units, c = (int)threadIdx.x - r * units;
  const int dr = (int)blockDim.x / units, dc = (int)blockDim.x - dr * units;
  while (r < rows) {
    if (vec)
      copyAsync16(dst + r * dld + 4 * c, src + (size_t)r * sld + 4 * c);
    else
      copyAsync4(dst + r * dld + c, src + (size_t)r * sld + c);
    r += dr;
    c += dc;
    if (c >= units) {
      c -= units;
      ++r;
    }
  }
}

__device__ __forceinline__ bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

struct Layout {
  const float *W1, *b1, *W2, *b2, *W3, *b3, *W4, *b4;
};

__host__ __device__ Layout layout(const float* p) {
  Layout L;
  L.W1 = p;
  L.b1 = L.W1 + H * NFEAT;
  L.W2 = L.b1 + H;
  L.b2 = L.W2 + H * H;
  L.W3 = L.b2 + H;
  L.b3 = L.W3 + H * H;
  L.W4 = L.b3 + H;
  L.b4 = L.W4 + H;
  return L;
}

// Rows a CTA takes: the fewest that fill the device once, so that small batches
// spread over it and large ones read the weights as seldom as possible.
int rowsPerCta(int batch, int sms) {
  return batch <= 8 * sms ? 8 : batch <= 16 * sms ? 16 : 32;
}

// A thread's outputs of a layer for R rows and 128 columns: TM rows from
// row(), TN columns col() + 64 * j (TN 2) or one column.
template <int R>
struct Place {
  static constexpr int TN = R == 32 ? 2 : 1;
  static constexpr int TM = R * H / MLP_THREADS / TN;
  static constexpr int COLS = H / TN;
  __device__ static int col() { return threadIdx.x % COLS; }
  __device__ static int row() { return threadIdx.x / COLS * TM; }
};

// acc += sum over k of in[row][k] * w(k)[col], products in input order; w(k, j)
// gives weights k .. k + 3 of column j.  The operands of the next four inputs
// are read ahead of this four's products: with two warps per scheduler the
// reads' latency otherwise bounds the loop.
template <int R, typename W4>
__device__ __forceinline__ void layerProducts(const float* in, W4 w4,
                                              float (&acc)[Place<R>::TM][Place<R>::TN]) {
  using P = Place<R>;
  const float* a = in + P::row() * LD;
  float4 w[P::TN], x[P::TM];
  auto read = [&](int k) {
#pragma unroll
    for (int j = 0; j < P::TN; ++j) w[j] = w4(k, j);
#pragma unroll
    for (int i = 0; i < P::TM; ++i) x[i] = *reinterpret_cast<const float4*>(a + i * LD + k);
  };
  read(0);
#pragma unroll 4
  for (int k = 0; k < H; k += 4) {
    float4 cw[P::TN], cx[P::TM];
#pragma unroll
    for (int j = 0; j < P::TN; ++j) cw[j] = w[j];
#pragma unroll
    for (int i = 0; i < P::TM; ++i) cx[i] = x[i];
    if (k + 4 < H) read(k + 4);
#pragma unroll
    for (int i = 0; i < P::TM; ++i)
#pragma unroll
      for (int j = 0; j < P::TN; ++j) acc[i][j] = __fmaf_rn(cx[i].x, cw[j].x, acc[i][j]);
#pragma unroll
    for (int i = 0; i < P::TM; ++i)
#pragma unroll
      for (int j = 0; j < P::TN; ++j) acc[i][j] = __fmaf_rn(cx[i].y, cw[j].y, acc[i][j]);
#pragma unroll
    for (int i = 0; i < P::TM; ++i)
#pragma unroll
      for (int j = 0; j < P::TN; ++j) acc[i][j] = __fmaf_rn(cx[i].z, cw[j].z, acc[i][j]);
#pragma unroll
    for (int i = 0; i < P::TM; ++i)
#pragma unroll
      for (int j = 0; j < P::TN; ++j) acc[i][j] = __fmaf_rn(cx[i].w, cw[j].w, acc[i][j]);
  }
}

// With the weights in padded rows of LD, one per output.
template <int R>
__device__ __forceinline__ void layerTimesRows(const float* in, const float* w,
                                               float (&acc)[Place<R>::TM][Place<R>::TN]) {
  using P = Place<R>;
  const float* b = w + P::col() * LD;
  layerProducts<R>(
      in, [&](int k, int j) { return *reinterpret_cast<const float4*>(b + j * P::COLS * LD + k); },
      acc);
}

// With the weights in rows of H, one per input.
template <int R>
__device__ __forceinline__ void layerTimesCols(const float* in, const float* w,
                                               float (&acc)[Place<R>::TM][Place<R>::TN]) {
  using P = Place<R>;
  const float* b = w + P::col();
  layerProducts<R>(
      in,
      [&](int k, int j) {
        const float* q = b + k * H + j * P::COLS;
        return make_float4(q[0], q[H], q[2 * H], q[3 * H]);
      },
      acc);
}

template <int R>
struct ForwardShared {
  float W2[H * LD], W3[H * LD];
  float X[R * XLD];
  float A[R * LD], B[R * LD];
  float W1[H * NFEAT];
  float b1[H], b2[H], b3[H], W4[H];
  Arrival first, second, third;  // W1 and X's CTA-wide part; W2; W3
};

// Bias, ReLU; the activation to shared memory and to global memory.
template <int R>
__device__ __forceinline__ void activate(const float (&acc)[Place<R>::TM][Place<R>::TN],
                                         const float* bias, float* shared, float* global, int rows) {
  using P = Place<R>;
#pragma unroll
  for (int i = 0; i < P::TM; ++i)
#pragma unroll
    for (int j = 0; j < P::TN; ++j) {
      const int r = P::row() + i, c = P::col() + j * P::COLS;
      float v = acc[i][j] + bias[c];
      v = v < 0.f ? 0.f : v;
      shared[r * LD + c] = v;
      if (r < rows) global[(size_t)r * H + c] = v;
    }
}

template <int R>
__global__ void __launch_bounds__(MLP_THREADS)
mlpForwardKernel(const float* params, const float* X, int batch,
                 float* ws, float* out, ExtraBytes extra) {
  using P = Place<R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  ForwardShared<R>& s = *reinterpret_cast<ForwardShared<R>*>(smraw);
  dependencyRelease();
  const int r0 = blockIdx.x * R, rows = min(R, batch - r0);
  const Layout L = layout(params);
  const bool vec = aligned16(params);
  if (threadIdx.x == 0) {
    mbarInit(sharedAddr(&s.first.bar), 1);
    mbarInit(sharedAddr(&s.second.bar), 1);
    mbarInit(sharedAddr(&s.third.bar), 1);
    mbarInitFence();
  }
  __syncthreads();
  dependencyWait();
  if (vec) {
    if (threadIdx.x == 0) {
      expect(s.first, H * NFEAT * 4 + extra.wait[0]);
      bulkFloats(s.W1, L.W1, H * NFEAT, s.first);
      expect(s.second, H * H * 4 + extra.wait[1]);
      expect(s.third, H * H * 4 + extra.wait[2]);
    }
    __syncthreads();  // the counts are armed before a copy completes
    if (threadIdx.x < H) {
      bulkFloats(s.W2 + threadIdx.x * LD, L.W2 + threadIdx.x * H, H, s.second);
      bulkFloats(s.W3 + threadIdx.x * LD, L.W3 + threadIdx.x * H, H, s.third);
    }
  } else {
    copyRows(s.W1, H * NFEAT, L.W1, 0, 1, H * NFEAT, false);
    copyRows(s.W2, LD, L.W2, H, H, H, false);
    copyRows(s.W3, LD, L.W3, H, H, H, false);
  }
  copyRows(s.X, XLD, X + (size_t)r0 * NFEAT, NFEAT, rows, NFEAT, false);
  copyRows(s.b1, H, L.b1, 0, 1, H, vec);
  copyRows(s.b2, H, L.b2, 0, 1, H, vec);
  copyRows(s.b3, H, L.b3, 0, 1, H, vec);
  copyRows(s.W4, H, L.W4, 0, 1, H, vec);
  copyCommit();
  float* A1 = ws + (size_t)r0 * H;
  float* A2 = A1 + (size_t)batch * H;
  float* A3 = A2 + (size_t)batch * H;
  auto giveUp = [&] {
    fillNaN(A1, rows * H);
    fillNaN(A2, rows * H);
    fillNaN(A3, rows * H);
    fillNaN(out + r0, rows);
    outlast(s.first);
    outlast(s.second);
    outlast(s.third);
  };
  // rows past the batch: any finite input
  for (int i = rows * XLD + threadIdx.x; i < R * XLD; i += MLP_THREADS) s.X[i] = 0.f;
  copyWait<0>();
  if (!__syncthreads_and(!vec || arrived(s.first))) return giveUp();
  {
    float acc[P::TM][P::TN] = {};
    const float* a = s.X + P::row() * XLD;
    const float* w = s.W1 + P::col() * NFEAT;  // NFEAT odd: no bank conflict
#pragma unroll 8
    for (int k = 0; k < NFEAT; ++k) {
      float wv[P::TN];
#pragma unroll
      for (int j = 0; j < P::TN; ++j) wv[j] = w[j * P::COLS * NFEAT + k];
#pragma unroll
      for (int i = 0; i < P::TM; ++i)
#pragma unroll
        for (int j = 0; j < P::TN; ++j) acc[i][j] = __fmaf_rn(a[i * XLD + k], wv[j], acc[i][j]);
    }
    activate<R>(acc, s.b1, s.A, A1, rows);
  }
  if (!__syncthreads_and(!vec || arrived(s.second))) return giveUp();
  {
    float acc[P::TM][P::TN] = {};
    layerTimesRows<R>(s.A, s.W2, acc);
    activate<R>(acc, s.b2, s.B, A2, rows);
  }
  if (!__syncthreads_and(!vec || arrived(s.third))) return giveUp();
  {
    float acc[P::TM][P::TN] = {};
    layerTimesRows<R>(s.B, s.W3, acc);
    activate<R>(acc, s.b3, s.A, A3, rows);
  }
  __syncthreads();
  if ((int)threadIdx.x < rows) {
    const float* a = s.A + threadIdx.x * LD;
    float v = 0.f;
#pragma unroll 8
    for (int k = 0; k < H; k += 4) {
      const float4 av = *reinterpret_cast<const float4*>(a + k);
      const float4 wv = *reinterpret_cast<const float4*>(s.W4 + k);
      v = __fmaf_rn(av.x, wv.x, v);
      v = __fmaf_rn(av.y, wv.y, v);
      v = __fmaf_rn(av.z, wv.z, v);
      v = __fmaf_rn(av.w, wv.w, v);
    }
    out[r0 + threadIdx.x] = v + *L.b4;
  }
}

// The gradient of the network's output with respect to activation 3 of a row,
// where that is positive (ReLU'): dout * W4.
__device__ __forceinline__ float outputGrad(float a3, float dout, float w4) {
  return a3 > 0.f ? __fmaf_rn(dout, w4, 0.f) : 0.f;
}

template <int R>
struct BackwardShared {
  float W3[H * H], W2[H * H];
  float D[R * LD], E[R * LD];
  Arrival first, second;  // W3, W2
};

// A thread's outputs' places in an activation or gradient of H columns.
template <int R, typename F>
__device__ __forceinline__ void forOutputs(F f) {
  using P = Place<R>;
#pragma unroll
  for (int i = 0; i < P::TM; ++i)
#pragma unroll
    for (int j = 0; j < P::TN; ++j) f(i, j, P::row() + i, P::col() + j * P::COLS);
}

// D2 = (D3 W3) masked by A2 and D1 = (D2 W2) masked by A1, with D3 = dout W4
// masked by A3.  D2 goes to the workspace's fifth part, D1 to its fourth.
template <int R>
__global__ void __launch_bounds__(MLP_THREADS)
mlpBackwardRows(const float* params, int batch, float* ws,
                const float* dout, ExtraBytes extra) {
  using P = Place<R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  BackwardShared<R>& s = *reinterpret_cast<BackwardShared<R>*>(smraw);
  dependencyRelease();
  const int r0 = blockIdx.x * R, rows = min(R, batch - r0);
  const Layout L = layout(params);
  const bool vec = aligned16(params);
  if (threadIdx.x == 0) {
    mbarInit(sharedAddr(&s.first.bar), 1);
    mbarInit(sharedAddr(&s.second.bar), 1);
    mbarInitFence();
  }
  __syncthreads();
  dependencyWait();
  if (vec) {
    if (threadIdx.x == 0) {
      constexpr int PIECE = H * H / 4;
      expect(s.first, H * H * 4 + extra.wait[0]);
      for (int i = 0; i < H * H; i += PIECE) bulkFloats(s.W3 + i, L.W3 + i, PIECE, s.first);
      expect(s.second, H * H * 4 + extra.wait[1]);
      for (int i = 0; i < H * H; i += PIECE) bulkFloats(s.W2 + i, L.W2 + i, PIECE, s.second);
    }
  } else {
    copyRows(s.W3, H * H, L.W3, 0, 1, H * H, false);
    copyRows(s.W2, H * H, L.W2, 0, 1, H * H, false);
    copyCommit();
  }
  const size_t part = (size_t)batch * H;
  const float* A1 = ws + (size_t)r0 * H;
  const float* A2 = A1 + part;
  const float* A3 = A2 + part;
  float* D1 = ws + 3 * part + (size_t)r0 * H;
  float* D2 = D1 + part;
  auto giveUp = [&] {
    fillNaN(D1, rows * H);
    fillNaN(D2, rows * H);
    outlast(s.first);
    outlast(s.second);
  };
  constexpr int PER = R * H / MLP_THREADS;  // elements of D3 a thread makes
  float a3[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = threadIdx.x + q * MLP_THREADS;
    a3[q] = i / H < rows ? A3[i] : 0.f;
  }
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int i = threadIdx.x + q * MLP_THREADS, r = i / H, c = i % H;
    s.D[r * LD + c] = r < rows ? outputGrad(a3[q], dout[r0 + r], L.W4[c]) : 0.f;
  }
  // the masks of both products, read while the weights are on their way
  bool on2[P::TM][P::TN], on1[P::TM][P::TN];
  forOutputs<R>([&](int i, int j, int r, int c) {
    on2[i][j] = r < rows && A2[(size_t)r * H + c] > 0.f;
    on1[i][j] = r < rows && A1[(size_t)r * H + c] > 0.f;
  });
  if (!vec) copyWait<0>();
  if (!__syncthreads_and(!vec || arrived(s.first))) return giveUp();
  {
    float acc[P::TM][P::TN] = {};
    layerTimesCols<R>(s.D, s.W3, acc);
    forOutputs<R>([&](int i, int j, int r, int c) {
      const float v = on2[i][j] ? acc[i][j] : 0.f;
      s.E[r * LD + c] = v;
      if (r < rows) D2[(size_t)r * H + c] = v;
    });
  }
  if (!__syncthreads_and(!vec || arrived(s.second))) return giveUp();
  {
    float acc[P::TM][P::TN] = {};
    layerTimesCols<R>(s.E, s.W2, acc);
    forOutputs<R>([&](int i, int j, int r, int c) {
      if (r < rows) D1[(size_t)r * H + c] = on1[i][j] ? acc[i][j] : 0.f;
    });
  }
}

// Weight gradients: gW[o][i] = sum over rows of D[row][o] * In[row][i] and gb[o]
// = sum of D[row][o], in tiles of GO x GI.  A cluster of GC CTAs shares a tile;
// CTA c takes GROWS-row chunks c, c + GC, ... of the batch (the next chunk on its
// way while one is summed), each GPARTS-th of its threads every GPARTS-th row.
// A thread sums 4 x 8 products per row for three 16-byte reads, so the kernel is
// bound by the FMA pipe; 22 tiles x 8 CTAs cover the device.
constexpr int GO = 32, GI = 64, GC = 8, GROWS = 128, GTHREADS = 256;
constexpr int GPART = (GO / 4) * (GI / 8), GPARTS = GTHREADS / GPART;
constexpr int DLD = GO + 4, ILD = GI + 4;
constexpr int GW_TILES = (H / GO) * (H / GI);  // of W3 and of W2
constexpr int GTILES = 2 * GW_TILES + H / GO + H / GI;
static_assert(NFEAT <= GI, "one tile width covers the features");

struct GradShared {
  struct Chunk {
    float D[GROWS * DLD], In[GROWS * ILD], dout[GROWS];
  } chunk[2];
  float W4[H];
  float bias[GPARTS][GO];
};
constexpr int GPARTIAL = GO * ILD;  // floats of a part's tile, in the chunks' place
static_assert(GPARTS * GPARTIAL * sizeof(float) <= sizeof(GradShared::chunk), "parts' tiles fit");

__global__ void __cluster_dims__(GC, 1, 1) __launch_bounds__(GTHREADS)
mlpWeightGrads(const float* params, const float* X, int batch, const float* ws, const float* dout,
               float* grads) {
  extern __shared__ __align__(16) unsigned char smraw[];
  GradShared& s = *reinterpret_cast<GradShared*>(smraw);
  cg::cluster_group cluster = cg::this_cluster();
  dependencyRelease();
  const int tile = blockIdx.x / GC, rank = (int)cluster.block_rank(), tid = threadIdx.x;
  const Layout L = layout(params);
  const size_t part = (size_t)batch * H;
  // which gradient: its D and In with their first column and width, and where
  // the tile goes
  int layer, o0 = 0, i0 = 0, width = GI, ild = H;
  const float *Dg = ws, *Ig;
  if (tile < 2 * GW_TILES) {
    layer = tile < GW_TILES ? 3 : 2;
    const int t = tile % GW_TILES;
    o0 = t / (H / GI) * GO;
    i0 = t % (H / GI) * GI;
    Dg = layer == 3 ? ws + 2 * part : ws + 4 * part;  // layer 3: A3, made D3 below
    Ig = layer == 3 ? ws + part : ws;
  } else if (tile < 2 * GW_TILES + H / GO) {
    layer = 1;
    o0 = (tile - 2 * GW_TILES) * GO;
    Dg = ws + 3 * part;
    Ig = X;
    ild = width = NFEAT;
  } else {
    layer = 4;  // one row of gradients: D is dout
    i0 = (tile - 2 * GW_TILES - H / GO) * GI;
    Ig = ws + 2 * part;
  }
  const bool vec = aligned16(ws), bias = i0 == 0;
  const int sub = tid / GPART, tx = tid % 8, ty = tid / 8 % (GO / 4);
  float acc[4][8] = {}, accD[4] = {};  // the tile: columns 4 tx + j, then 32 + 4 tx + j; the bias
  dependencyWait();
  if (layer == 3) copyRows(s.W4, H, L.W4, 0, 1, H, aligned16(params));
  auto fetch = [&](int b0, GradShared::Chunk& c) {
    const int rows = min(GROWS, batch - b0);
    if (layer != 4) copyRows(c.D, DLD, Dg + (size_t)b0 * H + o0, H, rows, GO, vec);
    copyRows(c.In, ILD, Ig + (size_t)b0 * ild + i0, ild, rows, width, vec && layer != 1);
    if (layer >= 3) copyRows(c.dout, GROWS, dout + b0, 0, 1, rows, false);
    copyCommit();
  };
  const int first = rank * GROWS, stride = GC * GROWS;
  if (first < batch) fetch(first, s.chunk[0]);
  int buf = 0;
  for (int b0 = first; b0 < batch; b0 += stride, buf ^= 1) {
    const int rows = min(GROWS, batch - b0);
    GradShared::Chunk& c = s.chunk[buf];
    if (b0 + stride < batch) {
      fetch(b0 + stride, s.chunk[buf ^ 1]);
      copyWait<1>();
    } else {
      copyWait<0>();
    }
    __syncthreads();
    if (layer == 3) {
#pragma unroll 4
      for (int i = tid; i < rows * GO; i += GTHREADS) {
        float& d = c.D[i / GO * DLD + i % GO];
        d = outputGrad(d, c.dout[i / GO], s.W4[o0 + i % GO]);
      }
      __syncthreads();
    }
    if (layer == 4) {
      const float* x = c.In + tid % GI;
#pragma unroll 8
      for (int r = tid / GI; r < rows; r += GTHREADS / GI) {
        acc[0][0] = __fmaf_rn(c.dout[r], x[r * ILD], acc[0][0]);
        accD[0] += c.dout[r];
      }
    } else if (tx * 4 < width) {
      auto sum = [&](auto withBias) {
#pragma unroll 4
        for (int r = sub; r < rows; r += GPARTS) {
          const float4 d = *reinterpret_cast<const float4*>(c.D + r * DLD + ty * 4);
          const float4 x = *reinterpret_cast<const float4*>(c.In + r * ILD + tx * 4);
          const float4 y = *reinterpret_cast<const float4*>(c.In + r * ILD + GI / 2 + tx * 4);
          const float dv[4] = {d.x, d.y, d.z, d.w};
          const float xv[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (decltype(withBias)::value) accD[i] += dv[i];
#pragma unroll
            for (int j = 0; j < 8; ++j) acc[i][j] = __fmaf_rn(dv[i], xv[j], acc[i][j]);
          }
        }
      };
      if (bias)
        sum(std::true_type{});
      else
        sum(std::false_type{});
    }
    __syncthreads();  // the chunk after the next reuses this buffer
  }
  cpAsyncWaitAll();  // W4's copy, in a CTA that had no rows
  // the parts' sums to shared memory, added in part order
  float* partial = s.chunk[0].D;  // the chunks' place, from its start
  if (layer == 4) {
    partial[tid] = acc[0][0];
    if (tid % GI == 0) s.bias[tid / GI][0] = accD[0];
  } else {
    float* at = partial + sub * GPARTIAL + ty * 4 * ILD + tx * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      *reinterpret_cast<float4*>(at + i * ILD) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4*>(at + i * ILD + GI / 2) =
          make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      if (tx == 0) s.bias[sub][ty * 4 + i] = accD[i];
    }
  }
  __syncthreads();
  const int outs = layer == 4 ? GI : GO * ILD, apart = layer == 4 ? GI : GPARTIAL;
  for (int i = tid; i < outs; i += GTHREADS) {
    float v = partial[i];
#pragma unroll
    for (int k = 1; k < GPARTS; ++k) v += partial[k * apart + i];
    partial[i] = v;
  }
  if (tid < GO) {
    float v = s.bias[0][tid];
#pragma unroll
    for (int k = 1; k < GPARTS; ++k) v += s.bias[k][tid];
    s.bias[0][tid] = v;
  }
  cluster.sync();
  // CTA `rank` adds the eight CTAs' sums of its share, in rank order
  auto total = [&](float* at) {
    float v = 0.f;
#pragma unroll
    for (int c = 0; c < GC; ++c) v += *cluster.map_shared_rank(at, c);
    return v;
  };
  const Layout G = layout(grads);
  if (layer == 4) {
    constexpr int OUT = GI / GC;
    if (tid < OUT) const_cast<float*>(G.W4)[i0 + rank * OUT + tid] = total(partial + rank * OUT + tid);
    if (bias && rank == 0 && tid == OUT) *const_cast<float*>(G.b4) = total(&s.bias[0][0]);
  } else {
    float* gW = const_cast<float*>(layer == 3 ? G.W3 : layer == 2 ? G.W2 : G.W1);
    float* gb = const_cast<float*>(layer == 3 ? G.b3 : layer == 2 ? G.b2 : G.b1);
    constexpr int OUT = GO / GC;  // rows of the tile
    const int o = rank * OUT + tid / GI, c = tid % GI;
    static_assert(OUT * GI == GTHREADS, "one output a thread");
    if (c < width) gW[(size_t)(o0 + o) * ild + i0 + c] = total(partial + o * ILD + c);
    if (bias && tid < OUT) gb[o0 + rank * OUT + tid] = total(&s.bias[0][rank * OUT + tid]);
  }
  cluster.sync();  // no CTA leaves while another reads its shared memory
}

// dout[b] = 2 (out[b] - y[b]) / batch; *loss += sum (out - y)^2 / batch.
__global__ void mseGradKernel(const float* out, const float* y, int batch, float* dout,
                              float* loss) {
  __shared__ float red[256];
  float s = 0.f;
  dependencyRelease();
  dependencyWait();
  for (int b = blockIdx.x * blockDim.x + threadIdx.x; b < batch; b += gridDim.x * blockDim.x) {
    const float d = out[b] - y[b];
    dout[b] = 2.f * d / batch;
    s += d * d / batch;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w) red[threadIdx.x] += red[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0 && loss != nullptr) atomicAdd(loss, red[0]);
}

// Adam (Kingma & Ba, 2015) with bias correction.
__global__ void adamKernel(float* p, const float* g, float* m, float* v, int n, float lr,
                           float b1, float b2, float eps, float c1, float c2) {
  dependencyRelease();
  dependencyWait();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  }
}

int gridFor(size_t n) {
  size_t g = (n + 255) / 256;
  return (int)(g > 4096 ? 4096 : (g < 1 ? 1 : g));
}

// Launches kernel<R> for the rows a CTA takes; shared: its structure by R.
template <typename K8, typename K16, typename K32, typename... Args>
cudaError_t launchRowsOf(int batch, cudaStream_t s, size_t sm8, size_t sm16, size_t sm32, K8 k8,
                         K16 k16, K32 k32, Args... args) {
  int dev = 0, sms = 0;
  if (!currentDevice(dev, sms)) return cudaErrorInvalidDevice;
  const int R = rowsPerCta(batch, sms);
  const size_t smem = R == 8 ? sm8 : R == 16 ? sm16 : sm32;
  const auto kernel = R == 8 ? k8 : R == 16 ? k16 : k32;
  if (cachedOccupancy((const void*)kernel, MLP_THREADS, (int)smem) < 1)
    return cudaErrorInvalidConfiguration;
  return launchDependent(kernel, (unsigned)((batch + R - 1) / R), MLP_THREADS, smem, s, args...);
}

cudaError_t forwardRows(const float* params, const float* X, int batch, float* ws, float* out,
                        cudaStream_t s, const ExtraBytes& extra) {
  return launchRowsOf(batch, s, sizeof(ForwardShared<8>), sizeof(ForwardShared<16>),
                      sizeof(ForwardShared<32>), mlpForwardKernel<8>, mlpForwardKernel<16>,
                      mlpForwardKernel<32>, params, X, batch, ws, out, extra);
}

cudaError_t backwardRows(const float* params, int batch, float* ws, const float* dout,
                         cudaStream_t s, const ExtraBytes& extra) {
  return launchRowsOf(batch, s, sizeof(BackwardShared<8>), sizeof(BackwardShared<16>),
                      sizeof(BackwardShared<32>), mlpBackwardRows<8>, mlpBackwardRows<16>,
                      mlpBackwardRows<32>, params, batch, ws, dout, extra);
}

}  // namespace
}  // namespace lt

extern "C" {

int librett_c_mlp_param_count(void) { return lt::mlpParamCount(); }

int librett_c_mlp_feature_count(void) { return lt::NFEAT; }

int librett_c_mlp_workspace_floats(int batch) { return 5 * batch * lt::H; }

int librett_c_mlp_forward(const float* params, const float* X, int batch, float* ws, float* out,
                          void* stream) {
  using namespace lt;
  if (!params || !X || !ws || !out || batch < 1) return LIBRETT_INVALID_PARAMETER;
  const cudaError_t err = forwardRows(params, X, batch, ws, out, (cudaStream_t)stream, {});
  return err == cudaSuccess ? LIBRETT_SUCCESS : LIBRETT_INTERNAL_ERROR;
}

int librett_c_mlp_backward(const float* params, const float* X, int batch, float* ws,
                           const float* dout, float* grads, void* stream) {
  using namespace lt;
  if (!params || !X || !ws || !dout || !grads || batch < 1) return LIBRETT_INVALID_PARAMETER;
  cudaStream_t s = (cudaStream_t)stream;
  cudaError_t err = backwardRows(params, batch, ws, dout, s, {});
  if (err == cudaSuccess)
    err = cachedOccupancy((const void*)mlpWeightGrads, GTHREADS, (int)sizeof(GradShared)) < 1
              ? cudaErrorInvalidConfiguration
              : launchDependent(mlpWeightGrads, GTILES * GC, GTHREADS, sizeof(GradShared), s, params, X,
                                batch, (const float*)ws, dout, grads);
  return err == cudaSuccess ? LIBRETT_SUCCESS : LIBRETT_INTERNAL_ERROR;
}

int librett_c_mlp_wait_test(int backward, int wait, unsigned extra_bytes, const float* params,
                            const float* X, int batch, float* ws, float* out, void* stream) {
  using namespace lt;
  if (!params || (!backward && !X) || !ws || !out || batch < 1 || batch > 4096 ||
      (uintptr_t)params % 16 || wait < 0 || wait >= (backward ? 2 : 3) || extra_bytes == 0 ||
      extra_bytes > 4096)
    return LIBRETT_INVALID_PARAMETER;
  ExtraBytes extra = {};
  extra.wait[wait] = (int)extra_bytes;
  cudaStream_t s = (cudaStream_t)stream;
  const cudaError_t err = backward ? backwardRows(params, batch, ws, out, s, extra)
                                   : forwardRows(params, X, batch, ws, out, s, extra);
  return err == cudaSuccess && cudaStreamSynchronize(s) == cudaSuccess ? LIBRETT_SUCCESS
                                                                       : LIBRETT_INTERNAL_ERROR;
}

int librett_c_mlp_mse_grad(const float* out, const float* y, int batch, float* dout, float* loss,
                           void* stream) {
  if (!out || !y || !dout || batch < 1) return LIBRETT_INVALID_PARAMETER;
  const cudaError_t err = lt::launchDependent(lt::mseGradKernel, (unsigned)lt::gridFor(batch), 256, 0,
                                              (cudaStream_t)stream, out, y, batch, dout, loss);
  return err == cudaSuccess ? LIBRETT_SUCCESS : LIBRETT_INTERNAL_ERROR;
}

int librett_c_mlp_adam(float* params, const float* grads, float* m, float* v, int n, float lr,
                       float beta1, float beta2, float eps, int step, void* stream) {
  if (!params || !grads || !m || !v || n < 1 || step < 1) return LIBRETT_INVALID_PARAMETER;
  const float c1 = 1.f - powf(beta1, (float)step), c2 = 1.f - powf(beta2, (float)step);
  const cudaError_t err =
      lt::launchDependent(lt::adamKernel, (unsigned)lt::gridFor(n), 256, 0, (cudaStream_t)stream, params,
                          grads, m, v, n, lr, beta1, beta2, eps, c1, c2);
  return err == cudaSuccess ? LIBRETT_SUCCESS : LIBRETT_INTERNAL_ERROR;
}

}  // extern "C"
