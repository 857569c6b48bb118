// Tile kernel of the transpose engine (sm_103a): covers LibreTT's Tiled,
// Packed and PackedSplit methods (src/kernel.cpp:48-170, :175-296, :304-444).
//
// A tile is the sub-tensor with extent trE[t] along each tile rank.  Its
// elements are numbered j in input order and q in output order.  One CTA
// walks its tiles (blockIdx.x, blockIdx.x + gridDim.x, ...):
//   load  : load unit u (LV consecutive j, one 16-byte access when LV > 1)
//           goes from global memory to shared memory at smemIndex(u * LV);
//   store : store unit w (SV consecutive q) gathers its SV elements from
//           shared memory and leaves as one global store.
// Units never straddle a run boundary and are 16-byte aligned in global
// memory; the planner only picks LV/SV > 1 when the layout guarantees this.
//
// Every tile is full: along a rank whose dim is not a multiple of the
// extent, the last chunk starts at dim - extent and overlaps its neighbour
// (the overlap is loaded and stored twice with identical bits).  So no tile
// needs bounds checks.  Offsets of units relative to the tile base are the
// same for every tile; each CTA computes them once into shared-memory tables
// and only two 64-bit bases change per tile.
#pragma once

#include <type_traits>

#include "group.h"
#include "kernels.cuh"
#include "slots.h"

namespace lt {

// P: TileParams or FlatParams (the same grid-rank fields).
template <typename P>
__device__ __forceinline__ void decodeTile(const P& p, uint32_t tile, long long& bin,
                                           long long& bout) {
  bin = 0;
  bout = 0;
  uint32_t rem = tile;
  for (int g = 0; g < p.nGR; ++g) {
    const uint32_t q = fdiv(rem, p.grDiv[g]);
    const uint32_t c = rem - q * p.grDiv[g].d;
    rem = q;
    const bool last = c + 1 == p.grDiv[g].d;
    bin += last ? p.grLastIn[g] : (long long)c * p.grSin[g];
    bout += last ? p.grLastOut[g] : (long long)c * p.grSout[g];
  }
}

// Returns x unchanged, but the compiler cannot see through it: values derived
// from it are recomputed where used instead of being hoisted out of the tile
// loop and kept live in registers for every slot.
__device__ __forceinline__ int opaque(int x) {
  asm volatile("" : "+r"(x));
  return x;
}

__device__ __forceinline__ int smemIndex(const TileParams& p, int j) {
  return j + ((j >> p.padShift) << p.padLog);
}

__device__ __forceinline__ void cpAsync16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
}

// cp.async of one 4-, 8- or 16-byte unit (16 bytes bypass L1); PF: L2
// prefetch size in bytes (0 none, 128 or 256: the .L2::128B / .L2::256B
// qualifier).
template <int BYTES, int PF = 0>
__device__ __forceinline__ void cpAsyncUnit(uint32_t dst, const void* src) {
  static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async unit");
  static_assert(PF == 0 || PF == 128 || PF == 256, "L2 prefetch size");
  if constexpr (BYTES == 16 && PF == 256)
    asm volatile("cp.async.cg.shared.global.L2::256B [%0], [%1], 16;\n" ::"r"(dst), "l"(src)
                 : "memory");
  else if constexpr (BYTES == 16 && PF == 128)
    asm volatile("cp.async.cg.shared.global.L2::128B [%0], [%1], 16;\n" ::"r"(dst), "l"(src)
                 : "memory");
  else if constexpr (BYTES == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src) : "memory");
  else if constexpr (PF == 256)
    asm volatile("cp.async.ca.shared.global.L2::256B [%0], [%1], %2;\n" ::"r"(dst), "l"(src),
                 "n"(BYTES)
                 : "memory");
  else if constexpr (PF == 128)
    asm volatile("cp.async.ca.shared.global.L2::128B [%0], [%1], %2;\n" ::"r"(dst), "l"(src),
                 "n"(BYTES)
                 : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(dst), "l"(src), "n"(BYTES)
                 : "memory");
}

// L2 prefetch size of the grouped kernel's data copies: 0 (none) or 256
// bytes (the .L2::256B qualifier of cp.async).  256: the 10,000-member batch
// 0.3 % faster than none (two interleaved runs each, one box); 128 made no
// difference.  The single-plan flat kernel uses none: on the 200-problem
// float64 suite 256 bytes measured 0.2 % slower and 128 bytes the same.
#ifndef LT_GROUP_L2_PREFETCH
#define LT_GROUP_L2_PREFETCH 256
#endif

// Flat tile kernels with at least this many load units per thread load
// through cp.async rather than registers: 8 (measured best on the float64
// suite: 4 is 0.1 % and register loads throughout 0.7 % slower), but 4 for
// 4-byte elements (the float32 small-leading-dim case 1.1 % faster).
#ifndef LT_FLAT_ASYNC_MIN_NL
#define LT_FLAT_ASYNC_MIN_NL 8
#endif

template <int ES>
__host__ __device__ constexpr int flatAsyncMinNL() {
  return ES == 4 && LT_FLAT_ASYNC_MIN_NL > 4 ? 4 : LT_FLAT_ASYNC_MIN_NL;
}

__device__ __forceinline__ void cpAsyncWaitAll() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

__device__ __forceinline__ void cpAsyncCommit() {
  asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <int N>
__device__ __forceinline__ void cpAsyncWait() {
  asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Shared-memory tables, built once per CTA:
//   ldOff[u]  global input offset (elements) of load unit u,
//   stOff[w]  global output offset (elements) of store unit w,
//   stSm[q]   shared-memory data index of output-order element q.
struct TileTables {
  int* ldOff;
  int* stOff;
  unsigned short* stSm;
  unsigned char* data;  // data buffers follow the tables (16-byte aligned)
};

// Layout: stSm (2 bytes per element, padded to 16 bytes); ldOff and stOff
// (4 bytes per unit), padded to 16 bytes; then the data buffers.
__host__ __device__ inline int tileSmIndexBytes(int vol) { return ((2 * vol + 15) / 16) * 16; }

__host__ __device__ inline int tileTableBytes(int vol, int lv, int sv) {
  return tileSmIndexBytes(vol) + ((4 * (vol / lv + vol / sv) + 15) / 16) * 16;
}

__device__ __forceinline__ TileTables buildTileTables(const TileParams& p, unsigned char* smraw) {
  TileTables tt;
  tt.stSm = reinterpret_cast<unsigned short*>(smraw);
  tt.ldOff = reinterpret_cast<int*>(smraw + tileSmIndexBytes(p.tileVol));
  tt.stOff = tt.ldOff + p.nIn;
  tt.data = smraw + tileTableBytes(p.tileVol, p.lv, p.sv);
  for (int u = threadIdx.x; u < p.nIn; u += blockDim.x) {
    int rem = u * p.lv, off = 0;
    for (int t = 0; t < p.nTR; ++t) {
      const int e = p.trE[t];
      const int q = rem / e;
      off += (rem - q * e) * p.trSin[t];
      rem = q;
    }
    tt.ldOff[u] = off;
  }
  for (int q = threadIdx.x; q < p.tileVol; q += blockDim.x) {
    int rem = q, off = 0, jj = 0;
    for (int i = 0; i < p.nTR; ++i) {
      const int t = p.trOut[i];
      const int e = p.trE[t];
      const int d = rem / e;
      const int c = rem - d * e;
      rem = d;
      off += c * p.trSout[t];
      jj += c * p.trInTile[t];
    }
    tt.stSm[q] = (unsigned short)smemIndex(p, jj);
    if (q % p.sv == 0) tt.stOff[q / p.sv] = off;
  }
  __syncthreads();
  return tt;
}

// Store phase shared by all pipelines: gather SV elements per store unit
// from shared memory and write them as one access.  stOff / stSm point to
// the offset tables (shared memory or device memory).
template <int ES, int SV>
__device__ __forceinline__ void storeTile(const TileParams& p, const int* __restrict__ stOff,
                                          const unsigned short* __restrict__ stSm,
                                          const typename Word<ES>::T* s,
                                          typename Word<ES>::T* outBase) {
  using T = typename Word<ES>::T;
  using ST = typename Word<ES * SV>::T;
  static_assert(sizeof(ST) == SV * sizeof(T), "unit size");
  const int tv = opaque(threadIdx.x);
#pragma unroll 4
  for (int w = tv; w < p.nOut; w += TILE_THREADS) {
    T* dst = outBase + stOff[w];
    if constexpr (SV == 1) {
      *dst = s[stSm[w]];
    } else {
      T e[SV];
      if constexpr (SV == 2) {
        const unsigned idx = *reinterpret_cast<const unsigned*>(stSm + 2 * w);
        e[0] = s[idx & 0xffffu];
        e[1] = s[idx >> 16];
      } else {
        const uint2 idx = *reinterpret_cast<const uint2*>(stSm + 4 * w);
        e[0] = s[idx.x & 0xffffu];
        e[1] = s[idx.x >> 16];
        e[2] = s[idx.y & 0xffffu];
        e[3] = s[idx.y >> 16];
      }
      ST v;
      __builtin_memcpy(&v, e, sizeof(ST));
      *reinterpret_cast<ST*>(dst) = v;
    }
  }
}

// Shared indices of store unit w's SV elements (stSm entries) in one word.
template <int SV> struct SmIdx;
template <> struct SmIdx<1> { using T = unsigned short; };
template <> struct SmIdx<2> { using T = unsigned; };
template <> struct SmIdx<4> { using T = uint2; };

template <int SV>
__device__ __forceinline__ typename SmIdx<SV>::T loadSmIdx(const unsigned short* __restrict__ stSm,
                                                           int w) {
  return __ldg(reinterpret_cast<const typename SmIdx<SV>::T*>(stSm + SV * w));
}

// Store unit w: gathers its SV elements at shared indices idx and writes
// them as one access at dst.
template <int ES, int SV>
__device__ __forceinline__ void storeUnit(const typename Word<ES>::T* s,
                                          typename SmIdx<SV>::T idx, typename Word<ES>::T* dst) {
  using T = typename Word<ES>::T;
  using ST = typename Word<ES * SV>::T;
  if constexpr (SV == 1) {
    *dst = s[idx];
  } else {
    T e[SV];
    if constexpr (SV == 2) {
      e[0] = s[idx & 0xffffu];
      e[1] = s[idx >> 16];
    } else {
      e[0] = s[idx.x & 0xffffu];
      e[1] = s[idx.x >> 16];
      e[2] = s[idx.y & 0xffffu];
      e[3] = s[idx.y >> 16];
    }
    ST v;
    __builtin_memcpy(&v, e, sizeof(ST));
    *reinterpret_cast<ST*>(dst) = v;
  }
}

// Table entries of a thread's first store units, fetched while the tile's
// data loads are in flight so that the stores can start as soon as the
// barrier opens: the tables are a dependent device-memory read otherwise.
template <int SV, int PF>
struct StorePrefetch {
  int off[PF > 0 ? PF : 1];
  typename SmIdx<SV>::T idx[PF > 0 ? PF : 1];

  __device__ __forceinline__ void load(const TileParams& p, const int* __restrict__ stOff,
                                       const unsigned short* __restrict__ stSm) {
#pragma unroll
    for (int i = 0; i < PF; ++i) {
      const int w = threadIdx.x + i * TILE_THREADS;
      if (w < p.nOut) {
        off[i] = __ldg(stOff + w);
        idx[i] = loadSmIdx<SV>(stSm, w);
      }
    }
  }
};

// Store phase of the flat pipeline: the prefetched units first, then the
// rest as in storeTile.
template <int ES, int SV, int PF>
__device__ __forceinline__ void storeTileFlat(const TileParams& p, const int* __restrict__ stOff,
                                              const unsigned short* __restrict__ stSm,
                                              const StorePrefetch<SV, PF>& pf,
                                              const typename Word<ES>::T* s,
                                              typename Word<ES>::T* outBase) {
#pragma unroll
  for (int i = 0; i < PF; ++i) {
    const int w = threadIdx.x + i * TILE_THREADS;
    if (w < p.nOut) storeUnit<ES, SV>(s, pf.idx[i], outBase + pf.off[i]);
  }
  const int tv = opaque(threadIdx.x);
#pragma unroll 4
  for (int w = tv + PF * TILE_THREADS; w < p.nOut; w += TILE_THREADS)
    storeUnit<ES, SV>(s, loadSmIdx<SV>(stSm, w), outBase + stOff[w]);
}

// Register-staged pipeline: load units go global -> registers -> shared
// memory; the next tile's loads are issued before the current tile's
// stores.  Two shared data buffers, one barrier per tile.
template <int ES, int LV, int SV, int NL>
__global__ void __launch_bounds__(TILE_THREADS)
tileKernelReg(const __grid_constant__ TileParams p, const typename Word<ES>::T* __restrict__ in,
              typename Word<ES>::T* __restrict__ out) {
  using T = typename Word<ES>::T;
  using LT = typename Word<ES * LV>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const TileTables tt = buildTileTables(p, smraw);
  T* sm = reinterpret_cast<T*>(tt.data);

  uint32_t tile = blockIdx.x;
  if (tile >= p.numTiles) return;
  long long bin, bout;
  decodeTile(p, tile, bin, bout);

  LT v[NL];
  auto load = [&](long long base) {
    const int tv = opaque(threadIdx.x);
#pragma unroll
    for (int k = 0; k < NL; ++k) {
      const int u = tv + k * TILE_THREADS;
      if (u < p.nIn) v[k] = *reinterpret_cast<const LT*>(in + base + tt.ldOff[u]);
    }
  };
  load(bin);

  int buf = 0;
  for (;;) {
    T* s = sm + buf * p.smStride;
    {
      const int tv = opaque(threadIdx.x);
#pragma unroll
      for (int k = 0; k < NL; ++k) {
        const int u = tv + k * TILE_THREADS;
        if (u < p.nIn) *reinterpret_cast<LT*>(s + smemIndex(p, u * LV)) = v[k];
      }
    }
    __syncthreads();
    const uint32_t next = tile + gridDim.x;
    const bool more = next < p.numTiles;
    long long nbin = 0, nbout = 0;
    if (more) {
      decodeTile(p, next, nbin, nbout);
      load(nbin);
    }
    storeTile<ES, SV>(p, tt.stOff, tt.stSm, s, out + bout);
    if (!more) break;
    tile = next;
    bin = nbin;
    bout = nbout;
    buf ^= 1;
  }
}

// cp.async pipeline (16-byte load units only): load units are copied from
// global straight into a TILE_STAGES-deep ring of shared buffers, so
// TILE_STAGES - 1 tiles of loads are in flight while one tile is stored.
template <int ES, int LV, int SV>
__global__ void __launch_bounds__(TILE_THREADS)
tileKernelAsync(const __grid_constant__ TileParams p, const typename Word<ES>::T* __restrict__ in,
                typename Word<ES>::T* __restrict__ out) {
  static_assert(ES * LV == 16, "cp.async pipeline moves 16-byte units");
  using T = typename Word<ES>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  const TileTables tt = buildTileTables(p, smraw);
  T* sm = reinterpret_cast<T*>(tt.data);
  const uint32_t smBase = (uint32_t)__cvta_generic_to_shared(tt.data);

  const uint32_t first = blockIdx.x;
  if (first >= p.numTiles) return;
  const uint32_t G = gridDim.x;
  const uint32_t nMine = (p.numTiles - first + G - 1) / G;

  auto issue = [&](uint32_t i) {
    long long bin, bout;
    decodeTile(p, first + i * G, bin, bout);
    const T* src = in + bin;
    const uint32_t dst = smBase + (uint32_t)((i % TILE_STAGES) * p.smStride) * ES;
    const int tv = opaque(threadIdx.x);
#pragma unroll 4
    for (int u = tv; u < p.nIn; u += TILE_THREADS)
      cpAsync16(dst + (uint32_t)smemIndex(p, u * LV) * ES, src + tt.ldOff[u]);
  };

#pragma unroll
  for (int s = 0; s < TILE_STAGES - 1; ++s) {
    if ((uint32_t)s < nMine) issue(s);
    cpAsyncCommit();
  }
  for (uint32_t i = 0; i < nMine; ++i) {
    cpAsyncWait<TILE_STAGES - 2>();
    __syncthreads();
    // The stage refilled here was last read in iteration i - 1, which every
    // thread has finished (barrier above).
    if (i + TILE_STAGES - 1 < nMine) issue(i + TILE_STAGES - 1);
    cpAsyncCommit();
    long long bin, bout;
    decodeTile(p, first + i * G, bin, bout);
    storeTile<ES, SV>(p, tt.stOff, tt.stSm, sm + (i % TILE_STAGES) * p.smStride, out + bout);
  }
  cpAsyncWait<0>();
}

// p + i * scale bytes.  With a scale the compiler cannot see (opaque), the
// offset is one wide integer multiply-add on the FMA pipe instead of a
// sign extension and a shift-add pair on the ALU pipe, which the grouped
// kernel's narrow units would otherwise saturate.
template <typename P>
__device__ __forceinline__ P* offsetBytes(P* p, int i, int scale) {
  using B = typename std::conditional<std::is_const<P>::value, const unsigned char,
                                      unsigned char>::type;
  return reinterpret_cast<P*>(reinterpret_cast<B*>(p) + (long long)i * scale);
}

// cp.async of one unit, issued only where live: the guard is a predicate on
// the instruction rather than a branch around it (the compiler cannot
// if-convert inline assembly, so a guarded asm costs a branch per slot).
template <int BYTES, int PF>
__device__ __forceinline__ void cpAsyncUnitIf(bool live, uint32_t dst, const void* src) {
  static_assert(BYTES == 4 || BYTES == 8 || BYTES == 16, "cp.async unit");
  static_assert(PF == 0 || PF == 256, "L2 prefetch size");
#define LT_CP_ASYNC_IF(OP, SIZE)                                                             \
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %2, 0;\n @p " OP " [%0], [%1], " SIZE \
               ";\n}\n" ::"r"(dst),                                                          \
               "l"(src), "r"((int)live)                                                      \
               : "memory")
  if constexpr (BYTES == 16 && PF == 256)
    LT_CP_ASYNC_IF("cp.async.cg.shared.global.L2::256B", "16");
  else if constexpr (BYTES == 16)
    LT_CP_ASYNC_IF("cp.async.cg.shared.global", "16");
  else if constexpr (BYTES == 8 && PF == 256)
    LT_CP_ASYNC_IF("cp.async.ca.shared.global.L2::256B", "8");
  else if constexpr (BYTES == 8)
    LT_CP_ASYNC_IF("cp.async.ca.shared.global", "8");
  else if constexpr (PF == 256)
    LT_CP_ASYNC_IF("cp.async.ca.shared.global.L2::256B", "4");
  else
    LT_CP_ASYNC_IF("cp.async.ca.shared.global", "4");
#undef LT_CP_ASYNC_IF
}

// Kernel parameters of a table-free tile (NTR rank class, NI load rank class;
// the host builds them per launch from the plan's TileParams).
template <int ES, int LV, int SV, int NL, int NI, int NTR>
struct FlatParams {
  static constexpr int NS = (NL * LV + SV - 1) / SV;  // store slots
  int nIn, nOut, tileVol;
  int padShiftB;     // shared byte address of byte x: x + (x >> padShiftB) * padBytes
  int padBytes;
  int ldSmStep;      // padded shared bytes between two load slots
  int elemStep;      // shared bytes between the elements of a store unit
  int storeStraddle; // a store unit's elements may cross output tile rank 0
  int segLen, testExtraTx;  // as in TileParams
  uint32_t statusTag;
  LoadSlots<NL, NI> ld;
  StoreSlots<NS, NTR> st;
  int nGR;           // grid ranks, as in TileParams
  static constexpr int NG = gridCapacity(NTR);
  FastDiv grDiv[NG];
  long long grSin[NG], grSout[NG], grLastIn[NG], grLastOut[NG];
};

// tp.nGR <= gridCapacity(NTR), as storeRankClass gives.
template <int ES, int LV, int SV, int NL, int NI, int NTR>
FlatParams<ES, LV, SV, NL, NI, NTR> makeFlatParams(const TileParams& tp) {
  FlatParams<ES, LV, SV, NL, NI, NTR> p;
  p.nIn = tp.nIn;
  p.nOut = tp.nOut;
  p.tileVol = tp.tileVol;
  // in-tile byte indices are below 2^20: shift 31 gives no padding
  p.padShiftB = tp.padShift >= PAD_NONE ? 31 : tp.padShift + (ES == 4 ? 2 : ES == 8 ? 3 : 4);
  p.padBytes = ES << tp.padLog;
  constexpr int B = TILE_THREADS * LV;  // a multiple of every padding period (2^2 .. 2^8)
  p.ldSmStep = B * ES + (tp.padShift >= PAD_NONE ? 0 : (B >> tp.padShift) * p.padBytes);
  p.elemStep = tp.toInTile[0] * ES;
  p.storeStraddle = tp.storeStraddle;
  p.segLen = tp.segLen;
  p.testExtraTx = tp.testExtraTx;
  p.statusTag = tp.statusTag;
  makeLoadSlots(tp, p.ld);
  makeStoreSlots(tp, ES, p.st);
  p.nGR = tp.nGR;
  for (int g = 0; g < tp.nGR; ++g) {
    p.grDiv[g] = tp.grDiv[g];
    p.grSin[g] = tp.grSin[g];
    p.grSout[g] = tp.grSout[g];
    p.grLastIn[g] = tp.grLastIn[g];
    p.grLastOut[g] = tp.grLastOut[g];
  }
  return p;
}

template <typename P>
__device__ __forceinline__ uint32_t padByte(const P& p, uint32_t x) {
  return x + (x >> p.padShiftB) * (uint32_t)p.padBytes;
}

// A thread's part of the store addresses, decoded while the loads are in
// flight.
template <int NTR>
struct StoreThread {
  uint32_t off, j;
  int d[NTR - 1];
};

// Store phase of the table-free flat and bulk-copy kernels.  Slots go in
// chunks of four, whole chunks without a guard.
template <int ES, int LV, int SV, int NL, int NI, int NTR>
__device__ __forceinline__ void storeTileSlots(const FlatParams<ES, LV, SV, NL, NI, NTR>& p,
                                               const StoreThread<NTR>& t,
                                               const unsigned char* s,
                                               typename Word<ES>::T* outBase) {
  using T = typename Word<ES>::T;
  using ST = typename Word<ES * SV>::T;
  constexpr int NS = FlatParams<ES, LV, SV, NL, NI, NTR>::NS;
  constexpr int CH = NS < 4 ? NS : 4;
  const int wMax = p.nOut - (int)threadIdx.x;
  const int esR = opaque(ES);
  auto slot = [&](int k) {
    uint32_t off, j;
    storeSlotOffset<NS, NTR>(p.st, k, t.off, t.j, t.d, off, j);
    T e[SV];
    e[0] = *reinterpret_cast<const T*>(s + padByte(p, j));
    if constexpr (SV > 1) {
      if (!p.storeStraddle) {
#pragma unroll
        for (int m = 1; m < SV; ++m)
          e[m] = *reinterpret_cast<const T*>(s + padByte(p, j + (uint32_t)(m * p.elemStep)));
      } else {
#pragma unroll
        for (int m = 1; m < SV; ++m) {
          StoreThread<NTR> u;
          storeThreadOffset<NS, NTR>(
              p.st, (uint32_t)((threadIdx.x + k * TILE_THREADS) * SV + m), u.d, u.off, u.j);
          e[m] = *reinterpret_cast<const T*>(s + padByte(p, u.j));
        }
      }
    }
    ST v;
    __builtin_memcpy(&v, e, sizeof(ST));
    *reinterpret_cast<ST*>(offsetBytes(outBase, (int)off, esR)) = v;
  };
#pragma unroll
  for (int k0 = 0; k0 < NS; k0 += CH) {
    if ((k0 + CH) * TILE_THREADS <= p.nOut) {
#pragma unroll
      for (int i = 0; i < CH; ++i) slot(k0 + i);
    } else if (k0 * TILE_THREADS < p.nOut) {
#pragma unroll
      for (int i = 0; i < CH; ++i)
        if ((k0 + i) * TILE_THREADS < wMax) slot(k0 + i);
    }
  }
}

// Flat pipeline, tiles of at most ARITH_MAX_NTR ranks: one tile per CTA and
// no persistent loop, so the hardware block scheduler streams tiles through
// the SMs in order.  Unit addresses come from the slot sums (slots.h).
template <int ES, int LV, int SV, int NL, int NI, int NTR>
__global__ void __launch_bounds__(TILE_THREADS)
tileKernelFlat(const __grid_constant__ FlatParams<ES, LV, SV, NL, NI, NTR> p,
               const typename Word<ES>::T* __restrict__ in, typename Word<ES>::T* __restrict__ out) {
  using LT = typename Word<ES * LV>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  dependencyRelease();
  long long bin, bout;
  decodeTile(p, blockIdx.x, bin, bout);
  const uint32_t jT = threadIdx.x * LV;
  int d[NI - 1];
  const uint32_t offT = loadThreadOffset<NL, NI>(p.ld, jT, d);
  const auto* src = in + bin;
  const int esR = opaque(ES);
  const int uMax = p.nIn - (int)threadIdx.x;
  const uint32_t dst0 = padByte(p, jT * ES);
  auto source = [&](int k) {
    return offsetBytes(src, (int)loadSlotOffset<NL, NI>(p.ld, k, offT, d), esR);
  };
  StoreThread<NTR> t;
  dependencyWait();
  if constexpr (NL >= flatAsyncMinNL<ES>()) {
    // many load units per thread: cp.async straight into shared memory
    // instead of NL data registers per thread
    const uint32_t sBase = (uint32_t)__cvta_generic_to_shared(smraw) + dst0;
    constexpr int CH = 4;
#pragma unroll
    for (int k0 = 0; k0 < NL; k0 += CH) {
      if ((k0 + CH) * TILE_THREADS <= p.nIn) {
#pragma unroll
        for (int k = k0; k < k0 + CH; ++k)
          cpAsyncUnit<ES * LV>(sBase + (uint32_t)(k * p.ldSmStep), source(k));
      } else if (k0 * TILE_THREADS < p.nIn) {
#pragma unroll
        for (int k = k0; k < k0 + CH; ++k)
          cpAsyncUnitIf<ES * LV, 0>(k * TILE_THREADS < uMax, sBase + (uint32_t)(k * p.ldSmStep),
                                    source(k));
      }
    }
    storeThreadOffset<FlatParams<ES, LV, SV, NL, NI, NTR>::NS, NTR>(p.st, threadIdx.x * SV, t.d,
                                                                    t.off, t.j);
    cpAsyncWaitAll();
  } else {
    LT v[NL];
#pragma unroll
    for (int k = 0; k < NL; ++k)
      if (k * TILE_THREADS < uMax) v[k] = ldGlobal<ES * LV>(source(k));
    storeThreadOffset<FlatParams<ES, LV, SV, NL, NI, NTR>::NS, NTR>(p.st, threadIdx.x * SV, t.d,
                                                                    t.off, t.j);
#pragma unroll
    for (int k = 0; k < NL; ++k)
      if (k * TILE_THREADS < uMax)
        *reinterpret_cast<LT*>(smraw + dst0 + (uint32_t)(k * p.ldSmStep)) = v[k];
  }
  __syncthreads();
  storeTileSlots<ES, LV, SV, NL, NI, NTR>(p, t, smraw, out + bout);
}

// Span loads (slots.h): the flat kernel for 4-byte elements whose input only
// allows element units.  Each run comes as the 16-byte blocks around it, with the
// neighbours' bytes that share its first and last block (a run that fills one
// block less reads one more; all of them lie inside the tensor).  The block at
// the tensor's either end that reaches past it is read element by element.
// A quarter of the load instructions and 9 sectors instead of 10 per 256 bytes;
// what bounds it then are the stores and the partly written sectors of output
// runs.  float32 (127, 63, 65, 33) perm (3, 1, 2, 0): 29.1 -> 28.4 us; (256, 128,
// 512) perm (2, 1, 0) one element off alignment: 26.9 -> 25.6; (142010, 2, 12, 38)
// perm (3, 1, 0, 2): 189.9 -> 174.7.  One bulk copy per run instead: 31.6 us for the
// first, whose runs each take a copy's issue and the mbarrier's wait.
template <int SV, int NL, int NI, int NTR>
struct SpanParams {
  FlatParams<SPAN_ES, 1, SV, NL, NI, NTR> flat;
  StoreSlots<spanSlots(NL), NI> blocks;
  int units;
  long long inBytes;  // the tensor's
};

template <int SV, int NL, int NI, int NTR>
SpanParams<SV, NL, NI, NTR> makeSpanParams(const TileParams& tp, const SpanLayout& L,
                                           long long inBytes) {
  SpanParams<SV, NL, NI, NTR> p;
  p.flat = makeFlatParams<SPAN_ES, 1, SV, NL, NI, NTR>(tp);
  p.flat.padShiftB = 31;  // rows have their own steps
  p.flat.elemStep = L.stepJ[0];
  makeStoreSlots(tp, L.stepJ, p.flat.st);
  makeSpanSlots(L, p.blocks);
  p.units = L.units;
  p.inBytes = inBytes;
  return p;
}

template <int SV, int NL, int NI, int NTR>
__global__ void __launch_bounds__(TILE_THREADS)
tileKernelSpan(const __grid_constant__ SpanParams<SV, NL, NI, NTR> q,
               const typename Word<SPAN_ES>::T* __restrict__ in,
               typename Word<SPAN_ES>::T* __restrict__ out) {
  constexpr int ES = SPAN_ES, NLS = spanSlots(NL);
  using Flat = FlatParams<ES, 1, SV, NL, NI, NTR>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const Flat& p = q.flat;
  dependencyRelease();
  long long bin, bout;
  decodeTile(p, blockIdx.x, bin, bout);
  const unsigned char* first = reinterpret_cast<const unsigned char*>(in);
  const unsigned char* end = first + q.inBytes;
  const unsigned char* base = first + bin * ES;
  const uint32_t start = (uint32_t)(reinterpret_cast<uintptr_t>(base) & 15);
  const uint32_t sTile = (uint32_t)__cvta_generic_to_shared(smraw) + start;
  int d[NI - 1];
  uint32_t offT, jT;
  storeThreadOffset<NLS, NI>(q.blocks, threadIdx.x, d, offT, jT);
  const int esR = opaque(ES);
  dependencyWait();
#pragma unroll
  for (int k = 0; k < NLS; ++k) {
    if (k * TILE_THREADS + (int)threadIdx.x < q.units) {
      uint32_t off, j;
      storeSlotOffset<NLS, NI>(q.blocks, k, offT, jT, d, off, j);
      const unsigned char* a = reinterpret_cast<const unsigned char*>(
          reinterpret_cast<uintptr_t>(offsetBytes(base, (int)off, esR)) & ~(uintptr_t)15);
      const uint32_t sa = (sTile + j) & ~15u;
      if (a >= first && a + 16 <= end) {
        cpAsyncUnit<16>(sa, a);
      } else {
#pragma unroll 1
        for (int i = 0; i < 16; i += ES)
          if (a + i >= first && a + i + ES <= end) cpAsyncUnit<ES>(sa + i, a + i);
      }
    }
  }
  StoreThread<NTR> t;
  storeThreadOffset<Flat::NS, NTR>(p.st, threadIdx.x * SV, t.d, t.off, t.j);
  cpAsyncWaitAll();
  __syncthreads();
  storeTileSlots<ES, 1, SV, NL, NI, NTR>(p, t, smraw + start, out + bout);
}

// The flat pipeline for larger tiles: the offset tables were written at plan
// time and are read from device memory (L1/L2-resident: every CTA of the
// launch reads the same few kilobytes).
template <int ES, int LV, int SV, int NL>
__global__ void __launch_bounds__(TILE_THREADS)
tileKernelTables(const __grid_constant__ TileParams p, const typename Word<ES>::T* __restrict__ in,
                 typename Word<ES>::T* __restrict__ out, const int* __restrict__ ldOff,
                 const int* __restrict__ stOff, const unsigned short* __restrict__ stSm) {
  using T = typename Word<ES>::T;
  using LT = typename Word<ES * LV>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  T* s = reinterpret_cast<T*>(smraw);
  long long bin, bout;
  decodeTile(p, blockIdx.x, bin, bout);
  // store units per thread: nOut <= NL * TILE_THREADS * LV / SV; up to two
  // are prefetched, except where the register pipeline already holds
  // NL >= 4 data words (measured slower there)
  constexpr int NS = (NL * LV + SV - 1) / SV;
  constexpr int PF_MAX = (NL >= flatAsyncMinNL<ES>() || NL < 4) ? 2 : 0;
  constexpr int PF = NS < PF_MAX ? NS : PF_MAX;
  StorePrefetch<SV, PF> pf;
  if constexpr (NL >= flatAsyncMinNL<ES>()) {
    const uint32_t sBase = (uint32_t)__cvta_generic_to_shared(s);
#pragma unroll
    for (int k = 0; k < NL; ++k) {
      const int u = threadIdx.x + k * TILE_THREADS;
      if (u < p.nIn)
        cpAsyncUnit<ES * LV>(sBase + (uint32_t)smemIndex(p, u * LV) * ES, in + bin + __ldg(ldOff + u));
    }
    pf.load(p, stOff, stSm);
    cpAsyncWaitAll();
  } else {
    LT v[NL];
#pragma unroll
    for (int k = 0; k < NL; ++k) {
      const int u = threadIdx.x + k * TILE_THREADS;
      if (u < p.nIn) v[k] = *reinterpret_cast<const LT*>(in + bin + __ldg(ldOff + u));
    }
    pf.load(p, stOff, stSm);
#pragma unroll
    for (int k = 0; k < NL; ++k) {
      const int u = threadIdx.x + k * TILE_THREADS;
      if (u < p.nIn) *reinterpret_cast<LT*>(s + smemIndex(p, u * LV)) = v[k];
    }
  }
  __syncthreads();
  storeTileFlat<ES, SV>(p, stOff, stSm, pf, s, out + bout);
}

// mbarrier and bulk-copy primitives (PTX ISA: mbarrier, cp.async.bulk).
__device__ __forceinline__ void mbarInit(uint32_t mb, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(mb), "r"(count) : "memory");
}

// Makes an initialised mbarrier visible to the asynchronous proxy (the bulk
// copies that complete on it).
__device__ __forceinline__ void mbarInitFence() {
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

__device__ __forceinline__ void mbarArriveExpectTx(uint32_t mb, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(mb), "r"(bytes)
               : "memory");
}

__device__ __forceinline__ bool mbarTryWait(uint32_t mb, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(mb), "r"(parity)
      : "memory");
  return ok != 0;
}

// One bulk copy global -> shared (16-byte aligned addresses, size a
// multiple of 16) that completes `bytes` transactions on mbarrier mb.
__device__ __forceinline__ void bulkLoad(uint32_t dst, const void* src, uint32_t bytes,
                                         uint32_t mb) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::
          "r"(dst),
      "l"(src), "r"(bytes), "r"(mb)
      : "memory");
}

__device__ __forceinline__ unsigned long long globalTimerNs() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;\n" : "=l"(t));
  return t;
}

// Waits for phase `parity` of mbarrier mb for at most limitNs nanoseconds.
__device__ __forceinline__ bool mbarWaitBounded(uint32_t mb, uint32_t parity,
                                                unsigned long long limitNs) {
  if (mbarTryWait(mb, parity)) return true;
  const unsigned long long t0 = globalTimerNs();
  for (;;) {
    if (mbarTryWait(mb, parity)) return true;
    if (globalTimerNs() - t0 > limitNs) return false;
  }
}

constexpr unsigned long long BULK_WAIT_NS = 1000000000ull;  // 1 s

// Bulk-copy pipeline: the flat kernel with its load phase as bulk copies.
// The tile's input-order elements form segments of p.segLen elements, each
// contiguous in global memory (inside one input run) and in shared memory
// (between two padding gaps); segment k starts at tile element k * segLen,
// whose global offset is the load-unit table entry of that element.  The
// CTA's threads issue one cp.async.bulk per segment (no per-unit
// instruction, no data registers), all completing on one mbarrier that
// thread 0 arms with the tile's byte count; every thread then waits on it
// and the stores run as in the flat pipeline.  The wait is bounded: after
// BULK_WAIT_NS without completion the CTA writes the plan's tag p.statusTag
// to *status, waits once more (bounded) for its copies in flight, and
// returns without storing.
// Issue half of the bulk-copy kernels: `off` gives a tile element's global
// input offset, `pad` its shared byte address.  Returns after the copies are
// issued and the mbarrier is armed.
template <int ES, typename P, typename Off, typename Pad>
__device__ __forceinline__ void bulkIssue(const P& p, const typename Word<ES>::T* src,
                                          uint32_t sBase, uint32_t mb, Off off, Pad pad) {
  if (threadIdx.x == 0) {
    mbarInit(mb, 1);
    mbarInitFence();
  }
  __syncthreads();
  dependencyWait();
  const int L = p.segLen;
  const int nSeg = p.tileVol / L;
  const uint32_t segBytes = (uint32_t)(L * ES);
  for (int k = threadIdx.x; k < nSeg; k += TILE_THREADS) {
    const int j0 = k * L;
    bulkLoad(sBase + pad(j0), src + off(j0), segBytes, mb);
  }
  if (threadIdx.x == 0) mbarArriveExpectTx(mb, (uint32_t)nSeg * segBytes + (uint32_t)p.testExtraTx);
}

// Wait half: false after the time limit, with the plan's tag in *status.
template <typename P>
__device__ __forceinline__ bool bulkWait(const P& p, uint32_t mb, unsigned* status) {
  if (mbarWaitBounded(mb, 0, BULK_WAIT_NS)) return true;
  if (threadIdx.x == 0) atomicExch(status, p.statusTag);
  mbarWaitBounded(mb, 0, BULK_WAIT_NS);  // copies in flight write this CTA's shared memory
  return false;
}

template <int ES, int LV, int SV, int NL, int NI, int NTR>
__global__ void __launch_bounds__(TILE_THREADS)
tileKernelBulk(const __grid_constant__ FlatParams<ES, LV, SV, NL, NI, NTR> p,
               const typename Word<ES>::T* __restrict__ in, typename Word<ES>::T* __restrict__ out,
               unsigned* status) {
  static_assert(ES * LV == 16, "bulk copies need 16-byte load units");
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(8) unsigned long long bar;
  dependencyRelease();
  long long bin, bout;
  decodeTile(p, blockIdx.x, bin, bout);
  const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&bar);
  bulkIssue<ES>(
      p, in + bin, (uint32_t)__cvta_generic_to_shared(smraw), mb,
      [&](int j) {
        int d[NI - 1];
        return (int)loadThreadOffset<NL, NI>(p.ld, (uint32_t)j, d);
      },
      [&](int j) { return padByte(p, (uint32_t)(j * ES)); });
  StoreThread<NTR> t;
  storeThreadOffset<FlatParams<ES, LV, SV, NL, NI, NTR>::NS, NTR>(p.st, threadIdx.x * SV, t.d,
                                                                  t.off, t.j);
  if (!bulkWait(p, mb, status)) return;
  storeTileSlots<ES, LV, SV, NL, NI, NTR>(p, t, smraw, out + bout);
}

// Bulk copies with offset tables (tiles of more than ARITH_MAX_NTR ranks).
template <int ES, int LV, int SV, int NL>
__global__ void __launch_bounds__(TILE_THREADS)
tileKernelBulkTables(const __grid_constant__ TileParams p,
                     const typename Word<ES>::T* __restrict__ in,
                     typename Word<ES>::T* __restrict__ out, const int* __restrict__ ldOff,
                     const int* __restrict__ stOff, const unsigned short* __restrict__ stSm,
                     unsigned* status) {
  static_assert(ES * LV == 16, "bulk copies need 16-byte load units");
  using T = typename Word<ES>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ __align__(8) unsigned long long bar;
  T* s = reinterpret_cast<T*>(smraw);
  long long bin, bout;
  decodeTile(p, blockIdx.x, bin, bout);
  const uint32_t mb = (uint32_t)__cvta_generic_to_shared(&bar);
  bulkIssue<ES>(
      p, in + bin, (uint32_t)__cvta_generic_to_shared(s), mb,
      [&](int j) { return __ldg(ldOff + j / LV); },
      [&](int j) { return (uint32_t)smemIndex(p, j) * ES; });
  constexpr int NS = (NL * LV + SV - 1) / SV;
  constexpr int PF = NS < 2 ? NS : 2;
  StorePrefetch<SV, PF> pf;
  pf.load(p, stOff, stSm);
  if (!bulkWait(p, mb, status)) return;
  storeTileFlat<ES, SV>(p, stOff, stSm, pf, s, out + bout);
}

template <int BYTES>
__device__ __forceinline__ typename Word<BYTES>::T ldShared(uint32_t addr) {
  typename Word<BYTES>::T v;
  if constexpr (BYTES == 4) {
    asm volatile("ld.shared.b32 %0, [%1];\n" : "=r"(v) : "r"(addr));
  } else if constexpr (BYTES == 8) {
    asm volatile("ld.shared.v2.b32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(addr));
  } else {
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "r"(addr));
  }
  return v;
}

template <int BYTES>
__device__ __forceinline__ void stShared(uint32_t addr, const typename Word<BYTES>::T& v) {
  if constexpr (BYTES == 4) {
    asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(addr), "r"(v) : "memory");
  } else if constexpr (BYTES == 8) {
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(addr), "r"(v.x), "r"(v.y) : "memory");
  } else {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(addr), "r"(v.x), "r"(v.y),
                 "r"(v.z), "r"(v.w)
                 : "memory");
  }
}

// Grouped flat kernel: CTA b moves one tile of tensor tileTensor[b] of a
// bucket; the tile list gives the tensor and the tile's corner offsets, the
// tensor's descriptor its pointers and run tables.  Unit
// offsets come from the run split (GroupTensor): a small table entry per
// run plus the position inside the run, so the tables stay in L1 even when
// consecutive CTAs belong to different tensors; when they are small enough
// the store-side tables are copied into shared memory with the data.  The load
// units are staged in registers or, with ASYNC, copied with cp.async straight
// into shared memory (no data registers, so more CTAs fit an SM).  Every
// access stays inside the member's input and output tensors.
//
// Index arithmetic is kept off the ALU pipe where it can be: with element-
// size units the kernel does little else, and integer adds, shifts and
// compares issue at half the rate of multiply-adds.  Load slot k of a thread
// starts at tile element jT + k * B (B = TILE_THREADS * LV).  Padding puts
// 2^padLog elements after every 2^padShift, with padShift <= 8 <= log2(B) or
// padShift = 31 (none), so slot k's padded index is padT + k * padStep: one
// multiply-add per slot.  Byte offsets are multiply-adds by a scale the
// compiler cannot fold into shifts.
template <int ES, int LV, int SV, int NL, bool ASYNC>
__device__ __forceinline__ void groupTileBody(const GroupTensor* __restrict__ g, long long bin,
                                              long long bout) {
  using T = typename Word<ES>::T;
  using LT = typename Word<ES * LV>::T;
  using ST = typename Word<ES * SV>::T;
  extern __shared__ __align__(16) unsigned char smraw[];
  // shared memory: [store-side run tables, when staged][tile data]
  const int tabBytes = g->tabBytes;
  T* s = reinterpret_cast<T*>(smraw + tabBytes);
  const T* in = reinterpret_cast<const T*>(g->in) + bin;
  T* out = reinterpret_cast<T*>(g->out) + bout;
  const int* ldRow = g->ldRow;
  const RunDiv inRun = g->inRun;
  const int nIn = g->nIn, nOut = g->nOut, padShift = g->padShift, padLog = g->padLog;
  const uint32_t sBase = (uint32_t)__cvta_generic_to_shared(s);
  const int esR = opaque(ES);
  const int padMul = 1 << padLog;
  {
    constexpr int B = TILE_THREADS * LV;
    const int jT = threadIdx.x * LV;
    const int bR = opaque(B);
    const uint32_t dst0 = sBase + (uint32_t)((jT + (jT >> padShift) * padMul) * esR);
    const int stepBytes = (B + (B >> padShift) * padMul) * esR;
    const int uMax = nIn - threadIdx.x;  // slot k is live while k * TILE_THREADS < uMax
    const int inD = (int)inRun.d;
    const int four = opaque(4);
    const int jT1 = jT + 1;
    const T* inM1 = in - 1;  // indexed by a + 1
    const int ldStepB = g->ldStepBytes;
    // STEP: input runs evenly spaced (no table read on the load path)
    auto loadAll = [&](auto step) {
      constexpr bool STEP = decltype(step)::value;
      auto unitSrc = [&](int k) {
        // j + 1 = k * B + jT + 1; run r = j / inRun, a + 1 = j + 1 - r * inRun
        const int j1 = k * bR + jT1;
        const uint32_t r = __umulhi((uint32_t)j1, inRun.mul);
        const int a1 = j1 - (int)r * inD;
        const T* runBase;
        if constexpr (STEP)
          runBase = offsetBytes(inM1, (int)r, ldStepB);
        else
          runBase = offsetBytes(inM1, __ldg(offsetBytes(ldRow, (int)r, four)), esR);
        return reinterpret_cast<const LT*>(offsetBytes(runBase, a1, esR));
      };
      if constexpr (ASYNC) {
#pragma unroll
        for (int k = 0; k < NL; ++k)
          if constexpr (STEP)  // the source is arithmetic only: predicate the copy
            cpAsyncUnitIf<ES * LV, LT_GROUP_L2_PREFETCH>(k * TILE_THREADS < uMax, dst0 + (uint32_t)(k * stepBytes),
                                   unitSrc(k));
          else if (k * TILE_THREADS < uMax)  // a dead slot's run would index past ldRow
            cpAsyncUnit<ES * LV>(dst0 + (uint32_t)(k * stepBytes), unitSrc(k));
        cpAsyncWaitAll();
      } else {
        LT v[NL];
#pragma unroll
        for (int k = 0; k < NL; ++k)
          if (k * TILE_THREADS < uMax) v[k] = ldGlobal<ES * LV>(unitSrc(k));
#pragma unroll
        for (int k = 0; k < NL; ++k)
          if (k * TILE_THREADS < uMax) stShared<ES * LV>(dst0 + (uint32_t)(k * stepBytes), v[k]);
      }
    };
    // the tile list, descriptor and tables are written once, at group creation
    // (which synchronises), so only the tensors' data waits for the stream
    dependencyWait();
    if (ldStepB >= 0)
      loadAll(std::true_type{});
    else
      loadAll(std::false_type{});
  }
  if (tabBytes > 0) {
    // the store-side tables (outRows and smRun are contiguous, 16-byte
    // aligned) into shared memory, in flight with the data loads
    const uint32_t tBase = (uint32_t)__cvta_generic_to_shared(smraw);
    const unsigned char* src = reinterpret_cast<const unsigned char*>(g->outRows);
    for (int c = threadIdx.x; c < (tabBytes >> 4); c += TILE_THREADS)
      cpAsyncUnit<16>(tBase + 16u * c, src + 16 * c);
    cpAsyncWaitAll();
  }
  __syncthreads();
  const RunDiv outRun = g->outRun;
  const int outD = (int)outRun.d;
  const int qT1 = threadIdx.x * SV + 1;
  T* outM1 = out - 1;  // indexed by a + 1
  const int bQ = opaque(TILE_THREADS * SV);
  const int wMax = nOut - threadIdx.x;  // store slot i is live while i * TILE_THREADS < wMax
  const int padBytes = padMul * esR;
  // shared address of (unpadded) tile element x
  auto smAddr = [&](int x) { return sBase + (uint32_t)(x * esR + (x >> padShift) * padBytes); };
  // nOut <= NL * TILE_THREADS * LV / SV
  constexpr int NS = (NL * LV + SV - 1) / SV;
  constexpr int UNROLL = NS <= 16 ? NS : 8;
  // ROWS: output runs evenly spaced (no outRows read); POS: positions of a
  // run evenly spaced in the tile (no smRun read)
  const int outStepB = g->outStepBytes, rowSmStep = g->rowSmStep, smStep = g->smStep;
  auto storeAll = [&](auto rowsStepped, auto posStepped, const int2* outRows, const int* smRun) {
    constexpr bool ROWS = decltype(rowsStepped)::value;
    constexpr bool POS = decltype(posStepped)::value;
#pragma unroll UNROLL
    for (int i = 0; i < NS; ++i) {
      if (i * TILE_THREADS < wMax) {
        const int q1 = i * bQ + qT1;  // q + 1
        const uint32_t r = __umulhi((uint32_t)q1, outRun.mul);
        const int a1 = q1 - (int)r * outD;  // a + 1
        const int a = a1 - 1;
        ST* dst;
        int jb;
        if constexpr (ROWS) {
          dst = reinterpret_cast<ST*>(offsetBytes(offsetBytes(outM1, a1, esR), (int)r, outStepB));
          jb = (int)r * rowSmStep;
        } else {
          const int2 row = outRows[r];
          dst = reinterpret_cast<ST*>(offsetBytes(offsetBytes(outM1, a1, esR), row.x, esR));
          jb = row.y;
        }
        if constexpr (SV == 1) {
          if constexpr (POS)
            *dst = ldShared<ES>(smAddr(a * smStep + jb));
          else
            *dst = ldShared<ES>(smAddr(jb + smRun[a]));
        } else {
          T e[SV];
          if constexpr (POS) {
            const int x0 = a * smStep + jb;
#pragma unroll
            for (int c = 0; c < SV; ++c) e[c] = ldShared<ES>(smAddr(x0 + c * smStep));
          } else if constexpr (SV == 2) {
            const int2 jr = *reinterpret_cast<const int2*>(smRun + a);
            e[0] = ldShared<ES>(smAddr(jb + jr.x));
            e[1] = ldShared<ES>(smAddr(jb + jr.y));
          } else {
            const int4 jr = *reinterpret_cast<const int4*>(smRun + a);
            e[0] = ldShared<ES>(smAddr(jb + jr.x));
            e[1] = ldShared<ES>(smAddr(jb + jr.y));
            e[2] = ldShared<ES>(smAddr(jb + jr.z));
            e[3] = ldShared<ES>(smAddr(jb + jr.w));
          }
          ST val;
          __builtin_memcpy(&val, e, sizeof(ST));
          *dst = val;
        }
      }
    }
  };
  // tables that are read come from shared memory when staged, else from
  // device memory (two instantiations, so shared reads stay shared loads)
  auto withTables = [&](auto rowsStepped, auto posStepped) {
    if (tabBytes > 0) {
      const int* t = reinterpret_cast<const int*>(smraw);
      storeAll(rowsStepped, posStepped, reinterpret_cast<const int2*>(smraw), t + g->smRunOff);
    } else {
      storeAll(rowsStepped, posStepped, g->outRows, g->smRun);
    }
  };
  using Yes = std::true_type;
  using No = std::false_type;
  if (outStepB >= 0) {
    if (smStep >= 0)
      storeAll(Yes{}, Yes{}, nullptr, nullptr);
    else
      withTables(Yes{}, No{});
  } else {
    if (smStep >= 0)
      withTables(No{}, Yes{});
    else
      withTables(No{}, No{});
  }
}

// Tile `index` of a bucket: its tensor's descriptor and its corner offsets.
__device__ __forceinline__ const GroupTensor* groupTile(const GroupTensor* __restrict__ tens,
                                                        const GroupTile* __restrict__ tiles,
                                                        uint32_t index, long long& bin,
                                                        long long& bout) {
  const longlong2 tile = __ldg(reinterpret_cast<const longlong2*>(tiles) + index);
  bin = tile.x & ((1LL << GROUP_TILE_SHIFT) - 1);
  bout = tile.y;
  return tens + (int)(tile.x >> GROUP_TILE_SHIFT);
}

// One tile of a group bucket per CTA, loads through registers (LOADS 0), or
// persistent CTAs (grid = SMs x occupancy) that walk the bucket's tile list with a
// grid stride, cp.async loads (LOADS 2).  One tile per CTA with cp.async is the mixed
// launch (k_groupmix.cu).
template <int ES, int LV, int SV, int NL, int LOADS>
__global__ void __launch_bounds__(TILE_THREADS)
groupTileKernel(const GroupTensor* __restrict__ tens, const GroupTile* __restrict__ tiles,
                uint32_t numTiles) {
  long long bin, bout;
  dependencyRelease();
  if constexpr (LOADS == 2) {
    for (uint32_t t = blockIdx.x; t < numTiles; t += gridDim.x) {
      const GroupTensor* g = groupTile(tens, tiles, t, bin, bout);
      groupTileBody<ES, LV, SV, NL, true>(g, bin, bout);
      __syncthreads();  // the next tile reuses the shared buffers
    }
  } else {
    const GroupTensor* g = groupTile(tens, tiles, blockIdx.x, bin, bout);
    groupTileBody<ES, LV, SV, NL, false>(g, bin, bout);
  }
}

}  // namespace lt
