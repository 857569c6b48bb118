// Slot addressing of the flat and bulk-copy tile kernels (table-free tiles).
//
// Thread t of a CTA handles in-tile elements x = t * V + k * B of one side,
// k = 0, 1, ... ("slots"), with B = TILE_THREADS * V.  The offset of x is the
// sum of its mixed-radix digits times their steps.  Decoding every x costs a
// multiply-high and two multiply-adds per rank and element; here the digits
// of t * V are decoded once per thread, the digits c of k * B are the same
// for every thread and are worked out on the host, and the sum of the two is
// formed by adding with carry:
//   d[r] + c[r] + carry >= ext[r]  <=>  d[r] + carry >= lim = ext[r] - c[r],
// and each carry replaces ext[r] steps of rank r by one of rank r + 1
// (corr = step[r + 1] - ext[r] * step[r]).  A slot then costs one addition
// plus, per rank but the last, one comparison and one predicated addition
// with operands in the parameter block.
//
// Narrow units are bound by instruction issue: float32 (127, 63, 65, 33) perm
// (3, 1, 2, 0), which moved in 4-byte units on both sides, issued 74 warp
// instructions per 32 elements with every element decoded on its own and 45
// with slot sums (39.9 -> 30.9 us; 28.7 us with dependent launches as well).
//
// Unused high ranks have ext 2^16 (in-tile indices are smaller, so their
// lower neighbour never carries into them) and step 0.  Sums are unsigned: a
// sum before its carries are applied may pass 2^31, the offset itself never
// does.
#pragma once

#include <cstdint>

#include "plan.h"

#ifdef __CUDACC__
#define LT_HD __host__ __device__ __forceinline__
#else
#define LT_HD inline
#endif

namespace lt {

constexpr int SLOT_EXT_NONE = 1 << 16;

LT_HD uint32_t slotMulHi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// Load side: NS slots, NR ranks (>= 2), one offset.
template <int NS, int NR>
struct LoadSlots {
  uint32_t mul[NR - 1];  // ceil(2^32 / ext)
  int ext[NR - 1];
  uint32_t step[NR];
  uint32_t corr[NR - 1];
  int lim[NS][NR - 1];
  uint32_t off[NS];  // offset of k * B
};

// Store side: the global output offset and the input-order index (in bytes).
template <int NS, int NR>
struct StoreSlots {
  uint32_t mul[NR - 1];
  int ext[NR - 1];
  uint32_t step[NR], stepJ[NR];
  uint32_t corr[NR - 1], corrJ[NR - 1];
  int lim[NS][NR - 1];
  uint32_t off[NS], offJ[NS];
};

// Digits of in-tile index x (below 2^16): d[0 .. NR-2], the last digit
// returned.
template <int NR>
LT_HD int slotDigits(const uint32_t* mul, const int* ext, uint32_t x, int* d) {
#pragma unroll
  for (int r = 0; r + 1 < NR; ++r) {
    const uint32_t q = slotMulHi(x, mul[r]);
    d[r] = (int)(x - q * (uint32_t)ext[r]);
    x = q;
  }
  return (int)x;
}

template <int NS, int NR>
LT_HD uint32_t loadThreadOffset(const LoadSlots<NS, NR>& s, uint32_t x, int* d) {
  uint32_t off = (uint32_t)slotDigits<NR>(s.mul, s.ext, x, d) * s.step[NR - 1];
#pragma unroll
  for (int r = 0; r + 1 < NR; ++r) off += (uint32_t)d[r] * s.step[r];
  return off;
}

template <int NS, int NR>
LT_HD uint32_t loadSlotOffset(const LoadSlots<NS, NR>& s, int k, uint32_t offT, const int* d) {
  uint32_t off = offT + s.off[k];
  int carry = 0;
#pragma unroll
  for (int r = 0; r + 1 < NR; ++r) {
    const bool c = d[r] + carry >= s.lim[k][r];
    if (c) off += s.corr[r];
    carry = c ? 1 : 0;
  }
  return off;
}

template <int NS, int NR>
LT_HD void storeThreadOffset(const StoreSlots<NS, NR>& s, uint32_t x, int* d, uint32_t& off,
                             uint32_t& j) {
  const uint32_t top = (uint32_t)slotDigits<NR>(s.mul, s.ext, x, d);
  off = top * s.step[NR - 1];
  j = top * s.stepJ[NR - 1];
#pragma unroll
  for (int r = 0; r + 1 < NR; ++r) {
    off += (uint32_t)d[r] * s.step[r];
    j += (uint32_t)d[r] * s.stepJ[r];
  }
}

template <int NS, int NR>
LT_HD void storeSlotOffset(const StoreSlots<NS, NR>& s, int k, uint32_t offT, uint32_t jT,
                           const int* d, uint32_t& off, uint32_t& j) {
  off = offT + s.off[k];
  j = jT + s.offJ[k];
  int carry = 0;
#pragma unroll
  for (int r = 0; r + 1 < NR; ++r) {
    const bool c = d[r] + carry >= s.lim[k][r];
    if (c) {
      off += s.corr[r];
      j += s.corrJ[r];
    }
    carry = c ? 1 : 0;
  }
}

// Load-side ranks of a tile: its ranks in input order, a rank whose input
// stride continues the previous one's extent merged into it (a tile that
// covers whole leading dims has one contiguous run there).  Returns their
// number.
inline int loadRanks(const TileParams& tp, int* ext, int* step) {
  int n = 0;
  for (int t = 0; t < tp.nTR; ++t) {
    if (n > 0 && (int64_t)tp.trSin[t] == (int64_t)ext[n - 1] * step[n - 1]) {
      ext[n - 1] *= tp.trE[t];
    } else {
      ext[n] = tp.trE[t];
      step[n] = tp.trSin[t];
      ++n;
    }
  }
  return n;
}

namespace detail {

// Fields shared by both sides: digits by ext (n ranks, padded to NR), limits
// and offsets of slot k at element k * B for steps `step`.
template <int NS, int NR>
void fillSlots(int n, const int* ext, const int* step, int B, uint32_t* mul, int* extOut,
               uint32_t* stepOut, uint32_t* corr, int (*lim)[NR - 1], uint32_t* off) {
  int e[NR], st[NR];
  for (int r = 0; r < NR; ++r) {
    e[r] = r < n ? ext[r] : SLOT_EXT_NONE;
    st[r] = r < n ? step[r] : 0;
    stepOut[r] = (uint32_t)st[r];
  }
  for (int r = 0; r + 1 < NR; ++r) {
    mul[r] = (uint32_t)(((uint64_t(1) << 32) + e[r] - 1) / e[r]);
    extOut[r] = e[r];
    // an unused neighbour is never carried into
    corr[r] = r + 1 < n ? (uint32_t)st[r + 1] - (uint32_t)e[r] * (uint32_t)st[r] : 0;
  }
  for (int k = 0; k < NS; ++k) {
    uint32_t x = (uint32_t)(k * B);
    uint32_t o = 0;
    for (int r = 0; r + 1 < NR; ++r) {
      const uint32_t q = x / (uint32_t)e[r];
      const int c = (int)(x - q * (uint32_t)e[r]);
      lim[k][r] = e[r] - c;
      o += (uint32_t)c * (uint32_t)st[r];
      x = q;
    }
    off[k] = o + x * (uint32_t)st[NR - 1];  // slots past the tile are never used
  }
}

}  // namespace detail

template <int NS, int NR>
void makeLoadSlots(const TileParams& tp, LoadSlots<NS, NR>& s) {
  int ext[MAXR], step[MAXR];
  const int n = loadRanks(tp, ext, step);
  detail::fillSlots<NS, NR>(n, ext, step, TILE_THREADS * tp.lv, s.mul, s.ext, s.step, s.corr, s.lim,
                            s.off);
}

// stepJ: shared bytes between elements along each tile rank, in output order.
template <int NS, int NR>
void makeStoreSlots(const TileParams& tp, const int* stepJ, StoreSlots<NS, NR>& s) {
  detail::fillSlots<NS, NR>(tp.nTR, tp.toE, tp.toSout, TILE_THREADS * tp.sv, s.mul, s.ext, s.step,
                            s.corr, s.lim, s.off);
  detail::fillSlots<NS, NR>(tp.nTR, tp.toE, stepJ, TILE_THREADS * tp.sv, s.mul, s.ext, s.stepJ,
                            s.corrJ, s.lim, s.offJ);
}

template <int NS, int NR>
void makeStoreSlots(const TileParams& tp, int esize, StoreSlots<NS, NR>& s) {
  int stepJ[MAXR];
  for (int i = 0; i < tp.nTR; ++i) stepJ[i] = tp.toInTile[i] * esize;
  makeStoreSlots(tp, stepJ, s);
}

// Span loads of a tile whose input moves in element units: the contiguous runs
// of its input come as the aligned 16-byte blocks around them (tileKernelSpan).
// A run lies in shared memory at the same address modulo 16 as in global memory,
// for every tile: a rank's shared step is congruent to its global step modulo 16,
// so that shared addresses stay sums of digits times steps, and runs lie far
// enough apart for the blocks around them.
struct SpanLayout {
  int perRun, units;  // blocks of a run, of the tile
  int n;              // load ranks (loadRanks), the first of them the run
  int ext[MAXR], step[MAXR], stepS[MAXR];  // extents; global (elements) and shared (bytes) steps
  int stepJ[MAXR];    // shared step of each tile rank in output order
  int smBytes;
};

// 4-byte elements in runs of 128 bytes or more.  float32 (r, 4000, 53) perm (2, 1,
// 0), runs of r elements, in element units and in spans: r = 33 12.77 and 12.52 us,
// 45 16.6 and 15.7, 61 22.1 and 20.2, 65 23.3 and 22.2, 126 (runs of 63) 43.5 and
// 41.3.  Shorter runs read more than an eighth of their bytes again.  8-byte
// elements have half the load instructions to save and lost: float64 (127, 63, 65,
// 33) perm (3, 1, 2, 0) 46.5 and 47.7, (2, 4, 105, 294, 92) off alignment 55.2 and 61.5.
// The plan selector does not know spans: its timings of such candidates are the flat
// kernel's, up to 9 % above, and a plan's shared memory is the flat layout's.
constexpr int SPAN_ES = 4, SPAN_MIN_BYTES = 128, SPAN_MAX_SMEM = 48 * 1024;

// Load slots of a tile of at most NL elements per thread: a run of
// SPAN_MIN_BYTES or more takes at most 1/8 more blocks than its bytes fill.
LT_HD constexpr int spanSlots(int NL) { return NL * SPAN_ES / 16 + 1; }

inline bool makeSpan(const TileParams& tp, int esize, SpanLayout& L) {
  if (esize != SPAN_ES || tp.lv != 1 || tp.nTR < 1 || tp.trSin[0] != 1) return false;
  L.n = loadRanks(tp, L.ext, L.step);
  const int bytes = L.ext[0] * esize;
  if (bytes < SPAN_MIN_BYTES) return false;
  L.perRun = (16 - esize + bytes + 15) / 16;
  L.units = tp.tileVol / L.ext[0] * L.perRun;
  int room = L.perRun * 16 + 15;  // of the ranks so far, wherever a block starts
  L.stepS[0] = esize;
  for (int r = 1; r < L.n; ++r) {
    const int want = (int)((int64_t)L.step[r] * esize % 16);
    L.stepS[r] = room + (want - room % 16 + 16) % 16;
    // an odd number of 16-byte units at least: lanes that step along this rank
    // then meet in 4 of 32 banks' worth at most, not in one bank
    if (L.stepS[r] % 32 == 0) L.stepS[r] += 16;
    room = L.ext[r] * L.stepS[r];
  }
  L.smBytes = (room + 16 + 15) / 16 * 16;  // and the tile's own start modulo 16
  if (L.smBytes > SPAN_MAX_SMEM) return false;
  // tile ranks merged into a load rank continue each other
  int trStep[MAXR];
  for (int t = 0, r = -1, left = 1; t < tp.nTR; ++t) {
    if (left == 1) {
      ++r;
      left = L.ext[r];
      trStep[t] = L.stepS[r];
    } else {
      trStep[t] = trStep[t - 1] * tp.trE[t - 1];
    }
    left /= tp.trE[t];
  }
  for (int i = 0; i < tp.nTR; ++i) L.stepJ[i] = trStep[tp.trOut[i]];
  return true;
}

// Global offsets (elements) and shared addresses (bytes) of the blocks, before
// both are rounded down to 16 bytes.
template <int NS, int NR>
void makeSpanSlots(const SpanLayout& L, StoreSlots<NS, NR>& s) {
  int ext[MAXR], step[MAXR], stepS[MAXR];
  for (int r = 0; r < L.n; ++r) {
    ext[r] = r == 0 ? L.perRun : L.ext[r];
    step[r] = r == 0 ? 16 / SPAN_ES : L.step[r];
    stepS[r] = r == 0 ? 16 : L.stepS[r];
  }
  detail::fillSlots<NS, NR>(L.n, ext, step, TILE_THREADS, s.mul, s.ext, s.step, s.corr, s.lim, s.off);
  detail::fillSlots<NS, NR>(L.n, ext, stepS, TILE_THREADS, s.mul, s.ext, s.stepJ, s.corrJ, s.lim,
                            s.offJ);
}

// Grid ranks whose chunks fit the parameter block of rank class c.  The block
// is copied into every launch, so the classes of few tile ranks carry only as
// many grid ranks as a problem of rank 7 can have (float32 (64, 48, 32) in
// a loop of executes: 2.90 us a call with room for 16 in every class, 2.72 here).
constexpr int GRID_FEW = 7;
constexpr int gridCapacity(int rankClass) { return rankClass < ARITH_MAX_NTR ? GRID_FEW : MAXR; }

// Rank counts the kernels are instantiated for: tiles of 1..6 ranks run as
// 2, 3, 4 or 6 (high ranks unused), and as 6 with more than GRID_FEW grid
// ranks (a tensor of eight ranks or more); 0 for tiles with offset tables.
inline int storeRankClass(const TileParams& tp) {
  const int r = arithRanks(tp);
  if (r == 0) return 0;
  if (tp.nGR > GRID_FEW) return ARITH_MAX_NTR;
  return r <= 2 ? 2 : r <= 4 ? r : ARITH_MAX_NTR;
}

}  // namespace lt
