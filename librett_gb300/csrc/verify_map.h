// The verifier's check of its own addressing.
//
// The verifier reads tiles by the boxes that the grouped kernel moves them by
// (box.h), so a mistake there would be made on both sides and pass.  Therefore each
// check also replays the box of its tile, with input offsets in the place of data,
// against the transpose formula: an output offset's digits by the output's dims,
// times the input's strides.  The formula shares nothing with the planner's tile or
// the box but the fused dims and the tile's extents.  The replay accepts a box only
// when every element of the tile is loaded once and compared once, with the input
// element that the formula names.
//
// The formula is linear in the digits, and tiles start at multiples of the extents
// (or end at the dim), so the map of a tile at the origin and the corners, which
// verify.cu works out from the extents itself, are the map of the tensor.
#pragma once

#include <cstdint>

#include "box.h"
#include "plan.h"

namespace lt {

LT_HD uint32_t mapDiv(uint32_t n, const FastDiv& f) {
  return (uint32_t)(((uint64_t)n * f.mul) >> f.shift);
}

// The tile in output order.
struct TileMap {
  int rank, vol;
  FastDiv dim[MAXR];      // d 0: a dim of 2^31 or more, which no offset in a tile exceeds
  uint32_t ext[MAXR];     // of the tile
  uint32_t inStep[MAXR];  // input stride (extents of 2 and more: below 2^31)
};

inline TileMap makeTileMap(const Fused& f, const int64_t* extent) {
  TileMap m{};
  m.rank = f.rank;
  m.vol = 1;
  for (int i = 0; i < f.rank; ++i) {
    const int r = f.perm[i];
    m.dim[i] = f.dim[r] < (int64_t(1) << 31) ? makeFastDiv((uint32_t)f.dim[r]) : FastDiv{};
    m.ext[i] = (uint32_t)extent[r];
    m.inStep[i] = extent[r] > 1 ? (uint32_t)f.sin[r] : 0;
    m.vol *= (int)extent[r];
  }
  return m;
}

// What a shared-memory cell holds that no element was loaded to, and one that was
// compared.
constexpr uint32_t CELL_EMPTY = 0xffffffffu, CELL_USED = 0xfffffffeu;

LT_HD bool cellInside(uint32_t at, uint32_t smBytes, int es) {
  return at % 4 == 0 && at < smBytes && smBytes - at >= (uint32_t)es;
}

// A replay takes four steps, each of them for every thread before the next: cells
// empty; mapLoads; mapStores; mapMark.  A box is sound when
// all return true, both counts are map.vol and map.vol cells are marked: then all
// comparisons read different cells, none of them empty, so every cell was loaded
// once, and different output offsets, as the formula names each input offset once.

// A thread's loads: put(at, offset) puts each element's input offset into its cell, at
// byte `at` of the tile's shared memory.  Adds the elements to n; false where a cell
// is outside.
#ifdef __CUDACC__
#pragma nv_exec_check_disable  // put, get and mark are for the host or for the device
#endif
template <typename Put>
LT_HD bool mapLoads(const unsigned char* block, uint32_t thread, uint32_t smBytes, int& n, Put put) {
  const TileBlock& g = *reinterpret_cast<const TileBlock*>(block);
  const BoxSlot* slot = reinterpret_cast<const BoxSlot*>(block + g.ld.slotAt);
  const Place l = placeAt(block, g.ld, thread);
  const int es = g.es, unit = g.ld.unit;
  bool ok = true;
  for (int k = 0; k < l.slots; ++k)
    for (int m = 0; m < unit; ++m) {
      const uint32_t at = l.sm + slot[k].sm + (uint32_t)(m * es);
      if (cellInside(at, smBytes, es))
        put(at, l.off + slot[k].off + (uint32_t)m);
      else
        ok = false;
    }
  n += l.slots * unit;
  return ok;
}

// A thread's comparisons, as the kernel for ES and SV makes them: get(at) must be the
// input offset that the formula names for the element's output offset, and that must
// lie inside the tile.  Adds the elements to n.  Eight elements at a time, so that a
// rank's divider is read once for them.
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <int ES, int SV, typename Get>
LT_HD bool mapStores(const TileMap& map, const unsigned char* block, uint32_t thread,
                     uint32_t smBytes, int& n, Get get) {
  constexpr int N = 8;
  static_assert(N % SV == 0, "whole units");
  const TileBlock& g = *reinterpret_cast<const TileBlock*>(block);
  const BoxSlot* slot = reinterpret_cast<const BoxSlot*>(block + g.st.slotAt);
  const Place t = placeAt(block, g.st, thread);
  uint32_t sm[SV];
  elementsAt<SV>(block, g, thread, t.sm, sm);
  const int es = g.es, per = SV > 1 ? SV : ES / es, total = t.slots * per;
  bool ok = true;
  for (int e0 = 0; e0 < total; e0 += N) {
    uint32_t o[N], at[N], src[N];
#pragma unroll
    for (int j = 0; j < N; ++j) {
      const int e = e0 + j < total ? e0 + j : total - per + j % per;  // past the end: again
      const int m = SV > 1 ? j % SV : e % per;
      const BoxSlot s = slot[e / per];
      o[j] = t.off + s.off + (uint32_t)m;
      at[j] = (SV > 1 ? sm[j % SV] : sm[0] + (uint32_t)(m * es)) + s.sm;
      src[j] = 0;
      ok = ok && (o[j] >> 31) == 0;
    }
#pragma unroll 1
    for (int i = 0; i < map.rank; ++i) {
      const FastDiv d = map.dim[i];
      const uint32_t ext = map.ext[i], step = map.inStep[i];
#pragma unroll
      for (int j = 0; j < N; ++j) {
        const uint32_t q = d.d != 0 ? mapDiv(o[j], d) : 0, c = o[j] - q * d.d;
        ok = ok && c < ext;
        src[j] += c * step;
        o[j] = q;
      }
    }
#pragma unroll
    for (int j = 0; j < N; ++j)
      ok = ok && o[j] == 0 && cellInside(at[j], smBytes, es) && get(at[j]) == src[j];
  }
  n += total;
  return ok;
}

// The same elements' cells: mark(at).
#ifdef __CUDACC__
#pragma nv_exec_check_disable
#endif
template <int ES, int SV, typename Mark>
LT_HD void mapMark(const unsigned char* block, uint32_t thread, uint32_t smBytes, Mark mark) {
  const TileBlock& g = *reinterpret_cast<const TileBlock*>(block);
  const BoxSlot* slot = reinterpret_cast<const BoxSlot*>(block + g.st.slotAt);
  const Place t = placeAt(block, g.st, thread);
  uint32_t sm[SV];
  elementsAt<SV>(block, g, thread, t.sm, sm);
  for (int k = 0; k < t.slots; ++k)
#pragma unroll
    for (int m = 0; m < SV; ++m)
      for (int b = 0; b < ES; b += g.es) {
        const uint32_t at = sm[m] + slot[k].sm + (uint32_t)b;
        if (cellInside(at, smBytes, g.es)) mark(at);
      }
}

}  // namespace lt
