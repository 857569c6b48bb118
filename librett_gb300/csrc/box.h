// Addressing of a tile by boxes, which the grouped kernel reads instead of
// decoding every unit.
//
// On each side the tile's ranks are listed in that side's order (input order
// for loads, output order for stores), ranks that continue each other in
// global and in shared memory merged.  The CTA's threads cover a box: the
// leading ranks whole, then as much of the next rank (the top rank) as fits
// TILE_THREADS units.  Slots move that box over the tile: chunks of the top
// rank, times every digit of the ranks above it.  A thread decodes its place
// in the box once; a slot is the same for all threads, a global offset and a
// shared-memory offset that the host works out.  So a unit costs one 64-bit
// multiply-add for its global address and one addition for its shared one,
// with no division, for any number of ranks, and the code is one short loop
// per side and unit size.  Slots of whole chunks need no guard; the ones of
// the ragged last chunk apply to threads whose top digit is below rem.
//
// Where both sides move 16-byte units of V elements along whole multiples of V
// of the input's and the output's fastest rank, a store item is a block of V x
// V elements: V 16-byte reads of shared memory, transposed in registers, V
// 16-byte stores.  That takes a V-th of the shared-memory reads of single
// elements, and their 4-byte (float32) or 8-byte accesses V units apart cannot
// be free of bank conflicts under padding that keeps 16-byte units aligned.
//
// Shared memory holds the tile at strides of its own per rank (stepS), which
// place the padding: some elements after a rank, or after the V rows that one
// store unit reads (the output-fastest rank is split there).  The layout is
// picked by counting the bank wavefronts of the warps' real accesses.
#pragma once

#include <cstdint>
#include <vector>

#include "plan.h"

#ifdef __CUDACC__
#define LT_HD __host__ __device__ __forceinline__
#else
#define LT_HD inline
#endif

namespace lt {

constexpr int BOX_SLOTS = 64;         // of a side, at most
constexpr int BOX_RANKS = MAXR + 1;   // of a side, with one split

struct alignas(16) BoxRank {
  uint32_t mul;    // ceil(2^32 / ext)
  uint32_t ext;
  uint32_t step;   // global step (elements)
  uint32_t stepS;  // shared step (bytes)
};

struct alignas(8) BoxSlot {
  uint32_t off;  // elements
  uint32_t sm;   // bytes
};

// One side without its arrays.
struct alignas(16) BoxHead {
  int active;          // threads of the box
  int p;               // the top rank: a thread decodes ranks 0 .. p
  int rem;             // top digits below rem take part in the ragged chunk
  int nFull, nRagged;  // slots of whole chunks, then of the ragged chunk
  int rankAt, slotAt;  // grouped execution: byte offsets of the arrays in the block
  int unit;            // elements
};

struct BoxSide {
  BoxHead h;
  BoxRank rank[BOX_RANKS];
  BoxSlot slot[BOX_SLOTS];
};

struct BoxParams {
  BoxSide ld, st;
  int block;          // store items are V x V blocks (unit 1 in st.h: one item)
  long long colStep;  // global output step (elements) between a block's V stores
  int wide;           // a store unit's elements are one aligned piece of shared memory
  int straddle;       // a store unit's elements cross output rank 0
  uint32_t elemStep;  // shared bytes between a store unit's elements otherwise,
                      // and between a block's V reads
  int smBytes;        // shared memory of the tile
};

// Box addressing of a tile (its units lv and sv; the store unit may be 1
// where no box can be cut at a unit boundary).  False when a side needs more
// slots than BOX_SLOTS.
bool makeBox(const TileParams& tp, int esize, BoxParams& b, bool blocks = true);

// What a kernel reads of a box: this header, then the arrays of both sides at
// their byte offsets, in one block of 16-byte units.
struct alignas(16) TileBlock {
  const unsigned char* in;
  unsigned char* out;
  BoxHead ld, st;
  int es;
  int store;  // blockStore
  int straddle;
  uint32_t elemStep;
  long long colStep;  // bytes
  int unused[2];
};

constexpr int TILE_BLOCK_MAX =
    (int)(sizeof(TileBlock) + 2 * (BOX_RANKS * sizeof(BoxRank) + BOX_SLOTS * sizeof(BoxSlot)));

// Bytes of a shared-memory read and reads per store unit (0: blocks) as one
// number, which selects the store code.  A wide unit is one read of its bytes.
LT_HD constexpr int blockStore(int bytes, int reads) { return bytes * 8 + reads; }

// The block of a box, at most TILE_BLOCK_MAX bytes.
std::vector<unsigned char> packBlock(BoxParams& b, int esize, const void* in, void* out);

LT_HD uint32_t boxMulHi(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// Decodes box element x (below 2^16; the multiply-high is exact there): its
// offsets, and the top digit returned.
LT_HD int boxDecode(const BoxRank* rank, int p, uint32_t x, uint32_t& off, uint32_t& sm) {
  off = sm = 0;
  for (int r = 0; r < p; ++r) {
    const BoxRank k = rank[r];
    const uint32_t q = boxMulHi(x, k.mul);
    const uint32_t d = x - q * k.ext;
    off += d * k.step;
    sm += d * k.stepS;
    x = q;
  }
  off += x * rank[p].step;
  sm += x * rank[p].stepS;
  return (int)x;
}

struct Place {  // of a thread on one side
  uint32_t off, sm;
  int slots;  // it takes part in
};

LT_HD Place placeAt(const unsigned char* block, const BoxHead& h, uint32_t thread) {
  Place t;
  const BoxRank* rank = reinterpret_cast<const BoxRank*>(block + h.rankAt);
  const int top = boxDecode(rank, h.p, thread * h.unit, t.off, t.sm);
  t.slots = (int)thread >= h.active ? 0 : h.nFull + (top < h.rem ? h.nRagged : 0);
  return t;
}

// Shared addresses of the SV elements of a thread's store unit, the first at
// sm0.
template <int SV>
LT_HD void elementsAt(const unsigned char* block, const TileBlock& g, uint32_t thread, uint32_t sm0,
                      uint32_t (&sm)[SV]) {
  sm[0] = sm0;
#pragma unroll
  for (int m = 1; m < SV; ++m) sm[m] = sm0 + (uint32_t)m * g.elemStep;
  if (SV > 1 && g.straddle) {
    const BoxRank* rank = reinterpret_cast<const BoxRank*>(block + g.st.rankAt);
    uint32_t off, first, j;
    boxDecode(rank, g.st.p, thread * SV, off, first);
#pragma unroll
    for (int m = 1; m < SV; ++m) {
      boxDecode(rank, g.st.p, thread * SV + m, off, j);
      sm[m] = sm0 + j - first;
    }
  }
}

}  // namespace lt
