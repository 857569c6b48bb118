// Grouped execution, mixed launch: tiles of every element size and unit in
// one grid.
//
// A launch of one bucket costs about 5 us whatever its work (graph node, first
// descriptor reads, one tile), and a batch of small tensors has tens of buckets
// of a few CTAs each.  500 tensors of 2^10 .. 2^16 elements: 33 launches on 8
// graph branches 77.0 us, one mixed launch 18.2 us.  2,500 tensors of 2^10 ..
// 2^22 elements: 2567 us in buckets, 2406 us mixed (93 % of the copy rate); what
// is left there is partly filled sectors of narrow runs.
//
// The code of a tile must be short here, because neighbouring CTAs run
// different units: with the buckets' unrolled bodies behind a switch, warps
// waited for instructions 13 cycles per issue (29.5 us).  Box addressing
// (box.h) needs one rolled loop per side, chosen by the load unit's bytes and
// by element size and store unit.  A CTA first copies its member's block (a few
// hundred bytes) into shared memory, where the slots are read from.
#include "box_kernel.cuh"

namespace lt {
namespace {

template <int ES, int SV>
__device__ __forceinline__ void storeTileOf(const unsigned char* block, const TileBlock& g, int n,
                                            unsigned char* dst, uint32_t sm0) {
  // (a wide unit is one read of its bytes: ES is not the element size then)
  using T = typename Word<ES>::T;
  using ST = typename Word<ES * SV>::T;
  uint32_t sm[SV];
  elementsOf<SV>(block, g, sm0, sm);
  const int es = g.es;
  auto one = [&](const BoxSlot& s) {
    T e[SV];
#pragma unroll
    for (int m = 0; m < SV; ++m) e[m] = ldShared<ES>(sm[m] + s.sm);
    ST v;
    __builtin_memcpy(&v, e, sizeof(ST));
    return v;
  };
  forSlots<4>(block, g.st, n, [&](auto... s) {
    const ST v[] = {one(s)...};
    const uint32_t off[] = {s.off...};
#pragma unroll
    for (int i = 0; i < (int)sizeof...(s); ++i)
      *reinterpret_cast<ST*>(offsetBytes(dst, (int)off[i], es)) = v[i];
  });
}

// Blocks of V x V elements, transposed in registers.
template <int ES>
__device__ __forceinline__ void storeBlocks(const unsigned char* block, const TileBlock& g, int n,
                                            unsigned char* dst, uint32_t sm0) {
  using T = typename Word<ES>::T;
  constexpr int V = 16 / ES;
  const int esR = opaque(ES);
  forSlots<V == 2 ? 2 : 1>(block, g.st, n, [&](auto... s) {
    constexpr int N = (int)sizeof...(s);
    const uint32_t sm[] = {s.sm...}, off[] = {s.off...};
    T e[N][V][V];
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
      for (int m = 0; m < V; ++m) {
        const uint4 r = ldShared<16>(sm0 + sm[i] + (uint32_t)m * g.elemStep);
        __builtin_memcpy(e[i][m], &r, 16);
      }
#pragma unroll
    for (int i = 0; i < N; ++i) {
      unsigned char* d = offsetBytes(dst, (int)off[i], esR);
#pragma unroll
      for (int c = 0; c < V; ++c) {
        T col[V];
#pragma unroll
        for (int m = 0; m < V; ++m) col[m] = e[i][m][c];
        uint4 r;
        __builtin_memcpy(&r, col, 16);
        *reinterpret_cast<uint4*>(d) = r;
        d += g.colStep;
      }
    }
  });
}

// Tiles ahead of a CTA's own whose list entry (two steps) and block (one step) it
// brings into L2: about a wave of six CTAs on each of 152 SMs.  Without that, a
// CTA's first two reads wait for memory one after the other, with the tile's own
// traffic in front of them (2,500 tensors of 2^10 .. 2^22 elements: 2423 -> 2406 us;
// a step of 512: 2410; the list entries alone: 2414).
constexpr uint32_t AHEAD = 1024;

__device__ __forceinline__ void prefetchL2(const void* p) {
  asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

__global__ void __launch_bounds__(TILE_THREADS, 6)
groupMixedKernel(const uint4* __restrict__ blocks, const GroupTile* __restrict__ tiles,
                 int blockBytes) {
  extern __shared__ __align__(16) unsigned char smraw[];
  dependencyRelease();
  const longlong2 tile = __ldg(reinterpret_cast<const longlong2*>(tiles) + blockIdx.x);
  constexpr long long LOW = (1LL << GROUP_TILE_SHIFT) - 1;
  const uint32_t sBase = (uint32_t)__cvta_generic_to_shared(smraw);
  if (threadIdx.x < (uint32_t)(tile.y >> GROUP_TILE_SHIFT))
    cpAsyncUnit<16>(sBase + 16 * threadIdx.x, blocks + (tile.x >> GROUP_TILE_SHIFT) + threadIdx.x);
  if (threadIdx.x == 0 && blockIdx.x + 2 * AHEAD < gridDim.x)
    prefetchL2(tiles + blockIdx.x + 2 * AHEAD);
  cpAsyncWaitAll();
  __syncthreads();
  const TileBlock& g = *reinterpret_cast<const TileBlock*>(smraw);
  const uint32_t sData = sBase + (uint32_t)blockBytes;
  const int es = g.es;
  {
    const Place t = placeOf(smraw, g.ld);
    const unsigned char* src = g.in + (tile.x & LOW) * es;
    src = offsetBytes(src, (int)t.off, es);
    // blocks and tile list are written once, at group creation (which
    // synchronises), so only the tensors' data waits for the stream
    dependencyWait();
    switch (es * g.ld.unit) {
      case 16: loadTile<16>(smraw, g.ld, t.slots, src, sData + t.sm, es); break;
      case 8: loadTile<8>(smraw, g.ld, t.slots, src, sData + t.sm, es); break;
      default: loadTile<4>(smraw, g.ld, t.slots, src, sData + t.sm, es); break;
    }
  }
  // while the loads are in flight: one warp's lanes fetch 8 units (128 bytes) each
  if (threadIdx.x < 32 && blockIdx.x + AHEAD < gridDim.x) {
    const longlong2 next = __ldg(reinterpret_cast<const longlong2*>(tiles) + blockIdx.x + AHEAD);
    if (8 * threadIdx.x < (uint32_t)(next.y >> GROUP_TILE_SHIFT))
      prefetchL2(blocks + (next.x >> GROUP_TILE_SHIFT) + 8 * threadIdx.x);
  }
  const Place t = placeOf(smraw, g.st);
  unsigned char* dst = offsetBytes(g.out + (tile.y & LOW) * es, (int)t.off, es);
  cpAsyncWaitAll();
  __syncthreads();
  switch (g.store) {
#define LT_STORE(ES, SV) \
  case blockStore(ES, SV): storeTileOf<ES, SV>(smraw, g, t.slots, dst, sData + t.sm); break;
    LT_STORE(4, 4)
    LT_STORE(4, 2)
    LT_STORE(4, 1)
    LT_STORE(8, 2)
    LT_STORE(8, 1)
    LT_STORE(16, 1)
#undef LT_STORE
    case blockStore(4, 0): storeBlocks<4>(smraw, g, t.slots, dst, sData + t.sm); break;
    case blockStore(8, 0): storeBlocks<8>(smraw, g, t.slots, dst, sData + t.sm); break;
    default: break;
  }
}

}  // namespace

cudaError_t launchGroupMixed(const void* blocks, const GroupTile* tiles, uint32_t numTiles,
                             int blockBytes, int smem, cudaStream_t s) {
  if (smem > 48 * 1024 &&
      cachedOccupancy((const void*)groupMixedKernel, TILE_THREADS, smem) < 1)
    return cudaErrorInvalidConfiguration;
  return launchDependent(groupMixedKernel, numTiles, TILE_THREADS, smem, s, (const uint4*)blocks,
                         tiles, blockBytes);
}

}  // namespace lt
