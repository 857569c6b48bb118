// Device side of box addressing (box.h): a CTA's member block in shared memory,
// its threads' places, and the loops over slots.  Used by the grouped mixed
// launch and the verifier.
#pragma once

#include "tile_kernel.cuh"

namespace lt {

struct Place {  // of a thread on one side
  uint32_t off, sm;
  int slots;  // it takes part in
};

__device__ __forceinline__ Place placeOf(const unsigned char* block, const BoxHead& h) {
  Place t;
  const BoxRank* rank = reinterpret_cast<const BoxRank*>(block + h.rankAt);
  const int top = boxDecode(rank, h.p, threadIdx.x * h.unit, t.off, t.sm);
  t.slots = (int)threadIdx.x >= h.active ? 0 : h.nFull + (top < h.rem ? h.nRagged : 0);
  return t;
}

// Runs f(slots...) for slots 0 .. n - 1 (n may differ between threads), PER (1,
// 2 or 4) at a time and the rest one by one.
template <int PER, typename F>
__device__ __forceinline__ void forSlots(const unsigned char* block, const BoxHead& h, int n, F f) {
  const BoxSlot* slot = reinterpret_cast<const BoxSlot*>(block + h.slotAt);
  int k = 0;
  if constexpr (PER > 1) {
#pragma unroll 1
    for (; k + PER <= n; k += PER) {
      const uint4 a = reinterpret_cast<const uint4*>(slot + k)[0];
      if constexpr (PER == 4) {
        const uint4 b = reinterpret_cast<const uint4*>(slot + k)[1];
        f(BoxSlot{a.x, a.y}, BoxSlot{a.z, a.w}, BoxSlot{b.x, b.y}, BoxSlot{b.z, b.w});
      } else {
        f(BoxSlot{a.x, a.y}, BoxSlot{a.z, a.w});
      }
    }
  }
#pragma unroll 1
  for (; k < n; ++k) f(slot[k]);
}

template <int BYTES>
__device__ __forceinline__ void loadTile(const unsigned char* block, const BoxHead& h, int n,
                                         const unsigned char* src, uint32_t dst, int es) {
  forSlots<4>(block, h, n, [&](auto... s) {
    (cpAsyncUnit<BYTES, LT_GROUP_L2_PREFETCH>(dst + s.sm, offsetBytes(src, (int)s.off, es)), ...);
  });
}

// Shared addresses of the SV elements of a thread's store unit, the first at
// sm0.
template <int SV>
__device__ __forceinline__ void elementsOf(const unsigned char* block, const TileBlock& g,
                                           uint32_t sm0, uint32_t (&sm)[SV]) {
  sm[0] = sm0;
#pragma unroll
  for (int m = 1; m < SV; ++m) sm[m] = sm0 + (uint32_t)m * g.elemStep;
  if (SV > 1 && g.straddle) {
    const BoxRank* rank = reinterpret_cast<const BoxRank*>(block + g.st.rankAt);
    uint32_t off, first, j;
    boxDecode(rank, g.st.p, threadIdx.x * SV, off, first);
#pragma unroll
    for (int m = 1; m < SV; ++m) {
      boxDecode(rank, g.st.p, threadIdx.x * SV + m, off, j);
      sm[m] = sm0 + j - first;
    }
  }
}

}  // namespace lt
