// Device side of box addressing (box.h): a CTA's member block in shared memory,
// its threads' places, and the loops over slots.  Used by the grouped mixed
// launch and the verifier.
#pragma once

#include "tile_kernel.cuh"

namespace lt {

__device__ __forceinline__ Place placeOf(const unsigned char* block, const BoxHead& h) {
  return placeAt(block, h, threadIdx.x);
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

template <int SV>
__device__ __forceinline__ void elementsOf(const unsigned char* block, const TileBlock& g,
                                           uint32_t sm0, uint32_t (&sm)[SV]) {
  elementsAt<SV>(block, g, threadIdx.x, sm0, sm);
}

}  // namespace lt
