// Device-side verifier: compares every output element of a transpose with
// the input element the transpose formula names, on the GPU, without a host
// copy of the tensors.  The role of LibreTT's device checker
// (src/TensorTester.cpp:47-126, checkTransposeKernel), which compares the
// output with an index pattern; this one compares with the actual input, so
// any input data works.
//
// The input is read a tile at a time through shared memory (box.h), because the
// elements that consecutive output elements name lie far apart: gathering them
// one by one from global memory (verifyKernel, kept for problems without a sound tile)
// fetched 32 bytes for 4 and took 745 us for 66.8M float32 elements (64, 128,
// 96, 85) perm (3, 1, 0, 2), where the two tensors' bytes take 80 us; this
// kernel takes 118 us (4-byte output units: two thirds of the issue slots).
// The tile's addressing is the grouped kernel's, the grid and the proof that the
// addressing is the transpose formula's are this file's own: each check replays its
// tile's map (verify_map.h), and where that fails, which no problem is
// known to do, the check is made element by element.
#include <cuda_runtime.h>
#include <unistd.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

#include "box_kernel.cuh"
#include "librett.h"
#include "librett_c.h"
#include "plan.h"
#include "plans.h"
#include "verify_map.h"

namespace lt {
namespace {

struct VerifyParams {
  int rank;
  unsigned long long vol;
  unsigned long long outD[MAXR];  // output-order dims (fused; may exceed 2^31)
  FastDiv outDim[MAXR];           // their fast dividers (dims below 2^31)
  long long inStride[MAXR];       // input stride of output rank i (elements)
};

// Adds a CTA's findings to the result, one pair of atomics per CTA that has any
// (the result lies in host memory).
__device__ __forceinline__ void report(unsigned long long bad, unsigned long long first,
                                       unsigned long long* result) {
  if (bad == 0) return;
  atomicAdd_system(result, bad);
  atomicMax_system(result + 1, ~first);
}

// result[0]: mismatching elements; result[1]: complement of the smallest
// mismatching output index (both start at 0)
template <int ES>
__global__ void __launch_bounds__(256)
verifyKernel(const __grid_constant__ VerifyParams p, const typename Word<ES>::T* __restrict__ in,
             const typename Word<ES>::T* __restrict__ out, unsigned long long* result) {
  using T = typename Word<ES>::T;
  unsigned long long bad = 0, first = ~0ull;
  const unsigned long long stride = (unsigned long long)gridDim.x * blockDim.x;
  for (unsigned long long q = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; q < p.vol;
       q += stride) {
    unsigned long long rem = q;
    long long src = 0;
    for (int i = 0; i < p.rank; ++i) {
      const unsigned long long d = p.outD[i];
      unsigned long long c;
      if (rem < (1ull << 31) && d < (1ull << 31)) {
        const uint32_t qq = fdiv((uint32_t)rem, p.outDim[i]);
        c = rem - (unsigned long long)qq * d;
        rem = qq;
      } else {
        c = rem % d;
        rem /= d;
      }
      src += (long long)c * p.inStride[i];
    }
    T a = in[src], b = out[q];
    bool same;
    if constexpr (ES == 4) {
      same = a == b;
    } else if constexpr (ES == 8) {
      same = a.x == b.x && a.y == b.y;
    } else {
      same = a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w;
    }
    if (!same) {
      ++bad;
      if (q < first) first = q;
    }
  }
  __shared__ unsigned long long sum, low;
  if (threadIdx.x == 0) {
    sum = 0;
    low = ~0ull;
  }
  __syncthreads();
  if (bad) {
    atomicAdd(&sum, bad);
    atomicMin(&low, first);
  }
  __syncthreads();
  if (threadIdx.x == 0) report(sum, low, result);
}

// Launches the element-by-element check.
cudaError_t verifyElements(const Fused& f, int sms, const void* in, const void* out,
                           unsigned long long* d, cudaStream_t s) {
  VerifyParams p{};
  p.rank = f.rank;
  p.vol = (unsigned long long)f.vol;
  for (int i = 0; i < f.rank; ++i) {
    const int r = f.perm[i];
    p.outD[i] = (unsigned long long)f.dim[r];
    p.outDim[i] = makeFastDiv(f.dim[r] < (int64_t(1) << 31) ? (uint32_t)f.dim[r] : 1u);
    p.inStride[i] = f.sin[r];
  }
  unsigned long long blocks = (p.vol + 255) / 256;
  const unsigned long long cap = (unsigned long long)sms * 8;
  if (blocks > cap) blocks = cap;
  if (blocks < 1) blocks = 1;
  auto launch = [&](auto kernel, auto word) {
    using T = decltype(word);
    kernel<<<(unsigned)blocks, 256, 0, s>>>(p, (const T*)in, (const T*)out, d);
  };
  switch (f.esize) {
    case 4: launch(verifyKernel<4>, Word<4>::T()); break;
    case 8: launch(verifyKernel<8>, Word<8>::T()); break;
    default: launch(verifyKernel<16>, Word<16>::T()); break;
  }
  return cudaGetLastError();
}

// A tile's box and its place in the tensor.
struct VerifyTiles {
  uint32_t numTiles;
  int blockBytes;
  int nGR;  // grid ranks, decode order
  FastDiv grDiv[MAXR];
  long long grSin[MAXR], grSout[MAXR], grLastIn[MAXR], grLastOut[MAXR];
  // A ragged last chunk of grid rank g overlaps its neighbour, which owns the
  // first `overlap` digits of that rank; 0 where the chunks divide the rank.  The
  // digit of an output offset o inside a tile is o / outStep % outDim (outDim.d 0:
  // no rank above).
  uint32_t overlap[MAXR];
  FastDiv outStep[MAXR], outDim[MAXR];
  int smBytes;  // of the tile, behind the block
  TileMap map;
  uint4 block[TILE_BLOCK_MAX / 16];
};

// A CTA's findings, in shared memory.
struct Findings {
  unsigned long long bad, first;
};

constexpr uint32_t VERIFY_LIST = 64;  // tiles with differences a CTA lists

// Corners of a tile; returns the grid ranks along which it overlaps its neighbour,
// as bits.
LT_HD uint32_t tileCorner(const VerifyTiles& p, uint32_t tile, long long& bin, long long& bout) {
  bin = bout = 0;
  uint32_t rem = tile, shared = 0;
  for (int r = 0; r < p.nGR; ++r) {
    const uint32_t q = mapDiv(rem, p.grDiv[r]);
    const uint32_t c = rem - q * p.grDiv[r].d;
    rem = q;
    const bool last = c + 1 == p.grDiv[r].d;
    bin += last ? p.grLastIn[r] : (long long)c * p.grSin[r];
    bout += last ? p.grLastOut[r] : (long long)c * p.grSout[r];
    if (last && p.overlap[r] > 0) shared |= 1u << r;
  }
  return shared;
}

// Whether a tile that overlaps its neighbours along the ranks of `shared` owns its
// element at output offset o from its corner.
__device__ __forceinline__ bool owns(const VerifyTiles& p, uint32_t shared, uint32_t o) {
  for (; shared != 0; shared &= shared - 1) {
    const int g = __ffs((int)shared) - 1;
    uint32_t digit = fdiv(o, p.outStep[g]);
    if (p.outDim[g].d != 0) digit -= fdiv(digit, p.outDim[g]) * p.outDim[g].d;
    if (digit < p.overlap[g]) return false;
  }
  return true;
}

__device__ __forceinline__ void loadInput(const unsigned char* block, const TileBlock& g,
                                          const Place& l, long long bin, uint32_t sTile) {
  const int es = g.es;
  const unsigned char* src = offsetBytes(g.in + bin * es, (int)l.off, es);
  switch (es * g.ld.unit) {
    case 16: loadTile<16>(block, g.ld, l.slots, src, sTile + l.sm, es); break;
    case 8: loadTile<8>(block, g.ld, l.slots, src, sTile + l.sm, es); break;
    default: loadTile<4>(block, g.ld, l.slots, src, sTile + l.sm, es); break;
  }
}

// Persistent CTAs over the tensor's tiles: the input tile goes to shared memory
// by cp.async; output units are read in batches, the first of them while the
// tile is on its way, and compared with the elements gathered from the tile.
// ES and SV as in the grouped store (a wide unit is one read of its bytes).
template <int ES, int SV>
__global__ void __launch_bounds__(TILE_THREADS, 6)
verifyTilesKernel(const __grid_constant__ VerifyTiles p, unsigned long long* result) {
  using T = typename Word<ES>::T;
  using ST = typename Word<ES * SV>::T;
  constexpr int N = ES * SV == 16 ? 4 : 8;  // units of a batch
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ Findings found;
  __shared__ uint32_t listed[VERIFY_LIST], numListed;  // tiles with a difference
  if (threadIdx.x == 0) {
    found = {0ull, ~0ull};
    numListed = 0;
  }
  dependencyRelease();  // of the map's kernel
  dependencyWait();     // at once: launched ordinarily
  for (int c = threadIdx.x; c < p.blockBytes / 16; c += blockDim.x)
    reinterpret_cast<uint4*>(smraw)[c] = p.block[c];
  __syncthreads();
  const TileBlock& g = *reinterpret_cast<const TileBlock*>(smraw);
  const uint32_t sTile = (uint32_t)__cvta_generic_to_shared(smraw) + (uint32_t)p.blockBytes;
  {
    const BoxSlot* slot = reinterpret_cast<const BoxSlot*>(smraw + g.st.slotAt);
    const int es = g.es;
    const Place l = placeOf(smraw, g.ld), t = placeOf(smraw, g.st);
    uint32_t sm[SV];
    elementsOf<SV>(smraw, g, sTile + t.sm, sm);
    for (uint32_t tile = blockIdx.x; tile < p.numTiles; tile += gridDim.x) {
      long long bin, bout;
      tileCorner(p, tile, bin, bout);
      loadInput(smraw, g, l, bin, sTile);
      const unsigned char* out = g.out + (bout + (int)t.off) * es;
      ST w[N];
      auto read = [&](int k) {
#pragma unroll
        for (int i = 0; i < N; ++i)
          if (k + i < t.slots) w[i] = ldGlobal<ES * SV>(offsetBytes(out, (int)slot[k + i].off, es));
      };
      read(0);
      cpAsyncWaitAll();
      __syncthreads();
      uint32_t differ = 0;
#pragma unroll 1
      for (int k = 0; k < t.slots; k += N) {
        if (k > 0) read(k);
#pragma unroll
        for (int i = 0; i < N; ++i)
          if (k + i < t.slots) {
            T e[SV];
#pragma unroll
            for (int m = 0; m < SV; ++m) e[m] = ldShared<ES>(sm[m] + slot[k + i].sm);
            uint32_t a[ES * SV / 4], b[ES * SV / 4];
            __builtin_memcpy(a, e, ES * SV);
            __builtin_memcpy(b, &w[i], ES * SV);
#pragma unroll
            for (int x = 0; x < ES * SV / 4; ++x) differ |= a[x] ^ b[x];
          }
      }
      // (also: the next tile reuses the buffer)
      if (__syncthreads_or((int)differ) && threadIdx.x == 0) {
        if (numListed < VERIFY_LIST) listed[numListed] = tile;
        ++numListed;
      }
    }
  }
  // the tiles that differ once more, counted in registers; all of the CTA's when
  // there are too many to list.  (64, 128, 96, 85) perm (3, 1, 0, 2) float32, host
  // time of a check: no wrong element 135 us, 200 of them 148, 1 % 362, all 381; with
  // two shared atomics for every wrong element 138, 161, 698, 4529.
  __syncthreads();
  if (numListed == 0) return;
  const bool all = numListed > VERIFY_LIST;
  const uint32_t n = all ? (p.numTiles - blockIdx.x + gridDim.x - 1) / gridDim.x : numListed;
  const BoxSlot* slot = reinterpret_cast<const BoxSlot*>(smraw + g.st.slotAt);
  const int es = g.es, lastWord = es / 4 - 1, shift = es == 4 ? 0 : es == 8 ? 1 : 2;
  const Place l = placeOf(smraw, g.ld), t = placeOf(smraw, g.st);
  uint32_t sm[SV];
  elementsOf<SV>(smraw, g, sTile + t.sm, sm);
  uint32_t bad = 0;
  unsigned long long first = ~0ull;
  for (uint32_t i = 0; i < n; ++i) {
    long long bin, bout;
    const uint32_t shared =
        tileCorner(p, all ? blockIdx.x + i * gridDim.x : listed[i], bin, bout);
    loadInput(smraw, g, l, bin, sTile);
    cpAsyncWaitAll();
    __syncthreads();
    const unsigned char* out = g.out + bout * es;
#pragma unroll 1
    for (int k = 0; k < t.slots; ++k) {
      const BoxSlot at = slot[k];
      const ST w = ldGlobal<ES * SV>(offsetBytes(out, (int)(t.off + at.off), es));
      T e[SV];
#pragma unroll
      for (int m = 0; m < SV; ++m) e[m] = ldShared<ES>(sm[m] + at.sm);
      uint32_t a[ES * SV / 4], b[ES * SV / 4];
      __builtin_memcpy(a, e, ES * SV);
      __builtin_memcpy(b, &w, ES * SV);
      uint32_t differ = 0;
#pragma unroll
      for (int x = 0; x < ES * SV / 4; ++x) {
        differ |= a[x] ^ b[x];
        if ((x & lastWord) != lastWord) continue;
        const uint32_t o = t.off + at.off + (uint32_t)(x >> shift);
        if (differ != 0 && owns(p, shared, o)) {
          ++bad;
          first = min(first, (unsigned long long)bout + o);
        }
        differ = 0;
      }
    }
    __syncthreads();
  }
  // one pair of shared atomics a warp
  bad = __reduce_add_sync(~0u, bad);
#pragma unroll
  for (int x = 16; x > 0; x >>= 1) first = min(first, __shfl_xor_sync(~0u, first, x));
  if (threadIdx.x % 32 == 0 && bad > 0) {
    atomicAdd(&found.bad, (unsigned long long)bad);
    atomicMin(&found.first, first);
  }
  __syncthreads();
  if (threadIdx.x == 0) report(found.bad, found.first, result);
}

// Replays the tile's map (verify_map.h), one CTA, next to the check itself: it is
// launched dependently behind that and touches none of the tensors.  Inside the
// check's kernel, as its last CTA's first work, it cost the others registers (135 ->
// 149 us for 256 MB); behind it 1 to 3 us of any check.
template <int ES, int SV>
__global__ void __launch_bounds__(TILE_THREADS)
verifyMapKernel(const __grid_constant__ VerifyTiles p, unsigned long long* result) {
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ int count[3];  // loaded, compared, marked
  uint32_t* cell = reinterpret_cast<uint32_t*>(smraw + p.blockBytes);
  const uint32_t smBytes = (uint32_t)p.smBytes;
  for (uint32_t i = threadIdx.x; i < smBytes / 4; i += TILE_THREADS) cell[i] = CELL_EMPTY;
  for (int c = threadIdx.x; c < p.blockBytes / 16; c += TILE_THREADS)
    reinterpret_cast<uint4*>(smraw)[c] = p.block[c];
  if (threadIdx.x < 3) count[threadIdx.x] = 0;
  __syncthreads();
  int loaded = 0, compared = 0, marked = 0;
  bool ok = mapLoads(smraw, threadIdx.x, smBytes, loaded,
                     [&](uint32_t at, uint32_t v) { cell[at / 4] = v; });
  __syncthreads();
  ok = mapStores<ES, SV>(p.map, smraw, threadIdx.x, smBytes, compared,
                         [&](uint32_t at) { return cell[at / 4]; }) && ok;
  __syncthreads();
  mapMark<ES, SV>(smraw, threadIdx.x, smBytes, [&](uint32_t at) { cell[at / 4] = CELL_USED; });
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < smBytes / 4; i += TILE_THREADS)
    marked += cell[i] == CELL_USED ? 1 : 0;
  loaded = __reduce_add_sync(~0u, loaded);
  compared = __reduce_add_sync(~0u, compared);
  marked = __reduce_add_sync(~0u, marked);
  if (threadIdx.x % 32 == 0) {
    atomicAdd(&count[0], loaded);
    atomicAdd(&count[1], compared);
    atomicAdd(&count[2], marked);
  }
  ok = __syncthreads_and(ok) != 0;
  ok = ok && count[0] == p.map.vol && count[1] == p.map.vol && count[2] == p.map.vol;
  if (!ok && threadIdx.x == 0) atomicAdd_system(result + 2, 1ull);
  dependencyWait();
}


using VerifyKernel = void (*)(const VerifyTiles, unsigned long long*);

// The check's kernel and its map's.
struct VerifyKernels {
  VerifyKernel tiles = nullptr, map = nullptr;
};

VerifyKernels verifyKernelsOf(int store) {
  switch (store) {
#define LT_VERIFY(ES, SV) \
  case blockStore(ES, SV): return {verifyTilesKernel<ES, SV>, verifyMapKernel<ES, SV>};
    LT_VERIFY(4, 4)
    LT_VERIFY(4, 1)
    LT_VERIFY(8, 2)
    LT_VERIFY(8, 1)
    LT_VERIFY(16, 1)
#undef LT_VERIFY
    default: return {};
  }
}

// Launches the check over tiles and the replay of their map; an error where one of
// them cannot be launched (the check may have been).
cudaError_t checkTiles(const VerifyTiles& tiles, int sms, int smem, unsigned long long* d,
                       cudaStream_t s) {
  const VerifyKernels k = verifyKernelsOf(reinterpret_cast<const TileBlock*>(tiles.block)->store);
  if (k.tiles == nullptr) return cudaErrorInvalidConfiguration;
  const int occ = cachedOccupancy((const void*)k.tiles, TILE_THREADS, smem);
  if (occ < 1 || cachedOccupancy((const void*)k.map, TILE_THREADS, smem) < 1)
    return cudaErrorInvalidConfiguration;
  k.tiles<<<std::min(tiles.numTiles, (uint32_t)(sms * occ)), TILE_THREADS, smem, s>>>(tiles, d);
  const cudaError_t err = cudaGetLastError();
  return err != cudaSuccess ? err : launchDependent(k.map, 1, TILE_THREADS, smem, s, tiles, d);
}

// Adds a grid rank: chunks of ext along dim, the last one ending at dim.
void addGridRank(int64_t dim, int64_t ext, int64_t sin, int64_t sout, VerifyTiles& p) {
  const int g = p.nGR++;
  p.grDiv[g] = makeFastDiv((uint32_t)((dim + ext - 1) / ext));
  p.grSin[g] = ext * sin;
  p.grSout[g] = ext * sout;
  p.grLastIn[g] = (dim - ext) * sin;
  p.grLastOut[g] = (dim - ext) * sout;
  // extents of 2 and more have strides below 2^31 (the tile's span is)
  p.overlap[g] = dim % ext != 0 ? (uint32_t)(ext - dim % ext) : 0;
  if (p.overlap[g] == 0) return;
  p.outStep[g] = makeFastDiv((uint32_t)sout);
  p.outDim[g] = dim < (int64_t(1) << 31) ? makeFastDiv((uint32_t)dim) : FastDiv{};
}

// Fills p for a check of in against out; the kernel's shared memory returned,
// 0 when the problem has no tile with a box.
int verifyTiles(const Fused& f, int sms, const void* in, const void* out, VerifyTiles& p) {
  // for a small tensor, whose check takes less time than ranking the planner's
  // tiles (7 us of host time), the planner's first tile
  const bool few = f.vol * f.esize < (4 << 20);
  std::vector<PlanDesc> c = flatTileCandidates(f, sms, true, few ? 1 : 0);
  if (c.empty()) return 0;
  PlanDesc pd = c[chooseHeuristic(c)];
  if (!refineCandidate(pd, sms)) return 0;
  const GroupRunSplit rs = groupRunSplit(pd.tile);
  if (((uintptr_t)in | (uintptr_t)out) % 16 != 0 || rs.inRun % pd.tile.lv || rs.outRun % pd.tile.sv) {
    if (!finalizePlan(pd)) return 0;
    pd.tile = pd.tileScalar;
  }
  const TileParams& tp = pd.tile;
  static thread_local BoxParams b;
  if (!makeBox(tp, f.esize, b, false)) return 0;
  // The grid from the extents; the tile only says in which order its ranks go.
  int64_t tiles = 1;
  p.nGR = 0;
  uint32_t seen = 0;
  for (int g = 0; g < tp.nGR; ++g) {
    int r = 0;  // input strides of a chunk differ between ranks
    while (r < f.rank && (pd.extent[r] * f.sin[r] != tp.grSin[g] || pd.extent[r] >= f.dim[r])) ++r;
    if (r == f.rank || (seen >> r & 1) != 0) return 0;
    seen |= 1u << r;
    addGridRank(f.dim[r], pd.extent[r], f.sin[r], f.sout[r], p);
    tiles *= p.grDiv[g].d;
    if (tiles >= (int64_t(1) << 31)) return 0;
  }
  for (int r = 0; r < f.rank; ++r)  // every other rank lies in the tile whole
    if ((seen >> r & 1) == 0 && pd.extent[r] != f.dim[r]) return 0;
  p.numTiles = (uint32_t)tiles;
  p.smBytes = b.smBytes;
  p.map = makeTileMap(f, pd.extent);
  const std::vector<unsigned char> block =
      packBlock(b, f.esize, in, const_cast<void*>(out));
  p.blockBytes = (int)block.size();
  std::memcpy(p.block, block.data(), block.size());
  return p.blockBytes + b.smBytes;
}

// As verifyTiles; 0 also where the host has no memory for the choice of a tile.
int verifyTilesOrNone(const Fused& f, int sms, const void* in, const void* out,
                      VerifyTiles& p) noexcept {
  try {
    return verifyTiles(f, sms, in, out, p);
  } catch (const std::exception&) {
    return 0;
  }
}

// A call's result: three zeroed words (wrong elements, the complement of the first
// one's index, whether the tile's map failed) of mapped host memory that the kernel adds
// to and the host reads after its synchronisation, so that a call makes no
// device allocation, memset or copy (together 150 us a call, with the default
// pool giving its memory back at every synchronisation).  The slots lie in one page
// of the process's own memory, registered with CUDA by the first call and again by
// the first one after a cudaDeviceReset, which ends the registration; a call
// beyond the page's slots allocates its own.
class ResultSlot {
 public:
  ResultSlot() {
    {
      std::lock_guard<std::mutex> lk(mutex());
      std::vector<unsigned long long*>& f = freeSlots();
      static const bool made = addPage(f);
      if (made && !f.empty()) {
        p_ = f.back();
        f.pop_back();
      }
    }
    if (p_ != nullptr) d_ = pageAddress();
    if (d_ == nullptr) {
      giveBack();
      own_ = p_ = allocate();
      d_ = address();
    }
    if (p_ != nullptr) clear();
  }
  ~ResultSlot() {
    if (own_ != nullptr) {
      const Uncaptured relaxed;
      cudaFreeHost(own_);
    } else {
      giveBack();
    }
  }
  ResultSlot(const ResultSlot&) = delete;
  ResultSlot& operator=(const ResultSlot&) = delete;
  volatile unsigned long long* host() const { return p_; }
  void clear() { p_[0] = p_[1] = p_[2] = 0; }
  // Its address on the current device, nullptr when there is none.
  unsigned long long* device() const { return d_; }

 private:
  static constexpr size_t SLOTS = 64, SLOT = 64;  // bytes of a slot
  // Allocating and registering is no error, and ends no capture, while another
  // thread captures a stream.
  struct Uncaptured {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    Uncaptured() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~Uncaptured() { cudaThreadExchangeStreamCaptureMode(&mode); }
  };
  static unsigned long long* allocate() {
    const Uncaptured relaxed;
    void* p = nullptr;
    const unsigned flags = cudaHostAllocMapped | cudaHostAllocPortable;
    if (cudaHostAlloc(&p, SLOT, flags) == cudaSuccess) return static_cast<unsigned long long*>(p);
    cudaGetLastError();
    return nullptr;
  }
  // Whole pages of their own, so that no other registration touches them.
  static bool addPage(std::vector<unsigned long long*>& f) {
    const long unit = sysconf(_SC_PAGESIZE);
    pageBytes() = (SLOTS * SLOT + unit - 1) / unit * unit;
    try {
      f.reserve(SLOTS);  // for good: giving a slot back needs no memory
    } catch (const std::exception&) {
      return false;
    }
    if (posix_memalign(&page(), (size_t)unit, pageBytes()) != 0) return false;
    for (size_t k = 0; k < SLOTS; ++k)
      f.push_back(reinterpret_cast<unsigned long long*>(static_cast<char*>(page()) + k * SLOT));
    return true;
  }
  unsigned long long* address() const {
    void* d = nullptr;
    if (p_ == nullptr) return nullptr;
    if (cudaHostGetDevicePointer(&d, p_, 0) == cudaSuccess) return static_cast<unsigned long long*>(d);
    cudaGetLastError();  // not registered
    return nullptr;
  }
  unsigned long long* pageAddress() const {
    if (unsigned long long* d = address()) return d;
    const Uncaptured relaxed;
    // (an error when another thread was faster)
    if (cudaHostRegister(page(), pageBytes(), cudaHostRegisterMapped | cudaHostRegisterPortable) !=
        cudaSuccess)
      cudaGetLastError();
    return address();
  }
  void giveBack() {
    if (p_ == nullptr) return;
    std::lock_guard<std::mutex> lk(mutex());
    freeSlots().push_back(p_);
    p_ = nullptr;
  }
  static std::mutex& mutex() {
    static std::mutex m;
    return m;
  }
  static std::vector<unsigned long long*>& freeSlots() {
    // lives until the process exits
    alignas(std::vector<unsigned long long*>) static unsigned char place[sizeof(
        std::vector<unsigned long long*>)];
    static auto* f = new (place) std::vector<unsigned long long*>();
    return *f;
  }
  static void*& page() {
    static void* p = nullptr;
    return p;
  }
  static size_t& pageBytes() {
    static size_t n = 0;
    return n;
  }
  unsigned long long *p_ = nullptr, *own_ = nullptr, *d_ = nullptr;
};

}  // namespace
}  // namespace lt

namespace lt {
namespace {

// mapIsSound on the host.
template <int ES, int SV>
bool mapIsSoundHost(const VerifyTiles& p, const unsigned char* block) {
  std::vector<uint32_t> cells(p.smBytes / 4, CELL_EMPTY);
  int loaded = 0, compared = 0;
  bool ok = true;
  const uint32_t smBytes = (uint32_t)p.smBytes;
  for (uint32_t t = 0; t < TILE_THREADS; ++t)
    ok = mapLoads(block, t, smBytes, loaded, [&](uint32_t at, uint32_t v) { cells[at / 4] = v; }) && ok;
  for (uint32_t t = 0; t < TILE_THREADS; ++t)
    ok = mapStores<ES, SV>(p.map, block, t, smBytes, compared,
                           [&](uint32_t at) { return cells[at / 4]; }) && ok;
  for (uint32_t t = 0; t < TILE_THREADS; ++t)
    mapMark<ES, SV>(block, t, smBytes, [&](uint32_t at) { cells[at / 4] = CELL_USED; });
  const int marked = (int)std::count(cells.begin(), cells.end(), CELL_USED);
  return ok && loaded == p.map.vol && compared == p.map.vol && marked == p.map.vol;
}

bool mapIsSoundHost(const VerifyTiles& p) {
  const unsigned char* block = reinterpret_cast<const unsigned char*>(p.block);
  switch (reinterpret_cast<const TileBlock*>(block)->store) {
    case blockStore(4, 4): return mapIsSoundHost<4, 4>(p, block);
    case blockStore(4, 1): return mapIsSoundHost<4, 1>(p, block);
    case blockStore(8, 2): return mapIsSoundHost<8, 2>(p, block);
    case blockStore(8, 1): return mapIsSoundHost<8, 1>(p, block);
    default: return mapIsSoundHost<16, 1>(p, block);
  }
}

// Every tile's corner is the formula's, and the elements that the tiles own add up
// to the tensor.
bool gridIsSound(const Fused& f, const VerifyTiles& p) {
  uint64_t owned = 0;
  for (uint32_t tile = 0; tile < p.numTiles; ++tile) {
    long long bin, bout;
    uint32_t shared = tileCorner(p, tile, bin, bout);
    long long rem = bout, src = 0;
    uint64_t mine = 1;
    uint32_t ranks = 0;
    for (int i = 0; i < f.rank; ++i) {
      const int r = f.perm[i];
      const long long c = rem % f.dim[r];
      if (c + p.map.ext[i] > f.dim[r]) return false;
      src += c * f.sin[r];
      rem /= f.dim[r];
      // the rank's first digits, where the tile before owns them
      uint64_t digits = p.map.ext[i];
      for (int g = 0; g < p.nGR; ++g)
        if ((shared >> g & 1) != 0 && p.outStep[g].d == (uint64_t)f.sout[r]) {
          digits -= p.overlap[g];
          ranks |= 1u << g;
        }
      mine *= digits;
    }
    if (src != bin || rem != 0 || ranks != shared) return false;
    owned += mine;
  }
  return owned == (uint64_t)f.vol;
}

// Plants mistake 1 .. 9 in a check's addressing; false where it has no place.
bool plant(int mistake, VerifyTiles& p) {
  unsigned char* block = reinterpret_cast<unsigned char*>(p.block);
  TileBlock& g = *reinterpret_cast<TileBlock*>(block);
  BoxSlot* ld = reinterpret_cast<BoxSlot*>(block + g.ld.slotAt);
  BoxSlot* st = reinterpret_cast<BoxSlot*>(block + g.st.slotAt);
  BoxRank* rank = reinterpret_cast<BoxRank*>(block + g.ld.rankAt);
  switch (mistake) {
    case 1:  // two slots' input, exchanged: every element still arrives somewhere
      if (g.ld.nFull < 2) return false;
      std::swap(ld[0].off, ld[1].off);
      return true;
    case 2:  // two slots' places in shared memory, exchanged
      if (g.st.nFull < 2) return false;
      std::swap(st[0].sm, st[1].sm);
      return true;
    case 3:  // the output of a slot
      if (g.st.nFull < 2) return false;
      st[0].off = st[1].off;
      return true;
    case 4:  // a step of the input
      rank[0].step += 1;
      return g.ld.active > 1 && (g.ld.p == 0 || (int)rank[0].ext > g.ld.unit);
    case 5:  // elements left out
      if (g.st.nFull < 1) return false;
      g.st.nFull -= 1;
      return true;
    case 6:  // elements left out on both sides
      if (g.ld.nFull < 1) return false;
      g.ld.active -= 1;
      g.st.active -= 1;
      return true;
    case 7:  // a corner
      if (p.nGR < 1) return false;
      p.grSin[0] += 1;
      return p.grDiv[0].d > 2;
    case 8:  // a tile left out
      p.numTiles -= 1;
      return p.numTiles > 0;
    case 9:  // an overlap counted twice
      for (int r = 0; r < p.nGR; ++r)
        if (p.overlap[r] > 0) {
          p.overlap[r] -= 1;
          return true;
        }
      return false;
    default: return false;
  }
}

}  // namespace
}  // namespace lt

extern "C" int librett_c_verify_map_check(int rank, const int* dim, const int* permutation,
                                          size_t sizeofType, int num_sms, int element_units,
                                          int mistake) {
  if (lt::checkInput(rank, dim, permutation, sizeofType) != 0 || mistake < 0 || mistake > 9)
    return LIBRETT_INVALID_PARAMETER;
  lt::Fused f;
  lt::fuseRanks(rank, dim, permutation, (int)sizeofType, f);
  static thread_local lt::VerifyTiles tiles;
  const uintptr_t at = element_units ? 4096 + sizeofType % 16 : 4096;  // addresses, not followed
  if (lt::verifyTilesOrNone(f, num_sms > 0 ? num_sms : 152, reinterpret_cast<const void*>(at),
                      reinterpret_cast<const void*>(2 * at), tiles) <= 0 ||
      (mistake > 0 && !lt::plant(mistake, tiles)))
    return LIBRETT_INVALID_DEVICE;
  return lt::mapIsSoundHost(tiles) && lt::gridIsSound(f, tiles) ? LIBRETT_SUCCESS
                                                                 : LIBRETT_INTERNAL_ERROR;
}

extern "C" int librett_c_verify(int rank, const int* dim, const int* permutation,
                                size_t sizeofType, const void* idata, const void* odata,
                                void* stream, unsigned long long* mismatches,
                                long long* first_bad) {
  if (lt::checkInput(rank, dim, permutation, sizeofType) != 0 || idata == nullptr ||
      odata == nullptr || mismatches == nullptr)
    return LIBRETT_INVALID_PARAMETER;
  const size_t a = sizeofType < 16 ? sizeofType : 16;
  if ((uintptr_t)idata % a || (uintptr_t)odata % a) return LIBRETT_INVALID_PARAMETER;
  lt::Fused f;
  lt::fuseRanks(rank, dim, permutation, (int)sizeofType, f);
  int sms = 0, dev = 0;
  if (!lt::currentDevice(dev, sms)) return LIBRETT_INTERNAL_ERROR;
  cudaStream_t s = (cudaStream_t)stream;
  lt::ResultSlot slot;
  unsigned long long* d = slot.device();
  if (d == nullptr) return LIBRETT_INTERNAL_ERROR;
  static thread_local lt::VerifyTiles tiles;
  const int smem = lt::verifyTilesOrNone(f, sms, idata, odata, tiles);
  cudaError_t err = smem > 0 ? lt::checkTiles(tiles, sms, smem, d, s) : cudaErrorInvalidConfiguration;
  // also after an error: a launch may have been made
  cudaError_t done = cudaStreamSynchronize(s);
  // Element by element: without a tile, where its map is not the formula's, or where a
  // launch was refused
  const bool refused = err == cudaErrorInvalidConfiguration || err == cudaErrorInvalidValue;
  if (done == cudaSuccess && (refused || (err == cudaSuccess && slot.host()[2] != 0))) {
    slot.clear();
    cudaGetLastError();  // of what was refused
    err = lt::verifyElements(f, sms, idata, odata, d, s);
    done = cudaStreamSynchronize(s);
  }
  if (err != cudaSuccess || done != cudaSuccess) return LIBRETT_INTERNAL_ERROR;
  const unsigned long long host[2] = {slot.host()[0], slot.host()[1]};
  *mismatches = host[0];
  if (first_bad) *first_bad = host[0] ? (long long)~host[1] : -1;
  return LIBRETT_SUCCESS;
}
