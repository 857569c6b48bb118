// Host side of box addressing (box.h): the side builders and the choice of
// the shared-memory layout.
#include "box.h"

#include <algorithm>
#include <cstring>
#include <numeric>

namespace lt {
namespace {

struct Ranks {
  int n = 0;
  int ext[BOX_RANKS];
  uint32_t step[BOX_RANKS], stepS[BOX_RANKS];
  // Appends a rank, merging it into the last one when it continues it.
  void add(int e, uint32_t st, uint32_t ss) {
    if (n > 0 && st == (uint32_t)ext[n - 1] * step[n - 1] &&
        ss == (uint32_t)ext[n - 1] * stepS[n - 1]) {
      ext[n - 1] *= e;
      return;
    }
    ext[n] = e;
    step[n] = st;
    stepS[n++] = ss;
  }
};

// One side with units of V elements; false when the box cannot be cut at a
// unit boundary or needs too many slots.
bool buildSide(const Ranks& r, int V, BoxSide& s) {
  const int T = TILE_THREADS * V;
  int p = 0, Q = 1;  // the top rank, the volume below it
  while (p + 1 < r.n && Q * r.ext[p] <= T) Q *= r.ext[p++];
  if ((Q * r.ext[p]) % V != 0) return false;
  int rho = std::min(r.ext[p], T / Q);  // of the top rank, in the box
  if (rho < r.ext[p]) rho -= rho % (V / std::gcd(Q, V));
  if (rho < 1 || (Q * rho) % V != 0) return false;
  for (int k = 0; k <= p; ++k) {
    const uint32_t mul = (uint32_t)(((uint64_t(1) << 32) + r.ext[k] - 1) / r.ext[k]);
    s.rank[k] = {mul, (uint32_t)r.ext[k], r.step[k], r.stepS[k]};
  }
  const int whole = r.ext[p] / rho;
  int outer = 1;
  for (int k = p + 1; k < r.n; ++k) outer *= r.ext[k];
  s.h.unit = V;
  s.h.active = Q * rho / V;
  s.h.p = p;
  s.h.rem = r.ext[p] - whole * rho;
  s.h.nFull = outer * whole;
  s.h.nRagged = s.h.rem > 0 ? outer : 0;
  if (s.h.nFull + s.h.nRagged > BOX_SLOTS) return false;
  int full = 0, ragged = s.h.nFull;
  for (int o = 0; o < outer; ++o) {
    uint32_t off = 0, sm = 0;
    for (int k = p + 1, x = o; k < r.n; ++k) {
      off += (uint32_t)(x % r.ext[k]) * r.step[k];
      sm += (uint32_t)(x % r.ext[k]) * r.stepS[k];
      x /= r.ext[k];
    }
    for (int ch = 0; ch < whole; ++ch)
      s.slot[full++] = {off + (uint32_t)(ch * rho) * r.step[p], sm + (uint32_t)(ch * rho) * r.stepS[p]};
    if (s.h.rem > 0)
      s.slot[ragged++] = {off + (uint32_t)(whole * rho) * r.step[p],
                          sm + (uint32_t)(whole * rho) * r.stepS[p]};
  }
  return true;
}

// Wavefronts of one warp access: lane l touches `bytes` consecutive bytes at
// addr[l] (all lanes of a phase distinct); a phase is 128 bytes' worth of
// lanes and costs the largest number of its words in one bank.
int accessCost(const uint32_t* addr, int lanes, int bytes) {
  const int words = bytes / 4, perPhase = 32 / words;
  int cost = 0;
  for (int l0 = 0; l0 < lanes; l0 += perPhase) {
    unsigned char cnt[32] = {};
    int most = 0;
    for (int l = l0; l < std::min(lanes, l0 + perPhase); ++l) {
      // aligned groups of `words` banks
      unsigned char& c = cnt[(addr[l] / (unsigned)bytes) % (32u / words)];
      most = std::max<int>(most, ++c);
    }
    cost += most;
  }
  return cost;
}

// A candidate layout: pad elements after tile rank `after` (input order), or,
// with split, after `split` rows of the output-fastest rank.
struct Layout {
  int after, pad, split;
};

struct Built {
  Ranks ld, st;
  int vol;            // padded elements
  uint32_t elemStep;  // shared step of the output-fastest rank
};

// Ranks of both sides under a layout (shared steps in bytes).  blockV > 1: the
// store side in blocks of blockV along its fastest rank and input rank 0.
void applyLayout(const TileParams& tp, int esize, const Layout& L, int blockV, Built& b) {
  uint32_t P[MAXR], PS = 0;  // stride of each tile rank; of the split rank's upper part
  const int t0 = tp.trOut[0];
  int s = 1, last = 0;
  for (int t = 0; t < tp.nTR; ++t) {
    P[t] = (uint32_t)(s * esize);
    last += (tp.trE[t] - 1) * s;
    if (L.split > 0 && t == t0) {
      const int up = L.split * s + L.pad, n = tp.trE[t] / L.split;
      PS = (uint32_t)(up * esize);
      last += (n - 1) * L.pad;
      s = up * n;
    } else {
      s *= tp.trE[t];
      if (L.split == 0 && t == L.after) s += L.pad;
    }
  }
  b.vol = last + 1;
  b.ld.n = b.st.n = 0;
  auto add = [&](Ranks& r, int t, const int* gl) {
    if (L.split > 0 && t == t0) {
      r.add(L.split, (uint32_t)gl[t], P[t]);
      if (tp.trE[t] > L.split) r.add(tp.trE[t] / L.split, (uint32_t)(L.split * gl[t]), PS);
    } else {
      r.add(tp.trE[t], (uint32_t)gl[t], P[t]);
    }
  };
  for (int t = 0; t < tp.nTR; ++t) add(b.ld, t, tp.trSin);
  for (int i = 0; i < tp.nTR; ++i) {
    const int t = tp.trOut[i];
    if (blockV > 1 && (t == t0 || t == 0)) {
      const uint32_t so = (uint32_t)blockV * (uint32_t)tp.trSout[t];
      if (t == t0 && L.split > 0) {
        if (L.split > blockV) b.st.add(L.split / blockV, so, (uint32_t)blockV * P[t]);
        if (tp.trE[t] > L.split)
          b.st.add(tp.trE[t] / L.split, (uint32_t)L.split * (uint32_t)tp.trSout[t], PS);
      } else if (tp.trE[t] > blockV) {
        b.st.add(tp.trE[t] / blockV, so, (uint32_t)blockV * P[t]);
      }
    } else {
      add(b.st, t, tp.trSout);
    }
  }
  if (b.st.n == 0) b.st.add(1, 0, 0);  // one block
  b.elemStep = P[t0];
}

// Wavefronts of the first two warps' accesses on both sides; *ideal: without
// a conflict.
int layoutCost(const BoxParams& b, int esize, int* ideal) {
  int cost = 0;
  *ideal = 0;
  uint32_t addr[32], off;
  for (int w = 0; w < 2; ++w) {
    int lanes = std::min(32, b.ld.h.active - 32 * w);
    if (lanes > 0) {
      for (int l = 0; l < lanes; ++l)
        boxDecode(b.ld.rank, b.ld.h.p, (uint32_t)((32 * w + l) * b.ld.h.unit), off, addr[l]);
      cost += accessCost(addr, lanes, b.ld.h.unit * esize);
      *ideal += (lanes * b.ld.h.unit * esize + 127) / 128;
    }
    lanes = std::min(32, b.st.h.active - 32 * w);
    if (b.block && lanes > 0) {
      for (int l = 0; l < lanes; ++l)
        boxDecode(b.st.rank, b.st.h.p, (uint32_t)(32 * w + l), off, addr[l]);
      cost += accessCost(addr, lanes, 16);  // the V reads are shifted copies
      *ideal += (lanes * 16 + 127) / 128;
      continue;
    }
    const int reads = b.wide ? 1 : b.st.h.unit, bytes = b.wide ? b.st.h.unit * esize : esize;
    for (int m = 0; m < reads && lanes > 0; ++m) {
      for (int l = 0; l < lanes; ++l) {
        if (m == 0 || b.straddle)
          boxDecode(b.st.rank, b.st.h.p, (uint32_t)((32 * w + l) * b.st.h.unit + m), off, addr[l]);
        else
          addr[l] += b.elemStep;
      }
      cost += accessCost(addr, lanes, bytes);
      *ideal += (lanes * bytes + 127) / 128;
    }
  }
  return cost;
}

}  // namespace

bool makeBox(const TileParams& tp, int esize, BoxParams& b, bool blocks) {
  if (tp.nTR < 1) return false;
  const int t0 = tp.trOut[0];
  const int V = 16 / esize;
  b.block = blocks && V > 1 && tp.lv == V && tp.sv == V && t0 != 0 && tp.trE[0] % V == 0 && tp.trE[t0] % V == 0;
  b.colStep = tp.trSout[0];
  auto build = [&](const Layout& L, int sv) {
    Built r;
    applyLayout(tp, esize, L, b.block ? V : 1, r);
    if (b.block) sv = 1;  // an item of the store side is one block
    b.straddle = sv > 1 && tp.trE[t0] % sv != 0;
    b.elemStep = r.elemStep;
    b.smBytes = (r.vol * esize + 15) / 16 * 16;
    // shared memory is what limits the CTAs of an SM: an eighth for padding
    if (8 * r.vol > 9 * tp.tileVol && L.pad > 0) return false;
    if (tp.lv > 1 && (r.ld.step[0] != 1 || r.ld.ext[0] % tp.lv != 0)) return false;
    if (!buildSide(r.ld, tp.lv, b.ld) || !buildSide(r.st, sv, b.st)) return false;
    b.wide = sv > 1 && !b.straddle && b.elemStep == (uint32_t)esize;
    const uint32_t unit = (uint32_t)(sv * esize);
    for (int k = 1; k <= b.st.h.p; ++k) b.wide = b.wide && b.st.rank[k].stepS % unit == 0;
    for (int k = 0; k < b.st.h.nFull + b.st.h.nRagged; ++k)
      b.wide = b.wide && b.st.slot[k].sm % unit == 0;
    return true;
  };
  // Candidate layouts, likeliest first.  The padding keeps load units whole
  // and aligned (multiples of lv, after products that are multiples of lv), and
  // wide store units too.
  Layout cand[24];
  int n = 0;
  const int lv = tp.lv, unit = t0 == 0 ? std::max(lv, tp.sv) : lv;
  if (t0 > 0) {
    // after the rows of a unit; after each row; after a few short rows
    if (tp.sv > 1 && tp.trE[t0] % tp.sv == 0) cand[n++] = {0, lv, tp.sv};
    for (int k = 1; k <= 3; ++k) cand[n++] = {t0 - 1, k * lv, 0};
    for (int k = 2; k <= 32; k *= 2)
      if (k != tp.sv && k < tp.trE[t0] && tp.trE[t0] % k == 0) cand[n++] = {0, lv, k};
  }
  cand[n++] = {-1, 0, 0};
  for (int t = 0; t + 1 < tp.nTR && n < 20; ++t)
    if (t != t0 - 1) {
      cand[n++] = {t, unit, 0};
      cand[n++] = {t, 2 * unit, 0};
    }
  auto whole = [&](const Layout& L) {
    if (L.pad == 0) return true;
    int prod = 1;
    const int last = L.split > 0 ? t0 - 1 : L.after;
    for (int t = 0; t <= last; ++t) prod *= tp.trE[t];
    return prod % lv == 0;
  };
  for (int sv = tp.sv;;) {
    int best = -1, bestCost = 0;
    int tried = -1;  // the layout b holds, whole or in part
    for (int c = 0; c < n; ++c) {
      // (a store unit stays inside a split's lower part)
      if (!whole(cand[c]) || (cand[c].split > 0 && cand[c].split % sv != 0)) continue;
      tried = c;
      if (!build(cand[c], sv)) continue;
      int ideal;
      const int cost = layoutCost(b, esize, &ideal);
      if (best < 0 || cost < bestCost) {
        best = c;
        bestCost = cost;
      }
      if (cost <= ideal) break;
    }
    if (best >= 0) {
      if (tried != best) build(cand[best], sv);
      return true;
    }
    // no box of blocks: units; none cut at a unit boundary: elements
    if (b.block)
      b.block = 0;
    else if (sv > 1)
      sv = 1;
    else
      return false;
  }
}

std::vector<unsigned char> packBlock(BoxParams& b, int esize, const void* in, void* out) {
  auto align16 = [](size_t x) { return (x + 15) / 16 * 16; };
  size_t at = sizeof(TileBlock);
  for (BoxSide* side : {&b.ld, &b.st}) {
    side->h.rankAt = (int)at;
    at = align16(at + (size_t)(side->h.p + 1) * sizeof(BoxRank));
    side->h.slotAt = (int)at;
    at = align16(at + (size_t)(side->h.nFull + side->h.nRagged) * sizeof(BoxSlot));
  }
  std::vector<unsigned char> block(at, 0);
  TileBlock t{};
  t.in = static_cast<const unsigned char*>(in);
  t.out = static_cast<unsigned char*>(out);
  t.ld = b.ld.h;
  t.st = b.st.h;
  t.es = esize;
  t.store = b.block  ? blockStore(esize, 0)
            : b.wide ? blockStore(esize * b.st.h.unit, 1)  // as one element
                     : blockStore(esize, b.st.h.unit);
  t.straddle = b.straddle;
  t.elemStep = b.elemStep;
  t.colStep = b.colStep * esize;
  std::memcpy(block.data(), &t, sizeof(t));
  for (const BoxSide* side : {&b.ld, &b.st}) {
    std::memcpy(block.data() + side->h.rankAt, side->rank, (side->h.p + 1) * sizeof(BoxRank));
    std::memcpy(block.data() + side->h.slotAt, side->slot,
                (side->h.nFull + side->h.nRagged) * sizeof(BoxSlot));
  }
  return block;
}

}  // namespace lt
