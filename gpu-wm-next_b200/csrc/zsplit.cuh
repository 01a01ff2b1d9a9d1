// zsplit.cuh — how the columns of a grid are split over CTAs in the kernels that march up
// in k.
#pragma once

#include <algorithm>
#include <cuda_runtime.h>

namespace gwmb {

// Chunk z of a column: the first `nbig` chunks hold `big` levels, the others `small`.  The
// grid's z index is its slowest, so the long chunks start first and the short ones fill the
// last wave.
struct ZSplit {
  int big, nbig, small, chunks;
  __host__ __device__ int first(int z) const { return z < nbig ? z * big : nbig * big + (z - nbig) * small; }
  __host__ __device__ int last(int z, int nz) const {  // one past the chunk's last level
    const int e = first(z) + (z < nbig ? big : small);
    return e < nz ? e : nz;
  }
  int longest() const { return std::max(big, small); }
};

inline int sm_count() {
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
    return 148;
  return sms;
}

// The split for `tiles` tiles of nz levels on `slots` resident CTAs (SMs x CTAs per SM).
// With all levels in one CTA a small grid leaves most SMs idle and its plane loop is a serial
// chain of nz plane latencies; a large grid of few waves idles in its last one (the acoustic
// substep of 768 x 768 x 64, 1.95 waves: SMs active 70 % of the time).  A chunk costs its
// levels and `extra` more (start-up, the plane below it), so with every slot kept busy until
// the last chunks the kernel takes, in plane times,
//   sum over chunks (levels + extra) * tiles / slots + (last chunk's levels + extra),
// and never less than its longest chunk.  Uniform splits measured against that (1024^2 x 64
// acoustic substep, chunks of 64, 32, 22, 16, 11, 8 levels: 681, 619, 599, 595, 590, 600 us;
// the formula with extra = 0.7: 681, 611, 593, 583, 585, 590).
// Chunks go down to one level: two tiles of 40 levels (32 x 32 x 40) still fill 80 SMs with one
// CTA each, 10.6 us a substep and 16.2 us a slow stage against 12.8 and 20.8 in chunks of two.
inline ZSplit z_split_search(unsigned tiles, int nz, int slots, float extra) {
  const float load = (float)tiles / (float)slots;
  // with fewer tiles than slots a chunk's start-up has less to hide behind
  extra += 2.0f * std::max(0.0f, 1.0f - load);
  ZSplit best{nz, 1, nz, 1};
  float least = 0.0f;
  auto consider = [&](int big, int nbig, int small) {
    const int rest = nz - big * nbig;
    const int nsmall = rest > 0 ? (rest + small - 1) / small : 0;
    const int chunks = nbig + nsmall;
    const int end = rest > 0 ? small : big;
    // all chunks resident at once: no second wave to wait for (measured 0.62 of the load)
    const float share = load * (float)chunks <= 1.0f ? 0.62f : 1.0f;
    const float busy = ((float)nz + extra * (float)chunks) * load * share + (float)end + extra;
    const float cost = std::max(busy, (float)big + extra + 2.0f * load);
    if (least == 0.0f || cost < 0.99f * least) {
      least = cost;
      best = ZSplit{big, nbig, small, chunks};
    }
  };
  for (int n = 1; n <= nz; ++n) {
    const int big = (nz + n - 1) / n;
    consider(big, (nz + big - 1) / big, big);  // uniform
    if (n > 6 || load < 0.9f) continue;  // one uneven wave gains nothing
    for (int nbig = 1; nbig < n; ++nbig)  // long chunks, then a few short ones
      for (int m = 1; m <= 8; ++m) {
        const int rest = nz - big * nbig, small = (rest + m - 1) / m;
        if (rest > 0 && small >= 2 && small < big) consider(big, nbig, small);
      }
  }
  return best;
}
// Results kept: they depend on the arguments alone.  256 of them, in sets of four: an ensemble of
// uneven members asks for a handful per member and step, and a search takes 2.5 to 6 us.
struct SplitMemo {
  struct Entry {
    unsigned tiles = 0;
    int nz = 0, slots = 0;
    float extra = 0.0f;
    ZSplit s{};
  };
  static constexpr unsigned kSets = 64, kWays = 4;
  Entry entry[kSets][kWays];
  unsigned char next[kSets] = {};  // the way of a set that is replaced next
  unsigned searches = 0;
  ZSplit get(unsigned tiles, int nz, int slots, float extra) {
    const unsigned h = (tiles * 0x9e3779b1u) ^ ((unsigned)nz * 0x85ebca77u) ^ ((unsigned)slots * 0xc2b2ae3du) ^
                       ((unsigned)(extra * 1024.0f) * 0x27d4eb2fu);
    const unsigned set = h >> 26;
    for (const Entry& e : entry[set])
      if (e.tiles == tiles && e.nz == nz && e.slots == slots && e.extra == extra) return e.s;
    ++searches;
    Entry& e = entry[set][next[set]++ % kWays];
    e = Entry{tiles, nz, slots, extra, z_split_search(tiles, nz, slots, extra)};
    return e.s;
  }
};
inline ZSplit z_split(unsigned tiles, int nz, int ctas_per_sm, float extra) {
  thread_local SplitMemo memo;
  return memo.get(tiles, nz, sm_count() * ctas_per_sm, extra);
}

}  // namespace gwmb
