// How the batched affine accumulation of G2 (msm.cu) cuts a sorted list into
// tiles and lays out the scratch of a resident block.  Plain integer C++: the
// same code runs in the kernels and in a CPU test.
#pragma once
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define ZK_HDI __host__ __device__ __forceinline__
#else
#define ZK_HDI inline
#endif

namespace zk {

constexpr int kAffT = 128;      // threads per block
constexpr int kAffMaxSub = 3;   // sub-segments per thread
constexpr int kSub = 64;        // points per sub-segment, at most (a 64-bit mask)
constexpr int kAffMinS = 32;    // records per thread, at least
constexpr int kAffPoint = 128;  // bytes of an affine G2 point
constexpr int kAffPair = 64;    // bytes of a pair's prefix product and norm

// Slots of a sub-segment of len points: buffer 1 takes the first round's
// results, buffer 0 the second's, and so on in turn.  A round about halves the
// points, so these hold all but the shortest runs; up to eight points fit
// whatever their runs.
ZK_HDI int aff_slots(int len, int buf) {
  const int need = buf ? len - len / 4 : len / 2, all = len < 8 ? len : 8;
  return need < all ? all : need;
}

// Layout of one resident block's scratch, interleaved by thread, for at most
// S records per thread: full sub-segments and a last one of what is left, so
// the scratch grows with S and not in steps of 64 (2^18 points with 17-bit
// tables, S = 70: 0.8 GB a wave, 1.4 GB with a full second sub-segment).
// Equal sub-segments (2 x 36) cost 2.6 % of that MSM's time.
struct AffShape {
  int nsub;       // sub-segments per thread
  int slots[2];   // slots of a full sub-segment
  int last[2];    // and of the last one
  int rows;       // slots per thread of buffer 0
  uint32_t pre;   // byte offsets of the pairs' prefixes and norms,
  uint32_t mask;  // of the masks
  uint32_t state; // and of the final state
  uint32_t bytes;
  ZK_HDI int limit(int h, int buf) const { return h + 1 < nsub ? slots[buf] : last[buf]; }
};
ZK_HDI AffShape aff_shape(int S) {
  AffShape a;
  a.nsub = (S + kSub - 1) / kSub;
  const int full = a.nsub - 1, len = S - full * kSub;
  for (int buf = 0; buf < 2; buf++) {
    a.slots[buf] = aff_slots(kSub, buf);
    a.last[buf] = aff_slots(len, buf);
  }
  a.rows = full * a.slots[0] + a.last[0];
  const uint32_t points = (uint32_t)(a.rows + full * a.slots[1] + a.last[1]);
  const uint32_t pairs = (uint32_t)(full * (kSub / 2) + len / 2);
  a.pre = kAffT * kAffPoint * points;
  a.mask = a.pre + kAffT * kAffPair * pairs;
  a.state = a.mask + kAffT * 3 * (uint32_t)(a.nsub * sizeof(uint64_t));
  a.bytes = a.state + kAffT * (uint32_t)sizeof(uint32_t);
  return a;
}

static_assert(kAffMaxSub * kSub < 256 && kAffMinS % 4 == 0, "layout of the affine scratch");

// Records per thread (even) of a list of `total` over ntiles tiles: spread
// evenly by the actual number, so skewed scalars, whose zero digits make no
// records, leave no tile idle.
ZK_HDI int aff_span(size_t total, uint32_t ntiles) {
  const size_t lanes = (size_t)ntiles * kAffT;
  const int S = ((int)((total + lanes - 1) / lanes) + 1) & ~1;
  return S < kAffMinS ? kAffMinS : S;
}

}  // namespace zk
