// Pippenger MSM on G1 / G2 for sm_100a.  See msm.hpp for the pipeline; the
// reference counterpart is include/msm_g1.cuh:271-926 and
// include/msm_g2.cuh:256-880.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "affine_layout.hpp"
#include "curve_quad.cuh"
#include "host_field.hpp"
#include "msm.hpp"
#include "profile.hpp"
#include "scan.cuh"

namespace zk {
namespace {

constexpr uint32_t kInvalid = 0xffffffffu;
constexpr uint32_t kNeg = 0x80000000u;
// pairs per block in the bucket-reduction block passes
template <class F>
constexpr int red_pairs() { return sizeof(F) == 64 ? 64 : 128; }
// nodes per block (a quad each) of the later levels of the segmented reduction
constexpr int lvl_nodes(bool g2) { return g2 ? 64 : 128; }
template <class F>
constexpr int lvl_nodes() { return lvl_nodes(sizeof(F) == 64); }

// ------------------------------------------------------------------ shape
struct Shape {
  size_t n;
  int c, W;              // window bits, scalar windows
  int Wk;                // bucket sets: W, or one per instance when windows share buckets
                         // (fixed bases)
  bool fixed;            // points carry precomputed 2^(c w) multiples (table of W*n records)
  int inst;              // fixed-base instances sharing the launch (1 otherwise)
  uint32_t B;            // buckets per set (2^(c-1))
  size_t entries;        // W*B + 1 scan entries (last = total)
  size_t records;        // W*n upper bound on sorted records
  int k0, k1, chunk;
  size_t affine;         // tiles of level 0 as batched affine additions (G2; 0: XYZZ)
  int levels;            // segmented-reduction levels (>= 1)
  size_t lvl_records[24];
  size_t lvl_blocks[24];
  int lvl_k[24];         // records per thread of each level
  size_t J;              // bucket-reduction level-1 chunks per window
};

size_t affine_tiles(size_t records, size_t buckets);
size_t affine_scratch(size_t records, size_t tiles);

// n: points (summed over instances for fixed-base multi-instance MSMs)
Shape make_shape(size_t n, bool g2, const MsmConfig& cfg, bool fixed = false, int inst = 1) {
  const int seg_t = g2 ? 64 : 128;
  Shape s{};
  s.n = n;
  s.inst = fixed ? inst : 1;
  s.c = cfg.c > 0 ? cfg.c : msm_default_c(n, g2);
  // the top window holds < c bits, so no carry leaves it; fixed-base MSMs
  // reduce scalars mod r first (254 bits)
  s.fixed = fixed;
  s.W = (fixed ? 254 : 256) / s.c + 1;
  s.Wk = fixed ? s.inst : s.W;
  s.B = 1u << (s.c - 1);
  s.entries = (size_t)s.Wk * s.B + 1;
  s.records = std::max<size_t>((size_t)s.W * n, 1);
  s.k0 = cfg.k0 > 0 ? cfg.k0 : msm_default_k0(n, fixed);
  s.k1 = cfg.k1;
  s.chunk = cfg.chunk > 0 ? cfg.chunk : msm_default_chunk((size_t)s.Wk * s.B, fixed, g2);
  s.J = (s.B + s.chunk - 1) / s.chunk;
  size_t rec = s.records;
  int per_thread = s.k0;
  s.levels = 0;
  s.affine = g2 && cfg.affine ? affine_tiles(s.records, (size_t)s.Wk * s.B) : 0;
  if (s.affine) {
    s.lvl_records[0] = rec;
    s.lvl_blocks[0] = s.affine;
    s.levels = 1;
    rec = 2 * s.affine;
    per_thread = s.k1;
  }
  while (true) {
    // a level that fits one block spreads its records over every thread
    // (its depth is the per-thread run plus the block tree)
    if (s.levels > 0 && rec <= (size_t)seg_t * per_thread)
      per_thread = std::max<int>(2, (int)((rec + seg_t - 1) / seg_t));
    size_t per_block = (size_t)seg_t * per_thread;
    size_t blocks = (rec + per_block - 1) / per_block;
    s.lvl_records[s.levels] = rec;
    s.lvl_blocks[s.levels] = blocks;
    s.lvl_k[s.levels] = per_thread;
    s.levels++;
    if (blocks <= 1 || s.levels == 24) break;
    rec = 2 * blocks;
    per_thread = s.k1;
  }
  return s;
}

template <class F>
struct Layout {
  uint32_t* counts;   // entries (exclusive offsets after the scan), then the tile queue
  uint32_t* tileq;    // work-queue counter of the persistent level 0 (counts[entries])
  uint32_t* cursor;   // entries
  uint32_t* tiles;    // scan tile sums
  uint2* srec;        // records: (bucket key, point index | sign), one 8-byte store each
  xyzz<F>* buckets;   // W*B
  uint32_t* pkey[2];  // ping-pong partial records
  xyzz<F>* ppt[2];
  xyzz<F>* rrun[2];   // bucket-reduction (run, acc) pairs, ping-pong
  xyzz<F>* racc[2];
  xyzz<F>* outua;     // 2 * W: U_0..U_{W-1}, A_0..A_{W-1}
  unsigned char* aff;  // affine accumulation: scratch of its resident blocks
  size_t bytes;
};

template <class F>
Layout<F> carve(void* base, const Shape& s) {
  Layout<F> L{};
  Carver cv(base);
  L.counts = cv.take<uint32_t>(s.entries + 1);
  L.tileq = L.counts + s.entries;
  L.cursor = cv.take<uint32_t>(s.entries);
  L.tiles = cv.take<uint32_t>(scan::tile_count(s.entries) + 1);
  L.srec = cv.take<uint2>(s.records + 1);
  L.buckets = cv.take<xyzz<F>>((size_t)s.Wk * s.B);
  size_t pmax[2] = {1, 1};
  for (int l = 1; l < s.levels; l++) pmax[l & 1] = std::max(pmax[l & 1], s.lvl_records[l]);
  for (int i = 0; i < 2; i++) {
    L.pkey[i] = cv.take<uint32_t>(pmax[i]);
    L.ppt[i] = cv.take<xyzz<F>>(pmax[i]);
  }
  const size_t j2 = (s.J + red_pairs<F>() - 1) / red_pairs<F>();
  L.rrun[0] = cv.take<xyzz<F>>((size_t)s.Wk * s.J);
  L.racc[0] = cv.take<xyzz<F>>((size_t)s.Wk * s.J);
  L.rrun[1] = cv.take<xyzz<F>>((size_t)s.Wk * j2);
  L.racc[1] = cv.take<xyzz<F>>((size_t)s.Wk * j2);
  L.outua = cv.take<xyzz<F>>((size_t)s.Wk * 2);
  L.aff = cv.take<unsigned char>(s.affine ? affine_scratch(s.records, s.affine) : 0);
  L.bytes = cv.off + 256;
  return L;
}

// --------------------------------------------------------------- digits
__device__ __forceinline__ void load_scalar(const uint64_t* sc, size_t i, uint32_t s[8]) {
  const uint4* p = reinterpret_cast<const uint4*>(sc) + 2 * i;
  uint4 a = __ldg(p), b = __ldg(p + 1);
  s[0] = a.x; s[1] = a.y; s[2] = a.z; s[3] = a.w;
  s[4] = b.x; s[5] = b.y; s[6] = b.z; s[7] = b.w;
}

// Pops the next c-bit window off a 256-bit scalar (s >>= c) and returns it.
__device__ __forceinline__ uint32_t pop_window(uint32_t s[8], int c) {
  const uint32_t v = s[0] & ((1u << c) - 1u);
#pragma unroll
  for (int i = 0; i < 7; i++) s[i] = __funnelshift_r(s[i], s[i + 1], c);
  s[7] >>= c;
  return v;
}

// Signed-digit recoding, digit in [-2^(c-1), 2^(c-1)]: the same digit set as
// the reference's g1_extractAllSigned (include/msm_g1.cuh:271-329).
// Returns the (window, bucket) key or kInvalid for a zero digit.
__device__ __forceinline__ uint32_t next_digit(uint32_t s[8], int c, uint32_t B, int w,
                                               uint32_t& carry, bool& neg) {
  uint32_t raw = pop_window(s, c) + carry;
  uint32_t mag;
  if (raw > B) {
    mag = (1u << c) - raw;
    carry = 1;
    neg = true;
  } else {
    mag = raw;
    carry = 0;
    neg = false;
  }
  return mag ? (uint32_t)w * B + (mag - 1) : kInvalid;
}

// k mod r for a 256-bit k (at most 5 subtractions of r < 2^254): fixed-base
// tables hold multiples of points of order r, so k and k mod r give the same
// sum, and the reduced scalar fits the tables' 254-bit window range.
__device__ __forceinline__ void reduce_mod_r(uint32_t s[8]) {
  for (int it = 0; it < 5; it++) {
    uint32_t d[8], bw;
    asm("sub.cc.u32  %0, %9, %17;\n\t"
        "subc.cc.u32 %1, %10, %18;\n\t"
        "subc.cc.u32 %2, %11, %19;\n\t"
        "subc.cc.u32 %3, %12, %20;\n\t"
        "subc.cc.u32 %4, %13, %21;\n\t"
        "subc.cc.u32 %5, %14, %22;\n\t"
        "subc.cc.u32 %6, %15, %23;\n\t"
        "subc.cc.u32 %7, %16, %24;\n\t"
        "subc.u32    %8, 0, 0;"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]),
          "=r"(d[7]), "=r"(bw)
        : "r"(s[0]), "r"(s[1]), "r"(s[2]), "r"(s[3]), "r"(s[4]), "r"(s[5]), "r"(s[6]), "r"(s[7]),
          "n"(FrCfg::P0), "n"(FrCfg::P1), "n"(FrCfg::P2), "n"(FrCfg::P3), "n"(FrCfg::P4),
          "n"(FrCfg::P5), "n"(FrCfg::P6), "n"(FrCfg::P7));
    if (bw) return;  // s < r
#pragma unroll
    for (int q = 0; q < 8; q++) s[q] = d[q];
  }
}

// Scalar sources of one launch.  Windowed MSMs: one instance, key
// w * B + bucket, record value = point index.  Fixed-base MSMs: up to
// kMaxInst instances (grid.y), each with its own scalars and table; all
// windows of an instance share its bucket set, key = instance * B + bucket,
// and the record value names the instance's table entry (window w of point
// i: w * n + i).
constexpr int kMaxInst = 64;
struct ScalarSrc {
  const uint64_t* sc[kMaxInst];
  uint32_t n[kMaxInst];
};

template <bool kFixed>
__global__ void k_msm_hist(const __grid_constant__ ScalarSrc src, int c, int W, uint32_t B,
                           uint32_t* __restrict__ counts) {
  const int inst = blockIdx.y;
  const uint32_t n = src.n[inst];
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n;
  uint32_t s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (active) load_scalar(src.sc[inst], i, s);
  if (kFixed) reduce_mod_r(s);
  const int lane = threadIdx.x & 31;
  uint32_t carry = 0;
  for (int w = 0; w < W; w++) {
    bool neg;
    uint32_t key = next_digit(s, c, B, kFixed ? inst : w, carry, neg);
    if (!active) key = kInvalid;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (key != kInvalid && lane == __ffs(peers) - 1) atomicAdd(&counts[key], (uint32_t)__popc(peers));
  }
}

template <bool kFixed>
__global__ void k_msm_scatter(const __grid_constant__ ScalarSrc src, int c, int W, uint32_t B,
                              uint32_t* __restrict__ cursor, uint2* __restrict__ srec) {
  const int inst = blockIdx.y;
  const uint32_t n = src.n[inst];
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n;
  uint32_t s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  if (active) load_scalar(src.sc[inst], i, s);
  if (kFixed) reduce_mod_r(s);
  const int lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  uint32_t carry = 0;
  for (int w = 0; w < W; w++) {
    bool neg;
    uint32_t key = next_digit(s, c, B, kFixed ? inst : w, carry, neg);
    if (!active) key = kInvalid;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    uint32_t base = 0;
    if (key != kInvalid && lane == leader) base = atomicAdd(&cursor[key], (uint32_t)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (key != kInvalid) {
      const uint32_t pos = base + __popc(peers & lt);
      const uint32_t idx = kFixed ? (uint32_t)((size_t)w * n + i) : (uint32_t)i;
      srec[pos] = make_uint2(key, idx | (neg ? kNeg : 0u));
    }
  }
}

// ------------------------------------------------- segmented reduction
// Node of the block-level segmented reduction: the partial sums of the first
// and last key-segments of a contiguous record range (one sum if the range
// holds a single segment).  Complete segments are written to their bucket as
// soon as they are known to be complete.  Nodes live in shared memory (one
// per thread) so the serial phase only keeps its running sum in registers.
template <class F>
struct __align__(16) SegNode {
  xyzz<F> f, l;
  uint32_t fk, lk;  // first / last key (fk == kInvalid: empty node)
  uint32_t single;
  uint32_t pad_;
};

template <class F>
constexpr int seg_threads() { return sizeof(F) == 32 ? 128 : 64; }

// a = a ++ b by the lanes of a quad (every lane of the warp calls it;
// `on`: whether this quad has a merge to do).
template <class F>
__device__ __forceinline__ void seg_merge(SegNode<F>& a, const SegNode<F>& b, bool on,
                                          xyzz<F>* buckets) {
  const uint32_t afk = a.fk, alk = a.lk, bfk = b.fk, blk = b.lk;
  const bool as = a.single, bs = b.single;
  const bool join = on && afk != kInvalid && bfk != kInvalid && alk == bfk;
  const lane_t<F> al = quad_ld(as ? &a.f : &a.l), bf = quad_ld(&b.f);
  lane_t<F> sum = bf;
  if (__any_sync(0xffffffffu, join)) sum = quad_add(al, bf);
  __syncwarp();
  if (!on || bfk == kInvalid) return;
  if (afk == kInvalid) {
    quad_st(&a.f, bf);
    quad_st(&a.l, quad_ld(&b.l));
  } else if (join) {
    if (as) {
      quad_st(&a.f, sum);
      if (!bs) quad_st(&a.l, quad_ld(&b.l));
    } else if (bs) {
      quad_st(&a.l, sum);
    } else {
      quad_st(&buckets[alk], sum);
      quad_st(&a.l, quad_ld(&b.l));
    }
  } else {
    if (!as) quad_st(&buckets[alk], al);
    if (!bs) quad_st(&buckets[bfk], bf);
    quad_st(&a.l, quad_ld(bs ? &b.f : &b.l));
  }
  if (quad_lane<F>() == 0) {
    if (afk == kInvalid) a.fk = bfk;
    a.lk = blk;
    a.single = afk == kInvalid ? bs : (join && as && bs);
  }
}

// Closes the running segment `cur` (sum `acc`) of the thread's node.
template <class F>
__device__ __forceinline__ void seg_close(SegNode<F>& nd, const xyzz<F>& acc, uint32_t cur,
                                          xyzz<F>* buckets) {
  if (cur == kInvalid) return;
  if (nd.fk == kInvalid) {
    nd.fk = cur;
    nd.f = acc;
    nd.lk = cur;
    nd.single = 1;
  } else {
    // the previous last segment is now a middle segment: complete
    if (!nd.single) st_pod(&buckets[nd.lk], nd.l);
    nd.lk = cur;
    nd.l = acc;
    nd.single = 0;
  }
}

// Block tree over N nodes, then emit the block's boundary segments: complete
// ones go to their buckets, the others become partial records 2*block and
// 2*block+1 for the next level.  A merge is a quad's; the quads of a level are
// contiguous, so a level's merges occupy as few warps as hold them.
template <class F, int N>
__device__ __forceinline__ void seg_block_finish(SegNode<F>* sm, uint32_t key_before,
                                                 uint32_t key_after, xyzz<F>* buckets,
                                                 uint32_t* okey, xyzz<F>* opt, size_t b) {
  constexpr int Q = quad_lanes<F>();
  const int t = threadIdx.x;
  __syncthreads();
  for (int s = 1; s < N; s <<= 1) {
    const int merges = N / (2 * s);
    for (int m0 = (t & ~31) / Q; m0 < merges; m0 += blockDim.x / Q) {  // warp-uniform
      const int m = m0 + (t & 31) / Q;
      const bool on = m < merges;
      const int i = on ? 2 * s * m : 0;
      seg_merge(sm[i], sm[i + s], on, buckets);
    }
    __syncthreads();
  }
  if (t != 0) return;
  const SegNode<F>& r = sm[0];
  uint32_t hk = kInvalid, tk = kInvalid;
  if (r.fk != kInvalid) {
    const bool head = key_before == r.fk;
    if (r.single) {
      const bool tail = key_after == r.fk;
      if (!head && !tail) {
        st_pod(&buckets[r.fk], r.f);
      } else {
        hk = r.fk;
        st_pod(&opt[2 * b], r.f);
        if (tail) {
          tk = r.fk;
          st_pod(&opt[2 * b + 1], xyzz_inf<F>());
        }
      }
    } else {
      if (head) {
        hk = r.fk;
        st_pod(&opt[2 * b], r.f);
      } else {
        st_pod(&buckets[r.fk], r.f);
      }
      if (key_after == r.lk) {
        tk = r.lk;
        st_pod(&opt[2 * b + 1], r.l);
      } else {
        st_pod(&buckets[r.lk], r.l);
      }
    }
  }
  if (okey) {
    okey[2 * b] = hk;
    okey[2 * b + 1] = tk;
  }
}

// Where level 0 reads the points of its records.
template <class F>
struct PointSrc {
  const F* x;  // windowed: point i at x + i * stride, y likewise
  const F* y;
  uint32_t stride;
  int bshift;                 // fixed-base: instance = key >> bshift
  const F* table[kMaxInst];   // fixed-base: record r of an instance at table + 2 r (x, y)
};

// Level 0, one tile: records [b T K, (b + 1) T K) of the list sorted by
// (bucket key, point index | sign).
template <class F, bool kFixed>
__device__ __forceinline__ void accum0_tile(size_t b, SegNode<F>* sm,
                                            const uint2* __restrict__ srec, size_t total,
                                            const PointSrc<F>& src, int K,
                                            xyzz<F>* __restrict__ buckets,
                                            uint32_t* __restrict__ okey,
                                            xyzz<F>* __restrict__ opt) {
  constexpr int T = seg_threads<F>();
  SegNode<F>& nd = sm[threadIdx.x];
  nd.fk = nd.lk = kInvalid;
  nd.single = 1;
  const size_t bstart = b * T * K;
  const size_t bend = min(bstart + (size_t)T * K, total);
  uint32_t key_before = kInvalid, key_after = kInvalid;
  if (bstart < total) {
    key_before = bstart ? srec[bstart - 1].x : kInvalid;
    key_after = bend < total ? srec[bend].x : kInvalid;
    const size_t s = bstart + (size_t)threadIdx.x * K;
    const size_t e = min(s + K, bend);
    xyzz<F> acc = xyzz_inf<F>();
    uint32_t cur = kInvalid;
    for (size_t p = s; p < e; p++) {
      const uint2 rec = srec[p];
      const uint32_t key = rec.x;
      if (key != cur) {
        seg_close(nd, acc, cur, buckets);
        cur = key;
        acc = xyzz_inf<F>();
      }
      const uint32_t v = rec.y;
      const uint32_t idx = v & ~kNeg;
      F x, y;
      if (kFixed) {
        const F* t = src.table[key >> src.bshift];
        x = ld_pod(t + 2 * (size_t)idx);
        y = ld_pod(t + 2 * (size_t)idx + 1);
      } else {
        x = ld_pod(src.x + (size_t)idx * src.stride);
        y = ld_pod(src.y + (size_t)idx * src.stride);
      }
      if (!(fe_is_zero(x) && fe_is_zero(y))) {
        if (v & kNeg) y = fe_neg(y);
        acc = xyzz_madd(acc, x, y);
      }
    }
    seg_close(nd, acc, cur, buckets);
  }
  seg_block_finish<F, T>(sm, key_before, key_after, buckets, okey, opt, b);
}

// One tile per block.  The G1 form takes 148 registers (three blocks per
// SM); capping it at 128 for four blocks spilled ~450 B a thread and ran
// ~1 % slower.  The G2 form is at the 255-register limit either way.
template <class F, bool kFixed>
__global__ void __launch_bounds__(seg_threads<F>()) k_msm_accum0(
    const uint2* __restrict__ srec, const uint32_t* __restrict__ total_p,
    const __grid_constant__ PointSrc<F> src, int K,
    xyzz<F>* __restrict__ buckets, uint32_t* __restrict__ okey, xyzz<F>* __restrict__ opt) {
  __shared__ SegNode<F> sm[seg_threads<F>()];
  accum0_tile<F, kFixed>(blockIdx.x, sm, srec, *total_p, src, K, buckets, okey, opt);
}

// Persistent form for multi-instance chains (several proofs' MSMs): a grid
// of as many blocks as the device holds at once, each claiming record tiles
// (instance, bucket range) from a device work queue until all `ntiles` are
// taken.  `queue` starts at zero.  Uncapped like the one-tile form (156
// registers, three G1 blocks per SM): fused batches ran ~2 % faster than
// with a 128-register cap.
template <class F, bool kFixed>
__global__ void __launch_bounds__(seg_threads<F>()) k_msm_accum0_queue(
    const uint2* __restrict__ srec, const uint32_t* __restrict__ total_p,
    const __grid_constant__ PointSrc<F> src, int K,
    xyzz<F>* __restrict__ buckets, uint32_t* __restrict__ okey, xyzz<F>* __restrict__ opt,
    uint32_t ntiles, uint32_t* __restrict__ queue) {
  __shared__ SegNode<F> sm[seg_threads<F>()];
  __shared__ uint32_t tile;
  const size_t total = *total_p;
  for (;;) {
    __syncthreads();  // the previous tile's outputs (thread 0) are written
    if (threadIdx.x == 0) tile = atomicAdd(queue, 1u);
    __syncthreads();
    const uint32_t b = tile;
    if (b >= ntiles) return;
    accum0_tile<F, kFixed>(b, sm, srec, total, src, K, buckets, okey, opt);
  }
}

// ------------------------------------------- batched affine accumulation
// A large G2 MSM's sorted list holds long runs of one bucket.  They are added
// pairwise in affine coordinates before the XYZZ accumulation sees them.  An
// affine addition costs two Fp2 products, a square and an inversion, and
// Montgomery's trick over the norms in Fp makes the inversion five Fp products
// and a norm plus a shared one: about 3400 multiply instructions against 6300
// of the mixed XYZZ addition, with half the live registers (16 warps per SM
// instead of 8).
//
// A block takes T * S consecutive records, S per thread.  In a round every
// thread pairs neighbours of the same run among its own points:
//   forward: the norm of each pair's denominator joins the thread's running
//     product (the product before it is stored);
//   the block's T products are inverted by one warp, a lane for each column
//     of T / 32 of them (32 inversions at the cost of one);
//   backward: every pair with its own inverse; sums and then the left-over
//     points are written compactly into the other of two slot buffers.
// Rounds go on while they pay for their inversions.  The few points left of
// each run go through the XYZZ accumulation and the block tree.
//
// Fixed-base 2^20 points (20-bit windows, runs of 26): 5.6 ms against 7.5 ms
// for the XYZZ accumulation, 2^18: 1.8 against 2.5.  Bound by the latency of
// the gathers and of the scattered slots (about 690 B of DRAM traffic per
// record, 530 where the points stay in L2), not by the multiply pipe (58 %
// busy).  For the same reason G1 keeps
// the XYZZ accumulation, whose additions are 2.5 times cheaper: there the
// rounds measured 2.71 against 2.70 ms.  Copying pairs to shared memory ahead
// (cp.async) was slower: scattered 16-byte copies cost a shared-memory
// wavefront each.
//
// The run structure is kept as bit masks per sub-segment of 64 points: bit j
// of `ends` is set when point j is the last of its run.  A round about halves
// the points, and the slots are sized for that; a block with runs too short
// for it (or for one round to pay) skips the rounds.
constexpr int kAffLeast = 8;    // additions left per thread for a round to pay
constexpr uint32_t kAffUntouched = 1u << 31;  // state: points still the table's
constexpr uint32_t kAffFirst = 1u << 30;      // state: points in slot buffer 1
static_assert(sizeof(fp2_t) * 2 == kAffPoint && sizeof(fp_t) * 2 == kAffPair, "affine_layout.hpp");

struct AffScratch {
  unsigned char* base;
  const AffShape& a;
  __device__ __forceinline__ fp2_t* slot(int buf, int h, int j) const {
    const int row = h * a.slots[buf] + j + (buf ? a.rows : 0);
    return reinterpret_cast<fp2_t*>(base) + 2 * (uint32_t)(row * kAffT + threadIdx.x);
  }
  // prefix product and norm of pair k
  __device__ __forceinline__ fp_t* pair(int k) const {
    return reinterpret_cast<fp_t*>(base + a.pre) + 2 * (uint32_t)(k * kAffT + threadIdx.x);
  }
  // which: 0 run ends now, 1 run ends of the sorted records, 2 pairs of the round
  __device__ __forceinline__ uint64_t& mask(int h, int which) const {
    return reinterpret_cast<uint64_t*>(base + a.mask)[(3 * h + which) * kAffT + threadIdx.x];
  }
  // points of each sub-segment (8 bits each) and the kAff* flags
  __device__ __forceinline__ uint32_t& state() const {
    return reinterpret_cast<uint32_t*>(base + a.state)[threadIdx.x];
  }
};

__device__ __forceinline__ uint64_t aff_low(int n) { return n >= 64 ? ~0ull : (1ull << n) - 1; }
// Bit j set when points j and j + 1 of a sub-segment of cnt points belong to
// one run.
__device__ __forceinline__ uint64_t aff_links(uint64_t ends, int cnt) {
  return ~ends & aff_low(cnt);
}
// The pairs (j, j + 1) of the links, from the top of each run down, as the
// bits of their first points.
__device__ __forceinline__ uint64_t aff_pairs(uint64_t links) {
  uint64_t m = 0;
  while (links) {
    const int j = 63 - __clzll((long long)links);
    links &= j ? aff_low(j - 1) : 0;
    m |= 1ull << j;
  }
  return m;
}
// `ends` after the pairs m became one point each (their first points' bits,
// which are clear, drop out).
__device__ __forceinline__ uint64_t aff_squeeze(uint64_t ends, uint64_t m) {
  while (m) {
    const int j = 63 - __clzll((long long)m);
    m ^= 1ull << j;
    ends = (ends & aff_low(j)) | ((ends >> 1) & ~aff_low(j));
  }
  return ends;
}

// How two affine points add: in general, as a doubling, or without any
// arithmetic (one of them or the sum is the point at infinity).
enum AffKind { kAffGeneral, kAffDouble, kAffTakeSecond, kAffTakeFirst, kAffInfinity };
template <class LoadY>
__device__ __forceinline__ int aff_kind(const fp2_t& x1, const fp2_t& x2, const fp2_t& d,
                                        LoadY load_y) {
  const bool zd = fe_is_zero(d), z1 = fe_is_zero(x1), z2 = fe_is_zero(x2);
  if (!(zd || z1 || z2)) return kAffGeneral;
  const fp2_t y1 = load_y(0), y2 = load_y(1);
  if (z1 && fe_is_zero(y1)) return kAffTakeSecond;
  if (z2 && fe_is_zero(y2)) return kAffTakeFirst;
  if (!zd) return kAffGeneral;
  return fe_eq(y1, y2) && !fe_is_zero(y1) ? kAffDouble : kAffInfinity;
}

// Inverts the kAffT products in place (one warp; none of them is zero).
__device__ __forceinline__ void aff_invert(fp_t* tot) {
  constexpr int R = kAffT / 32;
  fp_t* v = tot + (threadIdx.x & 31);
  fp_t pre[R];
  pre[0] = v[0];
#pragma unroll
  for (int i = 1; i < R; i++) pre[i] = pre[i - 1] * v[32 * i];
  fp_t inv = fe_inv(pre[R - 1]);
#pragma unroll
  for (int i = R - 1; i > 0; i--) {
    const fp_t x = v[32 * i];
    v[32 * i] = inv * pre[i - 1];
    inv = inv * x;
  }
  v[0] = inv;
}

// The points of one thread: the table's (with the record's sign) before the
// first round, the thread's slots afterwards.
template <bool kFixed>
struct AffPoints {
  const uint2* rec;  // the thread's sorted records
  const PointSrc<fp2_t>& src;
  const AffScratch& scr;
  bool first;
  int buf;  // slot buffer that holds the points
  __device__ __forceinline__ const fp2_t* at(const uint2& r, bool y) const {
    const size_t idx = r.y & ~kNeg;
    if (kFixed) return src.table[r.x >> src.bshift] + 2 * idx + y;
    return (y ? src.y : src.x) + idx * src.stride;
  }
  __device__ __forceinline__ uint2 record(int h, int j) const { return rec[h * kSub + j]; }
  __device__ __forceinline__ fp2_t x(int h, int j) const {
    return ld_pod(first ? at(record(h, j), false) : scr.slot(buf, h, j));
  }
  __device__ __forceinline__ fp2_t y(int h, int j) const {
    if (!first) return ld_pod(scr.slot(buf, h, j) + 1);
    const uint2 r = record(h, j);
    const fp2_t v = ld_pod(at(r, true));
    return r.y & kNeg ? fe_neg(v) : v;
  }
};

// Walks the pairs of the thread's sub-segments, from the last one down or
// from the first one up.
template <bool kDown>
struct AffWalk {
  const AffScratch& scr;
  int nsub, h, j = 0;  // h: current sub-segment; -1 past the last pair
  uint64_t m;
  __device__ __forceinline__ AffWalk(const AffScratch& scr, int n) : scr(scr), nsub(n) {
    h = kDown ? n - 1 : 0;
    m = scr.mask(h, 2);
  }
  __device__ __forceinline__ void next() {
    while (!m && h >= 0) {
      h = kDown ? h - 1 : (h + 1 < nsub ? h + 1 : -1);
      if (h >= 0) m = scr.mask(h, 2);
    }
    if (h < 0) return;
    j = kDown ? 63 - __clzll((long long)m) : __ffsll((long long)m) - 1;
    m ^= 1ull << j;
  }
};

// The rounds of tile tile0 + blockIdx.x.  kBlocks per SM: 3 (168 registers,
// ~350 bytes a thread spilled, as many tail blocks fit) or 4 (128 registers,
// ~650 bytes spilled, a third more scratch); see affine_blocks.
template <bool kFixed, int kBlocks>
__global__ void __launch_bounds__(kAffT, kBlocks) k_msm_affine(
    const uint2* __restrict__ srec, const uint32_t* __restrict__ total_p,
    const __grid_constant__ PointSrc<fp2_t> src, const __grid_constant__ AffShape shape,
    unsigned char* __restrict__ scratch, uint32_t tile0, uint32_t ntiles) {
  __shared__ fp_t tot[kAffT];
  __shared__ uint32_t left[kAffT / 32];
  const size_t total = *total_p;
  const int S = aff_span(total, ntiles);
  const size_t b = tile0 + blockIdx.x;
  const AffScratch scr{scratch + (size_t)blockIdx.x * shape.bytes, shape};
  const int t = threadIdx.x;
  const size_t s = min((b * kAffT + t) * S, total);
  const int len = (int)min((size_t)S, total - s);
  const int nsub = (S + kSub - 1) / kSub;
  AffPoints<kFixed> pts{srec + s, src, scr, true, 0};
  uint32_t cnts = 0;  // points of each sub-segment, 8 bits each

  int links = 0;  // additions left
  bool fits = true;
  for (int h = 0; h < nsub; h++) {
    const int cnt = min(max(len - h * kSub, 0), kSub);
    // s is even: two records (16 bytes) at a time; the list has room for the
    // word after its last record
    const uint4* r = reinterpret_cast<const uint4*>(srec + s + h * kSub);
    uint64_t ends = 0;
    uint32_t key = kInvalid;  // of the record before
    for (int j = 0; j < cnt; j += 2) {
      const uint4 v = r[j / 2];
      if (j) ends |= (uint64_t)(v.x != key) << (j - 1);
      ends |= (uint64_t)(v.z != v.x) << j;
      key = v.z;
    }
    if (cnt) ends = (ends | 1ull << (cnt - 1)) & aff_low(cnt);
    const uint64_t C = aff_links(ends, cnt), M = aff_pairs(C);
    scr.mask(h, 0) = ends;
    scr.mask(h, 1) = ends;
    scr.mask(h, 2) = M;
    cnts |= (uint32_t)cnt << (8 * h);
    links += __popcll(C);
    const int o1 = cnt - __popcll(M);
    const int o2 = o1 - __popcll(aff_pairs(aff_links(aff_squeeze(ends, M), o1)));
    fits = fits && o1 <= shape.limit(h, 1) && o2 <= shape.limit(h, 0);
  }
  const int lanes = __syncthreads_count(len > 0);

  for (uint32_t round = 0;; round++) {
    const uint32_t wsum = __reduce_add_sync(0xffffffffu, (uint32_t)links);
    if ((t & 31) == 0) left[t >> 5] = wsum;
    if (!__syncthreads_and(fits)) break;
    uint32_t sum = 0;
#pragma unroll
    for (int w = 0; w < kAffT / 32; w++) sum += left[w];
    if (!sum || sum < (uint32_t)(kAffLeast * lanes)) break;

    fp_t run = fe_one<FpCfg>();
    int k = 0;
    {
      // a pair has only a norm and a product here, too short to hide its
      // gathers behind: two pairs are read at a time
      constexpr int kAhead = 2;
      AffWalk<true> w(scr, nsub);
      while (w.h >= 0) {
        int h[kAhead], j[kAhead];
        fp2_t x1[kAhead], x2[kAhead];
        uint2 r1[kAhead], r2[kAhead];
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
          w.next();
          h[i] = w.h;
          j[i] = w.j;
          if (pts.first && w.h >= 0) {
            r1[i] = pts.record(w.h, w.j);
            r2[i] = pts.record(w.h, w.j + 1);
          }
        }
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
          if (h[i] < 0) continue;
          x1[i] = ld_pod(pts.first ? pts.at(r1[i], false) : scr.slot(pts.buf, h[i], j[i]));
          x2[i] = ld_pod(pts.first ? pts.at(r2[i], false) : scr.slot(pts.buf, h[i], j[i] + 1));
        }
#pragma unroll
        for (int i = 0; i < kAhead; i++) {
          if (h[i] < 0) break;
          fp2_t d = x2[i] - x1[i];
          const int kind = aff_kind(x1[i], x2[i], d, [&](int q) { return pts.y(h[i], j[i] + q); });
          if (kind == kAffDouble) d = fe_dbl(pts.y(h[i], j[i]));
          fp_t n = fe_one<FpCfg>();
          if (kind <= kAffDouble) n = fe_norm(d);
          st_pod(scr.pair(k), run);
          st_pod(scr.pair(k) + 1, n);
          run = run * n;
          k++;
        }
      }
    }
    tot[t] = run;
    __syncthreads();
    // the inverting warp rotates, so that blocks that share an SM load its
    // four schedulers evenly
    if ((t >> 5) == (int)((round + b) % (kAffT / 32))) aff_invert(tot);
    __syncthreads();
    fp_t inv = tot[t];
    const int ob = pts.buf ^ 1;
    {
      AffWalk<false> w(scr, nsub);
      uint2 ra{}, rb{};  // the pair's records, read a step ahead (first round)
      const auto next = [&] {
        w.next();
        if (pts.first && w.h >= 0) {
          ra = pts.record(w.h, w.j);
          rb = pts.record(w.h, w.j + 1);
        }
      };
      next();
      while (w.h >= 0) {
        const int h = w.h, j = w.j;
        k--;
        const fp_t pre = ld_pod(scr.pair(k)), n = ld_pod(scr.pair(k) + 1);
        fp2_t x1, y1, x2, num;
        if (pts.first) {
          x1 = ld_pod(pts.at(ra, false));
          y1 = ld_pod(pts.at(ra, true));
          x2 = ld_pod(pts.at(rb, false));
          num = ld_pod(pts.at(rb, true));
          if (ra.y & kNeg) y1 = fe_neg(y1);
          if (rb.y & kNeg) num = fe_neg(num);
        } else {
          const fp2_t* q = scr.slot(pts.buf, h, j);
          x1 = ld_pod(q);
          y1 = ld_pod(q + 1);
          x2 = ld_pod(q + 2 * kAffT);
          num = ld_pod(q + 2 * kAffT + 1);
        }
        fp2_t* const out = scr.slot(ob, h, j - __popcll(scr.mask(h, 2) & aff_low(j)));
        next();
        fp2_t d = x2 - x1;
        const int kind = aff_kind(x1, x2, d, [&](int q) { return q ? num : y1; });
        fp2_t xo = x2, yo = num;
        if (kind <= kAffDouble) {
          if (kind == kAffDouble) {
            d = fe_dbl(y1);
            num = fe_triple(fe_sqr(x1));
          } else {
            num = num - y1;
          }
          const fp_t ni = inv * pre;
          inv = inv * n;
          const fp2_t lam = num * fe_inv_of(d, ni);
          xo = fe_sqr(lam) - x1 - x2;
          yo = lam * (x1 - xo) - y1;
        } else if (kind == kAffTakeFirst) {
          xo = x1;
          yo = y1;
        } else if (kind == kAffInfinity) {
          xo = fe_zero_of<fp2_t>();
          yo = fe_zero_of<fp2_t>();
        }
        st_pod(out, xo);
        st_pod(out + 1, yo);
      }
    }
    // the points without a partner move over, and the masks follow
    links = 0;
    for (int h = 0; h < nsub; h++) {
      const uint64_t ends = scr.mask(h, 0), M = scr.mask(h, 2);
      const int cnt = (cnts >> (8 * h)) & 255;
      uint64_t alone = ~(M | M << 1) & aff_low(cnt);
      while (alone) {
        const int j = __ffsll((long long)alone) - 1;
        alone &= alone - 1;
        const fp2_t x = pts.x(h, j), y = pts.y(h, j);
        fp2_t* const out = scr.slot(ob, h, j - __popcll(M & aff_low(j)));
        st_pod(out, x);
        st_pod(out + 1, y);
      }
      const int o = cnt - __popcll(M);
      const uint64_t e = aff_squeeze(ends, M), C = aff_links(e, o);
      scr.mask(h, 0) = e;
      scr.mask(h, 2) = aff_pairs(C);
      cnts = (cnts & ~(255u << (8 * h))) | ((uint32_t)o << (8 * h));
      links += __popcll(C);
    }
    pts.first = false;
    pts.buf = ob;
  }
  scr.state() = cnts | (pts.first ? kAffUntouched : 0) | (pts.buf ? kAffFirst : 0);
}

// The XYZZ accumulation of the points the rounds of a tile left, and the
// block tree over its threads.  A kernel of its own: its register need would
// halve the rounds' residency.  Beside four round blocks per SM the tail
// runs as two waves of two (255 registers): 7.78 against 7.95 ms for a 2^20
// MSM with three spilling ones.
template <bool kFixed, int kBlocks>
__global__ void __launch_bounds__(kAffT, kBlocks == 3 ? 3 : 1) k_msm_affine_tail(
    const uint2* __restrict__ srec, const uint32_t* __restrict__ total_p,
    const __grid_constant__ PointSrc<fp2_t> src, const __grid_constant__ AffShape shape,
    unsigned char* __restrict__ scratch, xyzz<fp2_t>* __restrict__ buckets,
    uint32_t* __restrict__ okey, xyzz<fp2_t>* __restrict__ opt, uint32_t tile0, uint32_t ntiles) {
  extern __shared__ __align__(16) unsigned char smem[];
  SegNode<fp2_t>* sm = reinterpret_cast<SegNode<fp2_t>*>(smem);
  const size_t total = *total_p;
  const int S = aff_span(total, ntiles);
  const size_t b = tile0 + blockIdx.x;
  const AffScratch scr{scratch + (size_t)blockIdx.x * shape.bytes, shape};
  const int t = threadIdx.x;
  const size_t bstart = min(b * kAffT * S, total);
  const size_t bend = min(bstart + (size_t)kAffT * S, total);
  const size_t s = min(bstart + (size_t)t * S, total);
  const int nsub = (S + kSub - 1) / kSub;
  const uint32_t state = scr.state();
  const AffPoints<kFixed> pts{srec + s, src, scr, (state & kAffUntouched) != 0,
                              (state & kAffFirst) ? 1 : 0};
  SegNode<fp2_t>& nd = sm[t];
  nd.fk = nd.lk = kInvalid;
  nd.single = 1;
  xyzz<fp2_t> acc = xyzz_inf<fp2_t>();
  uint32_t cur = kInvalid;
  // a step of the loop ends at a point that has to be added: the points that
  // only begin a run are passed on the way, so the lanes add together
  int h = -1, j = 0, cnt = 0;
  uint64_t ends = 0, runs = 0;
  bool begins = true;
  for (;;) {
    bool add = false;
    fp2_t x, y;
    while (!add) {
      while (j >= cnt && h + 1 < nsub) {
        h++;
        j = 0;
        cnt = (state >> (8 * h)) & 127;
        ends = scr.mask(h, 0);
        runs = scr.mask(h, 1);
        begins = true;
      }
      if (j >= cnt) break;
      if (begins) {
        const uint32_t key = srec[s + h * kSub + __ffsll((long long)runs) - 1].x;
        runs &= runs - 1;
        if (key != cur) {
          seg_close(nd, acc, cur, buckets);
          cur = key;
          acc = xyzz_inf<fp2_t>();
        }
      }
      begins = (ends >> j) & 1;
      x = pts.x(h, j);
      y = pts.y(h, j);
      j++;
      if (fe_is_zero(x) && fe_is_zero(y)) continue;
      if (xyzz_is_inf(acc))
        acc = {x, y, fe_one_of<fp2_t>(), fe_one_of<fp2_t>()};
      else
        add = true;
    }
    if (!add) break;
    acc = xyzz_madd(acc, x, y);
  }
  seg_close(nd, acc, cur, buckets);
  const uint32_t key_before = bstart && bstart < bend ? srec[bstart - 1].x : kInvalid;
  const uint32_t key_after = bend < total ? srec[bend].x : kInvalid;
  seg_block_finish<fp2_t, kAffT>(sm, key_before, key_after, buckets, okey, opt, b);
}

// Blocks of the rounds the device holds at once: one wave.
template <int kBlocks>
size_t affine_grid_of() {
  static PerDevice<size_t> known;
  return resident_blocks(known, k_msm_affine<true, kBlocks>, kAffT, 0);
}
size_t affine_grid(int blocks) { return blocks == 3 ? affine_grid_of<3>() : affine_grid_of<4>(); }
size_t affine_wave(int blocks) { return affine_grid(blocks) * kAffT * kAffMaxSub * kSub; }

// Blocks per SM for a list of at most `records`: three while the list fits
// one wave of them, four beyond.  Fixed-base 2^17 / 2^18 / 2^20 points (2.0 /
// 3.9 / 13.6 M records against a wave of 10.9 M): 1.03 / 1.80 / 5.88 ms with
// three, 1.14 / 1.78 / 5.60 ms with four; a 2^20 proof 20.1 against 19.4 ms.
int affine_blocks(size_t records) { return records <= affine_wave(3) ? 3 : 4; }

// Tiles of the affine accumulation for a sorted list of at most `records`
// records in `buckets` buckets; 0 where the XYZZ accumulation takes the list:
// runs too short, or too few records to fill two thirds of the device with
// tiles of the least size (where the rounds' inversions stop paying: windowed
// 2^15 points, 192 tiles, 0.59 ms XYZZ against 0.67; 2^16, 352 tiles, 1.09
// against 0.88).
size_t affine_tiles(size_t records, size_t buckets) {
  if (records < 6 * buckets) return 0;
  const int blocks = affine_blocks(records);
  const size_t grid = affine_grid(blocks), wave = affine_wave(blocks);
  size_t tiles = grid * ((records + wave - 1) / wave);
  if (records < tiles * kAffT * kAffMinS) tiles = (records + kAffT * kAffMinS - 1) / (kAffT * kAffMinS);
  return 3 * tiles < 2 * grid ? 0 : tiles;
}

size_t affine_scratch(size_t records, size_t tiles) {
  return std::min(tiles, affine_grid(affine_blocks(records))) *
         (size_t)aff_shape(aff_span(records, (uint32_t)tiles)).bytes;
}

// Level 0 as rounds and tail, a wave of tiles at a time (the scratch holds
// one wave).
template <bool kFixed, int kBlocks>
void affine_enqueue(const uint2* srec, const uint32_t* total_p, const PointSrc<fp2_t>& src,
                    size_t records, unsigned char* scratch, xyzz<fp2_t>* buckets, uint32_t* okey,
                    xyzz<fp2_t>* opt, uint32_t ntiles, cudaStream_t st) {
  constexpr size_t smem = kAffT * sizeof(SegNode<fp2_t>);
  // more than the default 48 KB
  static PerDevice<bool> allowed;
  allowed.get(current_device(), [&] {
    ZK_CUDA(cudaFuncSetAttribute(k_msm_affine_tail<kFixed, kBlocks>,
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return true;
  });
  const AffShape shape = aff_shape(aff_span(records, ntiles));
  const uint32_t wave = (uint32_t)affine_grid(kBlocks);
  for (uint32_t t0 = 0; t0 < ntiles; t0 += wave) {
    const uint32_t g = std::min(wave, ntiles - t0);
    k_msm_affine<kFixed, kBlocks><<<g, kAffT, 0, st>>>(srec, total_p, src, shape, scratch, t0,
                                                       ntiles);
    ZK_LAUNCHED();
    k_msm_affine_tail<kFixed, kBlocks><<<g, kAffT, smem, st>>>(srec, total_p, src, shape, scratch,
                                                               buckets, okey, opt, t0, ntiles);
    ZK_LAUNCHED();
  }
}

// Levels >= 1: records are (bucket key, XYZZ partial sum); kInvalid keys
// carry nothing and only ever separate different keys.  A quad per node: these
// levels are short lists, bound by the depth of their dependent additions.
template <class F>
__global__ void __launch_bounds__(lvl_nodes<F>() * quad_lanes<F>()) k_msm_accumN(
    const uint32_t* __restrict__ ikey, const xyzz<F>* __restrict__ ipt, size_t m, int K,
    xyzz<F>* __restrict__ buckets, uint32_t* __restrict__ okey, xyzz<F>* __restrict__ opt) {
  constexpr int T = lvl_nodes<F>();
  extern __shared__ __align__(16) unsigned char smem[];
  SegNode<F>* sm = reinterpret_cast<SegNode<F>*>(smem);
  const int node = threadIdx.x / quad_lanes<F>();
  SegNode<F>& nd = sm[node];
  const size_t bstart = min((size_t)blockIdx.x * T * K, m);
  const size_t bend = min(bstart + (size_t)T * K, m);
  const uint32_t key_before = bstart && bstart < m ? ikey[bstart - 1] : kInvalid;
  const uint32_t key_after = bend < m ? ikey[bend] : kInvalid;
  const size_t s = bstart + (size_t)node * K;
  // the node's segments so far (registers of all four lanes; `acc` and the
  // closed segments one coordinate per lane)
  uint32_t fk = kInvalid, lk = kInvalid, cur = kInvalid;
  bool single = true;
  lane_t<F> acc = quad_inf<F>(), f = acc, l = acc;
  auto close = [&] {
    if (cur == kInvalid) return;
    if (fk == kInvalid) {
      fk = lk = cur;
      f = acc;
    } else {
      if (!single) quad_st(&buckets[lk], l);
      lk = cur;
      l = acc;
      single = false;
    }
  };
  for (int i = 0; i < K; i++) {
    const size_t p = s + i;
    const uint32_t key = p < bend ? ikey[p] : kInvalid;
    const bool on = key != kInvalid;
    if (!__any_sync(0xffffffffu, on)) continue;
    const lane_t<F> v = on ? quad_ld(ipt + p) : quad_inf<F>();
    const bool same = on && key == cur;
    lane_t<F> sum = v;
    if (__any_sync(0xffffffffu, same)) sum = quad_add(acc, v);
    if (on && !same) {
      close();
      cur = key;
      acc = v;
    } else if (on) {
      acc = sum;
    }
  }
  close();
  quad_st(&nd.f, f);
  quad_st(&nd.l, l);
  if (quad_lane<F>() == 0) {
    nd.fk = fk;
    nd.lk = lk;
    nd.single = single;
  }
  seg_block_finish<F, T>(sm, key_before, key_after, buckets, okey, opt, (size_t)blockIdx.x);
}

// dst[i] += src[i]: the buckets of two MSMs whose results are added, so one
// reduction yields the sum.
template <class F>
__global__ void __launch_bounds__(128) k_msm_bucket_add(xyzz<F>* __restrict__ dst,
                                                        const xyzz<F>* __restrict__ src,
                                                        size_t count) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count) return;
  st_pod(&dst[i], xyzz_add(ld_pod(&dst[i]), ld_pod(&src[i])));
}

// ------------------------------------------------------ bucket reduction
// Window sums sum_b (b+1) S_b, without per-chunk scalar multiplications and
// without long serial chains above the first level.
//
// Additions are quad operations (curve_quad.cuh): these are dependent chains
// on a device that is far from full.
// Level 1: quad per (window, chunk of L buckets) -> (run, acc) with
// run = sum S_b and acc = sum (i+1) S_{lo+i} (running sums from the top).
// Block passes: block per (window, segment of up to red_pairs consecutive pairs,
// each covering 2^log_span buckets) -> run' = sum run_i and
// acc' = sum acc_i + 2^log_span * sum_i i run_i.  In the block,
// sum_i i run_i = sum_{i>=1} S_i with S_i = sum_{k>=i} run_k: a shared-memory
// suffix scan (log2 of the pairs, in steps) and a tree reduction, so the depth is
// logarithmic.  The final pass (one segment per window) stops before the
// doublings and leaves U = sum_i i run_i and A = sum_i acc_i; the host forms
// the window sum A + 2^log_span U, where a serial doubling chain is cheap.
template <class F>
__global__ void __launch_bounds__(128) k_msm_reduce_l1(const xyzz<F>* __restrict__ buckets, int c,
                                                       int W, uint32_t B, uint32_t L, uint32_t J,
                                                       xyzz<F>* __restrict__ run_out,
                                                       xyzz<F>* __restrict__ acc_out) {
  const size_t t = ((size_t)blockIdx.x * blockDim.x + threadIdx.x) / quad_lanes<F>();
  const bool on = t < (size_t)W * J;
  const int w = on ? (int)(t / J) : 0;
  const uint32_t j = (uint32_t)(t % J);
  const int nbits = 256 - w * c;
  const uint32_t Bw = nbits >= c ? B : (nbits <= 0 ? 1u : (1u << nbits));
  const uint32_t lo = on ? min(j * L, Bw) : 0, hi = on ? min(lo + L, Bw) : 0;
  const xyzz<F>* bw = buckets + (size_t)w * B;
  lane_t<F> run = quad_inf<F>(), acc = run;
  for (uint32_t i = L; i-- > 0;) {
    const bool has = lo + i < hi;
    if (!__any_sync(0xffffffffu, has)) continue;
    run = quad_add(run, has ? quad_ld(bw + lo + i) : quad_inf<F>());
    acc = quad_add(acc, run);
  }
  if (!on) return;
  quad_st(&run_out[t], run);
  quad_st(&acc_out[t], acc);
}

// tree sum over the first `width` quads' values (a power of two; result valid
// in quad 0)
template <class F>
__device__ __forceinline__ lane_t<F> block_sum(lane_t<F> v, xyzz<F>* sm, int width) {
  constexpr int Q = quad_lanes<F>();
  const int i = threadIdx.x / Q, i0 = (threadIdx.x & ~31) / Q;
  quad_st(&sm[i], v);
  __syncthreads();
  for (int s = width / 2; s > 0; s >>= 1) {
    if (i0 < s) {  // warp-uniform
      v = quad_add(v, quad_ld(&sm[min(i + s, red_pairs<F>() - 1)]));
      __syncwarp();
      if (i < s) quad_st(&sm[i], v);
    }
    __syncthreads();
  }
  v = quad_ld(&sm[0]);
  __syncthreads();
  return v;
}

// grid (segments, windows); out_u / out_a receive U and A of final passes.
// Depth: the scan and the trees run over the segment's width (the power of
// two covering its pairs), not the whole block.  When the doublings are few
// (always between passes, and in a final pass when log_span + 1 is below the
// tree depth) each quad folds 2^log_span S_i into its acc_i and one tree
// sums the result, instead of two trees and a serial doubling tail; a final
// pass then leaves U = infinity and the whole sum in A.
template <class F>
__global__ void __launch_bounds__(red_pairs<F>() * quad_lanes<F>()) k_msm_reduce_blk(
    const xyzz<F>* __restrict__ run_in, const xyzz<F>* __restrict__ acc_in, uint32_t Jin,
    int log_span, uint32_t Jout, xyzz<F>* __restrict__ run_out, xyzz<F>* __restrict__ acc_out,
    xyzz<F>* __restrict__ out_u, xyzz<F>* __restrict__ out_a) {
  constexpr int kRedT = red_pairs<F>(), Q = quad_lanes<F>();
  __shared__ xyzz<F> sm[kRedT];
  const int w = blockIdx.y, i = threadIdx.x / Q, i0 = (threadIdx.x & ~31) / Q;
  const uint32_t idx = blockIdx.x * kRedT + i;
  const size_t base = (size_t)w * Jin;
  const uint32_t len = min((uint32_t)kRedT, Jin - blockIdx.x * kRedT);
  int width = 1, depth = 0;
  while (width < (int)len) {
    width <<= 1;
    depth++;
  }
  const lane_t<F> zero = quad_inf<F>();
  lane_t<F> r = idx < Jin ? quad_ld(run_in + base + idx) : zero;
  // inclusive suffix scan: r = S_i = sum_{k >= i} run_k within the segment
  quad_st(&sm[i], r);
  __syncthreads();
  for (int off = 1; off < width; off <<= 1) {
    const lane_t<F> o = i + off < kRedT ? quad_ld(&sm[i + off]) : zero;
    __syncthreads();
    if (i0 < width) {  // warp-uniform
      r = quad_add(r, o);
      quad_st(&sm[i], r);
    }
    __syncthreads();
  }
  const lane_t<F> total = quad_ld(&sm[0]);  // S_0 = sum of the segment's runs
  __syncthreads();
  const lane_t<F> acc = idx < Jin ? quad_ld(acc_in + base + idx) : zero;
  const size_t o = (size_t)w * Jout + blockIdx.x;
  if (i == 0) r = zero;
  if (Jout > 1 || log_span + 1 < depth) {
    lane_t<F> t = zero;
    if (i0 < width) {
      if (__any_sync(0xffffffffu, !quad_zero(r, 2)))
        for (int d = 0; d < log_span; d++) r = quad_dbl(r);
      t = quad_add(r, acc);
    }
    const lane_t<F> s = block_sum<F>(t, sm, width);
    if (i != 0) return;
    if (Jout == 1) {
      quad_st(&out_u[w], zero);
      quad_st(&out_a[w], s);
    } else {
      quad_st(&run_out[o], total);
      quad_st(&acc_out[o], s);
    }
    return;
  }
  // final pass with many doublings: U and A separately, the host doubles U
  const lane_t<F> u = block_sum<F>(r, sm, width);
  const lane_t<F> a = block_sum<F>(acc, sm, width);
  if (i != 0) return;
  quad_st(&out_u[w], u);
  quad_st(&out_a[w], a);
}

// ------------------------------------------------------ fixed-base tables
// table record (w * n + i) = affine 2^(c w) P_i, stored (x, y) like a zkey
// section, for w < W = 254 / c + 1.  With these, all windows of a fixed-base
// MSM share one bucket set: one bucket reduction instead of W, and no
// doubling chain between windows.
//
// The affine conversions share inversions (Montgomery's trick): a thread
// doubles through kPreChunk windows, writing each multiple's X, Y into its
// table record and keeping ZZ, ZZZ and the running product of the ZZZs, then
// inverts that product once and walks back, so a chunk costs one inversion
// and ~7 products per record instead of one inversion per record.
constexpr int kPreChunk = 8;

template <class F>
__global__ void __launch_bounds__(128) k_msm_precompute(const F* __restrict__ px,
                                                        const F* __restrict__ py, uint32_t pstride,
                                                        size_t n, int c, int W,
                                                        F* __restrict__ table) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const F x = ld_pod(px + i * pstride), y = ld_pod(py + i * pstride);
  st_pod(table + 2 * i, x);
  st_pod(table + 2 * i + 1, y);
  const bool inf = fe_is_zero(x) && fe_is_zero(y);
  xyzz<F> acc;
  if (!inf) acc = xyzz<F>{x, y, fe_one_of<F>(), fe_one_of<F>()};
  for (int w0 = 1; w0 < W; w0 += kPreChunk) {
    const int cnt = min(kPreChunk, W - w0);
    F zz[kPreChunk], zzz[kPreChunk], pre[kPreChunk];
    F prod = fe_one_of<F>();
    for (int k = 0; k < cnt; k++) {
      const size_t rec = (size_t)(w0 + k) * n + i;
      if (!inf)
        for (int d = 0; d < c; d++) acc = xyzz_dbl(acc);
      // a multiple at infinity (only for points outside the order-r
      // subgroup) takes 1 in the product and is written as (0, 0)
      const bool at_inf = inf || xyzz_is_inf(acc);
      zz[k] = at_inf ? fe_zero_of<F>() : acc.zz;
      zzz[k] = at_inf ? fe_one_of<F>() : acc.zzz;
      prod = prod * zzz[k];
      pre[k] = prod;
      st_pod(table + 2 * rec, at_inf ? fe_zero_of<F>() : acc.x);
      st_pod(table + 2 * rec + 1, at_inf ? fe_zero_of<F>() : acc.y);
    }
    F inv = fe_inv(prod);  // 1 / (zzz_0 ... zzz_{cnt-1})
    for (int k = cnt - 1; k >= 0; k--) {
      const F zzzi = k ? inv * pre[k - 1] : inv;  // 1 / zzz_k
      inv = inv * zzz[k];
      if (fe_is_zero(zz[k])) continue;  // stored as (0, 0) already
      const size_t rec = (size_t)(w0 + k) * n + i;
      const F zi = zzzi * zz[k];  // ZZ / ZZZ = 1 / Z
      const F zzi = fe_sqr(zi);   // 1 / ZZ
      st_pod(table + 2 * rec, ld_pod(table + 2 * rec) * zzi);
      st_pod(table + 2 * rec + 1, ld_pod(table + 2 * rec + 1) * zzzi);
    }
  }
}


// Blocks of the persistent level 0 the device holds at once.
template <class F>
int queue_grid() {
  static PerDevice<size_t> known;
  return (int)resident_blocks(known, k_msm_accum0_queue<F, true>, seg_threads<F>(), 0);
}

// The GPU part of one launch chain: a windowed MSM (inst = 1, points from
// ps.x / ps.y) or inst fixed-base MSMs of one window size sharing the chain
// (tables in ps.table).  n_max: the largest instance, n_total: their sum.
template <class F>
MsmResult msm_enqueue(const ScalarSrc& ss, const PointSrc<F>& ps, int inst, size_t n_max,
                      size_t n_total, void* scratch, size_t scratch_bytes, const MsmConfig& cfg,
                      cudaStream_t st, bool fixed, MsmMerge* merge_out = nullptr,
                      const MsmMerge* merge_in = nullptr) {
  constexpr bool g2 = sizeof(F) == 64;
  ZK_REQUIRE(n_max < (size_t(1) << 31), ZK_EINVAL, "msm: too many points (max 2^31 - 1)");
  ZK_REQUIRE(inst >= 1 && inst <= kMaxInst, ZK_EINVAL, "msm: 1..64 instances per launch");
  const Shape s = make_shape(n_total, g2, cfg, fixed, inst);
  ZK_REQUIRE(!fixed || (size_t)s.W * n_max < (size_t(1) << 31), ZK_EINVAL,
             "msm: fixed-base table too large (windows x points >= 2^31)");
  ZK_REQUIRE(s.c >= 4 && s.c <= 24, ZK_EINVAL, "msm: window size must be in [4, 24]");
  ZK_REQUIRE(s.records < (size_t(1) << 32) - 1, ZK_EINVAL, "msm: too many (point, window) records");
  ZK_REQUIRE(!fixed || (size_t)inst * s.B < kInvalid, ZK_EINVAL, "msm: too many buckets");
  Layout<F> L = carve<F>(scratch, s);
  ZK_REQUIRE(L.bytes <= scratch_bytes, ZK_EINVAL, "msm: scratch buffer too small");

  ZK_CUDA(cudaMemsetAsync(L.counts, 0, (s.entries + 1) * sizeof(uint32_t), st));
  ZK_CUDA(cudaMemsetAsync(L.buckets, 0, (size_t)s.Wk * s.B * sizeof(xyzz<F>), st));
  const int th = 256;
  const dim3 g((unsigned)((n_max + th - 1) / th), (unsigned)inst);
  if (n_max) {
    if (fixed)
      k_msm_hist<true><<<g, th, 0, st>>>(ss, s.c, s.W, s.B, L.counts);
    else
      k_msm_hist<false><<<g, th, 0, st>>>(ss, s.c, s.W, s.B, L.counts);
    ZK_LAUNCHED();
  }
  scan::exclusive(L.counts, L.cursor, s.entries, L.tiles, st);
  if (n_max) {
    if (fixed)
      k_msm_scatter<true><<<g, th, 0, st>>>(ss, s.c, s.W, s.B, L.cursor, L.srec);
    else
      k_msm_scatter<false><<<g, th, 0, st>>>(ss, s.c, s.W, s.B, L.cursor, L.srec);
    ZK_LAUNCHED();
  }
  const uint32_t* total_p = L.counts + (s.entries - 1);
  // level 0
  {
    uint32_t* ok = s.levels > 1 ? L.pkey[1] : nullptr;
    ProfScope prof(g2 ? kProfAccumG2 : kProfAccumG1, (double)n_total, st);
    const unsigned blocks = (unsigned)s.lvl_blocks[0];
    bool affine = false;
    if constexpr (g2) {
      affine = s.affine != 0;
      if (affine) {
        const bool three = affine_blocks(s.records) == 3;
        const auto run = fixed ? (three ? affine_enqueue<true, 3> : affine_enqueue<true, 4>)
                               : (three ? affine_enqueue<false, 3> : affine_enqueue<false, 4>);
        run(L.srec, total_p, ps, s.records, L.aff, L.buckets, ok, L.ppt[1], blocks, st);
      }
    }
    if (!affine) {
      if (fixed && inst > 1) {
        const unsigned grid = std::min(blocks, (unsigned)queue_grid<F>());
        k_msm_accum0_queue<F, true><<<grid, seg_threads<F>(), 0, st>>>(
            L.srec, total_p, ps, s.k0, L.buckets, ok, L.ppt[1], blocks, L.tileq);
      } else {
        const auto kern = fixed ? k_msm_accum0<F, true> : k_msm_accum0<F, false>;
        kern<<<blocks, seg_threads<F>(), 0, st>>>(L.srec, total_p, ps, s.k0, L.buckets, ok,
                                                  L.ppt[1]);
      }
      ZK_LAUNCHED();
    }
  }
  for (int l = 1; l < s.levels; l++) {
    const int in = l & 1, out = in ^ 1;
    uint32_t* ok = (l + 1 < s.levels) ? L.pkey[out] : nullptr;
    k_msm_accumN<F><<<(unsigned)s.lvl_blocks[l], lvl_nodes<F>() * quad_lanes<F>(),
                      lvl_nodes<F>() * sizeof(SegNode<F>), st>>>(
        L.pkey[in], L.ppt[in], s.lvl_records[l], s.lvl_k[l], L.buckets, ok, L.ppt[out]);
    ZK_LAUNCHED();
  }
  const size_t nbuckets = (size_t)s.Wk * s.B;
  if (merge_out && inst == 1) {
    // producer: the consumer reduces these buckets together with its own
    merge_out->buckets = L.buckets;
    merge_out->count = nbuckets;
    merge_out->c = s.c;
    merge_out->fixed = fixed;
    merge_out->g2 = g2;
    if (merge_out->ready) ZK_CUDA(cudaEventRecord(merge_out->ready, st));
    MsmResult none;
    none.c = s.c;
    return none;
  }
  if (merge_in) {
    ZK_REQUIRE(merge_in->buckets, ZK_EINTERNAL, "msm: merged MSM left no buckets");
    ZK_REQUIRE(inst == 1 && merge_in->count == nbuckets && merge_in->c == s.c &&
                   merge_in->fixed == fixed && merge_in->g2 == g2,
               ZK_EINTERNAL, "msm: merged bucket sets differ in shape");
    ZK_CUDA(cudaStreamWaitEvent(st, merge_in->ready, 0));
    k_msm_bucket_add<F><<<(unsigned)((nbuckets + 127) / 128), 128, 0, st>>>(
        L.buckets, static_cast<const xyzz<F>*>(merge_in->buckets), nbuckets);
    ZK_LAUNCHED();
  }
  int log_span = 0;
  {
    uint32_t J = (uint32_t)s.J;
    const uint32_t Lc = (uint32_t)s.chunk;
    while ((1u << log_span) < Lc) log_span++;
    const size_t tot = (size_t)s.Wk * J;
    k_msm_reduce_l1<F><<<(unsigned)((quad_lanes<F>() * tot + 127) / 128), 128, 0, st>>>(
        L.buckets, s.fixed ? 0 : s.c, s.Wk, s.B, Lc, J, L.rrun[0], L.racc[0]);
    ZK_LAUNCHED();
    int cur = 0;
    for (;;) {
      constexpr int kRedT = red_pairs<F>();
      const uint32_t Jout = (J + kRedT - 1) / kRedT;
      k_msm_reduce_blk<F><<<dim3(Jout, s.Wk), kRedT * quad_lanes<F>(), 0, st>>>(
          L.rrun[cur], L.racc[cur], J, log_span, Jout, L.rrun[cur ^ 1], L.racc[cur ^ 1], L.outua,
          L.outua + s.Wk);
      ZK_LAUNCHED();
      if (Jout == 1) break;
      cur ^= 1;
      J = Jout;
      log_span += g2 ? 6 : 7;  // log2 of the pairs per block
    }
  }
  MsmResult res;
  res.d_data = L.outua;
  res.bytes = (size_t)2 * s.Wk * sizeof(xyzz<F>);
  res.windows = s.Wk;
  res.c = s.c;
  res.log_span = log_span;
  return res;
}

}  // namespace

// Defaults, from sweeps of lone MSMs over sizes 2^8 .. 2^22 (tables 2^10 ..
// 2^20) and of whole 2^13 .. 2^20 proofs.  Small MSMs are bound by the depth
// of their dependent additions, so they take short per-thread runs, few
// buckets and short reduction chains; sizes count by the nearest power of two
// (a circuit's point sets are a little larger than its domain).
namespace {
int nearest_log2(size_t n) {
  int lg = 0;
  while (lg < 63 && (size_t(1) << lg) < n) lg++;
  // below 2^(lg - 1/2): n^2 < 2^(2 lg - 1)
  if (lg && lg < 32 && n * n < (size_t(1) << (2 * lg - 1))) lg--;
  return lg;
}
}  // namespace

// Window bits: 6 up to 2^10 points (777 points on G1: 0.30 ms, with 4 bits
// 0.33, with 8 0.31), lg - 5 up to 2^17 (2^16 points: 11 bits 0.74 ms, 12 0.77,
// 13 0.82; 2^17: 12 bits 1.08, 13 1.11, 15 1.12), then 15 (2^18 points: 1.62,
// 13 bits 1.68, 14 1.69; 2^20: 4.33 ms, 16 bits 4.34; a third shorter runs of
// zero digits on circom-like scalars: 2.08 against 2.17), 16 from 2^22 and one
// more per doubling beyond.  On G2, whose affine accumulation likes long
// runs, 11 at 2^17 (2.25 ms, 12 bits 2.42) and 13 at 2^18 (3.47, 15 bits 3.68).
int msm_default_c(size_t n, bool g2) {
  const int lg = nearest_log2(n);
  if (lg <= 17) return std::max(6, g2 && lg == 17 ? lg - 6 : lg - 5);
  if (g2 && lg == 18) return 13;
  return lg < 22 ? 15 : std::min(lg - 6, 20);
}

int msm_effective_c(size_t n, bool g2, const MsmConfig& cfg) {
  return cfg.c > 0 ? cfg.c : msm_default_c(n, g2);
}

// Sorted records per thread of the XYZZ accumulation: 8 up to 2^13 points
// (fixed-base 2^12: 0.32 against 0.35 ms with 16), growing to 64 at 2^20
// (windowed 2^19: 32 2.51 ms, 128 2.96, whose blocks make 1.2 waves), 128 from
// 2^22 windowed.  Whole 2^20 proofs with tables: 64 19.0 ms, 32 19.4, 128 19.3.
// Windowed sets around 2^18 take 16, whose shorter blocks end the last wave
// sooner: 190000 points 1.36 ms, 32 1.39; 2^18 1.62 and 1.64; 300007 1.75 and
// 1.76, with circom-like scalars 1.14 and 1.18 (2^18 of those: 1.07 and 1.05).
int msm_default_k0(size_t n, bool fixed) {
  const int lg = nearest_log2(n);
  if (lg <= 13) return 8;
  if (lg <= 15) return 16;
  if (lg == 18 && !fixed) return 16;
  if (lg <= 19) return 32;
  return fixed || lg < 22 ? 64 : 128;
}

// Buckets per lane group of the first reduction level, from the buckets of
// all sets: enough groups to keep the device busy, then longer chains instead
// of more groups for the block passes above.  Fixed-base sets (few, large):
// 8192 groups (G1; 2^17 buckets 16: 1.34 ms, 32 1.39) or 4096 groups of eight
// lanes (G2); windowed ones ~3100, since every window has a block pass of its
// own (2^16 points, 24 windows of 2^10: 8 0.74 ms, 16 0.77).
int msm_default_chunk(size_t buckets, bool fixed, bool g2) {
  const size_t groups = !fixed ? 3100 : (g2 ? 4096 : 8192);
  const int most = fixed || buckets > 400000 ? 32 : 16;
  int chunk = 2;
  while (chunk < most && groups * chunk < buckets) chunk *= 2;
  return chunk;
}

namespace {
Shape shape_for(size_t n, bool g2, const MsmConfig& cfg, int fixed_c) {
  MsmConfig k = cfg;
  if (fixed_c) k.c = fixed_c;
  return make_shape(n, g2, k, fixed_c != 0);
}
}  // namespace

MsmConfig msm_resolve(size_t n, bool g2, const MsmConfig& cfg, int fixed_c) {
  const Shape s = shape_for(n, g2, cfg, fixed_c);
  MsmConfig k = cfg;
  k.c = s.c;
  k.k0 = s.k0;
  k.chunk = s.chunk;
  return k;
}

bool msm_takes_affine(size_t n, bool g2, const MsmConfig& cfg, int fixed_c) {
  return shape_for(n, g2, cfg, fixed_c).affine != 0;
}

size_t msm_scratch_bytes(size_t n, bool g2, const MsmConfig& cfg) {
  const Shape s = make_shape(n, g2, cfg);
  if (g2) return carve<fp2_t>(nullptr, s).bytes;
  return carve<fp_t>(nullptr, s).bytes;
}

size_t msm_table_bytes(size_t n, bool g2, int c) {
  return (size_t)(254 / c + 1) * n * (g2 ? 128 : 64);
}

size_t msm_scratch_bytes_fixed(size_t n, bool g2, int c, const MsmConfig& cfg, int inst) {
  MsmConfig k = cfg;
  k.c = c;
  const Shape s = make_shape(n, g2, k, true, inst);
  if (g2) return carve<fp2_t>(nullptr, s).bytes;
  return carve<fp_t>(nullptr, s).bytes;
}

void msm_precompute(bool g2, const PointsView& pts, size_t n, int c, void* table, cudaStream_t st) {
  ZK_REQUIRE(c >= 4 && c <= 24, ZK_EINVAL, "msm table: window size must be in [4, 24]");
  if (!n) return;
  const int W = 254 / c + 1;
  const unsigned g = (unsigned)((n + 127) / 128);
  if (g2)
    k_msm_precompute<fp2_t><<<g, 128, 0, st>>>(reinterpret_cast<const fp2_t*>(pts.x),
                                               reinterpret_cast<const fp2_t*>(pts.y), pts.stride, n,
                                               c, W, reinterpret_cast<fp2_t*>(table));
  else
    k_msm_precompute<fp_t><<<g, 128, 0, st>>>(reinterpret_cast<const fp_t*>(pts.x),
                                              reinterpret_cast<const fp_t*>(pts.y), pts.stride, n,
                                              c, W, reinterpret_cast<fp_t*>(table));
  ZK_LAUNCHED();
}

namespace {
template <class F>
MsmResult enqueue_fixed_multi(int inst, const void* const* tables, const uint64_t* const* scalars,
                              const size_t* n, int c, void* scratch, size_t bytes,
                              const MsmConfig& cfg, cudaStream_t st, MsmMerge* merge_out = nullptr,
                              const MsmMerge* merge_in = nullptr) {
  ZK_REQUIRE(inst >= 1 && inst <= kMaxInst, ZK_EINVAL, "msm: 1..64 instances per launch");
  MsmConfig k = cfg;
  k.c = c;
  ScalarSrc ss{};
  PointSrc<F> ps{};
  ps.bshift = c - 1;
  size_t n_max = 0, n_total = 0;
  for (int i = 0; i < inst; i++) {
    ZK_REQUIRE(n[i] < (size_t(1) << 31), ZK_EINVAL, "msm: too many points (max 2^31 - 1)");
    ss.sc[i] = scalars[i];
    ss.n[i] = (uint32_t)n[i];
    ps.table[i] = reinterpret_cast<const F*>(tables[i]);
    n_max = std::max(n_max, n[i]);
    n_total += n[i];
  }
  return msm_enqueue<F>(ss, ps, inst, n_max, n_total, scratch, bytes, k, st, true, merge_out,
                       merge_in);
}

template <class F>
MsmResult enqueue_windowed(const PointsView& pts, const uint64_t* scalars, size_t n, void* scratch,
                           size_t bytes, const MsmConfig& cfg, cudaStream_t st,
                           MsmMerge* merge_out = nullptr, const MsmMerge* merge_in = nullptr) {
  ScalarSrc ss{};
  ss.sc[0] = scalars;
  ss.n[0] = (uint32_t)std::min(n, size_t(0xffffffffu));
  PointSrc<F> ps{};
  ps.x = reinterpret_cast<const F*>(pts.x);
  ps.y = reinterpret_cast<const F*>(pts.y);
  ps.stride = pts.stride;
  return msm_enqueue<F>(ss, ps, 1, n, n, scratch, bytes, cfg, st, false, merge_out, merge_in);
}
}  // namespace

MsmResult msm_enqueue_fixed(bool g2, const void* table, const uint64_t* scalars, size_t n, int c,
                            void* scratch, size_t bytes, const MsmConfig& cfg, cudaStream_t st,
                            MsmMerge* merge_out, const MsmMerge* merge_in) {
  if (g2)
    return enqueue_fixed_multi<fp2_t>(1, &table, &scalars, &n, c, scratch, bytes, cfg, st,
                                      merge_out, merge_in);
  return enqueue_fixed_multi<fp_t>(1, &table, &scalars, &n, c, scratch, bytes, cfg, st, merge_out,
                                   merge_in);
}

MsmResult msm_enqueue_fixed_multi(bool g2, int inst, const void* const* tables,
                                  const uint64_t* const* scalars, const size_t* n, int c,
                                  void* scratch, size_t bytes, const MsmConfig& cfg,
                                  cudaStream_t st) {
  if (g2) return enqueue_fixed_multi<fp2_t>(inst, tables, scalars, n, c, scratch, bytes, cfg, st);
  return enqueue_fixed_multi<fp_t>(inst, tables, scalars, n, c, scratch, bytes, cfg, st);
}

MsmResult msm_g1_enqueue(const PointsView& pts, const uint64_t* scalars, size_t n, void* scratch,
                         size_t bytes, const MsmConfig& cfg, cudaStream_t st, MsmMerge* merge_out,
                         const MsmMerge* merge_in) {
  return enqueue_windowed<fp_t>(pts, scalars, n, scratch, bytes, cfg, st, merge_out, merge_in);
}
MsmResult msm_g2_enqueue(const PointsView& pts, const uint64_t* scalars, size_t n, void* scratch,
                         size_t bytes, const MsmConfig& cfg, cudaStream_t st) {
  return enqueue_windowed<fp2_t>(pts, scalars, n, scratch, bytes, cfg, st);
}

namespace {
host::Fp fp_from_words(const uint32_t* w) {
  host::Fp r;
  memcpy(r.v, w, 32);
  return r;
}
host::Fp2 fp2_from_words(const uint32_t* q) { return host::Fp2{fp_from_words(q), fp_from_words(q + 8)}; }

// window w = A_w + 2^log_span U_w, then Horner over windows with c doublings
template <class T, class Load>
host::Xyzz<T> combine(const uint8_t* data, const MsmResult& r, size_t pt_bytes, Load load) {
  using P = host::Xyzz<T>;
  P acc = P::inf();
  for (int w = r.windows - 1; w >= 0; w--) {
    for (int i = 0; i < r.c && !acc.is_inf(); i++) acc = acc.dbl();
    P u = load(data + (size_t)w * pt_bytes);
    const P a = load(data + (size_t)(r.windows + w) * pt_bytes);
    for (int i = 0; i < r.log_span && !u.is_inf(); i++) u = u.dbl();
    acc = acc.add(u).add(a);
  }
  return acc;
}
}  // namespace

// instance i of a multi-instance result: its (U_i, A_i) as a one-window result
MsmResult gather_instance(const void* h_data, const MsmResult& r, int inst, size_t pt_bytes,
                          uint8_t* buf) {
  const uint8_t* d = reinterpret_cast<const uint8_t*>(h_data);
  memcpy(buf, d + (size_t)inst * pt_bytes, pt_bytes);
  memcpy(buf + pt_bytes, d + (size_t)(r.windows + inst) * pt_bytes, pt_bytes);
  MsmResult one = r;
  one.windows = 1;
  one.bytes = 2 * pt_bytes;
  return one;
}

bool msm_g1_combine_inst(const void* h_data, const MsmResult& r, int inst, uint64_t out[8]) {
  alignas(16) uint8_t buf[256];
  const MsmResult one = gather_instance(h_data, r, inst, 128, buf);
  return msm_g1_combine(buf, one, out);
}

bool msm_g2_combine_inst(const void* h_data, const MsmResult& r, int inst, uint64_t out[16]) {
  alignas(16) uint8_t buf[512];
  const MsmResult one = gather_instance(h_data, r, inst, 256, buf);
  return msm_g2_combine(buf, one, out);
}

host::Xyzz<host::Fp> msm_g1_combine_xyzz(const void* h_data, const MsmResult& r, int inst) {
  using P = host::Xyzz<host::Fp>;
  alignas(16) uint8_t buf[256];
  MsmResult one = r;
  if (inst >= 0) {
    one = gather_instance(h_data, r, inst, 128, buf);
    h_data = buf;
  }
  return combine<host::Fp>(reinterpret_cast<const uint8_t*>(h_data), one, 128,
                           [](const uint8_t* p) {
                             const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
                             return P{fp_from_words(q), fp_from_words(q + 8), fp_from_words(q + 16),
                                      fp_from_words(q + 24)};
                           });
}

host::Xyzz<host::Fp2> msm_g2_combine_xyzz(const void* h_data, const MsmResult& r, int inst) {
  using P = host::Xyzz<host::Fp2>;
  alignas(16) uint8_t buf[512];
  MsmResult one = r;
  if (inst >= 0) {
    one = gather_instance(h_data, r, inst, 256, buf);
    h_data = buf;
  }
  return combine<host::Fp2>(reinterpret_cast<const uint8_t*>(h_data), one, 256,
                            [](const uint8_t* p) {
                              const uint32_t* q = reinterpret_cast<const uint32_t*>(p);
                              return P{fp2_from_words(q), fp2_from_words(q + 16),
                                       fp2_from_words(q + 32), fp2_from_words(q + 48)};
                            });
}

bool msm_g1_combine(const void* h_data, const MsmResult& r, uint64_t out[8]) {
  host::Fp x, y;
  const bool inf = msm_g1_combine_xyzz(h_data, r).to_affine(x, y);
  memcpy(out, x.v, 32);
  memcpy(out + 4, y.v, 32);
  return inf;
}

bool msm_g2_combine(const void* h_data, const MsmResult& r, uint64_t out[16]) {
  host::Fp2 x, y;
  const bool inf = msm_g2_combine_xyzz(h_data, r).to_affine(x, y);
  memcpy(out, x.c0.v, 32);
  memcpy(out + 4, x.c1.v, 32);
  memcpy(out + 8, y.c0.v, 32);
  memcpy(out + 12, y.c1.v, 32);
  return inf;
}

bool msm_g1_run(const PointsView& pts, const uint64_t* scalars, size_t n, DeviceBuffer& scratch,
                const MsmConfig& cfg, cudaStream_t st, uint64_t out[8]) {
  scratch.ensure(msm_scratch_bytes(n, false, cfg));
  const MsmResult r = msm_g1_enqueue(pts, scalars, n, scratch.ptr, scratch.cap, cfg, st);
  std::vector<uint8_t> h(r.bytes);
  ZK_CUDA(cudaMemcpyAsync(h.data(), r.d_data, r.bytes, cudaMemcpyDeviceToHost, st));
  ZK_CUDA(cudaStreamSynchronize(st));
  return msm_g1_combine(h.data(), r, out);
}

bool msm_g2_run(const PointsView& pts, const uint64_t* scalars, size_t n, DeviceBuffer& scratch,
                MsmConfig cfg, cudaStream_t st, uint64_t out[16]) {
  msm_ensure_scratch(scratch, cfg,
                     [&](const MsmConfig& k) { return msm_scratch_bytes(n, true, k); });
  const MsmResult r = msm_g2_enqueue(pts, scalars, n, scratch.ptr, scratch.cap, cfg, st);
  std::vector<uint8_t> h(r.bytes);
  ZK_CUDA(cudaMemcpyAsync(h.data(), r.d_data, r.bytes, cudaMemcpyDeviceToHost, st));
  ZK_CUDA(cudaStreamSynchronize(st));
  return msm_g2_combine(h.data(), r, out);
}

}  // namespace zk
