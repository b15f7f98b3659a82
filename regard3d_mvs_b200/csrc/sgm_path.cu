// Full-range SGM tiles as eight chain passes.
//
// Semantics are those of sgm.cu (Census costs, the 8-path recurrence with
// sentinel labels, the sum modulo 2^16, winner-takes-all and the acceptance
// rules of rhiestan/Regard3D_MVS src/r3d/stereo/stereo_matcher.cpp:305-353,
// 446-525 and sgm_kernels.cpp:176-263, 387-403). Because the aggregated cost
// is a sum of 8 independent 1-D recurrences restarted at tile borders, each
// path direction is a set of independent chains: the tile's rows for the
// horizontal paths, its columns for the vertical ones and its diagonals for
// the diagonal ones. This file runs them that way:
//
//   cost kernel     u8 costs of every cell of the wave (written once);
//   8 path passes   G lanes walk one chain, K label pairs per lane, 32 / G
//                   chains per warp, the predecessor vector in registers, the
//                   next pixels' costs streaming into a shared-memory ring.
//                   Each writes its path's byte terms, all eight in one launch
//                   (or, with a P2 above 255, adds to u16 sums, two a launch);
//   winner kernel   total sums, winner-takes-all, acceptance rules, subpixel
//                   fit and confidence per pixel, into the tile's disparity
//                   and confidence.
//
// No CTA barrier is on the chain's critical path and every tile spreads over
// as many SMs as it has chains, so one small pair fills the GPU as well as a
// batch does. Bytes per aggregated cell with terms: 1 cost write, 8 cost
// reads (6 of them from DRAM on a 2048x1536 pair of 128 labels: a tile's
// directions run close together, but the terms they write, eight times the
// costs, push the costs out of L2), 8 term writes, 9 reads.
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "common.cuh"
#include "sgm_path.h"
#include "sgm_simd.cuh"
#include "tuning.h"

namespace r3dgpu {

namespace {

using sgm_simd::group_umin;
using sgm_simd::kSent2;
constexpr float kInfF = __builtin_huge_valf();
constexpr int kPathThreads = 256;
constexpr int kPathMaxLabels = 768;  // more go to the one-CTA-per-tile kernels
constexpr int kPathCounters = 256;  // block counters of a wave's launches (one each)

inline size_t align256(size_t v) { return (v + 255) & ~static_cast<size_t>(255); }

// Last job whose prefix value (field selected by `key`) is <= v; jobs are
// ordered so that every prefix is non-decreasing.
template <class Key>
R3D_DEVICE int find_job(const SgmPathJob* jobs, int njobs, int64_t v, Key key) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (key(jobs[mid]) <= v) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Whether the caller's cancellation flag is set (read once per chain block,
// by lane 0 for the whole warp; never a wait).
R3D_DEVICE bool cancelled(const int* cancel) {
  int c = 0;
  if (cancel != nullptr) c = *reinterpret_cast<const volatile int*>(cancel);
  return r3dsimt::shfl(static_cast<uint32_t>(c), 0) != 0;
}

// Start pixel and length of chain c of a direction (dx, dy) in a w x h tile;
// length 0 for c past the class's last chain.
R3D_DEVICE void chain_geometry(int cls, int dx, int dy, int w, int h, int64_t c, int& sx, int& sy, int& len) {
  sx = 0;
  sy = 0;
  len = 0;
  if (cls == 0) {
    if (c < h) {
      sx = dx > 0 ? 0 : w - 1;
      sy = static_cast<int>(c);
      len = w;
    }
  } else if (cls == 1) {
    if (c < w) {
      sx = static_cast<int>(c);
      sy = dy > 0 ? 0 : h - 1;
      len = h;
    }
  } else if (c < w) {
    const int ci = static_cast<int>(c);
    sx = dx > 0 ? ci : w - 1 - ci;
    sy = dy > 0 ? 0 : h - 1;
    len = r3dsimt::imin(h, w - ci);
  } else if (c < static_cast<int64_t>(w) + h - 1) {
    const int k = static_cast<int>(c - w + 1);
    sx = dx > 0 ? 0 : w - 1;
    sy = dy > 0 ? k : h - 1 - k;
    len = r3dsimt::imin(w, h - k);
  }
}

// ---------------------------------------------------------------- costs
// C(p, a) of stereo_matcher.cpp:305-353, u8. One warp per tile row: the
// partner Census codes the row can reach (right columns x0 - dmin - nd + 1 ..
// x0 + w - 1 - dmin) are staged in the warp's shared memory, then the lanes
// take 32 consecutive pixels and write 32 labels (one sector) at a time.
constexpr int kCostStage = 2048;  // staged partner codes per warp at most (sgm_path_fits: w + nd - 1 <= 2048)

// Label of byte i of word w of a run of 16-label units (the byte order of
// unpack_unit).
R3D_DEVICE int unit_label(int w, int i) { return 16 * (w >> 2) + 2 * (w & 3) + (i & 1) + 8 * (i >> 1); }

// `stage_words` (<= kCostStage): the widest staged row of the wave (tile
// width + labels - 1), so that narrow waves run more CTAs per SM.
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_cost_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                         int64_t rows, uint8_t* R3D_RESTRICT cost, int stage_words, uint16_t* R3D_RESTRICT ints,
                         int* R3D_RESTRICT counters) {
  R3D_DYNAMIC_SMEM(smem);
  if (blockIdx.x == 0 && threadIdx.x < kPathCounters) counters[threadIdx.x] = 0;
  const int lane = static_cast<int>(threadIdx.x & 31u), warp = static_cast<int>(threadIdx.x >> 5);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  uint64_t* stage = reinterpret_cast<uint64_t*>(smem) + static_cast<size_t>(warp) * stage_words;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * wpb + warp; r < rows; r += nwarps) {
    const int j = find_job(jobs, njobs, r, [](const SgmPathJob& q) { return q.row_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    const int nd = m.nd, w = job.w;
    const int y = static_cast<int>(r - job.row_off), by = job.y0 + y;
    const RowInterval lv = m.bv[by], rv = m.pv[by];
    const uint64_t* crow = m.cpart + static_cast<int64_t>(by) * m.cp_stride;
    const uint64_t* lrow = m.cbase + static_cast<int64_t>(by) * m.cb_stride;
    // Staged right column xr is stage[xr - xr0]; columns outside the valid
    // right interval are never read (their cost is invalid_cost).
    const int xr0 = job.x0 - m.dmin - nd + 1;
    const int span = w + nd - 1;
    r3dsimt::syncwarp();
    for (int k = lane; k < span; k += 32) {
      const int xr = xr0 + k;
      stage[k] = (xr >= rv.first && xr <= rv.last) ? crow[xr] : 0;
    }
    // The row's base intensities, for the pass kernels.
    {
      const uint16_t* irow = m.base + static_cast<int64_t>(by) * m.base_stride + job.x0;
      uint16_t* iout = ints + job.px_off + static_cast<int64_t>(y) * w;
      for (int x = lane; x < w; x += 32) iout[x] = irow[x];
    }
    r3dsimt::syncwarp();
    const uint32_t inv = static_cast<uint32_t>(m.invalid_cost);
    uint8_t* row_out = cost + job.cell_off + static_cast<int64_t>(y) * w * nd;
    for (int xb = 0; xb < w; xb += 32) {
      const int x = xb + lane;
      if (x >= w) continue;
      const int bx = job.x0 + x;
      const bool inside = bx >= lv.first && bx <= lv.last;
      const uint64_t cl = inside ? lrow[bx] : 0;
      uint8_t* out = row_out + static_cast<int64_t>(x) * nd;
      for (int c = 0; c < nd; c += 32) {
        const int nl = nd - c < 32 ? 16 : 32;  // nd is a multiple of 16
        uint32_t q[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        if (inside) {
          // Label a = c + k reads right column bx - dmin - a = xr0 + (x + nd - 1 - a).
          const int base = x + nd - 1 - c;
          const int xr_first = bx - m.dmin - c;  // right column of label c; label c + k reads xr_first - k
          if (xr_first <= rv.last && xr_first - (nl - 1) >= rv.first) {
            // Every label of the run reads a valid right column: four costs a
            // word, the two 32-bit popcounts of each Census XOR packed
            // separately by multiply-adds (each byte at most 32, no carries).
#pragma unroll
            for (int w4 = 0; w4 < 8; ++w4) {
              if (4 * w4 < nl) {
                uint32_t lo = 0, hi = 0;
#pragma unroll
                for (int i = 3; i >= 0; --i) {
                  const uint64_t d = cl ^ stage[base - unit_label(w4, i)];
                  lo = lo * 256u + static_cast<uint32_t>(r3dsimt::popc(static_cast<uint32_t>(d)));
                  hi = hi * 256u + static_cast<uint32_t>(r3dsimt::popc(static_cast<uint32_t>(d >> 32)));
                }
                q[w4] = lo + hi;
              }
            }
          } else {
#pragma unroll
            for (int k = 0; k < 32; ++k) {
              if (k < nl) {
                const int xr = xr_first - k;
                const bool ok = xr >= rv.first && xr <= rv.last;
                const uint32_t v = ok ? static_cast<uint32_t>(r3dsimt::popc64(cl ^ stage[base - k])) : inv;
                q[4 * (k >> 4) + ((k & 7) >> 1)] |= v << (8 * ((k & 1) + 2 * ((k >> 3) & 1)));
              }
            }
          }
        }
        *reinterpret_cast<uint4*>(out + c) = make_uint4(q[0], q[1], q[2], q[3]);
        if (nl == 32) *reinterpret_cast<uint4*>(out + c + 16) = make_uint4(q[4], q[5], q[6], q[7]);
      }
    }
  }
}

// ---------------------------------------------------------------- passes
// Pass modes. With byte terms (every P2 <= 255) every direction writes its
// path's term T_r = L_r - C (in [0, P2]) as one byte per cell, and the
// per-pixel kernel forms S = 8 C + sum T_r (at most 8 (255 + 255) < 2^16, so
// the sum modulo 2^16 is the plain sum). With u16 sums (any penalties) the
// first launch writes the sums and the next ones add to them, two directions a
// launch, each with a volume of its own, where the scratch holds two: more
// chains in flight for the same bytes (P2 = 600, one volume and two: 640x480
// pair, 128 labels 1.58 and 1.08 ms; 1024x768, 512 labels 8.45 and 7.65;
// 2048x1536, 128 labels 9.2 and 8.4, where an adding launch runs at 0.88 of the
// copy rate; four levels of a 3072x2048 pair 29.4 and 19.2).
enum PassMode { kFirst = 0, kAccumulate = 1, kTerm = 3 };
constexpr int kTermArrays = 8;
constexpr int kMaxPasses = 8;
// The passes of one launch: n directions (slot = its term array), their
// number per chain class, and the chain blocks of all of them together. The
// blocks are numbered tile after tile, within a tile direction after
// direction: the directions of a tile run close together, so that some of its
// cost reads are served by L2 (2 of 8 on a 2048x1536 pair of 128 labels; seven
// of its directions took 2.84 ms direction after direction, 2.38 in this order).
struct PassSet {
  int n;
  uint32_t one;  // 1 (see fma_add)
  int cls[kMaxPasses], dx[kMaxPasses], dy[kMaxPasses], slot[kMaxPasses];
  int per_class[kPathClasses];
  int64_t total;
  int* next;  // the next block to hand out after one per resident warp (zeroed with the wave)
};

// The block a warp takes after its current one: warps take one each to begin
// with, then the next free one, since blocks differ in length (diagonals, wide
// ranges): a fixed stride left a second round half empty.
R3D_DEVICE int64_t next_block(const PassSet& ps, int64_t nwarps) {
  uint32_t n = 0;
  if (r3dsimt::lane_id() == 0) n = static_cast<uint32_t>(atomicAdd(ps.next, 1));
  return nwarps + static_cast<int64_t>(r3dsimt::shfl(n, 0));
}

// Tile j, direction and chain block (returned: the block's number within its
// tile and direction, of CPW chains) of block gblk of the launch.
template <int CPW>
R3D_DEVICE int64_t locate_block(const SgmPathJob* jobs, int njobs, const PassSet& ps, int64_t gblk, int& j, int& cls,
                                int& dx, int& dy, int& slot) {
  const int64_t n0 = ps.per_class[0], n1 = ps.per_class[1], n2 = ps.per_class[2];
  auto key = [n0, n1, n2](const SgmPathJob& q) { return n0 * q.blk[0] + n1 * q.blk[1] + n2 * q.blk[2]; };
  j = find_job(jobs, njobs, gblk, key);
  const SgmPathJob& job = jobs[j];
  int64_t blk = gblk - key(job);
  cls = ps.cls[0];
  dx = ps.dx[0];
  dy = ps.dy[0];
  slot = ps.slot[0];
  bool found = false;
#pragma unroll
  for (int q = 0; q < kMaxPasses; ++q) {  // static indices only: no local copy of ps
    if (q < ps.n && !found) {
      const int c = ps.cls[q];
      const int chains = c == 0 ? job.h : (c == 1 ? job.w : job.w + job.h - 1);
      const int nb = (chains + CPW - 1) / CPW;
      if (blk < nb) {
        found = true;
        cls = c;
        dx = ps.dx[q];
        dy = ps.dy[q];
        slot = ps.slot[q];
      } else {
        blk -= nb;
      }
    }
  }
  return blk;
}

// Per-halfword a + b modulo 2^16.
R3D_DEVICE uint32_t add2(uint32_t a, uint32_t b, bool no_carry) { return no_carry ? a + b : r3dsimt::vadd2(a, b); }

// a * one + b with one = 1 at run time: an integer multiply-add, which the
// FMA pipe executes, in place of an add on the ALU pipe (packed minima, masks
// and byte permutes keep the ALU pipe the busier one: 64 lanes per clock each).
R3D_DEVICE uint32_t fma_add(uint32_t a, uint32_t one, uint32_t b) { return a * one + b; }

// Labels of a vector are kept in units of 16: word k = 0..7 of a unit holds
// labels k and k + 8, so that the neighbours d -+ 1 of a word are the words
// next to it. Byte planes (costs, terms) store word j = 0..3 of a unit as the
// bytes of labels 2 j, 2 j + 1, 2 j + 8, 2 j + 9: one mask or permute unpacks a
// word of two labels, one multiply-add packs two of them.
R3D_DEVICE void unpack_unit(const uint4& v, uint32_t* c2) {
  const uint32_t cw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    c2[2 * k] = cw[k] & 0x00FF00FFu;
    c2[2 * k + 1] = r3dsimt::perm(cw[k], 0u, 0x4341u);
  }
}
R3D_DEVICE uint4 pack_unit(const uint32_t* tr) {
  return make_uint4(tr[0] + 256u * tr[1], tr[2] + 256u * tr[3], tr[4] + 256u * tr[5], tr[6] + 256u * tr[7]);
}

// best = min(L(q, d), L(q, d -+ 1) + P1, min L(q) + P2) for N words whose
// labels cl are already clamped to min L(q) + P2 (one 3-way minimum per word
// is left); `below` and `above` hold the clamped labels before the first unit
// (in the high half) and after the last (in the low half).
template <int N>
R3D_DEVICE void best_terms(const uint32_t (&cl)[N], uint32_t below, uint32_t above, uint32_t one, uint32_t p1x2,
                           uint32_t (&best)[N]) {
#pragma unroll
  for (int u = 0; u < N / 8; ++u) {
    // Words -1 and 8 of the unit: labels (16 u - 1, 16 u + 7) and (16 u + 8, 16 u + 16).
    uint32_t s[10];
    s[0] = fma_add(r3dsimt::perm(u > 0 ? cl[u > 0 ? 8 * u - 1 : 0] : below, cl[8 * u + 7], 0x5432u), one, p1x2);
#pragma unroll
    for (int k = 0; k < 8; ++k) s[1 + k] = fma_add(cl[8 * u + k], one, p1x2);
    s[9] = fma_add(r3dsimt::perm(cl[8 * u], 8 * u + 8 < N ? cl[8 * u + 8 < N ? 8 * u + 8 : 0] : above, 0x5432u), one, p1x2);
#pragma unroll
    for (int k = 0; k < 8; ++k) best[8 * u + k] = r3dsimt::vmin3(cl[8 * u + k], s[k], s[2 + k]);
  }
}

// Per-halfword minimum of N words.
template <int N>
R3D_DEVICE uint32_t min_words(const uint32_t (&v)[N]) {
  constexpr int N3 = (N + 2) / 3;
  uint32_t t3[N3];
#pragma unroll
  for (int k = 0; k < N3; ++k)
    t3[k] = r3dsimt::vmin3(v[3 * k], v[3 * k + 1 < N ? 3 * k + 1 : 3 * k], v[3 * k + 2 < N ? 3 * k + 2 : 3 * k]);
  uint32_t m = t3[0];
#pragma unroll
  for (int k = 1; k < N3; k += 2) m = r3dsimt::vmin3(m, t3[k], t3[k + 1 < N3 ? k + 1 : k]);
  return m;
}

// The eight words of unit u of a pixel's total sums, from its cost and term
// bytes (TERMS) or its stored u16 sums (tstride: values to the next array, 0
// with one sum volume).
template <bool TERMS>
R3D_DEVICE void sum_unit(const uint8_t* cp, const uint8_t* tp, int64_t tstride, const uint16_t* sp, int u,
                         uint32_t (&wv)[8]) {
  if constexpr (TERMS) {
    uint4 t[1 + kTermArrays];
    t[0] = r3dsimt::ld_stream(reinterpret_cast<const uint4*>(cp + 16 * u));
#pragma unroll
    for (int r = 0; r < kTermArrays; ++r)
      t[1 + r] = r3dsimt::ld_stream(reinterpret_cast<const uint4*>(tp + r * tstride + 16 * u));
#pragma unroll
    for (int r = 0; r <= kTermArrays; ++r) {
      uint32_t c2[8];
      unpack_unit(t[r], c2);
#pragma unroll
      for (int k = 0; k < 8; ++k) wv[k] = r == 0 ? 8u * c2[k] : wv[k] + c2[k];
    }
  } else {
    auto load = [u](const uint16_t* v, uint32_t (&w)[8]) {
      const uint4 a = reinterpret_cast<const uint4*>(v)[2 * u], b = reinterpret_cast<const uint4*>(v)[2 * u + 1];
      w[0] = a.x;
      w[1] = a.y;
      w[2] = a.z;
      w[3] = a.w;
      w[4] = b.x;
      w[5] = b.y;
      w[6] = b.z;
      w[7] = b.w;
    };
    load(sp, wv);
    if (tstride != 0) {  // a second volume
      uint32_t w2[8];
      load(sp + tstride, w2);
#pragma unroll
      for (int k = 0; k < 8; ++k) wv[k] = r3dsimt::vadd2(wv[k], w2[k]);
    }
  }
}
// Unit u's sums in label order.
R3D_DEVICE void store_unit(uint16_t* vol, const uint32_t (&wv)[8]) {
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    vol[k] = static_cast<uint16_t>(wv[k] & 0xFFFFu);
    vol[k + 8] = static_cast<uint16_t>(wv[k] >> 16);
  }
}

// Per-warp shared-memory ring of the full-range passes: Stages stages, each
// with one pixel per chain of the bytes the pass reads (the cost, and the u16
// sum of the adding passes), then one 4-byte word per lane: the aligned word
// of the intensities that holds its chain's pixel (every lane copies its own,
// since a cp.async wait covers only the waiting thread's copies). 4-warp CTAs
// pack an SM's registers and shared memory finely.
template <int G, int K, int MODE>
struct PathRing {
  static constexpr int kThreads = 128;
  static constexpr int kMinBlocks = K <= 8 ? 8 : 5;
  static constexpr int ND = 2 * G * K;
  static constexpr int kPlanes = MODE == kAccumulate ? 3 : 1;
  // The u16 modes with 4, 5 and 6 stages: 640x480 pair, 128 labels 1.12, 1.08
  // and 1.10 ms; 1024x768, 96 labels 2.07, 1.96 and 1.99; 256: 4.13, 4.13, 4.16.
  static constexpr int kStages = MODE == kTerm ? 8 : 5;
  static constexpr int kPlaneBytes = (32 / G) * kPlanes * ND;
  static constexpr int kStageBytes = kPlaneBytes + 32 * 4;
  static constexpr int kWarpBytes = kStages * kStageBytes;
  // Each warp's rings, then each warp's copy of its match's P2 table.
  static constexpr int kBlockBytes = (kThreads / 32) * (kWarpBytes + 512);
};

// G lanes walk one chain, 2 K consecutive labels per lane (K / 8 units), 32 / G
// chains per warp. The step loop is unrolled by the ring depth NS so that ring
// slots are indexed statically; each chain keeps running pointers (advanced by
// one pixel along the path per step). The first pixel needs no special case:
// with a zero clamp, best = 0, so T = 0 and L = C there. FULL: every unit of
// the group is inside the match's label count.
template <int G, int K, int MODE, bool FULL>
R3D_GLOBAL void R3D_LAUNCH_BOUNDS_MIN((PathRing<G, K, MODE>::kThreads), (PathRing<G, K, MODE>::kMinBlocks))
    sgm_path_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                    const PassSet ps, const uint8_t* R3D_RESTRICT cost, uint16_t* sum, uint8_t* terms,
                    int64_t tstride, const uint16_t* R3D_RESTRICT ints, const int* cancel) {
  constexpr int CPW = 32 / G;  // chains per warp
  constexpr int NV = K / 8;    // units per lane
  constexpr int NS = PathRing<G, K, MODE>::kStages;
  using Ring = PathRing<G, K, MODE>;
  R3D_DYNAMIC_SMEM(smem);
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const int gi = lane / G, t = lane % G;
  const int e0 = 2 * t * K;  // first label of the lane
  const int left_lane = (lane + 31) & 31, right_lane = (lane + 1) & 31;
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  unsigned char* const ring = smem + static_cast<size_t>(threadIdx.x >> 5) * Ring::kWarpBytes;
  // The warp's copy of the P2 table of the match it works on (256 u16),
  // reloaded when a chain block belongs to another match.
  uint16_t* const lut = reinterpret_cast<uint16_t*>(smem + static_cast<size_t>(wpb) * Ring::kWarpBytes +
                                                    static_cast<size_t>(threadIdx.x >> 5) * 512);
  int lut_match = -1;
  unsigned char* const ring_cost = ring + gi * Ring::ND + e0;
  unsigned char* const ring_sum = ring + CPW * Ring::ND + gi * 2 * Ring::ND + 2 * e0;
  unsigned char* const ring_int = ring + Ring::kPlaneBytes + lane * 4;
  const uint32_t one = ps.one;
  for (int64_t gblk = static_cast<int64_t>(blockIdx.x) * wpb + (threadIdx.x >> 5); gblk < ps.total;
       gblk = next_block(ps, nwarps)) {
    if (cancelled(cancel)) break;
    int j, cls, dx, dy, tslot;
    const int64_t blk = locate_block<CPW>(jobs, njobs, ps, gblk, j, cls, dx, dy, tslot);
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    if (job.match != lut_match) {  // the same for the whole warp (one chain block)
      r3dsimt::syncwarp();
      for (int k = lane; k < 128; k += 32)
        reinterpret_cast<uint32_t*>(lut)[k] = reinterpret_cast<const uint32_t*>(m.lut)[k];
      r3dsimt::syncwarp();
      lut_match = job.match;
    }
    const int w = job.w, nd = m.nd;
    const uint32_t p1x2 = static_cast<uint32_t>(m.p1) * 0x10001u;
    const bool no_carry = m.sum_no_carry != 0;
    int sx, sy, len;
    chain_geometry(cls, dx, dy, w, job.h, blk * CPW + gi, sx, sy, len);
    int maxlen = len;
#pragma unroll
    for (int o = G; o < 32; o <<= 1) maxlen = r3dsimt::imax(maxlen, static_cast<int>(r3dsimt::shfl_xor(maxlen, o)));
    bool uvalid[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) uvalid[v] = FULL || e0 + 16 * v < nd;
    // Running pointers of the pixel being issued (NS - 1 ahead) and of the
    // pixel being computed.
    const int64_t dcell = (static_cast<int64_t>(dy) * w + dx) * nd;
    const int64_t cell0 = job.cell_off + e0 + (static_cast<int64_t>(sy) * w + sx) * nd;
    const uint8_t* c_in = cost + cell0;
    const int64_t out0 = cell0 + static_cast<int64_t>(tslot) * tstride;
    const uint16_t* s_in = sum + out0;
    uint16_t* s_out = sum + out0;
    uint8_t* t_out = terms + out0;
    const int64_t dpx = static_cast<int64_t>(dy) * w + dx;
    // Intensity of the pixel being issued (each lane copies the aligned
    // 4-byte word holding it into the stage), and the parity of the
    // chain's first pixel (which half of a staged word holds the intensity:
    // pixel i's parity is par0 ^ (i & dpar)).
    const uint16_t* i_iss = ints + job.px_off + static_cast<int64_t>(sy) * w + sx;
    const uint32_t par0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(i_iss) >> 1) & 1u;
    const uint32_t dpar = static_cast<uint32_t>(dpx) & 1u;

    auto issue = [&](int i, int st) {
      if (i < len) {
        unsigned char* rc = ring_cost + st * Ring::kStageBytes;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          if (uvalid[v]) {
            r3dsimt::cp_async16(rc + 16 * v, c_in + 16 * v);
            if constexpr (MODE == kAccumulate) {
              r3dsimt::cp_async16(ring_sum + st * Ring::kStageBytes + 32 * v, s_in + 16 * v);
              r3dsimt::cp_async16(ring_sum + st * Ring::kStageBytes + 32 * v + 16, s_in + 16 * v + 8);
            }
          }
        }
        r3dsimt::cp_async4(ring_int + st * Ring::kStageBytes,
                           reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(i_iss) & ~uintptr_t{3}));
      }
      r3dsimt::cp_async_commit();
      c_in += dcell;
      if constexpr (MODE == kAccumulate) s_in += dcell;
      i_iss += dpx;
    };
#pragma unroll
    for (int k = 0; k < NS - 1; ++k) issue(k, k);
    uint32_t prev[K];
#pragma unroll
    for (int k = 0; k < K; ++k) prev[k] = 0;
    uint32_t pmin = 0;
    // The next pixel's stage has landed when this pixel is computed, so the
    // P2 of the step into the next pixel is looked up one step ahead, off the
    // step's critical path (iprev is then this pixel's intensity). The first
    // step's P2 is 0, with pmin = 0 the zero clamp of the first pixel.
    uint32_t p2next = 0;
    r3dsimt::cp_async_wait<NS - 2>();  // the first of the NS - 1 stages in flight
    const uint32_t iw0 = *reinterpret_cast<const uint32_t*>(ring_int);
    int iprev = static_cast<int>((iw0 >> (16u * par0)) & 0xFFFFu);

    auto step = [&](const int i, const int q) {
      const bool on = i < len;
      issue(i + NS - 1, (q + NS - 1) % NS);
      const uint32_t hl = r3dsimt::shfl(prev[K - 1], left_lane);
      const uint32_t hr = r3dsimt::shfl(prev[0], right_lane);
      r3dsimt::cp_async_wait<NS - 2>();  // this pixel's stage and the next one's
      const uint32_t iw = *reinterpret_cast<const uint32_t*>(ring_int + ((q + 1) % NS) * Ring::kStageBytes);
      const int inext =
          static_cast<int>((iw >> (16u * ((par0 ^ (static_cast<uint32_t>(i + 1) & dpar)) & 1u))) & 0xFFFFu);
      const uint32_t pen2 = (pmin + p2next) * 0x10001u;
      const uint32_t negmp = pmin * 0xFFFEFFFFu;  // -(pmin in both halves) modulo 2^32
      const int dn = inext - iprev;
      p2next = lut[(dn < 0 ? -dn : dn) >> 8];
      iprev = inext;
      uint32_t cl[K], best[K], c2[K], out[K], tr[K];
#pragma unroll
      for (int k = 0; k < K; ++k) cl[k] = r3dsimt::vmin2(prev[k], pen2);
      best_terms<K>(cl, t > 0 ? r3dsimt::vmin2(hl, pen2) : pen2, t + 1 < G ? r3dsimt::vmin2(hr, pen2) : pen2, one, p1x2,
                    best);
      const unsigned char* sc = ring_cost + q * Ring::kStageBytes;
#pragma unroll
      for (int v = 0; v < NV; ++v)
        unpack_unit(uvalid[v] ? *reinterpret_cast<const uint4*>(sc + 16 * v) : make_uint4(0, 0, 0, 0), c2 + 8 * v);
      // out = L_r = C + T_r with T_r = best - min L(q).
#pragma unroll
      for (int k = 0; k < K; ++k) {
        tr[k] = fma_add(best[k], one, negmp);
        out[k] = fma_add(tr[k], one, c2[k]);
        if (!uvalid[k / 8]) out[k] = kSent2;
      }
      // Minimum over the lane's labels, then over the chain's lanes.
      const uint32_t mm = min_words<K>(out);
      pmin = group_umin<G>(r3dsimt::umin(mm & 0xFFFFu, mm >> 16));
      if (on) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          if (!uvalid[v]) continue;
          const uint32_t* o = out + 8 * v;
          if constexpr (MODE == kTerm) {
            r3dsimt::st_stream(reinterpret_cast<uint4*>(t_out + 16 * v), pack_unit(tr + 8 * v));
          } else {
            uint4 a = make_uint4(o[0], o[1], o[2], o[3]), b = make_uint4(o[4], o[5], o[6], o[7]);
            if constexpr (MODE == kAccumulate) {
              const uint4* ss = reinterpret_cast<const uint4*>(ring_sum + q * Ring::kStageBytes + 32 * v);
              const uint4 x = ss[0], y = ss[1];
              a = make_uint4(add2(x.x, a.x, no_carry), add2(x.y, a.y, no_carry), add2(x.z, a.z, no_carry),
                             add2(x.w, a.w, no_carry));
              b = make_uint4(add2(y.x, b.x, no_carry), add2(y.y, b.y, no_carry), add2(y.z, b.z, no_carry),
                             add2(y.w, b.w, no_carry));
            }
            r3dsimt::st_stream(reinterpret_cast<uint4*>(s_out + 16 * v), a);
            r3dsimt::st_stream(reinterpret_cast<uint4*>(s_out + 16 * v + 8), b);
          }
        }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) prev[k] = out[k];
      if constexpr (MODE == kTerm) t_out += dcell;
      else s_out += dcell;
    };
    for (int i0 = 0; i0 < maxlen; i0 += NS) {
#pragma unroll
      for (int q = 0; q < NS; ++q)
        if (i0 + q < maxlen) step(i0 + q, q);
    }
    r3dsimt::cp_async_wait<0>();
  }
}

// ---------------------------------------------------------------- acceptance
// stereo_matcher.cpp:474-523: validity, the rejection of a minimum on the edge
// of a reduced range (:501-503), the diagonal left-right check (`keys` are the
// row's right-view keys, `shift` their offset), uniqueness, subpixel fit and confidence of one pixel.
struct Winner {
  int best;                    // label of the first minimum
  uint32_t bcost, sec, sm, sp;  // S there, second best, S at best -+ 1
};
R3D_DEVICE void accept_pixel(const SgmMatch& m, const SgmPathJob& job, int x, int y, int lo, int num, const Winner& v,
                             const uint32_t* keys, int shift, float& d, float& cf) {
  const int bx = job.x0 + x, by = job.y0 + y;
  const RowInterval rv = m.pv[by];
  const int jb = v.best - lo;
  const int xr = bx - m.dmin - v.best;
  bool ok = xr >= rv.first && xr <= rv.last;
  if ((jb == 0 && lo > 0) || (jb == num - 1 && lo + num < m.nd)) ok = false;
  if (ok && m.diagonal_lr) {
    const uint32_t key = keys[x - v.best + shift];
    const int rb = key == 0xFFFFFFFFu ? 0xFFFF : static_cast<int>(key & 0xFFFFu) - x + v.best;
    const int diff = rb - v.best;
    if ((diff < 0 ? -diff : diff) > m.lr_max_diff) ok = false;
  }
  const float best_cost = static_cast<float>(v.bcost);
  if (ok && m.uniqueness > 0.0F && v.sec != 0xFFFFu &&
      best_cost > __fmul_rn(__fsub_rn(1.0F, m.uniqueness), static_cast<float>(v.sec)))
    ok = false;
  if (!ok) return;
  float delta = 0.0F;
  if (jb > 0 && jb < num - 1)
    delta = sgm_simd::subpixel_delta(m.subpixel, static_cast<float>(v.sm), best_cost, static_cast<float>(v.sp));
  d = __fadd_rn(static_cast<float>(m.dmin + v.best), delta);
  if (m.confidence)
    cf = (v.sec != 0xFFFFu && v.sec > 0u) ? __fsub_rn(1.0F, __fdiv_rn(best_cost, static_cast<float>(v.sec))) : 0.0F;
}

R3D_DEVICE int4 pack_winner(const Winner& v) {
  return make_int4(static_cast<int>(static_cast<uint32_t>(v.best) | (v.bcost << 16)),
                   static_cast<int>(v.sec | (v.sm << 16)), static_cast<int>(v.sp), 0);
}
R3D_DEVICE Winner unpack_winner(int4 in) {
  return Winner{in.x & 0xFFFF, static_cast<uint32_t>(in.x) >> 16, static_cast<uint32_t>(in.y) & 0xFFFFu,
                static_cast<uint32_t>(in.y) >> 16, static_cast<uint32_t>(in.z)};
}


// ---------------------------------------------------------------- winners
// v[j] for a runtime j in [0, 8): selects on the bits of j (a register array
// cannot be indexed at run time without local memory).
R3D_DEVICE uint32_t pick8(const uint32_t (&v)[8], int j) {
  const bool b0 = (j & 1) != 0, b1 = (j & 2) != 0, b2 = (j & 4) != 0;
  const uint32_t a = b0 ? v[1] : v[0], b = b0 ? v[3] : v[2], c = b0 ? v[5] : v[4], d = b0 ? v[7] : v[6];
  const uint32_t e = b1 ? b : a, f = b1 ? d : c;
  return b2 ? f : e;
}
R3D_DEVICE uint32_t group_min_rt(uint32_t v, int g) {
  for (int o = g >> 1; o > 0; o >>= 1) v = r3dsimt::umin(v, r3dsimt::shfl_xor(v, o));
  return v;
}

// Full range (lo = 0, num = nd): total sums, winner-takes-all
// (sgm_kernels.cpp:332-358: the first minimum, the second best outside +-1, S
// at kb -+ 1) and acceptance of every pixel of a tile row, one warp per row. A
// pixel's labels are spread over g lanes, one unit of 16 each (NU units for
// more than 512 labels), 32 / g pixels at a time; every 32 pixels the lanes
// take one pixel each for the acceptance.
//
// The sums form here and not in an eighth path pass: a pixel's nine byte
// planes are independent of its neighbours', so the reads are wide, coalesced
// and as many as the memory system takes (the path pass kept two pixels of
// eight planes in flight per chain, 4.3 TB/s on a large pair and latency-bound
// on a small one), and all eight directions run as one launch.
//
// The right-view winners of the diagonal check (sgm_kernels.cpp:349-356: the
// smallest S << 16 | x per right column) live in shared memory for the row:
// one shared-memory atomic per cell where the path pass had a global one.
//
// The grid's second dimension cuts a row into parts (one with the diagonal
// check, whose keys need the row in one warp): a 640x480 pair has 1,920 tile
// rows for 3,552 resident warps.
template <bool TERMS, int NU>
R3D_GLOBAL void R3D_LAUNCH_BOUNDS_MIN(kPathThreads, (NU == 1 ? 3 : 2))
    sgm_path_wta_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                        int64_t rows, const uint8_t* R3D_RESTRICT cost, const uint16_t* R3D_RESTRICT sum,
                        const uint8_t* R3D_RESTRICT terms, int64_t tstride, int4* info, int key_words) {
  R3D_DYNAMIC_SMEM(smem);
  const int lane = static_cast<int>(threadIdx.x & 31u), warp = static_cast<int>(threadIdx.x >> 5);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  int4* const winners = reinterpret_cast<int4*>(smem) + warp * 32;
  uint32_t* const keys = reinterpret_cast<uint32_t*>(smem + static_cast<size_t>(wpb) * 512) +
                         static_cast<size_t>(warp) * key_words;
  const int part = static_cast<int>(blockIdx.y), parts = static_cast<int>(gridDim.y);
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * wpb + warp; r < rows; r += nwarps) {
    const int j = find_job(jobs, njobs, r, [](const SgmPathJob& q) { return q.row_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    const int nd = m.nd, w = job.w, nu = nd >> 4;
    const int y = static_cast<int>(r - job.row_off);
    const int64_t row_px = static_cast<int64_t>(y) * w;
    const RowInterval lv = m.bv[job.y0 + y];
    const bool diag = m.diagonal_lr != 0;
    int g = 1;
    while (g < nu && g < 32) g <<= 1;
    const int per = 32 / g, gi = lane / g, t = lane & (g - 1);
    const int64_t cell0 = job.cell_off + row_px * nd;
    // The item's columns, whole groups of 32.
    const int groups = (w + 31) / 32;
    const int xfirst = 32 * (groups * part / parts);
    const int xend = r3dsimt::imin(w, 32 * (groups * (part + 1) / parts));
    if (diag) {
      for (int k = lane; k < w + nd; k += 32) keys[k] = 0xFFFFFFFFu;
      r3dsimt::syncwarp();
    }
    if (y == 0 && xfirst == 0 && lane == 0)
      *job.cells = static_cast<unsigned long long>(w) * static_cast<unsigned long long>(job.h) * nd;
    for (int xb = xfirst; xb < xend; xb += 32) {
      for (int s = 0; s < g && xb + s * per < w; ++s) {
        const int x = xb + s * per + gi;
        const bool inside = x < w && job.x0 + x >= lv.first && job.x0 + x <= lv.last;
        const bool need = inside || (x < w && job.volume != nullptr);
        const int64_t cell = cell0 + static_cast<int64_t>(x) * nd;
        uint32_t wv[NU][8];
        uint32_t kmin = 0xFFFFFFFFu;
#pragma unroll
        for (int n = 0; n < NU; ++n) {
          const int u = t + 32 * n;
          if (need && u < nu) {
            sum_unit<TERMS>(cost + cell, terms + cell, tstride, sum + cell, u, wv[n]);
            const uint32_t e = static_cast<uint32_t>(16 * u);
#pragma unroll
            for (int k = 0; k < 8; ++k)
              kmin = r3dsimt::umin(kmin, r3dsimt::umin((wv[n][k] << 16) | (e + k), (wv[n][k] & 0xFFFF0000u) | (e + k + 8)));
            if (job.volume != nullptr) store_unit(job.volume + (row_px + x) * nd + 16 * u, wv[n]);
          } else {
#pragma unroll
            for (int k = 0; k < 8; ++k) wv[n][k] = 0xFFFFFFFFu;
          }
        }
        kmin = group_min_rt(kmin, g);
        const int kb = static_cast<int>(kmin & 0xFFFFu);
        uint32_t sec2 = 0xFFFFFFFFu;
#pragma unroll
        for (int n = 0; n < NU; ++n) {
          // Bit l: label l of the unit lies within kb -+ 1; its low and high
          // byte in the two halves line up with the halves of word k >> k.
          const int rel = kb - 1 - 16 * (t + 32 * n);
          const uint32_t ex = rel >= 16 || rel < -2 ? 0u : (rel >= 0 ? 7u << rel : 7u >> -rel);
          const uint32_t ex2 = (ex & 0xFFu) | ((ex & 0xFF00u) << 8);
#pragma unroll
          for (int k = 0; k < 8; ++k)
            sec2 = r3dsimt::vmin2(sec2, wv[n][k] | (((ex2 >> k) & 0x00010001u) * 0xFFFFu));
        }
        const uint32_t sec = group_min_rt(r3dsimt::umin(sec2 & 0xFFFFu, sec2 >> 16), g);
        const int km = kb > 0 ? kb - 1 : 0, kp = kb + 1 < nd ? kb + 1 : nd - 1;
        uint32_t vm = pick8(wv[0], km & 7), vp = pick8(wv[0], kp & 7);
        if constexpr (NU > 1) {
          if (km >= 512) vm = pick8(wv[NU - 1], km & 7);
          if (kp >= 512) vp = pick8(wv[NU - 1], kp & 7);
        }
        vm = r3dsimt::shfl(vm, (gi * g + ((km >> 4) & (g - 1))) & 31);
        vp = r3dsimt::shfl(vp, (gi * g + ((kp >> 4) & (g - 1))) & 31);
        const Winner win{kb, kmin >> 16, sec, (km & 8) ? vm >> 16 : vm & 0xFFFFu, (kp & 8) ? vp >> 16 : vp & 0xFFFFu};
        if (t == 0) winners[s * per + gi] = pack_winner(win);
        if (diag && inside) {
#pragma unroll
          for (int n = 0; n < NU; ++n) {
            const int u = t + 32 * n;
            if (u < nu) {
              uint32_t* kr = keys + x + nd - 1 - 16 * u;
#pragma unroll
              for (int k = 0; k < 8; ++k) {
                atomicMin(kr - k, (wv[n][k] << 16) | static_cast<uint32_t>(x));
                atomicMin(kr - k - 8, (wv[n][k] & 0xFFFF0000u) | static_cast<uint32_t>(x));
              }
            }
          }
        }
      }
      r3dsimt::syncwarp();
      const int x = xb + lane;
      if (x < w) {
        const int64_t p = row_px + x;
        if (diag) {
          info[job.px_off + p] = winners[lane];
        } else {
          float d = kInfF, cf = 0.0F;
          if (job.x0 + x >= lv.first && job.x0 + x <= lv.last)
            accept_pixel(m, job, x, y, 0, nd, unpack_winner(winners[lane]), nullptr, 0, d, cf);
          job.disp[p] = d;
          if (job.conf != nullptr) job.conf[p] = cf;
        }
      }
      r3dsimt::syncwarp();
    }
    if (diag) {  // the row's keys are complete
      for (int x = lane; x < w; x += 32) {
        const int64_t p = row_px + x;
        float d = kInfF, cf = 0.0F;
        if (job.x0 + x >= lv.first && job.x0 + x <= lv.last)
          accept_pixel(m, job, x, y, 0, nd, unpack_winner(info[job.px_off + p]), keys, nd - 1, d, cf);
        job.disp[p] = d;
        if (job.conf != nullptr) job.conf[p] = cf;
      }
      r3dsimt::syncwarp();
    }
  }
}

// ================================================================ ranged tiles
// Per-pixel label ranges (lo, num; num a multiple of 16): the same passes on
// costs, terms and sums packed per tile, pixel after pixel, in units of 16
// labels.

// Record of a pixel: x = cell offset / 16 within its tile | min(units, 31)
// << 27 (a tile has fewer than 2^31 labels; 31 stands for 31 or more, looked
// up in the ranges), y = lo | base intensity << 16.
constexpr int kRecShift = 27;
constexpr uint32_t kRecOffset = (1u << kRecShift) - 1u, kRecWide = 31u;

// Units of the pixel at (x, y) of the tile with record r.
R3D_DEVICE int rec_units(const uint2& r, const SgmMatch& m, const SgmPathJob& job, int x, int y) {
  const uint32_t n = r.x >> kRecShift;
  if (n != kRecWide) return static_cast<int>(n);
  return m.rnum[static_cast<int64_t>(job.y0 + y) * m.r_stride + job.x0 + x] >> 4;
}

// Per wave row: the row's label total and its right-WTA shift max(lo + num -
// 1 - x).
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_ranged_rows_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                                int64_t rows, int* R3D_RESTRICT rowsum, int* R3D_RESTRICT rowshift,
                                int* R3D_RESTRICT counters) {
  if (blockIdx.x == 0 && threadIdx.x < kPathCounters) counters[threadIdx.x] = 0;
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < rows; r += nwarps) {
    const int j = find_job(jobs, njobs, r, [](const SgmPathJob& q) { return q.row_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    const int64_t row = static_cast<int64_t>(job.y0 + static_cast<int>(r - job.row_off)) * m.r_stride + job.x0;
    int sum = 0, shift = -0x7FFFFFFF;
    for (int x = lane; x < job.w; x += 32) {
      const int num = m.rnum[row + x];
      sum += num;
      shift = r3dsimt::imax(shift, m.rlo[row + x] + num - 1 - x);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += static_cast<int>(r3dsimt::shfl_xor(static_cast<uint32_t>(sum), o));
      shift = r3dsimt::imax(shift, static_cast<int>(r3dsimt::shfl_xor(static_cast<uint32_t>(shift), o)));
    }
    if (lane == 0) {
      rowsum[r] = sum;
      rowshift[r] = shift;
    }
  }
}

// Per tile: exclusive prefix of the row totals (the cell offset of each row).
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_ranged_rowstart_kernel(const SgmPathJob* R3D_RESTRICT jobs, int njobs, const int* R3D_RESTRICT rowsum,
                                    int* R3D_RESTRICT rowstart) {
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  for (int j = static_cast<int>(blockIdx.x) * wpb + static_cast<int>(threadIdx.x >> 5); j < njobs;
       j += static_cast<int>(gridDim.x) * wpb) {
    const SgmPathJob& job = jobs[j];
    int carry = 0;
    for (int yb = 0; yb < job.h; yb += 32) {
      const int y = yb + lane;
      const int v = y < job.h ? rowsum[job.row_off + y] : 0;
      int incl = v;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int u = static_cast<int>(r3dsimt::shfl(static_cast<uint32_t>(incl), lane >= o ? lane - o : lane));
        if (lane >= o) incl += u;
      }
      if (y < job.h) rowstart[job.row_off + y] = carry + incl - v;
      carry += static_cast<int>(r3dsimt::shfl(static_cast<uint32_t>(incl), 31));
    }
    if (lane == 0) *job.cells = static_cast<unsigned long long>(carry);
  }
}

// Per wave row, one warp: every pixel's record and the u8 costs of its num
// labels, C(p, lo + j) of stereo_matcher.cpp:305-353.
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_ranged_cost_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                                int64_t rows, uint2* R3D_RESTRICT rec, const int* R3D_RESTRICT rowstart,
                                uint8_t* R3D_RESTRICT cost) {
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < rows; r += nwarps) {
    const int j = find_job(jobs, njobs, r, [](const SgmPathJob& q) { return q.row_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    const int y = static_cast<int>(r - job.row_off), by = job.y0 + y, w = job.w;
    const RowInterval lv = m.bv[by], rv = m.pv[by];
    const uint64_t* lrow = m.cbase + static_cast<int64_t>(by) * m.cb_stride;
    const uint64_t* crow = m.cpart + static_cast<int64_t>(by) * m.cp_stride;
    const uint16_t* irow = m.base + static_cast<int64_t>(by) * m.base_stride;
    const uint16_t* lorow = m.rlo + static_cast<int64_t>(by) * m.r_stride;
    const uint16_t* numrow = m.rnum + static_cast<int64_t>(by) * m.r_stride;
    const int safe = rv.first > 0 ? rv.first : 0;
    const uint32_t inv = static_cast<uint32_t>(m.invalid_cost);
    int run = rowstart[r] >> 4;
    // The inputs of the next 32 pixels are loaded while the present ones are
    // worked on.
    int lo_n = 0, nu_n = 0;
    uint32_t iv_n = 0;
    uint64_t cl_n = 0;
    auto load = [&](int x) {
      if (x >= w) return;
      const int bx = job.x0 + x;
      lo_n = lorow[bx];
      nu_n = numrow[bx] >> 4;
      iv_n = irow[bx];
      cl_n = lrow[bx];
    };
    load(lane);
    for (int xb = 0; xb < w; xb += 32) {
      const int x = xb + lane, bx = job.x0 + x;
      const int lo = lo_n, nu = x < w ? nu_n : 0;
      const uint32_t iv = iv_n;
      const uint64_t cl = cl_n;
      load(x + 32);
      int incl = nu;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int v = static_cast<int>(r3dsimt::shfl(static_cast<uint32_t>(incl), lane >= o ? lane - o : lane));
        if (lane >= o) incl += v;
      }
      const int off = run + incl - nu;
      run += static_cast<int>(r3dsimt::shfl(static_cast<uint32_t>(incl), 31));
      if (x < w)
        rec[job.px_off + static_cast<int64_t>(y) * w + x] =
            make_uint2(static_cast<uint32_t>(off) | (r3dsimt::umin(static_cast<uint32_t>(nu), kRecWide) << kRecShift),
                       static_cast<uint32_t>(lo) | (iv << 16));
      const bool inside = x < w && bx >= lv.first && bx <= lv.last;
      uint8_t* out = cost + job.cell_off + static_cast<int64_t>(off) * 16;
      for (int u = 0; u < nu; ++u) {
        uint32_t q[4] = {0, 0, 0, 0};
        const int xr0 = bx - m.dmin - lo - 16 * u;  // right column of the unit's label 0
        if (inside && xr0 <= rv.last && xr0 - 15 >= rv.first) {
          // Every label reads a valid right column: the two popcounts of each
          // Census XOR packed separately (each byte at most 32, no carries).
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            uint32_t a = 0, b = 0;
#pragma unroll
            for (int i = 3; i >= 0; --i) {
              const uint64_t d = cl ^ crow[xr0 - unit_label(k, i)];
              a = a * 256u + static_cast<uint32_t>(r3dsimt::popc(static_cast<uint32_t>(d)));
              b = b * 256u + static_cast<uint32_t>(r3dsimt::popc(static_cast<uint32_t>(d >> 32)));
            }
            q[k] = a + b;
          }
        } else if (inside) {
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const int xr = xr0 - k;
            const bool ok = xr >= rv.first && xr <= rv.last;
            const uint64_t cr = crow[ok ? xr : safe];
            const uint32_t v = ok ? static_cast<uint32_t>(r3dsimt::popc64(cl ^ cr)) : inv;
            q[(k & 7) >> 1] |= v << (8 * ((k & 1) + 2 * (k >> 3)));
          }
        }
        *reinterpret_cast<uint4*>(out + 16 * u) = make_uint4(q[0], q[1], q[2], q[3]);
      }
    }
  }
}

// Passes over ranged tiles: one lane walks one chain, 32 chains per warp, pixel
// by pixel in step. A pixel's labels are taken CH = 2 K at a time (chunks of
// K / 8 units): one chunk for most pixels, more for wider ones.
//
// The predecessor vector stays in registers as long as every lane's next
// pixel has exactly CH labels in the same range as its last one (70 to 89 % of
// the steps of smooth disparities): such a step is the plain recurrence on K
// words, with no realignment, no shuffle and no shared-memory vector. When the
// warp's next step is not of that kind, the lanes write their vectors in
// label order into their own buffers (up to kVecLabels labels in shared
// memory, wider ones in global memory that the L1 holds), and the step reads
// its predecessor labels at its range's shift there, sentinels around them.
// Everything is private to a lane: no barrier, no warp-wide minimum. A step
// takes about 250 instructions of 32 pixels (K = 8), 370 (K = 16), a quarter
// of the steps realigned; issue and shared-memory latency bound it (level 0 of
// a 3072x2048 pair, K = 16: 0.61 of the issue slots, DRAM at a third of the copy
// rate).
//
// One lane per chain against the lane group of the full-range passes: most
// ranges are one or two units, so a group would idle on the narrow pixels and
// pay shuffles for every minimum and neighbour. One warp per CTA: the shared
// memory of an SM is split as finely as the ring allows.
constexpr int kRangedThreads = 32;

// Per warp: the ring of D pixels' first chunks (16-byte pieces, [piece][lane]),
// pixel records, two predecessor buffers per lane (odd stride in words: the
// same word of all lanes lies in distinct banks) and the match's P2 table.
template <int K, int MODE>
struct RangedRing {
  static constexpr int CH = 2 * K;    // labels per chunk
  static constexpr int UF = K / 8;    // units per chunk
  static constexpr int D = 4;
  static constexpr int NR = 2 * D;    // record slots (a power of two)
  static constexpr int kPieces = UF * (MODE == kAccumulate ? 3 : 1);
  static constexpr int kStageBytes = kPieces * 512;
  static constexpr int kData = D * kStageBytes;
  static constexpr int kRec = NR * 32 * 8;
  static constexpr int kVecLabels = 32;          // labels of a vector in shared memory
  static constexpr int kVecStep = kVecLabels / 2 + 1;  // words of a buffer: a vector and a sentinel after it
  static constexpr int kVecStride = (2 * kVecStep) | 1;
  static constexpr int kVec = 32 * kVecStride * 4;
  static constexpr int kWarpBytes = kData + kRec + kVec + 512;
  static constexpr int kBlockBytes = (kRangedThreads / 32) * kWarpBytes;
};

template <int K, int MODE>
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kRangedThreads)
    sgm_path_ranged_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                           const PassSet ps, const uint2* R3D_RESTRICT rec, const uint8_t* R3D_RESTRICT cost,
                           uint16_t* sum, uint8_t* terms, int64_t tstride, uint32_t* ovf, int ovf_words,
                           const int* cancel) {
  // Modes: kFirst / kAccumulate write or add u16 sums; kTerm writes the
  // pass's byte terms (all eight directions in one launch).
  using R = RangedRing<K, MODE>;
  constexpr int CH = R::CH, UF = R::UF, D = R::D, NR = R::NR, NS = R::kVecLabels;
  R3D_DYNAMIC_SMEM(smem);
  const int lane = static_cast<int>(threadIdx.x & 31u), warp = static_cast<int>(threadIdx.x >> 5);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  unsigned char* const wb = smem + static_cast<size_t>(warp) * R::kWarpBytes;
  unsigned char* const data = wb + lane * 16;
  uint2* const recs = reinterpret_cast<uint2*>(wb + R::kData) + lane;  // slot q at recs[32 q]
  // The lane's buffer b at vec + b * kVecStep: the words of a vector, then one
  // of sentinels. Reads clamp their word index to it as an unsigned number, so
  // that words before the vector come from there too.
  uint32_t* const vec = reinterpret_cast<uint32_t*>(wb + R::kData + R::kRec) + lane * R::kVecStride;
  uint16_t* const lut = reinterpret_cast<uint16_t*>(wb + R::kData + R::kRec + R::kVec);
  // The lane's buffers of wide vectors: word q of buffer b at wide[(b * ovf_words + q) * 32].
  uint32_t* const wide = ovf + (static_cast<int64_t>(blockIdx.x) * wpb + warp) * 2 * ovf_words * 32 + lane;
  int lut_match = -1;
  const uint32_t one = ps.one;
  for (int64_t gblk = static_cast<int64_t>(blockIdx.x) * wpb + warp; gblk < ps.total;
       gblk = next_block(ps, nwarps)) {
    if (cancelled(cancel)) break;
    int j, cls, dx, dy, tslot;
    const int64_t blk = locate_block<32>(jobs, njobs, ps, gblk, j, cls, dx, dy, tslot);
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    if (job.match != lut_match) {  // the same for the whole warp (one chain block)
      r3dsimt::syncwarp();
      for (int k = lane; k < 128; k += 32)
        reinterpret_cast<uint32_t*>(lut)[k] = reinterpret_cast<const uint32_t*>(m.lut)[k];
      r3dsimt::syncwarp();
      lut_match = job.match;
    }
    const int w = job.w;
    const uint32_t p1x2 = static_cast<uint32_t>(m.p1) * 0x10001u;
    const bool no_carry = m.sum_no_carry != 0;
    // The lane's chain: pixel (sx, sy) + i (dx, dy) at step i, t0 <= i < t1.
    // Diagonals run in step by row (a lane waits t0 steps for its chain's first
    // row), so that the 32 lanes are on adjacent pixels of one row; chains that
    // start down the tile's side, each from its own first pixel, would put
    // every lane on a row of its own, 32 cache lines per load.
    int sx, sy, t0 = 0, t1;
    if (cls == 2) {
      const int c = static_cast<int>(blk) * 32 + lane - (job.h - 1);  // column at step 0, along dx
      sx = dx > 0 ? c : w - 1 - c;
      sy = dy > 0 ? 0 : job.h - 1;
      t0 = c < 0 ? -c : 0;
      t1 = c < w ? r3dsimt::imin(job.h, w - c) : 0;
      int first = t1 > t0 ? t0 : job.h;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) first = r3dsimt::imin(first, static_cast<int>(r3dsimt::shfl_xor(static_cast<uint32_t>(first), o)));
      t0 -= first;
      t1 -= first;
      sx += first * dx;
      sy += first * dy;
    } else {
      chain_geometry(cls, dx, dy, w, job.h, blk * 32 + lane, sx, sy, t1);
    }
    int maxlen = t1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) maxlen = r3dsimt::imax(maxlen, static_cast<int>(r3dsimt::shfl_xor(static_cast<uint32_t>(maxlen), o)));
    const uint32_t chain_len = t1 > t0 ? static_cast<uint32_t>(t1 - t0) : 0u;
    auto has = [&](int i) { return static_cast<uint32_t>(i - t0) < chain_len; };
    const uint8_t* const cbase = cost + job.cell_off;
    uint16_t* const sbase = sum + job.cell_off + tslot * tstride;
    uint8_t* const tout = terms + job.cell_off + tslot * tstride;
    const int dpx = dy * w + dx;
    const uint2* rp = rec + job.px_off + static_cast<int64_t>(sy) * w + sx;  // record of the next step to request
    auto units_of = [&](const uint2& r, int i) { return rec_units(r, m, job, sx + i * dx, sy + i * dy); };
    // Chunk of the pixel with `left` units from unit `at` on into ring slot st.
    auto issue_chunk = [&](int st, int at, int left) {
      unsigned char* dst = data + st * R::kStageBytes;
#pragma unroll
      for (int u = 0; u < UF; ++u) {
        if (u == 0 || left > u) {
          const int64_t off = static_cast<int64_t>(at + u) * 16;
          r3dsimt::cp_async16(dst + u * 512, cbase + off);
          if constexpr (MODE == kAccumulate) {
            r3dsimt::cp_async16(dst + (UF + 2 * u) * 512, sbase + off);
            r3dsimt::cp_async16(dst + (UF + 2 * u + 1) * 512, sbase + off + 8);
          }
        }
      }
    };
    // Records read ahead of their use (a step's first decisions and addresses
    // depend on them): this pixel's, the next one's, and that of the pixel
    // whose first chunk is issued in this step.
    uint2 rc = make_uint2(0, 0), rn = rc, ri = rc;
    // Pixel i + D - 1's first chunk into slot st, pixel i + 2 D - 1's record;
    // one group.
    auto issue = [&](int i, int st) {
      if (has(i + D - 1)) issue_chunk(st, static_cast<int>(ri.x & kRecOffset), static_cast<int>(ri.x >> kRecShift));
      if (has(i + 2 * D - 1)) r3dsimt::cp_async8(&recs[((i + 2 * D - 1) & (NR - 1)) * 32], rp);
      rp += dpx;
      r3dsimt::cp_async_commit();
    };
#pragma unroll
    for (int k = 0; k < 2 * D - 1; ++k) {
      if (has(k)) recs[k * 32] = *rp;
      rp += dpx;
    }
#pragma unroll
    for (int k = 0; k < D - 1; ++k) {
      if (has(k)) {
        const uint2 r = recs[k * 32];
        issue_chunk(k, static_cast<int>(r.x & kRecOffset), static_cast<int>(r.x >> kRecShift));
      }
      r3dsimt::cp_async_commit();
    }
    if (has(0)) rc = recs[0];
    rn = rc;
    if (has(1)) rn = recs[32];
    if (has(D - 1)) ri = recs[(D - 1) * 32];
    // The predecessor's range, its minimum over labels in both halves,
    // negated, and the clamp min L(q) + P2. A zero clamp makes the first
    // pixel's best term 0 whatever the predecessor words hold: T = 0, L = C.
    int lo_q = 0, num_q = 0;
    uint32_t pen2 = 0, negmp = 0;
    uint32_t prev[K];
#pragma unroll
    for (int k = 0; k < K; ++k) prev[k] = 0;
    bool single = static_cast<int>(rc.x >> kRecShift) == UF;  // this pixel is one full chunk
    bool fast = r3dsimt::ballot(has(0) && !single) == 0;
    // From the best terms of a chunk (its bytes in ring slot st, its cells
    // from unit `at` on): T = best - min L(q), L = C + T, and the outputs.
    uint32_t out[K], pm;
    auto finish = [&](const uint32_t (&best)[K], int st, int at, bool on, bool upper) {
      const unsigned char* src = data + st * R::kStageBytes;
      uint32_t c2[K], tr[K];
#pragma unroll
      for (int u = 0; u < UF; ++u) unpack_unit(*reinterpret_cast<const uint4*>(src + u * 512), c2 + 8 * u);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        tr[k] = fma_add(best[k], one, negmp);
        out[k] = fma_add(tr[k], one, c2[k]);
        if (k >= 8 && !upper) out[k] = kSent2;
      }
      pm = r3dsimt::vmin2(pm, min_words<K>(out));
      if (!on) return;
#pragma unroll
      for (int u = 0; u < UF; ++u) {
        if (u > 0 && !upper) continue;
        const int64_t off = static_cast<int64_t>(at + u) * 16;
        const int q = 8 * u;
        if constexpr (MODE == kTerm) {
          r3dsimt::st_stream(reinterpret_cast<uint4*>(tout + off), pack_unit(tr + q));
        } else {
          uint32_t v[8];
#pragma unroll
          for (int k = 0; k < 8; ++k) v[k] = out[q + k];
          if constexpr (MODE == kAccumulate) {
#pragma unroll
            for (int k = 0; k < 8; k += 4) {
              const uint4 t = *reinterpret_cast<const uint4*>(src + (UF + 2 * u + k / 4) * 512);
              v[k] = add2(t.x, v[k], no_carry);
              v[k + 1] = add2(t.y, v[k + 1], no_carry);
              v[k + 2] = add2(t.z, v[k + 2], no_carry);
              v[k + 3] = add2(t.w, v[k + 3], no_carry);
            }
          }
          uint4* dst = reinterpret_cast<uint4*>(sbase + off);
          r3dsimt::st_stream(dst, make_uint4(v[0], v[1], v[2], v[3]));
          r3dsimt::st_stream(dst + 1, make_uint4(v[4], v[5], v[6], v[7]));
        }
      }
    };
    // Chunk c of pixel i (n units) into the lane's buffer of the pixel.
    auto store_vec = [&](int i, int c, int n, bool upper) {
      uint32_t nat[K];
#pragma unroll
      for (int u = 0; u < UF; ++u) {
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          nat[8 * u + k] = r3dsimt::perm(out[8 * u + 2 * k], out[8 * u + 2 * k + 1], 0x5410u);
          nat[8 * u + 4 + k] = r3dsimt::perm(out[8 * u + 2 * k], out[8 * u + 2 * k + 1], 0x7632u);
        }
      }
      const bool last = (c + 1) * UF >= n;
      const int end = 8 * n - c * K;  // word after the vector, from the chunk's first word
      if (16 * n <= NS) {
        uint32_t* v = vec + (i & 1) * R::kVecStep + c * K;
#pragma unroll
        for (int k = 0; k < K; ++k) v[k] = nat[k];
        if (last) v[end] = kSent2;
      } else {
        uint32_t* v = wide + ((i & 1) * ovf_words + c * K) * 32;
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (k < 8 || upper) v[k * 32] = nat[k];
        if (last) v[end * 32] = kSent2;
      }
    };
    // best = min(L(q, d), L(q, d -+ 1) + P1, min L(q) + P2); clamping first
    // leaves one 3-way minimum per word. From the lane's buffer of pixel i -
    // 1, for the labels of chunk c at lo.
    auto best_from_memory = [&](uint32_t (&best)[K], int i, int c, int lo) {
      // Predecessor labels b - 1 .. b + CH (its own indexing).
      const int b = c * CH + lo - lo_q;
      // pr[k]: labels b - 1 + 2 k, b + 2 k, from the words holding them.
      const int f = (b - 1) >> 1;
      const uint32_t par = 16u * (static_cast<uint32_t>(b - 1) & 1u);
      const uint32_t end = static_cast<uint32_t>(num_q >> 1);
      uint32_t wd[K + 2], pr[K + 1];
      if (num_q <= NS) {
        const uint32_t* vq = vec + ((i & 1) ^ 1) * R::kVecStep;
#pragma unroll
        for (int k = 0; k < K + 2; ++k) wd[k] = vq[r3dsimt::umin(static_cast<uint32_t>(f + k), end)];
      } else {
        const uint32_t* oq = wide + ((i & 1) ^ 1) * ovf_words * 32;
#pragma unroll
        for (int k = 0; k < K + 2; ++k) wd[k] = oq[r3dsimt::umin(static_cast<uint32_t>(f + k), end) * 32];
      }
#pragma unroll
      for (int k = 0; k < K + 1; ++k) pr[k] = r3dsimt::funnel_r(wd[k], wd[k + 1], par);
#pragma unroll
      for (int u = 0; u < UF; ++u) {
        uint32_t cl[10], s[10];
#pragma unroll
        for (int k = 0; k < 10; ++k) {
          cl[k] = r3dsimt::vmin2(
              r3dsimt::perm(pr[8 * u + (k >> 1)], pr[8 * u + (k >> 1) + 4], (k & 1) ? 0x7632u : 0x5410u), pen2);
          s[k] = fma_add(cl[k], one, p1x2);
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) best[8 * u + k] = r3dsimt::vmin3(cl[k + 1], s[k], s[k + 2]);
      }
    };
    for (int i = 0; i < maxlen; ++i) {
      const int st = i & (D - 1), st_in = (i + D - 1) & (D - 1);  // slots of this pixel and of the one issued now
      const bool on = has(i), on_n = has(i + 1);
      const int at = static_cast<int>(rc.x & kRecOffset);
      const int lo = static_cast<int>(rc.y & 0xFFFFu);
      const bool single_n = static_cast<int>(rn.x >> kRecShift) == UF;
      const bool okn = !on_n || (single_n && (!on || (single && ((rn.y ^ rc.y) & 0xFFFFu) == 0)));
      const bool fast_next = r3dsimt::ballot(!okn) == 0;
      const int dn = static_cast<int>(rn.y >> 16) - static_cast<int>(rc.y >> 16);
      const uint32_t p2 = lut[(dn < 0 ? -dn : dn) >> 8];  // of the step into the next pixel
      pm = kSent2;
      uint32_t best[K];
      int n = UF;
      uint2 rn2 = rn, ri2 = ri;
      // The records of the next step; they landed with the group just waited
      // for (requested D - 1 steps ago or before).
      auto look_ahead = [&]() {
        if (has(i + 2)) rn2 = recs[((i + 2) & (NR - 1)) * 32];
        if (has(i + D)) ri2 = recs[((i + D) & (NR - 1)) * 32];
      };
      if (fast) {
        issue(i, st_in);
        r3dsimt::cp_async_wait<D - 1>();
        look_ahead();
        uint32_t cl[K];
#pragma unroll
        for (int k = 0; k < K; ++k) cl[k] = r3dsimt::vmin2(prev[k], pen2);
        best_terms<K>(cl, pen2, pen2, one, p1x2, best);
        finish(best, st, at, on, true);
        if (!fast_next && on) store_vec(i, 0, n, true);
      } else {
        n = on ? units_of(rc, i) : 1;
        const bool multi = r3dsimt::ballot(n > UF) != 0;
        if (!multi) {
          issue(i, st_in);
          r3dsimt::cp_async_wait<D - 1>();
          look_ahead();
          best_from_memory(best, i, 0, lo);
          finish(best, st, at, on, n > 1);
          if (!fast_next && on) store_vec(i, 0, n, n > 1);
        } else {
          // A lane's pixel has more chunks: they pass through this pixel's
          // slot and the free one, each requested while the one before it
          // is worked on; the next pixel is issued after them.
          int sa = st, sb = st_in;
          if (n > UF) issue_chunk(sb, at + UF, n - UF);
          r3dsimt::cp_async_commit();
          r3dsimt::cp_async_wait<D - 1>();
          look_ahead();
          for (int c = 0; r3dsimt::ballot(c * UF < n) != 0; ++c) {
            const bool have = c * UF < n, upper = n - c * UF > 1;
            if (have) {
              best_from_memory(best, i, c, lo);
              finish(best, sa, at + c * UF, on, upper);
              if (on) store_vec(i, c, n, upper);
            }
            // Slot sa is free: the chunk after the one in slot sb.
            if ((c + 2) * UF < n) issue_chunk(sa, at + (c + 2) * UF, n - (c + 2) * UF);
            r3dsimt::cp_async_commit();
            r3dsimt::cp_async_wait<1>();
            const int t = sa;
            sa = sb;
            sb = t;
          }
          issue(i, st_in);
        }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) prev[k] = out[k];
      {
        const uint32_t mp = r3dsimt::vmin2(pm, r3dsimt::perm(pm, pm, 0x1032u));
        // A chain that starts at the next step keeps the zero clamp.
        pen2 = on ? mp + p2 * 0x10001u : 0u;
        negmp = on ? 0u - mp : 0u;
      }
      lo_q = lo;
      num_q = 16 * n;
      rc = rn;
      rn = rn2;
      ri = ri2;
      single = single_n;
      fast = fast_next;
    }
    r3dsimt::cp_async_wait<0>();
  }
}

// Per pixel: the total sums (S = 8 C + the eight byte terms with TERMS, the
// stored u16 sums without), winner-takes-all (sgm_kernels.cpp:332-358; first
// minimum, second best outside +-1, S at kb -+ 1 within the range) and, without the diagonal check, the acceptance rules; with it the right-view
// keys and the pixel's record for the acceptance kernel. Also the optional
// volume copy. Summing here instead of in the eighth path pass keeps that pass
// as short as the others (in one launch with them: the chains of one direction
// alone leave most of the SMs idle on a single pair) and saves the stored sum:
// 11 bytes per cell against 12.
//
// One warp per tile row, a lane per pixel, the next 32 records loaded while the
// present pixels are worked on (a search for the tile and a record per pixel
// before its planes are known left the loads waiting on each other). The first
// two units of a pixel stay in registers.
template <bool TERMS>
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_ranged_wta_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                               int64_t rows, const uint2* R3D_RESTRICT rec, const uint8_t* R3D_RESTRICT cost,
                               const uint16_t* R3D_RESTRICT sum, const uint8_t* R3D_RESTRICT terms, int64_t tstride,
                               const int* R3D_RESTRICT rowshift, int4* R3D_RESTRICT info, uint32_t* rkeys) {
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  for (int64_t r = static_cast<int64_t>(blockIdx.x) * wpb + (threadIdx.x >> 5); r < rows; r += nwarps) {
    const int j = find_job(jobs, njobs, r, [](const SgmPathJob& q) { return q.row_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    const int w = job.w, y = static_cast<int>(r - job.row_off);
    const int64_t row_px = static_cast<int64_t>(y) * w;
    const RowInterval lv = m.bv[job.y0 + y];
    uint2 rn = make_uint2(0, 0);
    if (lane < w) rn = rec[job.px_off + row_px + lane];
    for (int x = lane; x < w; x += 32) {
      const uint2 rc = rn;
      if (x + 32 < w) rn = rec[job.px_off + row_px + x + 32];
      const int64_t p = row_px + x;
      const bool inside = job.x0 + x >= lv.first && job.x0 + x <= lv.last;
      if (!inside && job.volume == nullptr) {
        job.disp[p] = kInfF;
        if (job.conf != nullptr) job.conf[p] = 0.0F;
        continue;
      }
      const int lo = static_cast<int>(rc.y & 0xFFFFu), nu = rec_units(rc, m, job, x, y), num = 16 * nu;
      const int64_t off = static_cast<int64_t>(rc.x & kRecOffset) * 16;
      const uint8_t* cp = cost + job.cell_off + off;
      const uint8_t* tp = terms + job.cell_off + off;
      const uint16_t* sp = sum + job.cell_off + off;
      uint32_t w0[8], w1[8], wx[8];
      sum_unit<TERMS>(cp, tp, tstride, sp, 0, w0);
      if (nu > 1) sum_unit<TERMS>(cp, tp, tstride, sp, 1, w1);
      uint32_t kmin = 0xFFFFFFFFu;
      auto least = [&](int u, const uint32_t (&wv)[8]) {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const uint32_t e = static_cast<uint32_t>(16 * u + k);
          kmin = r3dsimt::umin(kmin, r3dsimt::umin((wv[k] << 16) | e, (wv[k] & 0xFFFF0000u) | (e + 8)));
        }
        if (job.volume != nullptr) store_unit(job.volume + off + 16 * u, wv);
      };
      least(0, w0);
      if (nu > 1) least(1, w1);
      for (int u = 2; u < nu; ++u) {
        sum_unit<TERMS>(cp, tp, tstride, sp, u, wx);
        least(u, wx);
      }
      const int kb = static_cast<int>(kmin & 0xFFFFu);
      const int km = kb > 0 ? kb - 1 : 0;
      const int kp = kb + 1 < num ? kb + 1 : num - 1;
      uint32_t sec2 = 0xFFFFFFFFu, sm = 0, spv = 0;
      auto second = [&](int u, const uint32_t (&wv)[8]) {
        // Bit l: label l of the unit lies within kb -+ 1; its low and high
        // byte in the two halves line up with the halves of word k >> k.
        const int rel = kb - 1 - 16 * u;
        const uint32_t ex = rel >= 16 || rel < -2 ? 0u : (rel >= 0 ? 7u << rel : 7u >> -rel);
        const uint32_t ex2 = (ex & 0xFFu) | ((ex & 0xFF00u) << 8);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          sec2 = r3dsimt::vmin2(sec2, wv[k] | (((ex2 >> k) & 0x00010001u) * 0xFFFFu));
        if ((km >> 4) == u) {
          const uint32_t v = pick8(wv, km & 7);
          sm = (km & 8) ? v >> 16 : v & 0xFFFFu;
        }
        if ((kp >> 4) == u) {
          const uint32_t v = pick8(wv, kp & 7);
          spv = (kp & 8) ? v >> 16 : v & 0xFFFFu;
        }
      };
      second(0, w0);
      if (nu > 1) second(1, w1);
      for (int u = 2; u < nu; ++u) {
        sum_unit<TERMS>(cp, tp, tstride, sp, u, wx);
        second(u, wx);
      }
      const Winner win{lo + kb, kmin >> 16, r3dsimt::umin(sec2 & 0xFFFFu, sec2 >> 16), sm, spv};
      if (m.diagonal_lr) {
        info[job.px_off + p] = pack_winner(win);
        if (inside) {
          uint32_t* keys = rkeys + job.rk_off + static_cast<int64_t>(y) * (w + m.nd);
          const int base = x - lo + rowshift[r];
          auto post = [&](int u, const uint32_t (&wv)[8]) {
#pragma unroll
            for (int k = 0; k < 8; ++k) {
              const int e = 16 * u + k;
              atomicMin(keys + (base - e), (wv[k] << 16) | static_cast<uint32_t>(x));
              atomicMin(keys + (base - e - 8), (wv[k] & 0xFFFF0000u) | static_cast<uint32_t>(x));
            }
          };
          post(0, w0);
          if (nu > 1) post(1, w1);
          for (int u = 2; u < nu; ++u) {
            sum_unit<TERMS>(cp, tp, tstride, sp, u, wx);
            post(u, wx);
          }
        }
        continue;
      }
      float d = kInfF, cf = 0.0F;
      if (inside) accept_pixel(m, job, x, y, lo, num, win, nullptr, 0, d, cf);
      job.disp[p] = d;
      if (job.conf != nullptr) job.conf[p] = cf;
    }
  }
}

// Acceptance of the pixels of matches with the diagonal check (their keys
// are complete after the kernel above).
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_ranged_accept_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs,
                                  int njobs, int64_t pixels, const uint2* R3D_RESTRICT rec,
                                  const int4* R3D_RESTRICT info, const uint32_t* R3D_RESTRICT rkeys,
                                  const int* R3D_RESTRICT rowshift) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < pixels; i += stride) {
    const int j = find_job(jobs, njobs, i, [](const SgmPathJob& q) { return q.px_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    if (!m.diagonal_lr) continue;
    const int p = static_cast<int>(i - job.px_off);
    const int y = p / job.w, x = p - y * job.w;
    const RowInterval lv = m.bv[job.y0 + y];
    float d = kInfF, cf = 0.0F;
    if (job.x0 + x >= lv.first && job.x0 + x <= lv.last) {
      const uint2 rc = rec[i];
      accept_pixel(m, job, x, y, static_cast<int>(rc.y & 0xFFFFu), 16 * rec_units(rc, m, job, x, y),
                   unpack_winner(info[i]), rkeys + job.rk_off + static_cast<int64_t>(y) * (job.w + m.nd),
                   rowshift[job.row_off + y], d, cf);
    }
    job.disp[p] = d;
    if (job.conf != nullptr) job.conf[p] = cf;
  }
}

// ---------------------------------------------------------------- launches
// The path directions; the long chains (rows, columns) before the diagonals, so
// that a tile, and a launch, ends on short blocks.
struct Pass {
  int cls, dx, dy;
};
constexpr Pass kPasses[kMaxPasses] = {{0, 1, 0}, {0, -1, 0}, {1, 0, 1},   {1, 0, -1},
                                      {2, 1, 1}, {2, -1, 1}, {2, -1, -1}, {2, 1, -1}};
constexpr int kAllPasses[kMaxPasses] = {0, 1, 2, 3, 4, 5, 6, 7};

template <class Kernel>
int resident_grid(Kernel kernel, int sms, int64_t work_items, int per_block, size_t smem = 0,
                  int threads = kPathThreads) {
  int per_sm = 1;
  R3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  const int64_t need = (work_items + per_block - 1) / per_block;
  const int64_t resident = static_cast<int64_t>(sms) * (per_sm > 0 ? per_sm : 1);
  return static_cast<int>(need < resident ? (need > 0 ? need : 1) : resident);
}

// Algorithmic HBM bytes of one pass over a segment's cells: costs read; terms
// written; sums read (not by the first pass) and written.
uint64_t pass_bytes(int mode, const SgmPathSegment& g) {
  const uint64_t c = static_cast<uint64_t>(g.cells);
  return (mode == kTerm ? 2 : (mode == kFirst ? 3 : 5)) * c;
}

template <int G, int K, int MODE, bool FULL = false>
void launch_pass(const PassSet& ps, const SgmMatch* dm, const SgmPathJob* jobs, int njobs, const uint8_t* cost,
                 uint16_t* sum, uint8_t* terms, int64_t tstride, const uint16_t* ints, int sms, cudaStream_t s,
                 const SgmPathSegment& seg, const int* cancel) {
  const cudaEvent_t ev0 = profile_on() ? profile_mark(s) : nullptr;
  auto* k = sgm_path_kernel<G, K, MODE, FULL>;
  constexpr size_t smem = PathRing<G, K, MODE>::kBlockBytes;
  static thread_local int configured[64] = {};
  int dev = 0;
  R3D_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    R3D_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    configured[dev] = 1;
  }
  const int64_t nb = ps.total;
  constexpr int threads = PathRing<G, K, MODE>::kThreads;
  R3D_LAUNCH(k, dim3(resident_grid(k, sms, nb, threads / 32, smem, threads)), dim3(threads), smem, s, dm, jobs, njobs,
             ps, cost, sum, terms, tstride, ints, cancel);
  launched("sgm_path_kernel");
  if (ev0 != nullptr) {
    char shape[32];
    std::snprintf(shape, sizeof(shape), "%dx%d/mode%d", G, K, MODE);
    const uint64_t n = static_cast<uint64_t>(ps.n);
    profile_pass(ev0, profile_mark(s), "sgm_path_kernel", shape, n * static_cast<uint64_t>(seg.cells),
                 n * static_cast<uint64_t>(seg.pixels), n * pass_bytes(MODE, seg));
  }
}

// Passes q of kPasses in `qs` (count n) as one PassSet with the block counter `next`.
PassSet pass_set(const SgmPathSegment& g, const int* qs, int n, int* next) {
  PassSet ps{};
  ps.one = 1;
  ps.n = n;
  ps.next = next;
  for (int i = 0; i < n; ++i) {
    const Pass& p = kPasses[qs[i]];
    ps.cls[i] = p.cls;
    ps.dx[i] = p.dx;
    ps.dy[i] = p.dy;
    ps.slot[i] = i;
    ++ps.per_class[p.cls];
    ps.total += g.blocks[p.cls];
  }
  return ps;
}

template <int G, int K>
void launch_passes(const SgmMatch* dm, const SgmPathJob* jobs, const SgmPathSegment& g, const uint8_t* cost,
                   uint16_t* sum, uint8_t* terms, int64_t tstride, const uint16_t* ints, int sms, cudaStream_t s,
                   const int* cancel, int* counters) {
  for (int q = 0; q < kMaxPasses; ++q)
    if (g.blocks[kPasses[q].cls] <= 0) return;  // no pixels: every class has chains otherwise
  if (terms != nullptr) {
    // The eight term passes in one launch (they only read the costs and each
    // writes its own term array). Segments whose matches fill every unit take
    // the kernel without the per-unit validity selects.
    const PassSet ps = pass_set(g, kAllPasses, kTermArrays, counters);
    if (g.full != 0)
      launch_pass<G, K, kTerm, true>(ps, dm, jobs, g.count, cost, sum, terms, tstride, ints, sms, s, g, cancel);
    else
      launch_pass<G, K, kTerm>(ps, dm, jobs, g.count, cost, sum, terms, tstride, ints, sms, s, g, cancel);
    return;
  }
  // Two directions at a time, each into its own volume, or one.
  const int per = tstride != 0 ? 2 : 1;
  for (int q = 0; q < kMaxPasses; q += per) {
    const PassSet ps = pass_set(g, kAllPasses + q, per, counters + q);
    if (q == 0)
      launch_pass<G, K, kFirst>(ps, dm, jobs, g.count, cost, sum, terms, tstride, ints, sms, s, g, cancel);
    else
      launch_pass<G, K, kAccumulate>(ps, dm, jobs, g.count, cost, sum, terms, tstride, ints, sms, s, g, cancel);
  }
}

// Shapes compiled into the library (lanes per chain G, label pairs per lane K).
#define R3D_PATH_SHAPES(X) \
  X(1, 8)                  \
  X(2, 8)                  \
  X(4, 8)                  \
  X(8, 8)                  \
  X(16, 8)                 \
  X(32, 8)                 \
  X(2, 16)                 \
  X(4, 16)                 \
  X(8, 16)                 \
  X(16, 16)                \
  X(32, 16)

}  // namespace

bool sgm_path_enabled() {
  const char* e = std::getenv("R3DGPU_FULL_KERNEL");
  return !(e != nullptr && std::strcmp(e, "wavefront") == 0);
}

namespace {
bool path_shape_compiled(int g, int k) {
  bool found = false;
#define R3D_SHAPE(gg, kk) found = found || (g == gg && k == kk);
  R3D_PATH_SHAPES(R3D_SHAPE)
#undef R3D_SHAPE
  return found;
}
}  // namespace

SgmPathShape sgm_path_shape(int nd, bool terms) {
  // A compiled shape from R3DGPU_PATH_SHAPE ("G,K": any label count it
  // covers) or the tuning table (an entry for exactly this label count), else
  // with the fewest lanes of 8 label pairs per lane (up to 64 labels, and
  // u16 sums up to 512) or of 16.
  // Byte terms, whole pair, 2048x1536 (1536x1152 for 384 labels): 64 labels
  // 3.57 ms with 8 pairs per lane, 3.65 with 16; 96: 5.54 and 5.38; 128: 5.85
  // and 5.76; 256: 11.35 and 10.21; 384: 13.01 and 10.89. 24 pairs per lane,
  // which fit 48, 96, 192 and 384 labels without idle lanes, took 3.84, 5.78,
  // 10.2 and 11.4 (longer steps, fewer chains in flight).
  // u16 sums run two directions at a time, so chains in flight count for more.
  // 1024x768 pair, P2 = 600, 8 and 16 pairs per lane: 64 labels 1.44 and 1.74
  // ms; 96: 1.96 and 2.58; 128: 2.33 and 2.67; 256: 4.13 and 4.47; 384: 6.34
  // and 6.72; 512: 7.65 and 8.34. 2048x1536, 128 labels: 8.40 and 9.02.
  if (const char* e = std::getenv("R3DGPU_PATH_SHAPE")) {
    int g = 0, k = 0;
    if (std::sscanf(e, "%d,%d", &g, &k) == 2 && path_shape_compiled(g, k) && 2 * g * k >= nd) return {g, k};
  }
  const auto it = tuning().path.find(nd);
  if (it != tuning().path.end() && path_shape_compiled(it->second.g, it->second.k) &&
      2 * it->second.g * it->second.k >= nd)
    return {it->second.g, it->second.k};
  const int k_want = nd <= (terms ? 64 : 512) ? 8 : 16;
  SgmPathShape best{0, 0};
  int best_nd = 1 << 30;
#define R3D_SHAPE(g, k)                                              \
  if (k == k_want && 2 * g * k >= nd && 2 * g * k < best_nd) { \
    best = SgmPathShape{g, k};                                       \
    best_nd = 2 * g * k;                                             \
  }
  if (nd <= kPathMaxLabels) {
    R3D_PATH_SHAPES(R3D_SHAPE)
  }
#undef R3D_SHAPE
  return best;
}

namespace {
// The arrays of the mode: their size, and b.stride.
size_t path_arrays(SgmPathBuffers& b, int64_t cells, SgmPathMode mode) {
  const int arrays = mode == kPathTerms ? kTermArrays : (mode == kPathTwoSums ? 2 : 1);
  const size_t value = mode == kPathTerms ? 1 : 2;
  const size_t bytes = align256(static_cast<size_t>(cells) * value);
  b.stride = static_cast<int64_t>(bytes / value);
  return static_cast<size_t>(arrays) * bytes;
}
}  // namespace

SgmPathBuffers sgm_path_buffers(int64_t cells, int64_t pixels, int64_t keys, SgmPathMode mode) {
  SgmPathBuffers b{};
  size_t o = 0;
  b.cost = o;
  o += align256(static_cast<size_t>(cells));
  b.paths = o;
  o += path_arrays(b, cells, mode);
  // Winners of a tile row until its right-view keys are complete: only for
  // matches with the diagonal check.
  b.info = o;
  if (keys > 0) o += align256(static_cast<size_t>(pixels) * 16);
  // The tiles' base intensities, pixel after pixel, and 16 bytes more: the
  // pass kernels copy the aligned 4-byte word holding a pixel's intensity.
  b.ints = o;
  o += align256(static_cast<size_t>(pixels) * 2 + 16);
  b.counters = o;
  o += align256(sizeof(int) * kPathCounters);
  b.total = o;
  return b;
}

void launch_sgm_path_wave(const SgmMatch* dm, const SgmPathWave& wave, int sms, cudaStream_t s) {
  if (wave.njobs <= 0 || wave.cells <= 0) return;
  const SgmPathBuffers B = sgm_path_buffers(wave.cells, wave.pixels, wave.keys, wave.mode);
  uint8_t* cost = wave.buffer + B.cost;
  uint16_t* sum = reinterpret_cast<uint16_t*>(wave.buffer + B.paths);
  uint8_t* terms = wave.mode == kPathTerms ? wave.buffer + B.paths : nullptr;
  // From one array to the next; 0: one sum volume.
  const int64_t stride = wave.mode == kPathSum ? 0 : B.stride;
  int4* info = reinterpret_cast<int4*>(wave.buffer + B.info);
  uint16_t* ints = reinterpret_cast<uint16_t*>(wave.buffer + B.ints);
  int* counters = reinterpret_cast<int*>(wave.buffer + B.counters);
  if (8 * wave.nsegs > kPathCounters) fail(R3DGPU_EINVAL, "stereo: too many path kernel shapes in a wave");
  {
    constexpr size_t max_smem = static_cast<size_t>(kPathThreads / 32) * kCostStage * 8;
    static thread_local int configured[64] = {};
    int dev = 0;
    R3D_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev]) {
      R3D_CUDA(cudaFuncSetAttribute(sgm_path_cost_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    static_cast<int>(max_smem)));
      configured[dev] = 1;
    }
    const int words = wave.max_span > 0 && wave.max_span <= kCostStage ? (wave.max_span + 1) & ~1 : kCostStage;
    const size_t smem = static_cast<size_t>(kPathThreads / 32) * words * 8;
    R3D_LAUNCH(sgm_path_cost_kernel,
               dim3(resident_grid(sgm_path_cost_kernel, sms, wave.rows, kPathThreads / 32, smem)),
               dim3(kPathThreads), smem, s, dm, wave.jobs, wave.njobs, wave.rows, cost, words, ints, counters);
    launched("sgm_path_cost_kernel");
  }
  for (int q = 0; q < wave.nsegs; ++q) {
    const SgmPathSegment& g = wave.segs[q];
    const SgmPathJob* jobs = wave.jobs + g.first;
    bool done = false;
#define R3D_SHAPE(gg, kk)                                                                                     \
  if (!done && g.shape.g_ == gg && g.shape.k_ == kk) {                                                        \
    launch_passes<gg, kk>(dm, jobs, g, cost, sum, terms, stride, ints, sms, s, wave.cancel,                   \
                          counters + 8 * q);                                                                  \
    done = true;                                                                                              \
  }
    R3D_PATH_SHAPES(R3D_SHAPE)
#undef R3D_SHAPE
    if (!done) fail(R3DGPU_EINVAL, "stereo: bad path kernel shape");
  }
  bool wide = false;  // more than 512 labels: two units per lane
  for (int q = 0; q < wave.nsegs; ++q) wide = wide || 2 * wave.segs[q].shape.g_ * wave.segs[q].shape.k_ > 512;
  auto* wta = terms != nullptr ? (wide ? sgm_path_wta_kernel<true, 2> : sgm_path_wta_kernel<true, 1>)
                               : (wide ? sgm_path_wta_kernel<false, 2> : sgm_path_wta_kernel<false, 1>);
  // A row's right-view keys: tile width + labels, at most kCostStage + 1.
  const int key_words = wave.keys > 0 ? kCostStage + 4 : 0;
  const size_t smem = static_cast<size_t>(kPathThreads / 32) * (512 + 4 * static_cast<size_t>(key_words));
  if (wave.keys > 0)
    R3D_CUDA(cudaFuncSetAttribute(wta, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  // Parts of a row, at most 8, while the rows alone give a resident warp (24 per
  // SM) less than two items (640x480: 0.727 ms a pair with four parts, 0.770
  // with one or two).
  const int64_t resident = static_cast<int64_t>(sms) * 48;
  const int64_t want = wave.keys > 0 || wave.rows <= 0 ? 1 : (resident + wave.rows - 1) / wave.rows;
  const int parts = static_cast<int>(want > 8 ? 8 : want);
  R3D_LAUNCH(wta, dim3(resident_grid(wta, sms, wave.rows, kPathThreads / 32, smem), parts), dim3(kPathThreads), smem, s,
             dm, wave.jobs, wave.njobs, wave.rows, cost, sum, terms, stride, info, key_words);
  launched("sgm_path_wta_kernel");
}

// ---------------------------------------------------------------- ranged launches
namespace {

// Resident one-warp CTAs per SM of a ranged pass launch (the overflow has one
// slot per resident warp). Registers and shared memory allow 20 to 25; more
// than 12 are slower on the largest pairs (6048x4032: 30.8 ms with 12, 31.5 with
// 16, 32.3 with 25; 33.5 with 6), smaller pairs do not care.
constexpr int kRangedMaxPerSm = 12;

template <int K, int MODE>
void launch_ranged_pass(const PassSet& ps, const SgmMatch* dm, const SgmPathJob* jobs, int njobs, const uint2* rec,
                        const uint8_t* cost, uint16_t* sum, uint8_t* terms, int64_t tstride, uint32_t* ovf,
                        int ovf_words, int sms, cudaStream_t s, const SgmPathSegment& seg, const int* cancel) {
  const cudaEvent_t ev0 = profile_on() ? profile_mark(s) : nullptr;
  auto* k = sgm_path_ranged_kernel<K, MODE>;
  constexpr size_t smem = RangedRing<K, MODE>::kBlockBytes;
  static thread_local int configured[64] = {};
  int dev = 0;
  R3D_CUDA(cudaGetDevice(&dev));
  if (dev >= 0 && dev < 64 && !configured[dev]) {
    R3D_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
    configured[dev] = 1;
  }
  int grid = resident_grid(k, sms, ps.total, kRangedThreads / 32, smem, kRangedThreads);
  grid = grid < sms * kRangedMaxPerSm ? grid : sms * kRangedMaxPerSm;
  R3D_LAUNCH(k, dim3(grid), dim3(kRangedThreads), smem, s, dm, jobs, njobs, ps, rec, cost, sum, terms, tstride, ovf,
             ovf_words, cancel);
  launched("sgm_path_ranged_kernel");
  if (ev0 != nullptr) {
    char shape[32];
    std::snprintf(shape, sizeof(shape), "1x%d/mode%d", K, MODE);
    // Per pixel and pass also the 8-byte record (range and cell offset).
    const uint64_t n = static_cast<uint64_t>(ps.n);
    profile_pass(ev0, profile_mark(s), "sgm_path_ranged_kernel", shape, n * static_cast<uint64_t>(seg.cells),
                 n * static_cast<uint64_t>(seg.pixels), n * (pass_bytes(MODE, seg) + 8 * static_cast<uint64_t>(seg.pixels)));
  }
}

template <int K>
void launch_ranged_passes(const SgmMatch* dm, const SgmPathJob* jobs, const SgmPathSegment& g, const uint2* rec,
                          const uint8_t* cost, uint16_t* sum, uint8_t* terms, int64_t tstride, uint32_t* ovf,
                          int ovf_words, int sms, cudaStream_t s, const int* cancel, int* counters) {
  for (int q = 0; q < 8; ++q)
    if (g.blocks[kPasses[q].cls] <= 0) return;  // no pixels: every class has chains otherwise
  if (terms != nullptr) {
    // Byte terms: all eight directions in one launch.
    launch_ranged_pass<K, kTerm>(pass_set(g, kAllPasses, kTermArrays, counters), dm, jobs, g.count, rec, cost, sum,
                                 terms, tstride, ovf, ovf_words, sms, s, g, cancel);
    return;
  }
  const int per = tstride != 0 ? 2 : 1;  // directions a launch, as in the full-range passes
  for (int q = 0; q < kMaxPasses; q += per) {
    const PassSet ps = pass_set(g, kAllPasses + q, per, counters + q);
    if (q == 0)
      launch_ranged_pass<K, kFirst>(ps, dm, jobs, g.count, rec, cost, sum, terms, tstride, ovf, ovf_words, sms, s, g,
                                    cancel);
    else
      launch_ranged_pass<K, kAccumulate>(ps, dm, jobs, g.count, rec, cost, sum, terms, tstride, ovf, ovf_words, sms, s,
                                         g, cancel);
  }
}

}  // namespace

bool sgm_path_ranged_enabled() {
  const char* e = std::getenv("R3DGPU_RANGED_KERNEL");
  return e == nullptr || std::strcmp(e, "path") == 0;
}

SgmPathShape sgm_path_ranged_shape(int64_t cells, int64_t pixels) {
  // Items of 32 labels where the pixels average more than one and a half units.
  return cells > 24 * pixels ? SgmPathShape{1, 16} : SgmPathShape{1, 8};
}

SgmPathBuffers sgm_path_ranged_buffers(int64_t cells, int64_t pixels, int64_t keys, int64_t rows, int maxnum,
                                       int sms, SgmPathMode mode) {
  SgmPathBuffers b{};
  size_t o = 0;
  b.cost = o;
  o += align256(static_cast<size_t>(cells));
  b.paths = o;
  o += path_arrays(b, cells, mode);
  // Winners and right-view keys: only for matches with the diagonal check.
  b.info = o;
  if (keys > 0) o += align256(static_cast<size_t>(pixels) * 16);
  b.rkeys = o;
  o += align256(static_cast<size_t>(keys) * 4);
  b.counters = o;
  o += align256(sizeof(int) * kPathCounters);
  b.rec = o;
  o += align256(static_cast<size_t>(pixels) * 8);
  b.rowsum = o;
  o += align256(static_cast<size_t>(rows) * 4);
  b.rowstart = o;
  o += align256(static_cast<size_t>(rows) * 4);
  b.rowshift = o;
  o += align256(static_cast<size_t>(rows) * 4);
  // Words of a wide vector's buffer: the vector and a word of sentinels (none
  // where every vector fits shared memory).
  b.overflow_words = maxnum > RangedRing<8, kTerm>::kVecLabels ? maxnum / 2 + 1 : 0;
  b.overflow = o;
  // One slot (two buffers for each of 32 lanes) per resident warp.
  const int64_t slots = static_cast<int64_t>(sms) * kRangedMaxPerSm * (kRangedThreads / 32);
  o += align256(static_cast<size_t>(slots) * 64 * static_cast<size_t>(b.overflow_words) * 4);
  b.total = o;
  return b;
}

void launch_sgm_path_ranged_wave(const SgmMatch* dm, const SgmPathRangedWave& wave, int sms, cudaStream_t s) {
  if (wave.njobs <= 0 || wave.pixels <= 0) return;
  const SgmPathBuffers B =
      sgm_path_ranged_buffers(wave.cells, wave.pixels, wave.keys, wave.rows, wave.maxnum, sms, wave.mode);
  uint8_t* cost = wave.buffer + B.cost;
  uint16_t* sum = reinterpret_cast<uint16_t*>(wave.buffer + B.paths);
  uint8_t* terms = wave.mode == kPathTerms ? wave.buffer + B.paths : nullptr;
  const int64_t stride = wave.mode == kPathSum ? 0 : B.stride;
  int4* info = reinterpret_cast<int4*>(wave.buffer + B.info);
  uint32_t* rkeys = reinterpret_cast<uint32_t*>(wave.buffer + B.rkeys);
  uint2* rec = reinterpret_cast<uint2*>(wave.buffer + B.rec);
  int* rowsum = reinterpret_cast<int*>(wave.buffer + B.rowsum);
  int* rowstart = reinterpret_cast<int*>(wave.buffer + B.rowstart);
  int* rowshift = reinterpret_cast<int*>(wave.buffer + B.rowshift);
  uint32_t* ovf = reinterpret_cast<uint32_t*>(wave.buffer + B.overflow);
  int* counters = reinterpret_cast<int*>(wave.buffer + B.counters);
  if (wave.keys > 0) R3D_CUDA(cudaMemsetAsync(rkeys, 0xFF, static_cast<size_t>(wave.keys) * 4, s));
  R3D_LAUNCH(sgm_path_ranged_rows_kernel,
             dim3(resident_grid(sgm_path_ranged_rows_kernel, sms, wave.rows, kPathThreads / 32)), dim3(kPathThreads),
             0, s, dm, wave.jobs, wave.njobs, wave.rows, rowsum, rowshift, counters);
  launched("sgm_path_ranged_rows_kernel");
  R3D_LAUNCH(sgm_path_ranged_rowstart_kernel,
             dim3(resident_grid(sgm_path_ranged_rowstart_kernel, sms, wave.njobs, kPathThreads / 32)),
             dim3(kPathThreads), 0, s, wave.jobs, wave.njobs, rowsum, rowstart);
  launched("sgm_path_ranged_rowstart_kernel");
  R3D_LAUNCH(sgm_path_ranged_cost_kernel,
             dim3(resident_grid(sgm_path_ranged_cost_kernel, sms, wave.rows, kPathThreads / 32)), dim3(kPathThreads),
             0, s, dm, wave.jobs, wave.njobs, wave.rows, rec, rowstart, cost);
  launched("sgm_path_ranged_cost_kernel");
  for (int q = 0; q < wave.nsegs; ++q) {
    const SgmPathSegment& g = wave.segs[q];
    const SgmPathJob* jobs = wave.jobs + g.first;
    if (g.shape.k_ == 8)
      launch_ranged_passes<8>(dm, jobs, g, rec, cost, sum, terms, stride, ovf, B.overflow_words, sms, s,
                              wave.cancel, counters + 8 * q);
    else if (g.shape.k_ == 16)
      launch_ranged_passes<16>(dm, jobs, g, rec, cost, sum, terms, stride, ovf, B.overflow_words, sms, s,
                               wave.cancel, counters + 8 * q);
    else
      fail(R3DGPU_EINVAL, "stereo: bad ranged path kernel shape");
  }
  auto* wta = terms != nullptr ? sgm_path_ranged_wta_kernel<true> : sgm_path_ranged_wta_kernel<false>;
  R3D_LAUNCH(wta, dim3(resident_grid(wta, sms, wave.rows, kPathThreads / 32)), dim3(kPathThreads), 0, s, dm, wave.jobs,
             wave.njobs, wave.rows, rec, cost, sum, terms, stride, rowshift, info, rkeys);
  launched("sgm_path_ranged_wta_kernel");
  if (wave.keys > 0) {  // matches with the diagonal left-right check
    R3D_LAUNCH(sgm_path_ranged_accept_kernel,
               dim3(resident_grid(sgm_path_ranged_accept_kernel, sms, wave.pixels, kPathThreads)), dim3(kPathThreads),
               0, s, dm, wave.jobs, wave.njobs, wave.pixels, rec, info, rkeys, rowshift);
    launched("sgm_path_ranged_accept_kernel");
  }
}

}  // namespace r3dgpu
