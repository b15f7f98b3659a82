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
//   8 path passes   one launch per direction (and kernel shape); G lanes walk
//                   one chain, K label pairs per lane, 32 / G chains per warp,
//                   the predecessor vector in registers (its d -+ 1 neighbours
//                   across lanes by shuffle), the next pixel's costs and sums
//                   loaded while the current one is computed. The first pass
//                   writes the sum volume, the next six add to it, the last
//                   adds its path and takes the winner-takes-all records;
//   accept kernel   the acceptance rules, subpixel fit and confidence per
//                   pixel, into the tile's disparity and confidence.
//
// No CTA barrier is on the chain's critical path and every tile spreads over
// as many SMs as it has chains, so one small pair fills the GPU as well as a
// batch does. HBM traffic per aggregated cell: 1 B cost write, 8 x 1 B cost
// reads, 2 B + 6 x 4 B + 2 B sum traffic.
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
                  const uint64_t d = cl ^ stage[base - 4 * w4 - i];
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
                q[k >> 2] |= v << (8 * (k & 3));
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
// Pass modes. With u16 sums (any penalties): the first pass writes the sum
// volume, the next six add to it, the last adds its path and takes the
// winner-takes-all. With byte terms (every P2 <= 255): passes 1..7 write
// their path's term T_r = L_r - C (in [0, P2]) as one byte per cell, and the
// last pass forms S = L_8 + 7 C + sum T_r (at most 8 (255 + 255) < 2^16, so
// the sum modulo 2^16 is the plain sum) and takes the winner-takes-all.
enum PassMode { kFirst = 0, kAccumulate = 1, kLast = 2, kTerm = 3, kLastTerm = 4 };
constexpr int kTermArrays = 7;    // of the full-range passes (the last pass adds its own path)
constexpr int kRangedTerms = 8;   // of the ranged passes (summed per pixel)
constexpr int kMaxPasses = 8;
// The passes of one launch: n directions (slot = its term array), their
// number per chain class, and the chain blocks of all of them together. The
// blocks are numbered tile after tile, within a tile direction after
// direction: the directions of a tile run close together, so that its costs
// are read from DRAM about once and from L2 after that.
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
// FMA pipe executes, in place of an add on the ALU pipe (the pass kernels'
// packed min, byte permutes and adds keep the ALU pipe the busier one).
R3D_DEVICE uint32_t fma_add(uint32_t a, uint32_t one, uint32_t b) { return a * one + b; }

// v[j] for a runtime j in [0, K): a tree of K - 1 selects on the bits of j
// (a register array cannot be indexed at run time without local memory).
template <int N>
R3D_DEVICE void pick_level(uint32_t* t, bool hi) {
#pragma unroll
  for (int k = 0; 2 * k < N; ++k) t[k] = (2 * k + 1 < N && hi) ? t[2 * k + 1] : t[2 * k];
}
template <int K>
R3D_DEVICE uint32_t pick(const uint32_t (&v)[K], int j) {
  static_assert(K >= 2 && K <= 16, "pick: 2..16 words");
  constexpr int n1 = (K + 1) / 2, n2 = (n1 + 1) / 2, n3 = (n2 + 1) / 2;
  uint32_t t[K];
#pragma unroll
  for (int k = 0; k < K; ++k) t[k] = v[k];
  pick_level<K>(t, (j & 1) != 0);
  if constexpr (n1 > 1) pick_level<n1>(t, (j & 2) != 0);
  if constexpr (n2 > 1) pick_level<n2>(t, (j & 4) != 0);
  if constexpr (n3 > 1) pick_level<n3>(t, (j & 8) != 0);
  return t[0];
}

// Per-warp shared-memory ring of the pass kernels: Stages stages, each with
// one pixel per chain of the bytes the pass reads (Planes bytes per label:
// the cost, plus the u16 sum or the seven byte terms).
// The term passes read one byte per label and keep 8 stages in flight (their
// step is short, so 3 stages ahead left them waiting on DRAM).
// The last pass with byte terms stages eight byte planes per pixel: two
// stages (its step is long, one pixel ahead covers the DRAM latency).
template <int MODE>
struct PathMode {
  static constexpr int kPlanes = MODE == kAccumulate || MODE == kLast ? 3 : (MODE == kLastTerm ? 1 + kTermArrays : 1);
  static constexpr int kStages = MODE == kLastTerm ? 2 : (MODE == kTerm ? 8 : 4);
};
// A stage ends with one 4-byte word per lane: the aligned word of the
// intensities that holds its chain's pixel (every lane copies its own, since
// a cp.async wait covers only the waiting thread's copies).
// CTA size and resident CTAs per SM: 4-warp CTAs for the byte-term last
// pass (its eight-plane ring) and the 16-word term passes (92 registers),
// so that CTAs pack an SM's registers and shared memory finely (the 12-word
// term passes measured 12-19 % slower that way than in two 8-warp CTAs).
template <int G, int K, int MODE>
struct PathRing {
  static constexpr int kThreads = (MODE == kLastTerm || (MODE == kTerm && K >= 16)) ? 128 : kPathThreads;
  static constexpr int kMinBlocks = MODE == kLastTerm ? (K <= 8 ? 6 : 3)
                                    : MODE == kTerm   ? (K <= 8 ? 4 : (K >= 16 ? 5 : 2))
                                                      : (K <= 8 ? 3 : 2);
  static constexpr int ND = 2 * G * K;
  static constexpr int kStages = PathMode<MODE>::kStages;
  static constexpr int kPlaneBytes = (32 / G) * PathMode<MODE>::kPlanes * ND;
  static constexpr int kIntBytes = 32 * 4;
  static constexpr int kStageBytes = kPlaneBytes + kIntBytes;
  static constexpr int kWarpBytes = kStages * kStageBytes;
  // Each warp's rings, then each warp's copy of its match's P2 table.
  static constexpr int kBlockBytes = (kThreads / 32) * (kWarpBytes + 512);
};

// CTAs per SM (PathRing): four 8-warp CTAs for the 8-word term passes (64
// registers, no spills), two for the 12-word ones, five 4-warp CTAs for the
// 16-word ones; six or three 4-warp CTAs for the byte-term last pass; three
// or two 8-warp CTAs for the u16-sum passes.
//
// The step loop is unrolled by the ring depth NS so that ring slots and the
// intensity queue are indexed statically; each chain keeps running pointers
// (advanced by one pixel along the path per step) instead of recomputing
// addresses. The first pixel needs no special case: with a zero predecessor
// vector and a zero minimum, best = 0, so T = 0 and L = C there.
//
// One launch runs the passes of a PassSet: a single pass, or the seven term
// passes of a segment at once (they only read the costs and each writes its
// own term array, so their chain blocks can be taken in any order).
template <int G, int K, int MODE, bool FULL>
R3D_GLOBAL void R3D_LAUNCH_BOUNDS_MIN((PathRing<G, K, MODE>::kThreads), (PathRing<G, K, MODE>::kMinBlocks))
    sgm_path_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                    const PassSet ps, const uint8_t* R3D_RESTRICT cost, uint16_t* sum, uint8_t* terms,
                    int64_t tstride, int4* R3D_RESTRICT info, uint32_t* rkeys, const uint16_t* R3D_RESTRICT ints,
                    const int* cancel) {
  constexpr int CPW = 32 / G;  // chains per warp
  constexpr int U = K / 4;     // units of 8 labels per lane
  constexpr int NS = PathRing<G, K, MODE>::kStages;
  constexpr bool kReadsSum = MODE == kAccumulate || MODE == kLast;
  constexpr bool kWta = MODE == kLast || MODE == kLastTerm;
  // K a multiple of 8: a lane's 2 K labels are NV 16-byte aligned pieces of
  // every byte plane (piece v = units 2 v, 2 v + 1, valid together since
  // label counts are multiples of 16).
  constexpr bool kVec = K % 8 == 0;
  constexpr int NV = K / 8;
  R3D_DYNAMIC_SMEM(smem);
  const int lane = static_cast<int>(threadIdx.x & 31u);
  const int gi = lane / G, t = lane % G;
  const int e0 = 2 * t * K;  // first label of the lane
  const int left_lane = (lane + 31) & 31, right_lane = (lane + 1) & 31;
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  using Ring = PathRing<G, K, MODE>;
  unsigned char* const ring = smem + static_cast<size_t>(threadIdx.x >> 5) * Ring::kWarpBytes;
  // The warp's copy of the P2 table of the match it works on (256 u16),
  // reloaded when a chain block belongs to another match.
  uint16_t* const lut = reinterpret_cast<uint16_t*>(smem + static_cast<size_t>(wpb) * Ring::kWarpBytes +
                                                    static_cast<size_t>(threadIdx.x >> 5) * 512);
  int lut_match = -1;
  unsigned char* const ring_cost = ring + gi * Ring::ND + e0;
  unsigned char* const ring_sum = ring + CPW * Ring::ND + gi * 2 * Ring::ND + 2 * e0;
  unsigned char* const ring_term = ring + CPW * Ring::ND + gi * Ring::ND + e0;  // + r * CPW * ND
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
    bool uvalid[U];
#pragma unroll
    for (int u = 0; u < U; ++u) uvalid[u] = FULL || e0 + 8 * u < nd;
    // Running offsets (cells, pixels) of the pixel being issued (NS - 1
    // ahead) and of the pixel being computed.
    const int64_t dcell = (static_cast<int64_t>(dy) * w + dx) * nd;
    const int64_t cell0 = job.cell_off + e0 + (static_cast<int64_t>(sy) * w + sx) * nd;
    const uint8_t* c_in = cost + cell0;
    const uint16_t* s_in = sum + cell0;
    const uint8_t* t_in = terms + cell0;
    uint16_t* s_out = sum + cell0;
    uint8_t* t_out = terms + cell0 + static_cast<int64_t>(tslot) * tstride;
    int64_t px_out = job.px_off + static_cast<int64_t>(sy) * w + sx;
    const int64_t dpx = static_cast<int64_t>(dy) * w + dx;
    // Intensity of the pixel being issued (each lane copies the aligned
    // 4-byte word holding it into the stage), and the parity of the
    // chain's first pixel (which half of a staged word holds the intensity:
    // pixel i's parity is par0 ^ (i & dpar)).
    const uint16_t* i_iss = ints + job.px_off + static_cast<int64_t>(sy) * w + sx;
    const uint32_t par0 = static_cast<uint32_t>(reinterpret_cast<uintptr_t>(i_iss) >> 1) & 1u;
    const uint32_t dpar = static_cast<uint32_t>(dpx) & 1u;
    int x = sx, y = sy;

    auto issue = [&](int i, int st) {
      if (i < len) {
        unsigned char* rc = ring_cost + st * Ring::kStageBytes;
        if constexpr (kVec) {
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            if (uvalid[2 * v]) {
              r3dsimt::cp_async16(rc + 16 * v, c_in + 16 * v);
              if constexpr (kReadsSum) {
                r3dsimt::cp_async16(ring_sum + st * Ring::kStageBytes + 32 * v, s_in + 16 * v);
                r3dsimt::cp_async16(ring_sum + st * Ring::kStageBytes + 32 * v + 16, s_in + 16 * v + 8);
              }
              if constexpr (MODE == kLastTerm) {
#pragma unroll
                for (int r = 0; r < kTermArrays; ++r)
                  r3dsimt::cp_async16(ring_term + st * Ring::kStageBytes + r * CPW * Ring::ND + 16 * v,
                                      t_in + r * tstride + 16 * v);
              }
            }
          }
        } else {
#pragma unroll
          for (int u = 0; u < U; ++u) {
            if (uvalid[u]) {
              r3dsimt::cp_async8(rc + 8 * u, c_in + 8 * u);
              if constexpr (kReadsSum) r3dsimt::cp_async16(ring_sum + st * Ring::kStageBytes + 16 * u, s_in + 8 * u);
              if constexpr (MODE == kLastTerm) {
#pragma unroll
                for (int r = 0; r < kTermArrays; ++r)
                  r3dsimt::cp_async8(ring_term + st * Ring::kStageBytes + r * CPW * Ring::ND + 8 * u,
                                     t_in + r * tstride + 8 * u);
              }
            }
          }
        }
        r3dsimt::cp_async4(ring_int + st * Ring::kStageBytes,
                           reinterpret_cast<const void*>(reinterpret_cast<uintptr_t>(i_iss) & ~uintptr_t{3}));
      }
      r3dsimt::cp_async_commit();
      c_in += dcell;
      if constexpr (kReadsSum) s_in += dcell;
      if constexpr (MODE == kLastTerm) t_in += dcell;
      i_iss += dpx;
    };
#pragma unroll
    for (int k = 0; k < NS - 1; ++k) issue(k, k);
    uint32_t prev[K];
#pragma unroll
    for (int k = 0; k < K; ++k) prev[k] = 0;
    uint32_t pmin = 0;
    // Intensities and P2. With four stages or more, the next pixel's stage
    // has landed when this pixel is computed, so the P2 of the step into the
    // next pixel is looked up one step ahead, off the step's critical path
    // (iprev is then this pixel's intensity); with two stages the P2 of the
    // step into this pixel is looked up in its step (iprev is the previous
    // pixel's intensity). The first step's P2 is unused: its predecessor
    // vector is zero.
    constexpr bool kAheadP2 = NS >= 4;
    int iprev = 0;
    uint32_t p2next = 0;
    if constexpr (kAheadP2) {
      r3dsimt::cp_async_wait<NS - 2>();  // the first of the NS - 1 stages in flight
      const uint32_t iw0 = *reinterpret_cast<const uint32_t*>(ring_int);
      iprev = static_cast<int>((iw0 >> (16u * par0)) & 0xFFFFu);
    }

    auto step = [&](const int i, const int q) {
      const bool on = i < len;
      constexpr int kNext = NS - 1;
      issue(i + kNext, (q + kNext) % NS);
      uint32_t pen;
      if constexpr (kAheadP2) {
        r3dsimt::cp_async_wait<NS - 2>();  // this pixel's stage and the next one's
        const uint32_t iw = *reinterpret_cast<const uint32_t*>(ring_int + ((q + 1) % NS) * Ring::kStageBytes);
        const int inext =
            static_cast<int>((iw >> (16u * ((par0 ^ (static_cast<uint32_t>(i + 1) & dpar)) & 1u))) & 0xFFFFu);
        pen = pmin + p2next;
        const int dn = inext - iprev;
        p2next = lut[(dn < 0 ? -dn : dn) >> 8];
        iprev = inext;
      } else {
        r3dsimt::cp_async_wait<NS - 1>();
        const uint32_t iw = *reinterpret_cast<const uint32_t*>(ring_int + q * Ring::kStageBytes);
        const int icur =
            static_cast<int>((iw >> (16u * ((par0 ^ (static_cast<uint32_t>(i) & dpar)) & 1u))) & 0xFFFFu);
        const int dn = icur - iprev;
        iprev = icur;
        pen = pmin + lut[(dn < 0 ? -dn : dn) >> 8];
      }
      const unsigned char* sc = ring_cost + q * Ring::kStageBytes;
      uint2 craw[U];
      if constexpr (kVec) {
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          const uint4 w4 = uvalid[2 * v] ? *reinterpret_cast<const uint4*>(sc + 16 * v) : make_uint4(0, 0, 0, 0);
          craw[2 * v] = make_uint2(w4.x, w4.y);
          craw[2 * v + 1] = make_uint2(w4.z, w4.w);
        }
      } else {
#pragma unroll
        for (int u = 0; u < U; ++u)
          craw[u] = uvalid[u] ? *reinterpret_cast<const uint2*>(sc + 8 * u) : make_uint2(0, 0);
      }
      uint32_t c2[K];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        c2[4 * u + 0] = r3dsimt::perm(craw[u].x, 0u, 0x4140u);
        c2[4 * u + 1] = r3dsimt::perm(craw[u].x, 0u, 0x4342u);
        c2[4 * u + 2] = r3dsimt::perm(craw[u].y, 0u, 0x4140u);
        c2[4 * u + 3] = r3dsimt::perm(craw[u].y, 0u, 0x4342u);
      }
      // out = L_r = C + T_r with T_r = best - min L(q).
      const uint32_t pen2 = pen * 0x10001u;
      const uint32_t negmp = pmin * 0xFFFEFFFFu;  // -(pmin in both halves) modulo 2^32
      const uint32_t hl = r3dsimt::shfl(prev[K - 1], left_lane);
      const uint32_t hr = r3dsimt::shfl(prev[0], right_lane);
      uint32_t wv[K + 2];
      wv[0] = t > 0 ? hl : kSent2;
#pragma unroll
      for (int k = 0; k < K; ++k) wv[1 + k] = prev[k];
      wv[K + 1] = t + 1 < G ? hr : kSent2;
      uint32_t out[K], tr[K];
      uint32_t mprev = r3dsimt::perm(wv[0], wv[1], 0x5432u);
#pragma unroll
      for (int k = 0; k < K; ++k) {
        const uint32_t mnext = r3dsimt::perm(wv[k + 1], wv[k + 2], 0x5432u);
        const uint32_t nb = r3dsimt::vmin2(mprev, mnext);
        const uint32_t best = r3dsimt::vmin2(wv[k + 1], r3dsimt::vaddmin2(nb, p1x2, pen2));
        tr[k] = fma_add(best, one, negmp);
        out[k] = fma_add(tr[k], one, c2[k]);
        mprev = mnext;
      }
      // Minimum over the lane's labels (a tree), then over the chain's lanes.
      uint32_t mm[K];
#pragma unroll
      for (int k = 0; k < K; ++k) {
        if (!uvalid[k / 4]) out[k] = kSent2;
        mm[k] = out[k];
      }
#pragma unroll
      for (int s = 1; s < K; s <<= 1) {
#pragma unroll
        for (int k = 0; k + s < K; k += 2 * s) mm[k] = r3dsimt::vmin2(mm[k], mm[k + s]);
      }
      pmin = group_umin<G>(r3dsimt::umin(mm[0] & 0xFFFFu, mm[0] >> 16));
      uint32_t s[K];
      if constexpr (MODE == kFirst) {
        if (on) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (uvalid[u])
              r3dsimt::st_stream(reinterpret_cast<uint4*>(s_out + 8 * u),
                                 make_uint4(out[4 * u], out[4 * u + 1], out[4 * u + 2], out[4 * u + 3]));
        }
      } else if constexpr (MODE == kTerm) {
        if (on) {
          if constexpr (kVec) {
#pragma unroll
            for (int v = 0; v < NV; ++v)
              if (uvalid[2 * v])
                r3dsimt::st_stream(reinterpret_cast<uint4*>(t_out + 16 * v),
                                   make_uint4(r3dsimt::perm(tr[8 * v], tr[8 * v + 1], 0x6420u),
                                              r3dsimt::perm(tr[8 * v + 2], tr[8 * v + 3], 0x6420u),
                                              r3dsimt::perm(tr[8 * v + 4], tr[8 * v + 5], 0x6420u),
                                              r3dsimt::perm(tr[8 * v + 6], tr[8 * v + 7], 0x6420u)));
          } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (uvalid[u])
                r3dsimt::st_stream8(reinterpret_cast<uint2*>(t_out + 8 * u),
                                    make_uint2(r3dsimt::perm(tr[4 * u], tr[4 * u + 1], 0x6420u),
                                               r3dsimt::perm(tr[4 * u + 2], tr[4 * u + 3], 0x6420u)));
          }
        }
      } else if constexpr (MODE == kLastTerm) {
        // S = L_8 + 7 C + sum of the seven byte terms (no halfword overflows).
#pragma unroll
        for (int k = 0; k < K; ++k) s[k] = out[k] + 7u * c2[k];
        const unsigned char* stt = ring_term + q * Ring::kStageBytes;
#pragma unroll
        for (int r = 0; r < kTermArrays; ++r) {
          uint2 tw[U];
          if constexpr (kVec) {
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              const uint4 w4 = uvalid[2 * v] ? *reinterpret_cast<const uint4*>(stt + r * CPW * Ring::ND + 16 * v)
                                             : make_uint4(0, 0, 0, 0);
              tw[2 * v] = make_uint2(w4.x, w4.y);
              tw[2 * v + 1] = make_uint2(w4.z, w4.w);
            }
          } else {
#pragma unroll
            for (int u = 0; u < U; ++u)
              tw[u] = uvalid[u] ? *reinterpret_cast<const uint2*>(stt + r * CPW * Ring::ND + 8 * u) : make_uint2(0, 0);
          }
#pragma unroll
          for (int u = 0; u < U; ++u) {
            s[4 * u + 0] = fma_add(r3dsimt::perm(tw[u].x, 0u, 0x4140u), one, s[4 * u + 0]);
            s[4 * u + 1] = fma_add(r3dsimt::perm(tw[u].x, 0u, 0x4342u), one, s[4 * u + 1]);
            s[4 * u + 2] = fma_add(r3dsimt::perm(tw[u].y, 0u, 0x4140u), one, s[4 * u + 2]);
            s[4 * u + 3] = fma_add(r3dsimt::perm(tw[u].y, 0u, 0x4342u), one, s[4 * u + 3]);
          }
        }
      } else {
        const unsigned char* ss = ring_sum + q * Ring::kStageBytes;
#pragma unroll
        for (int u = 0; u < U; ++u) {
          const uint4 sraw = uvalid[u] ? *reinterpret_cast<const uint4*>(ss + 16 * u) : make_uint4(0, 0, 0, 0);
          s[4 * u + 0] = add2(sraw.x, out[4 * u + 0], no_carry);
          s[4 * u + 1] = add2(sraw.y, out[4 * u + 1], no_carry);
          s[4 * u + 2] = add2(sraw.z, out[4 * u + 2], no_carry);
          s[4 * u + 3] = add2(sraw.w, out[4 * u + 3], no_carry);
        }
        if constexpr (MODE == kAccumulate) {
          if (on) {
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (uvalid[u])
                r3dsimt::st_stream(reinterpret_cast<uint4*>(s_out + 8 * u),
                                   make_uint4(s[4 * u], s[4 * u + 1], s[4 * u + 2], s[4 * u + 3]));
          }
        }
      }
      if constexpr (kWta) {
        // Winner-takes-all over the total sums (sgm_kernels.cpp:332-358):
        // the first minimum, the second best outside +-1, and S at kb -+ 1.
        // Labels of units past nd count as 0xFFFF (they follow every valid
        // label, so they never come first among equal minima); with byte
        // terms their sum is the sentinel 0x7FFF, above every valid S (at
        // most 8 (255 + 255)), which serves as well.
        uint32_t sv[K];
#pragma unroll
        for (int k = 0; k < K; ++k) sv[k] = (MODE == kLastTerm || uvalid[k / 4]) ? s[k] : 0xFFFFFFFFu;
        // The lane's minimum and its first label, as one key S << 16 | label
        // whose minimum over the lane group is (bcost, kb).
        uint32_t mv = sv[0];
#pragma unroll
        for (int k = 1; k < K; ++k) mv = r3dsimt::vmin2(mv, sv[k]);
        const uint32_t lmin = r3dsimt::umin(mv & 0xFFFFu, mv >> 16);
        // Per word min(S - lmin, 1) is 0 in the halves at the minimum (every
        // half is >= lmin, so the subtraction borrows nothing).
        const uint32_t l2 = lmin * 0x10001u;
        uint32_t miss = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) miss |= r3dsimt::vmin2(sv[k] - l2, 0x00010001u) << k;
        const uint32_t hit = ~miss & (((1u << K) - 1u) * 0x10001u);
        const uint32_t he = hit & 0xFFFFu, ho = hit >> 16;
        const uint32_t fe = he != 0 ? static_cast<uint32_t>(2 * (r3dsimt::ffs(he) - 1)) : 0xFFFFu;
        const uint32_t fo = ho != 0 ? static_cast<uint32_t>(2 * (r3dsimt::ffs(ho) - 1) + 1) : 0xFFFFu;
        const uint32_t key = group_umin<G>((lmin << 16) | (r3dsimt::umin(fe, fo) + static_cast<uint32_t>(e0)));
        const uint32_t bcost = key >> 16;
        const int kb = static_cast<int>(key & 0xFFFFu);
        // The second best outside kb -+ 1. Label kb - 1 lies in the lane's
        // word wa = (kb - 1 - e0) >> 1 (arithmetic shift; out of [0, K) in
        // other lanes): its high half only when kb - 1 - e0 is odd, then kb and
        // kb + 1 fill word wa + 1; its both halves when even, then kb + 1 is the
        // low half of word wa + 1.
        const int wo = kb - 1 - e0;
        const int wa = wo >> 1;
        const uint32_t mask_a = (wo & 1) ? 0xFFFF0000u : 0xFFFFFFFFu;
        const uint32_t mask_b = (wo & 1) ? 0xFFFFFFFFu : 0x0000FFFFu;
        uint32_t sec2 = 0xFFFFFFFFu;
#pragma unroll
        for (int k = 0; k < K; ++k) {
          const uint32_t m = (k == wa ? mask_a : 0u) | (k == wa + 1 ? mask_b : 0u);
          sec2 = r3dsimt::vmin2(sec2, sv[k] | m);
        }
        const uint32_t sec = group_umin<G>(r3dsimt::umin(sec2 & 0xFFFFu, sec2 >> 16));
        const int km = kb > 0 ? kb - 1 : 0, kp = kb + 1 < nd ? kb + 1 : nd - 1;
        const int base_lane = gi * G;
        uint32_t vm = pick<K>(s, (km % (2 * K)) >> 1);
        uint32_t vp = pick<K>(s, (kp % (2 * K)) >> 1);
        vm = r3dsimt::shfl(vm, (base_lane + km / (2 * K)) & 31);
        vp = r3dsimt::shfl(vp, (base_lane + kp / (2 * K)) & 31);
        const uint32_t sm = (km & 1) ? (vm >> 16) : (vm & 0xFFFFu);
        const uint32_t sp = (kp & 1) ? (vp >> 16) : (vp & 0xFFFFu);
        if (on) {
          if (t == 0)
            info[px_out] = make_int4(static_cast<int>(static_cast<uint32_t>(kb) | (bcost << 16)),
                                     static_cast<int>(sec | (sm << 16)), static_cast<int>(sp), 0);
          if (job.volume != nullptr) {
            uint16_t* vb = job.volume + (static_cast<int64_t>(y) * w + x) * nd + e0;
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (uvalid[u])
                *reinterpret_cast<uint4*>(vb + 8 * u) = make_uint4(s[4 * u], s[4 * u + 1], s[4 * u + 2], s[4 * u + 3]);
          }
          if (m.diagonal_lr) {
            // Right-view WTA along the diagonal (sgm_kernels.cpp:349-356): the
            // smallest (S, x) key per right column.
            const RowInterval lv = m.bv[job.y0 + y];
            const int bx = job.x0 + x;
            if (bx >= lv.first && bx <= lv.last) {
              uint32_t* keys = rkeys + job.rk_off + static_cast<int64_t>(y) * (w + nd);
              const int b0 = x + nd - 1;
#pragma unroll
              for (int k = 0; k < K; ++k) {
                if (uvalid[k / 4]) {
                  const int e = e0 + 2 * k;
                  atomicMin(keys + (b0 - e), ((s[k] & 0xFFFFu) << 16) | static_cast<uint32_t>(x));
                  atomicMin(keys + (b0 - e - 1), (s[k] & 0xFFFF0000u) | static_cast<uint32_t>(x));
                }
              }
            }
          }
        }
      }
      (void)s;
#pragma unroll
      for (int k = 0; k < K; ++k) prev[k] = out[k];
      if constexpr (MODE == kFirst || MODE == kAccumulate) s_out += dcell;
      if constexpr (MODE == kTerm) t_out += dcell;
      if constexpr (kWta) {
        px_out += dpx;
        x += dx;
        y += dy;
      }
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
// of a reduced range (:501-503), the diagonal left-right check (`shift` is the
// row's key offset), uniqueness, subpixel fit and confidence of one pixel.
struct Winner {
  int best;                    // label of the first minimum
  uint32_t bcost, sec, sm, sp;  // S there, second best, S at best -+ 1
};
R3D_DEVICE void accept_pixel(const SgmMatch& m, const SgmPathJob& job, int x, int y, int lo, int num, const Winner& v,
                             const uint32_t* rkeys, int shift, float& d, float& cf) {
  const int bx = job.x0 + x, by = job.y0 + y;
  const RowInterval rv = m.pv[by];
  const int jb = v.best - lo;
  const int xr = bx - m.dmin - v.best;
  bool ok = xr >= rv.first && xr <= rv.last;
  if ((jb == 0 && lo > 0) || (jb == num - 1 && lo + num < m.nd)) ok = false;
  if (ok && m.diagonal_lr) {
    const uint32_t key = rkeys[job.rk_off + static_cast<int64_t>(y) * (job.w + m.nd) + (x - v.best + shift)];
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

// Full range: lo = 0, num = nd for every pixel.
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_accept_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                           int64_t pixels, const int4* R3D_RESTRICT info, const uint32_t* R3D_RESTRICT rkeys) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < pixels; i += stride) {
    const int j = find_job(jobs, njobs, i, [](const SgmPathJob& q) { return q.px_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    const int nd = m.nd, w = job.w;
    const int p = static_cast<int>(i - job.px_off);
    const int y = p / w, x = p - (p / w) * w;
    const RowInterval lv = m.bv[job.y0 + y];
    float d = kInfF, cf = 0.0F;
    if (job.x0 + x >= lv.first && job.x0 + x <= lv.last)
      accept_pixel(m, job, x, y, 0, nd, unpack_winner(info[i]), rkeys, nd - 1, d, cf);
    job.disp[p] = d;
    if (job.conf != nullptr) job.conf[p] = cf;
    if (p == 0) *job.cells = static_cast<unsigned long long>(w) * static_cast<unsigned long long>(job.h) * nd;
  }
}

// ================================================================ ranged tiles
// Per-pixel label ranges (lo, num; num a multiple of 16): the same passes on
// costs, terms and sums packed per tile, pixel after pixel, in units of 16
// labels. Within a unit the labels are interleaved so that a 32-bit word of
// the passes holds labels k and k + 8: the neighbours d -+ 1 of word k are
// then words k -+ 1, without byte permutes. Byte planes (costs, terms) store
// the bytes of word j = 0..3 of a unit as labels 2 j, 2 j + 1, 2 j + 8, 2 j + 9
// (one mask or permute unpacks a word, one multiply-add packs two); sums
// store word k = 0..7 as the halves of labels k and k + 8.

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
    for (int xb = 0; xb < w; xb += 32) {
      const int x = xb + lane, bx = job.x0 + x;
      const int lo = x < w ? lorow[bx] : 0, nu = x < w ? numrow[bx] >> 4 : 0;
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
                       static_cast<uint32_t>(lo) | (static_cast<uint32_t>(irow[bx]) << 16));
      const bool inside = x < w && bx >= lv.first && bx <= lv.last;
      const uint64_t cl = inside ? lrow[bx] : 0;
      uint8_t* out = cost + job.cell_off + static_cast<int64_t>(off) * 16;
      for (int u = 0; u < nu; ++u) {
        uint32_t q[4] = {0, 0, 0, 0};
        const int xr0 = bx - m.dmin - lo - 16 * u;  // right column of the unit's label 0
        if (inside && xr0 <= rv.last && xr0 - 15 >= rv.first) {
          // Every label reads a valid right column: the two popcounts of each
          // Census XOR packed separately (each byte at most 32, no carries).
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const int l[4] = {2 * k, 2 * k + 1, 2 * k + 8, 2 * k + 9};
            uint32_t a = 0, b = 0;
#pragma unroll
            for (int i = 3; i >= 0; --i) {
              const uint64_t d = cl ^ crow[xr0 - l[i]];
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
// Everything is private to a lane: no barrier, no warp-wide minimum.
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
  static constexpr int kPadWords = (CH + 2) / 2;  // sentinels before and after a vector
  static constexpr int kVecStep = kVecLabels / 2 + kPadWords;  // from buffer 0 to buffer 1
  static constexpr int kVecStride = (2 * kVecStep + kPadWords + 1) | 1;
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
  constexpr int CH = R::CH, UF = R::UF, D = R::D, NR = R::NR, NS = R::kVecLabels, PAD = R::kPadWords;
  R3D_DYNAMIC_SMEM(smem);
  const int lane = static_cast<int>(threadIdx.x & 31u), warp = static_cast<int>(threadIdx.x >> 5);
  const int wpb = static_cast<int>(blockDim.x) >> 5;
  const int64_t nwarps = static_cast<int64_t>(gridDim.x) * wpb;
  unsigned char* const wb = smem + static_cast<size_t>(warp) * R::kWarpBytes;
  unsigned char* const data = wb + lane * 16;
  uint2* const recs = reinterpret_cast<uint2*>(wb + R::kData) + lane;  // slot q at recs[32 q]
  // Buffer b of the lane: words -PAD .. NS / 2 + PAD - 1 around vec + b * kVecStep.
  uint32_t* const vec = reinterpret_cast<uint32_t*>(wb + R::kData + R::kRec) + lane * R::kVecStride + PAD;
  uint16_t* const lut = reinterpret_cast<uint16_t*>(wb + R::kData + R::kRec + R::kVec);
  // The lane's buffers of wide vectors: word q (from -PAD on) of buffer b at
  // wide[(b * ovf_words + q) * 32].
  uint32_t* const wide =
      ovf + ((static_cast<int64_t>(blockIdx.x) * wpb + warp) * 2 * ovf_words + PAD) * 32 + lane;
  if (ovf_words > 0) {
    for (int k = 1; k <= PAD; ++k) {
      wide[-32 * k] = kSent2;
      wide[(ovf_words - k) * 32] = kSent2;
    }
  }
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
    int sx, sy, len;
    chain_geometry(cls, dx, dy, w, job.h, blk * 32 + lane, sx, sy, len);
    int maxlen = len;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) maxlen = r3dsimt::imax(maxlen, static_cast<int>(r3dsimt::shfl_xor(maxlen, o)));
    const uint8_t* const cbase = cost + job.cell_off;
    uint16_t* const sbase = sum + job.cell_off;
    uint8_t* const tout = terms + job.cell_off + tslot * tstride;
    const int dpx = dy * w + dx;
    const uint2* rp = rec + job.px_off + static_cast<int64_t>(sy) * w + sx;  // record of the next pixel to request
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
    // Pixel i + D - 1's first chunk into slot st, pixel i + 2 D - 1's record;
    // one group. (Records: requested D steps before the data, so landed.)
    auto issue = [&](int i, int st) {
      if (i + D - 1 < len) {
        const uint2 r = recs[((i + D - 1) & (NR - 1)) * 32];
        issue_chunk(st, static_cast<int>(r.x & kRecOffset), static_cast<int>(r.x >> kRecShift));
      }
      if (i + 2 * D - 1 < len) r3dsimt::cp_async8(&recs[((i + 2 * D - 1) & (NR - 1)) * 32], rp);
      rp += dpx;
      r3dsimt::cp_async_commit();
    };
#pragma unroll
    for (int k = 0; k < 2 * D - 1; ++k) {
      if (k < len) recs[k * 32] = *rp;
      rp += dpx;
    }
#pragma unroll
    for (int k = 0; k < D - 1; ++k) {
      if (k < len) {
        const uint2 r = recs[k * 32];
        issue_chunk(k, static_cast<int>(r.x & kRecOffset), static_cast<int>(r.x >> kRecShift));
      }
      r3dsimt::cp_async_commit();
    }
    uint2 rc = make_uint2(0, 0);  // this pixel's record
    if (len > 0) rc = recs[0];
    // The predecessor's range, its minimum over labels in both halves,
    // negated, and the clamp min L(q) + P2. A zero clamp makes the first
    // pixel's best term 0 whatever the predecessor words hold: T = 0, L = C.
    int lo_q = 0, num_q = 0;
    uint32_t pen2 = 0, negmp = 0;
    uint32_t prev[K];
#pragma unroll
    for (int k = 0; k < K; ++k) prev[k] = 0;
    bool single = static_cast<int>(rc.x >> kRecShift) == UF;  // this pixel is one full chunk
    bool fast = r3dsimt::ballot(len > 0 && !single) == 0;
    bool clean = false;  // the buffers hold sentinels outside what this chain wrote
    int high = 0;        // labels of the longest vector written
    auto make_clean = [&]() {
      if (clean) return;
      for (int k = -PAD; k < R::kVecStride - PAD; ++k) vec[k] = kSent2;
      clean = true;
    };
    // From the best terms of a chunk (its bytes in ring slot st, its cells
    // from unit `at` on): T = best - min L(q), L = C + T, and the outputs.
    uint32_t out[K], pm;
    auto finish = [&](const uint32_t (&best)[K], int st, int at, bool on, bool upper) {
      const unsigned char* src = data + st * R::kStageBytes;
      uint32_t c2[K], tr[K];
#pragma unroll
      for (int u = 0; u < UF; ++u) {
        const uint4 v = *reinterpret_cast<const uint4*>(src + u * 512);
        const uint32_t cw[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          c2[8 * u + 2 * k] = cw[k] & 0x00FF00FFu;
          c2[8 * u + 2 * k + 1] = r3dsimt::perm(cw[k], 0u, 0x4341u);
        }
      }
#pragma unroll
      for (int k = 0; k < K; ++k) {
        tr[k] = fma_add(best[k], one, negmp);
        out[k] = fma_add(tr[k], one, c2[k]);
        if (k >= 8 && !upper) out[k] = kSent2;
      }
      {
        constexpr int N3 = (K + 2) / 3;
        uint32_t t3[N3];
#pragma unroll
        for (int k = 0; k < N3; ++k)
          t3[k] = r3dsimt::vmin3(out[3 * k], out[3 * k + 1 < K ? 3 * k + 1 : 3 * k], out[3 * k + 2 < K ? 3 * k + 2 : 3 * k]);
#pragma unroll
        for (int k = 0; k < N3; k += 2) pm = r3dsimt::vmin3(pm, t3[k], t3[k + 1 < N3 ? k + 1 : k]);
      }
      if (!on) return;
#pragma unroll
      for (int u = 0; u < UF; ++u) {
        if (u > 0 && !upper) continue;
        const int64_t off = static_cast<int64_t>(at + u) * 16;
        const int q = 8 * u;
        if constexpr (MODE == kTerm) {
          r3dsimt::st_stream(reinterpret_cast<uint4*>(tout + off),
                             make_uint4(tr[q] + 256u * tr[q + 1], tr[q + 2] + 256u * tr[q + 3],
                                        tr[q + 4] + 256u * tr[q + 5], tr[q + 6] + 256u * tr[q + 7]));
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
        if (last) {
          // Sentinels after the vector where a longer one was written before.
          if (n < high) {
#pragma unroll
            for (int k = 0; k < PAD; ++k) v[end + k] = kSent2;
          }
          high = r3dsimt::imax(high, n);
        }
      } else {
        uint32_t* v = wide + ((i & 1) * ovf_words + c * K) * 32;
#pragma unroll
        for (int k = 0; k < K; ++k)
          if (k < 8 || upper) v[k * 32] = nat[k];
        if (last) {
#pragma unroll
          for (int k = 0; k < PAD; ++k) v[(end + k) * 32] = kSent2;
        }
      }
    };
    // best = min(L(q, d), L(q, d -+ 1) + P1, min L(q) + P2); clamping first
    // leaves one 3-way minimum per word. From the lane's buffer of pixel i -
    // 1, for the labels of chunk c at lo.
    auto best_from_memory = [&](uint32_t (&best)[K], int i, int c, int lo) {
      // Predecessor labels b - 1 .. b + CH (its own indexing).
      int b = c * CH + lo - lo_q;
      b = r3dsimt::imax(r3dsimt::imin(b, num_q + 1), -(CH + 1));
      // pr[k]: labels b - 1 + 2 k, b + 2 k, from the words holding them.
      const int f = (b - 1) >> 1;
      const uint32_t par = 16u * (static_cast<uint32_t>(b - 1) & 1u);
      uint32_t wd[K + 2], pr[K + 1];
      if (num_q <= NS) {
        const uint32_t* vq = vec + ((i & 1) ^ 1) * R::kVecStep + f;
#pragma unroll
        for (int k = 0; k < K + 2; ++k) wd[k] = vq[k];
      } else {
        const uint32_t* oq = wide + (((i & 1) ^ 1) * ovf_words + f) * 32;
#pragma unroll
        for (int k = 0; k < K + 2; ++k) wd[k] = oq[k * 32];
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
      const bool on = i < len;
      const int at = static_cast<int>(rc.x & kRecOffset);
      const int lo = static_cast<int>(rc.y & 0xFFFFu);
      uint2 rn = rc;  // the next pixel's record
      if (i + 1 < len) rn = recs[((i + 1) & (NR - 1)) * 32];
      const bool single_n = static_cast<int>(rn.x >> kRecShift) == UF;
      const bool okn = i + 1 >= len || (single && single_n && ((rn.y ^ rc.y) & 0xFFFFu) == 0);
      const bool fast_next = r3dsimt::ballot(!okn) == 0;
      pm = kSent2;
      uint32_t best[K];
      int n = UF;
      if (fast) {
        issue(i, st_in);
        r3dsimt::cp_async_wait<D - 1>();
        uint32_t cl[K];
#pragma unroll
        for (int k = 0; k < K; ++k) cl[k] = r3dsimt::vmin2(prev[k], pen2);
#pragma unroll
        for (int u = 0; u < UF; ++u) {
          // Words -1 and 8 of the unit: labels (16 u - 1, 16 u + 7) and (16 u + 8, 16 u + 16).
          uint32_t s[10];
          s[0] = fma_add(r3dsimt::perm(u > 0 ? cl[8 * (u > 0 ? u - 1 : 0) + 7] : pen2, cl[8 * u + 7], 0x5432u), one, p1x2);
#pragma unroll
          for (int k = 0; k < 8; ++k) s[1 + k] = fma_add(cl[8 * u + k], one, p1x2);
          s[9] = fma_add(r3dsimt::perm(cl[8 * u], u + 1 < UF ? cl[8 * (u + 1 < UF ? u + 1 : 0)] : pen2, 0x5432u), one,
                         p1x2);
#pragma unroll
          for (int k = 0; k < 8; ++k) best[8 * u + k] = r3dsimt::vmin3(cl[8 * u + k], s[k], s[2 + k]);
        }
        finish(best, st, at, on, true);
        if (!fast_next) {
          make_clean();
          if (on) store_vec(i, 0, n, true);
        }
      } else {
        make_clean();
        n = on ? units_of(rc, i) : 1;
        const bool multi = r3dsimt::ballot(n > UF) != 0;
        if (!multi) {
          issue(i, st_in);
          r3dsimt::cp_async_wait<D - 1>();
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
        const int dn = static_cast<int>(rn.y >> 16) - static_cast<int>(rc.y >> 16);
        pen2 = mp + lut[(dn < 0 ? -dn : dn) >> 8] * 0x10001u;
        negmp = 0u - mp;
      }
      lo_q = lo;
      num_q = 16 * n;
      rc = rn;
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
template <bool TERMS>
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kPathThreads)
    sgm_path_ranged_wta_kernel(const SgmMatch* R3D_RESTRICT matches, const SgmPathJob* R3D_RESTRICT jobs, int njobs,
                               int64_t pixels, const uint2* R3D_RESTRICT rec, const uint8_t* R3D_RESTRICT cost,
                               const uint16_t* R3D_RESTRICT sum, const uint8_t* R3D_RESTRICT terms, int64_t tstride,
                               const int* R3D_RESTRICT rowshift, int4* R3D_RESTRICT info, uint32_t* rkeys) {
  const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < pixels; i += stride) {
    const int j = find_job(jobs, njobs, i, [](const SgmPathJob& q) { return q.px_off; });
    const SgmPathJob& job = jobs[j];
    const SgmMatch& m = matches[job.match];
    const int p = static_cast<int>(i - job.px_off);
    const int y = p / job.w, x = p - y * job.w;
    const uint2 rc = rec[i];
    const int lo = static_cast<int>(rc.y & 0xFFFFu), nu = rec_units(rc, m, job, x, y), num = 16 * nu;
    const int64_t off = static_cast<int64_t>(rc.x & kRecOffset) * 16;
    const uint8_t* cp = cost + job.cell_off + off;
    const uint8_t* tp = terms + job.cell_off + off;
    const uint4* sp4 = reinterpret_cast<const uint4*>(sum + job.cell_off + off);
    // Word k of a unit holds labels k and k + 8.
    auto unit = [&](int u, uint32_t (&wv)[8]) {
      if constexpr (TERMS) {
        uint4 t[1 + kRangedTerms];
        t[0] = *reinterpret_cast<const uint4*>(cp + 16 * u);
#pragma unroll
        for (int r = 0; r < kRangedTerms; ++r)
          t[1 + r] = r3dsimt::ld_stream(reinterpret_cast<const uint4*>(tp + r * tstride + 16 * u));
#pragma unroll
        for (int r = 0; r <= kRangedTerms; ++r) {
          const uint32_t tw[4] = {t[r].x, t[r].y, t[r].z, t[r].w};
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const uint32_t a = tw[k] & 0x00FF00FFu, b = r3dsimt::perm(tw[k], 0u, 0x4341u);
            wv[2 * k] = r == 0 ? 8u * a : wv[2 * k] + a;
            wv[2 * k + 1] = r == 0 ? 8u * b : wv[2 * k + 1] + b;
          }
        }
        return;
      }
      const uint4 a = sp4[2 * u], b = sp4[2 * u + 1];
      wv[0] = a.x;
      wv[1] = a.y;
      wv[2] = a.z;
      wv[3] = a.w;
      wv[4] = b.x;
      wv[5] = b.y;
      wv[6] = b.z;
      wv[7] = b.w;
    };
    uint32_t wv[8];
    uint32_t kmin = 0xFFFFFFFFu;
    for (int u = nu - 1; u >= 0; --u) {  // ends with unit 0 in wv: the only one of most pixels
      unit(u, wv);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const uint32_t e = static_cast<uint32_t>(16 * u + k);
        kmin = r3dsimt::umin(kmin, r3dsimt::umin((wv[k] << 16) | e, (wv[k] & 0xFFFF0000u) | (e + 8)));
      }
      if (job.volume != nullptr) {
        uint16_t* vol = job.volume + off + 16 * u;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          vol[k] = static_cast<uint16_t>(wv[k] & 0xFFFFu);
          vol[k + 8] = static_cast<uint16_t>(wv[k] >> 16);
        }
      }
    }
    const int kb = static_cast<int>(kmin & 0xFFFFu);
    const int km = kb > 0 ? kb - 1 : 0;
    const int kp = kb + 1 < num ? kb + 1 : (num > 0 ? num - 1 : 0);
    uint32_t sec = 0xFFFFu, sm = 0, spv = 0;
    for (int u = 0; u < nu; ++u) {
      if (u > 0) unit(u, wv);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          const int e = 16 * u + k + 8 * hf;
          const uint32_t v = hf != 0 ? wv[k] >> 16 : wv[k] & 0xFFFFu;
          if (e + 1 < kb || e > kb + 1) sec = r3dsimt::umin(sec, v);
          if (e == km) sm = v;
          if (e == kp) spv = v;
        }
      }
    }
    const Winner win{lo + kb, kmin >> 16, sec, sm, spv};
    const RowInterval lv = m.bv[job.y0 + y];
    const bool inside = job.x0 + x >= lv.first && job.x0 + x <= lv.last;
    if (m.diagonal_lr) {
      info[i] = pack_winner(win);
      if (inside) {
        uint32_t* keys = rkeys + job.rk_off + static_cast<int64_t>(y) * (job.w + m.nd);
        const int base = x - lo + rowshift[job.row_off + y];
        for (int u = 0; u < nu; ++u) {
          unit(u, wv);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const int e = 16 * u + k;
            atomicMin(keys + (base - e), (wv[k] << 16) | static_cast<uint32_t>(x));
            atomicMin(keys + (base - e - 8), (wv[k] & 0xFFFF0000u) | static_cast<uint32_t>(x));
          }
        }
      }
      continue;
    }
    float d = kInfF, cf = 0.0F;
    if (inside) accept_pixel(m, job, x, y, lo, num, win, rkeys, 0, d, cf);
    job.disp[p] = d;
    if (job.conf != nullptr) job.conf[p] = cf;
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
                   unpack_winner(info[i]), rkeys, rowshift[job.row_off + y], d, cf);
    }
    job.disp[p] = d;
    if (job.conf != nullptr) job.conf[p] = cf;
  }
}

// ---------------------------------------------------------------- launches
// Pass order: the first pass writes the sums, the last takes the WTA.
struct Pass {
  int cls, dx, dy;
};
constexpr Pass kPasses[8] = {{0, 1, 0},  {1, 0, 1},   {2, 1, 1},  {2, -1, 1},
                             {1, 0, -1}, {2, -1, -1}, {2, 1, -1}, {0, -1, 0}};

template <class Kernel>
int resident_grid(Kernel kernel, int sms, int64_t work_items, int per_block, size_t smem = 0,
                  int threads = kPathThreads) {
  int per_sm = 1;
  R3D_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
  const int64_t need = (work_items + per_block - 1) / per_block;
  const int64_t resident = static_cast<int64_t>(sms) * (per_sm > 0 ? per_sm : 1);
  return static_cast<int>(need < resident ? (need > 0 ? need : 1) : resident);
}

// Algorithmic HBM bytes of one pass over `cells` cells of `pixels` pixels:
// costs read, sums read (not by the first pass) and written (not by the
// full-range last pass, which writes the WTA records instead); byte terms:
// one written per cell by passes 1..7, seven read by the last pass.
uint64_t pass_bytes(int mode, bool ranged, const SgmPathSegment& g) {
  const uint64_t c = static_cast<uint64_t>(g.cells), px = static_cast<uint64_t>(g.pixels);
  if (mode == kFirst) return 3 * c;
  if (mode == kTerm) return 2 * c;
  if (mode == kLastTerm) return (1 + kTermArrays) * c + 16 * px;
  if (mode == kLast && !ranged) return 3 * c + 16 * px;
  return 5 * c;
}

template <int G, int K, int MODE, bool FULL = false>
void launch_pass(const PassSet& ps, const SgmMatch* dm, const SgmPathJob* jobs, int njobs, const uint8_t* cost,
                 uint16_t* sum, uint8_t* terms, int64_t tstride, int4* info, uint32_t* rkeys, const uint16_t* ints,
                 int sms, cudaStream_t s, const SgmPathSegment& seg, const int* cancel) {
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
             ps, cost, sum, terms, tstride, info, rkeys, ints, cancel);
  launched("sgm_path_kernel");
  if (ev0 != nullptr) {
    char shape[32];
    std::snprintf(shape, sizeof(shape), "%dx%d/mode%d", G, K, MODE);
    const uint64_t n = static_cast<uint64_t>(ps.n);
    profile_pass(ev0, profile_mark(s), "sgm_path_kernel", shape, n * static_cast<uint64_t>(seg.cells),
                 n * static_cast<uint64_t>(seg.pixels), n * pass_bytes(MODE, false, seg));
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
                   uint16_t* sum, uint8_t* terms, int64_t tstride, int4* info, uint32_t* rkeys, const uint16_t* ints,
                   int sms, cudaStream_t s, const int* cancel, int* counters) {
  for (int q = 0; q < 8; ++q)
    if (g.blocks[kPasses[q].cls] <= 0) return;  // no pixels: every class has chains otherwise
  if (terms != nullptr) {
    // The seven term passes in one launch, then the last pass, which finds
    // all seven term arrays written.
    const int qs[kTermArrays] = {0, 1, 2, 3, 4, 5, 6};
    const int last = 7;
    // Segments whose matches fill every label unit take the kernels without
    // the per-unit validity selects.
    if (g.full != 0) {
      launch_pass<G, K, kTerm, true>(pass_set(g, qs, kTermArrays, counters), dm, jobs, g.count, cost, sum, terms, tstride, info,
                                     rkeys, ints, sms, s, g, cancel);
      launch_pass<G, K, kLastTerm, true>(pass_set(g, &last, 1, counters + 1), dm, jobs, g.count, cost, sum, terms, tstride, info,
                                         rkeys, ints, sms, s, g, cancel);
    } else {
      launch_pass<G, K, kTerm>(pass_set(g, qs, kTermArrays, counters), dm, jobs, g.count, cost, sum, terms, tstride, info,
                               rkeys, ints, sms, s, g, cancel);
      launch_pass<G, K, kLastTerm>(pass_set(g, &last, 1, counters + 1), dm, jobs, g.count, cost, sum, terms, tstride, info, rkeys,
                                   ints, sms, s, g, cancel);
    }
    return;
  }
  for (int q = 0; q < 8; ++q) {
    const PassSet ps = pass_set(g, &q, 1, counters + q);
    if (q == 0)
      launch_pass<G, K, kFirst>(ps, dm, jobs, g.count, cost, sum, terms, tstride, info, rkeys, ints, sms, s, g,
                                cancel);
    else if (q < 7)
      launch_pass<G, K, kAccumulate>(ps, dm, jobs, g.count, cost, sum, terms, tstride, info, rkeys, ints, sms, s, g,
                                     cancel);
    else
      launch_pass<G, K, kLast>(ps, dm, jobs, g.count, cost, sum, terms, tstride, info, rkeys, ints, sms, s, g,
                               cancel);
  }
}

// Shapes compiled into the library (lanes per chain G, label pairs per lane K).
#define R3D_PATH_SHAPES(X) \
  X(1, 8)                  \
  X(2, 8)                  \
  X(2, 12)                 \
  X(2, 16)                 \
  X(4, 8)                  \
  X(4, 12)                 \
  X(4, 16)                 \
  X(8, 8)                  \
  X(8, 12)                 \
  X(8, 16)                 \
  X(16, 8)                 \
  X(16, 12)                \
  X(16, 16)                \
  X(32, 8)                 \
  X(32, 12)

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

SgmPathShape sgm_path_shape(int nd) {
  // A compiled shape from R3DGPU_PATH_SHAPE ("G,K": any label count it
  // covers) or the tuning table (an entry for exactly this label count),
  // else the narrowest row of 8 or 12 label pairs per lane, ties to fewer
  // lanes per chain.
  if (const char* e = std::getenv("R3DGPU_PATH_SHAPE")) {
    int g = 0, k = 0;
    if (std::sscanf(e, "%d,%d", &g, &k) == 2 && path_shape_compiled(g, k) && 2 * g * k >= nd) return {g, k};
  }
  const auto it = tuning().path.find(nd);
  if (it != tuning().path.end() && path_shape_compiled(it->second.g, it->second.k) &&
      2 * it->second.g * it->second.k >= nd)
    return {it->second.g, it->second.k};
  SgmPathShape best{0, 0};
  int best_nd = 1 << 30;
#define R3D_SHAPE(g, k)                                       \
  if (k != 16 && 2 * g * k >= nd && 2 * g * k < best_nd) { \
    best = SgmPathShape{g, k};                                \
    best_nd = 2 * g * k;                                      \
  }
  R3D_PATH_SHAPES(R3D_SHAPE)
#undef R3D_SHAPE
  return best;
}

SgmPathBuffers sgm_path_buffers(int64_t cells, int64_t pixels, int64_t keys, bool terms) {
  SgmPathBuffers b{};
  size_t o = 0;
  b.cost = o;
  o += align256(static_cast<size_t>(cells));
  b.sum = o;
  b.term_stride = terms ? static_cast<int64_t>(align256(static_cast<size_t>(cells))) : 0;
  b.terms = b.sum;
  o += terms ? static_cast<size_t>(kTermArrays) * static_cast<size_t>(b.term_stride)
             : align256(static_cast<size_t>(cells) * 2);
  b.info = o;
  o += align256(static_cast<size_t>(pixels) * 16);
  b.rkeys = o;
  o += align256(static_cast<size_t>(keys) * 4);
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
  const SgmPathBuffers B = sgm_path_buffers(wave.cells, wave.pixels, wave.keys, wave.terms != 0);
  uint8_t* cost = wave.buffer + B.cost;
  uint16_t* sum = reinterpret_cast<uint16_t*>(wave.buffer + B.sum);
  uint8_t* terms = wave.terms != 0 ? wave.buffer + B.terms : nullptr;
  int4* info = reinterpret_cast<int4*>(wave.buffer + B.info);
  uint32_t* rkeys = reinterpret_cast<uint32_t*>(wave.buffer + B.rkeys);
  uint16_t* ints = reinterpret_cast<uint16_t*>(wave.buffer + B.ints);
  int* counters = reinterpret_cast<int*>(wave.buffer + B.counters);
  if (8 * wave.nsegs > kPathCounters) fail(R3DGPU_EINVAL, "stereo: too many path kernel shapes in a wave");
  if (wave.keys > 0) R3D_CUDA(cudaMemsetAsync(rkeys, 0xFF, static_cast<size_t>(wave.keys) * 4, s));
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
    launch_passes<gg, kk>(dm, jobs, g, cost, sum, terms, B.term_stride, info, rkeys, ints, sms, s, wave.cancel, \
                          counters + 8 * q);                                                                  \
    done = true;                                                                                              \
  }
    R3D_PATH_SHAPES(R3D_SHAPE)
#undef R3D_SHAPE
    if (!done) fail(R3DGPU_EINVAL, "stereo: bad path kernel shape");
  }
  R3D_LAUNCH(sgm_path_accept_kernel, dim3(resident_grid(sgm_path_accept_kernel, sms, wave.pixels, kPathThreads)),
             dim3(kPathThreads), 0, s, dm, wave.jobs, wave.njobs, wave.pixels, info, rkeys);
  launched("sgm_path_accept_kernel");
}

// ---------------------------------------------------------------- ranged launches
namespace {

// Largest number of resident CTAs per SM any ranged pass kernel is launched
// with (the overflow has one slot per resident warp).
constexpr int kRangedMaxPerSm = 24;

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
                 n * static_cast<uint64_t>(seg.pixels), n * (pass_bytes(MODE, true, seg) + 8 * static_cast<uint64_t>(seg.pixels)));
  }
}

// The ranged passes' order: the long chains (rows, columns) before the
// diagonals of the same tile, so that a launch ends on short blocks.
constexpr int kRangedOrder[8] = {0, 7, 1, 4, 2, 3, 5, 6};

template <int K>
void launch_ranged_passes(const SgmMatch* dm, const SgmPathJob* jobs, const SgmPathSegment& g, const uint2* rec,
                          const uint8_t* cost, uint16_t* sum, uint8_t* terms, int64_t tstride, uint32_t* ovf,
                          int ovf_words, int sms, cudaStream_t s, const int* cancel, int* counters) {
  for (int q = 0; q < 8; ++q)
    if (g.blocks[kPasses[q].cls] <= 0) return;  // no pixels: every class has chains otherwise
  if (terms != nullptr) {
    // Byte terms: all eight directions in one launch.
    launch_ranged_pass<K, kTerm>(pass_set(g, kRangedOrder, kRangedTerms, counters), dm, jobs, g.count, rec, cost, sum,
                                 terms, tstride, ovf, ovf_words, sms, s, g, cancel);
    return;
  }
  for (int q = 0; q < 8; ++q) {
    const PassSet ps = pass_set(g, kRangedOrder + q, 1, counters + q);
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
                                       int sms, bool terms) {
  SgmPathBuffers b{};
  size_t o = 0;
  b.cost = o;
  o += align256(static_cast<size_t>(cells));
  // Eight byte-term arrays, or the u16 sums.
  b.sum = b.terms = o;
  b.term_stride = terms ? static_cast<int64_t>(align256(static_cast<size_t>(cells))) : 0;
  o += terms ? static_cast<size_t>(kRangedTerms) * static_cast<size_t>(b.term_stride)
             : align256(static_cast<size_t>(cells) * 2);
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
  // Words of a wide vector's buffer (none where every vector fits shared
  // memory), with the sentinels around it, for both item sizes.
  b.overflow_words = maxnum > RangedRing<8, kTerm>::kVecLabels ? maxnum / 2 + 2 * RangedRing<16, kTerm>::kPadWords + 2 : 0;
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
      sgm_path_ranged_buffers(wave.cells, wave.pixels, wave.keys, wave.rows, wave.maxnum, sms, wave.terms != 0);
  uint8_t* cost = wave.buffer + B.cost;
  uint16_t* sum = reinterpret_cast<uint16_t*>(wave.buffer + B.sum);
  uint8_t* terms = wave.terms != 0 ? wave.buffer + B.terms : nullptr;
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
      launch_ranged_passes<8>(dm, jobs, g, rec, cost, sum, terms, B.term_stride, ovf, B.overflow_words, sms, s,
                              wave.cancel, counters + 8 * q);
    else if (g.shape.k_ == 16)
      launch_ranged_passes<16>(dm, jobs, g, rec, cost, sum, terms, B.term_stride, ovf, B.overflow_words, sms, s,
                               wave.cancel, counters + 8 * q);
    else
      fail(R3DGPU_EINVAL, "stereo: bad ranged path kernel shape");
  }
  auto* wta = terms != nullptr ? sgm_path_ranged_wta_kernel<true> : sgm_path_ranged_wta_kernel<false>;
  R3D_LAUNCH(wta, dim3(resident_grid(wta, sms, wave.pixels, kPathThreads)), dim3(kPathThreads), 0, s, dm, wave.jobs,
             wave.njobs, wave.pixels, rec, cost, sum, terms, B.term_stride, rowshift, info, rkeys);
  launched("sgm_path_ranged_wta_kernel");
  if (wave.keys > 0) {  // matches with the diagonal left-right check
    R3D_LAUNCH(sgm_path_ranged_accept_kernel,
               dim3(resident_grid(sgm_path_ranged_accept_kernel, sms, wave.pixels, kPathThreads)), dim3(kPathThreads),
               0, s, dm, wave.jobs, wave.njobs, wave.pixels, rec, info, rkeys, rowshift);
    launched("sgm_path_ranged_accept_kernel");
  }
}

}  // namespace r3dgpu
