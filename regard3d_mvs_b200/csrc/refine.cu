// Patch-based depth refinement (r3dgpu_refine_depth_map) and its input images
// (r3dgpu_make_refinement_image), the reference's src/r3d/mvs/refinement.cpp.
//
// A first kernel lists the pixels to refine (a depth, the window inside the
// image); the refinement runs over that list, so that a sparse map costs what
// its depths cost: four neighbours of which one has a depth would keep a warp
// as long as four depths (1024 x 768 pixels, one in ten with a depth, float
// terms: 4.8 ms with four neighbours per warp, 1.1 from the list; all with a
// depth: 9.5 and 9.0).
//
// Four pixels per warp, 8 lanes each. The lanes of a pixel split into one
// group per view (two lanes each for 4 views); a lane warps, samples and
// normalises every second (or so) of its view's window samples (25 for the
// default 9 x 9 window at step 2, 49 for a 7 x 7 window at step 1, at most
// 225), and every sum of the NCC and of the Gauss-Newton terms is an
// xor-butterfly over the pixel's lanes. After a butterfly these hold the same
// bits (the partial sums meet in mirrored order, and IEEE addition commutes),
// so the per-pixel decisions — view selection, the damped Gauss-Newton loop
// with step shrinking, the acceptance test — are the same in all of them. The
// four pixels run in step: a pixel that is done idles until the last is.
//
// Four pixels per warp against one: the warp-wide set-up of a view's warp, the
// 3 x 3 solve and the butterflies, half of the instructions of a warp per
// pixel, serve four pixels at once (786,432 pixels of 49 samples in 4 views:
// 12.5 G warp instructions with one pixel per warp).
//
// The window terms compute in double precision as the reference does; with
// fp32 = 1 the Gauss-Newton terms (Jacobian, J^T J, J^T e: the bulk of the
// work) are float while the objective that decides which steps are taken
// (sampled values, window normalisation, NCC) and the 3 x 3 LDL^T solve stay
// double. Sums run in a different order than the reference's sequential loops,
// so results agree with a double-precision CPU restatement to rounding, not
// bit for bit.
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "common.cuh"
#include "geom.cuh"
#include "kernels.h"
#include "api_guard.h"
#include "matcher_internal.h"

namespace r3dgpu {
namespace {

constexpr int kMaxSamples = 225;  // refinement.cpp:21
constexpr int kMaxViews = 8;      // refinement.cpp:22
constexpr double kDiscontinuity = 0.05;
enum : int { kInput, kRefined, kUnconfirmed, kCounters, kListed = kCounters };  // kListed: slot 0 only
constexpr int kSlots = 128, kSlotStride = 4;  // copies of the counters (one address takes an addition at a time)
constexpr int kPixels = 4;                    // pixels per warp
constexpr int kLanes = 32 / kPixels;          // lanes per pixel (at least one per view)
constexpr int kRefineThreads = 128;
static_assert(kLanes >= kMaxViews, "a lane per view");

// A view's pixel as the kernels read it, 16 bytes: the intensity already in
// double (a sample has four, and a conversion runs at a quarter of the double
// rate), and the derivatives in float. (32 bytes with double derivatives made
// the double path wait on its loads.)
R3D_DEVICE void load_texel(const float4* p, double& v, float& gx, float& gy) {
  const float4 a = __ldg(p);
  memcpy(&v, &a, 8);
  gx = a.z;
  gy = a.w;
}

// A window sample: its pixel offset and offset / radius.
template <class T>
struct alignas(4 * sizeof(T)) Sample {
  T dx, dy, sx, sy;
};

// Plane-induced warp into a view (refinement.cpp:24-30): h = m (qx, qy, 1) + b w(q).
struct ViewGeo {
  double m[9];  // K_j R_j R_0^T K_0^-1, row-major
  double b[3];  // K_j R_j (C_0 - C_j)
  const float4* data;  // the view's texels
  int64_t stride;      // texels per row
  int width, height;
};

struct Params {
  int width, height;
  int radius, step, side, n;  // `side` samples per window row, n = side^2
  int iterations, num_views;
  double min_ncc, max_shift_px, min_gain, min_texture2n;
  int drop_unconfirmed;
};

template <class T>
R3D_DEVICE T shfl_xor_t(T v, int mask) {
  uint32_t w[sizeof(T) / 4];
  memcpy(w, &v, sizeof(T));
  for (int i = 0; i < static_cast<int>(sizeof(T) / 4); ++i) w[i] = r3dsimt::shfl_xor(w[i], mask);
  memcpy(&v, w, sizeof(T));
  return v;
}

// The value of lane `src` (every lane reads one source lane).
template <class T>
R3D_DEVICE T shfl_t(T v, int src) {
  uint32_t w[sizeof(T) / 4];
  memcpy(w, &v, sizeof(T));
  for (int i = 0; i < static_cast<int>(sizeof(T) / 4); ++i) w[i] = r3dsimt::shfl(w[i], src);
  memcpy(&v, w, sizeof(T));
  return v;
}

// Butterfly sums of K values over aligned groups of `to / from` lanes: masks
// from .. to / 2 (below a view's lane count: over its lanes; from there on: over
// the pixel's views). After them all lanes of a group hold the same bits: the
// partial sums meet in mirrored order and IEEE addition commutes.
template <class T, int K>
R3D_DEVICE void sums(T (&v)[K], int from, int to) {
  for (int m = from; m < to; m <<= 1) {
#pragma unroll
    for (int i = 0; i < K; ++i) v[i] += shfl_xor_t(v[i], m);
  }
}

template <class T>
R3D_DEVICE T pixel_sum(T v) {
  T a[1] = {v};
  sums(a, 1, kLanes);
  return a[0];
}

// Finite (neither infinite nor NaN): v - v is 0 exactly then, NaN otherwise.
R3D_DEVICE bool finite_d(double v) { return v - v == 0.0; }

using r3dsimt::fmadd;

// Smallest power of two >= m (m in 1..8): the number of lane groups.
R3D_DEVICE int groups_for(int m) { return m <= 1 ? 1 : (m <= 2 ? 2 : (m <= 4 ? 4 : 8)); }

// One view's terms at plane theta (refinement.cpp:46-152), computed by the
// `gsize` lanes of a group: lane `gl` of the group takes the window samples
// gl, gl + gsize, ... NCC of the warped window with the normalised base
// window, J^T J (xx xy xz yy yz zz) and J^T e of
// sum (n_q - n0_q)^2 in (w, a, b). `valid` is false if a sample leaves the
// image or the window has no texture. All lanes of the group return the same
// values; `active` false (a group without a view) returns zeros and valid.
//
// One pass: the lanes accumulate raw moments and one butterfly sums them.
// With v = (raw - mean) / |raw - mean| (sum v = 0, sum v^2 = 1),
// a = dv (1, sx, sy), d = a - mean(a) and p = sum v d, the reference's terms
// are ncc = sum raw n0 / |raw - mean| (n0 has zero mean),
// J^T J = (sum d d^T - p p^T) / |raw - mean|^2 and
// J^T e = (p ncc - sum a n0) / |raw - mean|. The objective moments are double
// (intensities shifted by `shift`, the base window's mean, to keep the
// variance well conditioned); the Jacobian moments are T. Products and sums of
// a sample are contracted (fmadd): a rounding less each, and a fifth of the
// instructions.
template <class T>
R3D_DEVICE void evaluate_group(const ViewGeo& g, bool active, double x, double y, const double* theta,
                               const Params& p, const Sample<T>* samples, const double* n0s, double shift, int gl,
                               int gsize, bool& valid, double& ncc_out, double* hh, double* gg) {
  double ob[3] = {0.0, 0.0, 0.0};
  T jm[15];
#pragma unroll
  for (int i = 0; i < 15; ++i) jm[i] = T(0);
  bool bad = false;
  if (active) {
    const T b0 = static_cast<T>(g.b[0]), b1 = static_cast<T>(g.b[1]), b2 = static_cast<T>(g.b[2]);
    const T m0 = static_cast<T>(g.m[0]), m1 = static_cast<T>(g.m[1]), m3 = static_cast<T>(g.m[3]),
            m4 = static_cast<T>(g.m[4]), m6 = static_cast<T>(g.m[6]), m7 = static_cast<T>(g.m[7]);
    const T max_x = static_cast<T>(g.width - 1), max_y = static_cast<T>(g.height - 1);
    const T th0 = static_cast<T>(theta[0]), th1 = static_cast<T>(theta[1]), th2 = static_cast<T>(theta[2]);
    // In float, pixel positions of a few thousand carry about 1e-4 px of
    // rounding. The float path therefore projects the window centre at the
    // current depth in double once and each sample as a small float offset:
    // (H + d).xy / (H + d).z = c + (d.xy - c d.z) / (H + d).z, c = H.xy / H.z.
    const bool rel = sizeof(T) == 4;
    double hz = 0.0;
    int ic0 = 0, ic1 = 0;
    T fc0 = 0, fc1 = 0, cf0 = 0, cf1 = 0, hzf = 0, ft0 = 0, ft1 = 0, hc0 = 0, hc1 = 0, hc2 = 0;
    if (rel) {
      const double H0 = row3(g.m, 0, x, y, 1.0) + g.b[0] * theta[0];
      const double H1 = row3(g.m, 1, x, y, 1.0) + g.b[1] * theta[0];
      hz = row3(g.m, 2, x, y, 1.0) + g.b[2] * theta[0];
      if (hz > 0.0) {
        const double c0 = H0 / hz, c1 = H1 / hz;
        const double f0 = floor(c0), f1 = floor(c1);
        if (fabs(f0) < 1e8 && fabs(f1) < 1e8) {
          ic0 = static_cast<int>(f0);
          ic1 = static_cast<int>(f1);
          fc0 = static_cast<T>(c0 - f0);
          fc1 = static_cast<T>(c1 - f1);
          cf0 = static_cast<T>(c0);
          cf1 = static_cast<T>(c1);
          hzf = static_cast<T>(hz);
          ft0 = static_cast<T>(f0);
          ft1 = static_cast<T>(f1);
        } else {
          hz = 0.0;
        }
      }
    }
    const bool offsets = rel && hz > 0.0;
    if (!offsets) {
      hc0 = static_cast<T>(row3(g.m, 0, x, y, 1.0));
      hc1 = static_cast<T>(row3(g.m, 1, x, y, 1.0));
      hc2 = static_cast<T>(row3(g.m, 2, x, y, 1.0));
    }
    for (int s = gl; s < p.n; s += gsize) {
      const Sample<T> q = samples[s];
      const T dx = q.dx, dy = q.dy, sx = q.sx, sy = q.sy;
      T inv_z, px, py, fx, fy;
      int ix, iy;
      if (offsets) {
        const T ws = fmadd(th1, sx, th2 * sy);  // w(q) - w at the window centre
        const T d0 = fmadd(b0, ws, fmadd(m0, dx, m1 * dy));
        const T d1 = fmadd(b1, ws, fmadd(m3, dx, m4 * dy));
        const T d2 = fmadd(b2, ws, fmadd(m6, dx, m7 * dy));
        const T h2 = hzf + d2;
        inv_z = T(1) / h2;
        const T q0 = fmadd(fmadd(-cf0, d2, d0), inv_z, fc0), q1 = fmadd(fmadd(-cf1, d2, d1), inv_z, fc1);
        const T fl0 = floor_small(static_cast<float>(q0), ic0, ix), fl1 = floor_small(static_cast<float>(q1), ic1, iy);
        fx = q0 - fl0;
        fy = q1 - fl1;
        // ix and iy as floats: exact wherever they are inside an image.
        px = (ft0 + fl0) + fx;
        py = (ft1 + fl1) + fy;
        // In front of the camera, px in [0, width - 1) and py in [0, height - 1), as below.
        if (!(h2 > T(0) && fabs(q0) < T(1e6) && fabs(q1) < T(1e6) && ix >= 0 && iy >= 0 && ix <= g.width - 2 &&
              iy <= g.height - 2)) {
          bad = true;
          break;
        }
      } else {
        const T wq = fmadd(th2, sy, fmadd(th1, sx, th0));
        const T h0 = fmadd(b0, wq, fmadd(m1, dy, fmadd(m0, dx, hc0)));
        const T h1 = fmadd(b1, wq, fmadd(m4, dy, fmadd(m3, dx, hc1)));
        const T h2 = fmadd(b2, wq, fmadd(m7, dy, fmadd(m6, dx, hc2)));
        if (!(h2 > T(0))) {
          bad = true;
          break;
        }
        inv_z = T(1) / h2;
        px = h0 * inv_z;
        py = h1 * inv_z;
        if (!(px >= T(0) && py >= T(0) && px < max_x && py < max_y)) {
          bad = true;
          break;
        }
        ix = static_cast<int>(px);
        iy = static_cast<int>(py);
        fx = px - static_cast<T>(ix);
        fy = py - static_cast<T>(iy);
      }
      const float4* r0 = g.data + static_cast<int64_t>(iy) * g.stride + ix;
      const float4* r1 = r0 + g.stride;
      double v00, v01, v10, v11;
      float x00, x01, x10, x11, y00, y01, y10, y11;
      load_texel(r0, v00, x00, y00);
      load_texel(r0 + 1, v01, x01, y01);
      load_texel(r1, v10, x10, y10);
      load_texel(r1 + 1, v11, x11, y11);
      const double fxd = fx, fyd = fy;
      const double ux = 1.0 - fxd, uy = 1.0 - fyd;
      const double raw = fmadd(uy, fmadd(ux, v00, fxd * v01), fyd * fmadd(ux, v10, fxd * v11)) - shift;
      const double n0 = n0s[s];
      ob[0] += raw;
      ob[1] = fmadd(raw, raw, ob[1]);
      ob[2] = fmadd(raw, n0, ob[2]);
      {
        const T ax = T(1) - fx, ay = T(1) - fy;
        const T tx00 = x00, tx01 = x01, tx10 = x10, tx11 = x11, ty00 = y00, ty01 = y01, ty10 = y10, ty11 = y11;
        const T gx = fmadd(ay, fmadd(ax, tx00, fx * tx01), fy * fmadd(ax, tx10, fx * tx11));
        const T gy = fmadd(ay, fmadd(ax, ty00, fx * ty01), fy * fmadd(ax, ty10, fx * ty11));
        const T dpx = fmadd(-px, b2, b0) * inv_z, dpy = fmadd(-py, b2, b1) * inv_z;
        const T dv = fmadd(gx, dpx, gy * dpy);
        const T a0 = dv, a1 = dv * sx, a2 = dv * sy;
        const T rf = static_cast<T>(raw), nf = static_cast<T>(n0);
        jm[0] += a0;
        jm[1] += a1;
        jm[2] += a2;
        jm[3] = fmadd(rf, a0, jm[3]);
        jm[4] = fmadd(rf, a1, jm[4]);
        jm[5] = fmadd(rf, a2, jm[5]);
        jm[6] = fmadd(a0, a0, jm[6]);
        jm[7] = fmadd(a0, a1, jm[7]);
        jm[8] = fmadd(a0, a2, jm[8]);
        jm[9] = fmadd(a1, a1, jm[9]);
        jm[10] = fmadd(a1, a2, jm[10]);
        jm[11] = fmadd(a2, a2, jm[11]);
        jm[12] = fmadd(nf, a0, jm[12]);
        jm[13] = fmadd(nf, a1, jm[13]);
        jm[14] = fmadd(nf, a2, jm[14]);
      }
    }
  }
  // The group is invalid if any of its lanes left the image.
  const uint32_t lane = r3dsimt::lane_id();
  const uint32_t gmask = (gsize == 32 ? 0xFFFFFFFFu : ((1u << gsize) - 1u) << (lane & ~static_cast<uint32_t>(gsize - 1)));
  const bool group_bad = (r3dsimt::ballot(bad) & gmask) != 0;
  sums(ob, 1, gsize);
  sums(jm, 1, gsize);
  for (int i = 0; i < 6; ++i) hh[i] = 0.0;
  for (int i = 0; i < 3; ++i) gg[i] = 0.0;
  ncc_out = 0.0;
  valid = true;
  if (!active) return;
  const double nd = p.n;
  const double mean = ob[0] / nd;  // of the shifted values
  const double norm2 = ob[1] - ob[0] * mean;
  if (group_bad || !(norm2 > 1e-6 * nd)) {
    valid = false;
    return;
  }
  const double inv_norm = 1.0 / sqrt(norm2);
  const double ncc = ob[2] * inv_norm;
  ncc_out = ncc;
  const T inv = static_cast<T>(inv_norm), n = static_cast<T>(p.n), meanf = static_cast<T>(mean);
  const T dm[3] = {jm[0] / n, jm[1] / n, jm[2] / n};
  const T pr[3] = {inv * (jm[3] - meanf * jm[0]), inv * (jm[4] - meanf * jm[1]), inv * (jm[5] - meanf * jm[2])};
  // sum d d^T = sum a a^T - dm (sum a)^T, then minus p p^T, times inv^2.
  const int ti[6] = {0, 0, 0, 1, 1, 2}, tj[6] = {0, 1, 2, 1, 2, 2};
#pragma unroll
  for (int e = 0; e < 6; ++e)
    hh[e] = static_cast<double>(inv * inv * ((jm[6 + e] - dm[ti[e]] * jm[tj[e]]) - pr[ti[e]] * pr[tj[e]]));
  const T nccf = static_cast<T>(ncc);
#pragma unroll
  for (int i = 0; i < 3; ++i) gg[i] = static_cast<double>(inv * (pr[i] * nccf - jm[12 + i]));
}

// refinement.cpp:155-165: pixels of motion in the view per unit of inverse depth.
R3D_DEVICE double centre_motion(const ViewGeo& g, double x, double y, double w) {
  const double h0 = row3(g.m, 0, x, y, 1.0) + g.b[0] * w;
  const double h1 = row3(g.m, 1, x, y, 1.0) + g.b[1] * w;
  const double h2 = row3(g.m, 2, x, y, 1.0) + g.b[2] * w;
  if (!(h2 > 0.0)) return 0.0;
  const double px = h0 / h2, py = h1 / h2;
  return hypot(g.b[0] - px * g.b[2], g.b[1] - py * g.b[2]) / h2;
}

// refinement.cpp:167-196: inverse-depth slope from the neighbours at +-1.
R3D_DEVICE double initial_slope(const float* depth, int w, int h, int x, int y, int ax, int ay) {
  const float z = depth[static_cast<int64_t>(y) * w + x];
  auto neighbour = [&](int k, double& wn) {
    const int nx = x + k * ax, ny = y + k * ay;
    if (nx < 0 || ny < 0 || nx >= w || ny >= h) return false;
    const float zn = depth[static_cast<int64_t>(ny) * w + nx];
    if (!(zn > 0.0F) || static_cast<double>(fabsf(zn - z)) > kDiscontinuity * static_cast<double>(fminf(z, zn)))
      return false;
    wn = 1.0 / zn;
    return true;
  };
  double wp = 0.0, wm = 0.0;
  const bool pl = neighbour(1, wp);
  const bool mi = neighbour(-1, wm);
  const double w0 = 1.0 / z;
  if (pl && mi) return 0.5 * (wp - wm);
  if (pl) return wp - w0;
  if (mi) return w0 - wm;
  return 0.0;
}

// delta = -(H (1 + 1e-6 on the diagonal) + 1e-12 I)^-1 g by LDL^T with
// symmetric diagonal pivoting (the largest remaining diagonal first).
R3D_DEVICE void solve_damped(const double* hh, const double* gg, double* delta) {
  double a[3][3] = {{hh[0], hh[1], hh[2]}, {hh[1], hh[3], hh[4]}, {hh[2], hh[4], hh[5]}};
  for (int i = 0; i < 3; ++i) a[i][i] = a[i][i] * (1.0 + 1e-6) + 1e-12;
  int perm[3] = {0, 1, 2};
  double l[3][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}}, d[3];
  for (int k = 0; k < 3; ++k) {
    int piv = k;
    for (int i = k + 1; i < 3; ++i)
      if (fabs(a[i][i]) > fabs(a[piv][piv])) piv = i;
    if (piv != k) {
      for (int j = 0; j < 3; ++j) {
        const double t = a[k][j];
        a[k][j] = a[piv][j];
        a[piv][j] = t;
      }
      for (int i = 0; i < 3; ++i) {
        const double t = a[i][k];
        a[i][k] = a[i][piv];
        a[i][piv] = t;
      }
      for (int j = 0; j < k; ++j) {
        const double t = l[k][j];
        l[k][j] = l[piv][j];
        l[piv][j] = t;
      }
      const int t = perm[k];
      perm[k] = perm[piv];
      perm[piv] = t;
    }
    d[k] = a[k][k];
    for (int i = k + 1; i < 3; ++i) l[i][k] = d[k] != 0.0 ? a[i][k] / d[k] : 0.0;
    for (int i = k + 1; i < 3; ++i)
      for (int j = k + 1; j <= i; ++j) {
        a[i][j] -= l[i][k] * d[k] * l[j][k];
        a[j][i] = a[i][j];
      }
  }
  double y[3];
  for (int i = 0; i < 3; ++i) {
    y[i] = gg[perm[i]];
    for (int j = 0; j < i; ++j) y[i] -= l[i][j] * y[j];
  }
  for (int i = 0; i < 3; ++i) y[i] = d[i] != 0.0 ? y[i] / d[i] : 0.0;
  for (int i = 2; i >= 0; --i)
    for (int j = i + 1; j < 3; ++j) y[i] -= l[j][i] * y[j];
  for (int i = 0; i < 3; ++i) delta[perm[i]] = -y[i];
}

// The pixels to refine, runs of kListRun pixels in the order their blocks come
// to it (a run's pixels in image order): those with a depth whose window lies
// inside the image, if there are views. Every pixel with a depth is counted
// and its confidence zeroed.
constexpr int kListThreads = 256, kListRun = 4 * kListThreads;
R3D_GLOBAL void R3D_LAUNCH_BOUNDS(kListThreads)
    list_kernel(const float* R3D_RESTRICT input, float* conf, int64_t stride, Params p, int64_t* R3D_RESTRICT list,
                unsigned long long* counters) {
  constexpr int kWarps = kListThreads / 32, kParts = kListRun / 32;
  R3D_DYNAMIC_SMEM(smem);
  int64_t* const start = reinterpret_cast<int64_t*>(smem);  // of the run's 32-pixel parts in the list
  const int lane = static_cast<int>(r3dsimt::lane_id()), warp = static_cast<int>(threadIdx.x >> 5);
  const int64_t total = static_cast<int64_t>(p.width) * p.height;
  const int64_t first = static_cast<int64_t>(blockIdx.x) * kListRun;
  unsigned long long* const slot = counters + (blockIdx.x % kSlots) * kSlotStride;
  uint32_t mine[kListRun / kListThreads];
#pragma unroll
  for (int k = 0; k < kListRun / kListThreads; ++k) {
    const int part = k * kWarps + warp;
    const int64_t pix = first + part * 32 + lane;
    const bool valid = pix < total && input[pix] > 0.0F;
    const int y = static_cast<int>(pix / p.width), x = static_cast<int>(pix - static_cast<int64_t>(y) * p.width);
    if (valid) conf[static_cast<int64_t>(y) * stride + x] = 0.0F;
    const uint32_t v = r3dsimt::ballot(valid);
    if (lane == 0 && v != 0) atomicAdd(slot + kInput, static_cast<unsigned long long>(r3dsimt::popc(v)));
    mine[k] = r3dsimt::ballot(valid && p.num_views > 0 && x >= p.radius && y >= p.radius && x < p.width - p.radius &&
                              y < p.height - p.radius);
    if (lane == 0) start[part] = r3dsimt::popc(mine[k]);
  }
  r3dsimt::syncthreads();
  if (threadIdx.x == 0) {
    int64_t n = 0;
    for (int i = 0; i < kParts; ++i) {
      const int64_t c = start[i];
      start[i] = n;
      n += c;
    }
    start[kParts] = n > 0 ? static_cast<int64_t>(atomicAdd(counters + kListed, static_cast<unsigned long long>(n))) : 0;
  }
  r3dsimt::syncthreads();
#pragma unroll
  for (int k = 0; k < kListRun / kListThreads; ++k) {
    const int part = k * kWarps + warp;
    if ((mine[k] >> lane) & 1u)
      list[start[kParts] + start[part] + r3dsimt::popc(mine[k] & ((1u << lane) - 1u))] = first + part * 32 + lane;
  }
}

// Dynamic shared memory: the window's p.n samples, then per pixel of the block
// its p.n normalised base window values.
template <class T>
R3D_GLOBAL void R3D_LAUNCH_BOUNDS_MIN(kRefineThreads, 4)
    refine_kernel(const float* R3D_RESTRICT input, float* depth, float* conf, int64_t stride,
                  const float* R3D_RESTRICT base, int64_t bstride, const ViewGeo* R3D_RESTRICT views, Params p,
                  const int64_t* R3D_RESTRICT list, unsigned long long* counters) {
  R3D_DYNAMIC_SMEM(smem);
  const int lane = static_cast<int>(r3dsimt::lane_id()), warp = static_cast<int>(threadIdx.x >> 5);
  const int sub = lane / kLanes, wl = lane % kLanes;  // the pixel of the warp, the lane of the pixel
  const bool lead = wl == 0;
  const int64_t listed = static_cast<int64_t>(counters[kListed]);  // complete: written by the launch before
  const int64_t first = ((static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * kPixels;
  if (first - warp * kPixels >= listed) return;  // whole block
  const int r = p.radius;
  Sample<T>* const samples = reinterpret_cast<Sample<T>*>(smem);
  for (int s = static_cast<int>(threadIdx.x); s < p.n; s += static_cast<int>(blockDim.x)) {
    const int ox = (s % p.side) * p.step - r, oy = (s / p.side) * p.step - r;
    samples[s] = Sample<T>{static_cast<T>(ox), static_cast<T>(oy), static_cast<T>(static_cast<double>(ox) / r),
                           static_cast<T>(static_cast<double>(oy) / r)};
  }
  r3dsimt::syncthreads();
  if (first >= listed) return;  // whole warp
  bool live = first + sub < listed;
  const int64_t pix = list[live ? first + sub : first];
  const int y = static_cast<int>(pix / p.width), x = static_cast<int>(pix - static_cast<int64_t>(y) * p.width);
  const float z0 = input[pix];
  const int64_t at = static_cast<int64_t>(y) * stride + x;
  unsigned long long* const slot = counters + (blockIdx.x % kSlots) * kSlotStride;
  auto count = [&](int counter, bool pred) {  // pixels of the warp with pred (one vote each)
    const uint32_t b = r3dsimt::ballot(pred && lead);
    if (lane == 0 && b != 0) atomicAdd(slot + counter, static_cast<unsigned long long>(r3dsimt::popc(b)));
  };

  // The normalised base window into the pixel's table.
  double* const n0s = reinterpret_cast<double*>(samples + p.n) + static_cast<size_t>(warp * kPixels + sub) * p.n;
  double sum = 0.0;
  for (int s = wl; s < p.n; s += kLanes) {
    const int dx = (s % p.side) * p.step - r, dy = (s / p.side) * p.step - r;
    const double v = live ? base[static_cast<int64_t>(y + dy) * bstride + 3 * (x + dx)] : 0.0;
    n0s[s] = v;
    sum += v;
  }
  const double mean = pixel_sum(sum) / p.n;
  double norm2 = 0.0;
  for (int s = wl; s < p.n; s += kLanes) {
    const double v = n0s[s] - mean;
    n0s[s] = v;
    norm2 += v * v;
  }
  norm2 = pixel_sum(norm2);
  live = live && !(norm2 < p.min_texture2n);
  const double inv_norm = 1.0 / sqrt(norm2);
  for (int s = wl; s < p.n; s += kLanes) n0s[s] *= inv_norm;
  r3dsimt::syncwarp();
  if (r3dsimt::ballot(live) == 0) return;

  const double w0 = 1.0 / z0;
  const double theta0[3] = {w0, live ? r * initial_slope(input, p.width, p.height, x, y, 1, 0) : 0.0,
                            live ? r * initial_slope(input, p.width, p.height, x, y, 0, 1) : 0.0};
  const double xd = x, yd = y;

  // The lane's view: gsize lanes each, the same for all pixels of the launch.
  const int gsize = kLanes / groups_for(p.num_views);
  const int my_t = wl / gsize, gl = wl % gsize;
  const ViewGeo& my_view = views[my_t < p.num_views ? my_t : 0];
  const uint32_t px_mask = (1u << kLanes) - 1u;

  // Local view selection at the initial plane; the selected views' terms there
  // are those of the first Gauss-Newton step.
  double ncc, hh_v[6], gg_v[3];
  bool use = live && my_t < p.num_views;  // the lane's view is used by its pixel
  int m = 0;
  double s0 = 0.0;
  {
    bool valid;
    evaluate_group<T>(my_view, use, xd, yd, theta0, p, samples, n0s, mean, gl, gsize, valid, ncc, hh_v, gg_v);
    use = use && valid && ncc >= p.min_ncc;
    const uint32_t ok = (r3dsimt::ballot(use) >> (sub * kLanes)) & px_mask;
    for (int j = 0; j < p.num_views; ++j) {
      const double nj = shfl_t(ncc, sub * kLanes + j * gsize);  // group j's value
      if ((ok >> (j * gsize)) & 1u) {
        ++m;
        s0 += nj;
      }
    }
  }
  const bool unconfirmed = live && m == 0 && p.drop_unconfirmed != 0;
  count(kUnconfirmed, unconfirmed);
  if (unconfirmed && lead) depth[at] = 0.0F;
  live = live && m > 0;
  if (r3dsimt::ballot(live) == 0) return;
  const int views_used = m > 0 ? m : 1;
  s0 /= views_used;
  if (live && lead) conf[at] = static_cast<float>(s0);
  double max_motion = use ? centre_motion(my_view, xd, yd, w0) : 0.0;
  for (int o = gsize; o < kLanes; o <<= 1) max_motion = fmax(max_motion, shfl_xor_t(max_motion, o));

  // Mean NCC and Gauss-Newton terms over the used views, from each lane's view's.
  auto total_terms = [&](double* hh, double* gg) {
    double tot[10] = {ncc, hh_v[0], hh_v[1], hh_v[2], hh_v[3], hh_v[4], hh_v[5], gg_v[0], gg_v[1], gg_v[2]};
    if (!use)
      for (int i = 0; i < 10; ++i) tot[i] = 0.0;
    sums(tot, gsize, kLanes);
    for (int i = 0; i < 6; ++i) hh[i] = tot[1 + i];
    for (int i = 0; i < 3; ++i) gg[i] = tot[7 + i];
    return tot[0] / views_used;
  };
  // The same at plane theta; -inf if a view drops out.
  auto evaluate = [&](const double* theta, bool active, double* hh, double* gg) {
    bool valid;
    evaluate_group<T>(my_view, active && use, xd, yd, theta, p, samples, n0s, mean, gl, gsize, valid, ncc, hh_v, gg_v);
    const bool dropped = ((r3dsimt::ballot(!valid) >> (sub * kLanes)) & px_mask) != 0;
    const double score = total_terms(hh, gg);
    return dropped ? -__builtin_huge_val() : score;
  };

  double hh[6], gg[3];
  double best[3] = {theta0[0], theta0[1], theta0[2]};
  double best_score = total_terms(hh, gg);
  live = live && finite_d(best_score);
  double scale = 1.0;
  bool stepping = live;
  for (int it = 0; it < p.iterations && r3dsimt::ballot(stepping) != 0; ++it) {
    double delta[3];
    solve_damped(hh, gg, delta);
    stepping = stepping && finite_d(delta[0]) && finite_d(delta[1]) && finite_d(delta[2]);
    // At most one pixel of motion per step at the window border.
    const double motion = max_motion * ((fabs(delta[0]) + fabs(delta[1])) + fabs(delta[2]));
    if (motion > 1.0)
      for (int i = 0; i < 3; ++i) delta[i] /= motion;
    for (int i = 0; i < 3; ++i) delta[i] *= scale;
    if (max_motion * ((fabs(delta[0]) + fabs(delta[1])) + fabs(delta[2])) < 1e-3) stepping = false;
    double h2[6], g2[3];
    const double cand[3] = {best[0] + delta[0], best[1] + delta[1], best[2] + delta[2]};
    const double score = evaluate(cand, stepping, h2, g2);
    if (stepping) {
      if (score > best_score) {
        for (int i = 0; i < 3; ++i) best[i] = cand[i];
        best_score = score;
        for (int i = 0; i < 6; ++i) hh[i] = h2[i];
        for (int i = 0; i < 3; ++i) gg[i] = g2[i];
        scale = 1.0;
      } else {
        scale *= 0.25;
      }
    }
  }
  const bool taken =
      live && best_score > s0 + p.min_gain && best[0] > 0.0 && max_motion * fabs(best[0] - w0) <= p.max_shift_px;
  count(kRefined, taken);
  if (taken && lead) {
    depth[at] = static_cast<float>(1.0 / best[0]);
    conf[at] = static_cast<float>(best_score);
  }
}

// ------------------------------------------------------------------ refinement images
// refinement.cpp:198-238: separable Gaussian, taps (normalised floats) from the host.
R3D_GLOBAL void blur_rows_kernel(const float* in, int64_t istride, int w, int h, const float* taps, int r,
                                 float* out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const float* row = in + static_cast<int64_t>(y) * istride;
  float acc = 0.0F;
  for (int i = -r; i <= r; ++i) {
    const int xx = x + i < 0 ? 0 : (x + i > w - 1 ? w - 1 : x + i);
    acc = __fadd_rn(acc, __fmul_rn(taps[i + r], row[xx]));
  }
  out[static_cast<int64_t>(y) * w + x] = acc;
}

R3D_GLOBAL void blur_cols_kernel(const float* in, int w, int h, const float* taps, int r, float* out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  float acc = 0.0F;
  for (int i = -r; i <= r; ++i) {
    const int yy = y + i < 0 ? 0 : (y + i > h - 1 ? h - 1 : y + i);
    acc = __fadd_rn(acc, __fmul_rn(taps[i + r], in[static_cast<int64_t>(yy) * w + x]));
  }
  out[static_cast<int64_t>(y) * w + x] = acc;
}

// refinement.cpp:249-266: intensity and central-difference derivatives.
R3D_GLOBAL void gradient_kernel(const float* gray, int64_t gstride, int w, int h, float* out, int64_t ostride) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const float* row = gray + static_cast<int64_t>(y) * gstride;
  const float* up = gray + static_cast<int64_t>(y > 0 ? y - 1 : 0) * gstride;
  const float* down = gray + static_cast<int64_t>(y < h - 1 ? y + 1 : h - 1) * gstride;
  const float sy = (y > 0 && y < h - 1) ? 0.5F : 1.0F;
  const int xl = x > 0 ? x - 1 : 0, xr = x < w - 1 ? x + 1 : w - 1;
  float* o = out + static_cast<int64_t>(y) * ostride + 3 * x;
  o[0] = row[x];
  o[1] = __fdiv_rn(__fsub_rn(row[xr], row[xl]), static_cast<float>(xr - xl > 1 ? xr - xl : 1));
  o[2] = __fmul_rn(__fsub_rn(down[x], up[x]), h > 1 ? sy : 0.0F);
}

// A view's 3-channel refinement image as texels.
R3D_GLOBAL void repack_kernel(const float* in, int64_t istride, int w, int h, float4* out) {
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
  if (x >= w || y >= h) return;
  const float* p = in + static_cast<int64_t>(y) * istride + 3 * x;
  const double v = p[0];
  float4 a;
  memcpy(&a, &v, 8);
  a.z = p[1];
  a.w = p[2];
  out[static_cast<int64_t>(y) * w + x] = a;
}

// ------------------------------------------------------------------ host side
struct Scratch {
  DeviceBuffer<unsigned long long> counters;
  DeviceBuffer<float> input, blur_tmp, blur_out, taps;
  DeviceBuffer<int64_t> list;  // the pixels to refine
  DeviceBuffer<ViewGeo> views;
  DeviceBuffer<float4> packed;  // the views' repacked images
};

Scratch& scratch() {
  thread_local Scratch s;
  s.counters.reserve(kSlots * kSlotStride);
  s.views.reserve(kMaxViews);
  return s;
}

// Row-major 3x3 products in the reference's left-to-right order.
void mat3(const double* a, const double* b, double* out) {
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) out[3 * i + j] = (a[3 * i] * b[j] + a[3 * i + 1] * b[3 + j]) + a[3 * i + 2] * b[6 + j];
}

// refinement.cpp:297-309.
ViewGeo view_geometry(const r3dgpu_pinhole_camera& c0, const r3dgpu_refinement_image& v) {
  const r3dgpu_pinhole_camera& cj = v.camera;
  const double kj[9] = {cj.intrinsics.fx, 0.0, cj.intrinsics.cx, 0.0, cj.intrinsics.fy, cj.intrinsics.cy,
                        0.0, 0.0, 1.0};
  double r0t[9];
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) r0t[3 * i + j] = c0.rotation[3 * j + i];
  double kr[9], krr[9];
  ViewGeo g{};
  mat3(kj, cj.rotation, kr);
  mat3(kr, r0t, krr);
  mat3(krr, c0.k_inv, g.m);
  const double dc[3] = {c0.center[0] - cj.center[0], c0.center[1] - cj.center[1], c0.center[2] - cj.center[2]};
  for (int i = 0; i < 3; ++i) g.b[i] = (kr[3 * i] * dc[0] + kr[3 * i + 1] * dc[1]) + kr[3 * i + 2] * dc[2];
  g.data = nullptr;  // set to the repacked image by the caller
  g.stride = cj.intrinsics.width;
  g.width = cj.intrinsics.width;
  g.height = cj.intrinsics.height;
  return g;
}

r3dgpu_refinement_options options_or_default(const r3dgpu_refinement_options* o) {
  r3dgpu_refinement_options out{};
  if (o != nullptr) return *o;
  r3dgpu_default_refinement_options(&out);
  return out;
}

template <class T>
void launch_refine(const float* input, float* depth, float* conf, int64_t stride, const float* base,
                   int64_t bstride, const ViewGeo* views, const Params& p, int64_t* list, unsigned long long* counters,
                   cudaStream_t s) {
  const int64_t total = static_cast<int64_t>(p.width) * p.height;
  R3D_LAUNCH(list_kernel, static_cast<unsigned>(ceil_div64(total, kListRun)), kListThreads,
             sizeof(int64_t) * (kListRun / 32 + 1), s, input, conf, stride, p, list, counters);
  launched("list_kernel");
  // Blocks for a full list; those past its end return at once.
  constexpr int per_block = kRefineThreads / 32 * kPixels;
  const size_t smem = (sizeof(Sample<T>) + sizeof(double) * per_block) * static_cast<size_t>(p.n);
  auto kernel = refine_kernel<T>;
  R3D_LAUNCH(kernel, static_cast<unsigned>(ceil_div64(total, per_block)), kRefineThreads, smem, s, input, depth, conf,
             stride, base, bstride, views, p, list, counters);
  launched(sizeof(T) == 8 ? "refine_kernel<f64>" : "refine_kernel<f32>");
}

void refine(float* depth, float* conf, int64_t stride, const r3dgpu_pinhole_camera& cam, int w, int h,
            const r3dgpu_refinement_image& base, const r3dgpu_refinement_image* views, int num_views,
            const r3dgpu_refinement_options& o, r3dgpu_refinement_stats* stats, cudaStream_t s) {
  if (o.radius < 1 || o.step < 1 || o.iterations < 0)
    fail(R3DGPU_EINVAL, "refinement: invalid window (radius " + std::to_string(o.radius) + ", step " +
                            std::to_string(o.step) + ") or iterations " + std::to_string(o.iterations));
  if (base.camera.intrinsics.width != w || base.camera.intrinsics.height != h || base.data == nullptr ||
      base.stride < 3LL * w)
    fail(R3DGPU_EINVAL, "refinement: base image does not match the depth map");
  if (w < 0 || h < 0 || (w > 0 && h > 0 && (depth == nullptr || conf == nullptr || stride < w)))
    fail(R3DGPU_EINVAL, "refinement: bad depth map");
  const int side = 2 * o.radius / o.step + 1;
  const int n = side * side;
  if (n > kMaxSamples)
    fail(R3DGPU_EINVAL, "refinement: window of " + std::to_string(n) + " samples (at most 225)");
  if (num_views < 0 || (num_views > 0 && views == nullptr)) fail(R3DGPU_EINVAL, "refinement: null views");
  const int nv = std::min(num_views, std::min(o.max_views, kMaxViews));
  Scratch& sc = scratch();
  ViewGeo geo[kMaxViews];
  for (int j = 0; j < nv; ++j) {
    const r3dgpu_refinement_image& v = views[j];
    if (v.data == nullptr || v.camera.intrinsics.width < 2 || v.camera.intrinsics.height < 2 ||
        v.stride < 3LL * v.camera.intrinsics.width)
      fail(R3DGPU_EINVAL, "refinement: view " + std::to_string(j) + " has no image");
    geo[j] = view_geometry(cam, v);
  }
  R3D_CUDA(cudaMemsetAsync(sc.counters.get(), 0, sizeof(unsigned long long) * kSlots * kSlotStride, s));
  if (w > 0 && h > 0) {
    // The views' images as texels.
    size_t total = 0;
    for (int j = 0; j < nv; ++j)
      total += static_cast<size_t>(views[j].camera.intrinsics.width) * views[j].camera.intrinsics.height;
    sc.packed.reserve(total > 0 ? total : 1);
    size_t off = 0;
    for (int j = 0; j < nv; ++j) {
      const int vw = views[j].camera.intrinsics.width, vh = views[j].camera.intrinsics.height;
      float4* dst = sc.packed.get() + off;
      const dim3 b(32, 8), g(static_cast<unsigned>(ceil_div(vw, 32)), static_cast<unsigned>(ceil_div(vh, 8)));
      R3D_LAUNCH(repack_kernel, g, b, 0, s, views[j].data, views[j].stride, vw, vh, dst);
      launched("repack_kernel");
      geo[j].data = dst;
      off += static_cast<size_t>(vw) * vh;
    }
    if (nv > 0)
      R3D_CUDA(cudaMemcpyAsync(sc.views.get(), geo, sizeof(ViewGeo) * nv, cudaMemcpyHostToDevice, s));
    sc.list.reserve(static_cast<size_t>(w) * h);
    sc.input.reserve(static_cast<size_t>(w) * h);
    R3D_CUDA(cudaMemcpy2DAsync(sc.input.get(), sizeof(float) * w, depth, sizeof(float) * stride, sizeof(float) * w,
                               h, cudaMemcpyDeviceToDevice, s));
    Params p{w, h, o.radius, o.step, side, n, o.iterations, nv, o.min_ncc, o.max_shift_px, o.min_gain,
             o.min_texture * o.min_texture * n, o.drop_unconfirmed};
    if (o.fp32)
      launch_refine<float>(sc.input.get(), depth, conf, stride, base.data, base.stride, sc.views.get(), p,
                           sc.list.get(), sc.counters.get(), s);
    else
      launch_refine<double>(sc.input.get(), depth, conf, stride, base.data, base.stride, sc.views.get(), p,
                            sc.list.get(), sc.counters.get(), s);
  }
  unsigned long long slots[kSlots * kSlotStride], c[kCounters] = {};
  R3D_CUDA(cudaMemcpyAsync(slots, sc.counters.get(), sizeof(slots), cudaMemcpyDeviceToHost, s));
  R3D_CUDA(cudaStreamSynchronize(s));
  for (int k = 0; k < kSlots; ++k)
    for (int i = 0; i < kCounters; ++i) c[i] += slots[k * kSlotStride + i];
  if (stats != nullptr) *stats = r3dgpu_refinement_stats{c[kInput], c[kRefined], c[kInput] - c[kRefined] - c[kUnconfirmed],
                                                         c[kUnconfirmed]};
}

void make_image(const float* gray, int64_t gstride, int w, int h, double sigma, float* out, int64_t ostride,
                cudaStream_t s) {
  if (w < 0 || h < 0 || (w > 0 && h > 0 && (gray == nullptr || out == nullptr || gstride < w || ostride < 3LL * w)))
    fail(R3DGPU_EINVAL, "refinement image: bad size, stride or pointer");
  if (w == 0 || h == 0) return;
  const dim3 b(32, 8), g(static_cast<unsigned>(ceil_div(w, 32)), static_cast<unsigned>(ceil_div(h, 8)));
  const float* src = gray;
  int64_t sstride = gstride;
  if (sigma > 0.0) {
    // refinement.cpp:200-210: taps up to 3 sigma, normalised in float.
    const int r = std::max(1, static_cast<int>(std::ceil(3.0 * sigma)));
    std::vector<float> k(static_cast<size_t>(2 * r + 1));
    float ksum = 0.0F;
    for (int i = -r; i <= r; ++i) {
      k[i + r] = static_cast<float>(std::exp(-0.5 * i * i / (sigma * sigma)));
      ksum += k[i + r];
    }
    for (float& v : k) v /= ksum;
    Scratch& sc = scratch();
    sc.taps.reserve(k.size());
    sc.blur_tmp.reserve(static_cast<size_t>(w) * h);
    sc.blur_out.reserve(static_cast<size_t>(w) * h);
    float* taps = sc.taps.get();
    float* tmp = sc.blur_tmp.get();
    float* blurred = sc.blur_out.get();
    R3D_CUDA(cudaMemcpyAsync(taps, k.data(), sizeof(float) * k.size(), cudaMemcpyHostToDevice, s));
    R3D_LAUNCH(blur_rows_kernel, g, b, 0, s, gray, gstride, w, h, taps, r, tmp);
    launched("blur_rows_kernel");
    R3D_LAUNCH(blur_cols_kernel, g, b, 0, s, tmp, w, h, taps, r, blurred);
    launched("blur_cols_kernel");
    src = blurred;
    sstride = w;
  }
  R3D_LAUNCH(gradient_kernel, g, b, 0, s, src, sstride, w, h, out, ostride);
  launched("gradient_kernel");
}

}  // namespace
}  // namespace r3dgpu

using namespace r3dgpu;

extern "C" {

void r3dgpu_default_refinement_options(r3dgpu_refinement_options* out) {
  if (out == nullptr) return;
  *out = r3dgpu_refinement_options{4, 2, 6, 4, 0.3, 2.0, 0.02, 1.0, 0.0, 1, 0};
}

r3dgpu_status r3dgpu_make_refinement_image(const float* gray, int64_t gray_stride, int32_t width, int32_t height,
                                           double blur_sigma, float* out, int64_t out_stride, void* stream) {
  return guard([&] {
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    make_image(gray, gray_stride, width, height, blur_sigma, out, out_stride, s);
    R3D_CUDA(cudaStreamSynchronize(s));
  });
}

r3dgpu_status r3dgpu_refine_depth_map(float* depth, float* confidence, int64_t stride,
                                      const r3dgpu_pinhole_camera* camera, int32_t width, int32_t height,
                                      const r3dgpu_refinement_image* base, const r3dgpu_refinement_image* views,
                                      int32_t num_views, const r3dgpu_refinement_options* options,
                                      r3dgpu_refinement_stats* stats, void* stream) {
  return guard([&] {
    if (camera == nullptr || base == nullptr) fail(R3DGPU_EINVAL, "refinement: null argument");
    refine(depth, confidence, stride, *camera, width, height, *base, views, num_views, options_or_default(options),
           stats, static_cast<cudaStream_t>(stream));
  });
}

r3dgpu_status r3dgpu_refine_depth_map_host(float* depth, float* confidence, int64_t stride,
                                           const r3dgpu_pinhole_camera* camera, int32_t width, int32_t height,
                                           const r3dgpu_refinement_image* base,
                                           const r3dgpu_refinement_image* views, int32_t num_views,
                                           const r3dgpu_refinement_options* options, r3dgpu_refinement_stats* stats) {
  return guard([&] {
    if (camera == nullptr || base == nullptr) fail(R3DGPU_EINVAL, "refinement: null argument");
    if (num_views < 0 || (num_views > 0 && views == nullptr)) fail(R3DGPU_EINVAL, "refinement: null views");
    if (width < 0 || height < 0 || stride < width || (width > 0 && height > 0 && (depth == nullptr || confidence == nullptr)))
      fail(R3DGPU_EINVAL, "refinement: bad depth map");
    const r3dgpu_refinement_options o = options_or_default(options);
    const int nv = std::min(num_views, std::min(o.max_views, kMaxViews));
    cudaStream_t s = nullptr;
    auto up = [](size_t n) { return (n + 255) & ~static_cast<size_t>(255); };
    auto image_bytes = [](const r3dgpu_refinement_image& v) {
      return sizeof(float) * 3 * static_cast<size_t>(v.camera.intrinsics.width) * v.camera.intrinsics.height;
    };
    const size_t px = static_cast<size_t>(width) * height;
    size_t bytes = 2 * up(4 * px) + up(image_bytes(*base));
    for (int j = 0; j < nv; ++j) bytes += up(image_bytes(views[j]));
    thread_local DeviceBuffer<unsigned char> io;
    io.reserve(bytes > 0 ? bytes : 1);
    unsigned char* p = io.get();
    auto take = [&](size_t n) {
      unsigned char* at = p;
      p += up(n);
      return at;
    };
    auto upload = [&](const r3dgpu_refinement_image& v) {
      r3dgpu_refinement_image d = v;
      const int vw = v.camera.intrinsics.width, vh = v.camera.intrinsics.height;
      float* dst = reinterpret_cast<float*>(take(image_bytes(v)));
      if (vw > 0 && vh > 0) {
        if (v.data == nullptr || v.stride < 3LL * vw) fail(R3DGPU_EINVAL, "refinement: image without data");
        R3D_CUDA(cudaMemcpy2DAsync(dst, sizeof(float) * 3 * vw, v.data, sizeof(float) * v.stride,
                                   sizeof(float) * 3 * vw, vh, cudaMemcpyHostToDevice, s));
      }
      d.data = dst;
      d.stride = 3LL * vw;
      return d;
    };
    float* dd = reinterpret_cast<float*>(take(4 * px));
    float* dc = reinterpret_cast<float*>(take(4 * px));
    if (px > 0) {
      R3D_CUDA(cudaMemcpy2DAsync(dd, 4 * static_cast<size_t>(width), depth, 4 * stride, 4 * static_cast<size_t>(width),
                                 height, cudaMemcpyHostToDevice, s));
      R3D_CUDA(cudaMemcpy2DAsync(dc, 4 * static_cast<size_t>(width), confidence, 4 * stride,
                                 4 * static_cast<size_t>(width), height, cudaMemcpyHostToDevice, s));
    }
    const r3dgpu_refinement_image dbase = upload(*base);
    std::vector<r3dgpu_refinement_image> dviews;
    for (int j = 0; j < nv; ++j) dviews.push_back(upload(views[j]));
    refine(dd, dc, width, *camera, width, height, dbase, dviews.data(), nv, o, stats, s);
    if (px > 0) {
      R3D_CUDA(cudaMemcpy2DAsync(depth, 4 * stride, dd, 4 * static_cast<size_t>(width), 4 * static_cast<size_t>(width),
                                 height, cudaMemcpyDeviceToHost, s));
      R3D_CUDA(cudaMemcpy2DAsync(confidence, 4 * stride, dc, 4 * static_cast<size_t>(width),
                                 4 * static_cast<size_t>(width), height, cudaMemcpyDeviceToHost, s));
    }
    R3D_CUDA(cudaStreamSynchronize(s));
  });
}

}  // extern "C"
