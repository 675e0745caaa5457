// Differentiable form: weighted-ray focal-plane image, the MSE between two
// images, and the adjoint of the image with respect to the 18 geometry and
// pointing parameters.
//
// Forward: one persistent kernel traces each ray in FP64 (ray_front and
// ray_image, on the trace's own shell records) and splats it with an 11 x 11
// Gaussian.  The splat is
// accumulated in 64-bit fixed point -- exact integer sums, so the image does
// not depend on the order of the atomics and repeats bit for bit -- first in
// a 64 x 64 shared-memory window about the image centre, which takes nearly
// every ray of a point source, and then in the global accumulator.  A warp
// splats its 32 rays together, one ray at a time, each lane adding four of
// the 121 taps, so the lanes of one atomic instruction never collide.
//
// Adjoint: the recorded rays are traced again with mxd::Dual scalars (FP64
// value, FP32 tangents of the four parameters that bend the ray's path: its
// shell's two tilts and the source's two offsets; the decenters shift the
// image); dL/dimage over the ray's 11 x 11 window gives dL/d(u, v, w), and the
// tangents of (u, v, w) turn that into six parameter contributions.  Nothing
// per ray is stored between the passes except the decision byte.  A block
// takes the rays of a tile whose decision byte says they reached the focal
// plane, in ascending order, and traces only those, so that its lanes do not
// idle through the rays that were lost.  Sums are deterministic: fixed tiles
// per block, fixed warp order, fixed block order, one final reduction.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <string>

#include "mx_context.h"
#include "mx_diff.cuh"

using mxd::Dual6;
namespace cg = cooperative_groups;

namespace {

constexpr int DBLOCK = 256;
constexpr int DWARPS = DBLOCK / 32;
constexpr int WIN = 64;                             // shared window side, pixels
constexpr int STAGE_W = 2 + 2 * mxd::TAPS;          // ic, jc, 11 y taps x w, 11 z taps
constexpr int STAGE_STRIDE = STAGE_W + 1;           // odd stride: conflict-free per-lane rows
constexpr int ADJ_STAGE = 9;                        // 6 contributions, shell, 2 pad
constexpr int ADJ_TILE = 8 * DBLOCK;                // rays a block sorts its hits out of at a time
constexpr int NP = MX_DIFF_NPARAM;

struct ImageGeom {
  int nx, ny;
  int wx0, wy0, wnx, wny;        // shared window: origin and extent in pixels
  int shift;                     // fixed-point right shift of each tap product
  int pad;
  double cy, cz, inv_pitch, cx_pix, cz_pix;
  float half_inv_s2;             // 1 / (2 sigma^2)
  float inv_s2;                  // 1 / sigma^2
  float knorm;                   // 1 / (sqrt(2 pi) sigma)
  float pad2;
  long long top_u, top_v;        // mx::dkey of nx + HALF and ny + HALF
};

// One shell at theta: its geometry in the trace's own record (so that the
// rays take the trace's conics, screens and struts), the source direction in
// the paraboloid's frame, and the reflection's constants.
struct DiffShell {
  MxShellDev h;
  double p1[3];                  // fwd[0] p0
  double wscale;                 // vignetting times the square of the effective-area correction
  float p1f[3], beta, delta;     // p1 and the optical constants at the ray energy
  float pad[19];                 // 992 bytes: the four shells start on distinct banks
};
static_assert(sizeof(DiffShell) % 128 == 96, "four shells on distinct bank offsets");

struct FwdArgs {
  DiffShell sh[4];
  double p0[3];
  double vig;
  int32_t ideal, area_uniform, weighted, pad;
  ImageGeom g;
};

// One shell's geometry with its tangents.
struct ShellTangents {
  mxd::Turn front[3], fwd[9];    // of the paraboloid
  mxd::Turn mid[9], off[3];
  mxd::Turn bwd[9], back[3];     // of the hyperboloid: bwd[1] and -to_osac[1] (its decenters taken apart)
  mxd::Dual p1[3];               // fwd p0, made on the device
  double corr;                   // effective-area correction per reflection
  double pad[4];                 // 688 bytes: lanes that load one field of different shells do not conflict
};
static_assert(sizeof(ShellTangents) == 688, "four shells on distinct bank offsets");

struct AdjArgs {
  FwdArgs f;
  ShellTangents d[4];
  mxd::Dual p0[3];
  mxd::Fresnel fr;
};

__host__ __device__ constexpr size_t align_up(size_t b) { return (b + 15) & ~(size_t) 15; }

// The pixel nearest to coordinate u, floor(u + 1/2), and the offset u - pixel
// rounded to float; false unless -(HALF + 1) < u < n + HALF (the ray's 11 x 11
// window misses the image).  Two FP64 additions; floor, comparisons and
// conversions on the integer and FP32 pipes.
__device__ __forceinline__ bool nearest_pixel(double u, long long top, int &ic, float &f) {
  const long long k = mx::dkey(u);
  if (!(k > mx::dkey(-(mxd::HALF + 1.0)) && k < top)) return false;
  const double s = MX_DADD(u, 0.5);
  const float t = mx::d2f_trunc(s);
  float c = floorf(t);                          // of s >= 0: truncation does not cross an integer
  if (s < 0.0 && c == t && mx::f2d_normal(t) != s) c -= 1.0f;
  ic = (int) c;
  f = mx::d2f_rn(MX_DADD(u, -mx::f2d_normal(c)));
  return true;
}

// Nearest pixel and the ray's offset from it on both axes; false when the
// ray's 11 x 11 window misses the image.
__device__ __forceinline__ bool splat_origin(const ImageGeom &g, double y, double z, int &ic, int &jc, float &fu,
                                             float &fv) {
  return nearest_pixel(mxd::pixel_coord(y, g.cy, g.inv_pitch, g.cx_pix), g.top_u, ic, fu) &&
         nearest_pixel(mxd::pixel_coord(z, g.cz, g.inv_pitch, g.cz_pix), g.top_v, jc, fv);
}

__device__ __forceinline__ float tap(const ImageGeom &g, int k, float f) {
  const float d = FSUB((float) (k - mxd::HALF), f);
  return FMUL(g.knorm, mxd::exp_neg(FMUL(FMUL(d, d), g.half_inv_s2)));
}

}  // namespace

// ------------------------------------------------------------ forward --
namespace {

constexpr int FWD_BLOCKS = 3;
constexpr int LIST = 64;                            // a warp's rays waiting: up to 31 left over and 32 new
constexpr int WSTRIDE = WIN + mxd::TAPS;            // window row stride, 11 mod 32 words: tap t of 121 falls on bank t

// A warp's list of rays that passed the aperture: index, shell, radius and
// the azimuth's sine and cosine.
struct RayList {
  double r[LIST];
  mx::F2 s[LIST], c[LIST];
  uint32_t i[LIST], shell[LIST];
};

// w 2^31 rounded to the nearest integer (ties to even), at most 2^32 - 1, on
// the integer pipe; 0 < w.
__device__ __forceinline__ uint32_t weight_fixed(double w) {
  const unsigned long long b = mx::dbits(w);
  const int sh = 1044 - (int) (b >> 52);              // w 2^31 = m 2^-sh
  if (sh < 21) return 0xffffffffu;                    // w >= 2
  if (sh > 54) return 0u;
  const unsigned long long m = (b & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
  const unsigned long long q = (m + ((1ull << (sh - 1)) - 1ull) + ((m >> sh) & 1ull)) >> sh;
  return q > 0xffffffffull ? 0xffffffffu : (uint32_t) q;
}

// The 121 taps as the lanes of a warp take them: tap t = lane + 32 j is
// (t % 11, t / 11).
struct TapLane {
  int ky[4], kz[4], at[4];
  __device__ __forceinline__ explicit TapLane(int lane) {
#pragma unroll
    for (int j = 0; j < 4; j++) {
      kz[j] = (lane + 32 * j) / mxd::TAPS;
      ky[j] = lane + 32 * j - mxd::TAPS * kz[j];
      at[j] = kz[j] * WSTRIDE + ky[j];
    }
  }
};

// The shared window as the splat tests it, in registers: its origin, the
// last origin of an 11 x 11 patch inside it (images
// are 16 pixels or more on a side) and the fixed-point shift, below 32 for every n_rays and sigma.
struct SplatWindow {
  int x0, y0;
  unsigned last_x, last_y, shift;
};

// Splat the warp's rays: lane L's ray is valid when valid is set; its window
// origin and taps go to a row of the stage, then the warp adds the 121 taps
// of each valid ray together.  The window's 64-bit
// sums are kept as two planes of 32-bit words, the carry added to the upper
// one: 9.5 cycles of the SM for a warp's update where a 64-bit shared atomic
// takes 13.6.
// Half the rays at a time (16 rows of the stage), a lane making the eleven
// taps of one ray along one axis.
__device__ __forceinline__ void splat_warp(const ImageGeom &g, const SplatWindow &W, bool valid, double y, double z, double w, uint32_t *stage,
                                           uint32_t *lo, uint32_t *hi, unsigned long long *acc, const TapLane &tl,
                                           int lane) {
  int ic = 0, jc = 0;
  float fu = 0.f, fv = 0.f;
  if (valid) valid = mx::is_pos(w) && splat_origin(g, y, z, ic, jc, fu, fv);
  const uint32_t wq = valid ? weight_fixed(w) : 0u;
  const unsigned vm = __ballot_sync(0xffffffffu, valid);
#pragma unroll 1
  for (int half = 0; half < 32; half += 16) {
  {
    const int src = half + (lane & 15);
    const float f0 = __shfl_sync(0xffffffffu, fu, src), f1 = __shfl_sync(0xffffffffu, fv, src);
    const int c = __shfl_sync(0xffffffffu, ic, src), r = __shfl_sync(0xffffffffu, jc, src);
    const uint32_t ww = __shfl_sync(0xffffffffu, wq, src);
    if ((vm >> src) & 1u) {
      uint32_t *row = stage + (lane & 15) * STAGE_STRIDE;
      const bool second = lane >= 16;
      const float f = second ? f1 : f0;
      row[second] = (uint32_t) (second ? r : c);
      row += second ? 2 + mxd::TAPS : 2;
#pragma unroll 1
      for (int k = 0; k < mxd::TAPS; k++) {
        const uint32_t t = __float2uint_rn(FMUL(tap(g, k, f), 2147483648.0f));   // K 2^31
        row[k] = second ? t : __umulhi(ww, t);                                   // w K 2^30
      }
    }
  }
  __syncwarp();
  for (unsigned hm = (vm >> half) & 0xffffu; hm; hm &= hm - 1) {
    const uint32_t *row = stage + (__ffs(hm) - 1) * STAGE_STRIDE;
    const int c0 = (int) row[0] - mxd::HALF, r0 = (int) row[1] - mxd::HALF;
    const int wc0 = c0 - W.x0, wr0 = r0 - W.y0;
    if ((unsigned) wc0 <= W.last_x && (unsigned) wr0 <= W.last_y) {   // all 121 in the window
      const int at = wr0 * WSTRIDE + wc0;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        if (j < 3 || lane < mxd::TAPS * mxd::TAPS - 96) {
          const unsigned long long c = (unsigned long long) row[2 + tl.ky[j]] * row[2 + mxd::TAPS + tl.kz[j]];
          const int k = at + tl.at[j];
          const uint32_t cl = __funnelshift_r((uint32_t) c, (uint32_t) (c >> 32), W.shift), old = atomicAdd(lo + k, cl);
          atomicAdd(hi + k, ((uint32_t) (c >> 32) >> W.shift) + (old + cl < cl ? 1u : 0u));
        }
      }
    } else {
#pragma unroll 1
      for (int t = lane; t < mxd::TAPS * mxd::TAPS; t += 32) {
        const int kz = t / mxd::TAPS, ky = t - mxd::TAPS * kz;
        const int col = c0 + ky, rr = r0 + kz;
        if ((unsigned) col >= (unsigned) g.nx || (unsigned) rr >= (unsigned) g.ny) continue;
        const unsigned long long c = ((unsigned long long) row[2 + ky] * row[2 + mxd::TAPS + kz]) >> g.shift;
        const unsigned wc = (unsigned) (col - g.wx0), wr = (unsigned) (rr - g.wy0);
        if (wc < (unsigned) g.wnx && wr < (unsigned) g.wny) {
          const int k = (int) wr * WSTRIDE + (int) wc;
          const uint32_t cl = (uint32_t) c, old = atomicAdd(lo + k, cl);
          atomicAdd(hi + k, (uint32_t) (c >> 32) + (old + cl < cl ? 1u : 0u));
        } else if (c)
          atomicAdd(acc + (size_t) rr * g.nx + col, c);
      }
    }
  }
  __syncwarp();
  }
}

// Part 1 of a ray: its point on the aperture (the shell pick, radius and
// azimuth the mirror stage draws for the photon of that tag, mirror_front,
// with the vignetting draw consumed but turned into a weight), and unless it
// is replayed the pre-collimator struts and the float screen for rays that
// certainly miss the paraboloid.  False for a ray that ends here.
__device__ __forceinline__ bool ray_front(const FwdArgs &A, const MxTables *T, uint64_t seed, uint32_t tag, bool replay,
                                          int &si, double &radius, mx::F2 &s, mx::F2 &c) {
  mx::Rng rng;
  rng.U = nullptr; rng.N = nullptr; rng.seed = seed; rng.n = 0; rng.i = 0; rng.tag = tag; rng.overrun = false;
  rng.window(MX_U_MIRROR, 12, MX_N_MIRROR, 2);
  if (!A.ideal) rng.skip_uniform();
  si = -1;
  for (int guard = 0; guard < 64 && si < 0; guard++) {
    const double r = rng.uniform();
    if (rng.overrun) return false;
    for (int i = 0; i < 4; i++)
      if (mx::lt_pos(r, A.sh[i].h.area_fraction)) { si = i; break; }
  }
  if (si < 0) return false;
  const MxShellDev &h = A.sh[si].h;
  if (A.area_uniform) {
    const double r0 = h.min_radius, r1 = h.max_radius;
    radius = mx::sqrt_fast(r0 * r0 + (r1 * r1 - r0 * r0) * rng.uniform());
  } else
    radius = fma(h.dr, rng.uniform(), h.min_radius);
  unsigned long long theta;
  for (int guard = 0;; guard++) {
    theta = rng.uniform_fixed();
    if (rng.overrun || guard >= 64) return false;
    if (h.shutter & (1u << (unsigned) (theta >> 62))) break;
  }
  mx::df_turn_sincos(theta, true, s, c);   // of the angle 2 pi (u - 1/8)
  if (replay) return true;
  const float rf = mx::d2f_trunc(radius), yf = rf * s.h, zf = rf * c.h;
  if (T->use_struts) {
    const float pxf = mx::d2f_trunc(A.p0[0]), pyf = mx::d2f_trunc(A.p0[1]), pzf = mx::d2f_trunc(A.p0[2]);
    int blocked = mx::struts_screen(*T, 0, h.frontf, yf - h.osac0f[1], zf - h.osac0f[2], pxf, pyf, pzf);
    if (blocked < 0)
      blocked = mx::struts_block_exact(*T, 0, mx::mk(h.front_position, radius * mx::df_join(s) - h.to_osac[0][1],
                                                    radius * mx::df_join(c) - h.to_osac[0][2]),
                                       mx::mk(A.p0[0], A.p0[1], A.p0[2])) ? 1 : 0;
    if (blocked) return false;
  }
  const double *f = h.fwd[0];
  const float f1 = mx::d2f_trunc(f[1]), f2 = mx::d2f_trunc(f[2]), f4 = mx::d2f_trunc(f[4]), f5 = mx::d2f_trunc(f[5]);
  const float f7 = mx::d2f_trunc(f[7]), f8 = mx::d2f_trunc(f[8]);
  return !mx::paraboloid_missed(h, fmaf(f2, zf, fmaf(f1, yf, h.front_fwdf)),
                                fmaf(f5, zf, fmaf(f4, yf, mx::d2f_trunc(h.front_fwd[1]))),
                                fmaf(f8, zf, fmaf(f7, yf, mx::d2f_trunc(h.front_fwd[2]))), A.sh[si].p1f[0], A.sh[si].p1f[1],
                                A.sh[si].p1f[2]);
}

static_assert(mxd::RAY_ROOT_P == 2 && mxd::RAY_ROOT_H == 4, "optic o's root is bit o + 1 of the decision byte");
// Part 2: through both mirrors to the focal plane x = 0.  root holds the
// recorded conic roots (RAY_ROOT_* bits) of a replayed ray, and receives
// those taken otherwise.
__device__ __forceinline__ bool ray_image(const FwdArgs &A, const MxTables &T, int si, double ry, double rz, bool replay,
                                          int &root, double &y, double &z, double &w) {
  const DiffShell &S = A.sh[si];
  const MxShellDev &h = S.h;
  // fwd (x + to) with x + to = (front + to[0], ry, rz): (ry - to[1]) + to[1]
  // is ry to within an ulp of to[1]
  const double *f = h.fwd[0];
  mx::D3 x = mx::mk(fma(f[2], rz, fma(f[1], ry, h.front_fwd[0])), fma(f[5], rz, fma(f[4], ry, h.front_fwd[1])),
                    fma(f[8], rz, fma(f[7], ry, h.front_fwd[2])));
  mx::D3 p = mx::mk(S.p1[0], S.p1[1], S.p1[2]);
  mx::F2 num{1.0f, 0.0f}, den{1.0f, 0.0f};
  int taken = 0;
#pragma unroll 1
  for (int o = 0; o < 2; o++) {   // one copy of the code: the warps of a block are at different places in it
    mx::D3 n;
    const int r = mxd::conic_root(h, o, x, p, n, replay ? (root >> (o + 1)) & 1 : -1);
    if (r < 0) return false;
    taken |= r << (o + 1);
    const double pdn = mx::dot(p, n);
    if (A.weighted) {
      mx::F2 a, b;
      mx::reflectivity_df(mx::split(fabs(pdn)), S.beta, S.delta, a, b);
      num = mx::df_mul(num, a);
      den = mx::df_mul(den, b);
    }
    p = mxd::reflected(p, n, pdn);
    if (o == 0) {
      if (!replay && T.use_struts && mx::cap_struts_block(T, h, x, p)) return false;
      const double *M = h.mid, *c = h.mid_off;
      p = mx::mat_mul(M, p);
      x = mx::mk(fma(M[0], x.x, fma(M[1], x.y, fma(M[2], x.z, c[0]))), fma(M[3], x.x, fma(M[4], x.y, fma(M[5], x.z, c[1]))),
                 fma(M[6], x.x, fma(M[7], x.y, fma(M[8], x.z, c[2]))));
    }
  }
  w = A.weighted ? mx::f2_double(mx::df_div(num, den)) * S.wscale : A.vig;   // NaN stays NaN, which df_join does not keep
  p = mx::mat_mul(h.bwd[1], p);
  x = mx::mat_mul(h.bwd[1], x);
  x = x - mx::mk(h.to_osac[1][0], h.to_osac[1][1], h.to_osac[1][2]);
  if (!replay && T.use_struts && mx::struts_block(T, 2, x, p)) return false;
  const double t = -x.x * mx::rcp_fast(p.x);
  y = fma(t, p.y, x.y);
  z = fma(t, p.z, x.z);
  root = taken;
  return true;
}

// SPLAT: accumulate the image; otherwise write each ray's y, z, w.
// MOMENTS: part[block][4], the block's sum w, sum w y, sum w z and hits.
//
// A warp takes 32 rays at a time through the aperture, keeps those that go on
// in a list of its own and traces 32 of the list together: half the rays miss
// the paraboloid, and traced where they stood they left 24 lanes of a warp
// busy on average and the FP64 work of a whole ray to every warp.  With the
// Newton intersections the FP64 instructions fall from 8.3 to 2.6 million per
// 1e6 rays: 697 -> 315 us.  The warps of a block are at different places of the
// kernel, so its length counts: with one copy of the code for both optics and
// for all taps (a third of the issue slots waited for instructions before)
// 255 us, FP64 pipe 58 % and issue 50 % busy.  Three blocks per SM (68
// registers, 72 with the moments); two took 3.38 ms for a gradient step over
// 4e6 rays where three took 3.05.
template <bool SPLAT, bool MOMENTS>
__global__ void __launch_bounds__(DBLOCK, FWD_BLOCKS) diff_forward_kernel(const __grid_constant__ FwdArgs args, const __grid_constant__ MxTables T,
                                                               uint64_t n, uint64_t seed, uint8_t *codes, int mode,
                                                               unsigned long long *acc, double *part, double *yzw) {
  extern __shared__ __align__(16) unsigned char smem[];
  FwdArgs &A = *reinterpret_cast<FwdArgs *>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  RayList &list = reinterpret_cast<RayList *>(smem + align_up(sizeof(FwdArgs)))[warp];
  uint32_t *lo = reinterpret_cast<uint32_t *>(smem + align_up(sizeof(FwdArgs)) + DWARPS * sizeof(RayList));
  uint32_t *hi = lo + WIN * WSTRIDE;
  uint32_t *stage = hi + WIN * WSTRIDE + warp * 16 * STAGE_STRIDE;   // SPLAT only, as lo and hi
  {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(&args);
    uint32_t *dst = reinterpret_cast<uint32_t *>(smem);
    for (int k = threadIdx.x; k < (int) (sizeof(FwdArgs) / 4); k += DBLOCK) dst[k] = src[k];
    if (SPLAT)
      for (int k = threadIdx.x; k < 2 * WIN * WSTRIDE; k += DBLOCK) lo[k] = 0u;
  }
  __syncthreads();
  const bool replay = mode == MX_DIFF_REPLAY;
  const TapLane tl(lane);
  const SplatWindow W{args.g.wx0, args.g.wy0, (unsigned) (args.g.wnx - mxd::TAPS), (unsigned) (args.g.wny - mxd::TAPS),
                      (unsigned) args.g.shift};
  double sw = 0.0, swy = 0.0, swz = 0.0;
  uint32_t hits = 0;
  const uint64_t step = (uint64_t) gridDim.x * DWARPS * 32;
  uint64_t base = ((uint64_t) blockIdx.x * DWARPS + warp) * 32;
  int have = 0;
  while (base < n || have > 0) {
    if (base < n) {
      const uint64_t i = base + lane;
      base += step;
      int si = 0;
      double radius = 0.0;
      mx::F2 s{0.f, 0.f}, c{0.f, 0.f};
      bool on = i < n;
      if (on && replay) on = (codes[i] & mxd::RAY_HIT) != 0;
      if (on) on = ray_front(A, &T, seed, (uint32_t) i, replay, si, radius, s, c);
      if (i < n && !on) {
        if (mode == MX_DIFF_RECORD) codes[i] = 0;
        if (!SPLAT) {
          yzw[i] = yzw[n + i] = __longlong_as_double(0x7ff8000000000000ll);
          yzw[2 * n + i] = 0.0;
        }
      }
      const unsigned m = __ballot_sync(0xffffffffu, on);
      if (on) {
        const int k = have + __popc(m & ((1u << lane) - 1u));
        list.r[k] = radius; list.s[k] = s; list.c[k] = c;
        list.i[k] = (uint32_t) i; list.shell[k] = (uint32_t) si;
      }
      have += __popc(m);
      __syncwarp();
      if (have < 32 && base < n) continue;
    }
    const int take = have < 32 ? have : 32;
    have -= take;
    bool hit = false;
    double y = 0.0, z = 0.0, w = 0.0;
    if (lane < take) {
      const int k = have + lane, si = (int) list.shell[k];
      const uint64_t i = list.i[k];
      const double radius = list.r[k], ry = radius * mx::df_join(list.s[k]), rz = radius * mx::df_join(list.c[k]);
      int root = replay ? codes[i] : 0;
      hit = ray_image(A, T, si, ry, rz, replay, root, y, z, w);
      if (mode == MX_DIFF_RECORD) codes[i] = hit ? (uint8_t) (mxd::RAY_HIT | root) : (uint8_t) 0;
      if (MOMENTS && hit) { sw += w; swy += w * y; swz += w * z; hits++; }
      if (!SPLAT) {
        yzw[i] = hit ? y : __longlong_as_double(0x7ff8000000000000ll);
        yzw[n + i] = hit ? z : __longlong_as_double(0x7ff8000000000000ll);
        yzw[2 * n + i] = hit ? w : 0.0;
      }
    }
    __syncwarp();   // the list's entries are read before they are written again
    if (SPLAT) splat_warp(A.g, W, hit, y, z, w, stage, lo, hi, acc, tl, lane);
  }
  __shared__ double red[4 * DWARPS];
  if (MOMENTS) {   // block partial moments, fixed order
    double nh = (double) hits;
    for (int o = 16; o > 0; o >>= 1) {
      sw += __shfl_down_sync(0xffffffffu, sw, o);
      swy += __shfl_down_sync(0xffffffffu, swy, o);
      swz += __shfl_down_sync(0xffffffffu, swz, o);
      nh += __shfl_down_sync(0xffffffffu, nh, o);
    }
    if (lane == 0) { red[4 * warp] = sw; red[4 * warp + 1] = swy; red[4 * warp + 2] = swz; red[4 * warp + 3] = nh; }
  }
  __syncthreads();
  if (SPLAT) {
    for (int k = threadIdx.x; k < A.g.wnx * A.g.wny; k += DBLOCK) {
      const int r = k / A.g.wnx, c = k - r * A.g.wnx;
      const unsigned long long v = ((unsigned long long) hi[r * WSTRIDE + c] << 32) | lo[r * WSTRIDE + c];
      if (v) atomicAdd(acc + (size_t) (A.g.wy0 + r) * A.g.nx + A.g.wx0 + c, v);
    }
  }
  if (MOMENTS && threadIdx.x < 4) {
    double s = 0.0;
    for (int k = 0; k < DWARPS; k++) s += red[4 * k + threadIdx.x];
    part[4 * blockIdx.x + threadIdx.x] = s;
  }
}

// image = acc 2^(shift - 61) / n_rays
__global__ void diff_image_kernel(const unsigned long long *acc, size_t npix, double scale, double *image) {
  for (size_t k = (size_t) blockIdx.x * blockDim.x + threadIdx.x; k < npix; k += (size_t) gridDim.x * blockDim.x)
    image[k] = (double) acc[k] * scale;
}

// out[v] = scale * sum over b of part[b * nv + v]: warp v, its lanes' strided
// sums added in a tree (a fixed order).  7 us for the 18 sums of a gradient; one
// thread a value waited for one load after the other, 39 us.
__global__ void __launch_bounds__(32 * NP) diff_sum_kernel(const double *part, int nblocks, int nv, double scale,
                                                           double *out) {
  const int v = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (v >= nv) return;
  double s = 0.0;
#pragma unroll 4
  for (int b = lane; b < nblocks; b += 32) s += part[(size_t) b * nv + v];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (lane == 0) out[v] = s * scale;
}

// loss = mean (image - target)^2 and, optionally, its gradient.  One cluster
// of blocks: each sums its part in a fixed order, and the first adds theirs
// from distributed shared memory, in the order of their ranks.  256 x 256
// pixels: 14 us; one block alone took 81 us, waiting for its loads.
constexpr int MSE_BLOCKS = 8, MSE_THREADS = 1024;
__global__ void __cluster_dims__(MSE_BLOCKS, 1, 1) __launch_bounds__(MSE_THREADS)
    diff_mse_kernel(const double *image, const double *target, size_t npix, double inv, double *dl, double *loss) {
  __shared__ double red[MSE_THREADS / 32];
  __shared__ double total;
  double s = 0.0;
  const double inv2 = 2.0 * inv;
#pragma unroll 4
  for (size_t k = (size_t) blockIdx.x * MSE_THREADS + threadIdx.x; k < npix; k += (size_t) MSE_BLOCKS * MSE_THREADS) {
    const double r = image[k] - target[k];
    s += r * r;
    if (dl) dl[k] = r * inv2;
  }
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = red[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) total = s;
  }
  cg::cluster_group cluster = cg::this_cluster();
  cluster.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    double t = 0.0;
    for (int b = 0; b < MSE_BLOCKS; b++) t += *cluster.map_shared_rank(&total, b);
    *loss = t * inv;
  }
  cluster.sync();   // every block's shared memory stays until it is read
}

}  // namespace

// ------------------------------------------------------------ adjoint --
namespace {

// dl/dimage at pixel (row, col): from the shared window, else from global
// memory, 0 outside the image.
__device__ __forceinline__ float resid_at(const ImageGeom &g, const float *rw, const double *dl, int row, int col) {
  const unsigned wc = (unsigned) (col - g.wx0), wr = (unsigned) (row - g.wy0);
  if (wc < (unsigned) g.wnx && wr < (unsigned) g.wny) return rw[wr * (WIN + 1) + wc];
  if ((unsigned) col < (unsigned) g.nx && (unsigned) row < (unsigned) g.ny)
    return (float) __ldg(dl + (size_t) row * g.nx + col);
  return 0.f;
}

// A recorded ray again, from the aperture to the focal plane x = 0, with
// tangents.
__device__ __forceinline__ bool ray_tangents(const AdjArgs &A, int si, double ry, double rz, int root, mxd::Dual &y,
                                             mxd::Dual &z, float &w, float (&wd)[mxd::NT]) {
  const ShellTangents &S = A.d[si];
  const MxShellDev &h = A.f.sh[si].h;
  mxd::V3 x = {mxd::turned(S.front[0], S.fwd[1], S.fwd[2], ry, rz), mxd::turned(S.front[1], S.fwd[4], S.fwd[5], ry, rz),
               mxd::turned(S.front[2], S.fwd[7], S.fwd[8], ry, rz)};
  mxd::V3 p = {S.p1[0], S.p1[1], S.p1[2]};
  mx::F2 w1{1.0f, 0.0f}, corr{1.0f, 0.0f};
  if (A.f.weighted) corr = mx::split(S.corr);
#pragma unroll 1
  for (int o = 0; o < 2; o++) {   // one copy of the code, as in ray_image
    mxd::V3 n;
    if (!mxd::conic_tangents(h, o, x, p, n, (root >> (o + 1)) & 1)) return false;
    const mxd::Dual pdn = mxd::dotp(p, n);
    mx::F2 wo{1.0f, 0.0f};
    float slope = 0.0f;
    if (A.f.weighted) {
      mx::F2 r;
      mxd::fresnel_slope(A.fr, mx::split(fabs(pdn.v)), r, slope);
      wo = mx::df_mul(r, corr);
      slope = mxd::tof(S.corr) * (mx::neg_bit(pdn.v) ? -slope : slope);
    }
    if (o == 0) {
      w1 = wo;
#pragma unroll
      for (int k = 0; k < mxd::NT; k++) wd[k] = slope * pdn.d[k];
    } else {
      const float w1f = mxd::tof(w1), w2f = mxd::tof(wo);
#pragma unroll
      for (int k = 0; k < mxd::NT; k++) wd[k] = w1f * (slope * pdn.d[k]) + w2f * wd[k];
      w = mx::df_mul(w1, wo).h;
    }
    const mxd::Dual q = 2.0 * pdn;
    p = {p.x - q * n.x, p.y - q * n.y, p.z - q * n.z};
    // into the hyperboloid's frame, then back to the MARX frame
    const mxd::Turn *m = o ? S.bwd : S.mid, *c = o ? S.back : S.off;
    p = mxd::matv(m, p);
    x = mxd::matv(m, x);
    x = {x.x + c[0], x.y + c[1], x.z + c[2]};
  }
  const mxd::Dual t = (0.0 - x.x) * mxd::drcp(p.x);
  y = x.y + t * p.y;
  z = x.z + t * p.z;
  return true;
}

// part[block][NP] = sum over the block's rays of dl/dimage . d(image)/dtheta
// (before the 1/n_rays factor).
//
// Per 1e6 rays: 500 -> 305 us with 3.1 instead of 5.9 million FP64 instructions
// (the rest are the tangents' FP32 steps and the window sums).  What went: the
// library's roots and divisions, the decenters' tangents, which are constants,
// the Fresnel chain in six directions (one slope, its values in double-float),
// the root that is not followed.  305 -> 279 us with one copy of the code for
// both optics and for the window's rows (a tenth of the issue slots waited for
// instructions): FP64 pipe 68 %, issue 42 %.  Two blocks per SM (128
// registers): three of 80 spill and took 2.40 instead of 2.35 ms for a gradient
// step over 4e6 rays.
__global__ void __launch_bounds__(DBLOCK, 2) diff_adjoint_kernel(const __grid_constant__ AdjArgs args, uint64_t n,
                                                               uint64_t seed, const uint8_t *codes,
                                                               const double *dl, double *part) {
  extern __shared__ __align__(16) unsigned char smem[];
  AdjArgs &A = *reinterpret_cast<AdjArgs *>(smem);
  float *rw = reinterpret_cast<float *>(smem + align_up(sizeof(AdjArgs)));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  float *stage = rw + WIN * (WIN + 1) + warp * 32 * ADJ_STAGE;
  uint32_t *wcnt = reinterpret_cast<uint32_t *>(rw + WIN * (WIN + 1) + DWARPS * 32 * ADJ_STAGE);   // DWARPS entries
  uint16_t *list = reinterpret_cast<uint16_t *>(wcnt + DWARPS);                                    // ADJ_TILE entries
  {
    const uint32_t *src = reinterpret_cast<const uint32_t *>(&args);
    uint32_t *dst = reinterpret_cast<uint32_t *>(smem);
    for (int k = threadIdx.x; k < (int) (sizeof(AdjArgs) / 4); k += DBLOCK) dst[k] = src[k];
    const ImageGeom &q = args.f.g;
    for (int k = threadIdx.x; k < q.wnx * q.wny; k += DBLOCK) {
      const int r = k / q.wnx, c = k - r * q.wnx;
      rw[r * (WIN + 1) + c] = (float) dl[(size_t) (q.wy0 + r) * q.nx + q.wx0 + c];
    }
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    ShellTangents &S = A.d[threadIdx.x];
    const mxd::V3 p = mxd::matv(S.fwd, {A.p0[0], A.p0[1], A.p0[2]});
    S.p1[0] = p.x; S.p1[1] = p.y; S.p1[2] = p.z;
  }
  const ImageGeom &g = A.f.g;
  double pacc = 0.0;               // lane p < NP: this warp's sum for parameter p
  for (uint64_t tile = (uint64_t) blockIdx.x * ADJ_TILE; tile < n; tile += (uint64_t) gridDim.x * ADJ_TILE) {
    // The rays of the tile that reached the focal plane, in ascending order:
    // only they contribute, and lanes given the others would idle through
    // the whole ray.  A thread takes eight decision bytes.
    const uint64_t i0 = tile + 8 * threadIdx.x;
    unsigned long long word = 0;
    if (i0 + 8 <= n) word = *reinterpret_cast<const unsigned long long *>(codes + i0);
    else
      for (int b = 0; b < 8; b++)
        if (i0 + b < n) word |= (unsigned long long) codes[i0 + b] << (8 * b);
    word &= 0x0101010101010101ull * mxd::RAY_HIT;
    const uint32_t mine = (uint32_t) __popcll(word);
    uint32_t off = mine;
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, off, o);
      if (lane >= o) off += v;
    }
    if (lane == 31) wcnt[warp] = off;
    __syncthreads();
    off -= mine;
    uint32_t nh = 0;
    for (int k = 0; k < DWARPS; k++) {
      const uint32_t c = wcnt[k];
      off += k < warp ? c : 0u;
      nh += c;
    }
    for (int b = 0; b < 8; b++)
      if ((word >> (8 * b)) & 1ull) list[off++] = (uint16_t) (8 * threadIdx.x + b);
    __syncthreads();
    for (uint32_t b0 = warp * 32; b0 < nh; b0 += DBLOCK) {
      float c6[mxd::ND];
#pragma unroll
      for (int k = 0; k < mxd::ND; k++) c6[k] = 0.f;
      int si = -1;
      double radius;
      mx::F2 s2, c2;
      const bool valid = b0 + lane < nh;
      const uint32_t i = valid ? (uint32_t) (tile + list[b0 + lane]) : 0u;
      if (valid && ray_front(A.f, nullptr, seed, i, true, si, radius, s2, c2)) {
        mxd::Dual y, z;
        float w, wd[mxd::NT];
        int ic, jc;
        float fu, fv;
        if (ray_tangents(A, si, radius * mx::df_join(s2), radius * mx::df_join(c2), codes[i], y, z, w, wd) && w > 0.0f &&
            splat_origin(g, y.v, z.v, ic, jc, fu, fv)) {
          float ky[mxd::TAPS], kyd[mxd::TAPS];
#pragma unroll
          for (int k = 0; k < mxd::TAPS; k++) {
            ky[k] = tap(g, k, fu);
            kyd[k] = ((float) (k - mxd::HALF) - fu) * g.inv_s2 * ky[k];
          }
          float sw = 0.f, su = 0.f, sv = 0.f;
          const bool inside = ic - mxd::HALF >= g.wx0 && ic + mxd::HALF < g.wx0 + g.wnx &&
                              jc - mxd::HALF >= g.wy0 && jc + mxd::HALF < g.wy0 + g.wny;
          const float *base_row = rw + (jc - mxd::HALF - g.wy0) * (WIN + 1) + (ic - mxd::HALF - g.wx0);
#pragma unroll 1
          for (int a = 0; a < mxd::TAPS; a++) {
            float t = 0.f, td = 0.f;
            if (inside) {
              const float *q = base_row + a * (WIN + 1);
#pragma unroll
              for (int b = 0; b < mxd::TAPS; b++) { t += q[b] * ky[b]; td += q[b] * kyd[b]; }
            } else {
#pragma unroll
              for (int b = 0; b < mxd::TAPS; b++) {
                const float r = resid_at(g, rw, dl, jc - mxd::HALF + a, ic - mxd::HALF + b);
                t += r * ky[b]; td += r * kyd[b];
              }
            }
            const float kz = tap(g, a, fv), kzd = ((float) (a - mxd::HALF) - fv) * g.inv_s2 * kz;
            sw += kz * t; su += kz * td; sv += kzd * t;
          }
          const float vig = (float) A.f.vig, wi = w * vig * (float) g.inv_pitch;
#pragma unroll
          for (int k = 0; k < mxd::NT; k++)
            c6[k < 2 ? k : k + 2] = vig * sw * wd[k] + wi * (su * y.d[k] + sv * z.d[k]);
          c6[2] = wi * (su * 1e-3f);    // the decenters shift the image, by a micrometre
          c6[3] = wi * (sv * -1e-3f);   // each: x0 towards +y, y0 towards -z
        } else
          si = -1;
      }
      float *row = stage + lane * ADJ_STAGE;
#pragma unroll
      for (int k = 0; k < mxd::ND; k++) row[k] = c6[k];
      row[mxd::ND] = __int_as_float(si);
      __syncwarp();
      if (lane < NP) {
        // lanes 0..15: shell lane/4, slot lane%4; lanes 16, 17: source slots 4, 5
        const int want = lane < 16 ? (lane >> 2) : -2, slot = lane < 16 ? (lane & 3) : lane - 12;
        float s = 0.f;
        for (int r = 0; r < 32; r++) {
          const float *q = stage + r * ADJ_STAGE;
          const int sr = __float_as_int(q[mxd::ND]);
          if (sr == want || (want == -2 && sr >= 0)) s += q[slot];
        }
        pacc += (double) s;
      }
      __syncwarp();
    }
    __syncthreads();   // the list is refilled for the next tile
  }
  __syncthreads();
  double *red = reinterpret_cast<double *>(rw);   // the window is no longer read
  if (lane < NP) red[warp * NP + lane] = pacc;
  __syncthreads();
  if (threadIdx.x < NP) {
    double s = 0.0;
    for (int k = 0; k < DWARPS; k++) s += red[k * NP + threadIdx.x];
    part[(size_t) blockIdx.x * NP + threadIdx.x] = s;
  }
}

}  // namespace

// --------------------------------------------------------------- host --
struct mx_diff {
  mx_context *ctx = nullptr;
  mx_diff_config cfg;
  ImageGeom g;
  int32_t weighted = 0;              // 0: unit weights (ideal mirrors)
  float beta = 0.f, delta = 1.f;     // optical constants at the ray energy
  double corr[4] = {1.0, 1.0, 1.0, 1.0};   // effective-area correction per reflection
  double vig = 1.0;
  DevBuf codes, acc, part, out;   // out: 4 moments, then NP gradient values
  double *h_out = nullptr;        // pinned: moments and gradient read back
  bool recorded = false;
  int fwd_blocks = 0, mom_blocks = 0, rays_blocks = 0, adj_blocks = 0;
  size_t fwd_smem = 0, rays_smem = 0, adj_smem = 0;
};

namespace {

constexpr double PI_D = 3.14159265358979323846264338327950288;
constexpr double ARCSEC = PI_D / (180.0 * 3600.0);

int diff_fail(mx_diff *d, int code, const std::string &msg) { return mx_fail(d ? d->ctx : nullptr, code, msg); }

// Both optics of every shell at theta, with derivatives: tilts enter az_mis
// and el_mis (degrees in the geometry file) and decenters x0 and y0 (mm),
// as read_hrma_geometry_file (hrma.c:319-391) and init_hrma_shells take
// them; the rotations are rebuilt as init_yaw_pitch does.
int build_optics(mx_diff *d, const double *theta, mxd::Optic opt[4][2], mxd::Between mid[4], Dual6 p0[3]) {
  mx_context *c = d->ctx;
  std::string err;
  size_t cnt = 0;
  const double *rdb = c->pack.get<double>("hrma/rdb", &cnt, err);
  if (!rdb || cnt != 72) return diff_fail(d, MX_EPACK, "mx_diff: hrma/rdb missing from the table pack");
  for (int s = 0; s < 4; s++) {
    const MxShellDev &h = c->hm.shells[s];
    const double cap_pos = c->cfg.hrma_cap_x + c->cfg.shell_xoffset[s];
    for (int o = 0; o < 2; o++) {
      const double *q = rdb + (4 * o + s) * 9;   // x0 y0 z0 p k rho0 az el l
      mxd::Optic &op = opt[s][o];
      Dual6 x0 = mxd::mkd(q[0] + theta[4 * s + 2] * 1e-3);
      x0.d[2] = 1e-3f;
      Dual6 y0 = mxd::mkd(q[1] + theta[4 * s + 3] * 1e-3);
      y0.d[3] = 1e-3f;
      op.to[0] = mxd::mkd(-(-q[2]) - cap_pos);
      op.to[1] = 0.0 - x0;
      op.to[2] = y0;
      Dual6 az = mxd::mkd(-(q[6] + theta[4 * s] / 3600.0) * (PI_D / 180.0));
      az.d[0] = (float) -ARCSEC;
      Dual6 el = mxd::mkd(-(q[7] + theta[4 * s + 1] / 3600.0) * (PI_D / 180.0));
      el.d[1] = (float) -ARCSEC;
      mxd::yaw_pitch(op.fwd, op.bwd, az, el);
      for (int r = 0; r < 3; r++) op.ff[r] = op.fwd[3 * r] * (h.front_position + op.to[0]);
    }
    const mxd::Optic &P = opt[s][0], &H = opt[s][1];
    mxd::Between &B = mid[s];
    mxd::mat3_mul(B.m, H.fwd, P.bwd);
    const Dual6 dt[3] = {H.to[0] - P.to[0], H.to[1] - P.to[1], H.to[2] - P.to[2]};
    for (int r = 0; r < 3; r++) B.c[r] = H.fwd[3 * r] * dt[0] + H.fwd[3 * r + 1] * dt[1] + H.fwd[3 * r + 2] * dt[2];
  }
  Dual6 ay = mxd::mkd((d->cfg.src_y + theta[16]) * ARCSEC);
  ay.d[4] = (float) ARCSEC;
  Dual6 az = mxd::mkd((d->cfg.src_z + theta[17]) * ARCSEC);
  az.d[5] = (float) ARCSEC;
  const Dual6 ty = 0.0 - mxd::dtan(ay), tz = 0.0 - mxd::dtan(az), inv = mxd::drsqrt(1.0 + ty * ty + tz * tz);
  p0[0] = 0.0 - inv; p0[1] = inv * ty; p0[2] = inv * tz;
  for (int s = 0; s < 4; s++)
    for (int r = 0; r < 3; r++) {
      const Dual6 *m = opt[s][0].fwd + 3 * r;
      mid[s].p1[r] = m[0] * p0[0] + m[1] * p0[1] + m[2] * p0[2];
    }
  return MX_OK;
}

int check_theta(mx_diff *d, const double *theta) {
  if (!theta) return diff_fail(d, MX_EINVAL, "mx_diff: theta is null");
  for (int k = 0; k < NP; k++)
    if (!std::isfinite(theta[k]) || fabs(theta[k]) > 3600.0)
      return diff_fail(d, MX_EINVAL, "mx_diff: theta[" + std::to_string(k) + "] must be finite and within +-3600");
  return MX_OK;
}

void fill_rays(mx_diff *d, const mxd::Optic opt[4][2], const mxd::Between mid[4], const Dual6 p0[3], FwdArgs &F) {
  for (int s = 0; s < 4; s++) {
    DiffShell &S = F.sh[s];
    MxShellDev &h = S.h;
    h = d->ctx->hm.shells[s];
    for (int o = 0; o < 2; o++) {
      for (int k = 0; k < 3; k++) h.to_osac[o][k] = opt[s][o].to[k].v;
      for (int k = 0; k < 9; k++) { h.fwd[o][k] = opt[s][o].fwd[k].v; h.bwd[o][k] = opt[s][o].bwd[k].v; }
    }
    for (int k = 0; k < 3; k++) { h.front_fwd[k] = opt[s][0].ff[k].v; h.osac0f[k] = (float) h.to_osac[0][k]; }
    h.front_fwdf = (float) h.front_fwd[0];
    for (int k = 0; k < 9; k++) { h.mid[k] = mid[s].m[k].v; h.bwd0f[k] = (float) h.bwd[0][k]; }
    for (int k = 0; k < 3; k++) h.mid_off[k] = mid[s].c[k].v;
    for (int k = 0; k < 3; k++) {
      S.p1[k] = mid[s].p1[k].v;
      S.p1f[k] = (float) S.p1[k];
    }
    S.beta = d->beta;
    S.delta = d->delta;
    S.wscale = d->corr[s] * d->corr[s] * d->vig;
  }
  for (int k = 0; k < 3; k++) F.p0[k] = p0[k].v;
  F.vig = d->vig;
  F.ideal = d->ctx->T.ideal;
  F.area_uniform = d->ctx->T.area_uniform;
  F.weighted = d->weighted;
  F.g = d->g;
}

int fill_fwd(mx_diff *d, const double *theta, FwdArgs &F) {
  mxd::Optic opt[4][2];
  mxd::Between mid[4];
  Dual6 p0[3];
  int r = build_optics(d, theta, opt, mid, p0);
  if (r) return r;
  memset(&F, 0, sizeof(F));
  fill_rays(d, opt, mid, p0, F);
  return MX_OK;
}

int fill_adj(mx_diff *d, const double *theta, AdjArgs &A) {
  mxd::Optic opt[4][2];
  mxd::Between mid[4];
  Dual6 p0[3];
  int r = build_optics(d, theta, opt, mid, p0);
  if (r) return r;
  memset(&A, 0, sizeof(A));
  fill_rays(d, opt, mid, p0, A.f);
  const auto turn = [](const Dual6 &a) { return mxd::Turn{a.v, {a.d[0], a.d[1]}}; };
  for (int s = 0; s < 4; s++) {
    ShellTangents &D = A.d[s];
    for (int j = 0; j < 3; j++) { D.front[j] = turn(opt[s][0].ff[j]); D.off[j] = turn(mid[s].c[j]); }
    for (int j = 0; j < 9; j++) { D.fwd[j] = turn(opt[s][0].fwd[j]); D.mid[j] = turn(mid[s].m[j]); D.bwd[j] = turn(opt[s][1].bwd[j]); }
    for (int j = 0; j < 3; j++) D.back[j] = mxd::Turn{-opt[s][1].to[j].v, {0.f, 0.f}};
    D.corr = d->corr[s];
  }
  for (int k = 0; k < 3; k++) A.p0[k] = mxd::Dual{p0[k].v, {0.f, 0.f, p0[k].d[4], p0[k].d[5]}};
  const double nr = 1.0 - (double) d->delta, ni = d->beta;
  const auto two = [](double v) { const float hi = (float) v; return mx::F2{hi, (float) (v - hi)}; };
  A.fr.sr = two(nr * nr - ni * ni);
  A.fr.si = two(2.0 * nr * ni);
  A.fr.lost = two(1.0 - (nr * nr - ni * ni));
  return MX_OK;
}

template <class K>
cudaError_t occupancy(K kernel, size_t smem, int num_sms, int *blocks) {
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
  if (e != cudaSuccess) return e;
  int per = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, DBLOCK, smem);
  if (e != cudaSuccess) return e;
  if (per < 1) return cudaErrorInvalidConfiguration;
  *blocks = per * num_sms;
  return cudaSuccess;
}

}  // namespace

extern "C" {

mx_diff *mx_diff_create(mx_context *c, const mx_diff_config *cfg) {
  if (!c || !cfg) { mx_fail(c, MX_EINVAL, "mx_diff_create: null argument"); return nullptr; }
  const mx_diff_config &k = *cfg;
  std::string bad;
  if (k.n_rays < 1 || k.n_rays > MX_DIFF_MAX_RAYS) bad = "n_rays must be in 1 .. 2^32-1";
  else if (!(k.energy > 0.0) || !std::isfinite(k.energy)) bad = "energy must be positive";
  else if (!(k.pitch > 0.0) || !std::isfinite(k.pitch)) bad = "pitch must be positive";
  else if (!(k.sigma >= 0.5 && k.sigma <= 1.0)) bad = "sigma must be within 0.5 .. 1 pixel";
  else if (k.nx < 16 || k.nx > 4096 || k.ny < 16 || k.ny > 4096) bad = "nx and ny must be within 16 .. 4096";
  else if (!std::isfinite(k.src_y) || !std::isfinite(k.src_z) || fabs(k.src_y) > 3600.0 || fabs(k.src_z) > 3600.0)
    bad = "source angles must be finite and within +-3600 arcsec";
  else if (!std::isfinite(k.center_y) || !std::isfinite(k.center_z)) bad = "image centre must be finite";
  else if (c->T.source_distance > 0.0) bad = "weighted rays need a source at infinity (SourceDistance 0)";
  if (!bad.empty()) { mx_fail(c, MX_EINVAL, "mx_diff_create: " + bad); return nullptr; }

  mx_diff *d = new mx_diff();
  d->ctx = c;
  d->cfg = k;
  ImageGeom &g = d->g;
  memset(&g, 0, sizeof(g));
  g.nx = (int) k.nx; g.ny = (int) k.ny;
  g.wnx = g.nx < WIN ? g.nx : WIN; g.wny = g.ny < WIN ? g.ny : WIN;
  g.wx0 = g.nx / 2 - g.wnx / 2; g.wy0 = g.ny / 2 - g.wny / 2;
  g.cy = k.center_y; g.cz = k.center_z;
  g.inv_pitch = 1.0 / k.pitch;
  g.cx_pix = 0.5 * g.nx - 0.5; g.cz_pix = 0.5 * g.ny - 0.5;
  g.half_inv_s2 = (float) (0.5 / (k.sigma * k.sigma));
  g.inv_s2 = (float) (1.0 / (k.sigma * k.sigma));
  g.knorm = (float) (1.0 / (std::sqrt(2.0 * PI_D) * k.sigma));
  g.top_u = mx::dkey(g.nx + (double) mxd::HALF);
  g.top_v = mx::dkey(g.ny + (double) mxd::HALF);
  // Each tap product is below w K^2 2^61 with w < 2; a pixel sums at most
  // n_rays of them, so shifting by log2(n K^2 / 4) + 1 keeps it in 64 bits.
  const double kmax = g.knorm;
  int shift = (int) std::ceil(std::log2((double) k.n_rays * kmax * kmax / 4.0)) + 1;
  g.shift = shift < 0 ? 0 : shift;

  const MxTables &T = c->T;
  d->weighted = T.opt_n > 0;
  if (d->weighted) {
    // the optical constants and correction at the ray energy, as the
    // mirror stage interpolates them (float tables, float energy)
    const float fe = (float) k.energy;
    const float *optc = c->hm.optc.data();
    const double *slope = c->hm.optc_slope.data();
    const unsigned on = (unsigned) T.opt_n;
    d->beta = mx::interp_f(fe, optc, optc + on, slope, on);
    d->delta = mx::interp_f(fe, optc, optc + 2 * on, slope + (on - 1), on);
    for (int s = 0; s < 4 && T.use_scale; s++) {
      const MxShellDev &h = c->hm.shells[s];
      const float *ce = optc + 3 * on + h.corr_off;
      d->corr[s] = std::sqrt((double) mx::interp_f(fe, ce, ce + h.corr_n, slope + h.corr_slope_off, (unsigned) h.corr_n));
    }
  }
  d->vig = T.ideal ? 1.0 : T.hrma_vig;

  cudaError_t e = cudaSetDevice(c->device);
  if (e == cudaSuccess) {
    d->rays_smem = align_up(sizeof(FwdArgs)) + DWARPS * sizeof(RayList);
    d->fwd_smem = d->rays_smem + 4 * (2 * WIN * WSTRIDE + DWARPS * 16 * STAGE_STRIDE);
    d->adj_smem = align_up(sizeof(AdjArgs)) + 4 * WIN * (WIN + 1) + 4 * DWARPS * (32 * ADJ_STAGE + 1) + 2 * ADJ_TILE;
    e = occupancy(diff_forward_kernel<true, false>, d->fwd_smem, c->num_sms, &d->fwd_blocks);
  }
  if (e == cudaSuccess) e = occupancy(diff_forward_kernel<true, true>, d->fwd_smem, c->num_sms, &d->mom_blocks);
  if (e == cudaSuccess) e = occupancy(diff_forward_kernel<false, false>, d->rays_smem, c->num_sms, &d->rays_blocks);
  if (e == cudaSuccess) e = occupancy(diff_adjoint_kernel, d->adj_smem, c->num_sms, &d->adj_blocks);
  const int maxb = std::max(d->mom_blocks, d->adj_blocks);
  if (e == cudaSuccess) e = d->codes.ensure(k.n_rays);
  if (e == cudaSuccess) e = d->acc.ensure(sizeof(unsigned long long) * k.nx * k.ny);
  if (e == cudaSuccess) e = d->part.ensure(sizeof(double) * (size_t) maxb * NP);
  if (e == cudaSuccess) e = d->out.ensure(sizeof(double) * (4 + NP));
  if (e == cudaSuccess) e = cudaMallocHost(&d->h_out, sizeof(double) * (4 + NP));
  if (e == cudaSuccess) e = cudaMemset(d->codes.ptr, 0, k.n_rays);
  if (e != cudaSuccess) {
    mx_cuda_fail(c, e, "mx_diff_create");
    mx_diff_destroy(d);
    return nullptr;
  }
  return d;
}

void mx_diff_destroy(mx_diff *d) {
  if (!d) return;
  d->codes.release(); d->acc.release(); d->part.release(); d->out.release();
  if (d->h_out) cudaFreeHost(d->h_out);
  delete d;
}

int mx_diff_forward(mx_diff *d, const double *theta, int mode, double *image, double *moments, void *stream) {
  if (!d) return mx_fail(nullptr, MX_EINVAL, "mx_diff_forward: null handle");
  if (!image) return diff_fail(d, MX_EINVAL, "mx_diff_forward: image is null");
  if (mode != MX_DIFF_RECORD && mode != MX_DIFF_REPLAY && mode != MX_DIFF_FRESH)
    return diff_fail(d, MX_EINVAL, "mx_diff_forward: unknown mode");
  if (mode == MX_DIFF_REPLAY && !d->recorded)
    return diff_fail(d, MX_EINVAL, "mx_diff_forward: MX_DIFF_REPLAY before any MX_DIFF_RECORD call");
  int r = check_theta(d, theta);
  if (r) return r;
  FwdArgs F;
  if ((r = fill_fwd(d, theta, F))) return r;
  mx_context *c = d->ctx;
  cudaStream_t st = (cudaStream_t) stream;
  const size_t npix = (size_t) d->cfg.nx * d->cfg.ny;
  cudaError_t e = cudaMemsetAsync(d->acc.ptr, 0, npix * sizeof(unsigned long long), st);
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "mx_diff_forward");
  unsigned long long *acc = (unsigned long long *) d->acc.ptr;
  if (moments)
    diff_forward_kernel<true, true><<<d->mom_blocks, DBLOCK, d->fwd_smem, st>>>(
        F, c->T, d->cfg.n_rays, d->cfg.seed, (uint8_t *) d->codes.ptr, mode, acc, (double *) d->part.ptr, nullptr);
  else
    diff_forward_kernel<true, false><<<d->fwd_blocks, DBLOCK, d->fwd_smem, st>>>(
        F, c->T, d->cfg.n_rays, d->cfg.seed, (uint8_t *) d->codes.ptr, mode, acc, nullptr, nullptr);
  const double scale = std::ldexp(1.0, d->g.shift - 61) / (double) d->cfg.n_rays;
  diff_image_kernel<<<2 * c->num_sms, 256, 0, st>>>(acc, npix, scale, image);
  if (moments)
    diff_sum_kernel<<<1, 32 * 4, 0, st>>>((const double *) d->part.ptr, d->mom_blocks, 4, 1.0, (double *) d->out.ptr);
  c->launches += moments ? 3 : 2;
  if ((e = cudaGetLastError()) != cudaSuccess) return mx_cuda_fail(c, e, "mx_diff_forward: launch");
  if (mode == MX_DIFF_RECORD) d->recorded = true;
  if (moments) {
    e = cudaMemcpyAsync(d->h_out, d->out.ptr, 4 * sizeof(double), cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return mx_cuda_fail(c, e, "mx_diff_forward: moments");
    memcpy(moments, d->h_out, 4 * sizeof(double));
  }
  return MX_OK;
}

int mx_diff_rays(mx_diff *d, const double *theta, int mode, double *yzw, void *stream) {
  if (!d) return mx_fail(nullptr, MX_EINVAL, "mx_diff_rays: null handle");
  if (!yzw) return diff_fail(d, MX_EINVAL, "mx_diff_rays: yzw is null");
  if (mode != MX_DIFF_RECORD && mode != MX_DIFF_REPLAY && mode != MX_DIFF_FRESH)
    return diff_fail(d, MX_EINVAL, "mx_diff_rays: unknown mode");
  if (mode == MX_DIFF_REPLAY && !d->recorded)
    return diff_fail(d, MX_EINVAL, "mx_diff_rays: MX_DIFF_REPLAY before any MX_DIFF_RECORD call");
  int r = check_theta(d, theta);
  if (r) return r;
  FwdArgs F;
  if ((r = fill_fwd(d, theta, F))) return r;
  mx_context *c = d->ctx;
  cudaStream_t st = (cudaStream_t) stream;
  diff_forward_kernel<false, false><<<d->rays_blocks, DBLOCK, d->rays_smem, st>>>(
      F, c->T, d->cfg.n_rays, d->cfg.seed, (uint8_t *) d->codes.ptr, mode, nullptr, nullptr, yzw);
  c->launches += 1;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "mx_diff_rays: launch");
  if (mode == MX_DIFF_RECORD) d->recorded = true;
  return MX_OK;
}

int mx_diff_mse(mx_diff *d, const double *image, const double *target, double *dl_dimage, double *loss,
                void *stream) {
  if (!d) return mx_fail(nullptr, MX_EINVAL, "mx_diff_mse: null handle");
  if (!image || !target || !loss) return diff_fail(d, MX_EINVAL, "mx_diff_mse: image, target and loss are required");
  const size_t npix = (size_t) d->cfg.nx * d->cfg.ny;
  diff_mse_kernel<<<MSE_BLOCKS, MSE_THREADS, 0, (cudaStream_t) stream>>>(
      image, target, npix, 1.0 / (double) npix, dl_dimage, loss);
  d->ctx->launches += 1;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MX_OK : mx_cuda_fail(d->ctx, e, "mx_diff_mse: launch");
}

int mx_diff_adjoint_async(mx_diff *d, const double *theta, const double *dl_dimage, double *grad_dev, void *stream) {
  if (!d) return mx_fail(nullptr, MX_EINVAL, "mx_diff_adjoint: null handle");
  if (!dl_dimage || !grad_dev) return diff_fail(d, MX_EINVAL, "mx_diff_adjoint: dl_dimage and grad are required");
  if (!d->recorded) return diff_fail(d, MX_EINVAL, "mx_diff_adjoint: no MX_DIFF_RECORD call yet");
  int r = check_theta(d, theta);
  if (r) return r;
  AdjArgs A;
  if ((r = fill_adj(d, theta, A))) return r;
  mx_context *c = d->ctx;
  cudaStream_t st = (cudaStream_t) stream;
  diff_adjoint_kernel<<<d->adj_blocks, DBLOCK, d->adj_smem, st>>>(A, d->cfg.n_rays, d->cfg.seed,
                                                                   (const uint8_t *) d->codes.ptr, dl_dimage,
                                                                   (double *) d->part.ptr);
  diff_sum_kernel<<<1, 32 * NP, 0, st>>>((const double *) d->part.ptr, d->adj_blocks, NP, 1.0 / (double) d->cfg.n_rays,
                                    grad_dev);
  c->launches += 2;
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? MX_OK : mx_cuda_fail(c, e, "mx_diff_adjoint: launch");
}

int mx_diff_adjoint(mx_diff *d, const double *theta, const double *dl_dimage, double *grad, void *stream) {
  if (!d) return mx_fail(nullptr, MX_EINVAL, "mx_diff_adjoint: null handle");
  if (!grad) return diff_fail(d, MX_EINVAL, "mx_diff_adjoint: grad is null");
  double *gdev = (double *) d->out.ptr + 4;
  int r = mx_diff_adjoint_async(d, theta, dl_dimage, gdev, stream);
  if (r) return r;
  cudaStream_t st = (cudaStream_t) stream;
  cudaError_t e = cudaMemcpyAsync(d->h_out + 4, gdev, NP * sizeof(double), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return mx_cuda_fail(d->ctx, e, "mx_diff_adjoint: reading the gradient");
  memcpy(grad, d->h_out + 4, NP * sizeof(double));
  return MX_OK;
}

}  // extern "C"
