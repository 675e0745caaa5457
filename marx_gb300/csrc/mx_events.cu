// marx2fits's per-event coordinates (marx/src/marx2fits.c) as a device pass
// over an event list: CHIPX/CHIPY, EXPNO, FLTGRADE/GRADE, DETX/DETY, sky
// X/Y and TDETX/TDETY.  Each event is independent except for ACIS frames:
// marx2fits keeps the dither state of a frame's first event for the whole
// frame (read_dither_value, marx2fits.c:3567-3581), so the pass finds each
// event's frame start with a max-scan over the event order.
//
// This file is compiled without fused multiply-add contraction: DETX/DETY
// are pure arithmetic in the reference (pixlib.c:135-222, detpix.c:182-208)
// and round bit for bit like it.  The sky columns are formed from the same
// unit vector in a well-conditioned form (sky_offsets).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "mx_context.h"
#include "mx_device.cuh"

using namespace mx;

namespace mx_ev {

constexpr int EV_BLOCK = 256;
constexpr int EV_MAX_FACETS = 6;

struct EvFacet {
  double x_ll[3], xhat[3], yhat[3];
  double xps, yps, xoff, yoff, tdx, tdy;   // pixel sizes, pixel of the LL corner, tiled offsets
  // of a detector that has neither moved nor turned: its corner from the
  // mirror's node (the params' offsets in), and its basis xps xhat, yps yhat
  double ofs[3], e1[3], e2[3];
  int32_t itdx, itdy;                      // tdx, tdy, which are whole numbers
  int32_t tiled, pad;                      // 0: ACIS-I chips 0, 2; 1: ACIS-I chips 1, 3; 2: x + tdx, y + tdy
};

struct EvGeom {
  EvFacet f[EV_MAX_FACETS];
  int32_t nf, first_id, acis, pad;
  double fp_delta, fp_x0, fp_y0;       // focal-plane system (detpix.c:42-63)
  const float *sp;                     // sub-pixel rows: energies, dx, dy (npoints each)
  const int32_t *sp_row;               // [2][256]: FI/BI x fltgrade -> offset of the row in sp, -1: none
  const int32_t *sp_n;                 // [2][256]: npoints
};

struct EvArgs {
  mx_events e;
  mx_event_params p;
  uint64_t seed;
  double roll_c, roll_s;               // cos, sin of Roll_Nom (host libm, as the reference)
  float inv_frame[2];                  // 1 / frame_time as hi + lo; NaN: divide
  float inv_delta[2];                  // 1 / fp_delta (pixels per radian) as hi + lo
  int frames;                          // frame runs decide the dither
  int rounds;                          // rounds of EV_BLOCK events in a block's tile
  unsigned long long *bad;
};

// FLTGRADE of each of the 3 x 3 sub-pixels, four equally likely values
// (Flight_Grade_Table, marx2fits.c:3838-3849): rows -- 0- +- -0 00 +0 -+ 0+ ++.
__constant__ int16_t kFlightGrades[9][4] = {
    {10, 11, 138, 139}, {2, 34, 130, 162}, {18, 22, 50, 54},
    {8, 12, 136, 140},  {0, 0, 0, 0},      {16, 17, 48, 49},
    {72, 76, 104, 108}, {64, 65, 68, 69},  {80, 81, 208, 209}};
// ASCA grade of each flight grade (the CALDB grade map the reference
// tabulates as Grade_Map, marx2fits.c:3792-3810), one digit per fltgrade.
__constant__ char kGradeMap[257] =
    "0125115735663577446755677777777711251157577757774467556777777777"
    "2277227767776777667777777777777755775577677767777777777777777777"
    "1125115735663577557777777777777711251157577757775577777777777777"
    "5577557777777777667777777777777777777777777777777777777777777777";

__device__ __forceinline__ double event_uniform(uint64_t seed, uint32_t k, uint32_t slot) {
  uint32_t c[4] = {k, slot, 0x5A5A0004u, 0u};
  philox(c, (uint32_t) seed, (uint32_t) (seed >> 32));
  uint64_t b = ((uint64_t) c[0] << 32) | c[1];
  return unit_from_bits(b >> 11);
}

__device__ __forceinline__ uint32_t row_of(const mx_events &e, uint32_t k) { return e.index ? e.index[k] : k; }

// time.dat as marx2fits reads it: a float.
__device__ __forceinline__ float event_time(const EvArgs &a, uint32_t row) {
  if (a.e.time) return a.e.time[row];
  return d2f_rn(a.e.time64[row] + a.p.time_offset);
}

// (int64) (t / frame_time), compute_expno (marx2fits.c:3741-3761).  The
// quotient in double-float (t exact, 1 / frame_time to 2^-48) is within
// 2^-45 of the true one and so within 2^-44 of the double quotient: unless
// an integer lies that close, both truncate alike, and no FP64 operation is
// needed.  Others (a time on a frame's edge), and times outside 0 .. 2^22
// frames, take the division.
__device__ __forceinline__ int64_t frame_number(const EvArgs &a, float t) {
  const F2 q = df_mul_f(F2{a.inv_frame[0], a.inv_frame[1]}, t);
  float i = floorf(q.h), f = (q.h - i) + q.l;
  if (f < 0.0f) { i -= 1.0f; f += 1.0f; }
  const float edge = q.h * 0x1p-40f + 0x1p-60f;
  if (q.h > 0.0f && q.h < 0x1p22f && f > edge && f < 1.0f - edge) return (int64_t) (int) i;
  return (int64_t) (f2d(t) / a.p.frame_time);
}

// JDMv_length (vector.c:77-97)
__device__ __forceinline__ double jdm_length(double ax, double ay, double az) {
  double x = fabs(ax), y = fabs(ay), z = fabs(az), t;
  if (z < x) { t = z; z = x; x = t; }
  if (z < y) { t = z; z = y; y = t; }
  if (z == 0.0) return 0.0;
  x = x / z; y = y / z;
  return z * sqrt(1.0 + x * x + y * y);
}
// JDMv_normalize (vector.c:99-109)
__device__ __forceinline__ D3 jdm_normalize(D3 a) {
  double len = jdm_length(a.x, a.y, a.z);
  if (len != 0.0) { a.x = a.x / len; a.y = a.y / len; a.z = a.z / len; }
  return a;
}
// 0 or a magnitude within 2^-400 .. 2^400
__device__ __forceinline__ bool mid_range(double x) {
  const unsigned e = (unsigned) (dbits(x) >> 52) & 0x7ffu;
  return e - 623u < 800u || is_zero(x);
}
// 1 / d, 2^-40 < |d| < 2^40: the float reciprocal and one Newton step on the
// FP32 pipe give it to 2^-45, a second step in double leaves half an ulp and
// 2^-37 of one: three FP64 operations where the correctly rounded
// reciprocal takes six.
__device__ __forceinline__ double rcp_seeded(double d) {
  const F2 z = split(d);
  const float s = __frcp_rn(z.h);
  const F2 p = df_mul_f(z, s);
  const F2 y2 = quick_sum(s, __fmul_rn(s, __fsub_rn(__fsub_rn(1.0f, p.h), p.l)));
  const double y = df_to(y2);
  return fma(fma(-d, y, 1.0), y, y);
}
// sqrt(v), 1 <= v < 4: the reciprocal root to 2^-44 on the FP32 pipe, then the
// root g = v y corrected by its exact remainder (v - g^2) y / 2, which is
// within 2^-88 of the true root before its one rounding: rounded as sqrt
// rounds it unless the root lies that close to a midpoint of two doubles.
// Four FP64 operations instead of nine.
__device__ __forceinline__ double sqrt_seeded(double v) {
  const F2 y2 = df_rsqrt(split(v));
  const double y = df_to(y2), g = v * y;
  return fma(fma(-g, g, v), 0.5 * y, g);
}
// JDMv_normalize's value, the bits too but where a reciprocal (within 2^-37 of
// an ulp) or the root falls on the other side of a midpoint: the five
// quotients by two divisors are Markstein divisions (div_by) from two
// reciprocals, and the comparisons run on the integer pipe; 36 FP64
// operations instead of about 60.  Components far outside the geometry's
// range take the divisions.
__device__ __forceinline__ D3 chip_direction(D3 a) {
  double x = fabs(a.x), y = fabs(a.y), z = fabs(a.z), t;
  if (lt_pos(z, x)) { t = z; z = x; x = t; }
  if (lt_pos(z, y)) { t = z; z = y; y = t; }
  if (!(mid_range(a.x) && mid_range(a.y) && mid_range(a.z) && lt_pos(0x1p-39, z) && lt_pos(z, 0x1p+38)))
    return jdm_normalize(a);
  const double rz = rcp_seeded(z);
  x = div_by(x, z, rz);
  y = div_by(y, z, rz);
  const double len = z * sqrt_seeded(1.0 + x * x + y * y), rl = rcp_seeded(len);
  return mk(div_by(a.x, len, rl), div_by(a.y, len, rl), div_by(a.z, len, rl));
}
// JDMv_rotate_unit_vector1 (vector.c:187-206)
__device__ __forceinline__ D3 jdm_rotate_unit(D3 p, D3 n, double c, double s) {
  double pn = p.x * n.x + p.y * n.y + p.z * n.z;
  double b = pn * (1.0 - c);
  D3 x3;   // JDMv_pcross_prod (n, p)
  x3.z = n.x * p.y - n.y * p.x;
  x3.x = n.y * p.z - n.z * p.y;
  x3.y = n.z * p.x - n.x * p.z;
  D3 d = mk(c * p.x + b * n.x + s * x3.x, c * p.y + b * n.y + s * x3.y, c * p.z + b * n.z + s * x3.z);
  return jdm_normalize(d);
}

// (float) of the double expression w0 a + w1 b of the sub-pixel tables, w1
// given in double-float: the double-float value is within 2^-42 of
// (|a| + |b|) (1 + |w1|), so unless a float rounding boundary lies within
// 2^-40 of that it rounds as the double expression does.  ok is cleared
// otherwise.
__device__ __forceinline__ float lerp_to_float(F2 w0, F2 w1, float a, float b, bool &ok) {
  if (a == 0.0f && b == 0.0f) return 0.0f;
  const F2 p = df_mul_f(w0, a), q = df_mul_f(w1, b);
  const F2 v = df_add(p, q);
  const float m = (fabsf(a) + fabsf(b)) * (1.0f + fabsf(w1.h));
  // v.h is the float nearest v; the boundary is half a step from it, and
  // half a step is 2^-25 |v.h| or more
  const uint32_t e = f2u(v.h) & 0x7f800000u;
  const float half = u2f(e) * 0x1p-24f;
  // a power of two has the nearer boundary, a quarter step, below it
  const float away = (f2u(v.h) & 0x7fffffu) ? half - fabsf(v.l) : 0.5f * half - fabsf(v.l);
  if (!(away > 0x1p-40f * m && fabsf(v.h) > 0x1p-60f && m < 0x1p60f)) ok = false;
  return v.h;
}

// marx_compute_acis_subpix (acis_subpix.c:284-320).  The interpolation runs
// in double-float on the FP32 pipe; where that does not settle the float the
// double expression does.
static __device__ void subpix(const EvGeom &G, int ccd, float energy, int fltgrade, float &dx, float &dy) {
  int kind = (ccd == 5 || ccd == 7) ? 1 : 0;   // BI chips (read_subpixel_file, acis_subpix.c:246-252)
  int off = __ldg(G.sp_row + kind * 256 + fltgrade);
  if (off < 0) { dx = dy = 0.0f; return; }
  unsigned n = (unsigned) __ldg(G.sp_n + kind * 256 + fltgrade);
  const float *e = G.sp + off, *xs = e + n, *ys = xs + n;
  unsigned j = bsearch_f(energy, e, n);
  if (j == 0) j++;
  if (j == n) j--;
  const float e0 = __ldg(e + j - 1), e1 = __ldg(e + j);
  const float x0 = __ldg(xs + j - 1), x1 = __ldg(xs + j), y0 = __ldg(ys + j - 1), y1 = __ldg(ys + j);
  {
    const float de = __fsub_rn(e1, e0);
    const F2 num = two_sum(energy, -e0);
    bool ok = de > 0x1p-30f && fabsf(num.h) < 0x1p30f;
    const F2 w1 = df_div(num, F2{de, 0.0f}), w0 = df_sub(F2{1.0f, 0.0f}, w1);
    dx = lerp_to_float(w0, w1, x0, x1, ok);
    dy = lerp_to_float(w0, w1, y0, y1, ok);
    if (ok) return;
  }
  double w1 = ((double) energy - e0) / (double) (e1 - e0);
  double w0 = 1.0 - w1;
  dx = (float) (w0 * x0 + w1 * x1);
  dy = (float) (w0 * y0 + w1 * y1);
}

// angle - (angle)^3 series: atan q = q - q^3 (1/3 - q^2/5 + ...) and
// asin z = z + z^3 (1/6 + 3 z^2/40 + ...) for |q|, |z| below 2^-5: the
// coefficients after the first in single precision (below 1e-7 of the
// value), the terms left out below 1e-15 of it.
__device__ __forceinline__ F2 atan_small(F2 q) {
  const F2 s = df_sqr(q);
  float g = __fmaf_rn(s.h, -0x1.745d18p-4f, 0x1.c71c72p-4f);           // 1/9 - s/11
  g = __fmaf_rn(s.h, -g, 0x1.24924ap-3f);                              // 1/7 - ...
  g = __fmaf_rn(s.h, -g, 0x1.99999ap-3f);                              // 1/5 - ...
  const F2 c = df_add(F2{0x1.555556p-2f, -0x1.555556p-27f}, df_mul_f(s, -g));
  return df_sub(q, df_mul(q, df_mul(s, c)));
}
__device__ __forceinline__ F2 asin_small(F2 z) {
  const F2 s = df_sqr(z);
  float g = __fmaf_rn(s.h, 0x1.6e8ba2p-6f, 0x1.f1c71cp-6f);            // 35/1152 + s 63/2816
  g = __fmaf_rn(s.h, g, 0x1.6db6dcp-5f);                               // 5/112 + ...
  g = __fmaf_rn(s.h, g, 0x1.333334p-4f);                               // 3/40 + ...
  const F2 c = df_add(F2{0x1.555556p-3f, -0x1.555556p-28f}, df_mul_f(s, g));
  return df_add(z, df_mul(z, df_mul(s, c)));
}

// Sine and cosine of a roll angle in double-float, |roll| < 8: k quarter
// turns off in three parts (k times the first is exact).
__device__ __forceinline__ void roll_sincos(float roll, F2 &s, F2 &c) {
  const float k = rintf(__fmul_rn(roll, 0x1.45f306p-1f));
  const F2 a = two_sum(__fmaf_rn(-k, 0x1.92p+0f, roll), __fmul_rn(-k, 0x1.fb4p-12f));
  const F2 r = df_add(a, df_mul_f(F2{-0x1.4442d2p-24f, 0x1.ee59dap-50f}, k));
  F2 sr, cr;
  df_sincos(r, sr, cr);
  const int q = (int) k & 3;
  s = (q & 1) ? cr : sr;
  c = (q & 1) ? sr : cr;
  if (q & 2) s = df_neg(s);
  if ((q + 1) & 2) c = df_neg(c);
}

// Sky X, Y of a dithered event (compute_xy_sky, marx2fits.c:3869-3910): the
// direction undithered (unapply_dither, dither.c:583-607), rolled, and its
// offsets in RA and Dec from (0, 0) in pixels.  The reference takes both
// angles as acos of numbers near 1 and passes them through cos, sin, atan
// and asin; about (0, 0) the offsets are atan(y / x) and -asin(z) of the
// rolled unit vector.  They are formed in double-float on the FP32 pipe
// (relative error of an offset below 2^-43, within 1e-10 pixel), 4 FP64
// operations in place of about 480.  The acos form's own rounding moves an
// event at angle t by up to 3e-16 / t, 2.5e-9 of the coordinate (1e-5 pixel) at
// SKY_NEAR and less from there out, which these values are free of; nearer the
// axes of the pointing (1 % of a field's events) sky_reference keeps the
// reference's rounding.
// False, with nothing written, also when the event is not within 0.03 rad
// of the pointing or its dither not below 1e-4 rad.
constexpr float SKY_NEAR = 1.2e-5f;
__device__ __forceinline__ bool sky_offsets(const EvArgs &a, const EvGeom &G, D3 mnc, float ra, float dec, F2 rs,
                                            F2 rc, double &sx, double &sy) {
  const F2 px = split(mnc.x), py = split(mnc.y), pz = split(mnc.z);
  if (!(fabsf(ra) < 1e-4f && fabsf(dec) < 1e-4f && px.h < -0.9f && fabsf(py.h) < 0.03f && fabsf(pz.h) < 0.03f))
    return false;
  // the dither's rotation undone as the change it makes to p: axis
  // (0, ny, nz) = (0, -sin dec, cos dec sin ra), d = 1 - cos dec cos ra;
  // the products with p.x in double-float, the terms below 1e-6 in single
  const float r2 = __fmul_rn(ra, ra), e2 = __fmul_rn(dec, dec);
  const F2 ny = quick_sum(-dec, __fmul_rn(__fmul_rn(dec, e2), 0x1.555556p-3f));
  const F2 nz = quick_sum(ra, -__fmul_rn(ra, __fmaf_rn(0.5f, e2, __fmul_rn(r2, 0x1.555556p-3f))));
  const float d = 0.5f * __fadd_rn(r2, e2), k = 0.5f * __fmaf_rn(py.h, ny.h, __fmul_rn(pz.h, nz.h));
  const F2 x = two_sum(px.h, __fadd_rn(px.l, __fmaf_rn(ny.h, pz.h, __fmaf_rn(-nz.h, py.h, -__fmul_rn(d, px.h)))));
  const float ty = __fmaf_rn(k, ny.h, -__fmul_rn(d, py.h)), tz = __fmaf_rn(k, nz.h, -__fmul_rn(d, pz.h));
  const F2 y = df_add(py, df_add(df_mul(nz, px), F2{ty, 0.0f}));
  const F2 z = df_add(pz, df_add(df_mul(df_neg(ny), px), F2{tz, 0.0f}));
  // roll about x
  const F2 y2 = df_sub(df_mul(rc, y), df_mul(rs, z)), z2 = df_add(df_mul(rc, z), df_mul(rs, y));
  const float ay = fabsf(y2.h), az = fabsf(z2.h);
  if (!(ay < 0.03f && az < 0.03f && ay > SKY_NEAR && az > SKY_NEAR)) return false;
  // y / x by the float reciprocal and one remainder
  const float rx = __frcp_rn(x.h), q0 = __fmul_rn(y2.h, rx);
  const F2 rem = df_sub(y2, df_mul_f(x, q0));
  const F2 q = quick_sum(q0, __fmul_rn(rem.h, rx));
  const F2 inv = {a.inv_delta[0], a.inv_delta[1]};
  const F2 u = df_mul(atan_small(q), inv), v = df_mul(asin_small(z2), inv);
  sx = (G.fp_x0 - f2d(u.h)) - f2d(u.l);
  sy = (G.fp_y0 - f2d(v.h)) - f2d(v.l);
  return true;
}

// acos(v) for v just below 1: with w = 1 - v (exact), sqrt(2 w) times the
// series 1 + w/12 + 3 w^2/160 + ...; false when v is not within 2^-10 of 1.
__device__ __forceinline__ bool acos_near_one(double v, double &t) {
  const double w = 1.0 - v;
  if (!(dbits(w) < dbits(0x1p-10))) return false;   // w = +0 .. 2^-10
  double c = fma(w, 63.0 / 90112.0, 35.0 / 18432.0);
  c = fma(c, w, 5.0 / 896.0);
  c = fma(c, w, 3.0 / 160.0);
  c = fma(c, w, 1.0 / 12.0);
  const double r = sqrt(w + w);
  t = fma(r * w, c, r);
  return true;
}

// The same columns in the reference's own steps, for any direction.  Within
// a few degrees of the pointing the offsets are the two acos values
// themselves (the reference's sin, cos, asin and atan undo each other).
__device__ __noinline__ void sky_reference(const EvGeom &G, D3 mnc, float ra_f, float dec_f, float roll_f, double &sx,
                                           double &sy) {
  const double d_ra = f2d(ra_f), d_dec = f2d(dec_f), d_roll = f2d(roll_f);
  // marx_undither_mnc -> unapply_dither (dither.c:583-607)
  // dither offsets are arcseconds: the short series rounds like the host's sin and cos
  double sra, cra, sdec, cdec;
  sincos_small(d_ra, &sra, &cra);
  sincos_small(d_dec, &sdec, &cdec);
  const double cos_t = cdec * cra;
  D3 n = mk(0.0, -sdec, cdec * sra);
  const double sin_t = jdm_length(n.x, n.y, n.z);
  if (sin_t >= 1e-20) {
    n = mk(n.x / sin_t, n.y / sin_t, n.z / sin_t);
    mnc = jdm_rotate_unit(mnc, n, cos_t, sin_t);
  }
  double roll_s, roll_c;
  sincos(d_roll, &roll_s, &roll_c);
  mnc = jdm_rotate_unit(mnc, mk(1.0, 0.0, 0.0), roll_c, roll_s);
  // marx_mnc_to_ra_dec (pixlib.c:499-523)
  double perp = sqrt(mnc.x * mnc.x + mnc.y * mnc.y);
  if (perp > 1.0) perp = 1.0;
  const double q = -mnc.x / perp;
  double dec, ra;
  if (acos_near_one(perp, dec) && acos_near_one(q, ra)) {
    sx = (mnc.y <= 0.0 ? -ra : ra) / G.fp_delta + G.fp_x0;
    sy = (mnc.z <= 0 ? dec : -dec) / G.fp_delta + G.fp_y0;
    return;
  }
  dec = mnc.z <= 0 ? acos(perp) : -acos(perp);
  ra = mnc.y <= 0.0 ? acos(q) : -acos(q);
  // marx_compute_ra_dec_offsets (pixlib.c:531-570) about (0, 0): cos(dec)
  // and cos(d_dec) are the same value there
  double sdec_s, c, sra_s, cra_s;
  sincos(dec, &sdec_s, &c);
  sincos(ra, &sra_s, &cra_s);
  const double factor = c * (1 - cra_s);
  double sin_dd = sdec_s + factor * 0.0;
  if (fabs(sin_dd) > 1.0) sin_dd = sin_dd < 0 ? -1.0 : 1.0;
  const double ddec = asin(sin_dd);
  const double num = c * sra_s, den = c - factor * 1.0;
  double dra;
  if (den >= 0) dra = atan(num / den);
  else dra = num >= 0 ? atan(num / den) + PI : atan(num / den) - PI;
  sx = -dra / G.fp_delta + G.fp_x0;
  sy = ddec / G.fp_delta + G.fp_y0;
}

// An event left to sky_reference.
struct EvLate {
  double mnc[3];
  uint32_t k, drow;
};

// The dither state of an event (read_dither_value): zero for an undithered
// run or a column the run does not have.
__device__ __forceinline__ float dither_value(const EvArgs &a, const float *col, uint32_t drow) {
  return a.p.dithered && col ? col[drow] : 0.0f;
}

__device__ __forceinline__ void late_event(const EvArgs &a, const EvGeom &G, const EvLate &l) {
  double sx, sy;
  sky_reference(G, mk(l.mnc[0], l.mnc[1], l.mnc[2]), dither_value(a, a.e.sky_ra, l.drow),
                dither_value(a, a.e.sky_dec, l.drow), dither_value(a, a.e.sky_roll, l.drow), sx, sy);
  if (a.e.x) a.e.x[l.k] = sx;
  if (a.e.y) a.e.y[l.k] = sy;
}

// Inclusive max-scan of v over the block (EV_BLOCK threads).
__device__ __forceinline__ uint32_t block_max_scan(uint32_t v, uint32_t *sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    uint32_t o = __shfl_up_sync(0xffffffffu, v, d);
    if (lane >= d) v = max(v, o);
  }
  if (lane == 31) sh[warp] = v;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < EV_BLOCK / 32 ? sh[lane] : 0u;
#pragma unroll
    for (int d = 1; d < EV_BLOCK / 32; d <<= 1) {
      uint32_t o = __shfl_up_sync(0xffffffffu, w, d);
      if (lane >= d) w = max(w, o);
    }
    if (lane < EV_BLOCK / 32) sh[lane] = w;
  }
  __syncthreads();
  uint32_t r = warp ? max(v, sh[warp - 1]) : v;
  __syncthreads();
  return r;
}

// A frame starts at event k when k is the first event or its frame number
// differs from the previous event's: k then, else 0.  t: event k's time.
// The previous event's frame number comes from the lane below.
__device__ __forceinline__ uint32_t frame_start(const EvArgs &a, uint32_t k, int64_t frame) {
  const unsigned lo = __shfl_up_sync(0xffffffffu, (unsigned) frame, 1);
  const unsigned hi = __shfl_up_sync(0xffffffffu, (unsigned) ((unsigned long long) frame >> 32), 1);
  if (k >= a.e.n || k == 0) return 0u;
  int64_t before = (int64_t) (((unsigned long long) hi << 32) | lo);
  if ((threadIdx.x & 31) == 0) before = frame_number(a, event_time(a, row_of(a.e, k - 1)));
  return frame != before ? k : 0u;
}

// Last frame start of each tile of rounds x EV_BLOCK events.
__global__ void __launch_bounds__(EV_BLOCK) mx_event_frame_tiles(EvArgs a, uint32_t ntiles, uint32_t *tile_max) {
  __shared__ uint32_t sh[32];
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    uint32_t m = 0u;
    for (int r = 0; r < a.rounds; r++) {
      const uint32_t k = (t * a.rounds + r) * EV_BLOCK + threadIdx.x;
      const int64_t f = k < a.e.n ? frame_number(a, event_time(a, row_of(a.e, k))) : 0;
      m = max(m, frame_start(a, k, f));
    }
    m = block_max_scan(m, sh);
    if (threadIdx.x == EV_BLOCK - 1) tile_max[t] = m;
  }
}

// Exclusive max-scan over the tiles, in place (one block of 1024 threads).
__global__ void __launch_bounds__(1024) mx_event_frame_prefix(uint32_t ntiles, uint32_t *tile_max) {
  __shared__ uint32_t carry;
  __shared__ uint32_t sh[32];
  if (threadIdx.x == 0) carry = 0u;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t base = 0; base < ntiles; base += 1024) {
    const uint32_t i = base + threadIdx.x;
    uint32_t incl = i < ntiles ? tile_max[i] : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl = max(incl, o);
    }
    if (lane == 31) sh[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      uint32_t w = sh[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        uint32_t o = __shfl_up_sync(0xffffffffu, w, d);
        if (lane >= d) w = max(w, o);
      }
      sh[lane] = w;
    }
    __syncthreads();
    const uint32_t before = max(warp ? sh[warp - 1] : 0u, carry);   // everything ahead of this warp
    incl = max(incl, before);
    uint32_t excl = __shfl_up_sync(0xffffffffu, incl, 1);
    if (lane == 0) excl = before;
    __syncthreads();
    if (i < ntiles) tile_max[i] = excl;
    if (threadIdx.x == 1023) carry = incl;
    __syncthreads();
  }
}

// The columns of event k (list row `row`, frame number `frame`, dither state
// of event `first`); true, with `late` filled, when its sky columns are left
// to sky_reference.  last_roll, roll_s, roll_c: the thread's latest roll.
__device__ __forceinline__ bool event_columns(const EvArgs &a, const EvGeom &G, const EvFacet *facets, uint32_t k,
                                              uint32_t row, uint32_t first, int64_t frame, bool numbered,
                                              float &last_roll, F2 &roll_s, F2 &roll_c, EvLate &late) {
  const mx_events &e = a.e;
  const mx_event_params &p = a.p;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const uint32_t drow = row_of(e, first);
  const int ccd = e.ccd_id[row];
  const int fi = ccd - G.first_id;
  // read_float32_add_1 (marx2fits.c:3460-3470): CHIPX is xpixel + 1 in float
  const float chipx = e.xpixel[row] + 1.0f, chipy = e.ypixel[row] + 1.0f;
  if (e.chipx) e.chipx[k] = chipx;
  if (e.chipy) e.chipy[k] = chipy;
  // EXPNO (compute_expno): the frame number, or the event number less one
  // when there are no frames
  if (e.expno) e.expno[k] = G.acis ? (numbered ? (int32_t) frame : (int32_t) k - 1) : 0;
  if (fi < 0 || fi >= G.nf) {
    atomicAdd(a.bad, 1ull);
    if (e.detx) e.detx[k] = nan;
    if (e.dety) e.dety[k] = nan;
    if (e.x) e.x[k] = nan;
    if (e.y) e.y[k] = nan;
    if (e.tdetx) e.tdetx[k] = -1;
    if (e.tdety) e.tdety[k] = -1;
    if (e.fltgrade) e.fltgrade[k] = 0;
    if (e.grade) e.grade[k] = 0;
    return false;
  }
  const EvFacet &g = facets[fi];
  // FLTGRADE (compute_fltgrade, marx2fits.c:3854-3866) and GRADE (compute_grade)
  const float fx = floorf(chipx), fy = floorf(chipy);
  int fltgrade = 0;
  if (G.acis) {
    // (int) (3 (c - floor c)): the float fraction is exact, and the floats
    // at and above 1/3 and 2/3 are those whose triple reaches 1 and 2
    const float rx = chipx - fx, ry = chipy - fy;
    const int sx = (rx >= 0x1.555556p-2f) + (rx >= 0x1.555556p-1f), sy = (ry >= 0x1.555556p-2f) + (ry >= 0x1.555556p-1f);
    const double ux = e.uniforms ? e.uniforms[k] : event_uniform(a.seed, k, 0);
    // (int) (4 u), u = 1 stays in the row
    const int pick = lt_pos(ux, 1.0) ? (int) quarter_of(ux) : min((int) (4 * ux), 3);
    fltgrade = kFlightGrades[3 * sy + sx][pick];
  }
  if (e.fltgrade) e.fltgrade[k] = (int16_t) fltgrade;
  if (e.grade) e.grade[k] = (int16_t) (G.acis ? kGradeMap[fltgrade & 0xff] - '0' : 0);
  // TDETX, TDETY (compute_tdetxy; acis_i_to_tiled, acis_s_to_tiled,
  // acis_geom.c:106-135, 183-203; hrc_i_to_tiled, hrc_i_geom.c:215-233;
  // hrc_s_to_tiled, hrc_s_geom.c:476-514)
  if (e.tdetx || e.tdety) {
    const unsigned ix = (unsigned) chipx, iy = (unsigned) chipy;
    int tx, ty;
    if ((ix | iy) < (1u << 22)) {   // whole numbers that a float holds: the same on integers
      tx = g.tiled == 0 ? g.itdx + (int) iy : (g.tiled == 1 ? g.itdx - (int) iy : (int) ix + g.itdx);
      ty = g.tiled == 0 ? g.itdy - (int) ix : (g.tiled == 1 ? g.itdy + (int) ix : (int) iy + g.itdy);
      tx = max(tx, 0) + 1;
      ty = max(ty, 0) + 1;
    } else {
      float xf, yf;
      if (g.tiled == 0) { xf = (float) (g.tdx + iy); yf = (float) (g.tdy - ix); }
      else if (g.tiled == 1) { xf = (float) (g.tdx - iy); yf = (float) (g.tdy + ix); }
      else { xf = (float) (ix + g.tdx); yf = (float) (iy + g.tdy); }
      if (xf < 0.0f) xf = 0.0f;
      if (yf < 0.0f) yf = 0.0f;
      tx = (int32_t) ((unsigned) xf + 1u);
      ty = (int32_t) ((unsigned) yf + 1u);
    }
    if (e.tdetx) e.tdetx[k] = tx;
    if (e.tdety) e.tdety[k] = ty;
  }
  const float d_dy = dither_value(a, e.det_dy, drow), d_dz = dither_value(a, e.det_dz, drow),
              d_th = dither_value(a, e.det_theta, drow);
  // compute_detxy (marx2fits.c:3676-3736): chip pixel from 1-based CHIPX.
  // Below 2^22 the pixel centres are floats; larger values in double.
  const bool small = fabsf(chipx) < 0x1p22f && fabsf(chipy) < 0x1p22f;
  double x, y;
  if (p.pixel_adjust == MX_PIXADJ_EXACT) {
    x = f2d(chipx) - 1.0;
    y = f2d(chipy) - 1.0;
  } else if (p.pixel_adjust == MX_PIXADJ_RANDOMIZE) {
    const double u1 = e.uniforms ? e.uniforms[(size_t) e.n + k] : event_uniform(a.seed, k, 1);
    const double u2 = e.uniforms ? e.uniforms[2 * (size_t) e.n + k] : event_uniform(a.seed, k, 2);
    x = (small ? f2d(fx - 1.0f) : floor((double) chipx - 1.0)) + u1;
    y = (small ? f2d(fy - 1.0f) : floor((double) chipy - 1.0)) + u2;
  } else {
    x = small ? f2d(fx - 0.5f) : floor((double) chipx - 1.0) + 0.5;
    y = small ? f2d(fy - 0.5f) : floor((double) chipy - 1.0) + 0.5;
    if (p.pixel_adjust != MX_PIXADJ_NONE) {   // EDSER
      float dx, dy;
      subpix(G, ccd, e.b_energy ? e.b_energy[row] : 0.0f, fltgrade, dx, dy);
      x = x + f2d(dx);
      y = y + f2d(dy);
    }
  }
  // marx_init_chip_to_mnc (pixlib.c:135-198) with the detector offsets and
  // motion, then marx_chip_to_mnc (pixlib.c:201-222)
  D3 ofs = mk(g.ofs[0], g.ofs[1], g.ofs[2]), e1 = mk(g.e1[0], g.e1[1], g.e1[2]), e2 = mk(g.e2[0], g.e2[1], g.e2[2]);
  if (d_th != 0.0f || d_dy != 0.0f || d_dz != 0.0f) {
    double ct = 1.0, st = 0.0;
    if (d_th != 0.0f) { ct = cos((double) d_th); st = sin((double) d_th); }
    const double yoff = p.det_offset[1] + f2d(d_dy), zoff = p.det_offset[2] + f2d(d_dz);
    ofs.y = yoff + ct * g.x_ll[1] - st * g.x_ll[2];
    ofs.z = zoff + st * g.x_ll[1] + ct * g.x_ll[2];
    e1 = mk(g.xhat[0], ct * g.xhat[1] - st * g.xhat[2], st * g.xhat[1] + ct * g.xhat[2]);
    e2 = mk(g.yhat[0], ct * g.yhat[1] - st * g.yhat[2], st * g.yhat[1] + ct * g.yhat[2]);
    e1 = mk(g.xps * e1.x, g.xps * e1.y, g.xps * e1.z);
    e2 = mk(g.yps * e2.x, g.yps * e2.y, g.yps * e2.z);
  }
  if (!G.acis) { x -= g.xoff; y -= g.yoff; }   // an ACIS corner is pixel 0
  const D3 mnc = chip_direction(mk(ofs.x + e1.x * x + e2.x * y, ofs.y + e1.y * x + e2.y * y, ofs.z + e1.z * x + e2.z * y));
  // marx_mnc_to_fpc (detpix.c:182-208)
  double detx = nan, dety = nan;
  if (!is_zero(mnc.x)) {
    const double factor = __drcp_rn(G.fp_delta * mnc.x);
    detx = G.fp_x0 - factor * mnc.y;
    dety = G.fp_y0 + factor * mnc.z;
  } else {
    atomicAdd(a.bad, 1ull);
  }
  if (e.detx) e.detx[k] = detx;
  if (e.dety) e.dety[k] = dety;
  if (!e.x && !e.y) return false;
  // compute_xy_sky (marx2fits.c:3869-3910)
  double sx, sy;
  if (!p.dithered) {
    const double dx = detx - G.fp_x0, dy = dety - G.fp_y0;
    sx = G.fp_x0 + a.roll_c * dx + a.roll_s * dy;
    sy = G.fp_y0 - a.roll_s * dx + a.roll_c * dy;
  } else {
    const float d_roll = dither_value(a, e.sky_roll, drow);
    const bool turn = fabsf(d_roll) < 8.0f;
    if (turn && d_roll != last_roll) {   // one roll for a whole run under INTERNAL dither
      roll_sincos(d_roll, roll_s, roll_c);
      last_roll = d_roll;
    }
    if (!turn || !sky_offsets(a, G, mnc, dither_value(a, e.sky_ra, drow), dither_value(a, e.sky_dec, drow), roll_s,
                              roll_c, sx, sy)) {
      late.mnc[0] = mnc.x; late.mnc[1] = mnc.y; late.mnc[2] = mnc.z;
      late.k = k; late.drow = drow;
      return true;
    }
  }
  if (e.x) e.x[k] = sx;
  if (e.y) e.y[k] = sy;
  return false;
}

// One event per thread, tiles of rounds x EV_BLOCK events per block.
// FP64-bound as the chain DETX/DETY round through is (about 65 operations:
// 12 for the chip position, 41 for its direction, 11 for the focal plane)
// with the rest, the sky angles and sub-pixel tables among it, on the FP32
// and integer pipes; the facets are read from shared memory, where lanes on
// different chips do not serialise as they do in the constant bank.  Events
// left to sky_reference are gathered in shared memory and worked on 256 at
// a time, every lane busy, instead of by the odd lane of a quarter of the
// warps.  1e7 ACIS-I events (EDSER, frames): 14.1 -> 1.63 ms.
__global__ void __launch_bounds__(EV_BLOCK) mx_event_kernel(const __grid_constant__ EvArgs a,
                                                            const __grid_constant__ EvGeom G, uint32_t ntiles,
                                                            const uint32_t *tile_pre) {
  __shared__ uint32_t sh[32];
  __shared__ EvFacet facets[EV_MAX_FACETS];
  __shared__ EvLate list[2 * EV_BLOCK];
  __shared__ int count;
  for (int w = threadIdx.x; w < (int) (sizeof(facets) / 4); w += EV_BLOCK)
    ((uint32_t *) facets)[w] = ((const uint32_t *) G.f)[w];
  if (threadIdx.x == 0) count = 0;
  __syncthreads();
  const uint32_t n = a.e.n;
  const bool numbered = G.acis && a.p.frame_time > 0.0, sky = a.p.dithered && (a.e.x || a.e.y);
  float last_roll = u2f(0x7fc00000u);   // NaN never equals a roll: the first event computes
  F2 roll_s = {0.0f, 0.0f}, roll_c = {1.0f, 0.0f};
  for (uint32_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    uint32_t before = a.frames ? tile_pre[t] : 0u;   // the last frame start ahead of the round
    for (int r = 0; r < a.rounds; r++) {
      const uint32_t k = (t * a.rounds + r) * EV_BLOCK + threadIdx.x;
      const uint32_t row = k < n ? row_of(a.e, k) : 0u;
      const int64_t frame = numbered && k < n ? frame_number(a, event_time(a, row)) : 0;
      uint32_t first = k;   // the event whose dither state this event uses
      if (a.frames) {
        first = max(block_max_scan(frame_start(a, k, frame), sh), before);
        if (threadIdx.x == EV_BLOCK - 1) sh[31] = first;
      }
      EvLate late;
      if (k < n && event_columns(a, G, facets, k, row, first, frame, numbered, last_roll, roll_s, roll_c, late))
        list[atomicAdd(&count, 1)] = late;   // count stays below 2 EV_BLOCK
      if (!sky && !a.frames) continue;
      __syncthreads();
      before = sh[31];
      const int c = count;
      if (c >= EV_BLOCK) {
        late_event(a, G, list[c - EV_BLOCK + threadIdx.x]);
        __syncthreads();
        if (threadIdx.x == 0) count = c - EV_BLOCK;
      }
      __syncthreads();
    }
  }
  __syncthreads();
  if ((int) threadIdx.x < count) late_event(a, G, list[threadIdx.x]);
}

// The facets, focal-plane system and sub-pixel tables of the context's
// detector.
struct EvTables {
  EvGeom G;
  std::vector<char> blob;
  size_t o_sp = 0, o_row = 0, o_n = 0;
};

static bool event_tables(const mx_context *c, EvTables &out, std::string &err) {
  const mx_config &cfg = c->cfg;
  const HostModel &M = c->hm;
  EvGeom &G = out.G;
  memset(&G, 0, sizeof(G));
  const double arcsec = PI / (3600.0 * 180.0);
  // AXAF-FP-1.1 (ACIS), AXAF-FP-2.1 (HRC-I), AXAF-FP-2.3 (HRC-S)
  // (Focal_Plane_Coord_Info, detpix.c:42-63)
  switch (cfg.detector) {
    case MX_DETECTOR_ACIS_I:
    case MX_DETECTOR_ACIS_S: G.fp_delta = 0.492 * arcsec; G.fp_x0 = G.fp_y0 = 4096.5; G.acis = 1; break;
    case MX_DETECTOR_HRC_I: G.fp_delta = 0.13175 * arcsec; G.fp_x0 = G.fp_y0 = 16384.5; break;
    case MX_DETECTOR_HRC_S: G.fp_delta = 0.1318 * arcsec; G.fp_x0 = G.fp_y0 = 32768.5; break;
    default: err = "event coordinates need an ACIS or HRC detector"; return false;
  }
  const MxTables &T = M.T;
  G.nf = T.nchips;
  if (G.nf < 1 || G.nf > EV_MAX_FACETS) { err = "detector without facets"; return false; }
  G.first_id = M.chips[T.chip_off].id;
  // tiled offsets (acis_geom.c:37-47, hrc_i_geom.c:136-137, hrc_s_geom.c:321-328)
  static const double acis_i_tx[4] = {3061, 5131, 3061, 5131}, acis_i_ty[4] = {5131, 4107, 4085, 3061};
  static const double acis_s_tx[6] = {791, 1833, 2875, 3917, 4959, 6001};
  static const double hrc_s_ty[3] = {-12.0, 16444.0, 32900.0};
  for (int i = 0; i < G.nf; i++) {
    const MxChipDev &ch = M.chips[T.chip_off + i];
    if (ch.id != G.first_id + i) { err = "facet ids are not consecutive"; return false; }
    EvFacet &f = G.f[i];
    memcpy(f.x_ll, ch.x_ll, sizeof(f.x_ll));
    memcpy(f.xhat, ch.xhat, sizeof(f.xhat));
    memcpy(f.yhat, ch.yhat, sizeof(f.yhat));
    f.tiled = 2;
    if (G.acis) {
      // tweak_acis_pixel_size (acis_geom.c:54-66); the LL corner is pixel 0
      f.xps = ch.xlen / 1024.0; f.yps = ch.ylen / 1024.0;
      if (cfg.detector == MX_DETECTOR_ACIS_I) {
        f.tdx = acis_i_tx[ch.id]; f.tdy = acis_i_ty[ch.id];
        f.tiled = (ch.id == 0 || ch.id == 2) ? 0 : 1;
      } else {
        f.tdx = acis_s_tx[ch.id - 4]; f.tdy = 1702;
      }
    } else {
      // 6.429 micron pixels (hrc_i_geom.c:277-278, hrc_s_geom.c:559-560)
      f.xps = f.yps = 6.429e-3;
      const MxHrcDev &h = T.hrc;
      if (cfg.detector == MX_DETECTOR_HRC_I) {
        f.xoff = h.ll_cxcy[0]; f.yoff = h.ll_cxcy[1];   // LL_CXCY (hrc_i_geom.c:139-140)
        f.tdx = -1.0; f.tdy = 0.0;
      } else {
        // _marx_hrc_s_compute_pixel (hrc_s_geom.c:343-392) at the LL corner
        const double u = h.u_active0 + 0.0 / h.pix[0], v = h.v_active0[i] + 0.0 / h.pix[1];
        f.xoff = h.cxcy0[i][0] + (u - h.uv0[i][0]);
        f.yoff = h.cxcy0[i][1] + (v - h.uv0[i][1]);
        f.tdx = 0.0; f.tdy = hrc_s_ty[i];
      }
    }
    for (int r = 0; r < 3; r++) { f.e1[r] = f.xps * f.xhat[r]; f.e2[r] = f.yps * f.yhat[r]; }
    f.itdx = (int32_t) f.tdx;
    f.itdy = (int32_t) f.tdy;
  }
  // ACIS sub-pixel offsets (read_subpix_ext, acis_subpix.c:96-186)
  std::vector<float> sp;
  std::vector<int32_t> row(512, -1), npts(512, 0);
  if (G.acis) {
    const char *kinds[2] = {"acis/subpix_fi", "acis/subpix_bi"};
    for (int kd = 0; kd < 2; kd++) {
      size_t ni, nt;
      const int32_t *idx = c->pack.get<int32_t>(std::string(kinds[kd]) + "/rows", &ni, err);
      const float *tab = c->pack.get<float>(std::string(kinds[kd]) + "/table", &nt, err);
      if (!idx || !tab) return false;
      // rows: (fltgrade, npoints) pairs; table: per row energies, dx, dy of `rep` floats
      const size_t nrows = ni / 2;
      if (nrows == 0 || nt % (3 * nrows)) { err = kinds[kd] + std::string(": malformed"); return false; }
      const size_t rep = nt / (3 * nrows);
      for (size_t r = 0; r < nrows; r++) {
        const int fg = idx[2 * r], np = idx[2 * r + 1];
        if (fg < 0 || fg >= 256) { err = "Illegal flight grade in subpix column"; return false; }
        if (np <= 0) { row[kd * 256 + fg] = -1; continue; }
        if (np == 1) { err = "Expecting Number of points (NPOINTS) to be greater than 1"; return false; }
        if ((size_t) np > rep) { err = "NPOINTS is greater than repeat count"; return false; }
        row[kd * 256 + fg] = (int32_t) sp.size();
        npts[kd * 256 + fg] = np;
        for (int w = 0; w < 3; w++) {
          const float *src = tab + (w * nrows + r) * rep;
          sp.insert(sp.end(), src, src + np);
        }
      }
    }
  }
  if (sp.empty()) sp.push_back(0.0f);
  auto put = [&](const void *d, size_t bytes) {
    size_t off = (out.blob.size() + 255) & ~(size_t) 255;
    out.blob.resize(off + bytes);
    memcpy(out.blob.data() + off, d, bytes);
    return off;
  };
  out.o_sp = put(sp.data(), sp.size() * sizeof(float));
  out.o_row = put(row.data(), row.size() * sizeof(int32_t));
  out.o_n = put(npts.data(), npts.size() * sizeof(int32_t));
  return true;
}

static int ensure_event_tables(mx_context *c) {
  if (c->events_ready) return MX_OK;
  EvTables t;
  std::string err;
  if (!event_tables(c, t, err)) return mx_fail(c, MX_EINVAL, err);
  cudaError_t e = c->ev_tab.ensure(t.blob.size());
  if (e == cudaSuccess) e = cudaMemcpy(c->ev_tab.ptr, t.blob.data(), t.blob.size(), cudaMemcpyHostToDevice);
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "uploading the event tables");
  char *b = (char *) c->ev_tab.ptr;
  t.G.sp = (const float *) (b + t.o_sp);
  t.G.sp_row = (const int32_t *) (b + t.o_row);
  t.G.sp_n = (const int32_t *) (b + t.o_n);
  static_assert(sizeof(EvGeom) <= sizeof(c->ev_geom), "event geometry larger than its slot");
  memcpy(c->ev_geom, &t.G, sizeof(EvGeom));
  c->events_ready = true;
  return MX_OK;
}

static int check_params(mx_context *c, const mx_event_params *p, const mx_events *ev) {
  if (!p || !ev) return mx_fail(c, MX_EINVAL, "mx_event_coords: null argument");
  if (ev->n == 0) return MX_OK;
  if (!ev->ccd_id || !ev->xpixel || !ev->ypixel) return mx_fail(c, MX_EINVAL, "mx_event_coords: ccd_id, xpixel and ypixel are required");
  if (!ev->time && !ev->time64) return mx_fail(c, MX_EINVAL, "mx_event_coords: no time column");
  if (p->pixel_adjust < MX_PIXADJ_EDSER || p->pixel_adjust > MX_PIXADJ_EXACT)
    return mx_fail(c, MX_EINVAL, "mx_event_coords: unknown pixel adjustment");
  if (!(p->focal_length > 0)) return mx_fail(c, MX_EINVAL, "mx_event_coords: focal length must be positive");
  return MX_OK;
}

static int launch_events(mx_context *c, const mx_event_params *params, const mx_events *ev, uint64_t seed, cudaStream_t st) {
  int rc = ensure_event_tables(c);
  if (rc != MX_OK) return rc;
  EvGeom G;
  memcpy(&G, c->ev_geom, sizeof(EvGeom));
  EvArgs a;
  a.e = *ev;
  a.p = *params;
  // marx2fits turns EDSER into RANDOMIZE for an HRC (marx2fits.c:3307-3308)
  if (!G.acis && a.p.pixel_adjust == MX_PIXADJ_EDSER) a.p.pixel_adjust = MX_PIXADJ_RANDOMIZE;
  a.seed = seed;
  const double theta = params->roll_nom * PI / 180.0;
  a.roll_c = cos(theta);
  a.roll_s = sin(theta);
  a.frames = G.acis && a.p.dithered && a.p.frame_time > 0.0 && a.p.pixel_adjust != MX_PIXADJ_EXACT;
  a.bad = c->d_event_bad;
  for (int i = 0; i < G.nf; i++) {
    EvFacet &f = G.f[i];
    f.ofs[0] = params->det_offset[0] - params->focal_length;
    f.ofs[1] = params->det_offset[1] + f.x_ll[1];
    f.ofs[2] = params->det_offset[2] + f.x_ll[2];
  }
  const double inv_frame = a.p.frame_time > 1e-9 && a.p.frame_time < 1e9 ? 1.0 / a.p.frame_time : std::nan("");
  a.inv_frame[0] = (float) inv_frame;
  a.inv_frame[1] = (float) (inv_frame - (double) a.inv_frame[0]);
  a.inv_delta[0] = (float) (1.0 / G.fp_delta);
  a.inv_delta[1] = (float) (1.0 / G.fp_delta - (double) a.inv_delta[0]);
  // tiles of one round spread a short list over the SMs; long lists take
  // four, a quarter of the tiles for the one-block scan over them
  a.rounds = ev->n >= (uint32_t) c->num_sms * 8 * 4 * EV_BLOCK ? 4 : 1;
  const uint32_t tile = (uint32_t) a.rounds * EV_BLOCK, ntiles = (uint32_t) (((uint64_t) ev->n + tile - 1) / tile);
  const uint32_t grid = (uint32_t) std::min<uint64_t>(ntiles, (uint64_t) c->num_sms * 8);
  uint32_t *tiles = nullptr;
  if (a.frames) {
    cudaError_t e = c->ev_scan.ensure((size_t) ntiles * sizeof(uint32_t));
    if (e == cudaSuccess) e = c->ev_turn.before(st);
    if (e != cudaSuccess) return mx_cuda_fail(c, e, "allocating the frame scan");
    tiles = (uint32_t *) c->ev_scan.ptr;
    mx_event_frame_tiles<<<grid, EV_BLOCK, 0, st>>>(a, ntiles, tiles);
    mx_event_frame_prefix<<<1, 1024, 0, st>>>(ntiles, tiles);
    c->launches += 2;
  }
  mx_event_kernel<<<grid, EV_BLOCK, 0, st>>>(a, G, ntiles, tiles);
  c->launches += 1;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && a.frames) e = c->ev_turn.after(st);
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "launching the event pass");
  return MX_OK;
}

}  // namespace mx_ev

using namespace mx_ev;

extern "C" {

int mx_event_coords(mx_context *c, const mx_event_params *params, const mx_events *ev, uint64_t seed, void *stream) {
  if (!c) return MX_EINVAL;
  int rc = check_params(c, params, ev);
  if (rc != MX_OK || ev->n == 0) return rc;
  return launch_events(c, params, ev, seed, (cudaStream_t) stream);
}

int mx_event_coords_host(mx_context *c, const mx_event_params *params, const mx_events *h, uint64_t seed) {
  if (!c) return MX_EINVAL;
  int rc = check_params(c, params, h);
  if (rc != MX_OK || h->n == 0) return rc;
  const size_t n = h->n;
  size_t rows = n;   // input rows: the largest index + 1
  if (h->index) {
    uint32_t m = 0;
    for (size_t k = 0; k < n; k++) m = std::max(m, h->index[k]);
    rows = (size_t) m + 1;
  }
  struct In { const void *src; size_t bytes; const void **dst; };
  mx_events d = *h;
  std::vector<In> ins = {
      {h->index, n * 4, (const void **) &d.index},       {h->ccd_id, rows, (const void **) &d.ccd_id},
      {h->xpixel, rows * 4, (const void **) &d.xpixel},  {h->ypixel, rows * 4, (const void **) &d.ypixel},
      {h->time, rows * 4, (const void **) &d.time},      {h->time64, rows * 8, (const void **) &d.time64},
      {h->sky_ra, rows * 4, (const void **) &d.sky_ra},  {h->sky_dec, rows * 4, (const void **) &d.sky_dec},
      {h->sky_roll, rows * 4, (const void **) &d.sky_roll}, {h->det_dy, rows * 4, (const void **) &d.det_dy},
      {h->det_dz, rows * 4, (const void **) &d.det_dz},  {h->det_theta, rows * 4, (const void **) &d.det_theta},
      {h->b_energy, rows * 4, (const void **) &d.b_energy}, {h->uniforms, 3 * n * 8, (const void **) &d.uniforms}};
  struct Out { void *dst; size_t bytes; void **dev; };
  std::vector<Out> outs = {
      {h->chipx, n * 4, (void **) &d.chipx}, {h->chipy, n * 4, (void **) &d.chipy},
      {h->detx, n * 8, (void **) &d.detx},   {h->dety, n * 8, (void **) &d.dety},
      {h->x, n * 8, (void **) &d.x},         {h->y, n * 8, (void **) &d.y},
      {h->tdetx, n * 4, (void **) &d.tdetx}, {h->tdety, n * 4, (void **) &d.tdety},
      {h->expno, n * 4, (void **) &d.expno}, {h->fltgrade, n * 2, (void **) &d.fltgrade},
      {h->grade, n * 2, (void **) &d.grade}};
  size_t total = 0;
  auto align = [](size_t b) { return (b + 255) & ~(size_t) 255; };
  for (auto &i : ins) if (i.src) total += align(i.bytes);
  for (auto &o : outs) if (o.dst) total += align(o.bytes);
  cudaError_t e = c->ev_io.ensure(total);
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "allocating event staging");
  cudaStream_t st = c->stream;
  char *b = (char *) c->ev_io.ptr;
  size_t off = 0;
  unsigned long long bad0 = 0;
  e = cudaMemcpyAsync(&bad0, c->d_event_bad, sizeof(bad0), cudaMemcpyDeviceToHost, st);
  for (auto &i : ins) {
    if (!i.src || e != cudaSuccess) continue;
    *i.dst = b + off;
    e = cudaMemcpyAsync(b + off, i.src, i.bytes, cudaMemcpyHostToDevice, st);
    off += align(i.bytes);
  }
  for (auto &o : outs) {
    if (!o.dst) continue;
    *o.dev = b + off;
    off += align(o.bytes);
  }
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "copying events to the device");
  rc = launch_events(c, params, &d, seed, st);
  if (rc != MX_OK) return rc;
  for (auto &o : outs) {
    if (!o.dst || e != cudaSuccess) continue;
    e = cudaMemcpyAsync(o.dst, *o.dev, o.bytes, cudaMemcpyDeviceToHost, st);
  }
  unsigned long long bad1 = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&bad1, c->d_event_bad, sizeof(bad1), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "event pass");
  if (bad1 != bad0) return mx_fail(c, MX_EINVAL, "event with a chip id outside the detector or without a focal-plane position");
  return MX_OK;
}

int mx_event_bad_count(mx_context *c, unsigned long long *count, int reset) {
  if (!c || !count) return MX_EINVAL;
  cudaError_t e = cudaMemcpy(count, c->d_event_bad, sizeof(*count), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && reset) e = cudaMemset(c->d_event_bad, 0, sizeof(unsigned long long));
  if (e != cudaSuccess) return mx_cuda_fail(c, e, "reading the bad-event counter");
  return MX_OK;
}

}  // extern "C"
