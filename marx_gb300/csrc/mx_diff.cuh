// Weighted-ray trace for the differentiable form.
//
// A weighted ray takes the aperture point a photon of the same tag would
// take in the plain trace (project_photon_to_hrma, hrma.c:984-1050), then
// follows the HRMA geometry (compute_conic_intersection hrma.c:411-478,
// reflect_from_conic hrma.c:488-545, _marx_hrma_mirror_reflect
// hrma.c:1183-1339) without normal blur or scattering, and is projected
// onto the focal plane x = 0.  Instead of being absorbed at random it
// carries a weight: vignetting times, at each reflection, the Fresnel
// reflectivity (reflect.c:39-77) times the effective-area correction.
//
// The values are FP64; the derivatives with respect to the parameters that can
// move a ray (its shell's two tilts and two decenters and the source's two
// angular offsets) are FP32: Dual6 carries both through the geometry that the
// host prepares, the adjoint kernel traces them ray by ray.
#pragma once
#include <stdint.h>

#include <cmath>

#include "mx_device.cuh"

#ifdef __CUDACC__
#define MXG __host__ __device__ __forceinline__
#else
#define MXG inline
#endif

namespace mxd {

constexpr int ND = 6;   // tangent slots: tilt az, tilt el, decenter x, decenter y, source y, source z

// A number with its derivatives, for the geometry that the host prepares.
struct Dual6 {
  double v;
  float d[ND];
};

inline Dual6 mkd(double v) {
  Dual6 r; r.v = v;
  for (int k = 0; k < ND; k++) r.d[k] = 0.f;
  return r;
}
// f(a) with value v and slope s
inline Dual6 chain(double v, float s, const Dual6 &a) {
  Dual6 r; r.v = v;
  for (int k = 0; k < ND; k++) r.d[k] = s * a.d[k];
  return r;
}
inline Dual6 operator+(const Dual6 &a, const Dual6 &b) {
  Dual6 r; r.v = a.v + b.v;
  for (int k = 0; k < ND; k++) r.d[k] = a.d[k] + b.d[k];
  return r;
}
inline Dual6 operator-(const Dual6 &a, const Dual6 &b) {
  Dual6 r; r.v = a.v - b.v;
  for (int k = 0; k < ND; k++) r.d[k] = a.d[k] - b.d[k];
  return r;
}
inline Dual6 operator*(const Dual6 &a, const Dual6 &b) {
  Dual6 r; r.v = a.v * b.v;
  const float av = (float) a.v, bv = (float) b.v;
  for (int k = 0; k < ND; k++) r.d[k] = av * b.d[k] + bv * a.d[k];
  return r;
}
inline Dual6 operator*(const Dual6 &a, double s) { return chain(s * a.v, (float) s, a); }
inline Dual6 operator+(double s, const Dual6 &a) { return chain(s + a.v, 1.0f, a); }
inline Dual6 operator-(double s, const Dual6 &a) { return chain(s - a.v, -1.0f, a); }
inline Dual6 dsin(const Dual6 &a) { return chain(std::sin(a.v), cosf((float) a.v), a); }
inline Dual6 dcos(const Dual6 &a) { return chain(std::cos(a.v), -sinf((float) a.v), a); }
inline Dual6 dtan(const Dual6 &a) {
  const float t = (float) std::tan(a.v);
  return chain(std::tan(a.v), 1.0f + t * t, a);
}
inline Dual6 drsqrt(const Dual6 &a) {
  const float t = (float) mx::mx_rsqrt(a.v);
  return chain(mx::mx_rsqrt(a.v), -0.5f * t * t * t, a);
}

// ------------------------------------------------ HRMA optic geometry --
// One optic of one shell: the MARX -> optic translation `to` and the
// pitch/yaw rotations fwd (into the optic's frame) and bwd (back).
struct Optic {
  Dual6 to[3], fwd[9], bwd[9];
  Dual6 ff[3];   // fwd (front + to[0], 0, 0): the aperture plane's part of fwd (x + to)
};

// A shell's way from the paraboloid's frame to the hyperboloid's: back to
// the MARX frame (P.bwd, less P.to), then in (plus H.to, H.fwd) as one
// matrix and offset, x' = m x + c, p' = m p, with m = H.fwd P.bwd and
// c = H.fwd (H.to - P.to); and the source direction in the paraboloid's
// frame, p1 = P.fwd p0.
struct Between {
  Dual6 m[9], c[3], p1[3];
};

// The rotation builders of init_yaw_pitch (hrma.c:842-880).
inline void rot_z(Dual6 m[9], const Dual6 &theta) {
  Dual6 c = dcos(theta), s = 0.0 - dsin(theta);
  m[0] = c; m[1] = s; m[2] = mkd(0.0);
  m[3] = 0.0 - s; m[4] = c; m[5] = m[2];
  m[6] = m[2]; m[7] = m[2]; m[8] = mkd(1.0);
}
inline void rot_axis(Dual6 m[9], const Dual6 n[3], const Dual6 &theta) {
  Dual6 c = dcos(theta), s = dsin(theta), c1 = 1.0 - c;
  Dual6 n0 = n[0], n1 = n[1], n2 = n[2];
  Dual6 n01 = n0 * n1 * c1, n02 = n0 * n2 * c1, n12 = n1 * n2 * c1;
  m[0] = n0 * n0 * c1 + c; m[1] = n01 - s * n2; m[2] = n02 + s * n1;
  m[3] = n01 + s * n2; m[4] = n1 * n1 * c1 + c; m[5] = n12 - s * n0;
  m[6] = n02 - s * n1; m[7] = n12 + s * n0; m[8] = n2 * n2 * c1 + c;
}
inline void mat3_mul(Dual6 c[9], const Dual6 a[9], const Dual6 b[9]) {
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) c[3 * i + j] = a[3 * i] * b[j] + a[3 * i + 1] * b[3 + j] + a[3 * i + 2] * b[6 + j];
}
// fwd = R(ny, -el) Rz(-az) and bwd = Rz(az) R(ny, el), ny = Rz(-az) e_y, as
// the reference builds them from the geometry file's az_mis and el_mis.
inline void yaw_pitch(Dual6 fwd[9], Dual6 bwd[9], const Dual6 &az, const Dual6 &el) {
  Dual6 rz[9], ry[9], ny[3];
  rot_z(rz, 0.0 - az);
  ny[0] = rz[1]; ny[1] = rz[4]; ny[2] = rz[7];
  rot_axis(ry, ny, 0.0 - el);
  mat3_mul(fwd, ry, rz);
  rot_axis(ry, ny, el);
  rot_z(rz, az);
  mat3_mul(bwd, rz, ry);
}

// Per-ray decision byte: what the ray did the last time it was traced
// afresh.  Replaying it keeps the traced function smooth in the parameters.
enum : uint8_t { RAY_HIT = 1, RAY_ROOT_P = 2, RAY_ROOT_H = 4 };

#ifdef __CUDACC__
// compute_conic_intersection (hrma.c:411-478) with the roots of
// JDMquadratic_root (qroot.c:36-70), in double, for the few rays conic_root
// leaves to it.  root < 0: choose as the reference does (a root inside
// [xmin, xmax), the larger x when both are); 0 = the -2c/(b f) root, 1 = the
// -b f/(2a) root: take that root without the x-limit test, so that the ray
// stays on the same branch while the optic moves.  The root taken, -1 for a
// miss.
static __device__ __noinline__ int conic_root_double(const MxShellDev &h, int o, mx::D3 &x, const mx::D3 &p, mx::D3 &n,
                                                     int root) {
  const double t_plus = -x.x * mx::rcp_fast(p.x);
  const double x_y = x.y + t_plus * p.y, x_z = x.z + t_plus * p.z;
  const double alpha = h.a[o] * (p.x * p.x) - 1.0;
  const double beta = h.b[o] * p.x - 2.0 * (p.y * x_y + p.z * x_z);
  const double gamma = h.c[o] - x_z * x_z - x_y * x_y;
  if (mx::is_zero(alpha)) return -1;
  const double bsqr = beta * beta, ac4 = alpha * gamma * 4.0;
  if (!(mx::dkey(ac4) < mx::dkey(bsqr))) return -1;
  // the roots -2 gamma / (beta f) and -beta f / (2 alpha) of the reference,
  // f = 1 + sqrt(1 - 4 alpha gamma / beta^2), from b f = beta + sign(beta)
  // sqrt(beta^2 - 4 alpha gamma) and one reciprocal of alpha b f
  const double bf = beta + copysign(sqrt(bsqr - ac4), beta), inv = mx::rcp_fast(alpha * bf);
  const double tp = (-2.0 * gamma) * alpha * inv, tm = (-0.5 * bf) * bf * inv;
  if (root < 0) {
    const double xp = p.x * tp, xm = p.x * tm;
    const bool okp = xp >= h.xmin[o] && xp < h.xmax[o], okm = xm >= h.xmin[o] && xm < h.xmax[o];
    if (!okp && !okm) return -1;
    root = okp && !(okm && xp < xm) ? 0 : 1;
  }
  const double t = root ? tm : tp;
  x = mx::mk(p.x * t, x_y + p.y * t, x_z + p.z * t);
  n = mx::mk((h.a[o] - 1.0) * x.x + 0.5 * h.b[o], -x.y, -x.z);
  n = mx::mx_rsqrt(mx::dot(n, n)) * n;
  return root;
}

// The same for a ray as the trace meets it, by Newton steps from the one
// crossing between the conic's ends (mx::conic_newton).  That crossing is
// root 0, the intersection nearer to the plane x = 0, when the sum of both,
// -beta / alpha, is more than twice as far from zero (in float, with room to
// spare: beta / alpha is of the order of 1e5 mm).  A ray without such a
// crossing certainly misses if it is not replayed and the screen says so;
// all others, those that follow root 1 among them, take the double form.
__device__ __forceinline__ int conic_root(const MxShellDev &h, int o, mx::D3 &x, const mx::D3 &p, mx::D3 &n, int root) {
  if (root <= 0) {
    mx::D3 r = x, m;
    const int hit = mx::conic_newton(h, o, r, p, m);
    if (hit > 0) {
      const float inv = 1.0f / mx::d2f_trunc(p.x), my = mx::d2f_trunc(p.y) * inv, mz = mx::d2f_trunc(p.z) * inv;
      const float xf = mx::d2f_trunc(r.x), m2 = fmaf(my, my, mz * mz), alpha = m2 - h.am1f[o];
      const float beta = fmaf(2.0f, fmaf(mx::d2f_trunc(r.y), my, mx::d2f_trunc(r.z) * mz) - xf * m2, -h.bf[o]);
      if (fabsf(beta) > fmaf(2.5f, fabsf(alpha * xf), 0.01f)) { x = r; n = m; return 0; }
    } else if (hit < 0 && root < 0)
      return -1;
  }
  return conic_root_double(h, o, x, p, n, root);
}

// p - 2 (p.n) n
__device__ __forceinline__ mx::D3 reflected(const mx::D3 &p, const mx::D3 &n, double pdn) {
  const double k = -2.0 * pdn;
  return mx::mk(fma(k, n.x, p.x), fma(k, n.y, p.y), fma(k, n.z, p.z));
}
// ------------------------------------------- the adjoint's arithmetic --
// A value of a recorded ray with its single-precision tangents in the four
// directions that bend its path: the shell's tilts (0, 1) and the source's
// offsets (2, 3); the decenters move both optics alike and shift the image
// alone.  Turn: an entry of the geometry, which only the tilts move.
constexpr int NT = 4;
struct Dual { double v; float d[NT]; };
struct Turn { double v; float d[2]; };

// A value rounded to single precision for the tangents: by truncation on the
// integer pipe (a conversion instruction would take an FP64-pipe slot).
__device__ __forceinline__ float tof(double x) { return mx::d2f_trunc(x); }
// The truncation of a double-float.
__device__ __forceinline__ float tof(mx::F2 a) {
  a = mx::quick_sum(a.h, a.l);
  const uint32_t u = __float_as_uint(a.h);
  return __uint_as_float(u - ((a.l != 0.0f && ((u ^ __float_as_uint(a.l)) >> 31)) ? 1u : 0u));
}

__device__ __forceinline__ Dual operator+(const Dual &a, const Dual &b) {
  Dual r; r.v = a.v + b.v;
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = a.d[k] + b.d[k];
  return r;
}
__device__ __forceinline__ Dual operator-(const Dual &a, const Dual &b) {
  Dual r; r.v = a.v - b.v;
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = a.d[k] - b.d[k];
  return r;
}
__device__ __forceinline__ Dual operator-(const Dual &a) {
  Dual r; r.v = -a.v;
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = -a.d[k];
  return r;
}
__device__ __forceinline__ Dual operator*(const Dual &a, const Dual &b) {
  Dual r; r.v = a.v * b.v;
  const float av = tof(a.v), bv = tof(b.v);
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = av * b.d[k] + bv * a.d[k];
  return r;
}
__device__ __forceinline__ Dual operator*(double s, const Dual &a) {
  Dual r; r.v = s * a.v;
  const float f = tof(s);
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = f * a.d[k];
  return r;
}
__device__ __forceinline__ Dual operator+(const Dual &a, double s) { Dual r = a; r.v = a.v + s; return r; }
__device__ __forceinline__ Dual operator-(const Dual &a, double s) { Dual r = a; r.v = a.v - s; return r; }
__device__ __forceinline__ Dual operator-(double s, const Dual &a) { Dual r = -a; r.v = s - a.v; return r; }
__device__ __forceinline__ Dual operator*(const Turn &a, const Dual &b) {
  Dual r; r.v = a.v * b.v;
  const float av = tof(a.v), bv = tof(b.v);
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = k < 2 ? av * b.d[k] + bv * a.d[k & 1] : __fmul_rn(av, b.d[k]);   // as with a zero a.d
  return r;
}
// a + b y + c z, the aperture point (0, y, z) in a turned frame
__device__ __forceinline__ Dual turned(const Turn &a, const Turn &b, const Turn &c, double y, double z) {
  Dual r; r.v = a.v + b.v * y + c.v * z;
  const float yf = tof(y), zf = tof(z);
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = k < 2 ? a.d[k & 1] + yf * b.d[k & 1] + zf * c.d[k & 1] : 0.0f;
  return r;
}
__device__ __forceinline__ Dual operator+(const Dual &a, const Turn &b) {
  Dual r = a; r.v = a.v + b.v;
  r.d[0] += b.d[0]; r.d[1] += b.d[1];
  return r;
}
// 1 / a, sqrt(a) and 1 / sqrt(a): Newton steps from a float seed (within one
// ulp); sizes outside 2^-39 .. 2^39, which no ray of a mirror meets, take the
// library's.
__device__ __forceinline__ bool usual(double a) { return (unsigned) (mx::dbits(a) >> 52) - (1023u - 39u) < 78u; }
static __device__ __noinline__ double rsqrt_library(double a) { return rsqrt(a); }
static __device__ __noinline__ double sqrt_library(double a) { return sqrt(a); }
__device__ __forceinline__ Dual drcp(const Dual &a) {
  Dual r; r.v = mx::rcp_fast(a.v);
  const float g = -tof(r.v) / tof(a.v);
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = g * a.d[k];
  return r;
}
__device__ __forceinline__ Dual dsqrt(const Dual &a) {
  Dual r; r.v = usual(a.v) ? a.v * mx::rsqrt_seeded(a.v) : sqrt_library(a.v);
  const float h = 0.5f / tof(r.v);
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = h * a.d[k];
  return r;
}
__device__ __forceinline__ Dual drsqrt(const Dual &a) {
  Dual r; r.v = usual(a.v) ? mx::rsqrt_seeded(a.v) : rsqrt_library(a.v);
  const float t = tof(r.v), h = -0.5f * t * t * t;
#pragma unroll
  for (int k = 0; k < NT; k++) r.d[k] = h * a.d[k];
  return r;
}

struct V3 { Dual x, y, z; };
__device__ __forceinline__ Dual dotp(const V3 &a, const V3 &b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 matv(const Turn *m, const V3 &v) {
  return {m[0] * v.x + m[1] * v.y + m[2] * v.z, m[3] * v.x + m[4] * v.y + m[5] * v.z, m[6] * v.x + m[7] * v.y + m[8] * v.z};
}

// conic_root_double with tangents for a ray that follows a recorded root.
// False when the ray misses the conic.
__device__ __forceinline__ bool conic_tangents(const MxShellDev &h, int o, V3 &x0, const V3 &p, V3 &n, int root) {
  const Dual t_plus = (0.0 - x0.x) * drcp(p.x);
  const Dual x_y = x0.y + t_plus * p.y, x_z = x0.z + t_plus * p.z;
  const Dual alpha = h.a[o] * (p.x * p.x) - 1.0;
  const Dual beta = h.b[o] * p.x - 2.0 * (p.y * x_y + p.z * x_z);
  const Dual gamma = h.c[o] - x_z * x_z - x_y * x_y;
  if (mx::is_zero(alpha.v)) return false;
  const Dual bsqr = beta * beta, ac4 = 4.0 * (alpha * gamma);
  if (!(mx::dkey(ac4.v) < mx::dkey(bsqr.v))) return false;
  const Dual sq = dsqrt(bsqr - ac4), bf = mx::neg_bit(beta.v) ? beta - sq : beta + sq, inv = drcp(alpha * bf);
  Dual t;
  if (root == 0) t = (-2.0 * gamma) * alpha * inv;
  else t = (-0.5 * bf) * bf * inv;
  x0 = {p.x * t, x_y + p.y * t, x_z + p.z * t};
  n = {(h.a[o] - 1.0) * x0.x + 0.5 * h.b[o], -x0.y, -x0.z};
  const Dual len = drsqrt(dotp(n, n));
  n = {len * n.x, len * n.y, len * n.z};
  return true;
}

// The Fresnel reflectivity of mx::reflectivity_df for refractive index
// n, sr + i si = n^2 and lost = 1 - sr, with its derivative by the grazing
// cosine: one chain of single-precision tangents beside the double-float
// values instead of one for every direction beside double values.
struct Fresnel { mx::F2 sr, si, lost; };
__device__ __forceinline__ void fresnel_slope(const Fresnel &f, mx::F2 c, mx::F2 &value, float &slope) {
  using mx::F2;
  const float cf = tof(c);
  const F2 wr = mx::df_sub(mx::df_prod(c, c), f.lost), wi = f.si;
  const float wrd = 2.0f * cf;
  const F2 r = mx::df_sqrt(mx::df_sum(mx::df_prod(wr, wr), mx::df_prod(wi, wi)));
  const float rd = 0.5f / tof(r) * (2.0f * tof(wr) * wrd);
  const bool right = wr.h >= 0.0f;
  const F2 h2 = mx::df_sum(r, right ? wr : mx::df_neg(wr));
  const F2 h = mx::quick_sum(0.5f * h2.h, 0.5f * h2.l), inv = mx::df_rsqrt(h), hw = {0.5f * wi.h, 0.5f * wi.l};
  const float hd = 0.5f * (right ? rd + wrd : rd - wrd), invf = tof(inv), invd = -0.5f * invf * invf * invf * hd;
  const F2 big = mx::df_prod(h, inv), small = mx::df_prod(hw, inv);
  const float bigd = tof(h) * invd + invf * hd, smalld = tof(hw) * invd;
  F2 rr = right ? big : small, ri = right ? small : big;
  float rrd = right ? bigd : smalld, rid = right ? smalld : bigd;
  if (!right && rr.h < 0.0f) { rr = mx::df_neg(rr); ri = mx::df_neg(ri); rrd = -rrd; rid = -rid; }
  const F2 ri2 = mx::df_prod(ri, ri), cm = mx::df_sub(c, rr), cp = mx::df_sum(c, rr);
  const float ri2d = 2.0f * tof(ri) * rid;
  const F2 a1 = mx::df_sum(mx::df_prod(cm, cm), ri2), b1 = mx::df_sum(mx::df_prod(cp, cp), ri2);
  const float a1d = 2.0f * tof(cm) * (1.0f - rrd) + ri2d, b1d = 2.0f * tof(cp) * (1.0f + rrd) + ri2d;
  const F2 pr = mx::df_prod(c, f.sr), pi = mx::df_prod(c, f.si);
  const float srf = tof(f.sr), sif = tof(f.si);
  const F2 pm = mx::df_sub(pr, rr), pp = mx::df_sum(pr, rr), im = mx::df_sub(pi, ri), ip = mx::df_sum(pi, ri);
  const F2 a2 = mx::df_sum(mx::df_prod(pm, pm), mx::df_prod(im, im)), b2 = mx::df_sum(mx::df_prod(pp, pp), mx::df_prod(ip, ip));
  const float a2d = 2.0f * tof(pm) * (srf - rrd) + 2.0f * tof(im) * (sif - rid);
  const float b2d = 2.0f * tof(pp) * (srf + rrd) + 2.0f * tof(ip) * (sif + rid);
  const F2 t = mx::df_sum(mx::df_prod(a1, b2), mx::df_prod(a2, b1)), den = mx::df_mul(b1, b2);
  const float numd = 0.5f * ((tof(a1) * b2d + tof(b2) * a1d) + (tof(a2) * b1d + tof(b1) * a2d));
  const float dend = tof(b1) * b2d + tof(b2) * b1d;
  value = mx::df_div(mx::quick_sum(0.5f * t.h, 0.5f * t.l), den);
  slope = (numd - tof(value) * dend) * (1.0f / tof(den));
}
#endif

// exp(-x) for x >= 0 in single precision with every operation explicitly
// rounded (Cody-Waite reduction x = n ln2 + r with ln2 in two parts, then
// the Taylor series of exp(-r) to r^7, |r| <= ln2 / 2: truncation error
// below 6e-9), so host and device give the same bits.  Used for the splat
// taps, whose image must be reproducible by the CPU restatement.
MXG float exp_neg(float x) {
  if (!(x < 80.0f)) return 0.0f;
  const int n = (int) FADD(FMUL(x, 1.44269502f), 0.5f);
  const float fn = (float) n;
  const float r = FSUB(FSUB(x, FMUL(fn, 0.693145752f)), FMUL(fn, 1.42860677e-06f));
  const float s = -r;
  float p = FADD(1.0f, FMUL(s, 1.0f / 7.0f));
  p = FADD(1.0f, FMUL(FMUL(s, 1.0f / 6.0f), p));
  p = FADD(1.0f, FMUL(FMUL(s, 0.2f), p));
  p = FADD(1.0f, FMUL(FMUL(s, 0.25f), p));
  p = FADD(1.0f, FMUL(FMUL(s, 1.0f / 3.0f), p));
  p = FADD(1.0f, FMUL(FMUL(s, 0.5f), p));
  p = FADD(1.0f, FMUL(s, p));
  return FMUL(p, mx::u2f((uint32_t) (127 - n) << 23));   // 2^-n, n <= 115
}

// Splat geometry shared by the forward image, the adjoint and the CPU
// restatement.  Pixel (row j, column i) is centred at focal-plane
// y = cy + (i - (nx/2 - 1/2)) pitch, z = cz + (j - (ny/2 - 1/2)) pitch.
constexpr int TAPS = 11, HALF = 5;

// Continuous pixel coordinate of a focal-plane position, its nearest
// pixel and the offset from it, in the explicitly rounded order the CPU
// restatement follows.
MXG double pixel_coord(double y, double c, double inv_pitch, double centre_pix) {
  return MX_DADD(MX_DMUL(y - c, inv_pitch), centre_pix);
}

}  // namespace mxd
