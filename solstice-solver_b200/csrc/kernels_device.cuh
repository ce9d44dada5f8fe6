/*
 * kernels_device.cuh - device code of the sm_100a realisation loop of
 * `ssol_solve`, and the templates of its host launchers. Included by the
 * kernels_*.cu translation units, each of which instantiates some of the
 * launchers, so that they compile in parallel.
 *
 * One thread traces whole optical paths; the warps of a persistent grid take
 * realisations, or segments of sorted ones, from a counter. Per path it
 * restates, on the flat device scene of device_scene.h:
 *   point_init             src/ssol_solver.c:207-358
 *   trace_radiative_path   src/ssol_solver.c:873-1127
 *   point_update_from_hit  src/ssol_solver.c:360-411
 *   point_shade            src/ssol_solver.c:419-494
 *   update_mc              src/ssol_solver.c:708-785
 *   hit_filter_function    src/ssol_scene.c:439-535
 *   quadric intersection   src/ssol_shape.c:864-1244, 1408-1494
 *   sun direction samplers src/ssol_ranst_sun_dir.c:177-310
 * Tallies are FP64 (sum w, sum w^2) of each realisation's total, exactly the
 * deferred mc_data semantics of src/ssol_estimator_c.h:59-126: a path keeps
 * its per-receiver contributions until it ends, applies the Russian-roulette
 * factor, then commits. The paths of a warp commit together: sums of the
 * global quantities and of the warp's sampled instance are added up by FP64
 * tensor-core products (commit_warp), the sparse ones (per primitive) by FP64
 * reductions in device memory.
 *
 * Geometry, sampling and BSDFs run in the template type R (float for the
 * plain build, double for the all-FP64 build); quadric roots found in FP32 get
 * one FP64 Newton step.
 */
#ifndef SSOL_B200_KERNELS_DEVICE_CUH
#define SSOL_B200_KERNELS_DEVICE_CUH

#include "device_scene.h"
#include "kernels.h"
#include "philox.h"

#include <cuda_runtime.h>
#include <algorithm>
#include <float.h>
#include <math.h>

#include <atomic>
#include <mutex>
#include <numeric>

namespace ssolb {

/*******************************************************************************
 * Small vector helpers
 ******************************************************************************/
template<class R> struct V3 { R x, y, z; };

template<class R> __device__ __forceinline__ V3<R> mk(R x, R y, R z)
{ V3<R> v; v.x = x; v.y = y; v.z = z; return v; }
template<class R> __device__ __forceinline__ V3<R> ld3(const R* p)
{ return mk(p[0], p[1], p[2]); }
template<class R> __device__ __forceinline__ V3<R> operator+(V3<R> a, V3<R> b)
{ return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
template<class R> __device__ __forceinline__ V3<R> operator-(V3<R> a, V3<R> b)
{ return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
template<class R> __device__ __forceinline__ V3<R> operator-(V3<R> a)
{ return mk(-a.x, -a.y, -a.z); }
template<class R> __device__ __forceinline__ V3<R> operator*(V3<R> a, R s)
{ return mk(a.x * s, a.y * s, a.z * s); }
/* Products rounded on their own. The sums below spell out which product is
 * fused into each addition: left to the compiler, the choice depends on the
 * code around, and the kernel variants and launch orders would round the same
 * path differently */
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
/* a0 b0 + a1 b1 + a2 b2 */
template<class R> __device__ __forceinline__ R sum3(R a0, R b0, R a1, R b1, R a2, R b2)
{ return fma(a2, b2, fma(a0, b0, mul_rn(a1, b1))); }
template<class R> __device__ __forceinline__ R dot(V3<R> a, V3<R> b)
{ return sum3(a.x, b.x, a.y, b.y, a.z, b.z); }
template<class R> __device__ __forceinline__ V3<R> cross(V3<R> a, V3<R> b)
{
  return mk(fma(a.y, b.z, -mul_rn(a.z, b.y)), fma(a.z, b.x, -mul_rn(a.x, b.z)),
            fma(a.x, b.y, -mul_rn(a.y, b.x)));
}

__device__ __forceinline__ float rsq(float x) { return rsqrtf(x); }
__device__ __forceinline__ double rsq(double x) { return rsqrt(x); }
__device__ __forceinline__ float sq_rt(float x) { return sqrtf(x); }
__device__ __forceinline__ double sq_rt(double x) { return sqrt(x); }
__device__ __forceinline__ float lg(float x) { return logf(x); }
__device__ __forceinline__ double lg(double x) { return log(x); }
__device__ __forceinline__ float ex(float x) { return expf(x); }
__device__ __forceinline__ double ex(double x) { return exp(x); }
__device__ __forceinline__ float cpsgn(float a, float b) { return copysignf(a, b); }
__device__ __forceinline__ double cpsgn(double a, double b) { return copysign(a, b); }
__device__ __forceinline__ float nxt(float a) { return nextafterf(a, FLT_MAX); }
__device__ __forceinline__ double nxt(double a) { return nextafter(a, DBL_MAX); }
__device__ __forceinline__ void sincos2pi(float u, float* s, float* c)
{ sincospif(2.f * u, s, c); }
__device__ __forceinline__ void sincos2pi(double u, double* s, double* c)
{ sincospi(2.0 * u, s, c); }
__device__ __forceinline__ float cs(float x) { return cosf(x); }
__device__ __forceinline__ double cs(double x) { return cos(x); }
__device__ __forceinline__ float sn(float x) { return sinf(x); }
__device__ __forceinline__ double sn(double x) { return sin(x); }

template<class R> __device__ __forceinline__ V3<R> normalize(V3<R> v)
{ const R len = sq_rt(dot(v, v)); return len > R(0) ? v * (R(1) / len) : v; }

/* A dot product and a normalisation with the first two products in the other
 * order, where the code has always rounded so */
template<class R> __device__ __forceinline__ R dot_yx(V3<R> a, V3<R> b)
{ return sum3(a.y, b.y, a.x, b.x, a.z, b.z); }
/* The same with the last product rounded on its own, too */
template<class R> __device__ __forceinline__ R dot_yx_rn(V3<R> a, V3<R> b)
{ return mul_rn(a.z, b.z) + fma(a.y, b.y, mul_rn(a.x, b.x)); }
template<class R> __device__ __forceinline__ V3<R> normalize_hit(V3<R> v)
{
  const R len = sq_rt(dot_yx(v, v));
  return len > R(0) ? v * (R(1) / len) : v;
}

template<class R> __device__ __forceinline__ R uni(uint32_t x);
template<> __device__ __forceinline__ float uni<float>(uint32_t x)
{ return u01f(x); }
template<> __device__ __forceinline__ double uni<double>(uint32_t x)
{ return u01d(x); }

template<class R> __device__ __forceinline__ R rmax();
template<> __device__ __forceinline__ float rmax<float>() { return FLT_MAX; }
template<> __device__ __forceinline__ double rmax<double>() { return DBL_MAX; }

/* Orthonormal basis whose third axis is n (Duff et al., "Building an
 * Orthonormal Basis, Revisited", JCGT 2017) */
template<class R>
__device__ __forceinline__ void onb(V3<R> n, V3<R>& b1, V3<R>& b2)
{
  const R sgn = n.z >= R(0) ? R(1) : R(-1);
  const R a = R(-1) / (sgn + n.z);
  const R b = n.x * n.y * a;
  b1 = mk(R(1) + sgn * n.x * n.x * a, sgn * b, -sgn * n.x);
  b2 = mk(b, sgn + n.y * n.y * a, -n.y);
}

/* Per-realisation Philox block */
struct Rng {
  uint32_t i_lo, i_hi, k0, k1;
  __device__ __forceinline__ U32x4 get(uint32_t event, uint32_t domain) const
  { return philox4x32_10(i_lo, i_hi, event, domain, k0, k1); }
};

/*******************************************************************************
 * Scalar data and media
 ******************************************************************************/
/* Clamped linear interpolation (src/ssol_spectrum.c:57-89) */
static __device__ __noinline__ double interp_clamped
  (const double* w, const double* v, int n, double x)
{
  int lo = 0, hi = n; /* first index with w[i] >= x */
  while(lo < hi) {
    const int mid = (lo + hi) >> 1;
    if(w[mid] < x) lo = mid + 1; else hi = mid;
  }
  if(lo == n) return v[n - 1];
  if(lo == 0) return v[0];
  const double slope = (v[lo] - v[lo - 1]) / (w[lo] - w[lo - 1]);
  return v[lo - 1] + (x - w[lo - 1]) * slope;
}

template<class R>
__device__ __forceinline__ double data_value
  (const DScene<R>& S, const DData& d, double wl)
{
  if(d.spectrum < 0) return d.real;
  const DSpectrum sp = S.spectra[d.spectrum];
  return interp_clamped(S.spec_wl + sp.first, S.spec_val + sp.first,
                        sp.count, wl);
}

/* Shader value of a material at wavelength wl: index 0 reflectivity,
 * 1 roughness */
template<class R>
__device__ __noinline__ R shader_lerp(const double* w, int n, const R* tab, int which, double wl)
{
  if(n == 1) return tab[which];
  int lo = 0, hi = n;
  while(lo < hi) {
    const int mid = (lo + hi) >> 1;
    if(w[mid] < wl) lo = mid + 1; else hi = mid;
  }
  if(lo == n) return tab[2 * (n - 1) + which];
  if(lo == 0) return tab[which];
  const double a = tab[2 * (lo - 1) + which], b = tab[2 * lo + which];
  return (R)(a + (wl - w[lo - 1]) * (b - a) / (w[lo] - w[lo - 1]));
}

/* One value at every node (all materials but spectral ones): from the record
 * itself. The search of the table, two dependent loads and an FP64 division
 * per value, and the sampling of a wavelength that nothing reads were the
 * longest chains of a bounce: field, 1e8 paths, 92.5 -> 79.5 ms; beam-down,
 * 6e7, 158 -> 144 ms; path-traced 1080p image, 16.2 -> 13.7 ms. Where the
 * values are the same the interpolation returns exactly them. */
template<class R>
__device__ __forceinline__ R shader_value
  (const DScene<R>& S, const DMaterial& m, int which, double wl)
{
  if((m.uniform >> which) & 1) return (R)m.value[which];
  return shader_lerp(S.shader_wl, S.shader_nodes, S.shader_tab + m.table, which, wl);
}

/* Shader value baked at the vertices of a triangle side (offset `bake` in
 * bake_tab), interpolated in wavelength then with the barycentric weights
 * (1 - b1 - b2, b1, b2) of the point */
template<class R>
__device__ __forceinline__ R baked_value
  (const DScene<R>& S, int bake, int which, double wl, R b1, R b2)
{
  const R* tab = S.bake_tab + bake;
  const int stride = 2 * S.shader_nodes;
  const R v0 = shader_lerp(S.shader_wl, S.shader_nodes, tab, which, wl);
  const R v1 = shader_lerp(S.shader_wl, S.shader_nodes, tab + stride, which, wl);
  const R v2 = shader_lerp(S.shader_wl, S.shader_nodes, tab + 2 * stride, which, wl);
  return sum3(v0, R(1) - b1 - b2, v1, b1, v2, b2);
}

/*******************************************************************************
 * Sun: direction and wavelength (src/ssol_ranst_sun_dir.c:177-310,
 * src/ssol_ranst_sun_wl.c:84-105)
 ******************************************************************************/
template<class R>
__device__ __forceinline__ V3<R> sun_local_to_world(const DScene<R>& S, V3<R> p)
{
  const R* B = S.sun_basis;
  return normalize(mk(sum3(B[0], p.x, B[3], p.y, B[6], p.z),
                      sum3(B[1], p.x, B[4], p.y, B[7], p.z),
                      sum3(B[2], p.x, B[5], p.y, B[8], p.z)));
}

/* Buie zenith angle by rejection (src/ssol_ranst_sun_dir.c:177-195); the
 * draws of attempt k come from event 2 + k of the primary domain.
 *
 * The warp repeats the loop until its last lane accepts, and an attempt's FP64
 * cosines, power, sine and division were a fifth of the kernel. The density
 * in FP32 decides all but the closest attempts: its relative error is below
 * 1e-5 (the cosines' arguments reach 1.52, where a cosine of 0.055 takes 18
 * times the 1.2e-7 of its argument), so outside a margin of 1e-3 the FP64
 * comparison has the same outcome, and inside it is made. Field of 317, 5.1e6
 * paths under CSR 0.05: kernel 4.46 -> 4.10 ms. */
static __device__ __noinline__ double buie_theta
  (double thetaSD, double dCSSD, double gamma, double ek1000g, double alpha, double h1,
   double h2, double p1, const Rng rng)
{
  double theta = 0;
  for(uint32_t k = 0; k < 64; ++k) {
    const U32x4 r = rng.get(2u + k, RNG_PRIMARY);
    double value;
    if(u01d(r.v[0]) < p1) {
      theta = u01d(r.v[1]) * thetaSD;
      value = u01d(r.v[2]) * h1;
    } else {
      theta = thetaSD + u01d(r.v[1]) * dCSSD;
      value = u01d(r.v[2]) * h2;
    }
    {
      const float t = (float)theta, v = (float)value;
      const float phi = theta < thetaSD ? cosf(326.f * t) / cosf(308.f * t)
                                        : (float)ek1000g * powf(t, (float)gamma);
      const float p = (float)alpha * phi * sinf(t);
      if(p > 1e-30f && p < 1e30f) {
        if(v < p * 0.999f) break;
        if(v > p * 1.001f) continue;
      }
    }
    const double phi = theta < thetaSD
      ? cos(326 * theta) / cos(308 * theta)
      : ek1000g * pow(theta, gamma);
    if(value <= alpha * phi * sin(theta)) break;
  }
  return theta;
}

template<class R>
__device__ __forceinline__ V3<R> sample_sun_dir(const DScene<R>& S, const Rng& rng, U32x4 r)
{
  if(S.sun_type == SUN_DIRAC) return ld3(S.sun_dir);
  R st, ct;
  if(S.sun_type == SUN_PILLBOX) {
    const R sin2 = uni<R>(r.v[0]) * S.sun_param;
    st = sq_rt(sin2);
    ct = sq_rt(R(1) - sin2);
  } else if(S.sun_type == SUN_GAUSSIAN) {
    /* 1 - u keeps the log argument in (0, 1] */
    st = S.sun_param * sq_rt(R(-2) * lg(R(1) - uni<R>(r.v[0])));
    st = st < R(1) ? st : R(1);
    ct = sq_rt(R(1) - st * st > R(0) ? R(1) - st * st : R(0));
  } else {
    const R theta = (R)buie_theta(S.buie[0], S.buie[1], S.buie[2], S.buie[3], S.buie[4],
                                  S.buie[5], S.buie[6], S.buie[7], rng);
    st = sn(theta);
    ct = cs(theta);
  }
  /* One copy of the azimuth and of the frame for every sunshape */
  R sp, cp; sincos2pi(uni<R>(r.v[1]), &sp, &cp);
  const R x = cp * st, y = sp * st;
  const bool buie = S.sun_type == SUN_BUIE;
  return sun_local_to_world(S, mk(buie ? y : x, buie ? x : y, ct));
}

/* Piecewise linear density over the sun spectrum nodes: pick the interval by
 * its trapezoid mass, then invert the quadratic CDF inside it */
static __device__ __noinline__ double sample_wavelength
  (const double* nodes, const double* pdf, const double* cdf, int n, double u)
{
  if(n == 1) return nodes[0];
  int lo = 0, hi = n - 1; /* interval j with cdf[j] <= u < cdf[j+1] */
  while(hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if(cdf[mid] <= u) lo = mid; else hi = mid;
  }
  const double mass = cdf[lo + 1] - cdf[lo];
  const double r = mass > 0 ? fmin(fmax((u - cdf[lo]) / mass, 0.0), 1.0) : 0;
  const double a = pdf[lo], b = pdf[lo + 1];
  double t;
  if(a == b) t = r;
  else {
    const double den = a + sqrt(a * a + r * (b * b - a * a));
    t = den > 0 ? r * (a + b) / den : r;
  }
  return nodes[lo] + t * (nodes[lo + 1] - nodes[lo]);
}
template<class R>
__device__ __forceinline__ double sample_wavelength(const DScene<R>& S, double u)
{ return sample_wavelength(S.wl_nodes, S.wl_pdf, S.wl_cdf, S.wl_count, u); }

/*******************************************************************************
 * Punched quadrics (src/ssol_shape.c:236-285, 864-1135, 1408-1494)
 ******************************************************************************/
template<class R>
__device__ __forceinline__ V3<R> xform_point(const R* M, V3<R> p)
{
  return mk(sum3(M[0], p.x, M[1], p.y, M[2], p.z) + M[3],
            sum3(M[4], p.x, M[5], p.y, M[6], p.z) + M[7],
            sum3(M[8], p.x, M[9], p.y, M[10], p.z) + M[11]);
}
template<class R>
__device__ __forceinline__ V3<R> xform_vec(const R* M, V3<R> v)
{
  return mk(sum3(M[0], v.x, M[1], v.y, M[2], v.z), sum3(M[4], v.x, M[5], v.y, M[6], v.z),
            sum3(M[8], v.x, M[9], v.y, M[10], v.z));
}
/* Normal to world: transpose of the world->local linear part */
template<class R>
__device__ __forceinline__ V3<R> xform_normal(const R* W, V3<R> n)
{
  return mk(sum3(W[0], n.x, W[4], n.y, W[8], n.z), sum3(W[1], n.x, W[5], n.y, W[9], n.z),
            sum3(W[2], n.x, W[6], n.y, W[10], n.z));
}

/* Front normal (local frame, unnormalised) at pl of the general form in
 * DQuadric::gen */
template<class R>
__device__ __forceinline__ V3<R> quadric_general_normal(const DQuadric<R>& Q, V3<R> pl)
{
  const R sg = (R)Q.gen[6];
  return mk(sg * R(2) * (R)Q.gen[0] * pl.x, sg * R(2) * (R)Q.gen[1] * pl.y,
            sg * (R(2) * (R)Q.gen[2] * (pl.z - (R)Q.gen[3]) + (R)Q.gen[4]));
}

/* Height of the surface above local (x, y): the linear case, or the
 * root on the side gen[7] of z0 (upper sheet of the hyperboloid, lower
 * hemisphere); src/ssol_shape.c:236-285 */
template<class R>
__device__ __forceinline__ R quadric_general_z(const DQuadric<R>& Q, R x, R y)
{
  const R kz = (R)Q.gen[2];
  const R rest = (R)Q.gen[0] * x * x + (R)Q.gen[1] * y * y + (R)Q.gen[5];
  if(kz == R(0)) return -rest / (R)Q.gen[4];
  const R w = -rest / kz;
  return (R)Q.gen[3] + (R)Q.gen[7] * sq_rt(w > R(0) ? w : R(0));
}

/* Roots in ascending order; stable form of src/ssol_shape.c:864-896. Two
 * divisions for every case (linear, double root, two roots) instead of one for
 * each, the carving loops rolled and the grid look-up out of line: the
 * beam-down loop is bound by instruction fetch. 6e7 paths, 87.9 -> 85.4 ms. */
template<class R>
__device__ __forceinline__ int solve_quadratic(R a, R b, R c, R t[2])
{
  const bool linear = a == R(0);
  const R delta = b * b - R(4) * a * c;
  if(linear ? b == R(0) : delta < R(0)) return 0;
  const R s = sq_rt(delta);
  const bool one = linear || delta == R(0);
  const R t1 = (linear ? -c : one ? -b : -b - cpsgn(s, b)) / (linear ? b : R(2) * a);
  t[0] = t1;
  if(one) return 1;
  const R t2 = (t1 != R(0) ? c : -b) / (t1 != R(0) ? a * t1 : a);
  t[0] = t1 < t2 ? t1 : t2;
  t[1] = t1 < t2 ? t2 : t1;
  return 2;
}

/* One FP64 Newton step of F(o + t d) on the FP32 root, general form */
__device__ __forceinline__ float refine_root_general
  (const double* g, V3<float> o, V3<float> d, float t)
{
  const double ox = o.x, oy = o.y, dx = d.x, dy = d.y, dz = d.z;
  const double zz = (double)o.z - g[3];
  const double a = g[0] * dx * dx + g[1] * dy * dy + g[2] * dz * dz;
  const double b = 2.0 * (g[0] * ox * dx + g[1] * oy * dy + g[2] * zz * dz) + g[4] * dz;
  const double c = g[0] * ox * ox + g[1] * oy * oy + g[2] * zz * zz + g[4] * (double)o.z
                 + g[5];
  const double td = t;
  const double f = (a * td + b) * td + c;
  const double df = 2.0 * a * td + b;
  return df != 0.0 ? (float)(td - f / df) : t;
}
__device__ __forceinline__ double refine_root_general
  (const double*, V3<double>, V3<double>, double t)
{ return t; }

template<class R>
__device__ bool in_carvings(const DScene<R>& S, const DQuadric<R>& Q, R x, R y)
{
  if(Q.type == QUAD_HEMISPHERE && x * x + y * y > Q.param[2]) return false;
  if(x < Q.carve_lo[0] || x > Q.carve_hi[0]
  || y < Q.carve_lo[1] || y > Q.carve_hi[1]) {
    if(Q.type != QUAD_HEMISPHERE || Q.carve_count) return false;
  }
#pragma unroll 1
  for(int k = 0; k < Q.carve_count; ++k) {
    const DCarving C = S.carvings[Q.carve_first + k];
    const R* v = S.carve_verts + 2 * C.first;
    bool in = false;
#pragma unroll 1
    for(int i = 0, j = C.count - 1; i < C.count; j = i++) {
      const R xi = v[2 * i], yi = v[2 * i + 1];
      const R xj = v[2 * j], yj = v[2 * j + 1];
      if(((yi > y) != (yj > y)) && (x < (xj - xi) * (y - yi) / (yj - yi) + xi))
        in = !in;
    }
    if(C.op == 0 ? !in : in) return false;
  }
  return true;
}

/*******************************************************************************
 * Ray casting with the reference hit filter (src/ssol_scene.c:439-535)
 ******************************************************************************/
struct SelfInfo {
  int gid; /* triangle the ray leaves, -1 if none */
  int sinst; /* shaded instance the ray leaves */
  int side; /* its side (SSOL_FRONT=1 / SSOL_BACK=2) */
  bool discard_virtual;
  bool reversed;
};

template<class R> struct Hit {
  R t;
  int sinst;
  int prim; /* triangle id in its shape (meshes) */
  int gid; /* global triangle id, -1 for quadrics */
  V3<R> n; /* world normal (unnormalised for triangles) */
};

struct Counters {
  uint32_t rays, nodes, tris, quads;
};

template<class R>
__device__ __forceinline__ bool side_passes
  (const DScene<R>& S, int sinst, int side, const SelfInfo& self)
{
  if(self.reversed) side = side == 1 ? 2 : 1;
  const DShadedInst si = ldg_record(S.sinsts + sinst);
  if(si.virtual_mask & (side == 1 ? 1 : 2)) {
    if(self.discard_virtual) return false;
    if(!(si.receiver_mask & side)) return false;
  }
  return true;
}

/* Differences rounded on their own (no FMA contraction): with mul_rn, the
 * edge functions of the watertight test must be exact negations on an edge
 * shared by two triangles */
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }

/* Per-ray shear of the watertight ray/triangle test (Woop, Benthin and Wald,
 * "Watertight Ray/Triangle Intersection", JCGT 2(1), 2013): rows that map a
 * vertex relative to the origin into a frame where the ray runs along +z,
 * x' = v[kx] - Sx v[kz], y' = v[ky] - Sy v[kz], z' = Sz v[kz], with kz the
 * dominant axis of the direction and kx, ky swapped when d[kz] < 0 so that
 * the winding is kept. Applying the rows is deterministic per vertex, which
 * is all watertightness needs. */
template<class R> struct Shear { V3<R> rx, ry, rz; };

template<class R>
__device__ __forceinline__ Shear<R> make_shear(V3<R> d)
{
  const R ax = fabs(d.x), ay = fabs(d.y), az = fabs(d.z);
  const int kz = ax > ay ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
  int kx = kz == 2 ? 0 : kz + 1;
  int ky = kx == 2 ? 0 : kx + 1;
  const R dz = kz == 0 ? d.x : kz == 1 ? d.y : d.z;
  if(dz < R(0)) { const int t = kx; kx = ky; ky = t; }
  const R dx = kx == 0 ? d.x : kx == 1 ? d.y : d.z;
  const R dy = ky == 0 ? d.x : ky == 1 ? d.y : d.z;
  const R sx = dx / dz, sy = dy / dz, sz = R(1) / dz;
  Shear<R> s;
  s.rx = mk(kx == 0 ? R(1) : kz == 0 ? -sx : R(0),
            kx == 1 ? R(1) : kz == 1 ? -sx : R(0),
            kx == 2 ? R(1) : kz == 2 ? -sx : R(0));
  s.ry = mk(ky == 0 ? R(1) : kz == 0 ? -sy : R(0),
            ky == 1 ? R(1) : kz == 1 ? -sy : R(0),
            ky == 2 ? R(1) : kz == 2 ? -sy : R(0));
  s.rz = mk(kz == 0 ? sz : R(0), kz == 1 ? sz : R(0), kz == 2 ? sz : R(0));
  return s;
}

template<class R>
__device__ __forceinline__ R shear_row(V3<R> r, V3<R> a)
{
  return fma(r.z, a.z, fma(r.y, a.y, mul_rn(r.x, a.x)));
}

/* A 16-byte aligned record through the read-only data path, 16 bytes at a
 * time */
template<class T>
__device__ __forceinline__ T ldg_record(const T* p)
{
  static_assert(sizeof(T) % 16 == 0 && alignof(T) >= 16, "16-byte records only");
  union { T t; int4 w[sizeof(T) / 16]; } u;
#pragma unroll
  for(int i = 0; i < (int)(sizeof(T) / 16); ++i)
    u.w[i] = __ldg(reinterpret_cast<const int4*>(p) + i);
  return u.t;
}

/* A triangle through the read-only data path: three 16-byte loads in FP32 */
__device__ __forceinline__ DTri<float> load_tri(const DTri<float>* p)
{
  const float4* q = reinterpret_cast<const float4*>(p);
  const float4 a = __ldg(q), b = __ldg(q + 1);
  const int4 c = __ldg(reinterpret_cast<const int4*>(q + 2));
  DTri<float> t;
  t.v0[0] = a.x; t.v0[1] = a.y; t.v0[2] = a.z;
  t.v1[0] = a.w; t.v1[1] = b.x; t.v1[2] = b.y;
  t.v2[0] = b.z; t.v2[1] = b.w; t.v2[2] = __int_as_float(c.x);
  t.sinst = c.y; t.prim = c.z; t.gid = c.w;
  return t;
}
__device__ __forceinline__ DTri<double> load_tri(const DTri<double>* p) { return *p; }

/* A BVH node through the read-only data path: four 16-byte loads in FP32 */
__device__ __forceinline__ DNode<float> load_node(const DNode<float>* p)
{
  const float4* q = reinterpret_cast<const float4*>(p);
  const float4 a = __ldg(q), b = __ldg(q + 1), c = __ldg(q + 2);
  const int4 d = __ldg(reinterpret_cast<const int4*>(q + 3));
  DNode<float> n;
  n.lo[0][0] = a.x; n.lo[0][1] = a.y; n.lo[0][2] = a.z;
  n.lo[1][0] = a.w; n.lo[1][1] = b.x; n.lo[1][2] = b.y;
  n.hi[0][0] = b.z; n.hi[0][1] = b.w; n.hi[0][2] = c.x;
  n.hi[1][0] = c.y; n.hi[1][1] = c.z; n.hi[1][2] = c.w;
  n.child[0] = d.x; n.child[1] = d.y; n.count[0] = d.z; n.count[1] = d.w;
  return n;
}
__device__ __forceinline__ DNode<double> load_node(const DNode<double>* p) { return *p; }

/* Entry distance `tent` of a box, and whether the ray meets it before tmax.
 * FUSED spells the fused products out, so that a triangle's own box rounds as
 * its leaf's; left to the compiler, which fuses them too, the variant with
 * quadrics spills less: beam-down, 6e7 paths, 82.0 ms, spelled out 84.9. */
template<bool FUSED, class R>
__device__ __forceinline__ R slab_term(R x, R inv, R oinv)
{ return FUSED ? fma(x, inv, -oinv) : x * inv - oinv; }
template<bool FUSED, class R>
__device__ __forceinline__ bool slab
  (const R* lo, const R* hi, V3<R> inv, V3<R> oinv, R tmin, R tmax, R& tent)
{
  const R tx0 = slab_term<FUSED>(lo[0], inv.x, oinv.x);
  const R tx1 = slab_term<FUSED>(hi[0], inv.x, oinv.x);
  const R ty0 = slab_term<FUSED>(lo[1], inv.y, oinv.y);
  const R ty1 = slab_term<FUSED>(hi[1], inv.y, oinv.y);
  const R tz0 = slab_term<FUSED>(lo[2], inv.z, oinv.z);
  const R tz1 = slab_term<FUSED>(hi[2], inv.z, oinv.z);
  const R t0 = fmax(fmax(fmin(tx0, tx1), fmin(ty0, ty1)),
                    fmax(fmin(tz0, tz1), tmin));
  const R t1 = fmin(fmin(fmax(tx0, tx1), fmax(ty0, ty1)),
                    fmin(fmax(tz0, tz1), tmax));
  tent = t0;
  return t0 <= t1;
}

/* Whether a ray meets the box that a triangle has in a leaf of its own */
template<class R>
__device__ __forceinline__ bool own_box(const DTri<R>& T, V3<R> inv, V3<R> oinv, R tmin, R tmax)
{
  R lo[3], hi[3], te;
#pragma unroll
  for(int c = 0; c < 3; ++c) {
    lo[c] = fmin(T.v0[c], fmin(T.v1[c], T.v2[c]));
    hi[c] = fmax(T.v0[c], fmax(T.v1[c], T.v2[c]));
  }
  return slab<true>(lo, hi, inv, oinv, tmin, tmax, te);
}

/* Mesh rule: reject t <= eps, t <= tmin and the starting triangle.
 * Inclusion by the watertight edge functions, so that no ray is lost between
 * two triangles; distance from the triangle's plane, dot(Ng, v0 - o) /
 * dot(Ng, d), so that the two triangles of a planar quad give the same t and
 * a ray crossing a virtual quad on its diagonal is not counted twice.
 * Ng = e2 x e1 is Star-3D's front face.
 *
 * A triangle of a pair (`own`) must have its own box hit too, before tleaf, so
 * that a ray meets the triangles that it would meet in leaves of their own. The
 * box test rounds: a triangle that is hit at a corner of its box can have the
 * box missed by an ulp of the distance and the pair's larger box hit, where a
 * leaf of its own would not have been tested: 2 of 1.6e9 paths of the field of
 * 1000, 3e-8 of its estimates. (A pair's box is never missed where a triangle's
 * own is hit: the rounded products are monotone in the bounds.) Asked of
 * accepted hits only, with the vertices read again rather than kept in
 * registers; asked once, of the hit a traversal ends with, 1 % slower. */
template<class R, int FEAT>
__device__ __forceinline__ void test_triangle
  (const DScene<R>& S, int idx, V3<R> o, V3<R> d, const Shear<R>& sh, R tmin,
   R eps, const SelfInfo& self, bool own, V3<R> inv, V3<R> oinv, R tleaf, Hit<R>& best,
   bool& found)
{
  const DTri<R> T = load_tri(S.tris + idx);
  const V3<R> p0 = ld3(T.v0), p1 = ld3(T.v1), p2 = ld3(T.v2);
  const V3<R> a = p0 - o, b = p1 - o, c = p2 - o;
  const R ax = shear_row(sh.rx, a), ay = shear_row(sh.ry, a);
  const R bx = shear_row(sh.rx, b), by = shear_row(sh.ry, b);
  const R cx = shear_row(sh.rx, c), cy = shear_row(sh.ry, c);
  const R u = sub_rn(mul_rn(cx, by), mul_rn(cy, bx));
  const R v = sub_rn(mul_rn(ax, cy), mul_rn(ay, cx));
  const R w = sub_rn(mul_rn(bx, ay), mul_rn(by, ax));
  if((u < R(0) || v < R(0) || w < R(0)) && (u > R(0) || v > R(0) || w > R(0)))
    return;
  if(u + v + w == R(0)) return;
  const V3<R> ng = cross(p2 - p0, p1 - p0);
  const R den = dot(ng, d);
  const R t = dot(ng, a) / den;
  if(!(t < best.t) || t <= eps || t <= tmin || T.gid == self.gid) return;
  if constexpr(Pairs<R, FEAT>::value) {
    if(own) {
      asm volatile("" : "+r"(idx)); /* not the registers of the loads above */
      if(!own_box(load_tri(S.tris + idx), inv, oinv, tmin, tleaf)) return;
    }
  }
  const int side = den < R(0) ? 1 : 2;
  if(!side_passes(S, T.sinst, side, self)) return;
  best.t = t;
  best.sinst = T.sinst;
  best.prim = T.prim;
  best.gid = T.gid;
  best.n = ng;
  found = true;
}

/* Triangle of the RT tessellation grid that contains local (x, y): cell
 * (ix, iy) holds triangles 2 (ix ny + iy) (below its diagonal) and + 1;
 * only used when no carving cut the grid */
template<class R>
__device__ __noinline__ int quad_grid_prim(const DQuadric<R>& Q, R x, R y)
{
  const R d = Q.grid_delta;
  int ix = (int)floor((x - Q.carve_lo[0]) / d);
  int iy = (int)floor((y - Q.carve_lo[1]) / d);
  ix = min(max(ix, 0), Q.grid_n[0] - 1);
  iy = min(max(iy, 0), Q.grid_n[1] - 1);
  const R x0 = Q.carve_lo[0] + (R)ix * d, y0 = Q.carve_lo[1] + (R)iy * d;
  const R x1 = fmin(x0 + d, Q.carve_hi[0]), y1 = fmin(y0 + d, Q.carve_hi[1]);
  const bool lower = (x - x0) * (y1 - y0) >= (y - y0) * (x1 - x0);
  return (ix * Q.grid_n[1] + iy) * 2 + (lower ? 0 : 1);
}

/* Punched rule: analytic roots inside the carved domain, not below tmin, and
 * not the opposite side of the shape the ray leaves */
template<class R>
__device__ __forceinline__ void test_quadric
  (const DScene<R>& S, int idx, V3<R> o, V3<R> d, R tmin,
   const SelfInfo& self, Hit<R>& best, bool& found)
{
  const DQuadric<R>& Q = S.quads[idx];
  const V3<R> ol = xform_point(Q.w2l, o);
  const V3<R> dl = xform_vec(Q.w2l, d);
  /* One code path for every kind: the general form of DQuadric::gen */
  const R kx = (R)Q.gen[0], ky = (R)Q.gen[1], kz = (R)Q.gen[2], z0 = (R)Q.gen[3];
  const R lz = (R)Q.gen[4], m = (R)Q.gen[5];
  const R zz = ol.z - z0;
  const R a = kx * dl.x * dl.x + ky * dl.y * dl.y + kz * dl.z * dl.z;
  const R b = R(2) * (kx * ol.x * dl.x + ky * ol.y * dl.y + kz * zz * dl.z) + lz * dl.z;
  const R c = kx * ol.x * ol.x + ky * ol.y * ol.y + kz * zz * zz + lz * ol.z + m;
  R roots[2];
  const int n = solve_quadratic(a, b, c, roots);
  /* Not unrolled: one inlined copy of the refinement, carving and normal
   * code for both roots */
#pragma unroll 1
  for(int k = 0; k < n; ++k) {
    const R t = refine_root_general(Q.gen, ol, dl, k == 0 ? roots[0] : roots[1]);
    if(t <= tmin) continue;
    if(!(t < best.t)) break;
    const V3<R> pl = ol + dl * t;
    if(Q.type == QUAD_HYPERBOL && !(pl.z + Q.param[1] > R(0))) continue;
    if(Q.type == QUAD_HEMISPHERE && pl.z > Q.param[0]) continue;
    if(!in_carvings(S, Q, pl.x, pl.y)) continue;
    const V3<R> nw = normalize(xform_normal(Q.w2l, quadric_general_normal(Q, pl)));
    const int side = dot(d, nw) < R(0) ? 1 : 2;
    if(Q.sinst == self.sinst && side != self.side) continue;
    if(!side_passes(S, Q.sinst, side, self)) continue;
    best.t = t;
    best.sinst = Q.sinst;
    best.prim = Q.grid_n[0] > 0 && Q.grid_n[1] > 0 && Q.grid_delta > R(0)
              ? quad_grid_prim(Q, pl.x, pl.y) : 0;
    best.gid = -1;
    best.n = nw;
    found = true;
    break;
  }
}

/* The builder bounds the BVH depth to 30, so a traversal never holds more
 * than 30 deferred nodes. They live in a per-thread array: the few entries in
 * use stay in L1, one line a warp where its lanes are equally deep, and the
 * loop has no second place to look. With the first 3 / 5 entries in shared
 * memory the field's 1e8 paths take 64.4 / 65.6 ms, without 63.4; beam-down,
 * 6e7, 89.6 / 90.8 and 87.9. */
constexpr int STACK_SIZE = 32;

/* Closest accepted hit, or the first accepted hit when `any` (shadow rays) */
template<class R, int FEAT = FEAT_ALL>
__device__ bool trace_ray
  (const DScene<R>& S, V3<R> o, V3<R> d, R tmin, const SelfInfo& self,
   bool any, Hit<R>& best, Counters& cnt)
{
  if(!(FEAT & FEAT_NOCOUNT)) ++cnt.rays;
  /* A zero direction component would make lo * inv - o * inv an inf - inf
   * NaN for boxes the ray runs parallel to; clamp it to +-2^-64 so that the
   * FMA form of the slab test stays finite (Aila and Laine, HPG 2009) */
  const R tiny = R(5.42101086242752217e-20);
  const V3<R> inv = mk(R(1) / (fabs(d.x) > tiny ? d.x : cpsgn(tiny, d.x)),
                       R(1) / (fabs(d.y) > tiny ? d.y : cpsgn(tiny, d.y)),
                       R(1) / (fabs(d.z) > tiny ? d.z : cpsgn(tiny, d.z)));
  const V3<R> oinv = mk(o.x * inv.x, o.y * inv.y, o.z * inv.z);
  /* Self-hit epsilon of the mesh rule: the reference's 1e-6, scaled by the
   * magnitude of the origin so that it stays above the FP32 resolution */
  const R amax = fmax(fmax(fabs(o.x), fabs(o.y)), fabs(o.z));
  const R eps = R(1e-6) * (R(1) + amax);
  const Shear<R> sh = make_shear(d);
  best.t = rmax<R>();
  bool found = false;
  int stack[STACK_SIZE];
  int sp = 0, node = 0;
  /* The hit leaves of the node last visited, slot 0's first: primitive counts
   * and references */
  int lc0 = 0, lf0 = 0, lc1 = 0, lf1 = 0;
  /* A lane visits nodes until one has hit leaves, then waits for the other
   * lanes' leaves, so that a warp tests its primitives together: testing them
   * inside the node loop had nearly every visit of the warp wait for some
   * lane's test. Each lane still meets nodes and primitives in the same order.
   * Beam-down, 6e7 paths, 115 -> 104 ms; the field is neutral. */
  for(;;) {
    while(lc0 == 0 && node >= 0 && !(Pairs<R, FEAT>::value && (node & PAIR_LEAF))) {
      const DNode<R> N = load_node(S.nodes + node);
      if(!(FEAT & FEAT_NOCOUNT)) ++cnt.nodes;
      R te[2];
      bool h[2];
      h[0] = slab<Pairs<R, FEAT>::value>(N.lo[0], N.hi[0], inv, oinv, tmin, best.t, te[0])
          && N.count[0] >= 0;
      h[1] = slab<Pairs<R, FEAT>::value>(N.lo[1], N.hi[1], inv, oinv, tmin, best.t, te[1])
          && N.count[1] >= 0;
      const bool l0 = h[0] && N.count[0] > 0, l1 = h[1] && N.count[1] > 0;
      lc0 = l0 ? N.count[0] : l1 ? N.count[1] : 0;
      lf0 = l0 ? N.child[0] : N.child[1];
      lc1 = l0 && l1 ? N.count[1] : 0;
      lf1 = N.child[1];
      const bool in0 = h[0] && N.count[0] == 0, in1 = h[1] && N.count[1] == 0;
      if(in0 && in1) {
        const bool first0 = te[0] <= te[1];
        const int far = first0 ? N.child[1] : N.child[0];
        stack[sp++ & (STACK_SIZE - 1)] = far;
        node = first0 ? N.child[0] : N.child[1];
      } else if(in0 || in1) {
        node = in0 ? N.child[0] : N.child[1];
      } else if(sp == 0) {
        node = -1;
      } else {
        --sp;
        node = stack[sp];
      }
    }
    /* A pair's turn comes where its node's would, so that of two triangles
     * met at one distance, on the edge they share, the same one is hit as in
     * leaves of their own. (Tested with the node that lists them, sooner, field,
     * 1e8 paths, 60.6 for 62.1 ms, but some hits changed places in flux maps.) */
    if(Pairs<R, FEAT>::value && lc0 == 0 && node >= 0 && (node & PAIR_LEAF)) {
      lc0 = 2 | PAIR_LEAF;
      lf0 = node ^ PAIR_LEAF;
      node = sp ? stack[--sp] : -1;
    }
    if(lc0 == 0) break;
    const bool own = Pairs<R, FEAT>::value && (lc0 & PAIR_LEAF);
    const int lc = Pairs<R, FEAT>::value ? lc0 & ~PAIR_LEAF : lc0, first = lf0;
    const R tleaf = best.t;
    lc0 = lc1;
    lf0 = lf1;
    lc1 = 0;
    for(int p = 0; p < lc; ++p) {
      const uint32_t ref = lc == 1 ? (uint32_t)first : S.primrefs[first + p];
      if(!(FEAT & FEAT_QUADRIC) || primref_kind(ref) == PRIM_TRIANGLE) {
        if(!(FEAT & FEAT_NOCOUNT)) ++cnt.tris;
        test_triangle<R, FEAT>(S, (int)primref_index(ref), o, d, sh, tmin, eps, self,
                               own, inv, oinv, tleaf, best, found);
      } else {
        if(!(FEAT & FEAT_NOCOUNT)) ++cnt.quads;
        test_quadric(S, (int)primref_index(ref), o, d, tmin, self, best, found);
      }
      if(any && found) return true;
    }
  }
  return found;
}

/* Per-thread FP64 path sums kept in shared memory (column `tid`, stride
 * blockDim): the first receiver entry's 6 values, the 3 global quantities
 * accumulated along the path and the cosine factor */
enum : int { PS_V0 = 0, PS_ABS = 6, PS_ATM = 7, PS_OTHER = 8, PS_COS = 9,
             PS_UV = 10 };
/* Path sums a kernel variant keeps: PS_UV only with shading attributes
 */
__host__ __device__ constexpr int ps_count(int feat)
{ return feat & FEAT_ATTRIBUTES ? 11 : 10; }

/* Barycentric weights (b1, b2) of vertices 1 and 2 of triangle gid at the
 * point x of its plane. DRAW: the determinant with its other product fused, as
 * the renderers have always rounded it. */
template<class R, bool DRAW = false>
__device__ __forceinline__ float2 tri_uv(const DScene<R>& S, int gid, V3<R> x)
{
  const DTri<R>& T = S.tris[gid];
  const V3<R> a = ld3(T.v0);
  const V3<R> e1 = ld3(T.v1) - a, e2 = ld3(T.v2) - a, q = x - a;
  const R d11 = dot(e1, e1), d12 = dot(e1, e2), d22 = dot(e2, e2);
  const R q1 = dot(q, e1), q2 = dot(q, e2);
  const R den = DRAW ? fma(d11, d22, -mul_rn(d12, d12)) : fma(-d12, d12, mul_rn(d11, d22));
  if(!(den != R(0))) return make_float2(0.f, 0.f);
  return make_float2((float)(fma(d22, q1, -mul_rn(d12, q2)) / den),
                     (float)(fma(d11, q2, -mul_rn(d12, q1)) / den));
}

/* Barycentric weights (b1, b2) of the current point, kept as two floats in
 * the PS_UV slot when the scene has shading attributes */
__device__ __forceinline__ void put_uv(double* ps, int stride, float b1, float b2)
{
  float2* q = reinterpret_cast<float2*>(ps + PS_UV * stride);
  *q = make_float2(b1, b2);
}
__device__ __forceinline__ float2 get_uv(const double* ps, int stride)
{
  return *reinterpret_cast<const float2*>(ps + PS_UV * stride);
}

/*******************************************************************************
 * BSDF sampling (Star-SF's BSDFs restated from published optics: Fresnel
 * equations, Walter et al. 2007 microfacet sampling, thin-slab series)
 ******************************************************************************/
enum { BXDF_REFLECTION = 1, BXDF_TRANSMISSION = 2 };

/* Unpolarised Fresnel reflectance at a dielectric interface */
template<class R>
__device__ __forceinline__ R fresnel(R cos_i, R cos_t, R eta_i, R eta_t)
{
  const R rs = (eta_i * cos_i - eta_t * cos_t) / (eta_i * cos_i + eta_t * cos_t);
  const R rp = (eta_t * cos_i - eta_i * cos_t) / (eta_t * cos_i + eta_i * cos_t);
  return R(0.5) * (rs * rs + rp * rp);
}

template<class R>
__device__ __forceinline__ V3<R> local_to(V3<R> n, R x, R y, R z)
{
  V3<R> b1, b2;
  onb(n, b1, b2);
  return mk(sum3(b1.x, x, b2.x, y, n.x, z), sum3(b1.y, x, b2.y, y, n.y, z),
            sum3(b1.z, x, b2.z, y, n.z, z));
}

/* One BSDF sample: the propagated fraction, the outgoing direction, the
 * sampled component (BXDF_*, 0 if none) and the medium beyond, through
 * references; false on an inconsistent medium (RES_BAD_OP). Inlined: a call
 * that takes the scene by reference gives every thread a copy of the kernel's
 * scene parameter in local memory (field, 1e8 paths, 73.8 -> 70.3 ms without
 * it), and spills the registers it may use. What scenes seldom need (spectral
 * tables, wavelengths, Buie's rejection loop, further receiver hits of a path)
 * stays out of line, as the bounce loop is bound by instruction fetch: 77.6
 * -> 73.9 ms. With the commit inlined as well: 70.2 -> 67.7 ms, beam-down,
 * 6e7, 104 -> 96 ms. */
template<class R, int FEAT = FEAT_ALL>
__device__ __forceinline__ bool shade
  (const DScene<R>& S, const Rng& rng, uint32_t scatter, int mtl_idx,
   int medium, double wl, V3<R> wo, V3<R> Ng, R& prop, V3<R>& out,
   int& type, int& next_medium, int gid, int side, const double* ps, int stride)
{
  const DMaterial m = S.mtls[mtl_idx];
  prop = R(0);
  type = 0;
  next_medium = medium;
  /* src/ssol_material.c:97-101 */
  if((FEAT & FEAT_DIELECTRIC) && m.type == MTL_DIELECTRIC && medium != m.out_medium)
    return false;
  /* Shading normal: the interpolated vertex normal turned toward the
   * incoming side, else Ng (src/ssol_material.c:630-654); shader values
   * baked per vertex where the material varies over the mesh */
  V3<R> N = Ng;
  int bake = -1;
  R b1 = R(0), b2 = R(0);
  if((FEAT & FEAT_ATTRIBUTES) && S.tshade && gid >= 0) {
    const float2 uv = get_uv(ps, stride);
    b1 = (R)uv.x;
    b2 = (R)uv.y;
    const DTriShade<R>& ts = S.tshade[gid];
    bake = ts.bake[side - 1];
    if(!isnan(ts.n[0])) {
      const V3<R> ns = ld3(ts.n) * (R(1) - b1 - b2) + ld3(ts.n + 3) * b1
                     + ld3(ts.n + 6) * b2;
      const R l2 = dot(ns, ns);
      if(l2 > R(0)) {
        N = ns * rsq(l2);
        if(dot(N, wo) < R(0)) N = -N;
      }
    }
  }
  const R cos_i = dot(wo, N);
  if(!(cos_i > R(0))) return true;
  const U32x4 r = rng.get(scatter, RNG_SCATTER);
  switch(m.type) {
    case MTL_MIRROR:
    case MTL_MATTE: {
      const bool matte = m.type == MTL_MATTE;
      const R refl = bake >= 0 ? baked_value(S, bake, 0, wl, b1, b2)
                               : shader_value(S, m, 0, wl);
      const R rough = matte ? R(1) : bake >= 0 ? baked_value(S, bake, 1, wl, b1, b2)
                                               : shader_value(S, m, 1, wl);
      type = BXDF_REFLECTION;
      if(rough == R(0)) {
        out = N * (R(2) * cos_i) - wo;
        prop = refl;
      } else {
        /* Matte: cosine weighted hemisphere. Mirror: microfacet normal drawn
         * around N (Beckmann: tan^2 = -a^2 ln(1-u); pillbox: tan^2 = a^2 u),
         * mirrored about; re-drawn while the reflection falls below the
         * surface. One copy of the angle and frame code for both, as a warp's
         * lanes on either run it together and less code is fetched: beam-down,
         * 6e7 paths, 85.4 -> 81.7 ms. The smooth and the thin dielectric in
         * one copy too, or out of line, 82.8 and 83.5. */
        U32x4 rr = r;
        bool ok = false;
#pragma unroll 1
        for(uint32_t k = 0; k < 16; ++k) {
          if(k) rr = rng.get((scatter << 6) | k, RNG_RETRY);
          const R u0 = uni<R>(rr.v[0]);
          R st, ct;
          if(matte) {
            st = sq_rt(u0);
            ct = sq_rt(R(1) - u0);
          } else {
            const R tan2 = m.distrib == DISTRIB_BECKMANN
              ? -rough * rough * lg(R(1) - u0)
              : rough * rough * u0;
            ct = rsq(R(1) + tan2);
            st = sq_rt(tan2) * ct;
          }
          R sp, cp; sincos2pi(uni<R>(rr.v[1]), &sp, &cp);
          const V3<R> h = local_to(N, cp * st, sp * st, ct);
          if(matte) { out = h; ok = true; break; }
          const R wh = dot(wo, h);
          if(!(wh > R(0))) continue;
          out = h * (R(2) * wh) - wo;
          ok = dot(out, N) > R(0);
          if(ok) break;
        }
        prop = ok ? refl : R(0);
      }
      break;
    }
    case MTL_DIELECTRIC: {
      if(!(FEAT & FEAT_DIELECTRIC)) break;
      const R eta_i = (R)data_value(S, S.media[m.out_medium].refractive_index, wl);
      const R eta_t = (R)data_value(S, S.media[m.in_medium].refractive_index, wl);
      const R eta = eta_i / eta_t;
      const R sin2_t = eta * eta * (R(1) - cos_i * cos_i);
      R F = R(1), cos_t = R(0);
      if(sin2_t < R(1)) {
        cos_t = sq_rt(R(1) - sin2_t);
        F = fresnel(cos_i, cos_t, eta_i, eta_t);
      }
      prop = R(1);
      if(uni<R>(r.v[0]) < F) {
        out = N * (R(2) * cos_i) - wo;
        type = BXDF_REFLECTION;
      } else {
        out = normalize(N * (eta * cos_i - cos_t) - wo * eta);
        type = BXDF_TRANSMISSION;
        next_medium = m.in_medium;
      }
      break;
    }
    case MTL_THIN_DIELECTRIC: {
      if(!(FEAT & FEAT_DIELECTRIC)) break;
      const R eta_i = (R)data_value(S, S.media[m.out_medium].refractive_index, wl);
      const R eta_t = (R)data_value(S, S.media[m.slab_medium].refractive_index, wl);
      const R alpha = (R)data_value(S, S.media[m.slab_medium].extinction, wl);
      const R eta = eta_i / eta_t;
      const R sin2_t = eta * eta * (R(1) - cos_i * cos_i);
      R Rt = R(1), Tt = R(0);
      if(sin2_t < R(1)) {
        const R cos_t = sq_rt(R(1) - sin2_t);
        const R F = fresnel(cos_i, cos_t, eta_i, eta_t);
        const R tau = ex(-alpha * (R)m.thickness / cos_t);
        const R den = R(1) - F * F * tau * tau;
        Rt = F + (R(1) - F) * (R(1) - F) * F * tau * tau / den;
        Tt = (R(1) - F) * (R(1) - F) * tau / den;
      }
      prop = Rt + Tt;
      if(prop > R(0) && uni<R>(r.v[0]) * prop < Rt) {
        out = N * (R(2) * cos_i) - wo;
        type = BXDF_REFLECTION;
      } else {
        out = -wo;
        type = BXDF_TRANSMISSION;
      }
      break;
    }
    default: break;
  }
  /* Wrong hemisphere for the sampled component, against the geometric
   * normal (src/ssol_solver.c:468-475) */
  const R cos_out = dot(Ng, out);
  if((cos_out > R(0) && (type & BXDF_TRANSMISSION))
  || (cos_out < R(0) && (type & BXDF_REFLECTION)))
    prop = R(0);
  return true;
}

/*******************************************************************************
 * Realisation state machine
 *
 * Each warp iteration casts exactly one ray per active lane, from a single
 * call site: the shadow ray of a new path (any hit) or the next segment of a
 * path (closest hit). Lanes start together, cast their shadow rays together
 * and then each segment; those that have ended wait (regen_lanes), commit
 * together and take the next realisations through a warp-aggregated atomic
 * counter.
 ******************************************************************************/
enum : int { PH_NONE = 0, PH_SHADOW = 1, PH_BOUNCE = 2, PH_ENDED = 3 };
enum : int {
  END_NONE = 0, END_SHADOW, END_MISS, END_ZERO, END_KILL, END_FAIL,
  END_OVERFLOW /* a failure: more receiver entries than a path keeps */
};

/* Extra (receiver side, primitive) entries of one path beyond the first,
 * kept in local memory: only paths reaching several receivers touch them */
constexpr int MAX_EXTRA = 7;

/* Sums into device memory, as reductions (no value comes back): an
 * atomicAdd through a pointer that may address shared memory is a generic
 * atomic whose sector returns to L1 */
__device__ __forceinline__ void red_add_global(double* p, double v)
{
  if(v != 0.0)
    asm volatile("red.global.add.f64 [%0], %1;"
                 :: "l"(__cvta_generic_to_global(p)), "d"(v) : "memory");
}
__device__ __forceinline__ void red_count_global(unsigned long long* p, unsigned long long n)
{
  asm volatile("red.global.add.u64 [%0], %1;"
               :: "l"(__cvta_generic_to_global(p)), "l"(n) : "memory");
}

/* (w, w^2) of the 10 receiver quantities of one path, from its 6
 * accumulated values (MC_RECEIVER_DATA order, src/ssol_solver.c:735-755:
 * incoming, incoming if no atmosphere loss, if no field loss, lost in the
 * field, lost in the atmosphere, then the same 5 absorbed), added to dst in
 * device memory. The values travel as scalars, so that none of them goes
 * through local memory. */
static __device__ __noinline__ void commit10
  (double* dst, double v0, double v1, double v2, double v3, double v4, double v5,
   double f)
{
  const double q[NRCV_Q] = {f * v0, f * v1, f * v2, f * (v2 - v0), f * (v1 - v0),
                            f * v3, f * v4, f * v5, f * (v5 - v3), f * (v4 - v3)};
#pragma unroll
  for(int k = 0; k < NRCV_Q; ++k) {
    red_add_global(dst + 2 * k, q[k]);
    red_add_global(dst + 2 * k + 1, q[k] * q[k]);
  }
}
__device__ __forceinline__ void commit10(double* dst, const double v[6], double f)
{
  commit10(dst, v[0], v[1], v[2], v[3], v[4], v[5], f);
}

template<class R> struct PathState {
  int phase;
  int end; /* END_* of a path in PH_ENDED */
  int samp;
  int tslot; /* tracked path slot, -1 if not tracked */
  uint32_t tseq; /* vertices recorded so far */
  /* current point / ray: the point is org (+ rd t after a hit) */
  int sinst, side, prim, gid, medium, out_medium;
  V3<R> N, org, rd;
  R tmin, hit_t;
  double wl;
  /* weights (FP64) */
  double prev[3];
  double inc0;
  bool virt;
  /* counters */
  uint32_t depth, interval, scatter, nroul, segments;
  int score;
  /* receiver entries: the first one's values live in shared memory */
  int nent;
  int r0, p0;
  bool overflow;
};

/* Sampled proxy primitive of a primary draw: Vose alias table, bucket =
 * floor(u * n) computed exactly on the 24-bit integer draw */
template<class R>
__device__ __forceinline__ int sample_prim(const DScene<R>& S, const U32x4& r0)
{
  int k = (int)(((unsigned long long)(r0.v[0] >> 8)
                 * (unsigned long long)S.nsamp) >> 24);
  if(!(uni<float>(r0.v[1]) < S.alias_prob[k])) k = S.alias_idx[k];
  return k;
}

/* point_init (src/ssol_solver.c:207-352) up to the shadow ray */
template<class R, int FEAT = FEAT_ALL>
__device__ __forceinline__ void init_path
  (const DScene<R>& S, const Rng& rng, PathState<R>& p, double* ps, int stride)
{
  const U32x4 r0 = rng.get(0u, RNG_PRIMARY);
  const int k = sample_prim(S, r0);
  const DSampTri<R> st = S.samp[k];
  const R sa = sq_rt(uni<R>(r0.v[2]));
  const R b2 = sa * uni<R>(r0.v[3]);
  const R b1 = sa - b2;
  V3<R> pos = ld3(st.v0) + ld3(st.e1) * b1 + ld3(st.e2) * b2;
  const V3<R> nproxy = ld3(st.n);
  if((FEAT & FEAT_ATTRIBUTES) && S.tshade) put_uv(ps, stride, (float)b1, (float)b2);

  const U32x4 r1 = rng.get(1u, RNG_PRIMARY);
  const V3<R> dir = sample_sun_dir(S, rng, r1);
  p.wl = S.spectral ? sample_wavelength(S, u01d(r1.v[2])) : 0.0;

  const DShadedInst si = S.sinsts[st.sinst];
  V3<R> N = nproxy;
  if((FEAT & FEAT_QUADRIC) && si.is_punched) {
    /* punched_shape_project_point (src/ssol_shape.c:1408-1447) */
    const DQuadric<R>& Q = S.quads[si.quadric];
    V3<R> pl = xform_point(Q.w2l, pos);
    pl.z = quadric_general_z(Q, pl.x, pl.y);
    N = normalize(xform_normal(Q.w2l, quadric_general_normal(Q, pl)));
    pos = xform_point(Q.l2w, pl);
  }
  int side = 1;
  if(dot(N, dir) >= R(0)) { side = 2; N = -N; }

  const V3<R> sun0 = ld3(S.sun_dir);
  const R surface_sun_cos = dot(N, dir);
  const R surface_sun0_cos = fabs(dot(sun0, N));
  const R sun0_sun_cos = dot(sun0, dir);
  const R surface_proxy_cos = si.is_punched ? fabs(dot(nproxy, N)) : R(1);
  const R cos_ratio = fabs(surface_sun_cos / (surface_proxy_cos * sun0_sun_cos));
  const double w0 = S.dni * S.area_proxy * (double)cos_ratio;
  ps[PS_COS * stride] = S.area_proxy / S.area_rt
    * (double)surface_sun0_cos / (double)surface_proxy_cos;
  ps[PS_ABS * stride] = ps[PS_ATM * stride] = ps[PS_OTHER * stride] = 0;
  p.samp = si.sampled;

  const DMaterial m = S.mtls[si.mtl[side - 1]];
  p.medium = S.air_medium;
  if((FEAT & FEAT_DIELECTRIC)
  && (m.type == MTL_DIELECTRIC || m.type == MTL_THIN_DIELECTRIC))
    p.medium = side == 1 ? m.in_medium : m.out_medium;

  p.sinst = st.sinst;
  p.side = side;
  p.prim = st.prim;
  p.gid = st.gid;
  p.N = N;
  p.hit_t = R(0);
  p.prev[0] = p.prev[1] = p.prev[2] = w0;
  p.inc0 = 0;
  p.virt = false;
  p.depth = p.scatter = p.nroul = p.segments = 0;
  p.interval = 64;
  p.score = 0;
  p.nent = 0;
  p.overflow = false;
  /* Shadow ray toward the sun (src/ssol_solver.c:320-352) */
  p.org = pos;
  p.rd = -dir;
  p.tmin = R(0);
  p.phase = PH_SHADOW;
}

/* A path's receiver hits beyond its first */
template<class R>
__device__ __noinline__ void add_entry_again
  (PathState<R>& p, int rslot, int pslot, const double v[6], double* ps,
   int stride, int* xr, int* xp, double (*xv)[6])
{
  if(p.r0 == rslot && p.p0 == pslot) {
    for(int q = 0; q < 6; ++q) ps[(PS_V0 + q) * stride] += v[q];
    return;
  }
  for(int e = 0; e < p.nent - 1; ++e) {
    if(xr[e] == rslot && xp[e] == pslot) {
      for(int q = 0; q < 6; ++q) xv[e][q] += v[q];
      return;
    }
  }
  if(p.nent - 1 >= MAX_EXTRA) { p.overflow = true; return; }
  const int e = p.nent - 1;
  xr[e] = rslot;
  xp[e] = pslot;
  for(int q = 0; q < 6; ++q) xv[e][q] = v[q];
  ++p.nent;
}

template<class R>
__device__ __forceinline__ void add_entry
  (PathState<R>& p, int rslot, int pslot, const double v[6], double* ps,
   int stride, int* xr, int* xp, double (*xv)[6])
{
  if(p.nent == 0) {
    p.nent = 1;
    p.r0 = rslot;
    p.p0 = pslot;
    for(int q = 0; q < 6; ++q) ps[(PS_V0 + q) * stride] = v[q];
    return;
  }
  add_entry_again(p, rslot, pslot, v, ps, stride, xr, xp, xv);
}

/* One surface interaction (src/ssol_solver.c:939-1011): extinction of the
 * incoming segment, virtual pass-through or BSDF sample, receiver tallies,
 * then either the next ray or the end of the path */
template<class R, int FEAT = FEAT_ALL>
__device__ int interact
  (const DScene<R>& S, const Rng& rng, PathState<R>& p, V3<R> pos, V3<R> dir,
   uint32_t& bounces, unsigned long long max_segments, double* ps, int stride,
   int* xr, int* xp, double (*xv)[6])
{
  const DShadedInst si = S.sinsts[p.sinst];
  const bool in_atm = p.medium == S.air_medium;
  const bool hit_receiver = (si.receiver_mask & p.side) != 0;
  const bool hit_virtual = (si.virtual_mask & p.side) != 0;
  double trans = 1;
  if(p.hit_t > R(0)) {
    const double kext = data_value(S, S.media[p.medium].extinction, p.wl);
    if(kext > 0) trans = (double)ex((R)(-kext * (double)p.hit_t));
  }
  const double inc0 = p.prev[0] * trans;
  const double inc1 = in_atm ? p.prev[1] : p.prev[1] * trans;
  const double inc2 = !in_atm ? p.prev[2] : p.prev[2] * trans;
  double out0, out1, out2, kabs;
  int out_medium = p.medium;
  if(hit_virtual) {
    kabs = 0;
    out0 = inc0; out1 = inc1; out2 = inc2;
  } else {
    ++bounces;
    R prop;
    V3<R> ndir;
    int type;
    if(!shade<R, FEAT>(S, rng, p.scatter++, si.mtl[p.side - 1], p.medium, p.wl, -dir,
              p.N, prop, ndir, type, out_medium, p.gid, p.side, ps, stride))
      return END_FAIL;
    const double pr = (double)prop;
    kabs = 1.0 - pr;
    out0 = inc0 * pr;
    out1 = inc1 * pr;
    out2 = hit_receiver ? inc2 * pr : inc2;
    if(type) dir = ndir;
  }
  if(hit_receiver) {
    const int s = p.side - 1;
    const double v[6] = {inc0, inc1, inc2, inc0 * kabs, inc1 * kabs, inc2 * kabs};
    const int pslot = si.prim_base[s] >= 0 ? si.prim_base[s] + p.prim : -1;
    add_entry(p, si.rcv_slot[s], pslot, v, ps, stride, xr, xp, xv);
    ps[PS_ABS * stride] += inc0 - out0;
  } else {
    ps[PS_OTHER * stride] += inc0 * kabs;
  }
  /* Loss along the incoming segment, accounted at non-virtual points or at
   * the end of the path (src/ssol_solver.c:1036-1054) */
  const double seg_loss = p.prev[0] - inc0;
  if(out0 == 0.0 || !hit_virtual)
    ps[(in_atm ? PS_ATM : PS_OTHER) * stride] += seg_loss;
  if(out0 == 0.0) return END_ZERO;
  if(!hit_virtual) {
    p.prev[0] = out0; p.prev[1] = out1; p.prev[2] = out2;
    p.org = pos;
    p.rd = dir;
    p.tmin = R(0);
  } else {
    /* Virtual: pursue the same ray beyond the hit (src/ssol_solver.c:988-995) */
    p.inc0 = inc0;
    p.tmin = nxt(p.hit_t);
  }
  p.virt = hit_virtual;
  p.out_medium = out_medium;
  if(++p.segments >= max_segments) return END_FAIL;
  p.phase = PH_BOUNCE;
  return END_NONE;
}

/* Running sums of a warp, kept in shared memory as the accumulators of four
 * FP64 tensor-core tiles (8 rows of 8 partial sums, two per lane):
 *   tile 0: (w, w^2) of the global quantities absorbed by receivers,
 *           missing, atmosphere, other, of item `gitem`;
 *   tile 1: cosine and shadowed of sampled instance `samp` of item `item`
 *           (rows 0-3), then, with tiles 2 and 3, the 10 receiver quantities
 *           of its slot `rbase` of samp_rcv (rows 4-7, 0-7, 0-7).
 * Only these are summed: a receiver side's totals are the sums of its
 * samp_rcv slots over the sampled instances, and the global cosine and
 * shadowed those of the samp slots, which finish_tallies adds up once a
 * launch.
 *
 * A commit is the sum of 32 lanes' values into few addresses: bound by the
 * atomics when each path sends its own (25 reductions a path to one sampled
 * instance's slots; with a single mirror every path of the GPU to the same
 * 25 addresses), by instructions when summed by shuffles (5 steps of two
 * per value). A product with a one-row matrix sums 32 lanes in one
 * instruction and keeps the running sum in its accumulator, in full FP64.
 * With the lock-step paths (regen_lanes): one mirror, 1e6 paths, 4.05 ->
 * 0.55 ms; field, 1e8 paths, 149 -> 92 ms (110 by the lock step alone). */
struct WarpKeys { int gitem, item, samp, rbase; };
constexpr int TILES = 4;

/* Row `row` (0..7) of a tile += the sum of v over the 32 lanes: an m8n8k4
 * product whose A is one in that row and zero elsewhere, and whose B holds
 * the lanes' values. v must be finite (0 x inf would reach every row). */
__device__ __forceinline__ void tile_add(double2& d, int row, unsigned lane, double v)
{
  const double a = (int)(lane >> 2) == row ? 1.0 : 0.0;
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 "
               "{%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d.x), "+d"(d.y) : "d"(a), "d"(v));
}
/* Sum of the lane's row (lane / 4) */
__device__ __forceinline__ double tile_row_sum(double2 d)
{
  double v = d.x + d.y;
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  return v;
}

/* The warp's tiles into the tallies they are keyed by: tile 0, the samp
 * rows, or the samp_rcv rows; all lanes call it */
static __device__ __noinline__ void flush_global
  (const DTallies* tallies, const WarpKeys* wk, double2* tile)
{
  const unsigned lane = threadIdx.x & 31u;
  const double v = tile_row_sum(tile[0]);
  const int row = (int)(lane >> 2);
  if((lane & 3u) == 0u && wk->gitem >= 0)
    red_add_global(tallies[wk->gitem].global + (row < 2 ? 2 * G_ABS_RCV : 2 * G_MISSING - 2) + row,
                   v);
  tile[0] = make_double2(0.0, 0.0);
}
static __device__ __noinline__ void flush_samp
  (const DTallies* tallies, const WarpKeys* wk, double2* tile, int stride, bool rcv_only)
{
  const unsigned lane = threadIdx.x & 31u;
  const int row = (int)(lane >> 2);
  double v[3];
#pragma unroll
  for(int k = 0; k < 3; ++k) v[k] = tile_row_sum(tile[(k + 1) * stride]);
  if((lane & 3u) == 0u && wk->item >= 0) {
    const DTallies& T = tallies[wk->item];
    if(row < 4) {
      if(!rcv_only) red_add_global(T.samp + (size_t)wk->samp * 4 + row, v[0]);
    }
    if(wk->rbase >= 0) {
      double* dst = T.samp_rcv + (size_t)wk->rbase * NRCV_Q * 2;
      if(row >= 4) red_add_global(dst + row - 4, v[0]);
      red_add_global(dst + 4 + row, v[1]);
      red_add_global(dst + 12 + row, v[2]);
    }
  }
  if(row >= 4 || !rcv_only) tile[stride] = make_double2(0.0, 0.0);
  tile[2 * stride] = tile[3 * stride] = make_double2(0.0, 0.0);
}

/* Lanes of one sampled instance below which their sums go straight to
 * device memory (id-ordered launches, whose lanes sample all over the
 * scene) */
constexpr int MIN_GROUP = 4;

/* A path's end: what commit_warp reads of it stays in p (the weight
 * shadowed or missing in prev[0]) */
template<class R>
__device__ __forceinline__ void path_ended(PathState<R>& p, int end)
{
  if(end == END_MISS && p.virt) p.prev[0] = p.inc0;
  p.end = p.overflow ? END_OVERFLOW : end;
  p.phase = PH_ENDED;
}

/* Commit the finished paths of the lanes with `ended`: FP64 (w, w^2) of each
 * path's totals, x 2^score for roulette survivors (src/ssol_solver.c:
 * 1087-1108). All lanes of the warp call it converged. The lanes of one
 * sampled instance (in the coherent order nearly always the whole warp) add
 * through the warp's tiles, the others, and any path with a weight that is
 * not finite, through reductions of their own. */
static __device__ __forceinline__ void commit_warp
  (int nrcv, const DTallies* tallies, int item, bool ended, int end, int p_samp, int score,
   int p_nent, int p_r0, int p0, double weight, const double* ps, int stride, double2* tile, WarpKeys* wk, const int* xr,
   const int* xp, const double (*xv)[6], const DControl* ctl)
{
  const unsigned FULL = 0xffffffffu;
  const unsigned lane = threadIdx.x & 31u;
  const DTallies& T = tallies[item];
  const bool good = ended && end < END_KILL;
  if(ended && end >= END_FAIL) {
    /* The failure that reaches the limit stops the launch's work fetch
     * (src/ssol_solver.c:1240-1245) */
    const unsigned long long nf = atomicAdd(&T.counters[0], 1ull) + 1ull;
    if(ctl && ctl->stop && nf >= ctl->max_failed) atomicExch(ctl->stop, 1ull);
    if(end == END_OVERFLOW) atomicAdd(&T.counters[2], 1ull);
  }
  if(ended && end == END_KILL) atomicAdd(&T.counters[1], 1ull);
  const int samp = ended ? p_samp : -1;
  const int nent = good ? p_nent : 0;
  const int r0 = nent ? p_r0 : -1;
  double f = 0, wcos = 0, wabs = 0, wsh = 0, wmiss = 0, watm = 0, woth = 0;
  double q[NRCV_Q] = {0, 0, 0, 0, 0, 0, 0, 0, 0, 0};
  double chk = 0;
  if(good) {
    f = (double)(1ull << score);
    wcos = f * ps[PS_COS * stride];
    wabs = f * ps[PS_ABS * stride];
    watm = f * ps[PS_ATM * stride];
    woth = f * ps[PS_OTHER * stride];
    const double w_end = f * weight;
    if(end == END_SHADOW) wsh = w_end;
    if(end == END_MISS) wmiss = w_end;
    chk = wcos * wcos + wabs * wabs + watm * watm + woth * woth + w_end * w_end;
    if(nent == 1) {
      const double a0 = ps[(PS_V0 + 0) * stride], a1 = ps[(PS_V0 + 1) * stride];
      const double a2 = ps[(PS_V0 + 2) * stride], a3 = ps[(PS_V0 + 3) * stride];
      const double a4 = ps[(PS_V0 + 4) * stride], a5 = ps[(PS_V0 + 5) * stride];
      q[0] = f * a0; q[1] = f * a1; q[2] = f * a2;
      q[3] = f * (a2 - a0); q[4] = f * (a1 - a0);
      q[5] = f * a3; q[6] = f * a4; q[7] = f * a5;
      q[8] = f * (a5 - a3); q[9] = f * (a4 - a3);
#pragma unroll
      for(int k = 0; k < NRCV_Q; ++k) chk += q[k] * q[k];
    }
  }
  /* Finite, and its squares too */
  const bool tame = chk < 1e300;

  /* Global quantities, item by item (one, unless a batch's warp straddles
   * two) */
  unsigned rest = __ballot_sync(FULL, good && tame);
#pragma unroll 1
  while(rest) {
    const int it = __shfl_sync(FULL, item, __ffs(rest) - 1);
    const bool in = good && tame && item == it;
    rest &= ~__ballot_sync(FULL, in);
    if(wk->gitem != it) {
      flush_global(tallies, wk, tile);
      __syncwarp();
      if(lane == 0) wk->gitem = it;
      __syncwarp();
    }
    double2 d = tile[0];
    tile_add(d, 0, lane, in ? wabs : 0.0);
    tile_add(d, 1, lane, in ? wabs * wabs : 0.0);
    tile_add(d, 2, lane, in ? wmiss : 0.0);
    tile_add(d, 3, lane, in ? wmiss * wmiss : 0.0);
    tile_add(d, 4, lane, in ? watm : 0.0);
    tile_add(d, 5, lane, in ? watm * watm : 0.0);
    tile_add(d, 6, lane, in ? woth : 0.0);
    tile_add(d, 7, lane, in ? woth * woth : 0.0);
    tile[0] = d;
  }
  if(good && !tame) {
    const double g[4] = {wabs, wmiss, watm, woth};
    const int at[4] = {G_ABS_RCV, G_MISSING, G_ATM, G_OTHER};
    for(int k = 0; k < 4; ++k) {
      red_add_global(T.global + 2 * at[k], g[k]);
      red_add_global(T.global + 2 * at[k] + 1, g[k] * g[k]);
    }
  }

  /* Sampled instances and their receivers: at most two of a warp's sampled
   * instances through the tiles */
  bool counted = !ended, samp_done = !good, rcv_done = nent != 1;
  rest = __ballot_sync(FULL, ended);
#pragma unroll 1
  for(int pass = 0; pass < 2 && rest; ++pass) {
    const int leader = __ffs(rest) - 1;
    const int ks = __shfl_sync(FULL, samp, leader), it = __shfl_sync(FULL, item, leader);
    const unsigned grp = __ballot_sync(FULL, ended && samp == ks && item == it);
    if(__popc(grp) < MIN_GROUP) break;
    rest &= ~grp;
    const bool in = ((grp >> lane) & 1u) && tame;
    if((int)lane == leader) red_count_global(&T.nb_samples[ks], (unsigned long long)__popc(grp));
    const unsigned have = __ballot_sync(FULL, in && nent == 1);
    int rb = have ? __shfl_sync(FULL, samp * nrcv + r0, __ffs(have) - 1) : -1;
    const bool on_r = in && nent == 1 && samp * nrcv + r0 == rb;
    if(wk->item != it || wk->samp != ks) {
      flush_samp(tallies, wk, tile, stride, false);
      __syncwarp();
      if(lane == 0) { wk->item = it; wk->samp = ks; wk->rbase = rb; }
    } else if(rb >= 0 && wk->rbase != rb) {
      flush_samp(tallies, wk, tile, stride, true);
      __syncwarp();
      if(lane == 0) wk->rbase = rb;
    }
    __syncwarp();
    double2 d = tile[stride];
    tile_add(d, 0, lane, in ? wcos : 0.0);
    tile_add(d, 1, lane, in ? wcos * wcos : 0.0);
    tile_add(d, 2, lane, in ? wsh : 0.0);
    tile_add(d, 3, lane, in ? wsh * wsh : 0.0);
    if(rb >= 0) {
      double2 e = tile[2 * stride], h = tile[3 * stride];
      double v[NRCV_Q];
#pragma unroll
      for(int k = 0; k < NRCV_Q; ++k) v[k] = on_r ? q[k] : 0.0;
#pragma unroll
      for(int k = 0; k < 4; ++k) {
        if(k < 2) {
          tile_add(d, 4 + 2 * k, lane, v[k]);
          tile_add(d, 5 + 2 * k, lane, v[k] * v[k]);
        }
        tile_add(e, 2 * k, lane, v[2 + k]);
        tile_add(e, 2 * k + 1, lane, v[2 + k] * v[2 + k]);
        tile_add(h, 2 * k, lane, v[6 + k]);
        tile_add(h, 2 * k + 1, lane, v[6 + k] * v[6 + k]);
      }
      tile[2 * stride] = e;
      tile[3 * stride] = h;
    }
    tile[stride] = d;
    counted = counted || ((grp >> lane) & 1u);
    samp_done = samp_done || in;
    rcv_done = rcv_done || on_r;
  }
  if(!counted) red_count_global(&T.nb_samples[samp], 1ull);
  if(!samp_done) {
    double* sp = T.samp + (size_t)samp * 4;
    red_add_global(sp + 0, wcos);
    red_add_global(sp + 1, wcos * wcos);
    red_add_global(sp + 2, wsh);
    red_add_global(sp + 3, wsh * wsh);
  }
  if(nent == 1) {
    const double a0 = ps[(PS_V0 + 0) * stride], a1 = ps[(PS_V0 + 1) * stride];
    const double a2 = ps[(PS_V0 + 2) * stride], a3 = ps[(PS_V0 + 3) * stride];
    const double a4 = ps[(PS_V0 + 4) * stride], a5 = ps[(PS_V0 + 5) * stride];
    if(!rcv_done)
      commit10(T.samp_rcv + ((size_t)samp * nrcv + r0) * NRCV_Q * 2, a0, a1, a2, a3, a4, a5, f);
    if(p0 >= 0)
      commit10(T.prim + (size_t)p0 * NRCV_Q * 2, a0, a1, a2, a3, a4, a5, f);
  } else if(nent > 1) {
    double v0[6];
    for(int k = 0; k < 6; ++k) v0[k] = ps[(PS_V0 + k) * stride];
    /* Several entries: sum per receiver side and per primitive before
     * squaring (deferred mc_data semantics) */
    for(int e = 0; e < nent; ++e) {
      const int re = e == 0 ? r0 : xr[e - 1];
      bool seen = false;
      for(int k = 0; k < e && !seen; ++k) seen = (k == 0 ? r0 : xr[k - 1]) == re;
      if(!seen) {
        double v[6] = {0, 0, 0, 0, 0, 0};
        for(int k = e; k < nent; ++k) {
          if((k == 0 ? r0 : xr[k - 1]) != re) continue;
          for(int c = 0; c < 6; ++c) v[c] += k == 0 ? v0[c] : xv[k - 1][c];
        }
        commit10(T.samp_rcv + ((size_t)samp * nrcv + re) * NRCV_Q * 2, v, f);
      }
      const int prim = e == 0 ? p0 : xp[e - 1];
      if(prim >= 0) {
        /* (receiver side, primitive) keys are unique among the entries */
        commit10(T.prim + (size_t)prim * NRCV_Q * 2, e == 0 ? v0 : xv[e - 1], f);
      }
    }
  }
  __syncwarp();
}

/* The sums that follow from others, once a launch (block y: the item): a
 * receiver side's from its samp_rcv slots, the global cosine and shadowed
 * from the samp slots. Block x: that group of `group` receiver sides, whose
 * slots of one sampled instance are neighbours; the last one: the globals.
 * Block z: its slice of the sampled instances; slices add up in what
 * finish_clear has zeroed, a single one stores. */
constexpr int FINISH_BLOCK = 960;
template<class R>
__global__ void __launch_bounds__(FINISH_BLOCK) finish_tallies
  (const DScene<R>* scenes, const DTallies* tallies, const DTallies one, int nrcv,
   int nsampled, int group)
{
  __shared__ double2 part[FINISH_BLOCK];
  const DTallies& T = tallies ? tallies[blockIdx.y] : one;
  if(scenes) { nrcv = scenes[blockIdx.y].nrcv; nsampled = scenes[blockIdx.y].nsampled; }
  const bool glob = blockIdx.x == gridDim.x - 1;
  const int r = (int)blockIdx.x * group;
  if(!glob && r >= nrcv) return;
  /* Sums in pairs (16-byte loads): 10 of a receiver side, 2 of the globals */
  const int width = glob ? 2 : min(group, nrcv - r) * NRCV_Q;
  const int lanes = FINISH_BLOCK / width;
  const int q = threadIdx.x % width, l = threadIdx.x / width;
  const double2* src = reinterpret_cast<const double2*>
    (glob ? T.samp : T.samp_rcv + (size_t)r * NRCV_Q * 2) + q;
  const size_t step = glob ? 2 : (size_t)nrcv * NRCV_Q;
  double2 v = make_double2(0.0, 0.0);
  const int per = (nsampled + (int)gridDim.z - 1) / (int)gridDim.z;
  const int last = min(nsampled, ((int)blockIdx.z + 1) * per);
  if(l < lanes)
#pragma unroll 8
    for(int s = (int)blockIdx.z * per + l; s < last; s += lanes) {
      const double2 w = __ldcs(src + (size_t)s * step); /* the scene stays in the L2 */
      v.x += w.x;
      v.y += w.y;
    }
  part[threadIdx.x] = v;
  /* Halves of the lanes, then the sums of the first one */
  for(int n = lanes; n > 1; ) {
    const int h = (n + 1) / 2;
    __syncthreads();
    if(l < n - h) {
      const double2 w = part[threadIdx.x + h * width];
      v.x += w.x;
      v.y += w.y;
      part[threadIdx.x] = v;
    }
    n = h;
  }
  if(l) return;
  double* dst = glob ? T.global + (q == 0 ? 2 * G_COS : 2 * G_SHADOW)
                     : T.rcv + (size_t)r * NRCV_Q * 2 + 2 * q;
  if(gridDim.z == 1) {
    dst[0] = v.x;
    dst[1] = v.y;
  } else {
    red_add_global(dst, v.x);
    red_add_global(dst + 1, v.y);
  }
}
template<class R>
__global__ void __launch_bounds__(256) finish_clear
  (const DScene<R>* scenes, const DTallies* tallies, const DTallies one, int nrcv)
{
  const DTallies& T = tallies ? tallies[blockIdx.x] : one;
  if(scenes) nrcv = scenes[blockIdx.x].nrcv;
  for(int i = threadIdx.x; i < nrcv * NRCV_Q * 2; i += blockDim.x) T.rcv[i] = 0.0;
  if(threadIdx.x < 2) {
    T.global[2 * G_COS + threadIdx.x] = 0.0;
    T.global[2 * G_SHADOW + threadIdx.x] = 0.0;
  }
}

/* Sampled instances that one block adds up by itself, and those of a slice
 * where there are more. One block for all of a receiver side's grew with the
 * plant: us a plan launch of 1e4 paths, one receiver side, one block / slices:
 * 2000 sampled instances 124 / 123 (of two launches), 2500 126 / 122, 5000
 * 138 / 125, 20,000 198 / 128, 1e5 418 / 127.
 * Many receiver sides of many instances fill more than a share of the L2 and
 * are bound by HBM. From 64 MB on a block takes FINISH_WIDE neighbouring sides
 * (1920 bytes of a row), in as many slices as one wave of blocks has, of
 * FINISH_DEEP rows a thread or more; below, the same takes as long. Plan launches
 * of 1e4 paths, a side a block / so: 20,000 x 100 sides (320 MB) 237 / 209 us,
 * 5000 x 400 227 / 207, 5000 x 100 168 / 160. */
constexpr int FINISH_SINGLE = 2048, FINISH_SLICE = 1024, FINISH_SLICES_MAX = 64;
constexpr int FINISH_WIDE = 12, FINISH_DEEP = 8, FINISH_WAVE = 2 * 148;
constexpr uint64_t FINISH_WIDE_SLOTS = 400000;
template<class R>
static void launch_finish(const DScene<R>* scenes, const DTallies* tallies, const DTallies& one,
                          int nitems, int nrcv, int nsampled, cudaStream_t st)
{
  int group = 1, slices = 1;
  if(nrcv > 1 && (uint64_t)nitems * nrcv * nsampled >= FINISH_WIDE_SLOTS) {
    group = std::min(nrcv, FINISH_WIDE);
    const int rows = FINISH_DEEP * (FINISH_BLOCK / (group * NRCV_Q));
    const int64_t blocks = (int64_t)nitems * ((nrcv + group - 1) / group + 1);
    slices = (int)std::min<int64_t>((nsampled + rows - 1) / rows,
                                    std::max<int64_t>(FINISH_WAVE / blocks, 1));
  } else if(nsampled > FINISH_SINGLE) {
    slices = std::min((nsampled + FINISH_SLICE - 1) / FINISH_SLICE, FINISH_SLICES_MAX);
  }
  if(slices > 1) finish_clear<R><<<(unsigned)nitems, 256, 0, st>>>(scenes, tallies, one, nrcv);
  const unsigned groups = (unsigned)((nrcv + group - 1) / group);
  for(int i = 0; i < nitems; i += 65535)
    finish_tallies<R><<<dim3(groups + 1, (unsigned)std::min(nitems - i, 65535),
                             (unsigned)slices), FINISH_BLOCK, 0, st>>>
      (scenes ? scenes + i : nullptr, tallies ? tallies + i : nullptr, one, nrcv, nsampled, group);
}

/*******************************************************************************
 * Kernel
 ******************************************************************************/
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
  for(int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long v)
{
#pragma unroll
  for(int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

constexpr int MAX_BLOCK = 256;
/* The paths of a warp advance together: its ended lanes wait until few are
 * still under way, then commit at once and start the next realisations
 * together. In the coherent order the lanes of a warp start on one heliostat,
 * so their shadow rays, and then their reflected rays, are nearly parallel
 * and visit the same nodes; refilling each lane as it ended (the former rule)
 * mixed shadow and path rays in every cast. `few`: none for the first
 * REGEN_AGE casts of meshes, 8 with quadrics or dielectrics, whose paths are
 * longer and uneven; after REGEN_AGE casts at least REGEN_LATE, so that deep
 * paths do not hold a warp. Field, 1e8 paths, lanes 32 (refill at once) / 16 /
 * 8 / 2 / 0: 145 / 107 / 97.0 / 94.5 / 92.5 ms; beam-down, 6e7: 216 / 161 /
 * 160 / 169 / 175 ms; a matte cavity, 1e7: 13.9 / 12.4 / 13.7 / 17.4 / 21.0,
 * with 2 and then more after 3 casts 12.9. */
constexpr int REGEN_AGE = 3, REGEN_LATE = 12;
static int regen_lanes(int features)
{ return features & (FEAT_QUADRIC | FEAT_DIELECTRIC) ? 8 : 0; }
/* SMs per item group of the batched kernel's work order: small items
 * (fewer than BATCH_LARGE_ITEM realisations on average) by groups of 8 SMs,
 * larger ones by 16. Measured on 256 field items (Mpaths/s, groups of 8 /
 * 16 / 37 SMs): 1e5 each 437 / 420 / 345, 1e6 each 482 / 489 / 485. */
constexpr int BATCH_GROUP_SMALL = 8, BATCH_GROUP_LARGE = 16;
constexpr unsigned long long BATCH_LARGE_ITEM = 400000;
/* Coherent order (see presort_count) */
constexpr int SORT_MAX_BINS = 12288; /* shared-memory histogram of primitives */
constexpr uint64_t SORT_CHUNK = 1ull << 24; /* realisations per sorted chunk */
/* Smaller launches keep the id order: there the presort (25 to 50 us) costs
 * more than it gives. us a launch, id order / sorted: field of 1000, 1e5
 * paths 172 / 179, 3e5 389 / 348, 1e6 1088 / 897, 7e6 7036 / 5549; field of
 * 30, 3e5 565 / 377; beam-down of 1000, 3e5 847 / 948, 1e6 2658 / 2650, 3e6
 * 7914 / 7262. A single sampled instance has its lanes on one surface already:
 * one mirror, 1e6, 349 / 377; a dish of 128 triangles, 1e6, 583 / 588, of
 * 2048, 1041 / 958. */
constexpr uint64_t SORT_MIN = 200000, SORT_MIN_QUADRIC = 1000000;
constexpr int SORT_SINGLE = 1024;
/* Launches that are being captured, whose scratch the graph would hold, sort
 * from here on only */
constexpr uint64_t SORT_MIN_CAPTURED = 6000000;
/* Segments a warp gets on average before they shrink from SORT_SEG to 32
 * realisations: with 1 / 2 / 4 / 8 the field's 1e6 paths take 1180 / 1007 /
 * 931 / 899 us, as the last segments leave fewer warps waiting */
constexpr uint64_t SORT_SHARE = 8;
constexpr uint32_t SORT_SEG = SORT_SEGMENT; /* sorted realisations per warp segment */

/* Append one vertex of a tracked path (src/ssol_solver.c:909-922, 1014-1019,
 * 1080-1083: the sun end, the sampled point, every hit and the end at
 * infinity, each with the flux carried to it) */
template<class R>
__device__ __forceinline__ void track_vertex
  (const DTrack& tr, PathState<R>& p, V3<R> x, double w)
{
  const unsigned long long k = atomicAdd(tr.nverts, 1ull);
  if(k < tr.cap) {
    TrackVertex& v = tr.verts[k];
    v.slot = (uint32_t)p.tslot;
    v.seq = p.tseq;
    v.pos[0] = (double)x.x;
    v.pos[1] = (double)x.y;
    v.pos[2] = (double)x.z;
    v.weight = w;
  }
  ++p.tseq;
}

template<class R, int MINB, bool TRACK, int FEAT>
__global__ void __launch_bounds__(MAX_BLOCK, sizeof(R) == 4 && MINB == 3 ? 4 : MINB)
realisation_kernel
  (const DScene<R> S, const DTallies T,
   uint64_t seed, uint64_t first, uint64_t count, unsigned long long max_segments,
   unsigned long long* next_path, const DTrack tr,
   const uint32_t* sorted_off, uint32_t seg_len, uint32_t seg_mul,
   const DControl ctl)
{
  /* Shared memory: per-thread FP64 path sums [ps_count][blockDim], the
   * warps' tally tiles [TILES][blockDim]; shared memory left unused goes to
   * the L1 cache */
  extern __shared__ double2 smem[];
  __shared__ double red[MAX_BLOCK / 32][8];
  __shared__ WarpKeys keys[MAX_BLOCK / 32];
  __shared__ DTallies tallies;
  const int bd = blockDim.x, tid = threadIdx.x;
  const unsigned lane = tid & 31u;
  double2* tile = smem + tid;
  double* ps = reinterpret_cast<double*>(smem + TILES * bd) + tid;
  WarpKeys* wk = keys + (tid >> 5);
  for(int k = 0; k < TILES; ++k) tile[k * bd] = make_double2(0.0, 0.0);
  if(lane == 0) *wk = {0, 0, -1, -1};
  if(tid == 0) tallies = T;
  __syncthreads();

  Rng rng;
  rng.k0 = (uint32_t)seed;
  rng.k1 = (uint32_t)(seed >> 32);
  PathState<R> p;
  p.phase = PH_NONE;
  bool done = false;
  Counters cnt = {0, 0, 0, 0};
  uint32_t bounces = 0, npaths = 0;
  int xr[MAX_EXTRA], xp[MAX_EXTRA];
  double xv[MAX_EXTRA][6];

  /* Coherent order: the warp's current segment [seg_cur, seg_end) of the
   * sorted realisations */
  uint32_t seg_cur = 0, seg_end = 0;
  const uint32_t nseg = sorted_off ? (uint32_t)((count + seg_len - 1) / seg_len) : 0u;
  const bool polled = ctl.stop || ctl.abort;
  uint32_t fetches = 0;
  int age = 0; /* casts since the warp last took realisations */

  for(;;) {
    /* The warp's paths advance together (regen_lanes) */
    unsigned need = 0;
    if(__popc(__ballot_sync(0xffffffffu, p.phase == PH_SHADOW || p.phase == PH_BOUNCE))
       <= (age <= REGEN_AGE ? ctl.regen : max(ctl.regen, REGEN_LATE))) {
      age = 0;
      if(__any_sync(0xffffffffu, p.phase == PH_ENDED)) {
        commit_warp(S.nrcv, &tallies, 0, p.phase == PH_ENDED, p.end, p.samp, p.score, p.nent,
                    p.r0, p.p0, p.prev[0], ps, bd, tile, wk, xr, xp, xv, &ctl);
        if(p.phase == PH_ENDED) p.phase = PH_NONE;
      }
      need = __ballot_sync(0xffffffffu, p.phase == PH_NONE && !done);
    }
    bool start = false;
    uint64_t off = 0;
    /* Early stop: every 4th fetch of the warp (of 32 realisations or so)
     * reads the stop and abort words (one L2 sector); a halted warp takes no
     * new realisation, also for the lanes whose paths end later */
    bool halt = false;
    if(need && polled && (fetches++ & 3u) == 0u) {
      const int leader = __ffs(need) - 1;
      int h = 0;
      if((int)lane == leader) {
        if(ctl.stop && *(volatile const unsigned long long*)ctl.stop) h = 1;
        if(ctl.abort && *(volatile const unsigned long long*)ctl.abort) h = 1;
      }
      halt = __shfl_sync(0xffffffffu, h, leader) != 0;
    }
    if(halt) {
      done = true;
    } else if(need && sorted_off) {
      /* Segments of SORT_SEG sorted realisations (one or two primitives) go
       * to warps whole, in a strided order, so that a warp's lanes start on
       * the same heliostat while the warps of the GPU spread over the field */
      const int leader = __ffs(need) - 1;
      const unsigned rank = __popc(need & ((1u << lane) - 1u));
      const unsigned c = __popc(need);
      const unsigned avail = seg_end - seg_cur;
      uint32_t idx = 0;
      bool got = rank < avail, exhausted = false;
      if(got) idx = seg_cur + rank;
      if(c > avail) {
        unsigned long long sg = 0;
        if((int)lane == leader) sg = atomicAdd(next_path, 1ull);
        sg = __shfl_sync(0xffffffffu, sg, leader);
        if(sg < nseg) {
          const uint32_t s0 = (uint32_t)((sg * seg_mul) % nseg) * seg_len;
          const uint32_t s1 = (uint32_t)min((uint64_t)s0 + seg_len, count);
          if(!got && rank - avail < s1 - s0) {
            idx = s0 + (rank - avail);
            got = true;
          }
          seg_cur = s0 + min(c - avail, s1 - s0);
          seg_end = s1;
        } else {
          seg_cur = seg_end;
          exhausted = true;
        }
      } else {
        seg_cur += c;
      }
      if(p.phase == PH_NONE && !done) {
        if(got) {
          start = true;
          /* read once: a streaming load, evicted from L2 first */
          off = __ldcs(&sorted_off[idx]);
        } else if(exhausted) {
          done = true;
        }
      }
    } else if(need) {
      const int leader = __ffs(need) - 1;
      unsigned long long base = 0;
      if((int)lane == leader)
        base = atomicAdd(next_path, (unsigned long long)__popc(need));
      base = __shfl_sync(0xffffffffu, base, leader);
      if(p.phase == PH_NONE && !done) {
        const unsigned long long idx = base + __popc(need & ((1u << lane) - 1u));
        if(idx >= count) {
          done = true;
        } else {
          start = true;
          off = idx;
        }
      }
    }
    /* One init_path for both orders, so that a realisation computes the same
     * bits whichever order it runs in */
    if(start) {
      const uint64_t id = first + off;
      rng.i_lo = (uint32_t)id;
      rng.i_hi = (uint32_t)(id >> 32);
      init_path<R, FEAT>(S, rng, p, ps, bd);
      ++npaths;
      if(TRACK) {
        p.tslot = off < tr.npaths ? (int)off : -1;
        p.tseq = 0;
        if(p.tslot >= 0) {
          if(tr.sun_len > 0)
            track_vertex(tr, p, p.org + p.rd * (R)tr.sun_len, S.dni);
          track_vertex(tr, p, p.org, p.prev[0]);
        }
      }
    }
    if(!__any_sync(0xffffffffu, p.phase == PH_SHADOW || p.phase == PH_BOUNCE)) break;
    ++age;

    /* One ray per active lane */
    Hit<R> h;
    bool found = false;
    if(p.phase == PH_SHADOW || p.phase == PH_BOUNCE) {
      const bool shadow = p.phase == PH_SHADOW;
      SelfInfo self;
      self.gid = p.gid;
      self.sinst = p.sinst;
      self.side = p.side;
      self.discard_virtual = shadow;
      self.reversed = shadow;
      found = trace_ray<R, FEAT>(S, p.org, p.rd, p.tmin, self, shadow, h, cnt);
    }

    int end = END_NONE;
    bool do_interact = false;
    V3<R> pos = p.org, dir = -p.rd;
    if(p.phase == PH_SHADOW) {
      if(found) end = END_SHADOW;
      else {
        /* The path starts at the sampled point along the sun direction; a
         * virtual sampled surface pursues that ray (src/ssol_solver.c:
         * 988-995), not the shadow ray */
        p.rd = dir;
        do_interact = true;
      }
    } else if(p.phase == PH_BOUNCE) {
      if(!found) {
        if(TRACK && p.tslot >= 0 && tr.inf_len > 0) {
          const V3<R> last = p.virt ? p.org + p.rd * p.hit_t : p.org;
          track_vertex(tr, p, last + p.rd * (R)tr.inf_len, p.virt ? p.inc0 : p.prev[0]);
        }
        /* Last segment: the medium the ray leaves into must be the air
         * (src/ssol_solver.c:1012-1032) */
        if(p.out_medium != S.air_medium) {
          end = END_FAIL;
        } else {
          if(p.virt) {
            const double loss = p.prev[0] - p.inc0;
            ps[(p.medium == S.air_medium ? PS_ATM : PS_OTHER) * bd] += loss;
          }
          end = END_MISS;
        }
      } else {
        /* Russian roulette on deep paths (src/ssol_solver.c:1056-1075) */
        p.depth += p.virt ? 0u : 1u;
        if(p.depth > p.interval && p.depth % p.interval == 1) {
          const double u = u01d(rng.get(p.nroul++, RNG_ROULETTE).v[0]);
          if(u > 0.5) {
            ++p.score;
            p.interval = 16;
          } else {
            end = END_KILL;
          }
        }
        if(end == END_NONE) {
          /* point_update_from_hit (src/ssol_solver.c:360-411) */
          p.sinst = h.sinst;
          p.prim = h.prim;
          p.gid = h.gid;
          dir = p.rd;
          p.N = normalize_hit(h.n);
          pos = p.org + p.rd * h.t;
          if((FEAT & FEAT_ATTRIBUTES) && S.tshade && h.gid >= 0) {
            const float2 uv = tri_uv(S, h.gid, pos);
            put_uv(ps, bd, uv.x, uv.y);
          }
          if(TRACK && p.tslot >= 0)
            track_vertex(tr, p, pos, p.virt ? p.inc0 : p.prev[0]);
          p.side = dot(p.rd, p.N) < R(0) ? 1 : 2;
          if(p.side == 2) p.N = -p.N;
          p.hit_t = h.t;
          p.medium = p.out_medium;
          do_interact = true;
        }
      }
    }
    if(do_interact)
      end = interact<R, FEAT>(S, rng, p, pos, dir, bounces, max_segments, ps, bd, xr, xp, xv);
    if(end != END_NONE) {
      if(TRACK && p.tslot >= 0 && end != END_KILL) {
        /* src/ssol_solver.c:931, 1092-1094, 1122-1125; killed paths are not
         * registered (1111) */
        tr.path_type[p.tslot] = end == END_SHADOW ? 1
          : (end == END_FAIL || p.overflow) ? 3 : (p.nent > 0 ? 2 : 0);
        tr.path_nv[p.tslot] = (int32_t)p.tseq;
      }
      path_ended(p, end);
    }
  }

  /* The warps' tiles: the sampled instance's, then the global sums through a
   * block reduction */
  const int warp = tid >> 5;
  flush_samp(&tallies, wk, tile, bd, false);
  {
    const double v = tile_row_sum(tile[0]);
    if((lane & 3u) == 0u) red[warp][lane >> 2] = v;
  }
  unsigned long long c[6] = {cnt.rays, cnt.nodes, cnt.tris, cnt.quads,
                             bounces, npaths};
  for(int q = 0; q < 6; ++q) c[q] = warp_sum_u64(c[q]);
  if(lane == 0) {
    unsigned long long* st = &T.stats->rays;
    for(int q = 0; q < 6; ++q) if(c[q]) atomicAdd(st + q, c[q]);
  }
  __syncthreads();
  if(tid < 8) {
    double v = 0;
    for(int w = 0; w < (bd >> 5); ++w) v += red[w][tid];
    red_add_global(T.global + (tid < 2 ? 2 * G_ABS_RCV : 2 * G_MISSING - 2) + tid, v);
  }
}

/* Batched form: several scenes (e.g. one re-aimed field per sun position)
 * and their realisation budgets in one persistent launch. Global work index
 * g maps to item it = max{i : prefix[i] <= g} and to realisation
 * firsts[it] + g - prefix[it] of that item's streams. Every item has its own
 * tallies; a warp's tiles are keyed by the item they sum for and flushed when
 * it commits for another one. The launch's total is prefix[nitems], read from device
 * memory so that a captured CUDA graph replays with new budgets. */
template<class R, int MINB, int FEAT>
__global__ void __launch_bounds__(MAX_BLOCK, sizeof(R) == 4 && MINB == 3 ? 4 : MINB)
batch_kernel
  (const DScene<R>* __restrict__ scenes, const DTallies* __restrict__ tallies,
   const unsigned long long* __restrict__ prefix,
   const unsigned long long* __restrict__ firsts, int nitems, uint64_t seed,
   unsigned long long max_segments, unsigned long long* next_items,
   DStats* stats, int regen, const uint32_t* __restrict__ sorted_off,
   const uint32_t* __restrict__ seg_mul)
{
  extern __shared__ double2 smem[];
  __shared__ WarpKeys keys[MAX_BLOCK / 32];
  const int bd = blockDim.x, tid = threadIdx.x;
  const unsigned lane = tid & 31u;
  double2* tile = smem + tid;
  double* ps = reinterpret_cast<double*>(smem + TILES * bd) + tid;
  WarpKeys* wk = keys + (tid >> 5);
  for(int k = 0; k < TILES; ++k) tile[k * bd] = make_double2(0.0, 0.0);
  if(lane == 0) *wk = {-1, -1, -1, -1};
  /* Two slots per warp tagged with an item (its current item and the
   * previous one, for the paths still running across an item boundary) hold
   * copies of the items' scene records, so that lanes on those items read
   * their scene from shared memory instead of device memory. Tags change
   * only where the warp is converged. */
  DScene<R>* wscene = reinterpret_cast<DScene<R>*>(
    reinterpret_cast<double*>(smem + TILES * bd) + ps_count(FEAT) * bd) + (size_t)(tid >> 5) * 2;
  __syncwarp();
  int stag[2] = {-1, -1};
  int cur = 0;
  auto scene_of = [&](int item) -> const DScene<R>& {
    return item == stag[cur] ? wscene[cur] : item == stag[cur ^ 1] ? wscene[cur ^ 1]
                                                                   : scenes[item];
  };

  /* Work: every item has its own counter (next_items). The SMs form groups
   * of group_sms; group g works through its own items g, g + G, g + 2G, ...
   * in turn, then through the next groups' lists, taking its realisations
   * from the first item of the sequence with work left. The warps of an SM
   * thus stay long on one item (its scene arrays stay warm in L1 and the
   * item tags rarely change), and only about G items are open at a time
   * (their arrays and tallies stay in L2). Positions q of the sequence map
   * to items (q % L) x G + q / L, L = ceil(nitems / G); those past the last
   * item are skipped. Measured on 256 field items: with one counter over
   * all items (every warp moved to the next item at the same time, its
   * arrays cold for all of them) 1e5 realisations per item ran at 199
   * Mpaths/s; with every SM starting on its own item 416, and 1e6 per item
   * 436 (about 150 items open). */
  const unsigned long long total = prefix[nitems];
  unsigned smid, nsmid;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
  asm volatile("mov.u32 %0, %%nsmid;" : "=r"(nsmid));
  const unsigned group_sms = total < BATCH_LARGE_ITEM * (unsigned long long)nitems
                            ? BATCH_GROUP_SMALL : BATCH_GROUP_LARGE;
  const int ngroups = min(nitems, max(1, (int)(nsmid / group_sms)));
  const int seq_len = (nitems + ngroups - 1) / ngroups;
  const int npos = ngroups * seq_len;
  int wq = (int)(min(smid, nsmid - 1) * (unsigned)ngroups / nsmid) * seq_len;
  int wit = 0;
  Rng rng;
  rng.k0 = (uint32_t)seed;
  rng.k1 = (uint32_t)(seed >> 32);
  PathState<R> p;
  p.phase = PH_NONE;
  int it = 0;
  bool done = total == 0;
  Counters cnt = {0, 0, 0, 0};
  uint32_t bounces = 0, npaths = 0;
  int xr[MAX_EXTRA], xp[MAX_EXTRA];
  double xv[MAX_EXTRA][6];
  int age = 0; /* casts since the warp last took realisations */

  for(;;) {
    /* The warp's paths advance together (regen_lanes) */
    unsigned need = 0;
    if(__popc(__ballot_sync(0xffffffffu, p.phase == PH_SHADOW || p.phase == PH_BOUNCE))
       <= (age <= REGEN_AGE ? regen : max(regen, REGEN_LATE))) {
      age = 0;
      if(__any_sync(0xffffffffu, p.phase == PH_ENDED)) {
        commit_warp(scene_of(it).nrcv, tallies, it, p.phase == PH_ENDED, p.end, p.samp, p.score,
                    p.nent, p.r0, p.p0, p.prev[0], ps, bd, tile, wk, xr, xp, xv,
                    (const DControl*)nullptr);
        if(p.phase == PH_ENDED) p.phase = PH_NONE;
      }
      need = __ballot_sync(0xffffffffu, p.phase == PH_NONE && !done);
    }
    if(need) {
      const int leader = __ffs(need) - 1;
      unsigned long long base = 0;
      int item = wit, got = 0, q = wq;
      if((int)lane == leader) {
        /* The warp's position, or the next ones in turn, until an item has
         * work */
        for(int k = 0; k < npos; ++k) {
          item = (q % seq_len) * ngroups + q / seq_len;
          if(item < nitems) {
            const unsigned long long budget = prefix[item + 1] - prefix[item];
            if(*(volatile const unsigned long long*)(next_items + item) < budget) {
              base = atomicAdd(next_items + item, (unsigned long long)__popc(need));
              if(base < budget) { got = 1; break; }
            }
          }
          q = q + 1 == npos ? 0 : q + 1;
        }
      }
      got = __shfl_sync(0xffffffffu, got, leader);
      item = __shfl_sync(0xffffffffu, item, leader);
      q = __shfl_sync(0xffffffffu, q, leader);
      base = __shfl_sync(0xffffffffu, base, leader);
      if(got) { wit = item; wq = q; }
      if(p.phase == PH_NONE && !done) {
        const unsigned long long g = base + __popc(need & ((1u << lane) - 1u));
        if(!got) {
          done = true;
        } else if(g < prefix[item + 1] - prefix[item]) {
          /* lanes past the item's end take work at the next fetch */
          it = item;
          /* Coherent order: the item's full warp segments of SORT_SEG
           * sorted realisations in a strided order (so that the warps of an
           * item group spread over its primitives), the ragged last one
           * last; each record is a realisation's offset in the item */
          uint64_t off = g;
          if(sorted_off) {
            const unsigned long long nfull = (prefix[it + 1] - prefix[it]) / SORT_SEG;
            unsigned long long sg = g / SORT_SEG;
            if(sg < nfull)
              sg = nfull < 65536ull
                ? (unsigned long long)((uint32_t)sg * seg_mul[it] % (uint32_t)nfull)
                : sg * seg_mul[it] % nfull;
            const unsigned long long rec = prefix[it] + sg * SORT_SEG + g % SORT_SEG;
            off = __ldcs(&sorted_off[rec]);
          }
          const uint64_t id = firsts[it] + off;
          rng.i_lo = (uint32_t)id;
          rng.i_hi = (uint32_t)(id >> 32);
          init_path<R, FEAT>(scene_of(it), rng, p, ps, bd);
          ++npaths;
        }
      }
      {
        /* Converged: the item fetched becomes the current slot */
        const int newest = got ? wit : -1;
        if(newest >= 0 && newest != stag[cur]) {
          const int prv = cur ^ 1;
          /* every lane's reads of the slot's old scene are done */
          __syncwarp();
          {
            const int* src = reinterpret_cast<const int*>(scenes + newest);
            int* dst = reinterpret_cast<int*>(wscene + prv);
            constexpr int words = (int)(sizeof(DScene<R>) / sizeof(int));
            for(int i = (int)lane; i < words; i += 32) dst[i] = src[i];
          }
          __syncwarp();
          stag[prv] = newest;
          cur = prv;
        }
      }
    }
    if(!__any_sync(0xffffffffu, p.phase == PH_SHADOW || p.phase == PH_BOUNCE)) break;
    ++age;

    const DScene<R>& S = scene_of(it);
    Hit<R> h;
    bool found = false;
    if(p.phase == PH_SHADOW || p.phase == PH_BOUNCE) {
      const bool shadow = p.phase == PH_SHADOW;
      SelfInfo self;
      self.gid = p.gid;
      self.sinst = p.sinst;
      self.side = p.side;
      self.discard_virtual = shadow;
      self.reversed = shadow;
      found = trace_ray<R, FEAT>(S, p.org, p.rd, p.tmin, self, shadow, h, cnt);
    }

    int end = END_NONE;
    bool do_interact = false;
    V3<R> pos = p.org, dir = -p.rd;
    if(p.phase == PH_SHADOW) {
      if(found) end = END_SHADOW;
      else {
        /* The path starts at the sampled point along the sun direction; a
         * virtual sampled surface pursues that ray (src/ssol_solver.c:
         * 988-995), not the shadow ray */
        p.rd = dir;
        do_interact = true;
      }
    } else if(p.phase == PH_BOUNCE) {
      if(!found) {
        if(p.out_medium != S.air_medium) {
          end = END_FAIL;
        } else {
          if(p.virt) {
            const double loss = p.prev[0] - p.inc0;
            ps[(p.medium == S.air_medium ? PS_ATM : PS_OTHER) * bd] += loss;
          }
          end = END_MISS;
        }
      } else {
        p.depth += p.virt ? 0u : 1u;
        if(p.depth > p.interval && p.depth % p.interval == 1) {
          const double u = u01d(rng.get(p.nroul++, RNG_ROULETTE).v[0]);
          if(u > 0.5) {
            ++p.score;
            p.interval = 16;
          } else {
            end = END_KILL;
          }
        }
        if(end == END_NONE) {
          p.sinst = h.sinst;
          p.prim = h.prim;
          p.gid = h.gid;
          dir = p.rd;
          p.N = normalize_hit(h.n);
          pos = p.org + p.rd * h.t;
          if((FEAT & FEAT_ATTRIBUTES) && S.tshade && h.gid >= 0) {
            const float2 uv = tri_uv(S, h.gid, pos);
            put_uv(ps, bd, uv.x, uv.y);
          }
          p.side = dot(p.rd, p.N) < R(0) ? 1 : 2;
          if(p.side == 2) p.N = -p.N;
          p.hit_t = h.t;
          p.medium = p.out_medium;
          do_interact = true;
        }
      }
    }
    if(do_interact)
      end = interact<R, FEAT>(S, rng, p, pos, dir, bounces, max_segments, ps, bd, xr, xp, xv);
    if(end != END_NONE) {
      path_ended(p, end);
    }
  }

  flush_samp(tallies, wk, tile, bd, false);
  flush_global(tallies, wk, tile);
  unsigned long long c[6] = {cnt.rays, cnt.nodes, cnt.tris, cnt.quads,
                             bounces, npaths};
  for(int q = 0; q < 6; ++q) c[q] = warp_sum_u64(c[q]);
  if(lane == 0) {
    unsigned long long* st = &stats->rays;
    for(int q = 0; q < 6; ++q) if(c[q]) atomicAdd(st + q, c[q]);
  }
}

/*******************************************************************************
 * Coherent order. The realisations of a launch, chunk by chunk, are sorted by
 * the primitive their primary draw samples (a counting sort), so that the
 * lanes of a warp start on the same or neighbouring heliostats and trace
 * nearly parallel shadow and reflected rays. Every realisation is traced once
 * with its own stream; only the order, and so the order of the FP64 sums,
 * changes. Only the sorted offsets are kept, 4 bytes a realisation: the
 * kernel draws the primary sample again (one Philox block) rather than read
 * it back. Bound by the rank atomics in shared memory: 16.8e6 realisations
 * take 57 us to count and 160 us to scatter (480 with tiles of 4096, which
 * sent four times the global atomics, and 16 bytes of draws scattered with
 * each offset).
 ******************************************************************************/

/* Bins of the sort: the sampled primitives, 2^shift neighbours to a bin where
 * there are more than the shared-memory histogram holds (neighbours belong to
 * one instance or to the next) */
__host__ __device__ inline int sort_shift(int nsamp)
{
  int s = 0;
  while(((nsamp - 1) >> s) + 1 > SORT_MAX_BINS) ++s;
  return s;
}

/* Bin of realisation first + j, counted per block in shared memory */
template<class R>
__global__ void __launch_bounds__(256) presort_count
  (const DScene<R> S, uint64_t seed, uint64_t first, uint32_t n, int shift, int nb,
   uint32_t* hist)
{
  __shared__ uint32_t h[SORT_MAX_BINS];
  for(int i = threadIdx.x; i < nb; i += blockDim.x) h[i] = 0;
  __syncthreads();
  Rng rng;
  rng.k0 = (uint32_t)seed;
  rng.k1 = (uint32_t)(seed >> 32);
  for(uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n;
      j += gridDim.x * blockDim.x) {
    const uint64_t id = first + j;
    rng.i_lo = (uint32_t)id;
    rng.i_hi = (uint32_t)(id >> 32);
    atomicAdd(&h[sample_prim(S, rng.get(0u, RNG_PRIMARY)) >> shift], 1u);
  }
  __syncthreads();
  for(int i = threadIdx.x; i < nb; i += blockDim.x)
    if(h[i]) atomicAdd(&hist[i], h[i]);
}

/* Exclusive prefix sums of histogram bins: block b scans the bins of item b
 * of a batch, from its first bin in bin_base to the next item's (`nb` for the
 * last), starting at prefix[b], the budgets before it; without bin_base one
 * block scans all `nb` */
constexpr int SCAN_BLOCK = 512;
static __global__ void __launch_bounds__(SCAN_BLOCK) presort_scan
  (const uint32_t* hist, uint32_t* off, int nb, const uint32_t* bin_base,
   const unsigned long long* prefix)
{
  __shared__ uint32_t part[SCAN_BLOCK];
  const int t = threadIdx.x;
  const int first = bin_base ? (int)bin_base[blockIdx.x] : 0;
  const int last = bin_base && blockIdx.x + 1 < gridDim.x ? (int)bin_base[blockIdx.x + 1] : nb;
  const int per = (last - first + SCAN_BLOCK - 1) / SCAN_BLOCK;
  const int b0 = min(first + t * per, last), b1 = min(b0 + per, last);
  uint32_t sum = 0;
  for(int i = b0; i < b1; ++i) sum += hist[i];
  part[t] = sum;
  __syncthreads();
  for(int d = 1; d < SCAN_BLOCK; d <<= 1) {
    const uint32_t v = t >= d ? part[t - d] : 0u;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  uint32_t run = (t ? part[t - 1] : 0u) + (prefix ? (uint32_t)prefix[blockIdx.x] : 0u);
  for(int i = b0; i < b1; ++i) {
    off[i] = run;
    run += hist[i];
  }
}

/* Each realisation to the next free place of its bin's range. A block ranks a
 * tile of SCATTER_PER x SCATTER_BLOCK realisations in shared memory, reserves
 * one range per bin of the tile with a single global atomic, then writes the
 * realisations' offsets */
constexpr int SCATTER_PER = 16, SCATTER_BLOCK = 1024;

template<class R>
__global__ void __launch_bounds__(SCATTER_BLOCK) presort_scatter
  (const DScene<R> S, uint64_t seed, uint64_t first, uint32_t n, int shift, int nb,
   uint32_t* off, uint32_t* out_off)
{
  __shared__ uint32_t cnt[SORT_MAX_BINS];
  const uint32_t tile = (uint32_t)SCATTER_BLOCK * SCATTER_PER;
  Rng rng;
  rng.k0 = (uint32_t)seed;
  rng.k1 = (uint32_t)(seed >> 32);
  for(uint64_t t0 = (uint64_t)blockIdx.x * tile; t0 < n; t0 += (uint64_t)gridDim.x * tile) {
    for(int i = threadIdx.x; i < nb; i += SCATTER_BLOCK) cnt[i] = 0;
    __syncthreads();
    uint32_t k[SCATTER_PER], rank[SCATTER_PER];
#pragma unroll
    for(int e = 0; e < SCATTER_PER; ++e) {
      const uint64_t j = t0 + e * SCATTER_BLOCK + threadIdx.x;
      k[e] = 0u;
      rank[e] = 0u;
      if(j < n) {
        const uint64_t id = first + j;
        rng.i_lo = (uint32_t)id;
        rng.i_hi = (uint32_t)(id >> 32);
        k[e] = (uint32_t)sample_prim(S, rng.get(0u, RNG_PRIMARY)) >> shift;
        rank[e] = atomicAdd(&cnt[k[e]], 1u);
      }
    }
    __syncthreads();
    for(int i = threadIdx.x; i < nb; i += SCATTER_BLOCK)
      if(cnt[i]) cnt[i] = atomicAdd(&off[i], cnt[i]);
    __syncthreads();
#pragma unroll
    for(int e = 0; e < SCATTER_PER; ++e) {
      const uint64_t j = t0 + e * SCATTER_BLOCK + threadIdx.x;
      if(j < n) out_off[cnt[k[e]] + rank[e]] = (uint32_t)j;
    }
    __syncthreads();
  }
}

/* Coherent order of a batched launch. Every size comes from the launch's
 * device arrays (prefix: the budgets' inclusive prefix, prefix[nitems] the
 * total), so that a captured graph serves any budgets. Item of realisation
 * j: prefix[item] <= j < prefix[item + 1]. */
__device__ __forceinline__ int batch_item_of
  (const unsigned long long* prefix, int nitems, unsigned long long j, int hint)
{
  if(prefix[hint] <= j && j < prefix[hint + 1]) return hint;
  int lo = 0, hi = nitems;
  while(hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if(prefix[mid] <= j) lo = mid; else hi = mid;
  }
  return lo;
}

/* The two passes of the batched sort: a block takes tiles of SCATTER_PER x
 * SCATTER_BLOCK realisations and, item by item of the tile (nearly always
 * one), ranks the item's realisations by bin in shared memory. SCATTER false:
 * counts into one histogram whose bins run item by item (bin_base). SCATTER
 * true: reserves the tile's range of every bin with one global atomic, then
 * writes the realisations' offsets in their item. (One global atomic per
 * realisation took 0.64 + 0.95 ms for 25e6 realisations of 32 suns.) */
template<class R, bool SCATTER>
__global__ void __launch_bounds__(SCATTER_BLOCK) batch_presort
  (const DScene<R>* scenes, const unsigned long long* prefix,
   const unsigned long long* firsts, int nitems, uint64_t seed,
   const uint32_t* bin_base, uint32_t* bins, uint32_t* sorted_off)
{
  __shared__ uint32_t cnt[SORT_MAX_BINS];
  const unsigned long long total = prefix[nitems];
  const unsigned long long tile = (unsigned long long)SCATTER_BLOCK * SCATTER_PER;
  Rng rng;
  rng.k0 = (uint32_t)seed;
  rng.k1 = (uint32_t)(seed >> 32);
  int item = 0;
  for(unsigned long long t0 = blockIdx.x * tile; t0 < total; t0 += gridDim.x * tile) {
    const unsigned long long t1 = t0 + tile < total ? t0 + tile : total;
    for(unsigned long long j0 = t0; j0 < t1;) {
      item = batch_item_of(prefix, nitems, j0, item);
      const unsigned long long start = prefix[item];
      const unsigned long long j1 = prefix[item + 1] < t1 ? prefix[item + 1] : t1;
      const DScene<R>& S = scenes[item];
      const int shift = sort_shift(S.nsamp), nb = ((S.nsamp - 1) >> shift) + 1;
      uint32_t* item_bins = bins + bin_base[item];
      for(int i = threadIdx.x; i < nb; i += SCATTER_BLOCK) cnt[i] = 0;
      __syncthreads();
      uint32_t k[SCATTER_PER], rank[SCATTER_PER];
#pragma unroll
      for(int e = 0; e < SCATTER_PER; ++e) {
        const unsigned long long j = j0 + e * SCATTER_BLOCK + threadIdx.x;
        k[e] = 0u;
        rank[e] = 0u;
        if(j < j1) {
          const uint64_t id = firsts[item] + (j - start);
          rng.i_lo = (uint32_t)id;
          rng.i_hi = (uint32_t)(id >> 32);
          k[e] = (uint32_t)sample_prim(S, rng.get(0u, RNG_PRIMARY)) >> shift;
          rank[e] = atomicAdd(&cnt[k[e]], 1u);
        }
      }
      __syncthreads();
      for(int i = threadIdx.x; i < nb; i += SCATTER_BLOCK)
        if(cnt[i]) {
          const uint32_t at = atomicAdd(&item_bins[i], cnt[i]);
          if(SCATTER) cnt[i] = at;
        }
      __syncthreads();
      if(SCATTER) {
#pragma unroll
        for(int e = 0; e < SCATTER_PER; ++e) {
          const unsigned long long j = j0 + e * SCATTER_BLOCK + threadIdx.x;
          if(j < j1) sorted_off[cnt[k[e]] + rank[e]] = (uint32_t)(j - start);
        }
        __syncthreads();
      }
      j0 = j1;
    }
  }
}

/* Per-device pool of the sort's scratch (kernels_plain.cu) */
cudaMemPool_t sort_pool(int dev);

static size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

/*******************************************************************************
 * Host launchers
 ******************************************************************************/

/* The dynamic shared-memory limit of a kernel is an attribute of one
 * device's context: raise it once per (kernel, device). `Tag` tells the
 * kernels apart (one set of flags per template instance). */
template<class Tag, class K>
static void raise_smem_limit(K kernel, int dev)
{
  static std::atomic<unsigned long long> done_mask{0};
  const unsigned long long bit = dev >= 0 && dev < 64 ? 1ull << dev : 0ull;
  if(bit && (done_mask.load(std::memory_order_acquire) & bit)) return;
  if(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                          160 * 1024) == cudaSuccess && bit)
    done_mask.fetch_or(bit, std::memory_order_acq_rel);
}
template<class R, int MINB, bool TRACK, int FEAT> struct RealisationTag {};
template<class R, int MINB, int FEAT> struct BatchTag {};

/* Shared memory of a block of the realisation kernels: tally tiles, path
 * sums */
static size_t path_smem(int feat, int block)
{
  return (size_t)block * (TILES * sizeof(double2) + ps_count(feat) * sizeof(double));
}

/* Scratch and kernels of the coherent order of one chunk of a launch */
struct SortScratch {
  unsigned char* buf = nullptr; /* null: id order */
  uint32_t* sorted_off = nullptr;
  uint32_t* hist = nullptr;
  uint32_t* off = nullptr;
  int shift = 0, nbins = 0;
};
template<class R>
static SortScratch sort_alloc(const DScene<R>& S, uint64_t chunk, int dev, cudaStream_t st)
{
  SortScratch q;
  q.shift = sort_shift(S.nsamp);
  q.nbins = ((S.nsamp - 1) >> q.shift) + 1;
  const size_t o_hist = align256(chunk * sizeof(uint32_t));
  const size_t o_off = o_hist + align256((size_t)q.nbins * sizeof(uint32_t));
  const size_t bytes = o_off + align256((size_t)q.nbins * sizeof(uint32_t));
  cudaMemPool_t pool = sort_pool(dev);
  if(!pool || cudaMallocFromPoolAsync((void**)&q.buf, bytes, pool, st) != cudaSuccess) {
    /* no room for the scratch: id order */
    cudaGetLastError();
    q.buf = nullptr;
    return q;
  }
  q.sorted_off = (uint32_t*)q.buf;
  q.hist = (uint32_t*)(q.buf + o_hist);
  q.off = (uint32_t*)(q.buf + o_off);
  return q;
}
template<class R>
static void sort_launch(const SortScratch& q, const DScene<R>& S, uint64_t seed, uint64_t first,
                        uint32_t n, int nsm, cudaStream_t st)
{
  cudaMemsetAsync(q.hist, 0, (size_t)q.nbins * sizeof(uint32_t), st);
  presort_count<R><<<(unsigned)nsm * 8u, 256, 0, st>>>(S, seed, first, n, q.shift, q.nbins,
                                                       q.hist);
  presort_scan<<<1, SCAN_BLOCK, 0, st>>>(q.hist, q.off, q.nbins, nullptr, nullptr);
  presort_scatter<R><<<(unsigned)nsm * 2u, SCATTER_BLOCK, 0, st>>>
    (S, seed, first, n, q.shift, q.nbins, q.off, q.sorted_off);
}
/* Realisations of a warp segment for n realisations on `warps` warps */
static uint32_t segment_length(uint64_t n, uint64_t warps)
{
  const uint64_t share = n / (warps * SORT_SHARE) / 32;
  return (uint32_t)std::min<uint64_t>(std::max<uint64_t>(share, 1) * 32, SORT_SEG);
}
/* Segment s of a launch is segment (s x mul) mod nseg of the sorted order,
 * mul coprime with nseg and near nseg / golden ratio */
static uint32_t segment_stride(uint32_t nseg)
{
  if(nseg <= 1) return 1;
  uint32_t mul = (uint32_t)(0.6180339887 * nseg) | 1u;
  while(std::gcd(mul, nseg) != 1u) mul += 2;
  return mul;
}
/* Whether a launch of `count` realisations runs in the coherent order */
template<class R>
static bool sort_pays(const DScene<R>& S, uint64_t count, int features, cudaStream_t st)
{
  const uint64_t least = features & (FEAT_QUADRIC | FEAT_DIELECTRIC) ? SORT_MIN_QUADRIC
                                                                     : SORT_MIN;
  if(count < least || (S.nsampled <= 1 && S.nsamp < SORT_SINGLE)) return false;
  if(count >= SORT_MIN_CAPTURED) return true;
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  return cudaStreamIsCapturing(st, &capture) == cudaSuccess
      && capture == cudaStreamCaptureStatusNone;
}

template<class R, int MINB, bool TRACK, int FEAT>
static int launch_variant
  (const DScene<R>& S, const DTallies& T, uint64_t seed, uint64_t first,
   uint64_t count, const LaunchConfig& cfg, void* stream, const DTrack& tr)
{
  int dev = 0;
  cudaGetDevice(&dev);
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int block = cfg.block_size > 0 ? cfg.block_size : MAX_BLOCK;
  if(block > MAX_BLOCK || block % 32) return (int)cudaErrorInvalidValue;
  const size_t smem = path_smem(FEAT, block);
  raise_smem_limit<RealisationTag<R, MINB, TRACK, FEAT>>(realisation_kernel<R, MINB, TRACK, FEAT>, dev);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor
    (&per_sm, realisation_kernel<R, MINB, TRACK, FEAT>, block, smem);
  if(per_sm < 1) per_sm = 1;
  uint64_t blocks = cfg.grid_blocks > 0
    ? (uint64_t)cfg.grid_blocks
    : (uint64_t)nsm * (uint64_t)per_sm * (uint64_t)(cfg.waves > 0 ? cfg.waves : 1);
  const uint64_t needed = (count + block - 1) / block;
  if(blocks > needed) blocks = needed;
  if(blocks < 1) blocks = 1;
  const cudaStream_t st = (cudaStream_t)stream;
  DControl ctl;
  ctl.max_failed = cfg.max_failed;
  ctl.stop = cfg.max_failed != ~0ull ? T.counters + 4 : nullptr;
  ctl.abort = cfg.abortable ? T.counters + 5 : nullptr;
  ctl.regen = regen_lanes(cfg.features);
  const uint64_t chunk = count < SORT_CHUNK ? count : SORT_CHUNK;
  SortScratch sort;
  if(!TRACK && cfg.coherent && sort_pays(S, count, cfg.features, st))
    sort = sort_alloc(S, chunk, dev, st);
  if(!sort.buf) {
    /* Work counter of this launch: counters[3] */
    cudaMemsetAsync(T.counters + 3, 0, sizeof(unsigned long long), st);
    realisation_kernel<R, MINB, TRACK, FEAT><<<(unsigned)blocks, block, smem, st>>>
      (S, T, seed, first, count, cfg.max_segments, T.counters + 3, tr, nullptr,
       1u, 1u, ctl);
    launch_finish<R>(nullptr, nullptr, T, 1, S.nrcv, S.nsampled, st);
    return (int)cudaGetLastError();
  }
  for(uint64_t c0 = 0; c0 < count; c0 += chunk) {
    const uint32_t n = (uint32_t)(count - c0 < chunk ? count - c0 : chunk);
    sort_launch(sort, S, seed, first + c0, n, nsm, st);
    uint64_t nb = (n + block - 1) / block;
    if(nb > blocks) nb = blocks;
    const uint32_t seg_len = segment_length(n, nb * (uint64_t)(block / 32));
    const uint32_t nseg = (uint32_t)((n + seg_len - 1) / seg_len);
    cudaMemsetAsync(T.counters + 3, 0, sizeof(unsigned long long), st);
    realisation_kernel<R, MINB, TRACK, FEAT><<<(unsigned)nb, block, smem, st>>>
      (S, T, seed, first + c0, n, cfg.max_segments, T.counters + 3, tr,
       sort.sorted_off, seg_len, segment_stride(nseg), ctl);
  }
  launch_finish<R>(nullptr, nullptr, T, 1, S.nrcv, S.nsampled, st);
  cudaFreeAsync(sort.buf, st);
  return (int)cudaGetLastError();
}

/* Feature variants: meshes with mirror and matte materials only, quadrics and
 * dielectrics, or everything (vertex attributes). The all-FP64 build has them
 * too: field, 2e6 paths, 4.25 ms a solve with the last one only, 3.87 with
 * the first. FP32 meshes whose tree has pairs get a variant of their own, as its
 * code costs trees without 3 %: field, 1e8 paths, leaves of one 64.2 -> 62.1 ms,
 * of two 60.6 -> 58.8. */
template<class R, int MINB, int NC>
static int launch_features
  (const DScene<R>& S, const DTallies& T, uint64_t seed, uint64_t first,
   uint64_t count, const LaunchConfig& cfg, void* stream)
{
  const DTrack none = {};
  if constexpr(sizeof(R) == sizeof(float))
    if(cfg.features == FEAT_PAIRS)
      return launch_variant<R, MINB, false, FEAT_PAIRS | NC>(S, T, seed, first, count, cfg,
                                                             stream, none);
  if(cfg.features == 0)
    return launch_variant<R, MINB, false, NC>(S, T, seed, first, count, cfg, stream, none);
  if(!(cfg.features & FEAT_ATTRIBUTES))
    return launch_variant<R, MINB, false, FEAT_QUADRIC | FEAT_DIELECTRIC | NC>
      (S, T, seed, first, count, cfg, stream, none);
  return launch_variant<R, MINB, false, FEAT_ALL | NC>(S, T, seed, first, count, cfg, stream,
                                                       none);
}

/* Register budget variants: at least MINB blocks of 256 threads per SM; NC
 * is FEAT_NOCOUNT for the variants without work counters (path tracking
 * always counts) */
template<class R, int NC = 0>
static int launch_impl
  (const DScene<R>& S, const DTallies& T, uint64_t seed, uint64_t first,
   uint64_t count, const LaunchConfig& cfg, void* stream, const DTrack* track)
{
  if(track)
    return launch_variant<R, 2, true, FEAT_ALL>(S, T, seed, first, count, cfg, stream, *track);
  switch(cfg.min_blocks) {
    case 1: return launch_features<R, 1, NC>(S, T, seed, first, count, cfg, stream);
    case 3: return launch_features<R, 3, NC>(S, T, seed, first, count, cfg, stream);
    default: return launch_features<R, 2, NC>(S, T, seed, first, count, cfg, stream);
  }
}

template<class R, int MINB, int FEAT>
static int launch_batch_variant(const BatchLaunch<R>& b, const LaunchConfig& cfg,
                                void* stream)
{
  int dev = 0;
  cudaGetDevice(&dev);
  int nsm = 0;
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  const int block = cfg.block_size > 0 ? cfg.block_size : MAX_BLOCK;
  if(block > MAX_BLOCK || block % 32) return (int)cudaErrorInvalidValue;
  const size_t smem = path_smem(FEAT, block) + (size_t)(block / 32) * 2 * sizeof(DScene<R>);
  raise_smem_limit<BatchTag<R, MINB, FEAT>>(batch_kernel<R, MINB, FEAT>, dev);
  int per_sm = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor
    (&per_sm, batch_kernel<R, MINB, FEAT>, block, smem);
  if(per_sm < 1) per_sm = 1;
  const uint64_t blocks = cfg.grid_blocks > 0
    ? (uint64_t)cfg.grid_blocks
    : (uint64_t)nsm * (uint64_t)per_sm * (uint64_t)(cfg.waves > 0 ? cfg.waves : 1);
  const cudaStream_t st = (cudaStream_t)stream;
  const BatchOrder& o = b.order;
  if(o.sorted_off) {
    cudaMemsetAsync(o.hist, 0, (size_t)o.nbins * sizeof(uint32_t), st);
    batch_presort<R, false><<<(unsigned)nsm * 2u, SCATTER_BLOCK, 0, st>>>
      (b.scenes, b.prefix, b.firsts, b.nitems, b.seed, o.bin_base, o.hist, nullptr);
    presort_scan<<<(unsigned)b.nitems, SCAN_BLOCK, 0, st>>>
      (o.hist, o.bin_off, (int)o.nbins, o.bin_base, b.prefix);
    batch_presort<R, true><<<(unsigned)nsm * 2u, SCATTER_BLOCK, 0, st>>>
      (b.scenes, b.prefix, b.firsts, b.nitems, b.seed, o.bin_base, o.bin_off, o.sorted_off);
  }
  cudaMemsetAsync(b.next_items, 0, (size_t)b.nitems * sizeof(unsigned long long), st);
  batch_kernel<R, MINB, FEAT><<<(unsigned)blocks, block, smem, st>>>
    (b.scenes, b.tallies, b.prefix, b.firsts, b.nitems, b.seed, cfg.max_segments,
     b.next_items, b.stats, regen_lanes(cfg.features), o.sorted_off, o.seg_mul);
  launch_finish<R>(b.scenes, b.tallies, {}, b.nitems, cfg.max_nrcv, cfg.max_nsampled, st);
  return (int)cudaGetLastError();
}

/* NC is FEAT_NOCOUNT for the variants without work counters */
template<class R, int NC = 0>
static int launch_batch_impl(const BatchLaunch<R>& b, const LaunchConfig& cfg,
                             void* stream)
{
  /* FP32 batches of meshes with mirror and matte materials only get the
   * smaller variant */
  if constexpr(sizeof(R) == sizeof(float))
    if((cfg.features & FEAT_ALL) == 0) {
      switch(cfg.min_blocks) {
        case 1: return launch_batch_variant<R, 1, FEAT_PAIRS | NC>(b, cfg, stream);
        case 3: return launch_batch_variant<R, 3, FEAT_PAIRS | NC>(b, cfg, stream);
        default: return launch_batch_variant<R, 2, FEAT_PAIRS | NC>(b, cfg, stream);
      }
    }
  switch(cfg.min_blocks) {
    case 1: return launch_batch_variant<R, 1, FEAT_ALL | NC>(b, cfg, stream);
    case 3: return launch_batch_variant<R, 3, FEAT_ALL | NC>(b, cfg, stream);
    default: return launch_batch_variant<R, 2, FEAT_ALL | NC>(b, cfg, stream);
  }
}

} /* namespace ssolb */

#endif /* SSOL_B200_KERNELS_DEVICE_CUH */
