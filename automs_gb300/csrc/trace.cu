// trace.cu -- the two-stage ray-traced channel simulator on GB300.
//
// Reference behaviour (file:line of the reference):
//   stage 1, forward discovery    optixPathTracer.cu:142-190, :285-331
//   stage 2, backward verify      optixPathTracer.cu:191-273, :332-417
//   sphere capture                optixPathTracer.cu:419-445
//   beam patterns                 optixPathTracer.cu:107-136
//   dedup + flood fill            optixPathTracer.cpp:127-354
//
// GB300 design:
//   * software BVH traversal over LBVHs (lbvh.cu) with a per-thread stack;
//     node culling is conservative, primitive tests are exact, and the
//     closest hit is chosen by (t, instance, primitive), so the hit does not
//     depend on traversal order.
//   * stage 1 inserts each forward record straight into a hashed path table
//     and a (cell x path) bitmap: no record buffer, no host round trip.
//   * stage 2 works on bitmaps: a round is "list new tasks -> trace the
//     25 x S backward rays of every task -> expand successes to the 4
//     neighbour cells"; the host only reads the new-task count.
//   * channel contributions are summed exactly in 64-bit fixed point, so H is
//     bit-reproducible whatever the launch order.
//   * this file is compiled with -fmad=false: the float arithmetic of every
//     decision matches the CPU oracle bit for bit.
#include <algorithm>

#include "ams_common.cuh"
#include "trace.h"

namespace {

// Largest floats not above cos((2k-1) pi / 72), k = 1..18: the 5-degree bin
// edges of theta_id = int((acos|c| / (pi/2) * 36 + 1) / 2)
// (optixPathTracer.cu:304-306).
__constant__ unsigned c_theta_thr_bits[18] = {
    0x3f7fc19fu, 0x3f7dcf54u, 0x3f79ee88u, 0x3f7426cbu, 0x3f6c835eu, 0x3f631324u,
    0x3f57e880u, 0x3f4b1934u, 0x3f3cbe35u, 0x3f2cf37au, 0x3f1bd7c9u, 0x3f098c77u,
    0x3eec6a50u, 0x3ec3ef15u, 0x3e99f61cu, 0x3e5da258u, 0x3e05a8a8u, 0x3d32aa3eu};

// The bin of |c| is the number of edges not below it.  An estimate of the
// angle (Abramowitz and Stegun 4.4.45, error below 7e-5 rad) gives the bin to
// within one, and the exact edges on both sides of it decide.
__device__ __forceinline__ int theta_id(float c) {
  const float a = fabsf(c);
  const float x = fminf(a, 1.0f);
  const float p = __fmaf_rn(x, __fmaf_rn(x, __fmaf_rn(x, -0.0187293f, 0.0742610f), -0.2121144f),
                            1.5707288f);
  const float th = __fsqrt_rn(1.0f - x) * p;  // acos
  // edges lie at (2k - 1) pi / 72, bins are 5 degrees wide
  int id = (int)__fmaf_rn(th, 36.0f / AMS_PIF, 0.5f);
  id = max(0, min(18, id));
  if (id > 0 && !(a <= __uint_as_float(c_theta_thr_bits[id - 1]))) id--;
  else if (id < 18 && a <= __uint_as_float(c_theta_thr_bits[id])) id++;
  return id;
}

// ------------------------------------------------------------------- RNG
// TEA-4 (Zafar, Olano, Curtis 2010) and the Numerical Recipes LCG
// (optix/SDK/cuda/random.h:31-61)
__device__ __forceinline__ uint32_t tea4(uint32_t v0, uint32_t v1) {
  uint32_t s0 = 0;
#pragma unroll
  for (int n = 0; n < 4; n++) {
    s0 += 0x9e3779b9u;
    v0 += ((v1 << 4) + 0xa341316cu) ^ (v1 + s0) ^ ((v1 >> 5) + 0xc8013ea4u);
    v1 += ((v0 << 4) + 0xad90777du) ^ (v0 + s0) ^ ((v0 >> 5) + 0x7e95761eu);
  }
  return v0;
}
__device__ __forceinline__ float rnd(uint32_t &seed) {
  seed = 1664525u * seed + 1013904223u;
  return (float)(seed & 0x00FFFFFFu) / (float)0x01000000;
}

// sin/cos of a float angle in [0, 7): Cody-Waite reduction by pi/2 with a
// two-part constant and Taylor series to degree 17/18 in double, rounded
// once to float (correctly rounded except within ~1e-16 of a midpoint).
__device__ __forceinline__ void sincos_exact(float a, float &s_out, float &c_out) {
  double x = (double)a;
  double kd = floor(x * 0.6366197723675814 + 0.5);
  double r = (x - kd * 1.5707963267341256) - kd * 6.077100506506192e-11;
  double r2 = r * r;
  double s = 2.8114572543455206e-15;
  s = s * r2 - 7.647163731819816e-13;
  s = s * r2 + 1.6059043836821613e-10;
  s = s * r2 - 2.505210838544172e-08;
  s = s * r2 + 2.7557319223985893e-06;
  s = s * r2 - 0.0001984126984126984;
  s = s * r2 + 0.008333333333333333;
  s = s * r2 - 0.16666666666666666;
  s = s * r2 + 1.0;
  s = s * r;
  double c = 1.5619206968586225e-16;
  c = c * r2 - 4.779477332387385e-14;
  c = c * r2 + 1.1470745597729725e-11;
  c = c * r2 - 2.08767569878681e-09;
  c = c * r2 + 2.755731922398589e-07;
  c = c * r2 - 2.48015873015873e-05;
  c = c * r2 + 0.001388888888888889;
  c = c * r2 - 0.041666666666666664;
  c = c * r2 + 0.5;
  c = 1.0 - c * r2;
  int q = ((int)kd) & 3;
  double so = q == 0 ? s : (q == 1 ? c : (q == 2 ? -s : -c));
  double co = q == 0 ? c : (q == 1 ? -s : (q == 2 ? -c : s));
  s_out = (float)so;
  c_out = (float)co;
}

// rand_dir, optixPathTracer.cu:56-68
__device__ __forceinline__ af3 rand_dir(uint32_t &seed, uint32_t ix, uint32_t iy, int lx, int ly) {
  float rnd1 = (rnd(seed) + (float)ix) / (float)lx;
  float rnd2 = (rnd(seed) + (float)iy) / (float)ly;
  float theta = (2.0f * AMS_PIF) * rnd1;
  float r = sqrtf(rnd2);
  float sn, cs;
  sincos_exact(theta, sn, cs);
  float u = r * cs, v = r * sn;
  float q = sqrtf(1.0f - r * r);
  return mk3((2.0f * u) * q, (2.0f * v) * q, 1.0f - (2.0f * r) * r);
}

// get_beampattern_factor, optixPathTracer.cu:107-136; branches on the float
// cosine against cos(120 deg) and cos(75 deg), taper value in float.
__device__ __forceinline__ float beampattern(af3 d1, af3 d2, int type) {
  if (type == 0) return 1.0f;
  float c = dot3(d1, d2) / (len3(d1) * len3(d2));
  switch (type) {
    case 1: return c < 0.0f ? 0.0f : c * 2.4495f;
    case 2: {
      if ((double)c < -0.5) return 0.1f;
      if ((double)c < 0.25881904510252074) {
        float th = acosf(c);
        float e = (2.0943951f - th) * 0.31830987f * 4.0f * 0.41299623f - 1.0f;
        return exp10f(e) * 2.4495f;
      }
      return (float)((double)c * 2.4495);
    }
    case 3: return c < 0.0f ? 0.0f : 1.4142f;
    default: return 0.0f;
  }
}

// ------------------------------------------------------------ primitives
struct RayT {
  af3 o, d;
  af3 inv;              // 1 / d clamped to +-1e30 (exact wherever it is smaller)
  float oix, oiy, oiz;  // o * inv for the node test
  int kx, ky, kz;
  float Sx, Sy, Sz;
};

// what the triangle test needs: the dominant axis and the shear
__device__ __forceinline__ void ray_setup_tri(RayT &r, af3 o, af3 d) {
  r.o = o;
  r.d = d;
  float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
  int kz = (ax > ay) ? ((ax > az) ? 0 : 2) : ((ay > az) ? 1 : 2);
  int kx = kz + 1; if (kx == 3) kx = 0;
  int ky = kx + 1; if (ky == 3) ky = 0;
  if (comp3(d, kz) < 0.0f) { int t = kx; kx = ky; ky = t; }
  r.kx = kx; r.ky = ky; r.kz = kz;
  float dz = comp3(d, kz);
  r.Sx = comp3(d, kx) / dz;
  r.Sy = comp3(d, ky) / dz;
  r.Sz = 1.0f / dz;
}
// what the box tests need (r.o and r.d are set)
__device__ __forceinline__ void ray_setup_box(RayT &r) {
  // The fused node test computes lo * inv - o * inv.  For an axis-parallel
  // ray (a zero direction component) an infinite inverse would give
  // inf - inf = NaN, or -inf for a box that reaches below 0, and cull nodes
  // the ray is inside of.  The clamp keeps every term finite; node boxes are
  // widened far beyond its rounding error.  prim_slab recovers the exact
  // inverse where the clamp applies.
  const float big = 1e30f;
  r.inv = mk3(fminf(fmaxf(1.0f / r.d.x, -big), big), fminf(fmaxf(1.0f / r.d.y, -big), big),
              fminf(fmaxf(1.0f / r.d.z, -big), big));
  r.oix = r.o.x * r.inv.x;
  r.oiy = r.o.y * r.inv.y;
  r.oiz = r.o.z * r.inv.z;
}
__device__ __forceinline__ void ray_setup(RayT &r, af3 o, af3 d) {
  ray_setup_tri(r, o, d);
  ray_setup_box(r);
}

// Watertight ray/triangle test (Woop, Benthin, Wald, JCGT 2(1) 2013).
__device__ __forceinline__ float tri_hit(const RayT &r, af3 v0, af3 v1, af3 v2) {
  af3 A = sub3(v0, r.o), B = sub3(v1, r.o), C = sub3(v2, r.o);
  float Az_ = comp3(A, r.kz), Bz_ = comp3(B, r.kz), Cz_ = comp3(C, r.kz);
  float Ax = comp3(A, r.kx) - r.Sx * Az_;
  float Ay = comp3(A, r.ky) - r.Sy * Az_;
  float Bx = comp3(B, r.kx) - r.Sx * Bz_;
  float By = comp3(B, r.ky) - r.Sy * Bz_;
  float Cx = comp3(C, r.kx) - r.Sx * Cz_;
  float Cy = comp3(C, r.ky) - r.Sy * Cz_;
  float U = Cx * By - Cy * Bx;
  float V = Ax * Cy - Ay * Cx;
  float W = Bx * Ay - By * Ax;
  if (U == 0.0f || V == 0.0f || W == 0.0f) {
    U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
    V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
    W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
  }
  if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return -1.0f;
  float det = U + V + W;
  if (det == 0.0f) return -1.0f;
  float Az = r.Sz * Az_, Bz = r.Sz * Bz_, Cz = r.Sz * Cz_;
  float T = U * Az + V * Bz + W * Cz;
  return T / det;
}

// slab gate in front of the sphere program (AABB given by the caller)
// exact 1 / d from the clamped inverse (recomputed only where clamped)
__device__ __forceinline__ float exact_inv(float clamped, float d) {
  return fabsf(clamped) < 1e30f ? clamped : 1.0f / d;
}

__device__ __forceinline__ bool prim_slab(const RayT &r, float4 lo, float4 hi) {
  const float ix = exact_inv(r.inv.x, r.d.x), iy = exact_inv(r.inv.y, r.d.y),
              iz = exact_inv(r.inv.z, r.d.z);
  float tx0 = (lo.x - r.o.x) * ix, tx1 = (hi.x - r.o.x) * ix;
  float ty0 = (lo.y - r.o.y) * iy, ty1 = (hi.y - r.o.y) * iy;
  float tz0 = (lo.z - r.o.z) * iz, tz1 = (hi.z - r.o.z) * iz;
  float tn = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fminf(tz0, tz1));
  float tf = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fmaxf(tz0, tz1));
  return tn <= tf && tf >= AMS_TMIN && tn <= AMS_TMAX;
}

// square of the distance at which a ray meets a sphere
__device__ __forceinline__ float sphere_acc(float radius) { return fmaxf(5e-5f, radius * radius); }
// __intersection__sphere, optixPathTracer.cu:419-445; t = closest approach
// D = d * (1 / |d|) is passed in: the same for every sphere of one query
__device__ __forceinline__ float sphere_hit(const RayT &r, af3 D, af3 center, float radius) {
  af3 O = sub3(center, r.o);
  float b = dot3(O, D);
  float c = dot3(O, O);
  if ((c - b * b < sphere_acc(radius)) && b > 0.0f && sqrtf(c) > radius) {
    if (b > AMS_TMIN && b < AMS_TMAX) return b;
  }
  return -1.0f;
}

struct Hit { float t; int inst; int prim; };

__device__ __forceinline__ bool better(float t, int inst, int prim, const Hit &h) {
  if (t < h.t) return true;
  if (t > h.t) return false;
  if (inst != h.inst) return inst < h.inst;
  return prim < h.prim;
}

// conservative child test: widened boxes, loosened far bound
__device__ __forceinline__ bool child_test(const RayT &r, float lx, float ly, float lz, float hx,
                                           float hy, float hz, float best, float &tn_out) {
  float tx0 = __fmaf_rn(lx, r.inv.x, -r.oix), tx1 = __fmaf_rn(hx, r.inv.x, -r.oix);
  float ty0 = __fmaf_rn(ly, r.inv.y, -r.oiy), ty1 = __fmaf_rn(hy, r.inv.y, -r.oiy);
  float tz0 = __fmaf_rn(lz, r.inv.z, -r.oiz), tz1 = __fmaf_rn(hz, r.inv.z, -r.oiz);
  float tn = fmaxf(fmaxf(fminf(tx0, tx1), fminf(ty0, ty1)), fminf(tz0, tz1));
  float tf = fminf(fminf(fmaxf(tx0, tx1), fmaxf(ty0, ty1)), fmaxf(tz0, tz1));
  tn_out = tn;
  // the o*inv form loses a little accuracy; the slack below covers it
  return tn <= __fmaf_rn(tf, 1.0001f, 1e-5f) && tf >= -1e-5f &&
         tn <= __fmaf_rn(best, 1.0001f, 1e-4f);
}

__device__ __forceinline__ af3 unit_dir(const RayT &r) { return scl3(r.d, 1.0f / len3(r.d)); }

// INST 2 (the many Rx spheres) uses the unit direction computed once per
// query; INST 1 (Tx spheres, rarely past the slab gate) computes it here
template <int INST>
__device__ __forceinline__ void test_prim(const float4 *prims, int j, const RayT &r, Hit &best,
                                          float radius, const af3 &Dq) {
  const float4 a = __ldg(prims + 3 * j);
  const float4 b = __ldg(prims + 3 * j + 1);
  const float4 c = __ldg(prims + 3 * j + 2);
  int orig = __float_as_int(a.w);
  if (INST == 0) {
    float t = tri_hit(r, mk3(a.x, a.y, a.z), mk3(b.x, b.y, b.z), mk3(c.x, c.y, c.z));
    if (t > AMS_TMIN && t < AMS_TMAX && better(t, 0, orig, best)) {
      best.t = t; best.inst = 0; best.prim = orig;
    }
  } else {
    if (!prim_slab(r, b, c)) return;
    float t = sphere_hit(r, INST == 2 ? Dq : unit_dir(r), mk3(a.x, a.y, a.z), radius);
    if (t >= 0.0f && better(t, INST, orig, best)) {
      best.t = t; best.inst = INST; best.prim = orig;
    }
  }
}

#define AMS_STACK 64
#define AMS_SEG_CAP 65536  // closest-hit queries per ray before giving up

template <int INST>
__device__ void traverse(const BvhNode *nodes, const float4 *prims, int n, const RayT &r,
                         Hit &best, float radius, unsigned *err) {
  if (n <= 0) return;
  af3 Dq = mk3(0.f, 0.f, 0.f);
  if (INST == 2) Dq = unit_dir(r);
  if (n == 1) { test_prim<INST>(prims, 0, r, best, radius, Dq); return; }
  int st_node[AMS_STACK];
  float st_t[AMS_STACK];
  int sp = 0;
  int node = 0;
  while (true) {
    if ((unsigned)node >= (unsigned)(n - 1)) { atomicOr(err, AMS_DERR_BVH); return; }
    const float4 *np = reinterpret_cast<const float4 *>(nodes + node);
    const float4 a = __ldg(np), b = __ldg(np + 1), c = __ldg(np + 2);
    const int4 d = __ldg(reinterpret_cast<const int4 *>(np + 3));
    float tn0, tn1;
    bool h0 = child_test(r, a.x, a.y, a.z, a.w, b.x, b.y, best.t, tn0);
    bool h1 = child_test(r, b.z, b.w, c.x, c.y, c.z, c.w, best.t, tn1);
    if (h0 && d.x < 0) {
      if (~d.x >= n) { atomicOr(err, AMS_DERR_BVH); return; }
      test_prim<INST>(prims, ~d.x, r, best, radius, Dq);
      h0 = false;
    }
    if (h1 && d.y < 0) {
      if (~d.y >= n) { atomicOr(err, AMS_DERR_BVH); return; }
      test_prim<INST>(prims, ~d.y, r, best, radius, Dq);
      h1 = false;
    }
    if (h0 && h1) {
      int nearn = d.x, farn = d.y;
      float tfar = tn1;
      if (tn1 < tn0) { nearn = d.y; farn = d.x; tfar = tn0; }
      if (sp < AMS_STACK) {
        st_node[sp] = farn; st_t[sp] = tfar; sp++;
      } else {
        atomicOr(err, AMS_DERR_STACK);
      }
      node = nearn;
    } else if (h0) {
      node = d.x;
    } else if (h1) {
      node = d.y;
    } else {
      bool found = false;
      while (sp > 0) {
        sp--;
        if (st_t[sp] <= __fmaf_rn(best.t, 1.0001f, 1e-4f)) { node = st_node[sp]; found = true; break; }
      }
      if (!found) break;
    }
  }
}

// ------------------------------------------------------------------ beams
// Stage 2 traces the rays of a warp together: from one Rx (or two
// neighbours) to the images of neighbouring Tx elements, so they differ by
// millimetres to centimetres.  A beam bounds them: at parameter t every
// active ray lies in the box [omin + t dmin, omax + t dmax].  The 32 lanes
// test the 32 children of one wide node against the beam at once, and each
// triangle that survives is tested exactly by every lane's own ray, nearest
// box first.  The closest hit is the lexicographic minimum over (t, instance,
// primitive) of exact tests, so it is the one that a traversal ray by ray
// finds; only the culling is shared.  Ray by ray, a query made 14 (2,172
// triangles) to 25 dependent visits of binary nodes; a beam makes 2.6 to 6.5
// visits of wide nodes and 4 to 5 triangle tests for 27 to 32 rays.  Stage-2
// kernels: 3.1 -> 2.2 ms on coverage-128, 42 -> 25 ms on a 62k-triangle room with
// 256 x 256 Rx, 90 -> 43 ms with 1,024 metasurface elements as Tx.
// Bound by instruction issue (70% of the slots) in large rounds, by a warp's
// latency in small ones.
constexpr unsigned kFullWarp = 0xffffffffu;

// n / d by the multiplier of make_fast_div (Granlund and Montgomery 1994)
__device__ __forceinline__ unsigned fdiv(unsigned n, const FastDiv &f) {
  if (f.mul == 0u) return n;  // d = 1
  const unsigned q = __umulhi(n, f.mul);
  return (((n - q) >> 1) + q) >> f.shift;
}
__device__ __forceinline__ float warp_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float warp_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}

struct BeamAxis { float o1, i1, o2, i2; };  // bounds on t from the near and the far box plane
struct Beam {
  BeamAxis x, y, z;
  // per axis k: bit k, directions negative (the hi plane is the near one);
  // bit 8 + k, directions of both signs (both planes bound t from below)
  unsigned flags;
  float spread;  // largest extent of the directions along an axis
  float reach;   // largest extent of the origins along an axis
};

// rcp.approx keeps the error (1 ulp) far inside the slack of the box test;
// the clamp as in ray_setup_box
__device__ __forceinline__ float beam_inv(float d) {
  return fminf(fmaxf(__fdividef(1.0f, d), -1e30f), 1e30f);
}
__device__ __forceinline__ BeamAxis beam_axis(float o, float d, bool on, int axis, Beam &b) {
  const float inf = 3.0e38f;
  const float omin = warp_min(on ? o : inf), omax = warp_max(on ? o : -inf);
  const float dmin = warp_min(on ? d : inf), dmax = warp_max(on ? d : -inf);
  // hi plane: omin + t dmin <= hi; lo plane: omax + t dmax >= lo.  A positive
  // dmin bounds t above by the first, a negative one below; and so on.
  const float ihi = dmin == 0.0f ? 1e30f : beam_inv(dmin);
  const float ilo = dmax == 0.0f ? (dmin < 0.0f ? -1e30f : 1e30f) : beam_inv(dmax);
  BeamAxis a;
  const bool neg = dmax <= 0.0f && dmin < 0.0f;
  if (neg) b.flags |= 1u << axis;
  if (dmin < 0.0f && dmax > 0.0f) b.flags |= 256u << axis;
  b.spread = fmaxf(b.spread, dmax - dmin);
  b.reach = fmaxf(b.reach, omax - omin);
  a.o1 = neg ? omin : omax; a.i1 = neg ? ihi : ilo;
  a.o2 = neg ? omax : omin; a.i2 = neg ? ilo : ihi;
  return a;
}
// bounds of the rays of the lanes with `on` (at least one)
__device__ __forceinline__ Beam beam_of(af3 o, af3 d, bool on) {
  Beam b;
  b.flags = 0u;
  b.spread = 0.0f;
  b.reach = 0.0f;
  b.x = beam_axis(o.x, d.x, on, 0, b);
  b.y = beam_axis(o.y, d.y, on, 1, b);
  b.z = beam_axis(o.z, d.z, on, 2, b);
  return b;
}
__device__ __forceinline__ void beam_slab(const BeamAxis &a, bool mixed, float v1, float v2,
                                          float &tn, float &tf) {
  const float t1 = (v1 - a.o1) * a.i1, t2 = (v2 - a.o2) * a.i2;
  tn = fmaxf(tn, mixed ? fmaxf(t1, t2) : t1);
  tf = fminf(tf, mixed ? 3.0e38f : t2);
}
// the slack of child_test, which covers the same rounding
__device__ __forceinline__ bool beam_in(float tn, float tf, float lim) {
  return tn <= __fmaf_rn(tf, 1.0001f, 1e-5f) && tf >= -1e-5f && tn <= lim;
}
__device__ __forceinline__ float beam_limit(float best) { return __fmaf_rn(best, 1.0001f, 1e-4f); }

// A lane's ray for the triangle tests of a beam: origin and shear in the
// order (kx, ky, kz) of its dominant axis (ray_setup_tri), so that a test
// reads the vertices' components in that order and selects nothing.
struct RayB { float ox, oy, oz, Sx, Sy, Sz; int kx, ky, kz; };
__device__ __forceinline__ RayB ray_b(af3 o, af3 d) {
  RayT r;
  ray_setup_tri(r, o, d);
  RayB b;
  b.kx = r.kx; b.ky = r.ky; b.kz = r.kz;
  b.Sx = r.Sx; b.Sy = r.Sy; b.Sz = r.Sz;
  b.ox = comp3(o, r.kx); b.oy = comp3(o, r.ky); b.oz = comp3(o, r.kz);
  return b;
}
// tri_hit on packed triangle p (v0, index, v1, -, v2, -), the same operations
__device__ __forceinline__ float tri_hit_b(const RayB &r, const float *p) {
  const float *px = p + r.kx, *py = p + r.ky, *pz = p + r.kz;
  const float Az_ = __ldg(pz) - r.oz, Bz_ = __ldg(pz + 4) - r.oz, Cz_ = __ldg(pz + 8) - r.oz;
  const float Ax = (__ldg(px) - r.ox) - r.Sx * Az_, Ay = (__ldg(py) - r.oy) - r.Sy * Az_;
  const float Bx = (__ldg(px + 4) - r.ox) - r.Sx * Bz_, By = (__ldg(py + 4) - r.oy) - r.Sy * Bz_;
  const float Cx = (__ldg(px + 8) - r.ox) - r.Sx * Cz_, Cy = (__ldg(py + 8) - r.oy) - r.Sy * Cz_;
  float U = Cx * By - Cy * Bx;
  float V = Ax * Cy - Ay * Cx;
  float W = Bx * Ay - By * Ax;
  if (U == 0.0f || V == 0.0f || W == 0.0f) {
    U = (float)((double)Cx * (double)By - (double)Cy * (double)Bx);
    V = (float)((double)Ax * (double)Cy - (double)Ay * (double)Cx);
    W = (float)((double)Bx * (double)Ay - (double)By * (double)Ax);
  }
  if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return -1.0f;
  const float det = U + V + W;
  if (det == 0.0f) return -1.0f;
  const float Az = r.Sz * Az_, Bz = r.Sz * Bz_, Cz = r.Sz * Cz_;
  const float T = U * Az + V * Bz + W * Cz;
  return T / det;
}

// Wide-node stack of a warp: child reference and near distance (bits).
#define AMS_BEAM_STACK 96
// node visits + triangle tests after which a beam is given up; its lanes then
// traverse the binary nodes one ray each
#define AMS_BEAM_WORK 64
// Directions (rays that met different surfaces) or origins (in m: neighbouring
// Rx of a coarse grid) further apart than this along an axis are taken as several
// beams of closer rays.  Where the rays around the one in the middle are less
// than half of them, no few beams will do, and they traverse the binary nodes
// one each.  38k triangles, Rx 0.5 m apart, all as beams / all one each / this
// rule: 1 Tx 6.2 / 1.5 / 1.4 ms, 4 Tx 4.1 / 1.7 / 1.8, 16 Tx 3.8 / 2.8 / 2.0, 36
// Tx 6.4 / 5.3 / 3.5 ms; Rx 0.1 m apart, 36 Tx 21.8 / 25.1 / 14.  A third, a
// quarter or a sixth instead of half: few Tx up to 1.5 times as long, many Tx the
// same; origins 0.2 or 0.5 m: within 4%, 36 Tx at 0.5 m 3.4 and 4.3 ms.
#define AMS_BEAM_SPREAD 0.1f
#define AMS_BEAM_REACH 0.3f
#define AMS_BEAM_SHARE 2

// Closest scene hit of every alive lane's ray, or with `any` whether there is
// one at all before `best` (such a lane's `alive` becomes false).  Warp
// collective; returns false when the beam was given up or the stack is full,
// with `best` holding only hits that exist.
__device__ __forceinline__ bool beam_scene(const TraceDev &P, const Beam &bm, const RayB &r,
                                           Hit &best, bool &alive, bool any, int2 *stk) {
  const int lane = threadIdx.x & 31;
  int sp = 0, node = 0, work = 0;
  float lim = beam_limit(warp_max(alive ? best.t : 0.0f));
  while (true) {
    if ((unsigned)node >= (unsigned)P.n_tri_wide) {
      if (lane == 0) atomicOr(P.err, AMS_DERR_BVH);
      return true;
    }
    const float *nd = P.tri_wide + (size_t)node * AMS_WIDE_WORDS + lane;
    const int px = (bm.flags & 1u) << 5, py = (bm.flags & 2u) << 4, pz = (bm.flags & 4u) << 3;
    const float x1 = __ldg(nd + px), x2 = __ldg(nd + (px ^ 32)), y1 = __ldg(nd + 64 + py),
                y2 = __ldg(nd + 64 + (py ^ 32)), z1 = __ldg(nd + 128 + pz),
                z2 = __ldg(nd + 128 + (pz ^ 32));
    const int child = __float_as_int(__ldg(nd + 192));
    float tn = -3.0e38f, tf = 3.0e38f;
    beam_slab(bm.x, bm.flags & 256u, x1, x2, tn, tf);
    beam_slab(bm.y, bm.flags & 512u, y1, y2, tn, tf);
    beam_slab(bm.z, bm.flags & 1024u, z1, z2, tn, tf);
    bool hit = beam_in(tn, tf, lim);
    // near distance in the high bits, lane in the low five: the order of
    // non-negative floats is that of their bits
    const unsigned key = (__float_as_uint(fmaxf(tn, 0.0f)) & ~31u) | (unsigned)lane;
    unsigned lk = hit && child < 0 ? key : 0xffffffffu;
    while (true) {
      const unsigned k = __reduce_min_sync(kFullWarp, lk);
      if (k == 0xffffffffu || __uint_as_float(k & ~31u) > lim) break;
      const int j = ~__shfl_sync(kFullWarp, child, (int)(k & 31u));
      if ((unsigned)j >= (unsigned)P.n_tri) {
        if (lane == 0) atomicOr(P.err, AMS_DERR_BVH);
        return true;
      }
      bool closer = false;
      if (alive) {
        const float *pj = reinterpret_cast<const float *>(P.tri_prims + 3 * (size_t)j);
        const float t = tri_hit_b(r, pj);
        if (t > AMS_TMIN && t < AMS_TMAX && t <= best.t) {
          const int orig = __float_as_int(__ldg(pj + 3));
          closer = better(t, 0, orig, best);
          if (closer) { best.t = t; best.inst = 0; best.prim = orig; alive = !any; }
        }
      }
      if (__any_sync(kFullWarp, closer)) {
        if (any && !__any_sync(kFullWarp, alive)) return true;
        lim = beam_limit(warp_max(alive ? best.t : 0.0f));
      }
      if (lk == k) lk = 0xffffffffu;
      work++;
    }
    hit = hit && child >= 0 && tn <= lim;
    const unsigned m = __ballot_sync(kFullWarp, hit);
    if (m) {
      // the nearest child next, the others on the stack, nearer ones on top
      int rank = 0;
      if (m & (m - 1u)) {
#pragma unroll 1
        for (unsigned q = m; q; q &= q - 1u)
          rank += __shfl_sync(kFullWarp, key, __ffs(q) - 1) < key ? 1 : 0;
      }
      const int more = __popc(m) - 1;
      if (sp + more > AMS_BEAM_STACK) return false;
      if (hit && rank > 0) stk[sp + more - rank] = make_int2(child, (int)(key & ~31u));
      node = __shfl_sync(kFullWarp, child, __ffs(__ballot_sync(kFullWarp, hit && rank == 0)) - 1);
      sp += more;
      __syncwarp();
    } else {
      bool found = false;
      while (sp > 0 && !found) {
        const int2 e = stk[--sp];
        found = __int_as_float(e.y) <= lim;
        node = e.x;
      }
      __syncwarp();
      if (!found) return true;
    }
    if (++work > AMS_BEAM_WORK) return false;
  }
}

// whether a ray (r.inv set) may meet the box of the whole Tx array (tx_info words
// 8-10 and 12-14)
__device__ __forceinline__ bool ray_near_tx(const TraceDev &P, const RayT &r) {
  const float4 lo = __ldg(P.tx_info + 2), hi = __ldg(P.tx_info + 3);
  float tn;
  return child_test(r, lo.x, lo.y, lo.z, hi.x, hi.y, hi.z, AMS_TMAX, tn);
}
// The Tx spheres that a ray can meet besides the one it meets, without asking
// the hierarchy.  A ray through the boxes of two Tx is nearly parallel to the
// line between them, so one steep enough to the plane (or the line) of the
// array meets only one: |D . n| > (eta + 2 rho) / (delta - 2 rho), with eta
// the array's extent along n, rho the boxes' radius and delta the smallest
// distance of two Tx (k_tx_info).
__device__ __forceinline__ bool tx_alone(const TraceDev &P, af3 D) {
  const float4 a = __ldg(P.tx_info), b = __ldg(P.tx_info + 1);
  return fabsf(dot3(D, mk3(a.x, a.y, a.z))) > a.w || fabsf(dot3(D, mk3(b.x, b.y, b.z))) > b.w;
}

// the paths that are rarely taken, out of line: their code would push the
// beam loop out of the instruction cache
__device__ __noinline__ Hit traverse_tx(const TraceDev &P, af3 o, af3 d, Hit h) {
  RayT r;
  ray_setup(r, o, d);
  traverse<1>(P.tx_nodes, P.tx_prims, P.n_src, r, h, P.src_r, P.err);
  return h;
}
__device__ __noinline__ Hit traverse_scene(const TraceDev &P, af3 o, af3 d, Hit h) {
  RayT r;
  ray_setup(r, o, d);
  traverse<0>(P.tri_nodes, P.tri_prims, P.n_tri, r, h, 0.0f, P.err);
  return h;
}

// Backward-ray query of stage 2 for a warp: optixTrace with the visibility
// mask of the scene and the Tx spheres (optixPathTracer.cpp:417-424), from
// (o, d) of the lanes with `on` towards Tx s.  On a path's last segment a
// triangle ends the ray wherever it is (optixPathTracer.cu:336-417), so there
// the Tx spheres come first, Tx s itself before the others; a ray that meets
// none has ended, and the scene is asked only for something in front of the
// Tx hit.  Elsewhere the scene comes first.  Returns the closest hit; on the
// last segment the triangle of an inst = 0 hit is any one in front, and
// inst = 3 may stand for a triangle behind no Tx.
__device__ __forceinline__ Hit closest_s2(const TraceDev &P, af3 o, af3 d, int s, bool last,
                                          bool on, int2 *stk) {
  Hit h;
  h.t = AMS_TMAX; h.inst = 3; h.prim = 0x7fffffff;
  if (last) {
    bool others = false;
    if (on) {
      RayT r;
      r.o = o;
      r.d = d;
      ray_setup_box(r);
      const float *bx = P.src_aabb + 6 * (size_t)s;
      const float4 lo = make_float4(__ldg(bx), __ldg(bx + 1), __ldg(bx + 2), 0.f),
                   hi = make_float4(__ldg(bx + 3), __ldg(bx + 4), __ldg(bx + 5), 0.f);
      if (prim_slab(r, lo, hi)) {
        const af3 D = unit_dir(r);
        const float t = sphere_hit(r, D, ld3(P.src + 3 * (size_t)s), P.src_r);
        if (t >= 0.0f && better(t, 1, s, h)) {
          h.t = t; h.inst = 1; h.prim = s;
          others = P.n_src > 1 && !tx_alone(P, D);
        }
      }
      if (h.inst != 1) others = P.n_src > 1 && ray_near_tx(P, r);
    }
    // from the start, as a ray that meets only others: where boxes are smaller than
    // their spheres the order of the hierarchy decides what comes first, and Tx s
    // would hide others that lie before it
    if (others) {
      h.t = AMS_TMAX; h.inst = 3; h.prim = 0x7fffffff;
      h = traverse_tx(P, o, d, h);
    }
    __syncwarp();
  }
  // the rays that the scene is asked for, as beams of close ones
  const int lane = threadIdx.x & 31;
  const bool ask = on && (!last || h.inst == 1);
  bool alone = ask && P.n_tri_wide == 0;  // traverses the binary nodes by itself
  const RayB r = ray_b(o, d);
  for (unsigned left = P.n_tri_wide == 0 ? 0u : __ballot_sync(kFullWarp, ask); left;) {
    bool in = (left >> lane) & 1u;
    Beam bm = beam_of(o, d, in);
    unsigned now = left;
    if (bm.spread > AMS_BEAM_SPREAD || bm.reach > AMS_BEAM_REACH) {
      // around the ray in the middle of them
      const int lead = __ffs(__ballot_sync(kFullWarp, in && __popc(left & ((1u << lane) - 1u)) ==
                                                                __popc(left) / 2)) - 1;
      const float dx = __shfl_sync(kFullWarp, d.x, lead), dy = __shfl_sync(kFullWarp, d.y, lead),
                  dz = __shfl_sync(kFullWarp, d.z, lead), ox = __shfl_sync(kFullWarp, o.x, lead),
                  oy = __shfl_sync(kFullWarp, o.y, lead), oz = __shfl_sync(kFullWarp, o.z, lead);
      const bool near =
          fmaxf(fmaxf(fabsf(d.x - dx), fabsf(d.y - dy)), fabsf(d.z - dz)) < 0.5f * AMS_BEAM_SPREAD &&
          fmaxf(fmaxf(fabsf(o.x - ox), fabsf(o.y - oy)), fabsf(o.z - oz)) < 0.5f * AMS_BEAM_REACH;
      now = __ballot_sync(kFullWarp, in && (near || lead == lane));
      if (__popc(now) * AMS_BEAM_SHARE < __popc(left)) {
        alone = alone || in;
        break;
      }
      in = (now >> lane) & 1u;
      bm = beam_of(o, d, in);
    }
    left &= ~now;
    bool alive = in;
    if (!beam_scene(P, bm, r, h, alive, last, stk)) alone = alone || alive;
    __syncwarp();
  }
  if (alone) h = traverse_scene(P, o, d, h);
  // (ray by ray: by the beams' bounds most rays of a loose beam seemed to pass
  // the Tx array, and every one of them asked its hierarchy: 34 -> 25 ms)
  if (!last && on) {
    RayT q;
    q.o = o;
    q.d = d;
    ray_setup_box(q);
    if (ray_near_tx(P, q)) h = traverse_tx(P, o, d, h);
  }
  __syncwarp();
  return h;
}

// ---------------------------------------------------------- image method
struct Mat34 { float m[12]; };

__device__ __forceinline__ af3 image_of(const Mat34 &M, af3 p) {
  const float *m = M.m;
  return mk3(m[0] * p.x + m[1] * p.y + m[2] * p.z + m[3] * 1.0f,
             m[4] * p.x + m[5] * p.y + m[6] * p.z + m[7] * 1.0f,
             m[8] * p.x + m[9] * p.y + m[10] * p.z + m[11] * 1.0f);
}

// updateImageTransform, optixPathTracer.cu:70-76 (sum order of Matrix.h:339-356)
__device__ __forceinline__ void image_update(Mat34 &M, af3 N, af3 A) {
  float n[3] = {N.x, N.y, N.z};
  float a[9];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      float p = (2.0f * n[i]) * n[j];
      a[i * 3 + j] = (i == j ? 1.0f : 0.0f) - p;
    }
  Mat34 r;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 4; j++) {
      float s = a[i * 3] * M.m[j];
      s = s + a[i * 3 + 1] * M.m[4 + j];
      s = s + a[i * 3 + 2] * M.m[8 + j];
      r.m[i * 4 + j] = s;
    }
  float k2 = 2.0f * dot3(A, N);
  r.m[3] = r.m[3] + k2 * N.x;
  r.m[7] = r.m[7] + k2 * N.y;
  r.m[11] = r.m[11] + k2 * N.z;
  M = r;
}

__device__ __forceinline__ int32_t fbits(float f) {
  int32_t b = __float_as_int(f);
  return b == (int32_t)0x80000000 ? 0 : b;  // -0 and +0 are one key
}

// Path-key hash: word-wise FNV-1a (Fowler, Noll, Vo) in 64 bits, finished
// by an avalanche mixer; it places the key in the open-addressed table.
__device__ __forceinline__ uint64_t key_hash64(const int32_t *k) {
  uint64_t h = 0xcbf29ce484222325ull;
#pragma unroll
  for (int i = 0; i < 14; i++) h = (h ^ (uint64_t)(uint32_t)k[i]) * 0x100000001b3ull;
  return mix64(h);
}

// OR a bit into a bitmap word (a reduction: the thread does not wait)
__device__ __forceinline__ void set_bit(unsigned *word, unsigned bit) { atomicOr(word, bit); }

// Key words are stored with the sign bit flipped.  A key never holds
// 0x80000000 (-0.0 is canonicalised to +0, and the hit count and reflect
// mask are small non-negative integers), so a stored word is never 0, and a
// 0 read back from a slot is a word its claiming thread has not written yet.
#define AMS_KEY_FLIP 0x80000000u
__device__ __forceinline__ int32_t key_word(const int32_t *slot_key, int i) {
  return (int32_t)((uint32_t)__ldg(slot_key + i) ^ AMS_KEY_FLIP);
}

// Claim or find the slot of a path key; returns -1 when the table is full.
// The 64-bit hash picks the first probe; a slot belongs to the key whose
// 14 words are stored in it.  One batch of loads reads a slot's hash and
// words: a slot with the same hash whose words are all written (non-zero)
// and equal is the key's slot; one whose words are still being written is
// re-read until they are (a few instructions of the claiming thread; the
// wait is bounded); a slot holding other words is passed over.  So two
// distinct keys never share a slot, and a key never takes two.
__device__ int path_insert(const TraceDev &P, const int32_t *key) {
  const uint64_t h = key_hash64(key) | 1ull;
  uint32_t enc[14];
#pragma unroll
  for (int i = 0; i < 14; i++) enc[i] = (uint32_t)key[i] ^ AMS_KEY_FLIP;
  uint32_t slot = (uint32_t)h & P.tab_mask;
#pragma unroll 1
  for (uint32_t probe = 0; probe <= P.tab_mask; probe++) {
    unsigned long long old = __ldcg(P.tab_h + slot);
    uint32_t *sk = reinterpret_cast<uint32_t *>(P.tab_key) + (size_t)slot * 14;
    if (old == 0ull) old = atomicCAS(P.tab_h + slot, 0ull, (unsigned long long)h);
    if (old == 0ull) {
#pragma unroll
      for (int i = 0; i < 14; i++) __stcg(sk + i, enc[i]);
      unsigned long long occ = atomicAdd(P.ctr + 2, 1ull);
      if (occ >= P.tab_limit) atomicOr(P.err, AMS_DERR_PATH_TABLE);
      return (int)slot;
    }
    if (old == (unsigned long long)h) {
      for (int spin = 0;; spin++) {
        uint32_t w[14];
        bool full = true, same = true;
#pragma unroll
        for (int i = 0; i < 14; i++) w[i] = __ldcg(sk + i);
#pragma unroll
        for (int i = 0; i < 14; i++) {
          full &= w[i] != 0u;
          same &= w[i] == enc[i];
        }
        if (same) return (int)slot;
        if (full) break;  // another key with this hash: probe on
        if (spin > (1 << 22)) { atomicOr(P.err, AMS_DERR_HASH); return -1; }
        __nanosleep(32);
      }
    }
    slot = (slot + 1u) & P.tab_mask;
  }
  atomicOr(P.err, AMS_DERR_PATH_TABLE);
  return -1;
}

// What the hit programs need of scene triangle `prim` (original index,
// optixPathTracer.cu:296-299): computed once per scene by k_tri_attr with
// the operations the programs would repeat at every hit.
struct TriAttr {
  af3 n;        // unit normal
  float n_len;  // its length as computed
  float max_d;  // longest edge
  af3 v0;
};
__device__ __forceinline__ TriAttr scene_tri(const TraceDev &P, int prim) {
  const float4 a = __ldg(P.tri_attr + 2 * (size_t)prim), b = __ldg(P.tri_attr + 2 * (size_t)prim + 1);
  TriAttr r;
  r.n = mk3(a.x, a.y, a.z);
  r.n_len = a.w;
  r.v0 = mk3(b.x, b.y, b.z);
  r.max_d = b.w;
  return r;
}
__global__ void k_tri_attr(const float *tris, int n, float4 *attr) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float *v = tris + (size_t)i * 9;
  const af3 v0 = ld3(v), v1 = ld3(v + 3), v2 = ld3(v + 6);
  const af3 N0 = nrm3(cross3(sub3(v1, v0), sub3(v2, v0)));
  const float max_d = fmaxf(fmaxf(len3(sub3(v0, v1)), len3(sub3(v1, v2))), len3(sub3(v2, v0)));
  // a normal turned towards the ray has the same length: squares lose the sign
  attr[2 * i] = make_float4(N0.x, N0.y, N0.z, len3(N0));
  attr[2 * i + 1] = make_float4(v0.x, v0.y, v0.z, max_d);
}

// ---------------------------------------------------------------- stage 1
// A branch slot whose ray waits while an earlier-indexed one is traced (the
// reference's 32-entry PRD stack, optixPathTracer.cu:152-190).  Its
// remaining levels follow from the index: a reflection spawned at hit count
// hc sets bit hc - 1 as the slot's highest bit and keeps L + 1 - hc levels.
struct Slot {
  af3 o, d;
  Mat34 M;
};

__device__ __forceinline__ int slot_ttl(int L, int j) { return L - (31 - __clz(j)); }

// Image matrix of the lane's current ray: slot 0 (the primary ray) is the
// identity and is never stored; any other slot's matrix sits in one per-lane
// array (48 bytes of local memory that stay in L1; a shared-memory copy
// measured 3% slower, its 6 KB per CTA taken from L1).
struct CurMatrix {
  float *cm;  // the lane's 12 floats
  __device__ __forceinline__ Mat34 get(int cur) const {
    Mat34 M;
#pragma unroll
    for (int k = 0; k < 12; k++)
      M.m[k] = cur == 0 ? ((k == 0 || k == 5 || k == 10) ? 1.0f : 0.0f) : cm[k];
    return M;
  }
  __device__ __forceinline__ void set(const Mat34 &M) const {
#pragma unroll
    for (int k = 0; k < 12; k++) cm[k] = M.m[k];
  }
};



// Stage 1 runs as a persistent loop per warp with dynamic fetching (after
// Aila & Laine, "Understanding the efficiency of ray traversal on GPUs",
// HPG 2009).  A round answers one closest-hit query of every lane: the Rx
// spheres (by their grid, or by their hierarchy where they form none) and
// the scene pruned at the sphere hit, visiting BVH nodes until every lane's
// query has ended; then all lanes handle their hits together and set up their
// next queries (the next segment, the next pending slot, the next sub-launch,
// or a launch index fetched from a global counter).  Lanes that finish a
// short ray take new work instead of idling behind the warp's longest ray, and
// the hit code runs once per round for the whole warp.  (Handling the hits
// of a subset of lanes while the others still traverse measured slower at
// every threshold tried: the hit code is long.)
// Per launch index the queries, hits and records come in the order of the
// sequential trace (slots in increasing index, which is the order
// __ffs(pending) gives because a spawned slot always has a higher index than
// its parent), so the per-thread min_hc dedup and the reserve cap see
// exactly what they see in the reference.
//
// Half of the node visits were spent on the Rx spheres (13 per query in a tree
// of 16,384); the grid needs a row or two.  Bound by the latency of dependent
// instructions and node fetches with 14 of 32 lanes active.  Code that is not
// in the loop any more was worth as much as fewer visits: short loops run
// rolled up (unrolled by the compiler they cost 3.1 instead of 2.6 ms on
// coverage-128).  k_stage1:
// coverage-128 3.84 -> 2.07 ms, 62k triangles and 256 x 256 Rx 14.8 -> 8.1 ms,
// the same scene and a 32 x 32 metasurface as Rx 9.6 -> 4.7 ms.

// warp-aggregated fetch of one launch index per calling lane
__device__ __forceinline__ long long fetch_launch(unsigned long long *ctr) {
  const unsigned m = __activemask();
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  unsigned long long base = 0;
  if (lane == leader) base = atomicAdd(ctr, (unsigned long long)__popc(m));
  base = __shfl_sync(m, base, leader);
  return (long long)(base + (unsigned long long)__popc(m & ((1u << lane) - 1u)));
}

struct S1Query {
  RayT r;
  af3 Dq;  // unit direction for the sphere tests
  Hit best;
};

// ------------------------------------------------------------- Rx grid
// Rx sets are mostly axis-aligned planar grids (gen_pos_from_endpoint,
// go.py:248-300): index i runs along axis ua, j along va, and axis wa is
// constant.  A ray crosses the slab of all Rx boxes over a short stretch, whose
// u and v intervals give the few Rx that it can meet; they are tested one by
// one with the tests that the hierarchy's leaves get.  rx_grid words: 0-2 the
// largest deviation of an Rx from its place in the grid along u, v, w; 3-5 the
// largest extent of a box from its Rx; 6 counts the CTAs of k_rx_grid that are
// done, whose last one writes 7: 1 where the grid can be used (the hierarchy
// of the Rx is not built then); 8 is set where a box is smaller than its sphere.
struct RxGrid {
  int ok, ua, va, wa;
  float u0, su, iu, v0, sv, iv, w0;  // steps and their inverses, 0 where there is one row
  float bu, bv, bw;          // reach of a box, with the deviation and a margin
};
// axes, origin and steps from three corners of the set
__device__ __forceinline__ RxGrid rx_grid_axes(const float *dst, int n0, int n1, float &du,
                                               float &dv) {
  RxGrid g;
  const af3 a = ld3(dst), e = sub3(ld3(dst + 3 * (size_t)(n0 - 1) * n1), a),
            f = sub3(ld3(dst + 3 * (size_t)(n1 - 1)), a);
  auto main_axis = [](af3 v) {
    const float x = fabsf(v.x), y = fabsf(v.y), z = fabsf(v.z);
    return x >= y ? (x >= z ? 0 : 2) : (y >= z ? 1 : 2);
  };
  g.ua = main_axis(e);
  g.va = main_axis(f);
  if (n0 == 1) g.ua = (g.va + 1) % 3;
  if (n1 == 1) g.va = (g.ua + 1) % 3;
  g.wa = 3 - g.ua - g.va;
  g.ok = g.ua != g.va && n0 * n1 > 1;
  if (!g.ok) g.wa = 0;
  du = n0 > 1 ? comp3(e, g.ua) / (float)(n0 - 1) : 0.0f;
  dv = n1 > 1 ? comp3(f, g.va) / (float)(n1 - 1) : 0.0f;
  g.u0 = comp3(a, g.ua);
  g.v0 = comp3(a, g.va);
  g.w0 = comp3(a, g.wa);
  return g;
}
__global__ void __launch_bounds__(256) k_rx_grid(const float *dst, const float *aabb, int n0, int n1,
                                                 float radius, float *out) {
  float du, dv;
  // A sphere's hit lies at the ray's closest approach (sphere_hit).  Only where
  // the box holds all of the sphere is that always inside the box, and the
  // nearest hit the same in whichever order the spheres are looked at; with a
  // smaller box the order of the hierarchy decides.
  const float need = sqrtf(sphere_acc(radius));
  bool small = false;
  const RxGrid g = rx_grid_axes(dst, n0, n1, du, dv);
  float m[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  const int ax[3] = {g.ua, g.va, g.wa};
  for (int d = blockIdx.x * blockDim.x + threadIdx.x; d < n0 * n1; d += gridDim.x * blockDim.x) {
    const int i = d / n1, j = d % n1;
    const af3 p = ld3(dst + 3 * (size_t)d), lo = ld3(aabb + 6 * (size_t)d),
              hi = ld3(aabb + 6 * (size_t)d + 3);
    const float at[3] = {g.u0 + (float)i * du, g.v0 + (float)j * dv, g.w0};
    for (int k = 0; k < 3; k++) {
      const float x = comp3(p, ax[k]);
      const float dev = fabsf(x - at[k]);
      m[k] = dev < 3.0e38f ? fmaxf(m[k], dev) : 3.0e38f;  // a NaN too
      const float up = comp3(hi, ax[k]) - x, down = x - comp3(lo, ax[k]);
      m[3 + k] = fmaxf(m[3 + k], fmaxf(fabsf(up), fabsf(down)));
      // (the rounding of a box that was made of the radius)
      small = small || !(fminf(up, down) >= need - (2e-6f + 1e-7f * fabsf(x)));
    }
  }
  for (int k = 0; k < 6; k++) {
    const float v = warp_max(m[k]);
    if ((threadIdx.x & 31) == 0)
      atomicMax(reinterpret_cast<int *>(out) + k, __float_as_int(v));
  }
  if (small) reinterpret_cast<int *>(out)[8] = 1;
  __threadfence();
  __syncthreads();
  if (threadIdx.x != 0 ||
      atomicAdd(reinterpret_cast<int *>(out) + 6, 1) != (int)gridDim.x - 1)
    return;
  __threadfence();
  for (int k = 0; k < 6; k++) m[k] = __ldcg(out + k);
  // (NaN compares false; without a step the rows lie on one another, and a ray
  // may meet any of them first)
  const bool ok = g.ok && (n0 == 1 || (du != 0.0f && m[0] <= 0.25f * fabsf(du))) &&
                  (n1 == 1 || (dv != 0.0f && m[1] <= 0.25f * fabsf(dv))) && m[2] <= m[5] &&
                  m[3] < 1e6f && m[4] < 1e6f && m[5] < 1e6f &&
                  __ldcg(reinterpret_cast<const int *>(out) + 8) == 0;
  reinterpret_cast<int *>(out)[7] = ok ? 1 : 0;
}
__device__ __forceinline__ RxGrid rx_grid(const TraceDev &P) {
  float du, dv;
  RxGrid g = rx_grid_axes(P.dst, P.n0_dst, P.n1_dst, du, dv);
  const float *m = P.rx_grid;
  g.ok = reinterpret_cast<const int *>(m)[7];
  g.su = du;
  g.sv = dv;
  g.iu = du != 0.0f ? 1.0f / du : 0.0f;
  g.iv = dv != 0.0f ? 1.0f / dv : 0.0f;
  // 0.1 mm and 10 ppm of the place for rounding
  g.bu = m[3] + m[0] + 1e-4f + 1e-5f * fabsf(g.u0);
  g.bv = m[4] + m[1] + 1e-4f + 1e-5f * fabsf(g.v0);
  g.bw = m[5] + m[2] + 1e-4f + 1e-5f * fabsf(g.w0);
  return g;
}
// index range along one axis whose boxes the ray meets for t in [tn, tf]
__device__ __forceinline__ void grid_range(float o, float d, float tn, float tf, float u0, float iu,
                                           float b, int n, int &i0, int &i1) {
  const float a0 = __fmaf_rn(tn, d, o), a1 = __fmaf_rn(tf, d, o);
  // 20 ppm of the far end for its rounding
  const float e = b + 2e-5f * fmaxf(fabsf(a0), fabsf(a1));
  const float lo = fminf(a0, a1) - e - u0, hi = fmaxf(a0, a1) + e - u0;
  if (iu == 0.0f) {  // one row
    i0 = 0;
    i1 = lo <= 0.0f && hi >= 0.0f ? 0 : -1;
    return;
  }
  const float x = lo * iu, y = hi * iu;
  i0 = (int)fminf(fmaxf(ceilf(fminf(x, y) - 1e-3f), 0.0f), (float)n);
  i1 = (int)fmaxf(fminf(floorf(fmaxf(x, y) + 1e-3f), (float)(n - 1)), -1.0f);
}
// Closest Rx sphere by the grid: rows of the axis that the ray crosses more of,
// in the order in which it meets them, until they lie behind the best hit.
__device__ __forceinline__ void rx_by_grid(const TraceDev &P, const RxGrid &g, S1Query &q) {
  const float ow = comp3(q.r.o, g.wa), iw = comp3(q.r.inv, g.wa);
  const float t1 = (g.w0 - g.bw - ow) * iw, t2 = (g.w0 + g.bw - ow) * iw;
  const float tn = fmaxf(__fmaf_rn(fminf(t1, t2), 0.9999f, -1e-4f), 0.0f);
  // (a ray in the plane of the Rx stays in it: 1000 km stand for ever)
  const float tf = fminf(__fmaf_rn(fmaxf(t1, t2), 1.0001f, 1e-4f), 1e6f);
  if (!(tn <= tf)) return;
  const float ou = comp3(q.r.o, g.ua), du = comp3(q.r.d, g.ua), ov = comp3(q.r.o, g.va),
              dv = comp3(q.r.d, g.va);
  int i0, i1, j0, j1;
  grid_range(ou, du, tn, tf, g.u0, g.iu, g.bu, P.n0_dst, i0, i1);
  grid_range(ov, dv, tn, tf, g.v0, g.iv, g.bv, P.n1_dst, j0, j1);
  if (i1 < i0 || j1 < j0) return;
  const bool by_u = i1 - i0 >= j1 - j0;  // rows of constant u or of constant v
  const float oo = by_u ? ou : ov, io = comp3(q.r.inv, by_u ? g.ua : g.va),
              o0 = by_u ? g.u0 : g.v0, so = by_u ? g.su : g.sv, bo = by_u ? g.bu : g.bv;
  const float on = by_u ? ov : ou, dn = by_u ? dv : du, n0 = by_u ? g.v0 : g.u0,
              in = by_u ? g.iv : g.iu, bn = by_u ? g.bv : g.bu;
  const int nn = by_u ? P.n1_dst : P.n0_dst, step = by_u ? 1 : P.n1_dst,
            row_step = by_u ? P.n1_dst : 1;
  const int first = by_u ? i0 : j0, last = by_u ? i1 : j1;
  const bool up = (io < 0.0f) == (so < 0.0f);
#pragma unroll 1
  for (int k = 0; k <= last - first; k++) {
    const int row = up ? first + k : last - k;
    const float c = o0 + (float)row * so - oo, ta = (c - bo) * io, tb = (c + bo) * io;
    const float r0 = fmaxf(__fmaf_rn(fminf(ta, tb), 0.9999f, -1e-4f), tn),
                r1 = fminf(__fmaf_rn(fmaxf(ta, tb), 1.0001f, 1e-4f), tf);
    if (r0 > __fmaf_rn(q.best.t, 1.0001f, 1e-4f)) break;
    if (!(r0 <= r1)) continue;
    int a, b;
    grid_range(on, dn, r0, r1, n0, in, bn, nn, a, b);
#pragma unroll 1
    for (; a <= b; a++) {
      const int d = row * row_step + a * step;
      const float *x = P.dst + 3 * (size_t)d;
      const float t = sphere_hit(q.r, q.Dq, mk3(__ldg(x), __ldg(x + 1), __ldg(x + 2)), P.dst_r);
      if (t >= 0.0f && better(t, 2, d, q.best)) {
        const float *y = P.dst_aabb + 6 * (size_t)d;
        if (prim_slab(q.r, make_float4(__ldg(y), __ldg(y + 1), __ldg(y + 2), 0.f),
                      make_float4(__ldg(y + 3), __ldg(y + 4), __ldg(y + 5), 0.f))) {
          q.best.t = t; q.best.inst = 2; q.best.prim = d;
        }
      }
    }
  }
}

struct S1Ray {
  long long li;
  int ix, iy, launch, res_cnt;
  uint32_t seed;
  bool capped;
  af3 spos;
  unsigned pending;
  int cur, ttl, guard;
  // path-table slot of the last record's key: the key is a function of
  // (slot, remaining levels) within one sub-launch, and consecutive records
  // along a ray mostly repeat it
  int key_cur, key_ttl, key_slot;
};

// the hit of the finished query (stage-1 closest-hit program,
// optixPathTracer.cu:285-331)
__device__ __forceinline__ void s1_hit(const TraceDev &P, S1Query &q, S1Ray &w, Slot *slots,
                                    const CurMatrix &cm, volatile int *los_slot, int *rec,
                                    unsigned long long &my_records) {
  const int L = P.L;
  if (q.best.inst == 3) { w.ttl = 0; return; }
  const af3 d = q.r.d;
  const af3 o = add3(q.r.o, scl3(d, q.best.t));
  q.r.o = o;
  if (q.best.inst == 0 && w.ttl > 1) {
    const TriAttr tri = scene_tri(P, q.best.prim);
    const af3 v0 = tri.v0, N0 = tri.n;
    af3 N = faceforward3(N0, neg3(d), N0);
    int m = __ldg(P.mat + q.best.prim);
    float ct = dot3(d, N) / (tri.n_len * len3(d));
    int tid = theta_id(ct);
    bool pen = __ldg(P.mat_prop + tid + m * AMS_NBINS) < 0.0f;
    w.ttl--;
    int hc = L + 1 - w.ttl;
    int j = w.cur | (1 << (hc - 1));
    Mat34 M = cm.get(w.cur);
    af3 V = sub3(v0, image_of(M, w.spos));
    af3 Nimg = faceforward3(N0, V, N0);
    image_update(M, Nimg, v0);
    const af3 dr = sub3(d, scl3(N, 2.0f * dot3(d, N)));
    if (!pen && (w.pending & ((1u << j) - 1u)) == 0u) {
      // the current ray stops and the new slot is the lowest pending one, so
      // it is the next to be traced: continue with it at once, without
      // storing it (always the case when no material is penetrable)
      w.cur = j;
      w.guard = 0;
      q.r.d = dr;
      cm.set(M);
    } else {
      Slot &c = slots[j];
      c.o = o;
      c.d = dr;
      c.M = M;
      w.pending |= 1u << j;
      if (!pen) w.ttl = 0;
    }
  } else if (q.best.inst == 2) {
    if (w.res_cnt < P.reserve) {
      int d0 = q.best.prim / P.n1_dst, d1 = q.best.prim % P.n1_dst;
      int cell = (d0 / P.gs) * P.n1g + d1 / P.gs;
      int hc = L + 1 - w.ttl;
      int mhc = 0;
#pragma unroll 1
      for (int k = w.res_cnt - 1; k >= 0; k--)
        if ((rec[k] >> 3) == cell) { mhc = (rec[k] & 7) + 1; break; }
      if (mhc <= hc) {
        rec[w.res_cnt++] = cell * 8 + hc;
        int slot = w.key_slot;
        if (w.key_cur != w.cur || w.key_ttl != w.ttl) {
          // the primary ray's key depends on the hit count only (identity
          // matrix, slot 0), so the CTA keeps its slot per hit count
          slot = w.cur == 0 ? los_slot[hc] : -1;
          if (slot < 0) {
            int32_t key[14];
            const Mat34 M = cm.get(w.cur);
#pragma unroll
            for (int k = 0; k < 12; k++) key[k] = fbits(M.m[k]);
            key[12] = hc;
            key[13] = w.cur;
            slot = path_insert(P, key);
            if (w.cur == 0 && slot >= 0) los_slot[hc] = slot;
          }
          w.key_cur = w.cur;
          w.key_ttl = w.ttl;
          w.key_slot = slot;
        }
        if (slot >= 0) set_bit(P.T + (size_t)cell * P.W + (slot >> 5), 1u << (slot & 31));
        my_records++;
      }
    } else {
      w.capped = true;
    }
  }
}

// next query of the lane: the current slot's next segment, the next pending
// slot, the next sub-launch, or the next launch index.  Returns false when
// no launch index is left.
__device__ __forceinline__ bool s1_next(const TraceDev &P, S1Query &q, S1Ray &w, const Slot *slots,
                                       const CurMatrix &cm, long long n_fetch, long long tiles_y,
                                       unsigned long long &my_capped) {
  while (true) {
    if (w.ttl > 0) {
      if (++w.guard > AMS_SEG_CAP) {
        atomicOr(P.err, AMS_DERR_LOOP);
        w.ttl = 0;
        continue;
      }
      return true;
    }
    if (w.pending) {
      w.cur = __ffs(w.pending) - 1;
      w.pending &= w.pending - 1u;
      q.r.o = slots[w.cur].o;
      q.r.d = slots[w.cur].d;
      cm.set(slots[w.cur].M);
      w.ttl = slot_ttl(P.L, w.cur);
      w.guard = 0;
      continue;
    }
    if (w.li >= 0 && w.launch < P.spl) {
      w.launch++;
      float rs = rnd(w.seed) * (float)P.n_src;
      uint32_t src = (uint32_t)rs;
      if (src >= (uint32_t)P.n_src) src = (uint32_t)P.n_src - 1u;
      w.spos = ld3(P.src + 3 * src);
      // slot 0 (the primary ray) starts at once: origin and direction go
      // straight into the query, and its image matrix is the identity,
      // which is never stored (CurMatrix)
      q.r.o = w.spos;
      q.r.d = rand_dir(w.seed, (uint32_t)w.ix, (uint32_t)w.iy, P.launch_x, P.launch_y);
      w.cur = 0;
      w.ttl = P.L + 1;
      w.guard = 0;
      w.pending = 0u;
      w.key_cur = -1;  // a new ray: forget the last key
      continue;
    }
    if (w.li >= 0 && w.capped) my_capped++;
    // launch indices are dealt in tiles of 4 (ix, azimuth) x 8 (iy, height)
    // cells, so lanes that fetch together trace neighbouring directions
    // (4.09 ms on coverage-128 against 4.26 ms for 1 x 32 runs of iy and
    // 4.24-4.39 ms for 8 x 4 .. 32 x 1); n_fetch counts the tiles' cells,
    // those outside the launch are skipped
    while (true) {
      const long long f = fetch_launch(P.ctr + 10);
      if (f >= n_fetch) return false;
      const long long tile = f >> 5;
      const int c = (int)(f & 31);
      const int ix = (int)(tile / tiles_y) * 4 + (c & 3);
      const int iy = (int)(tile % tiles_y) * 8 + (c >> 2);
      if (ix < P.launch_x && iy < P.launch_y) {
        w.li = f;
        w.ix = ix;
        w.iy = iy;
        break;
      }
    }
    w.seed = tea4((uint32_t)w.ix * (uint32_t)P.launch_y + (uint32_t)w.iy, 0u);
    w.launch = 0;
    w.res_cnt = 0;
    w.capped = false;
  }
}

// 8 CTAs of 128 per SM (64 registers) measured fastest among 4 to 12.
// LMAX bounds max_reflection: 2^LMAX branch slots (slot indices hold one bit
// per hit count below L).  GRID: the instance for Rx sets that form a grid; the
// other one visits the nodes of both hierarchies in one loop, so that a lane
// whose Rx are done goes on with the scene while others still look for theirs
// (64 x 64 rotated Rx: 4.3 ms, one hierarchy after the other 4.9; in a room of 60
// triangles 2.1 and 2.4).  Without that code the grid's instance is shorter too
// (coverage-128: 2.57 -> 2.07 ms).  Both are launched, and the one that the set is
// not for returns at once (the set is looked at on the device).
template <int LMAX, bool GRID>
__global__ void __launch_bounds__(128, 8) k_stage1(const __grid_constant__ TraceDev P) {
  const long long tiles_y = (P.launch_y + 7) / 8;
  const long long n_fetch = (long long)((P.launch_x + 3) / 4) * tiles_y * 32;
  unsigned long long my_records = 0, my_segs = 0, my_capped = 0;
  float curm[12];
  const CurMatrix cm{curm};
  // path-table slot of the primary ray's key per hit count (-1: not known)
  __shared__ int s_los[AMS_MAX_L + 2];
  __shared__ RxGrid s_grid;
  if (threadIdx.x < AMS_MAX_L + 2) s_los[threadIdx.x] = -1;
  if (threadIdx.x == 32) s_grid = rx_grid(P);
  __syncthreads();
  if ((s_grid.ok != 0) != GRID) return;
  int rec[AMS_MAX_RESERVE];  // cell * 8 + hit_cnt of the records kept so far
  Slot slots[1 << LMAX];     // deferred branch slots
  int2 stack[AMS_STACK];     // node, its near distance

  S1Ray w;
  w.li = -1; w.ix = 0; w.iy = 0; w.launch = 0; w.res_cnt = 0; w.seed = 0u; w.capped = false;
  w.spos = mk3(0.f, 0.f, 0.f); w.pending = 0u; w.cur = 0; w.ttl = 0; w.guard = 0;
  w.key_cur = -1; w.key_ttl = 0; w.key_slot = -1;
  S1Query q;
  q.r.o = mk3(0.f, 0.f, 0.f);
  q.r.d = mk3(0.f, 0.f, 1.f);
  bool live = s1_next(P, q, w, slots, cm, n_fetch, tiles_y, my_capped);

  while (__any_sync(kFullWarp, live)) {
    __syncwarp();
    ray_setup(q.r, q.r.o, q.r.d);
    q.Dq = unit_dir(q.r);
    q.best.t = AMS_TMAX; q.best.inst = 3; q.best.prim = 0x7fffffff;
    // ---- Rx spheres, then the scene, pruned at the sphere hit: node visits
    // until every lane's query has ended
    if (GRID && live) rx_by_grid(P, s_grid, q);
    __syncwarp();
    if (!GRID && live && P.n_dst == 1) test_prim<2>(P.rx_prims, 0, q.r, q.best, P.dst_r, q.Dq);
    if (live && P.n_tri == 1) test_prim<0>(P.tri_prims, 0, q.r, q.best, 0.0f, q.Dq);
    bool rx = !GRID && P.n_dst > 1;
    bool trav = live && (rx || P.n_tri > 1);
    int node = 0, sp = 0;
    while (trav) {
      const int n_prims = rx ? P.n_dst : P.n_tri;
      const float4 *prims = rx ? P.rx_prims : P.tri_prims;
      if ((unsigned)node >= (unsigned)(n_prims - 1)) {
        atomicOr(P.err, AMS_DERR_BVH);
        break;
      }
      const float4 *np = reinterpret_cast<const float4 *>((rx ? P.rx_nodes : P.tri_nodes) + node);
      const float4 a = __ldg(np), b = __ldg(np + 1), c = __ldg(np + 2);
      const int2 d = __ldg(reinterpret_cast<const int2 *>(np + 3));
      float tn0, tn1;
      bool h0 = child_test(q.r, a.x, a.y, a.z, a.w, b.x, b.y, q.best.t, tn0);
      bool h1 = child_test(q.r, b.z, b.w, c.x, c.y, c.z, c.w, q.best.t, tn1);
      // leaves: one test site for both children
      const int lf0 = (h0 && d.x < 0) ? ~d.x : -1;
      const int lf1 = (h1 && d.y < 0) ? ~d.y : -1;
      if (lf0 >= 0) h0 = false;
      if (lf1 >= 0) h1 = false;
      if (lf0 >= n_prims || lf1 >= n_prims) {
        atomicOr(P.err, AMS_DERR_BVH);
        break;
      }
#pragma unroll 1
      for (int k = 0; k < 2; k++) {
        const int lf = k == 0 ? lf0 : lf1;
        if (lf < 0) continue;
        if (!GRID && rx) test_prim<2>(prims, lf, q.r, q.best, P.dst_r, q.Dq);
        else test_prim<0>(prims, lf, q.r, q.best, 0.0f, q.Dq);
      }
      if (h0 && h1) {
        const bool swap = tn1 < tn0;
        if (sp < AMS_STACK) {
          stack[sp++] = make_int2(swap ? d.x : d.y, __float_as_int(swap ? tn0 : tn1));
        } else {
          atomicOr(P.err, AMS_DERR_STACK);
        }
        node = swap ? d.y : d.x;
      } else if (h0) {
        node = d.x;
      } else if (h1) {
        node = d.y;
      } else {
        trav = false;
        const float lim = __fmaf_rn(q.best.t, 1.0001f, 1e-4f);
#pragma unroll 1
        while (sp > 0) {
          const int2 e = stack[--sp];
          if (__int_as_float(e.y) <= lim) { node = e.x; trav = true; break; }
        }
        if (!GRID && !trav && rx) {  // the Rx are done
          rx = false;
          trav = P.n_tri > 1;
          node = 0;
        }
      }
    }
    __syncwarp();
    // ---- hits of all lanes, then their next queries
    if (live) {
      my_segs++;
      s1_hit(P, q, w, slots, cm, s_los, rec, my_records);
      live = s1_next(P, q, w, slots, cm, n_fetch, tiles_y, my_capped);
    }
  }
  // block-aggregated counters
  unsigned long long rr = my_records, sg = my_segs, cp = my_capped;
  for (int off = 16; off > 0; off >>= 1) {
    rr += __shfl_xor_sync(0xffffffffu, rr, off);
    sg += __shfl_xor_sync(0xffffffffu, sg, off);
    cp += __shfl_xor_sync(0xffffffffu, cp, off);
  }
  if ((threadIdx.x & 31) == 0) {
    if (rr) atomicAdd(P.ctr + 0, rr);
    if (sg) atomicAdd(P.ctr + 8, sg);
    if (cp) atomicAdd(P.ctr + 1, cp);
  }
}

// ------------------------------------------------------------- Tx array
// tx_info of the Tx positions, 4 float4 (ray_near_tx, tx_alone): two
// directions that the array is thin along (the normal of a planar array
// twice, two normals of a linear one), each with the sine above which a ray
// meets one Tx only; then the box of all Tx boxes, widened as a node's.  Word
// 11 holds the square of the smallest distance of two Tx (the bits of the
// largest float less its own, so that 0 stands for the largest), word 15 counts
// the CTAs that have done their share of the pairs; the last one, or CTA 0 alone beyond kTxPairs Tx where no
// ray counts as steep enough, writes the rest.
constexpr int kTxPairs = 4096;
__global__ void __launch_bounds__(256) k_tx_info(const float *src, const float *aabb, int n,
                                                 float *info) {
  __shared__ float sv[8];
  __shared__ int si[8];
  __shared__ bool fit;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  if (n <= kTxPairs) {
    float best = 3.0e38f;
    for (int i = blockIdx.x; i < n; i += gridDim.x) {
      const af3 a = ld3(src + 3 * i);
      for (int j = i + 1 + t; j < n; j += blockDim.x) {
        const af3 v = sub3(ld3(src + 3 * j), a);
        best = fminf(best, dot3(v, v));
      }
    }
    best = warp_min(best);
    if (lane == 0)
      atomicMax(reinterpret_cast<int *>(info) + 11, 0x7f7fffff - __float_as_int(best));
  }
  __threadfence();
  __syncthreads();
  if (t == 0)
    fit = atomicAdd(reinterpret_cast<int *>(info) + 15, 1) == (int)gridDim.x - 1;
  __syncthreads();
  if (!fit) return;
  __threadfence();
  // the largest f(i) over the Tx and its index
  auto farthest = [&](auto f) {
    float v = -3.0e38f;
    int at = 0;
    for (int i = t; i < n; i += blockDim.x) {
      const float x = f(i);
      if (x > v) { v = x; at = i; }
    }
    for (int o = 16; o > 0; o >>= 1) {
      const float x = __shfl_xor_sync(kFullWarp, v, o);
      const int i = __shfl_xor_sync(kFullWarp, at, o);
      if (x > v) { v = x; at = i; }
    }
    __syncthreads();
    if (lane == 0) { sv[w] = v; si[w] = at; }
    __syncthreads();
    v = sv[0]; at = si[0];
    for (int i = 1; i < 8; i++)
      if (sv[i] > v) { v = sv[i]; at = si[i]; }
    return make_float2(v, __int_as_float(at));
  };
  const af3 a = ld3(src);
  auto rel = [&](int i) { return sub3(ld3(src + 3 * i), a); };
  const float2 f1 = farthest([&](int i) { const af3 v = rel(i); return dot3(v, v); });
  const af3 v1 = rel(__float_as_int(f1.y));
  const float len = sqrtf(fmaxf(f1.x, 0.0f));
  const af3 u = len > 0.0f ? scl3(v1, 1.0f / len) : mk3(1.f, 0.f, 0.f);
  const float2 f2 = farthest([&](int i) { const af3 c = cross3(rel(i), u); return dot3(c, c); });
  af3 n1, n2;
  if (f2.x > 1e-6f * len * len) {  // a plane
    n1 = cross3(rel(__float_as_int(f2.y)), u);
    n1 = scl3(n1, 1.0f / len3(n1));
    n2 = n1;
  } else {  // a line
    const af3 e = fabsf(u.x) < 0.6f ? mk3(1.f, 0.f, 0.f) : mk3(0.f, 1.f, 0.f);
    n1 = cross3(u, e);
    n1 = scl3(n1, 1.0f / len3(n1));
    n2 = cross3(u, n1);
  }
  const float e1 = farthest([&](int i) { return fabsf(dot3(rel(i), n1)); }).x;
  const float e2 = farthest([&](int i) { return fabsf(dot3(rel(i), n2)); }).x;
  const float rh = farthest([&](int i) {
    const af3 c = ld3(src + 3 * i), lo = sub3(c, ld3(aabb + 6 * i)),
              hi = sub3(ld3(aabb + 6 * i + 3), c);
    return len3(mk3(fmaxf(fabsf(lo.x), fabsf(hi.x)), fmaxf(fabsf(lo.y), fabsf(hi.y)),
                    fmaxf(fabsf(lo.z), fabsf(hi.z))));
  }).x;
  float bx[6];
  for (int k = 0; k < 6; k++) {
    const float sign = k < 3 ? -1.0f : 1.0f;
    bx[k] = sign * farthest([&](int i) { return sign * aabb[6 * i + k]; }).x;
    bx[k] += sign * (1e-5f + 2e-6f * fabsf(bx[k]));
  }
  if (t == 0) {
    // two Tx may lie on either side of the first; 20 um of slack for the
    // rounding of positions and box tests over a building
    const float rho = 2.0f * (rh + 2e-5f);
    const float d2 = __int_as_float(0x7f7fffff - __ldcg(reinterpret_cast<int *>(info) + 11));
    const float gap = n <= kTxPairs ? sqrtf(d2) - rho : 0.0f;
    float4 *o = reinterpret_cast<float4 *>(info);
    o[0] = make_float4(n1.x, n1.y, n1.z, gap > 0.0f ? (2.0f * e1 + rho) / gap + 1e-3f : 3.0e38f);
    o[1] = make_float4(n2.x, n2.y, n2.z, gap > 0.0f ? (2.0f * e2 + rho) / gap + 1e-3f : 3.0e38f);
    o[2] = make_float4(bx[0], bx[1], bx[2], 0.0f);
    o[3] = make_float4(bx[3], bx[4], bx[5], 0.0f);
  }
}

// --------------------------------------------------------------- tasks
// Dense path ids: after stage 1 the path table is final, so stage 2 numbers
// its paths 0 .. n_paths - 1 (slot_of maps back to the table) and keeps its
// bitmaps [cell][W] with W = ceil(n_paths / 32) words instead of one bit per
// table slot.  The numbering follows the order in which threads claim ids;
// nothing computed depends on it (sums are exact, lists are per cell).
__global__ void k_dense_ids(TraceDev P, int *dense_of, unsigned long long *n) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s <= P.tab_mask;
       s += gridDim.x * blockDim.x) {
    if (P.tab_h[s] == 0ull) continue;
    const unsigned long long id = atomicAdd(n, 1ull);
    dense_of[s] = (int)id;
    P.slot_of[id] = (int)s;
  }
}

// out[cell][dense id] = the bits of in[cell][slot] (out zeroed before)
__global__ void k_to_dense(TraceDev P, const unsigned *in, int w_in, const int *dense_of,
                           unsigned *out) {
  const long long nwords = (long long)P.ng * w_in;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nwords;
       i += (long long)gridDim.x * blockDim.x) {
    unsigned b = in[i];
    if (!b) continue;
    const int cell = (int)(i / w_in), w = (int)(i % w_in);
    while (b) {
      const int k = __ffs(b) - 1;
      b &= b - 1u;
      const int d = dense_of[w * 32 + k];
      atomicOr(out + (size_t)cell * P.W + (d >> 5), 1u << (d & 31));
    }
  }
}

// With per-ray records (EXPORT) a round's tasks are listed in a fixed order,
// cell by cell: cell c's new paths (dense ids) are
// task_path[cell_off[c] .. cell_off[c + 1]) in increasing order, cut into
// chunks of up to kpi paths: chunk_at[chunk_off[c] ..] = (cell, first
// task).  A warp per cell counts, one CTA scans, a warp per cell fills.
__global__ void k_cell_counts(TraceDev P, const unsigned *bits) {
  const int lane = threadIdx.x & 31;
  const int nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int cell = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; cell < P.ng; cell += nwarp) {
    const unsigned *row = bits + (size_t)cell * P.W;
    int c = 0;
    for (int w = lane; w < P.W; w += 32) c += __popc(row[w]);
    for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
    if (lane == 0) P.cell_cnt[cell] = c;
  }
}

// exclusive scans of the task and chunk counts (cell_cnt) into cell_off and
// chunk_off ([ng] = totals); one CTA of 1024 threads
__global__ void __launch_bounds__(1024) k_cell_scan(TraceDev P) {
  __shared__ int wsum[32], wch[32];
  __shared__ int carry_s, ccarry_s;
  const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
  if (t == 0) { carry_s = 0; ccarry_s = 0; }
  __syncthreads();
  for (int base = 0; base < P.ng; base += 1024) {
    const int i = base + t;
    const int v = i < P.ng ? P.cell_cnt[i] : 0;
    const int ch = (v + P.kpi - 1) / P.kpi;
    int x = v, y = ch;
    for (int o = 1; o < 32; o <<= 1) {
      const int x2 = __shfl_up_sync(0xffffffffu, x, o);
      const int y2 = __shfl_up_sync(0xffffffffu, y, o);
      if (lane >= o) { x += x2; y += y2; }
    }
    if (lane == 31) { wsum[wid] = x; wch[wid] = y; }
    __syncthreads();
    int xb = 0, yb = 0;
    for (int k = 0; k < wid; k++) { xb += wsum[k]; yb += wch[k]; }
    const int carry = carry_s, ccarry = ccarry_s;
    if (i < P.ng) {
      P.cell_off[i] = carry + xb + x - v;
      P.chunk_off[i] = ccarry + yb + y - ch;
    }
    __syncthreads();
    if (t == 0) {
      int xs = 0, ys = 0;
      for (int k = 0; k < 32; k++) { xs += wsum[k]; ys += wch[k]; }
      carry_s = carry + xs;
      ccarry_s = ccarry + ys;
    }
    __syncthreads();
  }
  if (t == 0) {
    P.cell_off[P.ng] = carry_s;
    P.chunk_off[P.ng] = ccarry_s;
    RoundCount *rc = P.rounds + (P.round_slot & (AMS_ROUND_SLOTS - 1));
    rc->listed = (unsigned long long)carry_s;
    rc->chunks = (unsigned long long)ccarry_s;
  }
}

__global__ void k_cell_fill(TraceDev P, const unsigned *bits) {
  const int lane = threadIdx.x & 31;
  const int nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int cell = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; cell < P.ng; cell += nwarp) {
    const int first = P.cell_off[cell], end = P.cell_off[cell + 1];
    if (first == end) continue;
    const unsigned *row = bits + (size_t)cell * P.W;
    long long pos = first;
    for (int w0 = 0; w0 < P.W; w0 += 32) {
      const int w = w0 + lane;
      unsigned b = w < P.W ? row[w] : 0u;
      const int c = __popc(b);
      int x = c;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      long long q = pos + x - c;
      while (b) {
        const int k = __ffs(b) - 1;
        b &= b - 1u;
        const int id = w * 32 + k;
        if ((unsigned long long)q < P.task_cap)
          P.task_path[q] = make_int2(id, id < P.n_paths ? P.slot_of[id] : -1);
        else atomicOr(P.err, AMS_DERR_TASKS);
        q++;
      }
      pos += __shfl_sync(0xffffffffu, x, 31);
    }
    const int c0 = P.chunk_off[cell], c1 = P.chunk_off[cell + 1];
    for (int j = c0 + lane; j < c1; j += 32) {
      const int t0 = first + (j - c0) * P.kpi;
      if ((unsigned long long)j < P.task_cap) P.chunk_at[j] = make_int4(cell, t0, min(end, t0 + P.kpi), 0);
      else atomicOr(P.err, AMS_DERR_TASKS);
    }
  }
}

// Flood-fill step and task list of a round in one kernel, a warp per cell.
// EXPAND: N = (S of the 4 neighbour cells) & ~T; T |= N (cpp:257-300; the
// neighbours are linear cell indices +-1 and +-n1g with only the [0, ng)
// check, exactly as the reference, so row ends wrap), and S_next, where the
// coming stage 2 sets its success bits, is cleared.  Without EXPAND the new
// tasks are the bits of N already.  LIST: the cell's new tasks in path order
// go to a run of task_path that the warp claims, cut into chunks of up to kpi
// paths in chunk_at.  The order of the runs differs from one execution to the
// next; nothing computed depends on it.  The counts go to the round's slot of
// the ring `rounds`, whose next slot is zeroed.  Replaces four kernels and two
// copies a round (count, scan, fill, expand: 20 us of 33 us between the
// stage-2 kernels of coverage-128's late rounds).
template <bool EXPAND, bool LIST>
__global__ void __launch_bounds__(256) k_round(const __grid_constant__ TraceDev P) {
  const int lane = threadIdx.x & 31;
  RoundCount *rc = P.rounds + (P.round_slot & (AMS_ROUND_SLOTS - 1));
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    RoundCount *nx = P.rounds + ((P.round_slot + 1) & (AMS_ROUND_SLOTS - 1));
    nx->tasks = 0ull;
    nx->listed = 0ull;
    nx->chunks = 0ull;
  }
  const int nwarp = (gridDim.x * blockDim.x) >> 5;
  for (int cell = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; cell < P.ng; cell += nwarp) {
    const size_t row = (size_t)cell * P.W;
    int cnt = 0;
    for (int w = lane; w < P.W; w += 32) {
      unsigned n;
      if (EXPAND) {
        unsigned s = 0;
        const int nb[4] = {cell - 1, cell + 1, cell - P.n1g, cell + P.n1g};
#pragma unroll
        for (int k = 0; k < 4; k++)
          if (nb[k] >= 0 && nb[k] < P.ng) s |= __ldg(P.S + (size_t)nb[k] * P.W + w);
        const unsigned t = P.T[row + w];
        n = s & ~t;
        if (n) P.T[row + w] = t | n;
        P.N[row + w] = n;
        P.S_next[row + w] = 0u;
      } else {
        n = P.N[row + w];
      }
      cnt += __popc(n);
    }
    cnt = __reduce_add_sync(kFullWarp, cnt);
    if (cnt == 0) continue;
    unsigned long long first = 0, c0 = 0;
    const int nch = (cnt + P.kpi - 1) / P.kpi;
    if (lane == 0) {
      first = atomicAdd(EXPAND ? &rc->tasks : &rc->listed, (unsigned long long)cnt);
      if (LIST) c0 = atomicAdd(&rc->chunks, (unsigned long long)nch);
    }
    if (!LIST) continue;
    first = __shfl_sync(kFullWarp, first, 0);
    c0 = __shfl_sync(kFullWarp, c0, 0);
    if (first + cnt > P.task_cap) {
      if (lane == 0) atomicOr(P.err, AMS_DERR_TASKS);
      continue;
    }
    __syncwarp();
    unsigned long long pos = first;
    for (int w0 = 0; w0 < P.W; w0 += 32) {
      const int w = w0 + lane;
      unsigned b = w < P.W ? P.N[row + w] : 0u;
      const int c = __popc(b);
      int x = c;
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFullWarp, x, o);
        if (lane >= o) x += y;
      }
      unsigned long long q = pos + x - c;
      while (b) {
        const int id = w * 32 + __ffs(b) - 1;
        b &= b - 1u;
        P.task_path[q++] = make_int2(id, id < P.n_paths ? P.slot_of[id] : -1);
      }
      pos += __shfl_sync(kFullWarp, x, 31);
    }
    for (int j = lane; j < nch; j += 32) {
      const int t0 = (int)first + j * P.kpi;
      P.chunk_at[c0 + j] = make_int4(cell, t0, min((int)first + cnt, t0 + P.kpi), 0);
    }
  }
}

// ---------------------------------------------------------------- stage 2
// One backward ray per active lane (stage-2 raygen + closest-hit programs,
// optixPathTracer.cu:191-273, :332-417): the image source of the path key in
// `slot` (the same for the whole warp) seen from Rx position o, traced back to
// Tx `s`.  Every scene hit lowers the remaining levels by one, so the warp's
// rays stay at the same segment.  Returns true with the contribution as 2^-56
// fixed point when the ray arrives.  Warp collective.
template <bool EXPORT>
__device__ __forceinline__ bool s2_ray(const TraceDev &P, int slot, int s, af3 o,
                                       bool act, int2 *stk, unsigned &segs,
                                       unsigned long long &cre, unsigned long long &cim,
                                       ams_ray_record *rr) {
  const int32_t *key = P.tab_key + (size_t)slot * 14;
  Mat34 M;
#pragma unroll
  for (int k = 0; k < 12; k++) M.m[k] = __int_as_float(key_word(key, k));
  const int hc = key_word(key, 12), mask = key_word(key, 13);
  const float lam = P.lam_f;
  const af3 srcdir = mk3(P.src_dir[0], P.src_dir[1], P.src_dir[2]);
  const af3 dstdir = mk3(P.dst_dir[0], P.dst_dir[1], P.dst_dir[2]);
  af3 d = nrm3(sub3(image_of(M, ld3(P.src + 3 * s)), o));
  float amp = beampattern(d, dstdir, P.dst_bp);
  float xloss = 1.0f;  // exported: free-space factors only
  if (EXPORT) {
    rr->receive_angle = dot3(d, dstdir) / (len3(d) * len3(dstdir));
    rr->hit_cnt = 0;
  }
  float far = 1e6f, dd = 0.0f, dres = 0.0f;
  double D = 0.0;
  bool ok = false;
  for (int ttl = hc + 1; ttl > 0; ttl--) {
    if (!__any_sync(kFullWarp, act)) break;
    const bool last = ttl == 1;
    // a ray that meets another Tx's sphere goes on behind it; the warp's other
    // rays wait for it
    bool todo = act;
    int prim = 0;
    for (int guard = 0; __any_sync(kFullWarp, todo); guard++) {
      if (guard >= AMS_SEG_CAP) {
        if (todo) { atomicOr(P.err, AMS_DERR_LOOP); act = false; }
        break;
      }
      __syncwarp();
      const Hit h = closest_s2(P, o, d, s, last, todo, stk);
      if (todo) {
        segs++;
        const bool other = h.inst == 1 && h.prim != s;
        if (h.inst != 3) {
          o = add3(o, scl3(d, h.t));
          dd += h.t;
          D += (double)h.t;
        }
        prim = h.prim;
        todo = other;
        // the segment has to end on a triangle, the last one on Tx s
        if (!other && h.inst != (last ? 1 : 0)) act = false;
      }
      __syncwarp();
    }
    if (act && !last) {
      const TriAttr tri = scene_tri(P, prim);
      const float max_d = tri.max_d;
      const af3 N = faceforward3(tri.n, neg3(d), tri.n);
      int m = __ldg(P.mat + prim);
      float ct = dot3(d, N) / (tri.n_len * len3(d));
      float loss = fabsf(__ldg(P.mat_prop + theta_id(ct) + m * AMS_NBINS));
      int hcb = hc + 2 - ttl;
      int is_ref = (mask >> (hcb - 1)) & 1;
      float fspl = 1.0f;
      if (dd > far) { fspl = lam / ((4.0f * AMS_PIF) * dres); dres = 0.0f; }
      amp *= loss * fspl;
      dres += dd;
      if (EXPORT) {
        if (rr->hit_cnt < 5) rr->hit_loss_idx[rr->hit_cnt] = theta_id(ct) + m * AMS_NBINS;
        rr->hit_cnt++;
        xloss *= fspl;
      }
      // far_dist = 2 max_d^2 / lambda, divided in double and rounded to
      // float (optixPathTracer.cu:385-389).  Its value matters only when
      // the segment is longer; a float estimate (relative error < 3e-7)
      // with a 1e-5 margin settles the common near-field case without
      // the double division (FP64 is slow on this part).
      float far_next = 1e6f;
      if (dd > ((2.0f * max_d) * max_d / lam) * 0.99999f) {
        const float fd = (float)(2.0 * (double)max_d * (double)max_d / (double)lam);
        far_next = (dd > fd) ? fd : 1e6f;
      }
      far = far_next;
      dd = 0.0f;
      if (is_ref) d = sub3(d, scl3(N, 2.0f * dot3(d, N)));
    } else if (act) {
      float bp = beampattern(neg3(d), srcdir, P.src_bp);
      float af = lam / ((4.0f * AMS_PIF) * (dres + dd));
      amp *= bp * af;
      ok = true;
      if (EXPORT) {
        const af3 nd = neg3(d);
        rr->launch_angle = dot3(nd, srcdir) / (len3(nd) * len3(srcdir));
        rr->loss = xloss * af;
        rr->phase = D * P.two_pi_over_lam;
      }
    }
    __syncwarp();
  }
  if (ok) {
    // FP64 path length -> phase, reduced mod 2 pi in FP64 (products with
    // precomputed 2 pi / lambda and 1 / (2 pi): no FP64 division per ray)
    double ph = D * P.two_pi_over_lam;
    ph = ph - 6.283185307179586 * floor(ph * 0.15915494309189535);
    float sn, cs;
    sincosf((float)ph, &sn, &cs);
    // the contribution in 2^-56 fixed point, in FP32: the limit (64) and the
    // scale (2^56) are powers of two, so the range test and the scaling are
    // exact in float and the rounding to an integer sees the same value as
    // a conversion through double would (FP64 is slow on this part)
    const float re = amp * cs, im = -amp * sn;
    if (!(fabsf(re) < (float)AMS_ACC_LIMIT && fabsf(im) < (float)AMS_ACC_LIMIT)) {
      atomicOr(P.err, AMS_DERR_ACC_RANGE);
      return false;
    }
    cre = (unsigned long long)__float2ll_rn(re * (float)AMS_ACC_SCALE);
    cim = (unsigned long long)__float2ll_rn(im * (float)AMS_ACC_SCALE);
  }
  return ok;
}

// Stage 2: a warp takes an item = (a chunk of up to kpi of one cell's new
// paths, 32 consecutive (Rx within the cell, Tx) pairs, Tx fastest) and traces
// the chunk's paths one after the other, the 32 rays of a path as a beam; each
// lane sums its pair's contributions over the chunk in registers (exact
// 64-bit fixed point) and adds them once into the Rx-major accumulator
// acc[dst][s], so a warp's adds cover one or a few contiguous runs of Tx
// (coalesced), one atomic add per (Tx, Rx) and chunk instead of two per
// verified ray.  One warp per item, 8 per CTA: the block scheduler balances
// items of uneven cost (fixed strides over persistent warps and a fetch
// counter both measured slower); kpi is chosen per round by the host so that a
// round keeps several items per resident warp.  The launch covers the items
// when the host knows their number, else (late rounds, whose list the host has
// not seen) the resident warps stride over them.  With EXPORT (kpi = 1) every
// ray's record is written.
template <bool EXPORT>
__global__ void __launch_bounds__(256, 4) k_stage2(const __grid_constant__ TraceDev P) {
  __shared__ int2 stack[8][AMS_BEAM_STACK];
  const int lane = threadIdx.x & 31;
  const unsigned n_chunks = (unsigned)P.rounds[P.round_slot & (AMS_ROUND_SLOTS - 1)].chunks;
  const long long n_items = (long long)n_chunks * P.s2_groups;
  unsigned n_ok = 0, n_fail = 0, n_segs = 0, n_adds = 0;  // n_adds: warp total
  long long item = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (item >= n_items) return;
  for (; item < n_items; item += (long long)gridDim.x * (blockDim.x >> 5)) {
    unsigned ck, grp;  // chunk and group of 32 pairs
    if (n_items <= 0xffffffffll) {
      ck = fdiv((unsigned)item, P.div_groups);
      grp = (unsigned)item - ck * P.s2_groups;
    } else {
      ck = (unsigned)(item / P.s2_groups);
      grp = (unsigned)(item % P.s2_groups);
    }
    const int4 chunk = __ldg(P.chunk_at + ck);
    const int cell = chunk.x, t0 = chunk.y, t1 = chunk.z;
    if ((unsigned)cell >= (unsigned)P.ng || t0 < 0 || t1 < t0 ||
        (unsigned long long)t1 > P.task_cap) {
      if (lane == 0) atomicOr(P.err, AMS_DERR_TASKS);
      break;
    }
    const long long pairs = (long long)P.gs * P.gs * P.n_src;
    const long long pr = (long long)grp * 32 + lane;
    const bool pair = pr < pairs;
    const unsigned inner = !pair ? 0u : pr <= 0xffffffffll ? fdiv((unsigned)pr, P.div_src)
                                                          : (unsigned)(pr / P.n_src);
    const int s = pair ? (int)(pr - (long long)inner * P.n_src) : 0;
    const int ir = (int)fdiv(inner, P.div_gs), gi = (int)fdiv((unsigned)cell, P.div_n1g);
    const int di = ir + gi * P.gs, dj = (int)inner - ir * P.gs + (cell - gi * P.n1g) * P.gs;
    const int dst = di * P.n1_dst + dj;
    const bool act = pair && !(dst >= P.n_dst ||
                               (P.strict_grid && (di >= P.n0_dst || dj >= P.n1_dst)));
    const af3 o = act ? ld3(P.dst + 3 * (size_t)dst) : mk3(0.f, 0.f, 0.f);
    bool any_ok = false;
    unsigned long long sre = 0, sim = 0;
    for (int t = t0; t < t1; t++) {
      const int2 task = __ldg(P.task_path + t);
      const int path = task.x, slot = task.y;
      if ((unsigned)path >= (unsigned)P.n_paths || (unsigned)slot > P.tab_mask) {
        if (lane == 0) atomicOr(P.err, AMS_DERR_TASKS);
        break;
      }
      ams_ray_record rr;
      if (EXPORT) {
        rr.src = s; rr.dst = pair ? dst : -1; rr.path = path; rr.traced = act ? 1 : 0;
        rr.successful = 0; rr.hit_cnt = 0;
        rr.launch_angle = 0.f; rr.receive_angle = 0.f; rr.loss = 0.f; rr.pad0 = 0.f;
        rr.phase = 0.0; rr.pad1 = 0;
#pragma unroll
        for (int i = 0; i < 5; i++) rr.hit_loss_idx[i] = -1;
      }
      unsigned long long cre = 0, cim = 0;
      const bool ok = s2_ray<EXPORT>(P, slot, s, o, act, stack[threadIdx.x >> 5], n_segs, cre, cim,
                                     &rr);
      if (ok) { sre += cre; sim += cim; n_ok++; any_ok = true; } else if (act) { n_fail++; }
      if (EXPORT && pair) {
        if (!act) rr.receive_angle = 0.f;  // not traced
        rr.successful = ok ? 1 : 0;
        const unsigned long long at = P.rec_base + (unsigned long long)t * pairs + pr;
        if (at < P.rec_cap) P.rec[at] = rr;
      }
      if (__any_sync(kFullWarp, ok) && lane == 0)
        atomicOr(P.S + (size_t)cell * P.W + (path >> 5), 1u << (path & 31));
    }
    const bool add = P.kpi == 1 ? any_ok : act && (sre | sim);
    if (add) {
      unsigned long long *acc = P.acc + ((size_t)dst * P.n_src + s) * 2;
      atomicAdd(acc, sre);
      atomicAdd(acc + 1, sim);
    }
    n_adds += 2u * (unsigned)__popc(__ballot_sync(kFullWarp, add));
  }
  n_ok = __reduce_add_sync(kFullWarp, n_ok);
  n_fail = __reduce_add_sync(kFullWarp, n_fail);
  n_segs = __reduce_add_sync(kFullWarp, n_segs);
  if (lane == 0) {
    if (n_adds) atomicAdd(P.ctr + 13, (unsigned long long)n_adds);
    if (n_segs) atomicAdd(P.ctr + 9, (unsigned long long)n_segs);
    if (n_ok) atomicAdd(P.ctr + 3, (unsigned long long)n_ok);
    if (n_fail) atomicAdd(P.ctr + 4, (unsigned long long)n_fail);
  }
}

__global__ void k_popcount(const unsigned *bits, long long n, unsigned long long *out) {
  unsigned long long c = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x)
    c += __popc(bits[i]);
  for (int off = 16; off > 0; off >>= 1) c += __shfl_xor_sync(0xffffffffu, c, off);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(out, c);
}

// result[s][dst] += acc[dst][s] * 2^-56 (re, im): 32 x 32 tiles turned
// through shared memory, reads coalesced over s and writes over dst.
// Block (32, 8), grid (ceil(n_dst / 32), ceil(n_src / 32)).
__global__ void k_finalize(const unsigned long long *acc, float *result, int n_src, int n_dst) {
  __shared__ float2 tl[32][33];
  const int d0 = blockIdx.x * 32, s0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int d = d0 + i, s = s0 + threadIdx.x;
    float2 v = make_float2(0.f, 0.f);
    if (d < n_dst && s < n_src) {
      const unsigned long long *a = acc + ((size_t)d * n_src + s) * 2;
      v = make_float2((float)((double)(long long)a[0] * AMS_ACC_INV),
                      (float)((double)(long long)a[1] * AMS_ACC_INV));
    }
    tl[i][threadIdx.x] = v;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int s = s0 + i, d = d0 + threadIdx.x;
    if (s >= n_src || d >= n_dst) continue;
    const float2 v = tl[threadIdx.x][i];
    if (v.x != 0.f || v.y != 0.f) {
      float2 *r = reinterpret_cast<float2 *>(result) + (size_t)s * n_dst + d;
      float2 x = *r;
      x.x += v.x;
      x.y += v.y;
      *r = x;
    }
  }
}

__global__ void k_export(TraceDev P, int32_t *out, unsigned long long *n_out) {
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s <= P.tab_mask;
       s += gridDim.x * blockDim.x) {
    if (P.tab_h[s] == 0ull) continue;
    unsigned long long k = atomicAdd(n_out, 1ull);
    for (int i = 0; i < 14; i++)
      out[k * 14 + i] = (int32_t)((uint32_t)P.tab_key[(size_t)s * 14 + i] ^ AMS_KEY_FLIP);
  }
}

int grid_for(long long n, int block) {
  long long b = (n + block - 1) / block;
  const long long cap = (long long)ams_device_sms() * 16;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

}  // namespace

cudaError_t trace_tri_attr(const float *tris, int n, float4 *attr, cudaStream_t st) {
  if (n > 0) k_tri_attr<<<(n + 255) / 256, 256, 0, st>>>(tris, n, attr);
  return cudaGetLastError();
}

cudaError_t trace_tx_info(const float *src, const float *aabb, int n, float *info,
                          cudaStream_t st) {
  const int blocks = n > kTxPairs ? 1 : std::min(n, 304);
  k_tx_info<<<blocks, 256, 0, st>>>(src, aabb, n, info);
  return cudaGetLastError();
}

cudaError_t trace_rx_grid(const float *dst, const float *aabb, int n0, int n1, float radius,
                          float *out, cudaStream_t st) {
  k_rx_grid<<<grid_for((long long)n0 * n1, 256), 256, 0, st>>>(dst, aabb, n0, n1, radius, out);
  return cudaGetLastError();
}

cudaError_t trace_stage1(const TraceDev &P, cudaStream_t st) {
  // persistent: as many CTAs as are resident at once (lanes fetch launch
  // indices from ctr[10], zeroed with the other counters)
  long long n = (long long)P.launch_x * P.launch_y;
  // the smallest slot array that holds max_reflection's slots
  const int lk = P.L <= 2 ? 0 : (P.L == 3 ? 1 : 2);
  void (*const kern[2][3])(TraceDev) = {
      {k_stage1<2, false>, k_stage1<3, false>, k_stage1<AMS_MAX_L, false>},
      {k_stage1<2, true>, k_stage1<3, true>, k_stage1<AMS_MAX_L, true>}};
  static int per_sm[2][3][AMS_MAX_DEVICES] = {{{0}}};
  const int dev = ams_current_device();
  if (dev < 0) return cudaErrorInvalidDevice;
  for (int g = P.n_dst > 1 ? 1 : 0; g >= 0; g--) {  // (one Rx is no grid)
    int &ps = per_sm[g][lk][dev];
    if (ps == 0) {
      int b = 0;
      cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern[g][lk], 128, 0);
      if (e != cudaSuccess) return e;
      ps = b > 0 ? b : 1;
    }
    long long blocks = (long long)ps * ams_device_sms();
    const long long need = (n + 127) / 128;
    if (blocks > need) blocks = need;
    if (blocks < 1) blocks = 1;
    kern[g][lk]<<<(int)blocks, 128, 0, st>>>(P);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

namespace {
int stage2_per_sm() {
  static int per_sm[AMS_MAX_DEVICES] = {0};
  const int dev = ams_current_device();
  if (dev < 0) return 1;
  if (per_sm[dev] == 0) {
    int b = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_stage2<false>, 256, 0) != cudaSuccess) b = 1;
    per_sm[dev] = b > 0 ? b : 1;
  }
  return per_sm[dev];
}
}  // namespace

int trace_paths_per_item(const TraceDev &P, unsigned long long n_tasks) {
  // several paths per item (fewer atomic adds) only when a round still has
  // about 32 items per resident warp with them: long items at the end of a
  // smaller round leave the GPU idle.  (8 or 128 items per warp: the traces
  // take the same time, the adds differ.)
  const unsigned long long warps = (unsigned long long)stage2_per_sm() * ams_device_sms() * 8;
  const unsigned long long pairs = (unsigned long long)(P.gs * P.gs) * P.n_src;
  const unsigned long long work = n_tasks * ((pairs + 31) / 32);
  unsigned long long k = work / (32 * warps);
  if (k < 1) k = 1;
  if (k > 16) k = 16;
  return (int)k;
}

cudaError_t trace_dense_paths(const TraceDev &P, const unsigned *T_slots, int w_slots,
                              int *dense_of, unsigned *out, cudaStream_t st) {
  k_dense_ids<<<grid_for((long long)P.tab_mask + 1, 256), 256, 0, st>>>(P, dense_of, P.ctr + 12);
  k_to_dense<<<grid_for((long long)P.ng * w_slots, 256), 256, 0, st>>>(P, T_slots, w_slots,
                                                                      dense_of, out);
  return cudaGetLastError();
}

cudaError_t trace_round(const TraceDev &P, bool expand, bool list, cudaStream_t st) {
  const int blocks = grid_for((long long)P.ng * 32, 256);
  if (expand && list) k_round<true, true><<<blocks, 256, 0, st>>>(P);
  else if (expand) k_round<true, false><<<blocks, 256, 0, st>>>(P);
  else if (list) k_round<false, true><<<blocks, 256, 0, st>>>(P);
  return cudaGetLastError();
}

cudaError_t trace_list_ordered(const TraceDev &P, cudaStream_t st) {
  const int blocks = grid_for((long long)P.ng * 32, 256);
  k_cell_counts<<<blocks, 256, 0, st>>>(P, P.N);
  k_cell_scan<<<1, 1024, 0, st>>>(P);
  k_cell_fill<<<blocks, 256, 0, st>>>(P, P.N);
  return cudaGetLastError();
}

cudaError_t trace_stage2(const TraceDev &P, unsigned long long n_tasks, cudaStream_t st) {
  // one warp per item; the chunks number at most n_tasks / kpi + one per
  // cell (the exact count is on the device, warps beyond it return); with no
  // n_tasks, the warps that are resident at once
  unsigned long long blocks = (unsigned long long)stage2_per_sm() * ams_device_sms();
  if (n_tasks > 0) {
    const unsigned long long k = (unsigned long long)P.kpi;
    unsigned long long chunks = (n_tasks + k - 1) / k + (unsigned long long)P.ng;
    if (chunks > n_tasks) chunks = n_tasks;
    blocks = (chunks * P.s2_groups + 7) / 8;
    if (blocks > 0x7fffffffull) return cudaErrorInvalidConfiguration;
  }
  if (P.rec) {
    if (P.kpi != 1) return cudaErrorInvalidValue;
    k_stage2<true><<<(unsigned)blocks, 256, 0, st>>>(P);
  } else {
    k_stage2<false><<<(unsigned)blocks, 256, 0, st>>>(P);
  }
  return cudaGetLastError();
}

bool trace_round_is_small(const TraceDev &P, unsigned long long n_tasks) {
  // up to four items per resident warp
  const unsigned long long warps = (unsigned long long)stage2_per_sm() * ams_device_sms() * 8;
  return n_tasks * P.s2_groups <= 4 * warps;
}

cudaError_t trace_count_bits(const TraceDev &P, const unsigned *bits, unsigned long long *out,
                             cudaStream_t st) {
  long long n = (long long)P.ng * P.W;
  k_popcount<<<grid_for(n, 256), 256, 0, st>>>(bits, n, out);
  return cudaGetLastError();
}

cudaError_t trace_finalize(const TraceDev &P, float *result, cudaStream_t st) {
  dim3 grid((P.n_dst + 31) / 32, (P.n_src + 31) / 32), block(32, 8);
  k_finalize<<<grid, block, 0, st>>>(P.acc, result, P.n_src, P.n_dst);
  return cudaGetLastError();
}

cudaError_t trace_export_paths(const TraceDev &P, int32_t *out, unsigned long long *n_out,
                               cudaStream_t st) {
  k_export<<<grid_for((long long)P.tab_mask + 1, 256), 256, 0, st>>>(P, out, n_out);
  return cudaGetLastError();
}
