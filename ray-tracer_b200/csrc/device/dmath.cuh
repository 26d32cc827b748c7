#pragma once
// fp32 vector maths, the per-sample PCG32 stream, sampling routines and robust
// ray spawning for the sm_100a kernels.
//
// RNG: the stream for sample s of pixel p is keyed exactly as the reference's
// Rng::for_sample (include/raytracer/math/rng.hpp:10-46): SplitMix64 finaliser
// over (seed, pixel, sample), PCG32 (O'Neill 2014) with a 64-bit state and a
// per-stream increment. The integer outputs are bit-identical to the CPU's and
// are drawn in the same order; only the mapping to [0, 1) differs (24 bits here,
// so a float can never round up to 1).
#include <cstdint>

#include "device/layout.h"

namespace rtg {

__device__ __forceinline__ float3 f3(float a, float b, float c) { return make_float3(a, b, c); }
__device__ __forceinline__ float3 f3(float4 v) { return make_float3(v.x, v.y, v.z); }
// Pinned rounding, for everything a sample's value depends on: every product and sum
// is an explicit fmaf or an __fmul_rn / __fadd_rn / __fsub_rn, which the compiler
// never fuses, so the bits do not depend on the kernel the code is inlined into, on
// its register limit or on what else it computes. (Left to contract freely, the same
// source rounded differently in different instances of a kernel.) The vector operators
// round each operation; mad3, dot3 and dot3p say which product is fused. Where two forms
// would do, each place keeps the one its values have always had.
__device__ __forceinline__ float3 operator+(float3 a, float3 b) {
  return f3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z));
}
__device__ __forceinline__ float3 operator-(float3 a, float3 b) {
  return f3(__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z));
}
__device__ __forceinline__ float3 operator-(float3 a) { return f3(-a.x, -a.y, -a.z); }
__device__ __forceinline__ float3 operator*(float3 a, float3 b) {
  return f3(__fmul_rn(a.x, b.x), __fmul_rn(a.y, b.y), __fmul_rn(a.z, b.z));
}
__device__ __forceinline__ float3 operator*(float3 a, float s) {
  return f3(__fmul_rn(a.x, s), __fmul_rn(a.y, s), __fmul_rn(a.z, s));
}
__device__ __forceinline__ float3 operator*(float s, float3 a) { return a * s; }
// a b + c, fused.
__device__ __forceinline__ float3 mad3(float a, float3 b, float3 c) {
  return f3(fmaf(a, b.x, c.x), fmaf(a, b.y, c.y), fmaf(a, b.z, c.z));
}
__device__ __forceinline__ float3 mad3(float3 a, float3 b, float3 c) {
  return f3(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y), fmaf(a.z, b.z, c.z));
}
__device__ __forceinline__ float dot3(float3 a, float3 b) {
  return fmaf(a.z, b.z, fmaf(a.x, b.x, __fmul_rn(a.y, b.y)));
}
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
  return f3(fmaf(a.y, b.z, -__fmul_rn(a.z, b.y)), fmaf(a.z, b.x, -__fmul_rn(a.x, b.z)),
            fmaf(a.x, b.y, -__fmul_rn(a.y, b.x)));
}
__device__ __forceinline__ float max3(float3 a) { return fmaxf(a.x, fmaxf(a.y, a.z)); }
__device__ __forceinline__ bool is_zero3(float3 a) { return a.x == 0.f && a.y == 0.f && a.z == 0.f; }

// dot3 with the first product unfused instead of the second.
__device__ __forceinline__ float dot3p(float3 a, float3 b) { return fmaf(a.z, b.z, fmaf(a.y, b.y, __fmul_rn(a.x, b.x))); }

// The hit tests' own forms (dot3p fuses in another order than dot3).
__device__ __forceinline__ float3 sub3p(float3 a, float3 b) { return a - b; }
__device__ __forceinline__ float3 add3p(float3 a, float3 b) { return a + b; }
__device__ __forceinline__ float3 cross3p(float3 a, float3 b) { return cross3(a, b); }

// Normalise (pinned rounding), or return `fallback` for (near-)zero or non-finite input.
__device__ __forceinline__ float3 unit_or(float3 v, float3 fallback) {
  const float l2 = dot3p(v, v);
  if (!(l2 > 1e-30f) || !isfinite(l2)) return fallback;
  const float s = rsqrtf(l2);
  return f3(__fmul_rn(v.x, s), __fmul_rn(v.y, s), __fmul_rn(v.z, s));
}

__device__ __forceinline__ float3 reflect3(float3 v, float3 n) { return mad3(-__fmul_rn(2.f, dot3(v, n)), n, v); }

// Snell refraction of unit `v` through unit `n` (facing against v), eta = n_i / n_t.
__device__ __forceinline__ bool refract3(float3 v, float3 n, float eta, float3& out) {
  const float cos_i = fminf(-dot3(v, n), 1.f);
  const float sin2_t = __fmul_rn(__fmul_rn(eta, eta), fmaf(-cos_i, cos_i, 1.f));
  if (sin2_t > 1.f) return false;
  const float cos_t = sqrtf(__fsub_rn(1.f, sin2_t));
  out = mad3(eta, v, fmaf(eta, cos_i, -cos_t) * n);
  return true;
}

__device__ __forceinline__ float schlick(float cos_theta, float eta) {
  float r0 = __fsub_rn(1.f, eta) / __fadd_rn(1.f, eta);
  r0 = __fmul_rn(r0, r0);
  const float m = __fsub_rn(1.f, cos_theta);
  const float m2 = __fmul_rn(m, m);
  return fmaf(__fsub_rn(1.f, r0), __fmul_rn(__fmul_rn(m2, m2), m), r0);
}

// ---------------------------------------------------------------------------
// PCG32 stream keyed on (seed, pixel, sample)
__host__ __device__ __forceinline__ std::uint64_t mix64(std::uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

struct Pcg {
  std::uint64_t state, inc;

  __device__ __forceinline__ std::uint32_t next() {
    const std::uint64_t old = state;
    state = old * 6364136223846793005ull + inc;
    const std::uint32_t x = static_cast<std::uint32_t>(((old >> 18u) ^ old) >> 27u);
    const std::uint32_t r = static_cast<std::uint32_t>(old >> 59u);
    return __funnelshift_r(x, x, r);  // rotate right by r
  }
  // Uniform in [0, 1) from the top 24 bits of one draw.
  __device__ __forceinline__ float uniform() { return __fmul_rn(static_cast<float>(next() >> 8), 0x1p-24f); }
  // Uniform integer in [0, n): floor(u32 * n / 2^32), which equals the CPU's
  // floor(double(u32) / 2^32 * n) exactly for n < 2^21.
  __device__ __forceinline__ std::uint32_t below(std::uint32_t n) {
    return static_cast<std::uint32_t>((static_cast<std::uint64_t>(next()) * n) >> 32);
  }

  __device__ static __forceinline__ Pcg seeded(std::uint64_t seed, std::uint64_t stream) {
    Pcg p{0, (stream << 1u) | 1u};
    p.next();
    p.state += seed;
    p.next();
    return p;
  }
  __device__ static __forceinline__ Pcg for_sample(std::uint64_t seed, std::uint64_t pixel, std::uint64_t sample) {
    const std::uint64_t h = mix64(seed ^ mix64(pixel ^ mix64(sample)));
    return seeded(h, mix64(h));
  }
};

// ---------------------------------------------------------------------------
// Sampling (each follows the matching reference routine and draw order,
// include/raytracer/math/sampling.hpp:13-78).
__device__ __forceinline__ float2 unit_disk(Pcg& rng) {
  const float r = sqrtf(rng.uniform());
  float s, c;
  sincospif(2.f * rng.uniform(), &s, &c);
  return make_float2(__fmul_rn(r, c), __fmul_rn(r, s));
}

__device__ __forceinline__ float3 unit_vector(Pcg& rng) {
  const float z = fmaf(-2.f, rng.uniform(), 1.f);
  const float r = sqrtf(fmaxf(0.f, fmaf(-z, z, 1.f)));
  float s, c;
  sincospif(2.f * rng.uniform(), &s, &c);
  return f3(__fmul_rn(r, c), __fmul_rn(r, s), z);
}

__device__ __forceinline__ float3 cosine_hemisphere(Pcg& rng) {
  const float2 d = unit_disk(rng);
  return f3(d.x, d.y, sqrtf(fmaxf(0.f, fmaf(-d.y, d.y, fmaf(-d.x, d.x, 1.f)))));
}

// Uniform direction in the cone 1 - cos(theta) <= one_minus_cos_max around +Z.
// Written in terms of 1 - cos so narrow cones keep their precision in fp32.
__device__ __forceinline__ float3 uniform_cone(Pcg& rng, float one_minus_cos_max) {
  const float s = __fmul_rn(rng.uniform(), one_minus_cos_max);  // 1 - cos(theta)
  const float cos_t = __fsub_rn(1.f, s);
  const float sin_t = sqrtf(fmaxf(0.f, __fmul_rn(s, __fsub_rn(2.f, s))));
  float sp, cp;
  sincospif(2.f * rng.uniform(), &sp, &cp);
  return f3(__fmul_rn(sin_t, cp), __fmul_rn(sin_t, sp), cos_t);
}

// Uniform barycentrics (b1, b2) on a triangle (square-root parameterisation).
__device__ __forceinline__ float2 uniform_triangle(Pcg& rng) {
  const float su = sqrtf(rng.uniform());
  return make_float2(__fsub_rn(1.f, su), __fmul_rn(rng.uniform(), su));
}

// Orthonormal basis around unit w (Duff et al. 2017, "Building an Orthonormal
// Basis, Revisited", JCGT 6(1)).
struct Frame {
  float3 u, v, w;
  __device__ __forceinline__ explicit Frame(float3 n) : w(n) {
    const float sign = copysignf(1.f, n.z);
    const float a = -1.f / __fadd_rn(sign, n.z);
    const float b = __fmul_rn(__fmul_rn(n.x, n.y), a);
    u = f3(fmaf(__fmul_rn(__fmul_rn(sign, n.x), n.x), a, 1.f), __fmul_rn(sign, b), __fmul_rn(-sign, n.x));
    v = f3(b, fmaf(__fmul_rn(n.y, n.y), a, sign), -n.y);
  }
  __device__ __forceinline__ float3 to_world(float3 a) const { return f3(fmaf(a.z, w.x, fmaf(a.y, v.x, __fmul_rn(a.x, u.x))), fmaf(a.z, w.y, fmaf(a.y, v.y, __fmul_rn(a.x, u.y))),
              fmaf(a.z, w.z, fmaf(a.x, u.z, __fmul_rn(a.y, v.z)))); }
};

// ---------------------------------------------------------------------------
// Robust spawn point: move p off the surface along n (which must point to the
// side the new ray leaves towards) by a fixed number of float ulps, or by a
// small absolute amount near the origin. Wächter and Binder, "A Fast and Robust
// Method for Avoiding Self-Intersection", Ray Tracing Gems (2019), ch. 6. The
// fp32 replacement for the reference's 1.6e-6 * max(1, |p|) offset
// (include/raytracer/math/ray.hpp:41-58), which is below an fp32 ulp at the
// 555-unit scale of a Cornell room.
__device__ __forceinline__ float ulp_step(float p, float n, float scaled_n) {
  const int step = static_cast<int>(__fmul_rn(256.f, n));
  const float moved = __int_as_float(__float_as_int(p) + (p < 0.f ? -step : step));
  return fabsf(p) < (1.f / 32.f) ? __fadd_rn(p, scaled_n) : moved;
}
__device__ __forceinline__ float3 spawn_point(float3 p, float3 n) {
  constexpr float kNearScale = 1.f / 65536.f;
  const float3 near = kNearScale * n;  // exact: a power of two
  return f3(ulp_step(p.x, n.x, near.x), ulp_step(p.y, n.y, near.y), ulp_step(p.z, n.z, near.z));
}
// Whether direction `dir` leaves a surface with geometric normal `gn` on that side. dot3p:
// one in the surface's plane (total reflection's edge) leaves on the side that this form's
// rounding says, as it always has.
__device__ __forceinline__ bool leaves_outside(float3 gn, float3 dir) { return dot3p(dir, gn) > 0.f; }
// Spawn for direction `dir` from there.
__device__ __forceinline__ float3 spawn_towards(float3 p, float3 gn, float3 dir) {
  return spawn_point(p, leaves_outside(gn, dir) ? gn : -gn);
}

// The reference's shadow-ray shortening distance is 4 * 1.6e-6 * max(1, |p|inf)
// (src/rendering/integrator.cpp:69-70), ~100 fp32 ulps of |p|: kShadowMargin times this.
constexpr float kShadowMargin = 4.f * 1.6e-6f;
__device__ __forceinline__ float shadow_scale(float3 p) {
  const float m = fmaxf(fmaxf(fabsf(p.x), fabsf(p.y)), fmaxf(fabsf(p.z), 1.f));
  return m;
}

}  // namespace rtg
