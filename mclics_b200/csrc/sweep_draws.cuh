// What the sweeps on pairs of sites share (colour passes, resident sweep): the draws of a pair, its raw
// moments and their sums over a warp.
#pragma once
#include "common.cuh"
#include "physics.cuh"

namespace mcl {

// Lane values of a pair draw (one Philox block for sites x and x + 2, non-flip models), bit-identical to
// lane_draw(pair_half(out, 0), pair_half(out, 1), false).
__device__ __forceinline__ float unit21_bits(uint32_t bits_shifted, uint32_t exponent) {
  return __uint_as_float(exponent | (bits_shifted & 0x7FFFFCu));
}
__device__ __forceinline__ LaneDraw<float2> pair_draw_lanes(const U4 &o) {
  LaneDraw<float2> r;
  // u1 (angle field, bits 0..20 of lo): 2 u1 - 1 is used; keep u1 itself exact as (1 + f 2^-21) - 1
  r.u1 = __fadd2_rn(make_float2(unit21_bits(o.x << 2, 0x3F800000u), unit21_bits(o.z << 2, 0x3F800000u)),
                    make_float2(-1.f, -1.f));
  // u3 (acceptance field, bits 10..30 of hi)
  r.u3 = __fadd2_rn(make_float2(unit21_bits(o.y >> 8, 0x3F800000u), unit21_bits(o.w >> 8, 0x3F800000u)),
                    make_float2(-1.f, -1.f));
  r.u4 = make_float2(0.f, 0.f);
  // axis field: bits 21..41 of the 64-bit half (lo, hi)
  const uint32_t f0 = __funnelshift_r(o.x, o.y, 21) & 0x1FFFFFu, f1 = __funnelshift_r(o.z, o.w, 21) & 0x1FFFFFu;
  r.w0 = make_float2(f0 < 698352u ? 1.f : 0.f, f1 < 698352u ? 1.f : 0.f);
  r.w2 = make_float2(f0 >= 1396704u ? 1.f : 0.f, f1 >= 1396704u ? 1.f : 0.f);
  r.w1 = make_float2(1.f - r.w0.x - r.w2.x, 1.f - r.w0.y - r.w2.y);
  return r;
}

// Draws of the sites x and x + 2 with counter ctr (linear index of x; ctr + 2 for x + 2 in flip models).
template <bool FLIP>
__device__ __forceinline__ LaneDraw<float2> pair_draws(unsigned long long seed, unsigned long long sweep, uint32_t ctr) {
  if (FLIP) {
    const U4 u0 = site_draws(seed, sweep, ctr, 0), u1 = site_draws(seed, sweep, ctr + 2, 0);
    return lane_draw(Draw{u0.x >> 8, u0.y >> 8, u0.z >> 8, u0.w >> 8}, Draw{u1.x >> 8, u1.y >> 8, u1.z >> 8, u1.w >> 8},
                     true);
  }
  return pair_draw_lanes(site_draws(seed, sweep, ctr, 0));
}

// Raw moments of two pairs of sites (lanes paired): m[0..5] = sum v_a v_b (xx, xy, xz, yy, yz, zz), m[6..8] = sum v.
// Q and sum n follow per thread at the end: sum q_ab = 1.5 sum v_a v_b - 0.5 delta_ab (sites).
__device__ __forceinline__ void pair_moments(float2 (&m)[9], const float2 (&u)[3], const float2 (&v)[3]) {
  m[0] = __ffma2_rn(v[0], v[0], __fmul2_rn(u[0], u[0]));
  m[1] = __ffma2_rn(v[0], v[1], __fmul2_rn(u[0], u[1]));
  m[2] = __ffma2_rn(v[0], v[2], __fmul2_rn(u[0], u[2]));
  m[3] = __ffma2_rn(v[1], v[1], __fmul2_rn(u[1], u[1]));
  m[4] = __ffma2_rn(v[1], v[2], __fmul2_rn(u[1], u[2]));
  m[5] = __ffma2_rn(v[2], v[2], __fmul2_rn(u[2], u[2]));
  m[6] = __fadd2_rn(u[0], v[0]);
  m[7] = __fadd2_rn(u[1], v[1]);
  m[8] = __fadd2_rn(u[2], v[2]);
}

// Sums of ten values over a warp: the halves of the warp split the values between them at every step (12 double
// shuffles instead of 50). The lane that holds value k afterwards returns k, the others -1.
__device__ __forceinline__ int warp_sum10(const double (&v)[kPartials], double &out) {
  const int lane = threadIdx.x & 31;
  const bool b16 = lane & 16, b8 = lane & 8, b4 = lane & 4, b2 = lane & 2;
  double a[6], b[4], c[2];
#pragma unroll
  for (int i = 0; i < 5; i++) a[i] = (b16 ? v[5 + i] : v[i]) + __shfl_xor_sync(0xffffffffu, b16 ? v[i] : v[5 + i], 16);
  a[5] = 0.0;
#pragma unroll
  for (int i = 0; i < 3; i++) b[i] = (b8 ? a[3 + i] : a[i]) + __shfl_xor_sync(0xffffffffu, b8 ? a[i] : a[3 + i], 8);
  b[3] = 0.0;
#pragma unroll
  for (int i = 0; i < 2; i++) c[i] = (b4 ? b[2 + i] : b[i]) + __shfl_xor_sync(0xffffffffu, b4 ? b[i] : b[2 + i], 4);
  double d = (b2 ? c[1] : c[0]) + __shfl_xor_sync(0xffffffffu, b2 ? c[0] : c[1], 2);
  out = d + __shfl_xor_sync(0xffffffffu, d, 1);
  const int in4 = (b4 ? 2 : 0) + (b2 ? 1 : 0), in8 = (b8 ? 3 : 0) + in4;
  return (lane & 1) == 0 && in4 < 3 && in8 < 5 ? (b16 ? 5 : 0) + in8 : -1;
}

}  // namespace mcl
