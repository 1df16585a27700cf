// Reconstruction coefficients (PLM, PPM, PQM) and their integrals in plain
// single precision: the fused arithmetic of the acceleration and translation
// remaps.
#pragma once

namespace vlgpu {

// m >= 0 with the sign of a.
__device__ __forceinline__ float with_sign(float m, float a) {
   return __uint_as_float(__float_as_uint(m) | (__float_as_uint(a) & 0x80000000u));
}

// h8 face value and h7 face derivative of the left face of the cell whose
// stencil is w0..w7 = values k-4 .. k+3 (cpu_face_estimates.hpp:45-79).
__device__ __forceinline__ float h8_value(float w0, float w1, float w2, float w3, float w4, float w5, float w6,
                                          float w7) {
   return (float)(1.0 / 840.0) *
          (533.0f * (w3 + w4) - 139.0f * (w2 + w5) + 29.0f * (w1 + w6) - 3.0f * (w0 + w7));
}
__device__ __forceinline__ float h7_derivative(float w0, float w1, float w2, float w3, float w4, float w5, float w6,
                                               float w7) {
   return (float)(1.0 / 5040.0) *
          (7175.0f * (w4 - w3) - 889.0f * (w5 - w2) + 119.0f * (w6 - w1) - 9.0f * (w7 - w0));
}

// PQM coefficients (compute_pqm_coeff, cpu_1d_pqm.hpp:157-176) from the raw
// h8/h7 faces: the extremum / boundedness / slope filters of
// compute_filtered_face_values_derivatives (cpu_face_estimates.hpp:216-275)
// and the inflexion-point filter filter_pqm_monotonicity (cpu_1d_pqm.hpp:
// 31-156), in single precision.
//
// The faces enter as their distances from the cell's value, L = v0 - left and
// R = right - v0: the combinations of v0 and the faces in the reference's
// formulas cancel v0 exactly, so each is two products instead of three, without
// the rounding of 60 v0 and 360 v0.  The reconstruction's slope is a cubic with
// the Bernstein coefficients fd_l, fd_l + b0/3, fd_l + 2 b0/3 + b1/6, fd_r on
// the cell; where none opposes the cell's slope, neither does the slope at an
// inflexion point, and the roots (a square root and two quotients) are not
// needed.  Where they are, they are rounded ones: three sweeps of 256 cells with
// packing take 793 us, 750 with approximate ones (of which only the slope's sign
// is read: the error against 64-bit sweeps is the same 9.4e-6 of the peak), 1675
// with v0 in every product and the roots taken in every cell.
__device__ __forceinline__ void pqm_coeff_fused(float vm1, float v0, float vp1, float fv_l, float fv_r, float fd_l,
                                                float fd_r, float a[5]) {
   const float dr = vp1 - v0, dl = v0 - vm1;
   const bool same = dr * dl > 0.0f;
   const float adr = fabsf(dr), adl = fabsf(dl);
   const float slope = same ? copysignf(fminf(2.0f * fminf(adr, adl), fmaxf(adr, adl)), dr) : 0.0f;
   float L = v0 - fv_l, R = fv_r - v0;
   // a face outside the values of its two cells, or a derivative against the slope
   const float sign = with_sign(1.0f, slope);
   if (L * (dl - L) < 0.0f || sign * fd_l < 0.0f) {
      L = 0.5f * slope;
      fd_l = slope;
   }
   if (R * (dr - R) < 0.0f || sign * fd_r < 0.0f) {
      R = 0.5f * slope;
      fd_r = slope;
   }
   if (slope == 0.0f) L = R = fd_l = fd_r = 0.0f;
   // second-derivative coefficients (White and Adcroft 2008, eq. 23)
   const float d = R - L, e = fd_r - fd_l;
   const float b0 = fmaf(3.0f, fd_r, fmaf(-9.0f, fd_l, fmaf(36.0f, L, -24.0f * R)));
   const float b1 = fmaf(-24.0f, fd_r, fmaf(36.0f, fd_l, fmaf(168.0f, R, -192.0f * L)));
   const float third = (float)(1.0 / 3.0);
   const float s1 = fmaf(b0, third, fd_l), s2 = fmaf(b1, (float)(1.0 / 6.0), fmaf(b0, 2.0f * third, fd_l));
   if (fminf(sign * s1, sign * s2) < 0.0f) {
      const float b2 = fmaf(30.0f, e, -180.0f * d);
      const float disc = fmaf(b1, b1, -4.0f * b0 * b2);
      const float sq = disc < 0.0f ? b1 + 200.0f * b2 : sqrtf(disc);
      const float c2 = 0.5f * b1, c3 = b2 * third;
      float against = 0.0f;  // the lower of the slopes (times sign) at the roots on the cell
#pragma unroll 1
      for (int q = 0; q < 2; ++q) {
         const float root = ((q ? -sq : sq) - b1) / (2.0f * b2);
         const float at = sign * fmaf(root, fmaf(root, fmaf(root, c3, c2), b0), fd_l);
         if (root >= 0.0f && root <= 1.0f) against = fminf(against, at);
      }
      if (against < 0.0f) {
         if (adl <= adr) {
            // collapse to the left edge (eq. 21), then the PLM-slope checks (eqs. 28, 29)
            fd_l = third * fmaf(8.0f, L, -2.0f * R);
            fd_r = fmaf(6.0f, R, -4.0f * L);
            if (sign * fd_l < 0.0f) {
               fd_l = 0.0f;
               R = 4.0f * L;
               fd_r = 20.0f * L;
            } else if (sign * fd_r < 0.0f) {
               fd_r = 0.0f;
               L = 1.5f * R;
               fd_l = (float)(10.0 / 3.0) * R;
            }
         } else {
            fd_l = fmaf(6.0f, L, -4.0f * R);
            fd_r = third * fmaf(8.0f, R, -2.0f * L);
            if (sign * fd_l < 0.0f) {
               fd_l = 0.0f;
               R = 1.5f * L;
               fd_r = (float)(10.0 / 3.0) * L;
            } else if (sign * fd_r < 0.0f) {
               fd_r = 0.0f;
               L = 4.0f * R;
               fd_l = 20.0f * R;
            }
         }
      }
   }
   a[0] = v0 - L;
   a[1] = 0.5f * fd_l;
   a[2] = fmaf(0.5f, fd_r, fmaf(-1.5f, fd_l, fmaf(6.0f, L, -4.0f * R)));
   a[3] = fmaf(1.5f, fd_l, fmaf(7.0f, R, -8.0f * L)) - fd_r;
   a[4] = fmaf(0.5f, fd_r - fd_l, 3.0f * (L - R));
}

// Reconstruction orders of the acceleration remap (the reference's
// ACC_SEMILAG_PLM / _PPM / _PQM).
constexpr int RECON_PLM = 1, RECON_PPM = 2, RECON_PQM = 4;

// Integral of the quartic reconstruction from 0 to u (cpu_acc_map.cpp:590-601),
// Horner form with FMA.
__device__ __forceinline__ float pqm_integral(float u, const float a[5]) {
   return u * fmaf(u, fmaf(u, fmaf(u, fmaf(u, a[4], a[3]), a[2]), a[1]), a[0]);
}

// The h4 face of uniform cells, (-v_{-2} + 7 v_{-1} + 7 v_0 - v_1) / 12
// (cpu_face_estimates.hpp:160-167), and PPM for two columns at once, with the
// packed single-precision operations of sm_100 (__fadd2_rn, __fmul2_rn, __ffma2_rn);
// the limiter's comparisons and selections stay per component.
__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }

__device__ __forceinline__ float2 h4_face_x2(float2 vm2, float2 vm1, float2 v0, float2 vp1) {
   return __ffma2_rn(__fadd2_rn(vm1, v0), f2((float)(7.0 / 12.0)),
                     __fmul2_rn(__fadd2_rn(vm2, vp1), f2((float)(-1.0 / 12.0))));
}

// y - x of two columns.
__device__ __forceinline__ float2 p_minus(float2 y, float2 x) { return __fadd2_rn(y, make_float2(-x.x, -x.y)); }

// a b > 0 of two value differences as a factor: their product times 2^150,
// saturated.  Where a b > 0 holds in single precision the product is 2^-149 at
// least, so the factor is 1; it is 0 at an extremum.  (A positive product that
// single precision loses, of differences below 1e-22, gives 1 or a fraction,
// where the comparison would flatten the cell.)
constexpr float SAME_SCALE = 37778931862957161709568.0f;

// Half the superbee slope of two columns, h = min(|a|, |b|, max(|a|, |b|) / 2)
// for the differences a, b to the right and left, and its sign s (zero at an
// extremum).
__device__ __forceinline__ void half_slope_x2(float2 a, float2 b, float2& h, float2& s) {
   const float2 aS = __fmul2_rn(a, f2(SAME_SCALE)), bS = __fmul2_rn(b, f2(SAME_SCALE));
   s = make_float2(with_sign(__saturatef(aS.x * bS.x), a.x), with_sign(__saturatef(aS.y * bS.y), a.y));
   const float2 mx =
      __fmul2_rn(make_float2(fmaxf(fabsf(a.x), fabsf(b.x)), fmaxf(fabsf(a.y), fabsf(b.y))), f2(0.5f));
   h = make_float2(fminf(fminf(fabsf(a.x), fabsf(b.x)), mx.x), fminf(fminf(fabsf(a.y), fabsf(b.y)), mx.y));
}

// What a walk along the cells carries from one cell to the next: v - left
// face, whether that face lies outside the values of its two cells, and the
// difference to the cell below.
struct PpmWalk {
   float2 left, b;
   bool out_x, out_y;
   // before the cell v0 with the cells vm2, vm1 below it and vp1 above
   __device__ __forceinline__ void start(float2 vm2, float2 vm1, float2 v0, float2 vp1) {
      const float2 face = h4_face_x2(vm2, vm1, v0, vp1);
      left = p_minus(v0, face);
      b = p_minus(v0, vm1);
      const float2 t = __fmul2_rn(p_minus(face, vm1), left);
      out_x = !(t.x >= 0.0f);
      out_y = !(t.y >= 0.0f);
   }
};

// PPM of two columns in magnitudes (cpu_1d_ppm.hpp:35-54): l = |v0 - left
// face|, r = |right face - v0| after the limiters; with the slope's sign s the
// integral of the reconstruction from 0 to u is u (v0 + s (u-1) (l + u (r-l))).
// A face outside its two cells' values (or one that is not a number, next to a
// value that is not) gives half the superbee slope instead;
// the Colella-Woodward corrections are l = min(l, 2r), r = min(r, 2l), of
// which at most one acts; at an extremum s = 0 flattens the cell.
__device__ __forceinline__ void ppm_magnitudes_x2(PpmWalk& c, float2 vm1, float2 v0, float2 vp1, float2 vp2, float2& s,
                                                  float2& l, float2& r) {
   const float2 a = p_minus(vp1, v0);
   float2 h;
   half_slope_x2(a, c.b, h, s);
   const float2 fr = h4_face_x2(vm1, v0, vp1, vp2);
   const float2 right = p_minus(fr, v0), next = p_minus(vp1, fr);
   const float2 t = __fmul2_rn(right, next);
   const bool or_x = !(t.x >= 0.0f), or_y = !(t.y >= 0.0f);
   const float2 lf = make_float2(c.out_x ? h.x : c.left.x, c.out_y ? h.y : c.left.y);
   const float2 rf = make_float2(or_x ? h.x : right.x, or_y ? h.y : right.y);
   const float2 l2 = __fmul2_rn(lf, f2(2.0f)), r2 = __fmul2_rn(rf, f2(2.0f));
   l = make_float2(fminf(fabsf(lf.x), fabsf(r2.x)), fminf(fabsf(lf.y), fabsf(r2.y)));
   r = make_float2(fminf(fabsf(rf.x), fabsf(l2.x)), fminf(fabsf(rf.y), fabsf(l2.y)));
   c.left = next;
   c.b = a;
   c.out_x = or_x;
   c.out_y = or_y;
}

}  // namespace vlgpu
