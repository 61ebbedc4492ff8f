// hb_compat.cu -- the reference's torch-extension op surface as C-ABI entry
// points over caller-owned device arrays, for FP32 and FP64.
//
// Same compacted-cell layout, neighbour table and in-place semantics as the
// reference ops (paths relative to CHANS-HiPIMS/hipims/cuda):
//   hb_flux             fluxCal_2ndOrder_jh_improved.cpp:28-53  (order 2)
//                       fluxCal_jh_modified_surface.cpp:28-53   (order 1)
//   hb_friction_update  friction_implicit_andUpdate_jh_interface.cpp:29-53
//   hb_timestep         timeControl.cpp:27-41
//   hb_rain_station     stationPrecipitation_interface.cpp:26-38
//   hb_flux_mask        fluxMaskGenerator.cpp:22-29
//   hb_euler_update     euler_update.cpp:27-44
//   hb_infiltration     infiltration_interface.cpp (Green-Ampt)
// This file is compiled with -fmad=false so that FP64 results follow the
// reference's operation order without contraction.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "hb_common.cuh"
#include "hb_physics.cuh"

namespace hb {
namespace {

constexpr int kThreads = 256;

template <typename T>
__device__ __forceinline__ Cell<T> load_cell(const T *__restrict__ h,
                                             const T *__restrict__ wl,
                                             const T *__restrict__ qx,
                                             const T *__restrict__ qy,
                                             const T *__restrict__ z, int64_t i) {
  Cell<T> c;
  c.h = __ldg(h + i);
  c.wl = __ldg(wl + i);
  c.qx = __ldg(qx + i);
  c.qy = __ldg(qy + i);
  c.z = __ldg(z + i);
  return c;
}

// What every face of a call reads: the state, the neighbour table and the
// boundary rows at t.
template <typename T>
struct FluxArgs {
  int64_t N;
  const T *h, *wl, *z, *qx, *qy;
  const int32_t *index;
  const T *gd, *gw, *gq;  // the tables' rows at t
  int dc, wc, qc;
  T dx, dt;
};
template <typename T>
struct FluxSum {
  T h, qx, qy;
};

template <typename T>
__device__ __forceinline__ Cell<T> cell_at(const FluxArgs<T> &a, int64_t i) {
  return load_cell(a.h, a.wl, a.qx, a.qy, a.z, i);
}

// Ghost of cell c across a missing neighbour.
template <typename T, int ORDER>
__device__ __forceinline__ bool flux_ghost(const FluxArgs<T> &a, int32_t c_type, const Cell<T> &c,
                                           T n0, T n1, Cell<T> &r) {
  int bt, bid;
  decode_bc(c_type, bt, bid);
  // Table columns beyond the given width read as 0 (the reference reads
  // past the row there).
  const T hb = bid + 1 < a.dc ? a.gd[bid + 1] : T(0);
  const T wlb = bid + 1 < a.wc ? a.gw[bid + 1] : T(0);
  const T qxb = 2 + 2 * bid < a.qc ? a.gq[1 + 2 * bid] : T(0);
  const T qyb = 2 + 2 * bid < a.qc ? a.gq[2 + 2 * bid] : T(0);
  return ghost(bt, ORDER == 1, c, n0, n1, hb, wlb, qxb, qyb, r);
}

// One face of cell i along an arbitrary normal, operation for operation as the
// reference: faces of unusual normals, and faces with a non-finite quotient.
template <typename T, int ORDER>
__device__ __noinline__ FluxSum<T> flux_face_plain(const FluxArgs<T> &a, int32_t i, int j, T n0,
                                                   T n1, FluxSum<T> f) {
  const T hs = T(kHSmall), g = T(kG), dx = a.dx, dt = a.dt;
  Cell<T> c = cell_at(a, i);
  const T t0 = -n1, t1 = n0;
  const int rdir = j + 1;
  const int ldir = (rdir + 2) > 4 ? rdir - 2 : rdir + 2;
  const int32_t l_id = a.index[(int64_t)ldir * a.N + i];
  const int32_t r_id = a.index[(int64_t)rdir * a.N + i];
  Cell<T> r, eL, eR;
  T c_h = c.h, c_z = c.z;  // raw cell values for the 1st-order scheme
  T r_h = T(0), r_z = T(0);
  if (r_id == -1) {
    if (!flux_ghost<T, ORDER>(a, a.index[i], c, n0, n1, r)) return f;
    r_h = r.h;
    r_z = r.z;
    eL = c;
    eR = r;
  } else if (ORDER == 2) {
    Cell<T> l = (l_id == -1) ? c : cell_at(a, l_id);
    const int32_t rr_id = a.index[(int64_t)rdir * a.N + r_id];
    r = cell_at(a, r_id);
    Cell<T> rr = (rr_id == -1) ? r : cell_at(a, rr_id);
    muscl(c, l, r, eL);
    muscl(r, rr, c, eR);
  } else {
    const T l_z = (l_id == -1) ? c.z : __ldg(a.z + l_id);
    const int32_t rr_id = a.index[(int64_t)rdir * a.N + r_id];
    const T rr_z = (rr_id == -1) ? __ldg(a.z + r_id) : __ldg(a.z + rr_id);
    r = cell_at(a, r_id);
    r_h = r.h;
    r_z = r.z;
    T rb = minmod(c.z - l_z, r.z - c.z);
    if (r.h > hs) c.z += T(0.5) * rb;
    rb = minmod(r.z - rr_z, c_z - r.z);
    if (c.h > hs) r.z += T(0.5) * rb;
    eL = c;
    eR = r;
  }
  if (c.h < hs && r.h < hs) return f;
  // velocities of the edge states before the hydrostatic step
  const T ux_l = eL.h < hs ? T(0) : eL.qx / eL.h;
  const T uy_l = eL.h < hs ? T(0) : eL.qy / eL.h;
  const T ux_r = eR.h < hs ? T(0) : eR.qx / eR.h;
  const T uy_r = eR.h < hs ? T(0) : eR.qy / eR.h;
  if (ORDER == 2)
    hydro2(c.wl, r.wl, eL, eR);
  else
    hydro1(c_h, c_z, r_h, r_z, eL, eR);
  const T u_L = ux_l * n0 + uy_l * n1;
  const T u_R = ux_r * n0 + uy_r * n1;
  const T v_L = -ux_l * n1 + uy_l * n0;
  const T v_R = -ux_r * n1 + uy_r * n0;
  T Fh, Fn, Ft;
  if (hllc<T, false>(eL.h, eR.h, u_L, u_R, v_L, v_R, Fh, Fn, Ft)) {
    f.h -= (Fh / dx) * dt;
    f.qx -= ((Fn * n0 + Ft * t0) / dx) * dt;
    f.qy -= ((Fn * n1 + Ft * t1) / dx) * dt;
  }
  if (ORDER == 2) {
    f.qx -= ((T(0.5) * g * (c.h + eL.h) * (eL.z - c.z) * n0) / dx) * dt;
    f.qy -= ((T(0.5) * g * (c.h + eL.h) * (eL.z - c.z) * n1) / dx) * dt;
  } else {
    f.qx -= ((T(0.5) * g * (eL.h + c_h) * (eL.z - c_z) * n0) / dx) * dt;
    f.qy -= ((T(0.5) * g * (eL.h + c_h) * (eL.z - c_z) * n1) / dx) * dt;
  }
  return f;
}

// a / b, correctly rounded, from y = RN(1 / b): q = RN(a y), remainder a - b q
// (exact in one FMA) times y added back (Markstein's theorem; finite operands,
// no underflow).  A face takes nine quotients by four divisors.  `rest` gathers
// the remainders: it is not finite if an operand was not.
__device__ __forceinline__ double recip(double b) { return __drcp_rn(b); }
__device__ __forceinline__ float recip(float b) { return __frcp_rn(b); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
template <typename T>
__device__ __forceinline__ T quot(T a, T b, T y, T &rest) {
  const T q = a * y;
  const T r = fma_rn(-q, b, a);
  rest += r;
  return fma_rn(r, y, q);
}

// hllc<T, false> with the quotients above and the contact speed's sign read off
// its numerator and denominator (only the sign is used).
template <typename T>
__device__ __forceinline__ bool hllc_q(T hL, T hR, T u_L, T u_R, T v_L, T v_R, T &fh, T &fn,
                                       T &ft, T &rest) {
  const T hs = T(kHSmall), g = T(kG);
  if (hL < hs && hR < hs) return false;
  const T qx_L = u_L * hL, qx_R = u_R * hR;
  const T a_L = sqrt(g * hL), a_R = sqrt(g * hR);
  const T base = (a_L + a_R) * T(0.5) + (u_L - u_R) * T(0.25);
  const T u_star = (u_L + u_R) * T(0.5) + a_L - a_R;
  const T h_star = quot(base * base, g, T(1) / g, rest);
  const T a_star = sqrt(g * h_star);
  const T s_L = hL <= hs ? u_R - T(2) * a_R : fmin(u_L - a_L, u_star - a_star);
  const T s_R = hR <= hs ? u_L + T(2) * a_L : fmax(u_R + a_R, u_star + a_star);
  const T h_flux_L = qx_L, h_flux_R = qx_R;
  const T qx_flux_L = u_L * qx_L + T(0.5) * g * hL * hL;
  const T qx_flux_R = u_R * qx_R + T(0.5) * g * hR * hR;
  if (T(0) <= s_L) {
    fh = h_flux_L;
    fn = qx_flux_L;
    ft = u_L * (v_L * hL);
    return true;
  }
  const T num = s_L * hR * (u_R - s_R) - s_R * hL * (u_L - s_L);
  const T den = hR * (u_R - s_R) - hL * (u_L - s_L);
  // s_M = num / den; den = 0 (NaN or infinite s_M) is left to the plain face
  const bool pos = num == T(0) || (num > T(0)) == (den > T(0));
  if (den == T(0)) rest = INFINITY;
  if (!(s_L < T(0)) || (!pos && !(T(0) <= s_R))) {
    fh = h_flux_R;
    fn = qx_flux_R;
    ft = u_R * (v_R * hR);
    return true;
  }
  const T ds = s_R - s_L, y = recip(ds);
  fh = quot(s_R * h_flux_L - s_L * h_flux_R + s_L * s_R * (hR - hL), ds, y, rest);
  fn = quot(s_R * qx_flux_L - s_L * qx_flux_R + s_L * s_R * (qx_R - qx_L), ds, y, rest);
  ft = fh * (pos ? v_L : v_R);
  return true;
}

// Face J (0 E, 1 N, 2 W, 3 S, normals (1, 0), (0, 1), (-1, 0), (0, -1); X: E or W)
// of cell i with its slope s along the axis (towards E / N), the same results as
// flux_face_plain: a product with a normal's zero is not formed, and quotients
// by a shared divisor share its reciprocal.
template <typename T, int ORDER, bool X>
__device__ __forceinline__ FluxSum<T> flux_face(const FluxArgs<T> &a, int32_t i, int J,
                                                int32_t r_id, const Cell<T> &c, const Cell<T> &s,
                                                T ydx, const FluxSum<T> f) {
  const T hs = T(kHSmall), g = T(kG);
  const T sgn = J < 2 ? T(1) : T(-1);
  const T n0 = X ? sgn : T(0), n1 = X ? T(0) : sgn;
  Cell<T> r, eL = c, eR;
  T r_h, r_z;
  if (r_id == -1) {
    if (!flux_ghost<T, ORDER>(a, a.index[i], c, n0, n1, r)) return f;
    r_h = r.h;
    r_z = r.z;
    eR = r;
  } else {
    const int32_t rr_id = a.index[(int64_t)(J + 1) * a.N + r_id];
    r = cell_at(a, r_id);
    r_h = r.h;
    r_z = r.z;
    if constexpr (ORDER == 2) {
      const int64_t k = rr_id == -1 ? r_id : rr_id;
      eL.h = c.h + T(0.5) * (sgn * s.h);
      eL.z = c.z + T(0.5) * (sgn * s.z);
      const bool dry = c.h < hs;
      eL.qx = dry ? T(0) : c.qx + T(0.5) * (sgn * s.qx);
      eL.qy = dry ? T(0) : c.qy + T(0.5) * (sgn * s.qy);
      Cell<T> rr;
      rr.h = __ldg(a.h + k);
      rr.z = __ldg(a.z + k);
      rr.qx = __ldg(a.qx + k);
      rr.qy = __ldg(a.qy + k);
      muscl(r, rr, c, eR);
    } else {
      const T rr_z = __ldg(a.z + (rr_id == -1 ? r_id : rr_id));
      eR = r;
      if (r.h > hs) eL.z = c.z + T(0.5) * (sgn * s.z);
      if (c.h > hs) eR.z = r.z + T(0.5) * minmod(r.z - rr_z, c.z - r.z);
    }
  }
  if (c.h < hs && r.h < hs) return f;
  T rest = T(0);
  const T yl = recip(eL.h), yr = recip(eR.h);
  const bool dl = eL.h < hs, dr = eR.h < hs;
  T restl = T(0), restr = T(0);
  T ux_l = quot(eL.qx, eL.h, yl, restl), uy_l = quot(eL.qy, eL.h, yl, restl);
  T ux_r = quot(eR.qx, eR.h, yr, restr), uy_r = quot(eR.qy, eR.h, yr, restr);
  if (dl) ux_l = uy_l = T(0); else rest += restl;
  if (dr) ux_r = uy_r = T(0); else rest += restr;
  if constexpr (ORDER == 2)
    hydro2(c.wl, r.wl, eL, eR);
  else
    hydro1(c.h, c.z, r_h, r_z, eL, eR);
  const T u_L = X ? sgn * ux_l : sgn * uy_l, u_R = X ? sgn * ux_r : sgn * uy_r;
  const T v_L = X ? sgn * uy_l : -sgn * ux_l, v_R = X ? sgn * uy_r : -sgn * ux_r;
  FluxSum<T> o = f;
  T Fh, Fn, Ft;
  if (hllc_q(eL.h, eR.h, u_L, u_R, v_L, v_R, Fh, Fn, Ft, rest)) {
    o.h -= quot(Fh, a.dx, ydx, rest) * a.dt;
    const T mn = quot(sgn * Fn, a.dx, ydx, rest) * a.dt;
    const T mt = quot(X ? sgn * Ft : -sgn * Ft, a.dx, ydx, rest) * a.dt;
    o.qx -= X ? mn : mt;
    o.qy -= X ? mt : mn;
  }
  const T bed = ORDER == 2 ? T(0.5) * g * (c.h + eL.h) * (eL.z - c.z)
                           : T(0.5) * g * (eL.h + c.h) * (eL.z - c.z);
  const T mb = quot(sgn * bed, a.dx, ydx, rest) * a.dt;
  if (X) o.qx -= mb; else o.qy -= mb;
  if (!(fabs(rest) < T(INFINITY)))  // an infinite or NaN operand
    return flux_face_plain<T, ORDER>(a, i, J, n0, n1, f);
  return o;
}

// Slope of c between minus-side id m and plus-side id p (missing: c itself).
// `rest` stays finite while the differences do (with a NaN among them minmod is
// not odd under a swap of the sides).
template <typename T>
__device__ __forceinline__ T slope_at(const T *__restrict__ x, T c, int32_t m, int32_t p,
                                      T &rest) {
  const T lo = m == -1 ? c : __ldg(x + m), up = p == -1 ? c : __ldg(x + p);
  const T d = c - lo, e = up - c;
  rest += d + e;
  return minmod(d, e);
}

// Per active cell, its four faces E, N, W, S in order; each face is computed
// from this cell's side (the reference's scheme), accumulating -dt/dx * F and
// the bed-slope source into the update arrays.  FP64 issue binds it, IEEE
// divisions above all (13 a face: 1300 of 3760 instructions a cell), so the
// cell's slopes are formed once per axis (minmod is odd under a swap of the
// sides) and the quotients share reciprocals; the results are those of the
// plain form bit for bit (quotients near or below the least normal number: to a
// few units of the least number).  1024^2 cells, 2nd / 1st order: FP64 169 / 149 -> 123 /
// 100 us, FP32 86 / 76 -> 74 / 62 us.  64 registers (8 blocks of 128) although
// FP64 spills: at 80 registers 129 / 108 us, without a cap (142) 180 us.
template <typename T, int ORDER>
__global__ void __launch_bounds__(128, 8)
flux_kernel(int64_t M, int64_t N, const int32_t *__restrict__ wet,
            T *__restrict__ h_flux, T *__restrict__ qx_flux, T *__restrict__ qy_flux,
            const T *__restrict__ h, const T *__restrict__ wl, const T *__restrict__ z,
            const T *__restrict__ qx, const T *__restrict__ qy,
            const int32_t *__restrict__ index, const T *__restrict__ normal,
            const T *__restrict__ gd, int dr, int dc, const T *__restrict__ gw, int wr,
            int wc, const T *__restrict__ gq, int qr, int qc, const T *__restrict__ dxp,
            const T *__restrict__ tp, const T *__restrict__ dtp) {
  int64_t w = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= M) return;
  const int32_t i = wet[w];
  const int32_t e = index[1 * N + i], n = index[2 * N + i], ww = index[3 * N + i],
                so = index[4 * N + i];
  const double t = (double)tp[0];
  FluxArgs<T> a{N, h, wl, z, qx, qy, index, gd, gw, gq, dc, wc, qc, dxp[0], dtp[0]};
  if ((e | n | ww | so) < 0) {  // a missing neighbour: the tables' rows
    a.gd = gd + (int64_t)timelevel(t, gd, dr, dc) * dc;
    a.gw = gw + (int64_t)timelevel(t, gw, wr, wc) * wc;
    a.gq = gq + (int64_t)timelevel(t, gq, qr, qc) * qc;
  }
  FluxSum<T> f{h_flux[i], qx_flux[i], qy_flux[i]};
  const bool axes = normal[0] == T(1) && normal[1] == T(0) && normal[2] == T(0) &&
                    normal[3] == T(1) && normal[4] == T(-1) && normal[5] == T(0) &&
                    normal[6] == T(0) && normal[7] == T(-1);
  const Cell<T> c = cell_at(a, i);
  Cell<T> sx, sy;
  T rest = T(0);
  sx.z = slope_at(z, c.z, ww, e, rest);
  sy.z = slope_at(z, c.z, so, n, rest);
  if constexpr (ORDER == 2) {
    sx.h = slope_at(h, c.h, ww, e, rest);
    sx.qx = slope_at(qx, c.qx, ww, e, rest);
    sx.qy = slope_at(qy, c.qy, ww, e, rest);
    sy.h = slope_at(h, c.h, so, n, rest);
    sy.qx = slope_at(qx, c.qx, so, n, rest);
    sy.qy = slope_at(qy, c.qy, so, n, rest);
  }
  if (axes && fabs(rest) < T(INFINITY)) {
    const T ydx = recip(a.dx);
#pragma unroll 1
    for (int j = 0; j < 4; j += 2) {
      f = flux_face<T, ORDER, true>(a, i, j, j ? ww : e, c, sx, ydx, f);
      f = flux_face<T, ORDER, false>(a, i, j + 1, j ? so : n, c, sy, ydx, f);
    }
  } else {
    for (int j = 0; j < 4; j++)
      f = flux_face_plain<T, ORDER>(a, i, j, normal[j * 2], normal[j * 2 + 1], f);
  }
  h_flux[i] = f.h;
  qx_flux[i] = f.qx;
  qy_flux[i] = f.qy;
}

// Implicit Manning friction + Euler update, zeroing the accumulators.  The
// reference kernel writes this step with double literals, so its FP32 build
// evaluates C_f and the implicit update in double; D below reproduces those
// promotions (for T = double it changes nothing).
template <typename T>
__global__ void __launch_bounds__(kThreads)
friction_update_kernel(int64_t M, const int32_t *__restrict__ wet, T *__restrict__ hu,
                       T *__restrict__ qxu, T *__restrict__ qyu, T *__restrict__ zu,
                       const uint8_t *__restrict__ landuse, T *__restrict__ hp,
                       T *__restrict__ wlp, T *__restrict__ qxp, T *__restrict__ qyp,
                       T *__restrict__ zp, const T *__restrict__ manning,
                       const T *__restrict__ dtp) {
  using D = double;
  int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  const T hs = T(kHSmall), g = T(kG), dt = dtp[0];
  const int32_t i = wet[j];
  T h = hp[i] + hu[i];
  T qx = qxp[i], qy = qyp[i];
  if (h < hs) {
    qx = T(0);
    qy = T(0);
  } else {
    const T n = manning[landuse[i]];
    const T C_f = (T)((D)(g * n * n) * pow((D)h, -1.0 / 3.0));
    qx += qxu[i];
    qy += qyu[i];
    const T q_norm = sqrt(qx * qx + qy * qy);
    const T h2 = h * h;
    const bool fx = fabs(qx) > T(1.0e-10), fy = fabs(qy) > T(1.0e-10);
    if (n > T(0) && (fx || fy)) {
      // shared by both components (a copy in each branch: 35.8 us for 1024^2
      // cells in FP64, 33.1 so, at 4.5 TB/s)
      const D lim = 5.0 * (D)h * (D)sqrt(h * g);
      const D top = 1.0 - sqrt(1.0 + (4.0 * (D)dt * (D)C_f) / (D)h2 * (D)q_norm);
      const D bot = -2.0 * (D)dt * (D)C_f / (D)h2;
      if (fx) {
        const D temp = top / (bot * (D)(q_norm / qx));
        if (fabs(temp) > lim) {
          qx = (T)(2.0 * temp - (D)qx);
          if ((D)qx * temp <= 0.0) qx = T(0);
        } else {
          qx = (T)temp;
        }
      }
      if (fy) {
        const D temp = top / (bot * (D)(q_norm / qy));
        if (fabs(temp) > lim) {
          qy = (T)(2.0 * temp - (D)qy);
          if ((D)qy * temp <= 0.0) qy = T(0);
        } else {
          qy = (T)temp;
        }
      }
    }
  }
  const T z = zp[i] + zu[i];
  hp[i] = h;
  qxp[i] = qx;
  qyp[i] = qy;
  zp[i] = z;
  wlp[i] = z + h;
  hu[i] = T(0);
  qxu[i] = T(0);
  qyu[i] = T(0);
  zu[i] = T(0);
}

// CFL acceleration per listed cell and running maximum depth.  sqrtf is
// single precision in the reference kernel for both dtypes.
template <typename T>
__global__ void __launch_bounds__(kThreads)
timestep_kernel(int64_t M, const int32_t *__restrict__ wet, T *__restrict__ accel,
                T *__restrict__ h_max, const T *__restrict__ h, const T *__restrict__ qx,
                const T *__restrict__ qy, const T *__restrict__ dxp,
                const T *__restrict__ cflp) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= M) return;
  const int32_t j = wet[i];
  const T hj = h[j];
  h_max[j] = fmax(hj, h_max[j]);
  const T g = T(kG);
  accel[i] = hj > T(kHSmall)
                 ? cflp[0] * dxp[0] /
                       ((T)sqrtf((float)(g * hj)) + fmax(fabs(qx[j]), fabs(qy[j])) / hj)
                 : T(60.0);
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
rain_station_kernel(int64_t N, T *__restrict__ hu, const int16_t *__restrict__ mask,
                    const T *__restrict__ data, const T *__restrict__ dtp) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N) hu[i] += data[mask[i]] * dtp[0];
}

// Neighbour ids are tested with `> 0` as in the reference, so cell 0 never
// activates its neighbours (HC/fluxMaskGenerator_Kernel.cu:36).
template <typename T>
__global__ void __launch_bounds__(kThreads)
flux_mask_kernel(int64_t N, uint8_t *__restrict__ out, const T *__restrict__ h,
                 const int32_t *__restrict__ index, const T *__restrict__ tp) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N) return;
  if (tp[0] == T(0)) {
    out[i] = 1;
    return;
  }
  const T hs = T(kHSmall);
  bool m = h[i] > hs;
#pragma unroll
  for (int nei = 1; nei < 5; nei++) {
    const int32_t k = index[(int64_t)nei * N + i];
    if (k > 0) m = m || (h[k] > hs);
  }
  out[i] = m ? 1 : 0;
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
euler_update_kernel(int64_t M, const int32_t *__restrict__ mask,
                    const T *__restrict__ hu, const T *__restrict__ qxu,
                    const T *__restrict__ qyu, const T *__restrict__ zu, T *__restrict__ h,
                    T *__restrict__ wl, T *__restrict__ z, T *__restrict__ qx,
                    T *__restrict__ qy) {
  int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  const int32_t i = mask[j];
  const T hh = h[i] + hu[i];
  const T zz = z[i] + zu[i];
  h[i] = hh;
  qx[i] = qx[i] + qxu[i];
  qy[i] = qy[i] + qyu[i];
  z[i] = zz;
  wl[i] = hh + zz;
}

template <typename T>
__global__ void __launch_bounds__(kThreads)
infiltration_kernel(int64_t M, const int32_t *__restrict__ wet, T *__restrict__ hu,
                    const uint8_t *__restrict__ landuse, const T *__restrict__ hp,
                    const T *__restrict__ ks, const T *__restrict__ psi,
                    const T *__restrict__ dth, T *__restrict__ cum,
                    const T *__restrict__ dtp) {
  int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= M) return;
  const int32_t i = wet[j];
  const uint8_t lt = landuse[i];
  const T h = hp[i], dt = dtp[0];
  const T K_s = ks[lt], phi_s = psi[lt], d = dth[lt];
  const T F_0 = cum[i];
  const T total_head = phi_s + h;
  const T F_1 = T(0.5) * (F_0 + dt * K_s +
                          sqrt((F_0 + dt * K_s) * (F_0 + dt * K_s) +
                               T(4) * dt * K_s * total_head * d));
  const T dF = fmin(h, F_1 - F_0);
  cum[i] += dF;
  hu[i] -= dF;
}

// Ordered list of the cells that pass a test, as torch.nonzero gives it, in two
// kernels: a block tests kListCells cells, keeps their bits and counts them;
// then each block adds up the counts before its own and writes its ids.  Bound
// by the reads of h (and the neighbour table); against the mask, its fill, the
// comparison kernels, the three kernels of nonzero and the cast to int32 it is
// two launches instead of nine: a step of the solver object on 256 x 300 cells
// (FP32, host-bound) 349 -> 279 us, 241 with the raw stream handle.
constexpr int kListCells = 4096, kListThreads = 256, kListWords = kListCells / 32;

// RULE 0: fluxMask (HC/fluxMaskGenerator_Kernel.cu:19-42; x = t); 1: the update
// list of HP/SWE_CUDA.py:786-790, |h_update| > 0 or h >= 0 (x = h_update).
template <typename T, int RULE>
__global__ void __launch_bounds__(kListThreads)
list_test_kernel(int64_t N, const T *__restrict__ h, const int32_t *__restrict__ index,
                 const T *__restrict__ x, uint32_t *__restrict__ words,
                 int32_t *__restrict__ counts) {
  __shared__ int s_n;
  if (threadIdx.x == 0) s_n = 0;
  __syncthreads();
  const T hs = T(kHSmall);
  const bool first = RULE == 0 && x[0] == T(0);
  int mine = 0;
#pragma unroll 4
  for (int k = 0; k < kListCells / kListThreads; k++) {
    const int64_t i = (int64_t)blockIdx.x * kListCells + k * kListThreads + threadIdx.x;
    bool m = false;
    if (i < N) {
      if constexpr (RULE == 0) {
        m = first || h[i] > hs;
        if (!m) {
#pragma unroll
          for (int nei = 1; nei < 5; nei++) {
            const int32_t q = index[(int64_t)nei * N + i];
            if (q > 0) m = m || (h[q] > hs);  // cell 0 never activates its neighbours
          }
        }
      } else {
        m = fabs(x[i]) > T(0) || h[i] >= T(0);
      }
    }
    const unsigned b = __ballot_sync(0xffffffffu, m);
    if ((threadIdx.x & 31) == 0) {
      words[(int64_t)blockIdx.x * kListWords + (k * kListThreads + threadIdx.x) / 32] = b;
      mine += __popc(b);
    }
  }
  if ((threadIdx.x & 31) == 0) atomicAdd(&s_n, mine);
  __syncthreads();
  if (threadIdx.x == 0) counts[blockIdx.x] = s_n;
}

__global__ void __launch_bounds__(kListThreads)
list_write_kernel(const uint32_t *__restrict__ words, const int32_t *__restrict__ counts,
                  int32_t *__restrict__ list, int32_t *__restrict__ total) {
  __shared__ int s_red[kListThreads / 32], s_pos[kListWords];
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  int before = 0;
  for (int b = tid; b < (int)blockIdx.x; b += kListThreads) before += counts[b];
  for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
  if (lane == 0) s_red[w] = before;
  // exclusive scan of the block's words
  const uint32_t *bw = words + (int64_t)blockIdx.x * kListWords;
  int c = tid < kListWords ? __popc(bw[tid]) : 0, inc = c;
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += v;
  }
  __shared__ int s_warp[kListThreads / 32];
  if (lane == 31) s_warp[w] = inc;
  __syncthreads();
  int base = 0;
  for (int q = 0; q < kListThreads / 32; q++) base += s_red[q];
  int pos = base + inc - c;
  for (int q = 0; q < w; q++) pos += s_warp[q];
  if (tid < kListWords) s_pos[tid] = pos;
  __syncthreads();
  for (int k = w; k < kListWords; k += kListThreads / 32) {
    const uint32_t bits = bw[k];
    if ((bits >> lane) & 1u)
      list[s_pos[k] + __popc(bits & ((1u << lane) - 1u))] =
          (int32_t)((int64_t)blockIdx.x * kListCells + k * 32 + lane);
  }
  if (blockIdx.x == gridDim.x - 1 && tid == 0) *total = base + counts[blockIdx.x];
}

// Two-level min: blocks reduce to partials, the last block to finish reduces
// the partials (counter-based, no spinning).
constexpr int kMinThreads = 1024;
// two blocks an SM: with a block per 1024 values (up to 4096) the time went into
// their starts and the last-block count, 37.0 us for 2048^2 doubles; 10.1 us so
constexpr int kMinMaxBlocks = 296;

template <typename T>
__device__ __forceinline__ T block_min(T v, T *sh) {
  for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (lane == 0) sh[wid] = v;
  __syncthreads();
  if (wid == 0) {
    v = lane < (int)(blockDim.x >> 5) ? sh[lane] : sh[0];
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
  }
  return v;
}

template <typename T>
__global__ void __launch_bounds__(kMinThreads)
min_reduce_kernel(int64_t M, const T *__restrict__ x, T *__restrict__ out,
                  T *__restrict__ partial, unsigned int *__restrict__ counter) {
  __shared__ T sh[32];
  __shared__ bool last;
  T v = x[0];
#pragma unroll 4
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < M;
       i += (int64_t)gridDim.x * blockDim.x)
    v = fmin(v, x[i]);
  v = block_min(v, sh);
  if (gridDim.x == 1) {
    if (threadIdx.x == 0) out[0] = v;
    return;
  }
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = v;
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  T m = partial[0];
  for (int b = threadIdx.x; b < (int)gridDim.x; b += blockDim.x) m = fmin(m, partial[b]);
  __syncthreads();
  m = block_min(m, sh);
  if (threadIdx.x == 0) {
    out[0] = m;
    *counter = 0u;
  }
}

template <typename T>
__global__ void gather_kernel(int64_t n, const int64_t *__restrict__ off,
                              const T *__restrict__ h, const T *__restrict__ qx,
                              const T *__restrict__ qy, T *__restrict__ oh,
                              T *__restrict__ ou, T *__restrict__ ov) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t k = off[i];
  const T hh = h[k];
  if (oh) oh[i] = hh;
  const bool wet = hh > T(kHSmall);
  if (ou) ou[i] = wet ? qx[k] / hh : T(0);
  if (ov) ov[i] = wet ? qy[k] / hh : T(0);
}

// h, qx, qy between the dense arrays and compacted arrays (cell i at dense
// offset off[i]); TO_DENSE: scatter, else gather.
template <typename T, bool TO_DENSE>
__global__ void state_layout_kernel(int64_t n, const int64_t *__restrict__ off, T *h, T *qx,
                                    T *qy, T *ch, T *cqx, T *cqy) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int64_t k = off[i];
  if constexpr (TO_DENSE) {
    h[k] = ch[i];
    qx[k] = cqx[i];
    qy[k] = cqy[i];
  } else {
    ch[i] = h[k];
    cqx[i] = qx[k];
    cqy[i] = qy[k];
  }
}

bool bad_dtype(int dtype) { return dtype != HB_F32 && dtype != HB_F64; }

}  // namespace
}  // namespace hb

using namespace hb;

#define HB_REQUIRE(cond, ...) \
  do {                        \
    if (!(cond)) return set_error(HB_ERR_ARG, __VA_ARGS__); \
  } while (0)

extern "C" int hb_flux_mask(int dtype, int64_t N, uint8_t *flux_mask, const void *h,
                            const int32_t *index, const void *t, void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_flux_mask: bad dtype %d", dtype);
  HB_REQUIRE(N >= 0, "hb_flux_mask: negative N");
  if (N == 0) return HB_OK;
  HB_REQUIRE(flux_mask && h && index && t, "hb_flux_mask: null pointer");
  auto s = as_stream(stream);
  if (dtype == HB_F64)
    flux_mask_kernel<double><<<blocks_for(N, kThreads), kThreads, 0, s>>>(
        N, flux_mask, (const double *)h, index, (const double *)t);
  else
    flux_mask_kernel<float><<<blocks_for(N, kThreads), kThreads, 0, s>>>(
        N, flux_mask, (const float *)h, index, (const float *)t);
  return check_launch("hb_flux_mask");
}

extern "C" size_t hb_cell_list_workspace_size(int64_t N) {
  const int64_t nb = (N + kListCells - 1) / kListCells;
  return N <= 0 ? 0 : (size_t)nb * (kListWords + 1) * sizeof(uint32_t);
}

extern "C" int hb_cell_list(int dtype, int rule, int64_t N, const void *h, const int32_t *index,
                            const void *x, int32_t *list, int32_t *count, void *workspace,
                            void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_cell_list: bad dtype %d", dtype);
  HB_REQUIRE(rule == 0 || rule == 1, "hb_cell_list: rule must be 0 or 1 (got %d)", rule);
  HB_REQUIRE(N > 0 && N <= INT32_MAX, "hb_cell_list: bad N=%lld", (long long)N);
  HB_REQUIRE(h && x && list && count && workspace && (rule != 0 || index),
             "hb_cell_list: null pointer");
  auto s = as_stream(stream);
  const unsigned nb = (unsigned)((N + kListCells - 1) / kListCells);
  uint32_t *words = (uint32_t *)workspace;
  int32_t *counts = (int32_t *)(words + (size_t)nb * kListWords);
#define HB_LIST_TEST(T, R) \
  list_test_kernel<T, R><<<nb, kListThreads, 0, s>>>(N, (const T *)h, index, (const T *)x, words, counts)
  if (dtype == HB_F64) {
    if (rule == 0) HB_LIST_TEST(double, 0); else HB_LIST_TEST(double, 1);
  } else {
    if (rule == 0) HB_LIST_TEST(float, 0); else HB_LIST_TEST(float, 1);
  }
#undef HB_LIST_TEST
  list_write_kernel<<<nb, kListThreads, 0, s>>>(words, counts, list, count);
  return check_launch("hb_cell_list");
}

extern "C" int hb_flux(int order, int dtype, int64_t M, int64_t N, const int32_t *wet_mask,
                       void *h_flux, void *qx_flux, void *qy_flux, const void *h,
                       const void *wl, const void *z, const void *qx, const void *qy,
                       const int32_t *index, const void *normal, const void *given_depth,
                       int depth_rows, int depth_cols, const void *given_wl, int wl_rows,
                       int wl_cols, const void *given_q, int q_rows, int q_cols,
                       const void *dx, const void *t, const void *dt, void *stream) {
  HB_REQUIRE(order == 1 || order == 2, "hb_flux: order must be 1 or 2 (got %d)", order);
  HB_REQUIRE(!bad_dtype(dtype), "hb_flux: bad dtype %d", dtype);
  HB_REQUIRE(M >= 0 && N >= 0 && M <= N, "hb_flux: bad sizes M=%lld N=%lld",
             (long long)M, (long long)N);
  if (M == 0) return HB_OK;  // HC/flucCal_2ndOrder_jh_improved_Kernel.cu:537-540
  HB_REQUIRE(wet_mask && h_flux && qx_flux && qy_flux && h && wl && z && qx && qy &&
                 index && normal && given_depth && given_wl && given_q && dx && t && dt,
             "hb_flux: null pointer");
  HB_REQUIRE(depth_rows > 0 && depth_cols > 0 && wl_rows > 0 && wl_cols > 0 &&
                 q_rows > 0 && q_cols > 0,
             "hb_flux: empty boundary table");
  auto s = as_stream(stream);
  const unsigned nb = blocks_for(M, 128);
#define HB_FLUX_LAUNCH(T, O)                                                          \
  flux_kernel<T, O><<<nb, 128, 0, s>>>(                                          \
      M, N, wet_mask, (T *)h_flux, (T *)qx_flux, (T *)qy_flux, (const T *)h,           \
      (const T *)wl, (const T *)z, (const T *)qx, (const T *)qy, index,               \
      (const T *)normal, (const T *)given_depth, depth_rows, depth_cols,              \
      (const T *)given_wl, wl_rows, wl_cols, (const T *)given_q, q_rows, q_cols,      \
      (const T *)dx, (const T *)t, (const T *)dt)
  if (dtype == HB_F64) {
    if (order == 2) HB_FLUX_LAUNCH(double, 2); else HB_FLUX_LAUNCH(double, 1);
  } else {
    if (order == 2) HB_FLUX_LAUNCH(float, 2); else HB_FLUX_LAUNCH(float, 1);
  }
#undef HB_FLUX_LAUNCH
  return check_launch("hb_flux");
}

extern "C" int hb_friction_update(int dtype, int64_t M, const int32_t *wet_mask,
                                  void *h_update, void *qx_update, void *qy_update,
                                  void *z_update, const uint8_t *landuse, void *h, void *wl,
                                  void *qx, void *qy, void *z, const void *manning,
                                  const void *dt, void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_friction_update: bad dtype %d", dtype);
  HB_REQUIRE(M >= 0, "hb_friction_update: negative M");
  if (M == 0) return HB_OK;
  HB_REQUIRE(wet_mask && h_update && qx_update && qy_update && z_update && landuse && h &&
                 wl && qx && qy && z && manning && dt,
             "hb_friction_update: null pointer");
  auto s = as_stream(stream);
#define HB_FR_LAUNCH(T)                                                                 \
  friction_update_kernel<T><<<blocks_for(M, kThreads), kThreads, 0, s>>>(                \
      M, wet_mask, (T *)h_update, (T *)qx_update, (T *)qy_update, (T *)z_update, landuse, \
      (T *)h, (T *)wl, (T *)qx, (T *)qy, (T *)z, (const T *)manning, (const T *)dt)
  if (dtype == HB_F64) HB_FR_LAUNCH(double); else HB_FR_LAUNCH(float);
#undef HB_FR_LAUNCH
  return check_launch("hb_friction_update");
}

extern "C" int hb_timestep(int dtype, int64_t M, const int32_t *wet_mask, void *accelerator,
                           void *h_max, const void *h, const void *qx, const void *qy,
                           const void *dx, const void *cfl, const void *t, const void *dt,
                           void *stream) {
  (void)t;
  (void)dt;
  HB_REQUIRE(!bad_dtype(dtype), "hb_timestep: bad dtype %d", dtype);
  HB_REQUIRE(M >= 0, "hb_timestep: negative M");
  if (M == 0) return HB_OK;
  HB_REQUIRE(wet_mask && accelerator && h_max && h && qx && qy && dx && cfl,
             "hb_timestep: null pointer");
  auto s = as_stream(stream);
#define HB_TS_LAUNCH(T)                                                             \
  timestep_kernel<T><<<blocks_for(M, kThreads), kThreads, 0, s>>>(                  \
      M, wet_mask, (T *)accelerator, (T *)h_max, (const T *)h, (const T *)qx,       \
      (const T *)qy, (const T *)dx, (const T *)cfl)
  if (dtype == HB_F64) HB_TS_LAUNCH(double); else HB_TS_LAUNCH(float);
#undef HB_TS_LAUNCH
  return check_launch("hb_timestep");
}

extern "C" int hb_rain_station(int dtype, int64_t N, void *h_update, const int16_t *mask,
                               const void *station_data, const void *dt, void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_rain_station: bad dtype %d", dtype);
  HB_REQUIRE(N >= 0, "hb_rain_station: negative N");
  if (N == 0) return HB_OK;
  HB_REQUIRE(h_update && mask && station_data && dt, "hb_rain_station: null pointer");
  auto s = as_stream(stream);
  if (dtype == HB_F64)
    rain_station_kernel<double><<<blocks_for(N, kThreads), kThreads, 0, s>>>(
        N, (double *)h_update, mask, (const double *)station_data, (const double *)dt);
  else
    rain_station_kernel<float><<<blocks_for(N, kThreads), kThreads, 0, s>>>(
        N, (float *)h_update, mask, (const float *)station_data, (const float *)dt);
  return check_launch("hb_rain_station");
}

extern "C" int hb_euler_update(int dtype, int64_t M, const int32_t *update_mask,
                               const void *h_update, const void *qx_update,
                               const void *qy_update, const void *z_update, void *h,
                               void *wl, void *z, void *qx, void *qy, void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_euler_update: bad dtype %d", dtype);
  HB_REQUIRE(M >= 0, "hb_euler_update: negative M");
  if (M == 0) return HB_OK;
  HB_REQUIRE(update_mask && h_update && qx_update && qy_update && z_update && h && wl &&
                 z && qx && qy,
             "hb_euler_update: null pointer");
  auto s = as_stream(stream);
#define HB_EU_LAUNCH(T)                                                                  \
  euler_update_kernel<T><<<blocks_for(M, kThreads), kThreads, 0, s>>>(                   \
      M, update_mask, (const T *)h_update, (const T *)qx_update, (const T *)qy_update,  \
      (const T *)z_update, (T *)h, (T *)wl, (T *)z, (T *)qx, (T *)qy)
  if (dtype == HB_F64) HB_EU_LAUNCH(double); else HB_EU_LAUNCH(float);
#undef HB_EU_LAUNCH
  return check_launch("hb_euler_update");
}

extern "C" int hb_infiltration(int dtype, int64_t M, const int32_t *wet_mask,
                               void *h_update, const uint8_t *landuse, const void *h,
                               const void *ks, const void *psi, const void *dtheta,
                               void *cumulative, const void *dt, void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_infiltration: bad dtype %d", dtype);
  HB_REQUIRE(M >= 0, "hb_infiltration: negative M");
  if (M == 0) return HB_OK;
  HB_REQUIRE(wet_mask && h_update && landuse && h && ks && psi && dtheta && cumulative && dt,
             "hb_infiltration: null pointer");
  auto s = as_stream(stream);
#define HB_IN_LAUNCH(T)                                                                 \
  infiltration_kernel<T><<<blocks_for(M, kThreads), kThreads, 0, s>>>(                  \
      M, wet_mask, (T *)h_update, landuse, (const T *)h, (const T *)ks, (const T *)psi, \
      (const T *)dtheta, (T *)cumulative, (const T *)dt)
  if (dtype == HB_F64) HB_IN_LAUNCH(double); else HB_IN_LAUNCH(float);
#undef HB_IN_LAUNCH
  return check_launch("hb_infiltration");
}

extern "C" size_t hb_min_reduce_workspace_size(int64_t M) {
  int64_t nb = (M + kMinThreads - 1) / kMinThreads;
  if (nb <= 4) return 0;
  if (nb > kMinMaxBlocks) nb = kMinMaxBlocks;
  return (size_t)nb * sizeof(double) + 256;
}

extern "C" int hb_min_reduce(int dtype, int64_t M, const void *x, void *out, void *workspace,
                             void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_min_reduce: bad dtype %d", dtype);
  HB_REQUIRE(M > 0, "hb_min_reduce: M must be positive");
  HB_REQUIRE(x && out, "hb_min_reduce: null pointer");
  int64_t nb = (M + kMinThreads - 1) / kMinThreads;
  if (nb <= 4) nb = 1;
  if (nb > kMinMaxBlocks) nb = kMinMaxBlocks;
  HB_REQUIRE(nb == 1 || workspace, "hb_min_reduce: workspace required for M=%lld",
             (long long)M);
  // the block counter sits at a fixed offset (the first word) so that a
  // workspace reused for inputs of other sizes finds it where the last call
  // left it (zero); the block partials follow at 256 bytes
  unsigned int *counter = nb == 1 ? nullptr : (unsigned int *)workspace;
  void *partial = nb == 1 ? nullptr : (void *)((char *)workspace + 256);
  auto s = as_stream(stream);
  if (dtype == HB_F64)
    min_reduce_kernel<double><<<(unsigned)nb, kMinThreads, 0, s>>>(
        M, (const double *)x, (double *)out, (double *)partial, counter);
  else
    min_reduce_kernel<float><<<(unsigned)nb, kMinThreads, 0, s>>>(
        M, (const float *)x, (float *)out, (float *)partial, counter);
  return check_launch("hb_min_reduce");
}

extern "C" int hb_gather(int dtype, int64_t n, const int64_t *cell_offsets, const void *h,
                         const void *qx, const void *qy, void *out_h, void *out_u,
                         void *out_v, void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_gather: bad dtype %d", dtype);
  HB_REQUIRE(n >= 0, "hb_gather: negative n");
  if (n == 0) return HB_OK;
  HB_REQUIRE(cell_offsets && h, "hb_gather: null pointer");
  HB_REQUIRE(!(out_u || out_v) || (qx && qy), "hb_gather: velocities need qx and qy");
  auto s = as_stream(stream);
  if (dtype == HB_F64)
    gather_kernel<double><<<blocks_for(n, kThreads), kThreads, 0, s>>>(
        n, cell_offsets, (const double *)h, (const double *)qx, (const double *)qy,
        (double *)out_h, (double *)out_u, (double *)out_v);
  else
    gather_kernel<float><<<blocks_for(n, kThreads), kThreads, 0, s>>>(
        n, cell_offsets, (const float *)h, (const float *)qx, (const float *)qy,
        (float *)out_h, (float *)out_u, (float *)out_v);
  return check_launch("hb_gather");
}

extern "C" int hb_state_layout(int dtype, int64_t n, const int64_t *offsets, int to_dense,
                               void *h, void *qx, void *qy, void *ch, void *cqx, void *cqy,
                               void *stream) {
  HB_REQUIRE(!bad_dtype(dtype), "hb_state_layout: bad dtype %d", dtype);
  HB_REQUIRE(n >= 0, "hb_state_layout: negative n");
  if (n == 0) return HB_OK;
  HB_REQUIRE(offsets && h && qx && qy && ch && cqx && cqy, "hb_state_layout: null pointer");
  auto s = as_stream(stream);
  const unsigned nb = blocks_for(n, kThreads);
  if (dtype == HB_F64) {
    auto *a = (double *)h, *b = (double *)qx, *c = (double *)qy;
    auto *d = (double *)ch, *e = (double *)cqx, *f = (double *)cqy;
    if (to_dense)
      state_layout_kernel<double, true><<<nb, kThreads, 0, s>>>(n, offsets, a, b, c, d, e, f);
    else
      state_layout_kernel<double, false><<<nb, kThreads, 0, s>>>(n, offsets, a, b, c, d, e, f);
  } else {
    auto *a = (float *)h, *b = (float *)qx, *c = (float *)qy;
    auto *d = (float *)ch, *e = (float *)cqx, *f = (float *)cqy;
    if (to_dense)
      state_layout_kernel<float, true><<<nb, kThreads, 0, s>>>(n, offsets, a, b, c, d, e, f);
    else
      state_layout_kernel<float, false><<<nb, kThreads, 0, s>>>(n, offsets, a, b, c, d, e, f);
  }
  return check_launch("hb_state_layout");
}
