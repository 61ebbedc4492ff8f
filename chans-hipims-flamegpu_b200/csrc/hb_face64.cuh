// hb_face64.cuh -- one FP64 face of the scheme, shared by the step kernel
// (hb_rows64.cuh, which says how it is laid out and why) and the adjoint's
// forward pass.  Included inside namespace hb, after hb_fp64.cuh and the
// constants of hb_common.cuh.  Every operation is pinned (no contraction), so a
// face comes out bit for bit the same wherever it is evaluated.

__device__ __forceinline__ double ad(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sb(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double mu(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double fm(double a, double b, double c) { return __fma_rn(a, b, c); }

__device__ __forceinline__ double max64(double a, double b) { return a > b ? a : b; }
__device__ __forceinline__ double min64(double a, double b) { return a < b ? a : b; }
// max(x, 0) by the sign bit
__device__ __forceinline__ double pos64(double x) { return __double2hiint(x) < 0 ? 0.0 : x; }
// minmod(x, y) (HC/flucCal_2ndOrder_jh_improved_Kernel.cu:74-81): the sign test
// on the sign bits (a zero argument has the smaller magnitude and is selected)
__device__ __forceinline__ double mm64(double x, double y) {
  const double m = fabs(x) < fabs(y) ? x : y;
  return (__double2hiint(x) ^ __double2hiint(y)) < 0 ? 0.0 : m;
}

struct Cel64 {
  double h, qx, qy, z;
};
// fluxes in the global frame from the minus (west / south) side, bed-slope
// terms of both sides
struct Fc64 {
  double fh, fx, fy, sa, sb;
};

// One face in its own frame from the cells' depths and beds (A minus, B plus)
// and the edge states L, R (depth, bed, normal and tangential discharge).
template <int ORDER>
__device__ __forceinline__ void face_core64(double Ah, double Az, double Bh, double Bz,
                                            double Lh, double Lz, double Lqn, double Lqt,
                                            double Rh, double Rz, double Rqn, double Rqt,
                                            double &fh, double &fn, double &ft, double &sa,
                                            double &sbt) {
  const double hs = kHSmall, g = kG;
  const bool dryA = Ah < hs, dryB = Bh < hs;
  // velocities of the edge states before the hydrostatic step; a dry cell's
  // edge carries none
  const double il = (dryA || Lh < hs) ? 0.0 : rcp64(Lh);
  const double ir = (dryB || Rh < hs) ? 0.0 : rcp64(Rh);
  const double uL = mu(Lqn, il), vL = mu(Lqt, il), uR = mu(Rqn, ir), vR = mu(Rqt, ir);
  // hydrostatic reconstruction
  const double wa = ad(Az, Ah), wb = ad(Bz, Bh);
  const bool down = wa > wb;
  const double hi = down ? wa : wb, lo = down ? wb : wa;
  double Lw = max64(min64(ad(Lh, Lz), hi), lo);
  double Rw = max64(min64(ad(Rh, Rz), hi), lo);
  if constexpr (ORDER == 2) {
    const double m = max64(Lw, Rw);
    Lw = down ? m : Lw;
    Rw = down ? Rw : m;
  } else {
    const bool flip = mu(sb(wa, wb), sb(Lw, Rw)) < 0.0;
    const double avg = mu(ad(Lw, Rw), 0.5);
    Lw = flip ? avg : Lw;
    Rw = flip ? avg : Rw;
  }
  const double zbm = max64(sb(Lw, Lh), sb(Rw, Rh));
  const double hL = pos64(sb(Lw, zbm)), hR = pos64(sb(Rw, zbm));
  sa = mu(mu(0.5 * kG, ad(Ah, hL)), sb(sb(Lw, hL), Az));
  sbt = mu(mu(0.5 * kG, ad(Bh, hR)), sb(sb(Rw, hR), Bz));
  // HLLC
  const bool thinL = hL <= hs, thinR = hR <= hs;
  const double qL = mu(uL, hL), qR = mu(uR, hR);
  const double gL = mu(g, hL), gR = mu(g, hR);
  const double aL = sqrt64(gL), aR = sqrt64(gR);
  const double us = sb(fm(ad(uL, uR), 0.5, aL), aR);
  const double as = fabs(fm(ad(aL, aR), 0.5, mu(sb(uL, uR), 0.25)));
  const double sL = thinL ? fm(-2.0, aR, uR) : min64(sb(uL, aL), sb(us, as));
  const double sR = thinR ? fm(2.0, aL, uL) : max64(ad(uR, aR), ad(us, as));
  const double nL = fm(uL, qL, mu(mu(0.5, gL), hL)), nR = fm(uR, qR, mu(mu(0.5, gR), hR));
  const double pL = mu(hL, sb(uL, sL)), pR = mu(hR, sb(uR, sR));
  // contact speed sM = num / den: only its sign is needed (0 / 0 counts as
  // negative, as in the reference; so does 0, where no mass crosses)
  const double num = sb(mu(sL, pR), mu(sR, pL)), den = sb(pR, pL);
  const bool left = 0.0 <= sL;
  const bool up =
      left || (num != 0.0 && (__double2hiint(num) ^ __double2hiint(den)) >= 0);
  // the region's flux (wave speeds clamped at 0 in the star flux give it too, but
  // beside a thin side they may cross, which is 0 / 0, or both be negative with
  // sM > 0); a face between dry sides has the star flux's factor 0
  const bool dd = dryA && dryB, dry = (hL < hs && hR < hs) || dd;
  const bool outL = left && !dry, outR = !up && __double2hiint(sR) < 0 && !dry;
  double inv = rcp64(sb(sR, sL));
  if (dry) inv = 0.0;
  const double sLR = mu(sL, sR);
  fh = mu(fm(sLR, sb(hR, hL), sb(mu(sR, qL), mu(sL, qR))), inv);
  fn = mu(fm(sLR, sb(qR, qL), sb(mu(sR, nL), mu(sL, nR))), inv);
  fh = outL ? qL : (outR ? qR : fh);
  fn = outL ? nL : (outR ? nR : fn);
  // the tangential flux is the mass flux times the upwind tangential velocity
  ft = mu(fh, up ? vL : vR);
  if (dd) sa = sbt = 0.0;
}

// Ghost of cell C across a missing neighbour along DIR
// (HC/flucCal_2ndOrder_jh_improved_Kernel.cu:197-332; FALL, type 9:
// HC/fluxCal_jh_modified_surface_Kernel.cu:389-396).  False: no ghost rule.
template <int DIR, int ORDER>
__device__ __forceinline__ bool ghost64(int type, const double *bc, const Cel64 &C, Cel64 &G) {
  G = C;
  switch (type) {
    case 3:  // both components change sign on x-faces, neither on y-faces
      if (DIR == 0) {
        G.qx = -C.qx;
        G.qy = -C.qy;
      }
      return true;
    case 4:
      if (DIR == 0) G.qx = -C.qx; else G.qy = -C.qy;
      return true;
    case 5:
      return true;
    case 6:
      G.h = bc[0];
      return true;
    case 7:
      G.qx = bc[2];
      G.qy = bc[3];
      return true;
    case 8:
      G.h = sb(max64(bc[1], C.z), C.z);
      return true;
    case 9:
      if (ORDER != 1) return false;
      G.h = G.qx = G.qy = 0.0;
      return true;
    default:
      return false;
  }
}

// Slopes of c between its minus-side neighbour m and plus-side neighbour p (a
// missing one is replaced by c, HC/flucCal_2ndOrder_jh_improved_Kernel.cu:416-428);
// ORDER 1 uses the bed's only.
template <int ORDER, bool ALLV>
__device__ __forceinline__ Cel64 slope64(const Cel64 &c, const Cel64 &m, bool vm, const Cel64 &p,
                                         bool vp) {
  auto one = [&](double x, double a, double b) {
    const double lo = ALLV || vm ? a : x, up = ALLV || vp ? b : x;
    return mm64(sb(x, lo), sb(up, x));
  };
  Cel64 s{0.0, 0.0, 0.0, one(c.z, m.z, p.z)};
  if constexpr (ORDER == 2) {
    s.h = one(c.h, m.h, p.h);
    s.qx = one(c.qx, m.qx, p.qx);
    s.qy = one(c.qy, m.qy, p.qy);
  }
  return s;
}

// Face between A (minus side, code ca) and B (plus side, code cb) along DIR
// from the cells and their slopes; general tiles: a missing side becomes the
// other cell's ghost, without reconstruction, and the cell is the minus side, in
// its outward frame (with crossing wave speeds a face has the minus side's flux).
template <int DIR, int ORDER, bool ALLV>
__device__ __forceinline__ Fc64 face64(const int *bctype, const double (*bc)[4], Cel64 A,
                                       uint8_t ca, Cel64 B, uint8_t cb, Cel64 sA, Cel64 sB) {
  bool va = true, vb = true, rule = true;
  if constexpr (!ALLV) {
    va = (ca >> 4) != HB_NODATA_CLASS;
    vb = (cb >> 4) != HB_NODATA_CLASS;
    if (va != vb) {
      const int cls = (va ? ca : cb) >> 4;
      Cel64 G;
      rule = ghost64<DIR, ORDER>(bctype[cls], bc[cls], va ? A : B, G);
      if (!va) {
        A = Cel64{B.h, -B.qx, -B.qy, B.z};
        G.qx = -G.qx;
        G.qy = -G.qy;
      }
      B = G;
      sA = sB = Cel64{0.0, 0.0, 0.0, 0.0};
    }
  }
  Cel64 L, R;
  if constexpr (ORDER == 2) {
    L = Cel64{fm(0.5, sA.h, A.h), fm(0.5, sA.qx, A.qx), fm(0.5, sA.qy, A.qy), fm(0.5, sA.z, A.z)};
    R = Cel64{fm(-0.5, sB.h, B.h), fm(-0.5, sB.qx, B.qx), fm(-0.5, sB.qy, B.qy),
              fm(-0.5, sB.z, B.z)};
  } else {
    // the bed alone takes half its slope, on a side whose neighbour is wet
    L = A;
    R = B;
    if (B.h > kHSmall) L.z = fm(0.5, sA.z, A.z);
    if (A.h > kHSmall) R.z = fm(-0.5, sB.z, B.z);
  }
  Fc64 o;
  double fn, ft;
  if constexpr (DIR == 0) {
    face_core64<ORDER>(A.h, A.z, B.h, B.z, L.h, L.z, L.qx, L.qy, R.h, R.z, R.qx, R.qy, o.fh, fn,
                       ft, o.sa, o.sb);
    o.fx = fn;
    o.fy = ft;
  } else {
    // normal +y, tangent -x; the tangential flux is linear in the tangential
    // discharge, so +qx in gives +Fx out
    face_core64<ORDER>(A.h, A.z, B.h, B.z, L.h, L.z, L.qy, L.qx, R.h, R.z, R.qy, R.qx, o.fh, fn,
                       ft, o.sa, o.sb);
    o.fx = ft;
    o.fy = fn;
  }
  if constexpr (!ALLV) {
    if (!(va || vb) || !rule) o = Fc64{0.0, 0.0, 0.0, 0.0, 0.0};
    if (!va) {
      o.fh = -o.fh;
      o.sb = o.sa;
      o.sa = 0.0;
    } else if (!vb) {
      o.sb = 0.0;
    }
  }
  return o;
}
