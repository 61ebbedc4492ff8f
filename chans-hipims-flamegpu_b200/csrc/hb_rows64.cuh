// hb_rows64.cuh -- the FP64 step kernel.
//
// Included by hb_fused.cu inside its anonymous namespace (TilePartial, BcTable,
// close_group, mbarrier/TMA helpers, TileEntry).  Same scheme, decisions and
// data layout as the FP32 kernels (HC/flucCal_2ndOrder_jh_improved_Kernel.cu:43-506,
// HC/fluxCal_jh_modified_surface_Kernel.cu:96-139, 577-610 per face,
// HC/friction_implicit_andUpdate_jh_Kernel.cu:22-146 and
// HC/timeControl_Kernel.cu:164-198 per cell, HC/fluxMaskGenerator_Kernel.cu:19-42
// for the activity rule).
//
// What bounds it: latency and FP64 issue.  An SM starts 64 FP64 lanes a cycle,
// and a cell needs about 400 FP64 operations (two faces, eight slopes, one
// update), so the design spends as few of them as it can and keeps 16 warps an
// SM to cover their latency:
//  * a CTA of 4 warps owns 32 columns x TY rows staged by TMA, lane = column,
//    each warp walks TY/4 rows; every face is evaluated once (south faces are
//    kept for the next row, west faces go to the west lane by shuffle, the
//    faces east of lane 31 are evaluated by the first lanes of the same warp
//    before the walk, one row a lane, so no warp waits for another);
//  * reciprocals and square roots by one table-free cubic step from the
//    hardware's approximate seed (hb_fp64.cuh: 3 and 6 FP64 operations
//    instead of a division of about twelve and a root of about ten), one
//    reciprocal per edge for both velocities, one for the wave span, dt / dx once
//    per tile; the contact speed's sign is read off numerator and denominator,
//    beside the star flux, which the left or right state's flux replaces outside
//    the waves;
//  * a missing neighbour is replaced by its ghost state before the face, so
//    ghost faces go through the same code as interior ones and cost selects
//    instead of a second, divergent evaluation;
//  * minmod and the dry tests of non-negative values compare on the integer
//    pipe where that is exact.
// Measured (B200, 2nd order, steps back to back), against the FP64 build of the
// one-cell-per-lane kernel it replaced (IEEE divisions, pow, 191-230
// registers, two launches): 1024^2 282 -> 67 us a step, 2048^2 960 -> 218 us,
// 301 x 517 in 1st order 77 -> 20 us.  1024^2: 40 M warp instructions (81 M
// before), 15 M of them FP64; issue active 52 %, FP64 pipe 39 %, 16 warps an SM.
// Error against 64-bit references of the same steps: unchanged (1.1e-13 of the
// discharge's norm after 8 steps, set by the reference's friction form).
// Every operation is pinned (__dadd_rn, __dmul_rn, __fma_rn), so a face
// evaluated by two tiles, or by the general and the all-valid path, comes out
// bit for bit the same.

#include "hb_face64.cuh"

template <int TY>
struct Rows64Smem {
  static constexpr int SH = TY + 4;
  double f[4][SH * kSWF];  // h, qx, qy, z
  double hmax[TY * kTW];
  uint8_t code[SH * kSWC];
  alignas(8) unsigned long long bar;
  double xe[TY][4];   // face between cols 31 | 32: fh, fx, fy, sa
  double sxw[TY][4];  // x-slope of col -1: h, qx, qy, z
  double bc[HB_MAX_CLASSES][4];
  int bctype[HB_MAX_CLASSES];
  double manning[HB_MAX_ZONES];
  double red_d[2][kRowsNW];
  double red_s[kRowsNW];
  int red_i[kRowsNW];
  int last, last2;
  static constexpr unsigned kTxBytes =
      (unsigned)(4 * SH * kSWF * sizeof(double) + TY * kTW * sizeof(double) + SH * kSWC);
};

template <int TY>
struct View64 {
  const Rows64Smem<TY> &s;
  __device__ __forceinline__ int fi(int i, int j) const { return (i + 2) * kSWF + (j + 4); }
  __device__ __forceinline__ Cel64 cell(int i, int j) const {
    const int k = fi(i, j);
    return Cel64{s.f[0][k], s.f[1][k], s.f[2][k], s.f[3][k]};
  }
  __device__ __forceinline__ uint8_t code(int i, int j) const {
    return s.code[(i + 2) * kSWC + (j + 16)];
  }
};

// One block of TY rows of a step (tile or part of a tile); returns false when
// its data did not arrive within the bounded wait.
template <int TY, bool SOURCES, bool ALLV, int ORDER>
__device__ __forceinline__ bool rows64_tile(Rows64Smem<TY> &s, unsigned &phase, const TileEntry en,
                                            const hb_instance *__restrict__ insts,
                                            TilePartial *__restrict__ partials,
                                            TilePartial *__restrict__ gparts,
                                            unsigned *__restrict__ gcount,
                                            BcTable *__restrict__ bct,
                                            const CUtensorMap *__restrict__ maps) {
  using S = Rows64Smem<TY>;
  constexpr int R = TY / kRowsNW;
  constexpr int kPer = 32 / TY;
  const View64<TY> V{s};
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const double hs = kHSmall, g = kG;
  const bool skip = !ALLV && en.tile < 0;  // no valid cell: adds a zero partial
  const int tile = en.tile < 0 ? ~en.tile : en.tile;
  const int ii = en.inst;
  const hb_instance &in = insts[ii];
  hb_ctrl *ctrl = en.ctrl;
  if (__ldcg(&ctrl->halted)) return true;
  const int tile0 = in.tile_begin * kPer;
  const int lt = tile - tile0;
  const int tyi = lt / in.tiles_x, txi = lt - tyi * in.tiles_x;
  const int y0 = tyi * TY, x0 = txi * kTW;
  const int cur = __ldcg(&ctrl->cur);
  const double dt = __ldcg(&ctrl->dt);
  const bool first = __ldcg(&ctrl->t) == 0.0;
  const double rdt = mu(__ldcg(&ctrl->rain_rate), dt);
  const int P = in.pitch;
  if (tid == 0 && !skip) {
    const CUtensorMap *m = maps + (size_t)ii * kMapsPerInstance;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(&s.bar, S::kTxBytes);
    tma_load_2d(s.f[0], m + 0 + cur, x0, y0, &s.bar);
    tma_load_2d(s.f[1], m + 2 + cur, x0, y0, &s.bar);
    tma_load_2d(s.f[2], m + 4 + cur, x0, y0, &s.bar);
    tma_load_2d(s.f[3], m + 6, x0, y0, &s.bar);
    tma_load_2d(s.hmax, m + 7, x0 + HB_PAD_X, y0 + HB_PAD_Y, &s.bar);
    tma_load_2d(s.code, m + 8, x0, y0, &s.bar);
  }
  if (tid < HB_MAX_CLASSES) {
    if constexpr (!ALLV) {
      s.bctype[tid] = in.bc_type[tid];
      for (int q = 0; q < 4; q++) s.bc[tid][q] = __ldcg(&bct[ii].v[tid][q]);
    }
  } else if (tid >= 64 && tid < 64 + HB_MAX_ZONES) {
    s.manning[tid - 64] = in.manning[tid - 64];
  }
  const int bug_y = in.bug_y, bug_x = in.bug_x;
  const double r = dt / in.dx;
  if (!skip) {
    const bool arrived = mbar_wait(&s.bar, phase, 4000000000LL);
    if (__syncthreads_or(!arrived)) {
      if (tid == 0) atomicOr(&ctrl->status, 2);
      mbar_wait(&s.bar, phase, 4000000000LL);
      return false;
    }
    phase ^= 1u;
  }

  double vol = 0.0, smax = 0.0, outf = 0.0;
  int any_dry = 0;
  if (!skip) {
    const int j = lane, r0 = w * R;
    auto valid = [](uint8_t k) -> bool { return ALLV || is_valid(k); };
    // --- faces east of lane 31 and x-slopes of column -1, one row a lane
    if (lane < R) {
      const int i = r0 + lane;
      const Cel64 a = V.cell(i, 31), b = V.cell(i, 32);
      const uint8_t ca = V.code(i, 31), cb = V.code(i, 32);
      const Cel64 sa = slope64<ORDER, ALLV>(a, V.cell(i, 30), valid(V.code(i, 30)), b, valid(cb));
      const Cel64 sb_ = slope64<ORDER, ALLV>(b, a, valid(ca), V.cell(i, 33),
                                             valid(V.code(i, 33)));
      const Fc64 f = face64<0, ORDER, ALLV>(s.bctype, s.bc, a, ca, b, cb, sa, sb_);
      s.xe[i][0] = f.fh;
      s.xe[i][1] = f.fx;
      s.xe[i][2] = f.fy;
      s.xe[i][3] = f.sa;
      const Cel64 m1 = slope64<ORDER, ALLV>(V.cell(i, -1), V.cell(i, -2), valid(V.code(i, -2)),
                                            V.cell(i, 0), valid(V.code(i, 0)));
      s.sxw[i][0] = m1.h;
      s.sxw[i][1] = m1.qx;
      s.sxw[i][2] = m1.qy;
      s.sxw[i][3] = m1.z;
    }
    // --- column window: row r0, its y-slopes and its north face
    Cel64 C = V.cell(r0, j), Sx = V.cell(r0 + 1, j);
    uint8_t kC = V.code(r0, j), kS = V.code(r0 + 1, j), kN = V.code(r0 - 1, j);
    double Nh;
    Cel64 syC;
    Fc64 nf;
    {
      const Cel64 N = V.cell(r0 - 1, j);
      const Cel64 syN = slope64<ORDER, ALLV>(N, C, valid(kC), V.cell(r0 - 2, j),
                                             valid(V.code(r0 - 2, j)));
      syC = slope64<ORDER, ALLV>(C, Sx, valid(kS), N, valid(kN));
      nf = face64<1, ORDER, ALLV>(s.bctype, s.bc, C, kC, N, kN, syC, syN);
      Nh = N.h;
    }
    __syncwarp();  // this warp's xe and sxw
    double *hout = (double *)in.h[1 - cur];
    double *qxout = (double *)in.qx[1 - cur];
    double *qyout = (double *)in.qy[1 - cur];
    double *hmaxg = (double *)in.h_max;
    const bool infil = SOURCES && in.cum != nullptr;
    const bool stations = SOURCES && in.rain_station != nullptr;
    const bool fwd_tile = (y0 < HB_PAD_Y && in.halo_up[0] != nullptr) ||
                          (y0 + TY > in.rows - HB_PAD_Y && in.halo_down[0] != nullptr);
    const int rx = x0 + j;
#pragma unroll 1
    for (int i = r0; i < r0 + R; ++i) {
      const int ry = y0 + i;
      const size_t go = (size_t)(ry + HB_PAD_Y) * P + (rx + HB_PAD_X);
      unsigned sid = 0;
      double F0 = 0.0;
      if constexpr (SOURCES) {  // loaded ahead of the faces
        if (stations) sid = __ldg(in.rain_station + go);
        if (infil) F0 = ((const double *)in.cum)[go];
      }
      // --- west face; its flux is the west lane's east face
      double ehf, exf, eyf, eaf;
      double dh, dx_, dy_;   // flux differences (minus-side faces - plus-side faces)
      double wfh, Wh, Eh;
      bool vW, vE;
      {
        const Cel64 W = V.cell(i, j - 1), E = V.cell(i, j + 1);
        const uint8_t kW = V.code(i, j - 1), kE = V.code(i, j + 1);
        vW = valid(kW);
        vE = valid(kE);
        Wh = W.h;
        Eh = E.h;
        const Cel64 sxC = slope64<ORDER, ALLV>(C, W, vW, E, vE);
        Cel64 sxW{0.0, 0.0, 0.0, 0.0};
        sxW.z = __shfl_up_sync(0xffffffffu, sxC.z, 1);
        if constexpr (ORDER == 2) {
          sxW.h = __shfl_up_sync(0xffffffffu, sxC.h, 1);
          sxW.qx = __shfl_up_sync(0xffffffffu, sxC.qx, 1);
          sxW.qy = __shfl_up_sync(0xffffffffu, sxC.qy, 1);
        }
        if (lane == 0) sxW = Cel64{s.sxw[i][0], s.sxw[i][1], s.sxw[i][2], s.sxw[i][3]};
        const Fc64 wf = face64<0, ORDER, ALLV>(s.bctype, s.bc, W, kW, C, kC, sxW, sxC);
        ehf = __shfl_down_sync(0xffffffffu, wf.fh, 1);
        exf = __shfl_down_sync(0xffffffffu, wf.fx, 1);
        eyf = __shfl_down_sync(0xffffffffu, wf.fy, 1);
        eaf = __shfl_down_sync(0xffffffffu, wf.sa, 1);
        if (lane == 31) {
          ehf = s.xe[i][0];
          exf = s.xe[i][1];
          eyf = s.xe[i][2];
          eaf = s.xe[i][3];
        }
        dh = sb(wf.fh, ehf);
        dx_ = ad(sb(sb(wf.fx, exf), eaf), wf.sb);
        dy_ = sb(wf.fy, eyf);
        wfh = wf.fh;
      }
      // --- south face: the next row's north face
      const Cel64 SS = V.cell(i + 2, j);
      const uint8_t kSS = V.code(i + 2, j);
      const Cel64 syS = slope64<ORDER, ALLV>(Sx, SS, valid(kSS), C, valid(kC));
      const Fc64 sf = face64<1, ORDER, ALLV>(s.bctype, s.bc, Sx, kS, C, kC, syS, syC);

      // --- cell update
      if (valid(kC)) {
        bool active = first || C.h > hs;
        if (!active) {
          if constexpr (ALLV) {
            active = Eh > hs || Nh > hs || Wh > hs || Sx.h > hs;
          } else {
            auto nb = [&](bool v, int yy, int xx, double hh) {
              return v && !(yy == bug_y && xx == bug_x) && hh > hs;
            };
            active = nb(vE, ry, rx + 1, Eh) || nb(valid(kN), ry - 1, rx, Nh) ||
                     nb(vW, ry, rx - 1, Wh) || nb(valid(kS), ry + 1, rx, Sx.h);
          }
        }
        double hu = mu(ad(dh, sb(sf.fh, nf.fh)), r);
        double qxu = mu(ad(dx_, sb(sf.fx, nf.fx)), r);
        double qyu = mu(ad(dy_, ad(sb(sb(sf.fy, nf.fy), nf.sa), sf.sb)), r);
        if (!active) hu = qxu = qyu = 0.0;
        if constexpr (!ALLV) {
          // outflow through boundary faces of active cells
          const bool bE = !vE, bW = !vW, bN = !valid(kN), bS = !valid(kS);
          if (active && (bE | bW | bN | bS)) {
            double o = 0.0;
            if (bE) o += ehf;
            if (bN) o += nf.fh;
            if (bW) o -= wfh;
            if (bS) o -= sf.fh;
            outf += o;
          }
        }
        // rain (HP/SWE_CUDA.py:549 / HC/stationPrecipitation_Kernel.cu:27)
        if (stations) hu = ad(hu, mu(__ldcg(in.station_rate + sid), dt));
        else hu = ad(hu, rdt);
        if (infil && active) {
          // Green-Ampt infiltration on the active cells, after rain
          // (HC/infiltrationCUDA_Kernel.cu:20-46; order HP/CatchFlood_main.py:164-170)
          const int zc = kC & 15;
          const double K = in.ks[zc];
          const double a = ad(F0, mu(dt, K));
          const double F1 =
              mu(0.5, ad(a, sqrt(fm(a, a, mu(mu(mu(mu(4.0, dt), K), ad(in.psi[zc], C.h)),
                                            in.dtheta[zc])))));
          const double dF = min64(C.h, sb(F1, F0));
          ((double *)in.cum)[go] = ad(F0, dF);
          hu = sb(hu, dF);
        }
        // implicit friction + update (HC/friction_implicit_andUpdate_jh_Kernel.cu:22-146):
        // temp = q (sqrt(1 + 4 a |q|) - 1) / (2 a |q|), a = dt C_f / h^2, in the
        // reference's form of the root's difference (its rounding included)
        const double h = ad(C.h, hu);
        double qx = 0.0, qy = 0.0;
        const bool wet = !(h < hs);
        if (wet) {
          qx = ad(C.qx, qxu);
          qy = ad(C.qy, qyu);
          const double ih = rcp64(h);
          const double n = s.manning[kC & 15];
          if (n > 0.0) {
            const double qn = sqrt64(fm(qx, qx, mu(qy, qy)));
            const double a = mu(mu(mu(mu(mu(dt, g), mu(n, n)), rcbrt(h)), ih), ih);
            const double x = mu(a, qn);
            const double S = __dsqrt_rn(fm(4.0, x, 1.0));
            const double f = mu(sb(S, 1.0), rcp64(mu(2.0, x)));
            const double lim2 = mu(mu(mu(25.0 * kG, h), h), h);  // (5 h sqrt(g h))^2
            auto limit = [&](double q) {
              const double temp = mu(q, f);
              const double q2 = fm(2.0, temp, -q);
              const double over = (__double2hiint(q2) ^ __double2hiint(temp)) < 0 ? 0.0 : q2;
              const double t = mu(temp, temp) > lim2 ? over : temp;
              return fabs(q) > 1.0e-10 ? t : q;
            };
            qx = limit(qx);
            qy = limit(qy);
          }
          if (h > hs) {
            // CFL speed (HC/timeControl_Kernel.cu:186-189), its root in single precision
            const double sp = fm(max64(fabs(qx), fabs(qy)), ih,
                                 (double)__fsqrt_rn((float)mu(g, h)));
            smax = max64(smax, sp);
          }
        }
        if (!(h > hs)) any_dry = 1;
        hout[go] = h;
        qxout[go] = qx;
        qyout[go] = qy;
        const double hm = s.hmax[i * kTW + j];
        hmaxg[go] = h > hm ? h : hm;
        if (fwd_tile) {
          // into the neighbour strip's halo row of the same output buffer (plain
          // stores; the neighbour's arrays may be on a peer GPU)
          const int ob = 1 - cur;
          auto fwd = [&](void *const *dst, int row) {
            const size_t gh = (size_t)row * P + (rx + HB_PAD_X);
            ((double *)dst[ob])[gh] = h;
            ((double *)dst[2 + ob])[gh] = qx;
            ((double *)dst[4 + ob])[gh] = qy;
          };
          if (ry < HB_PAD_Y && in.halo_up[0] != nullptr)
            fwd(in.halo_up, in.halo_up_rows + HB_PAD_Y + ry);
          if (ry >= in.rows - HB_PAD_Y && in.halo_down[0] != nullptr)
            fwd(in.halo_down, ry - in.rows + HB_PAD_Y);
          // system-wide order before this block's partial, its count and the
          // host's next collective
          __threadfence_system();
        }
        vol = ad(vol, h);
      }
      // slide the column window down one row
      nf = sf;
      Nh = C.h;
      kN = kC;
      C = Sx;
      kC = kS;
      Sx = SS;
      kS = kSS;
      syC = syS;
    }
  }

  // the next step's CTAs may take this one's slots from here on (from the start
  // of the block instead: 512^2 26.2 -> 28.8 us a step, 301 x 517 20.4 -> 22.4)
  if constexpr (TY != 32) asm volatile("griddepcontrol.launch_dependents;");
  // --- partials and the instance's last-tile finalize
  vol = warp_sum(vol);
  if constexpr (!ALLV) outf = warp_sum(outf);
  smax = warp_max(smax);
  any_dry = __any_sync(0xffffffffu, any_dry);
  if (lane == 0) {
    s.red_d[0][w] = vol;
    s.red_d[1][w] = outf;
    s.red_s[w] = smax;
    s.red_i[w] = any_dry;
  }
  __syncthreads();
  const int n_inst_tiles = in.tiles_x * in.tiles_y * kPer;
  const int gt = group_tiles(n_inst_tiles);
  const int grp = lt / gt;
  const int gsize = min(gt, n_inst_tiles - grp * gt);
  const int gbase = tile0 / kGroupTiles + ii;
  if (tid == 0) {
    partials[tile] = block_sum<kRowsNT>(s.red_d, s.red_s, s.red_i);
    cuda::atomic_ref<unsigned, cuda::thread_scope_device> done(gcount[gbase + grp]);
    s.last = (done.fetch_add(1u, cuda::memory_order_acq_rel) == (unsigned)(gsize - 1));
  }
  __syncthreads();
  if (s.last)
    close_group<double, kRowsNT>(in, ii, partials + tile0 + grp * gt, gsize, gparts, gcount,
                                 gbase + grp, gbase, (n_inst_tiles + gt - 1) / gt, bct, s.red_d,
                                 s.red_s, s.red_i, &s.last2);
  __syncthreads();
  return true;
}

// The general path out of line, so that the all-valid path keeps its own
// register allocation.
template <int TY, bool SOURCES, int ORDER>
__device__ __noinline__ bool rows64_general(Rows64Smem<TY> &s, unsigned &phase, const TileEntry en,
                                            const hb_instance *__restrict__ insts,
                                            TilePartial *__restrict__ partials,
                                            TilePartial *__restrict__ gparts,
                                            unsigned *__restrict__ gcount,
                                            BcTable *__restrict__ bct,
                                            const CUtensorMap *__restrict__ maps) {
  return rows64_tile<TY, SOURCES, false, ORDER>(s, phase, en, insts, partials, gparts, gcount,
                                                bct, maps);
}

// The FP64 step: one programmatic launch over the prepared list (general
// blocks with a valid cell [0, n_live), all-valid blocks [n_live,
// n_valid_end), blocks without a valid cell), one CTA per block or a smaller
// grid that loops.  `order` (whole tiles only) stands in for the list.
template <int TY, bool SOURCES, int ORDER>
__global__ void __launch_bounds__(kRowsNT, 4)
rows64_kernel(const hb_instance *__restrict__ insts, const TileEntry *__restrict__ list,
              const int n_live, const int n_valid_end, const int n_list,
              TilePartial *__restrict__ partials, TilePartial *__restrict__ gparts,
              unsigned *__restrict__ gcount, BcTable *__restrict__ bct,
              const CUtensorMap *__restrict__ maps, const int32_t *__restrict__ order,
              const int32_t *__restrict__ tile_inst) {
  using S = Rows64Smem<TY>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  S &s = *reinterpret_cast<S *>(smem_raw);
  if (threadIdx.x == 0) {
    mbar_init(&s.bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if constexpr (TY == 32) asm volatile("griddepcontrol.launch_dependents;");
  unsigned phase = 0;
  for (int k = blockIdx.x; k < n_list; k += gridDim.x) {
    TileEntry en;
    if (TY == 32 && order) {
      en.tile = order[k];
      en.inst = tile_inst[en.tile < 0 ? ~en.tile : en.tile];
      en.ctrl = insts[en.inst].ctrl;
    } else {
      en = list[k];
    }
    const bool ok = k >= n_live && k < n_valid_end
                        ? rows64_tile<TY, SOURCES, true, ORDER>(s, phase, en, insts, partials,
                                                                gparts, gcount, bct, maps)
                        : rows64_general<TY, SOURCES, ORDER>(s, phase, en, insts, partials,
                                                             gparts, gcount, bct, maps);
    if (!ok) return;
  }
}
