// hb_adjoint.cu -- discrete adjoint of the FP64 fused HiPIMS step.
//
// For a loss J of the states, given lambda^{n+1} = dJ/dU^{n+1} it returns
// lambda^n = (dU^{n+1}/dU^n)^T lambda^{n+1} and accumulates
// (dU^{n+1}/dtheta)^T lambda^{n+1} for theta = (Manning n of each zone, rain
// multiplier), with the time step frozen (the forward's dt schedule replayed).
// Two passes per step over the dense raster of one catchment:
//  1. cells: recompute the block's faces (once each, in shared memory) and the
//     cell's update, reverse the update (friction, rain), write the direct part
//     of lambda^n and mu = dJ/d(flux increments) of active cells;
//  2. faces: every face once, owned by its east / south cell; reverse it with
//     the adjoints of its two cells' increments and scatter the result to its
//     four input cells with FP64 atomics.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "hb_adjoint.cuh"
#include "hb_common.cuh"
#include "hb_physics.cuh"
#include "hipims_b200.h"
#include "hipims_b200_fused.h"

static_assert(sizeof(hb_adjoint_args) == 184, "hb_adjoint_args layout (ctypes mirror)");

namespace hb {
namespace {

#include "hb_face64.cuh"

using namespace adj;

struct Grid {
  const hb_instance *in;
  int rows, cols, P, CP;
  const double *h, *qx, *qy, *z;
  const uint8_t *code;
  __device__ __forceinline__ size_t off(int r, int c) const {
    return (size_t)(r + HB_PAD_Y) * P + (c + HB_PAD_X);
  }
  __device__ __forceinline__ uint8_t cd(int r, int c) const {
    if ((unsigned)r >= (unsigned)rows || (unsigned)c >= (unsigned)cols)
      return (uint8_t)(HB_NODATA_CLASS << 4);
    return code[(size_t)(r + HB_PAD_Y) * CP + (c + HB_CODE_PAD_X)];
  }
  __device__ __forceinline__ bool valid(int r, int c) const {
    return (cd(r, c) >> 4) != HB_NODATA_CLASS;
  }
  // (r, c) within two cells of the raster: the dense arrays hold that margin
  __device__ __forceinline__ Cz cell(int r, int c) const {
    Cz v;
    const size_t k = off(r, c);
    v.h = h[k];
    v.qx = qx[k];
    v.qy = qy[k];
    v.z = z[k];
    return v;
  }
};

struct BcVals {
  double v[HB_MAX_CLASSES][4];
  int type[HB_MAX_CLASSES];
};

__device__ void load_bc(const hb_instance &in, double t, BcVals &bc) {
  const int k = threadIdx.x + threadIdx.y * blockDim.x;
  if (k >= HB_MAX_CLASSES) return;
  const int id = in.bc_id[k];
  double hb = 0, wlb = 0, qxb = 0, qyb = 0;
  if (in.given_depth && id + 1 < in.depth_cols) {
    const int tl = timelevel(t, in.given_depth, in.depth_rows, in.depth_cols);
    hb = in.given_depth[(int64_t)tl * in.depth_cols + id + 1];
  }
  if (in.given_wl && id + 1 < in.wl_cols) {
    const int tl = timelevel(t, in.given_wl, in.wl_rows, in.wl_cols);
    wlb = in.given_wl[(int64_t)tl * in.wl_cols + id + 1];
  }
  if (in.given_q && 2 + 2 * id < in.q_cols) {
    const int tl = timelevel(t, in.given_q, in.q_rows, in.q_cols);
    qxb = in.given_q[(int64_t)tl * in.q_cols + 1 + 2 * id];
    qyb = in.given_q[(int64_t)tl * in.q_cols + 2 + 2 * id];
  }
  bc.v[k][0] = hb;
  bc.v[k][1] = wlb;
  bc.v[k][2] = qxb;
  bc.v[k][3] = qyb;
  bc.type[k] = in.bc_type[k];
}

// Face (A at (ra, ca) minus side, B at (rb, cb) plus side) along DIR, any
// validity, reversed with the output adjoint `ob` and scattered into lam
// (atomics).
template <int DIR>
__device__ void face_at(const Grid &G, const BcVals &bc, int ra, int ca, int rb, int cb,
                        const FaceOut5 &ob, double *lh, double *lqx, double *lqy, double hreg) {
  const int dr = rb - ra, dc = cb - ca;  // unit step from A to B
  const bool va = G.valid(ra, ca), vb = G.valid(rb, cb);
  if (!va && !vb) return;
  FaceIn fi;
  FaceTape<DIR> tp;
  int rL = ra - dr, cL = ca - dc, rR = rb + dr, cR = cb + dc;
  double jac[3] = {1, 1, 1};
  bool ghostA = false;
  if (va && vb) {
    fi.A = G.cell(ra, ca);
    fi.B = G.cell(rb, cb);
    fi.L = G.cell(rL, cL);
    fi.R = G.cell(rR, cR);
    fi.vL = G.valid(rL, cL);
    fi.vR = G.valid(rR, cR);
    fi.noslope = false;
  } else {
    // boundary face: the valid cell against its ghost, no reconstruction
    const int rc = va ? ra : rb, cc = va ? ca : cb;
    const Cz C = G.cell(rc, cc);
    const int cls = G.cd(rc, cc) >> 4;
    Cz Gh;
    if (!ghost_of(bc.type[cls], DIR, C, bc.v[cls][0], bc.v[cls][1], bc.v[cls][2],
                  bc.v[cls][3], Gh, jac))
      return;
    fi.A = va ? C : Gh;
    fi.B = va ? Gh : C;
    fi.L = fi.A;
    fi.R = fi.B;
    fi.vL = fi.vR = false;
    fi.noslope = true;
    ghostA = !va;
  }
  face_fwd<DIR>(fi, tp);
  FaceBar xb{};
  face_rev<DIR>(fi, tp, ob, xb);
  // into a valid cell of depth h (a masked cell's state adjoint stays zero)
  auto add = [&](int r, int c, double h, const C3 &v) {
    if (h < hreg) return;
    const size_t k = G.off(r, c);
    if (v.h != 0.0) atomicAdd(lh + k, v.h);
    if (v.qx != 0.0) atomicAdd(lqx + k, v.qx);
    if (v.qy != 0.0) atomicAdd(lqy + k, v.qy);
  };
  if (va && vb) {
    if (fi.vL) add(rL, cL, fi.L.h, xb.L);
    add(ra, ca, fi.A.h, xb.A);
    add(rb, cb, fi.B.h, xb.B);
    if (fi.vR) add(rR, cR, fi.R.h, xb.R);
  } else {
    // only the valid cell receives: directly, and through its ghost
    C3 c = ghostA ? xb.B : xb.A;
    const C3 gb = ghostA ? xb.A : xb.B;
    c.h += gb.h * jac[0];
    c.qx += gb.qx * jac[1];
    c.qy += gb.qy * jac[2];
    add(va ? ra : rb, va ? ca : cb, va ? fi.A.h : fi.B.h, c);
  }
}

// Forward values of the face between (ra, ca) (minus side) and (rb, cb): the
// step's own face (hb_face64.cuh), cells by their place in the staged tile.
constexpr int kCellRows = 8;
constexpr int kTileRows = kCellRows + 4, kTileCols = 32 + 4;
struct CellTile {  // a block's cells and two around them: h, qx, qy, z and codes
  double f[4][kTileRows][kTileCols];
  uint8_t code[kTileRows][kTileCols];
  __device__ __forceinline__ Cel64 cell(int i, int j) const {
    return Cel64{f[0][i + 2][j + 2], f[1][i + 2][j + 2], f[2][i + 2][j + 2], f[3][i + 2][j + 2]};
  }
  __device__ __forceinline__ uint8_t cd(int i, int j) const { return code[i + 2][j + 2]; }
  __device__ __forceinline__ bool valid(int i, int j) const {
    return (code[i + 2][j + 2] >> 4) != HB_NODATA_CLASS;
  }
};
template <int DIR>
__device__ __forceinline__ Fc64 face_forward(const CellTile &T, const BcVals &bc, int ra, int ca) {
  constexpr int dr = DIR == 0 ? 0 : -1, dc = DIR == 0 ? 1 : 0;  // from A to B
  const int rb = ra + dr, cb = ca + dc;
  const Cel64 A = T.cell(ra, ca), B = T.cell(rb, cb);
  const Cel64 sA = slope64<2, false>(A, T.cell(ra - dr, ca - dc), T.valid(ra - dr, ca - dc), B,
                                     true);
  const Cel64 sB = slope64<2, false>(B, A, true, T.cell(rb + dr, cb + dc),
                                     T.valid(rb + dr, cb + dc));
  return face64<DIR, 2, false>(bc.type, bc.v, A, T.cd(ra, ca), B, T.cd(rb, cb), sA, sB);
}

// Pass 1: a block of 32 x 8 cells and nine warps.  The block's cells are staged
// in shared memory, each face of theirs is evaluated once into shared memory
// (warps 0-7: the west and north faces of their row's cells; warp 8: the last
// row of y-faces and the last column of x-faces), then the cells are updated
// and reversed.  FP64 issue and latency bind it.  512^2 cells, cold: faces in a
// pass of their own through global memory, IEEE divisions, pow and boundary
// tables searched by every block 27 + 41 us; one pass 34 us; the step's face,
// staged cells and three blocks an SM 28 us.
__global__ void __launch_bounds__(32 * (kCellRows + 1), 3)
adj_cell_kernel(hb_adjoint_args a) {
  __shared__ BcVals bc;
  __shared__ double red[HB_MAX_ZONES + 1][kCellRows + 1];
  __shared__ double sx[5][kCellRows][33], sy[5][kCellRows + 1][32];
  extern __shared__ __align__(16) unsigned char smem_raw[];
  CellTile &T = *reinterpret_cast<CellTile *>(smem_raw);
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const hb_instance &in = *a.instance;
  Grid G{a.instance, a.rows, a.cols, a.pitch, a.code_pitch, a.h, a.qx, a.qy,
         (const double *)in.z, in.code};
  const int lane = threadIdx.x, w = threadIdx.y;
  const int tid = lane + 32 * w;
  for (int q = tid; q < (HB_MAX_ZONES + 1) * (kCellRows + 1); q += 32 * (kCellRows + 1))
    (&red[0][0])[q] = 0.0;
  const int r0 = blockIdx.y * kCellRows, c0 = blockIdx.x * 32;
  const int r = r0 + w, c = c0 + lane;
  // this thread's x-face (rx, cx - 1) | (rx, cx) and y-face (r, c) | (r - 1, c)
  const bool extra = w == kCellRows;  // the last warp's x-faces: column c0 + 32, row = lane
  const int rx = extra ? r0 + lane : r, cx = extra ? c0 + 32 : c;
  const bool hasx = (!extra || lane < kCellRows) && rx < a.rows && cx <= a.cols;
  const bool hasy = r <= a.rows && c < a.cols;
  // stage the cells (the dense arrays hold two cells around the raster)
  for (int q = tid; q < kTileRows * kTileCols; q += 32 * (kCellRows + 1)) {
    const int i = q / kTileCols, j = q - i * kTileCols;
    const int rr = r0 + i - 2, cc = c0 + j - 2;
    Cz v{0, 0, 0, 0};
    if (rr < a.rows + 2 && cc < a.cols + 2) v = G.cell(rr, cc);
    T.f[0][i][j] = v.h;
    T.f[1][i][j] = v.qx;
    T.f[2][i][j] = v.qy;
    T.f[3][i][j] = v.z;
    T.code[i][j] = G.cd(rr, cc);
  }
  __syncthreads();
  const int lx = cx - c0;  // this thread's x-face in the block
  const bool ghosts = (hasx && T.valid(rx - r0, lx - 1) != T.valid(rx - r0, lx)) ||
                      (hasy && T.valid(w, lane) != T.valid(w - 1, lane));
  if (__syncthreads_or(ghosts)) {  // boundary tables: blocks with ghost faces only
    load_bc(in, a.t, bc);
    __syncthreads();
  }
  if (hasx) {
    const Fc64 f = face_forward<0>(T, bc, rx - r0, lx - 1);
    const int i = rx - r0, j = lx;
    sx[0][i][j] = f.fh; sx[1][i][j] = f.fx; sx[2][i][j] = f.fy; sx[3][i][j] = f.sa;
    sx[4][i][j] = f.sb;
  }
  if (hasy) {
    const Fc64 f = face_forward<1>(T, bc, w, lane);
    sy[0][w][lane] = f.fh; sy[1][w][lane] = f.fx; sy[2][w][lane] = f.fy; sy[3][w][lane] = f.sa;
    sy[4][w][lane] = f.sb;
  }
  __syncthreads();
  double gz = 0.0, gm = 0.0;
  int zone = 0;
  if (!extra && r < a.rows && c < a.cols) {
    const size_t k = G.off(r, c);
    double *mu_h = a.mu, *mu_qx = a.mu + a.mu_stride, *mu_qy = a.mu + 2 * a.mu_stride;
    if (!T.valid(w, lane)) {
      a.out_h[k] = a.out_qx[k] = a.out_qy[k] = 0.0;
      mu_h[k] = mu_qx[k] = mu_qy[k] = 0.0;
    } else {
      const Cel64 u = T.cell(w, lane);
      const C3 ob{a.lam_h[k], a.lam_qx[k], a.lam_qy[k]};
      const double hs = kHs;
      // fluxMask activity (HC/fluxMaskGenerator_Kernel.cu:19-42, cell 0 ignored)
      bool active = a.first || u.h > hs;
      if (!active) {
        auto wet = [&](int dr, int dc) {
          const bool bug = (r + dr == in.bug_y && c + dc == in.bug_x);
          return T.valid(w + dr, lane + dc) && !bug && T.cell(w + dr, lane + dc).h > hs;
        };
        active = wet(0, 1) || wet(-1, 0) || wet(0, -1) || wet(1, 0);
      }
      const double kk = a.dt / in.dx;
      C3 rr{0, 0, 0};
      if (active) {
        const int j = lane;
        rr.h = ((sx[0][w][j] + sy[0][w + 1][j]) - (sx[0][w][j + 1] + sy[0][w][j])) * kk;
        rr.qx = ((sx[1][w][j] + sy[1][w + 1][j]) - (sx[1][w][j + 1] + sy[1][w][j]) -
                 sx[3][w][j + 1] + sx[4][w][j]) * kk;
        rr.qy = ((sx[2][w][j] + sy[2][w + 1][j]) - (sx[2][w][j + 1] + sy[2][w][j]) -
                 sy[3][w][j] + sy[4][w + 1][j]) * kk;
      }
      rr.h += a.rain_rate * a.dt;
      zone = T.cd(w, lane) & 15;
      const double n = in.manning[zone];
      CellTape tp;
      const C3 uu{u.h, u.qx, u.qy};
      cell_fwd(uu, rr, n, a.dt, tp);
      C3 ub, rb;
      double nb;
      cell_rev(tp, ob, a.dt, ub, rb, nb);
      // Below h_reg the cell's state adjoint is held at zero.  The step never
      // clamps h >= 0 (as the reference); negative depths and films of a few
      // h_small on bumps between deeper cells, with discharges at rounding
      // level, have linearised gains above one per step that the nonlinear
      // step saturates, so the exact adjoint through them grows without bound.
      const bool keep = !(u.h < a.h_reg);
      a.out_h[k] = keep ? ub.h : 0.0;
      a.out_qx[k] = keep ? ub.qx : 0.0;
      a.out_qy[k] = keep ? ub.qy : 0.0;
      mu_h[k] = active ? rb.h : 0.0;
      mu_qx[k] = active ? rb.qx : 0.0;
      mu_qy[k] = active ? rb.qy : 0.0;
      gz = nb;
      gm = rb.h * a.rain_base * a.dt;
    }
  }
  asm volatile("griddepcontrol.launch_dependents;");
  // block reduction of the parameter gradient: each warp sums the zones it
  // holds (one or two as a rule)
  for (unsigned rem = __ballot_sync(0xffffffffu, gz != 0.0); rem;) {
    const int zz = __shfl_sync(0xffffffffu, zone, __ffs(rem) - 1);
    double v = (zone == zz) ? gz : 0.0;
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) red[zz][w] = v;
    rem &= ~__ballot_sync(0xffffffffu, zone == zz);
  }
  for (int o = 16; o > 0; o >>= 1) gm += __shfl_xor_sync(0xffffffffu, gm, o);
  if (lane == 0) red[HB_MAX_ZONES][w] = gm;
  __syncthreads();
  if (tid <= HB_MAX_ZONES) {
    double v = 0;
    for (int q = 0; q < kCellRows; q++) v += red[tid][q];
    if (v != 0.0) atomicAdd(a.grad + tid, v);
  }
}

// Pass 2: every face along DIR (x: owned by its east cell, y: by its south
// cell); blockIdx.z selects the direction, which halves a thread's chain and
// evens out the last wave.  Bound by latency at 16 warps an SM (the decision
// tape of a face fills 128 registers; 156 without the cap, 3 % slower): 62 us a
// step of 512^2 cells with both directions in one thread and IEEE divisions,
// 34 us so (cold).
template <int DIR>
__device__ __forceinline__ void face_rev_at(const hb_adjoint_args &a, const Grid &G,
                                            const hb_instance &in, BcVals &bc, int r, int c) {
  const int ra = r, ca = DIR == 0 ? c - 1 : c, rb = DIR == 0 ? r : r - 1, cb = c;
  const double *mu_h = a.mu, *mu_qx = a.mu + a.mu_stride, *mu_qy = a.mu + 2 * a.mu_stride;
  const bool has = DIR == 0 ? (r < a.rows && c <= a.cols) : (r <= a.rows && c < a.cols);
  const bool va = has && G.valid(ra, ca), vb = has && G.valid(rb, cb);
  auto mu = [&](bool v, int rr, int cc) {
    C3 m{0, 0, 0};
    if (v) {
      const size_t k = G.off(rr, cc);
      m = C3{mu_h[k], mu_qx[k], mu_qy[k]};
    }
    return m;
  };
  const double kk = a.dt / in.dx;
  const C3 mA = mu(va, ra, ca), mB = mu(vb, rb, cb);
  const FaceOut5 ob{kk * (mB.h - mA.h), kk * (mB.qx - mA.qx), kk * (mB.qy - mA.qy),
                    -kk * (DIR == 0 ? mA.qx : mA.qy), kk * (DIR == 0 ? mB.qx : mB.qy)};
  const bool work = (va || vb) && (ob.fh != 0.0 || ob.fx != 0.0 || ob.fy != 0.0 ||
                                   ob.sa != 0.0 || ob.sb != 0.0);
  if (__syncthreads_or(work && va != vb)) {  // boundary tables: blocks with ghost faces only
    load_bc(in, a.t, bc);
    __syncthreads();
  }
  if (work) face_at<DIR>(G, bc, ra, ca, rb, cb, ob, a.out_h, a.out_qx, a.out_qy, a.h_reg);
}

__global__ void __launch_bounds__(128, 4)
adj_face_kernel(hb_adjoint_args a) {
  __shared__ BcVals bc;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const hb_instance &in = *a.instance;
  Grid G{a.instance, a.rows, a.cols, a.pitch, a.code_pitch, a.h, a.qx, a.qy,
         (const double *)in.z, in.code};
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  const int r = blockIdx.y * blockDim.y + threadIdx.y;
  if (blockIdx.z == 0)
    face_rev_at<0>(a, G, in, bc, r, c);
  else
    face_rev_at<1>(a, G, in, bc, r, c);
  asm volatile("griddepcontrol.launch_dependents;");
}

__global__ void gauge_kernel(int64_t n, const int64_t *off, const double *h, const double *obs,
                             double *lam_h, double w) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) atomicAdd(lam_h + off[i], 2.0 * w * (h[off[i]] - obs[i]));
}

}  // namespace
}  // namespace hb

using namespace hb;

extern "C" int hb_adjoint_step(const hb_adjoint_args *a, void *stream) {
  if (!a || !a->instance || !a->h || !a->qx || !a->qy || !a->lam_h || !a->lam_qx ||
      !a->lam_qy || !a->out_h || !a->out_qx || !a->out_qy || !a->mu || !a->grad)
    return set_error(HB_ERR_ARG, "hb_adjoint_step: null pointer");
  if (a->rows <= 0 || a->cols <= 0 || a->pitch < a->cols + 8 || a->mu_stride <= 0)
    return set_error(HB_ERR_ARG, "hb_adjoint_step: bad geometry");
  if (a->faces && a->face_stride < (int64_t)(a->rows + 1) * (a->cols + 1))
    return set_error(HB_ERR_ARG, "hb_adjoint_step: face_stride below (rows + 1) * (cols + 1)");
  auto st = as_stream(stream);
  // Programmatic launches: each kernel waits for the one before it at its top.
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cfg.blockDim = dim3(32, kCellRows + 1);
  cfg.dynamicSmemBytes = sizeof(CellTile);
  cfg.gridDim = dim3((a->cols + 31) / 32, (a->rows + kCellRows - 1) / kCellRows);
  cudaError_t e = cudaLaunchKernelEx(&cfg, adj_cell_kernel, *a);
  if (e == cudaSuccess) {
    cfg.blockDim = dim3(32, 4);
    cfg.dynamicSmemBytes = 0;
    cfg.gridDim = dim3((a->cols + 1 + 31) / 32, (a->rows + 1 + 3) / 4, 2);
    e = cudaLaunchKernelEx(&cfg, adj_face_kernel, *a);
  }
  if (e != cudaSuccess) return set_error(HB_ERR_CUDA, "hb_adjoint_step: %s", cudaGetErrorString(e));
  return check_launch("hb_adjoint_step");
}

extern "C" int hb_adjoint_gauge(int64_t n, const int64_t *offsets, const double *h,
                                const double *obs, double *lam_h, double weight, void *stream) {
  if (n < 0) return set_error(HB_ERR_ARG, "hb_adjoint_gauge: negative n");
  if (n == 0) return HB_OK;
  if (!offsets || !h || !obs || !lam_h) return set_error(HB_ERR_ARG, "hb_adjoint_gauge: null");
  gauge_kernel<<<blocks_for(n, 256), 256, 0, as_stream(stream)>>>(n, offsets, h, obs, lam_h,
                                                                   weight);
  return check_launch("hb_adjoint_gauge");
}
