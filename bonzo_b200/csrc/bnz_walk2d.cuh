// bnz_walk2d.cuh -- the 2D stages as strip walks of single warps: large batches
// and large single grids (bnz_common.h: batch_walks, grid_variant).
//
// A warp owns a strip of at most 30 columns and walks its rows upwards; lane l
// is column x0 - 1 + l, so the strip and one column on either side fill the
// warp.  Per row it forms the y faces below the row, the x faces of the row and
// the corner EMFs between them, then finishes the row below: fluxes are used as
// they are formed and never stored for a tile.
// What a lane carries from row to row (the lower y fluxes, the row's x flux
// differences, then its half-done update, a corner EMF, a cell EMF) stays in
// its own slots of shared memory; values of a neighbouring column come by
// shuffles.  The next row's cells are copied in (cp.async) while this one
// computes.  There is no block barrier anywhere, which is what held the tile
// kernels of bnz_fused.cuh up most (their six phases a tile end in one each).
// The face work is about theirs: a strip of w x h cells forms (w + 1)(h + 2) x
// faces and (w + 2)(h + 1) y faces, 2.2 a cell at 30 x 32, 2.3 at 30 x 18 (5 M
// zones), 2.5 at 30 x 8, against 2.43 of 15 x 14 tiles.
// Expressions are stage_cell's and the flux stages', and what the fast build
// would contract another way is fixed by hand, so the bits are the same in both
// builds (test_gpu_walk2d.py).
// What bounds it is FP64 dependency latency at 12 (corrector: 15.8 KB of shared
// memory and 168 registers a thread) and 16 (predictor) warps an SM.  Measured,
// HLLD, 64 blasts of 6.4 M zones 2.15 ms a step against 2.35 on the persistent
// 15 x 14 tiles (corrector 1.27 against 1.52); one 1024^2 grid 411 us a step
// against 596 on 32 x 8 tiles (bnz_common.h has other sizes and solvers).
// Included inside the per-floating-point-mode namespace, after bnz_fused.cuh
// and bnz_split_flux.cuh (cp.async helpers).
#pragma once

namespace fused {

constexpr int WALK_NW = 4;  // warps a block, one strip each
static_assert(WALK_COLS + 2 == 32, "a lane a column of the strip, and one on either side");

// a lane's slots between rows: [U] the x part of the row's flux differences,
// then its hydro update, [BZ] likewise of bz; the row's x flux of by, its cell
// EMF, the y fluxes below it (six hydro ones and bz's), the corner EMF below
enum { SV_U = 0, SV_BZ = 6, SV_FXBY = 7, SV_EC = 8, SV_FY = 9, SV_EZ = 16, SV_N = 17 };

template <int ORDER>
struct WalkSmem {
  // a staged row: the predictor's w^n and b^n (12 fields) on the 32 columns,
  // the corrector's ws (9 fields) on them and one more on either side
  static constexpr int RW = ORDER ? 34 : 32, NV = ORDER ? NM : NM + 3;
  static constexpr int ROW = NV * RW;
  static constexpr int WARP = 3 * ROW + (ORDER ? 16 * 32 : 0) + SV_N * 32;  // doubles
  static constexpr int BYTES = 8 * WARP * WALK_NW;
};

// the states of the x face at a staged cell p with slopes d (bnz_device.cuh face_flux)
template <int ORDER>
struct WalkX {
  const double *p, *d;
  static constexpr int RW = WalkSmem<ORDER>::RW;
  __device__ __forceinline__ double L(int n) const { return ORDER ? p[n * RW - 1] + d[slot8(n) * 32 - 1] : p[n * RW - 1]; }
  __device__ __forceinline__ double R(int n) const { return ORDER ? p[n * RW] - d[slot8(n) * 32] : p[n * RW]; }
  __device__ __forceinline__ double at(bool left, int n) const {
    const double v = (left ? p - 1 : p)[n * RW];
    if (ORDER == 0) return v;
    return fma(left ? 1. : -1., (left ? d - 1 : d)[slot8(n) * 32], v);
  }
};

// the states of the y face between the staged cells lo and hi; with PLM lo is
// the lower state itself and the upper one hi minus its slope
template <int ORDER>
struct WalkY {
  const double *lo, *hi, *d;
  static constexpr int RW = WalkSmem<ORDER>::RW;
  __device__ __forceinline__ double L(int n) const { return ORDER ? lo[slot8(n) * 32] : lo[plain::perm<1>(n) * RW]; }
  __device__ __forceinline__ double R(int n) const {
    return ORDER ? hi[plain::perm<1>(n) * RW] - d[slot8(n) * 32] : hi[plain::perm<1>(n) * RW];
  }
  __device__ __forceinline__ double at(bool left, int n) const {
    if (ORDER == 0) return (left ? lo : hi)[plain::perm<1>(n) * RW];
    return left ? L(n) : R(n);
  }
};

// ORDER 0: the predictor on a strip of the predictor range; ORDER 1: the
// corrector (PLM, limiter LIM, no characteristic slopes) on active cells.
template <int ORDER, int RS, int LIM>
__global__ void __launch_bounds__(32 * WALK_NW, ORDER ? 3 : 4)
    k_walk2d(const Inst* __restrict__ insts, const Tile* __restrict__ tiles, int ntiles, int parity) {
  using M = WalkSmem<ORDER>;
  constexpr int RW = M::RW;
  extern __shared__ __align__(16) double walk_smem[];
  __shared__ Inst sI[WALK_NW];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int t0 = blockIdx.x * WALK_NW + wid;
  if (t0 >= ntiles) return;
  const Tile T = tiles[t0];
  {
    const int* src = reinterpret_cast<const int*>(insts + T.inst);
    int* dst = reinterpret_cast<int*>(&sI[wid]);
    for (int q = lane; q < (int)(sizeof(Inst) / sizeof(int)); q += 32) dst[q] = src[q];
    __syncwarp();
  }
  const Inst& I = sI[wid];
  const double dtf = I.ds->dt;
  if (!(dtf > 0.)) {
    if (ORDER) copy_tile(I, T, parity, lane, 32);  // time has reached tmax: carry the state over
    return;
  }
  const double dt = ORDER ? dtf : 0.5 * dtf;
  const int i = T.x0 - 1 + lane;
  const bool col = lane <= T.wx + 1;            // a column of the strip or beside it
  const bool xface = lane >= 1 && col;          // the x face on its left is formed
  const bool own = lane >= 1 && lane <= T.wx;   // its cells are updated
  const long long nx = I.nx, sv = I.sv;
  double* base = walk_smem + wid * M::WARP;
  double* rm = base + lane + ORDER;  // rows s - 1, s, s + 1 in turn
  double* rc = rm + M::ROW;
  double* rn = rc + M::ROW;
  double* sL = base + 3 * M::ROW + lane;         // PLM: lower state of the next y face
  double* sD = sL + 8 * 32;                     // PLM: half slopes
  double* sv_ = base + 3 * M::ROW + (ORDER ? 16 * 32 : 0) + lane;
  const double* __restrict__ wg = ORDER ? I.ws : I.w[parity];
  const double* __restrict__ bg = ORDER ? I.bs : I.b[parity];
  const AxisMap mx = axis_map(I, 0), my = axis_map(I, 1);
  const bool interior = ORDER || pred_interior(I, T);
  // ghost positions of the predictor's inputs: the lane's source columns; a
  // reflecting side flips signs, so its tiles copy through registers
  const bool flips = !interior && (I.bc[0][0] == 2 || I.bc[0][1] == 2 || I.bc[1][0] == 2 || I.bc[1][1] == 2);
  int ci = i, fi = i;
  if (!interior && col && !flips) {
    bool f, z;
    ci = map_cell(i, mx, f);
    fi = map_face(i, mx, f, z);
  }
  auto load = [&](double* r, int s) {
    if (!col) return;
    if (ORDER) {
      const double* q = wg + s * nx + i;
#pragma unroll
      for (int n = 0; n < NM; ++n) split::cpa::copy8(r + n * RW, q + n * sv);
      const int side = lane == 0 ? -1 : lane == T.wx + 1 ? 1 : 0;
      if (side) {
#pragma unroll
        for (int n = 0; n < NM; ++n) split::cpa::copy8(r + n * RW + side, q + n * sv + side);
      }
    } else if (!flips) {
      int cj = s, fj = s;
      if (!interior) {
        bool f, z;
        cj = map_cell(s, my, f);
        fj = map_face(s, my, f, z);
      }
      const double* q = wg + cj * nx + ci;
#pragma unroll
      for (int n = 0; n < NM; ++n) split::cpa::copy8(r + n * RW, q + n * sv);
      split::cpa::copy8(r + 9 * RW, bg + cj * nx + fi);
      split::cpa::copy8(r + 10 * RW, bg + sv + fj * nx + ci);
      split::cpa::copy8(r + 11 * RW, bg + 2 * sv + cj * nx + ci);
    } else {
      double v[NM];
      load_prim_all(I, wg, i, s, mx, my, false, v);
#pragma unroll
      for (int n = 0; n < NM; ++n) r[n * RW] = v[n];
      r[9 * RW] = load_face<0>(I, bg, i, s, mx, my, false);
      r[10 * RW] = load_face<1>(I, bg, i, s, mx, my, false);
      r[11 * RW] = load_face<2>(I, bg, i, s, mx, my, false);
    }
  };
  const double gm1i = 1. / (I.gam - 1.);
  const double dz = I.dlf2;
  double dx = 0., idx = 0.;
  if (own) {
    dx = I.dlf[0][i];
    idx = I.dlf_inv[0][i];
  }
  const int i2 = I.ng + I.N[0] - 1, j2 = I.ng + I.N[1] - 1;
  const CorrInGlobal in{&I, I.w[parity], I.b[parity], nullptr};
  unsigned e = 0;
  double cmax = 0.;
  const int ye = T.y0 + T.wy;
  if (ORDER) {
    load(rm, T.y0 - 2);
    load(rc, T.y0 - 1);
    load(rn, T.y0);
    split::cpa::commit();
  } else {
    load(rc, T.y0 - 1);
    split::cpa::commit();
    load(rn, T.y0);
    split::cpa::commit();
  }
  for (int s = T.y0 - 1; s <= ye; ++s) {
    const bool upper = s >= T.y0;    // the y face below row s is formed
    const bool fin = s > T.y0;       // row s - 1 is finished
    double bnx = 0., bny = 0.;
    if (ORDER) {
      if (col) {
        bnx = bg[s * nx + i];
        bny = bg[sv + s * nx + i];
      }
      split::cpa::wait<0>();
    } else {
      split::cpa::wait<1>();
    }
    __syncwarp();
    if (!ORDER) {
      bnx = rc[9 * RW];
      bny = rc[10 * RW];
    }
    if (ORDER) {
      if (col) {
#pragma unroll
        for (int n = 0; n < NM; ++n) {
          if (n == BX) continue;
          const int o = plain::perm<1>(n) * RW;
          sD[slot8(n) * 32] = half_slope<LIM>(rm[o], rc[o], rn[o]);
        }
      }
      // row s - 1 is done with (its x slopes were formed a step ago)
      if (s + 2 <= ye + 1) load(rm, s + 2);
      split::cpa::commit();
      // the step's input for the next row's update, into L2
      if (own && s >= T.y0 && s < ye) {
        const long long c = s * nx + i;
#pragma unroll
        for (int n = 0; n < NM; ++n) split::prefetch_l2(I.w[parity] + n * sv + c);
#pragma unroll
        for (int n = 0; n < 3; ++n) split::prefetch_l2(I.b[parity] + n * sv + c);
      }
    }
    // y faces below row s, and the y part of row s - 1's update
    double fybx = 0.;
    if (upper) {
      double f[NM];
#pragma unroll
      for (int n = 0; n < NM; ++n) f[n] = 0.;
      if (col) face_flux<RS>(f, WalkY<ORDER>{ORDER ? sL : rm, rc, sD}, bny, I.gam, gm1i, e);
      // local -> global (godunov.pyx:297-324 for the y sweep)
      const double fy[7] = {f[RHO], f[VZ], f[VX], f[VY], f[EN], f[PSC], f[BY]};
      fybx = f[BZ];
      if (fin && own) {
        const int j = s - 1;
        double wn[NM], un[NM];
        if (ORDER) {
          in.wn(i, j, wn);
        } else {
#pragma unroll
          for (int n = 0; n < NM; ++n) wn[n] = rm[n * RW];
        }
        prim2cons_g(un, wn, gm1i);
        const double bz0 = ORDER ? I.b[parity][2 * sv + j * nx + i] : rm[11 * RW];
#if BNZ_FAST_MATH
        const double idy = I.dlf_inv[1][j], idz = 1. / dz;
        const double dtdv = dt * idx * idy * idz;
        const double dtda = dt * idx * idy;
#else
        const double dy = I.dlf[1][j];
        const double vol = dx * dy * dz;
        const double dtdv = dt / vol;
        const double dtda = dt / (dx * dy);
#endif
        const double day = dx * dz;
#pragma unroll
        for (int n = 0; n < 6; ++n) {
          // (the predictor's un is rounded first, as the tile kernel's is)
          double v = BNZ_FAST_MATH && ORDER == 0 ? fma(-dtdv, sv_[(SV_U + n) * 32], un[n])
                                                 : un[n] - dtdv * sv_[(SV_U + n) * 32];
          v -= dtdv * (day * fy[n] - day * sv_[(SV_FY + n) * 32]);
          sv_[(SV_U + n) * 32] = v;
        }
        const double exb = -sv_[(SV_FY + 6) * 32], ext = -fy[6];
        double bz = bz0 - dtda * sv_[SV_BZ * 32];
        bz += dtda * (dx * ext - dx * exb);
        sv_[SV_BZ * 32] = bz;
      }
#pragma unroll
      for (int n = 0; n < 7; ++n) sv_[(SV_FY + n) * 32] = fy[n];
    }
    if (ORDER) {
      if (col) {
        // the lower state of the next y face, then the x slopes
#pragma unroll
        for (int n = 0; n < NM; ++n) {
          if (n == BX) continue;
          sL[slot8(n) * 32] = rc[plain::perm<1>(n) * RW] + sD[slot8(n) * 32];
        }
#pragma unroll
        for (int n = 0; n < NM; ++n) {
          if (n == BX) continue;
          sD[slot8(n) * 32] = half_slope<LIM>(rc[n * RW - 1], rc[n * RW], rc[n * RW + 1]);
        }
      }
      __syncwarp();
    }
    // x faces of row s
    double f[NM];
#pragma unroll
    for (int n = 0; n < NM; ++n) f[n] = 0.;
    if (xface) face_flux<RS>(f, WalkX<ORDER>{rc, sD}, bnx, I.gam, gm1i, e);
    // cell EMF of row s (ct.pyx:148) and the corner EMF (i, s) (ct.pyx:204-207)
    double ec = 0.;
    if (col) {
      const double vx = rc[VX * RW], vy = rc[VY * RW], bxc = rc[BX * RW], byc = rc[BY * RW];
      ec = -(vx * byc - vy * bxc);
    }
    const double ecp = sv_[SV_EC * 32];
    const double fybxl = __shfl_up_sync(0xffffffffu, fybx, 1);
    const double ecl = __shfl_up_sync(0xffffffffu, ec, 1), ecpl = __shfl_up_sync(0xffffffffu, ecp, 1);
    // (explicit additions: the tile kernels read these terms from shared
    // memory, so none is contracted with the product it comes from)
    const double es = __dadd_rn(__dadd_rn(__dsub_rn(-sv_[SV_FXBY * 32], f[BY]), fybxl), fybx);
    const double cs = __dadd_rn(__dadd_rn(__dadd_rn(ecl, ec), ecpl), ecp);
    const double ez = 0.5 * es - 0.25 * cs;
    const double e00 = sv_[SV_EZ * 32], e01 = ez;
    const double e10 = __shfl_down_sync(0xffffffffu, e00, 1), e11 = __shfl_down_sync(0xffffffffu, e01, 1);
    if (fin && own) {
      // row s - 1: the faces (ct.pyx:15-91), face-to-cell B (ct.pyx:96-123),
      // sources and cons2prim, as stage_cell
      const int j = s - 1;
      const long long c = j * nx + i;
      double bxl0, bxr0, byb0, byt0;
      if (ORDER) {
        const bool edge = (i == i2) || (j == j2) || (i == I.ng) || (j == I.ng);
        bxl0 = in.face(0, i, j, edge, mx, my);
        bxr0 = in.face(0, i + 1, j, edge, mx, my);
        byb0 = in.face(1, i, j, edge, mx, my);
        byt0 = in.face(1, i, j + 1, edge, mx, my);
      } else {
        bxl0 = rm[9 * RW];
        bxr0 = rm[9 * RW + 1];
        byb0 = rm[10 * RW];
        byt0 = rc[10 * RW];
      }
#if BNZ_FAST_MATH
      const double idy = I.dlf_inv[1][j], idz = 1. / dz;
      double dtda = dt * idy * idz;
#else
      const double dy = I.dlf[1][j];
      double dtda = dt / (dy * dz);
#endif
      const double bxl = bxl0 - dtda * (dz * e01 - dz * e00);
      const double bxr = bxr0 - dtda * (dz * e11 - dz * e10);
#if BNZ_FAST_MATH
      dtda = dt * idx * idz;
#else
      dtda = dt / (dx * dz);
#endif
      const double byb = byb0 + dtda * (dz * e10 - dz * e00);
      const double byt = byt0 + dtda * (dz * e11 - dz * e01);
      double u[NM];
#pragma unroll
      for (int n = 0; n < 6; ++n) u[n] = sv_[(SV_U + n) * 32];
      const double bz = sv_[SV_BZ * 32];
      u[BX] = ((I.lv[0][i] - I.lf[0][i]) * bxl + (I.lf[0][i + 1] - I.lv[0][i]) * bxr) * I.dlf_inv[0][i];
      u[BY] = ((I.lv[1][j] - I.lf[1][j]) * byb + (I.lf[1][j + 1] - I.lv[1][j]) * byt) * I.dlf_inv[1][j];
      u[BZ] = bz;
      if (I.src) {
        // integrator.pyx:132-170 with the stage input's state
        double fd[3];
        if (I.fdriv) {
          fd[0] = I.fdriv[c];
          fd[1] = I.fdriv[sv + c];
          fd[2] = I.fdriv[2 * sv + c];
        }
        const bool grav = I.grav[0] != 0. || I.grav[1] != 0. || I.grav[2] != 0.;
        double w0[4];
#pragma unroll
        for (int n = 0; n < 4; ++n) w0[n] = ORDER ? wg[n * sv + c] : rm[n * RW];
        srcterm::apply(u, w0[RHO], w0[VX], w0[VY], w0[VZ], I.grav, grav, I.fdriv ? fd : nullptr, dt);
      }
      double o[NM];
      cons2prim(o, u, I.gam);
      double* __restrict__ w1 = ORDER ? I.w[parity ^ 1] : I.ws;
      double* __restrict__ b1 = ORDER ? I.b[parity ^ 1] : I.bs;
#pragma unroll
      for (int n = 0; n < NM; ++n) w1[n * sv + c] = o[n];
      b1[c] = bxl;
      b1[sv + c] = byb;
      b1[2 * sv + c] = bz;
      if (i == (ORDER ? i2 : I.nx - 2)) b1[c + 1] = bxr;
      if (j == (ORDER ? j2 : I.ny - 2)) b1[sv + c + nx] = byt;
      if (ORDER) {
        e |= plain::check_prim(o);
        // next step's CFL (new_dt.pyx:55-99) on the new state
        const double vf = fms(o, I.gam);
        const double cx = fabs(o[VX]) + vf, cy = fabs(o[VY]) + vf;
#if BNZ_FAST_MATH
        const double cds = fmax(cx * I.dlf_inv[0][i], cy * I.dlf_inv[1][j]);
#else
        const double cds = fmax(fmax(cx / I.dlf[0][i], cy / I.dlf[1][j]), 0. / I.dlf2);
#endif
        if (cds > cmax) cmax = cds;
      }
    }
    if (s < ye) {
      // the x part of row s for the next step
      const double dy = I.dlf[1][s];
      const double dax = dy * dz;
#pragma unroll
      for (int n = 0; n < 6; ++n) {
        const double fr = __shfl_down_sync(0xffffffffu, f[n], 1);
        sv_[(SV_U + n) * 32] = dax * fr - dax * f[n];
      }
      const double eyl = f[BZ], eyr = __shfl_down_sync(0xffffffffu, f[BZ], 1);
      sv_[SV_BZ * 32] = dy * eyr - dy * eyl;
      sv_[SV_FXBY * 32] = f[BY];
      sv_[SV_EC * 32] = ec;
      sv_[SV_EZ * 32] = ez;
    }
    if (!ORDER) {
      // the neighbours' reads of row s - 1 are done: row s + 2 takes its place
      __syncwarp();
      if (s + 2 <= ye) load(rm, s + 2);
      split::cpa::commit();
    }
    double* t = rm;
    rm = rc;
    rc = rn;
    rn = t;
  }
  if (ORDER) {
    for (int o = 16; o > 0; o >>= 1) cmax = fmax(cmax, __shfl_xor_sync(0xffffffffu, cmax, o));
    if (lane == 0 && cmax > 0.)
      atomicMax(&I.ds->cds_bits[parity ^ 1], (unsigned long long)__double_as_longlong(cmax));
  }
  if (e) atomicOr(I.err, e);
}

}  // namespace fused
