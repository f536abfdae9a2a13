// bnz_split_flux.cuh -- the split path's face-flux kernels.
//
// A Riemann solve is a long FP64 dependency chain, so what bounds these
// kernels is how many warps can make progress, not bandwidth.  No thread here
// waits for another warp: there is no block barrier.
//   k_flux_march (y and z sweeps): a thread owns one column of faces along the
//     sweep axis and walks `len` of them.  Its cells live in its own slots of
//     shared memory, filled by 8-byte asynchronous copies (cp.async) one cell
//     ahead, so a cell is loaded once and its PLM half slopes are formed once
//     (by the thread that owns the column); lanes run along x, so that every
//     load and store of a warp is contiguous.
//   k_flux_row (x sweep): a warp walks segments of 32 consecutive cells of the
//     box's rows; neighbours are read from the warp's own shared memory.
// Rows and columns of any length and alignment take the same kernel.
// Measured (256^3, HLLD, PLM, ms per launch): y and z sweeps 0.75, x sweep
// 0.82, where block-wide tiles with barriers between their phases (cells by
// TMA into two buffers) took 1.24 and 1.21; donor cells 0.64 / 0.62 / 0.63
// against 0.71 / 0.76 / 0.68 for one thread per face reading global memory.
// Instructions per PLM face fell from 1240 to 770 (no tile coordinates, one
// slope per face), issue rose from 43 to 47 % of the slots; 16 (PLM march) to
// 20 warps an SM (a spill costs more than the warps it buys there: PLM march at
// 20 warps and 96 registers 0.80).  Characteristic slopes run at 16 warps and
// 128 registers: one 512^2 grid 175 us a step at 12 warps, 169 at 16; 128^3 1521
// and 1471.
// Included inside the per-floating-point-mode namespace, after bnz_plain.cuh.
#pragma once

namespace split {

using namespace dev;

__device__ __forceinline__ int ax_of(int3 v, int a) { return a == 0 ? v.x : a == 1 ? v.y : v.z; }

// slope slot of variable n (the normal field has none)
__device__ __forceinline__ constexpr int slot8(int n) { return n < BX ? n : n - 1; }

// reconstr_c.c:54-91 half slope; in the fast build the van Leer limiter's
// quotient 2ab/(a+b) is 2ab times the Newton-refined reciprocal of a + b
// (bnz_fastmath.cuh: within 2 ulp; ab > 0 makes a and b one-signed, so
// |a + b| >= 2 sqrt(ab) is a normal number)
template <int LIM>
__device__ __forceinline__ double half_slope_split(double wm, double wc, double wp) {
#if BNZ_FAST_MATH
  if (LIM == LIM_VL) {
    const double a = wc - wm, b = wp - wc, ab = a * b;
    return (ab > 0.) ? ab * bnz_nr_rcp(a + b) : 0.;
  }
#endif
  return half_slope<LIM>(wm, wc, wp);
}

namespace cpa {
__device__ __forceinline__ void copy8(double* dst, const double* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
}  // namespace cpa

// values staged per cell: the eight variables a face reads (without the normal
// field; all nine with characteristic slopes), then the face field
template <int CP>
struct RowVars {
  static constexpr int NV = CP ? 10 : 9;
  static constexpr int BF = NV - 1;
  __device__ static constexpr int slot(int n) { return CP ? n : slot8(n); }
};

constexpr int FLUX_NT = 128;

// states of a face in a column walk: lo / hi point at the cells beside it (in
// the thread's slots, FLUX_NT apart); with PLM, lo at the left state and the
// right one is hi minus its slope
template <int ORDER, int CP>
struct ColFace {
  const double *lo, *hi, *d;
  __device__ __forceinline__ static int o(int n) { return RowVars<CP>::slot(n) * FLUX_NT; }
  __device__ __forceinline__ double L(int n) const { return ORDER ? lo[slot8(n) * FLUX_NT] : lo[o(n)]; }
  __device__ __forceinline__ double R(int n) const { return ORDER ? hi[o(n)] - d[slot8(n) * FLUX_NT] : hi[o(n)]; }
  __device__ __forceinline__ double at(bool left, int n) const {
    if (ORDER == 0) return (left ? lo : hi)[o(n)];
    return left ? L(n) : R(n);
  }
};

template <int ORDER, int CP>
struct ColSmem {
  static constexpr int ROWS = 3 * RowVars<CP>::NV * FLUX_NT;
  static constexpr int BYTES = 8 * (ROWS + (ORDER ? 16 * FLUX_NT : 0));
};

// the half slopes of one cell into d, from the staged cells at m, c, p; with
// FIRST == 0 the left state of the next face (wm + the old slope) into l
// (CS, DS: the strides between a cell's variables and between slopes)
template <int LIM, int CP, int CS, int DS>
__device__ __forceinline__ void col_slopes(const double* m, const double* c, const double* p, double* d, double* l,
                                           bool first) {
#pragma unroll
  for (int n = 0; n < NM; ++n) {
    if (n == BX) continue;
    const int o = RowVars<CP>::slot(n) * CS, s = slot8(n) * DS;
    const double wm = m[o], wc = c[o], wp = p[o];
    if (!first) l[s] = wm + d[s];
    d[s] = half_slope_split<LIM>(wm, wc, wp);
  }
}

template <int LIM, int CS, int DS>
__device__ __forceinline__ void col_slopes_char(const double* m, const double* c, const double* p, double* d, double* l,
                                                bool first, double gam) {
  double wm[NM], wc[NM], wp[NM], h[NM];
#pragma unroll
  for (int n = 0; n < NM; ++n) {
    wm[n] = m[n * CS];
    wc[n] = c[n * CS];
    wp[n] = p[n * CS];
  }
  half_slopes_char<LIM>(wm, wc, wp, gam, h);
#pragma unroll
  for (int n = 0; n < NM; ++n) {
    if (n == BX) continue;
    if (!first) l[slot8(n) * DS] = wm[n] + d[slot8(n) * DS];
    d[slot8(n) * DS] = h[n];
  }
}

template <int CP, int CS, int DS>
__device__ __forceinline__ void col_slopes_rt(int lim, const double* m, const double* c, const double* p, double* d,
                                              double* l, bool first, double gam) {
  if constexpr (CP) {
    if (lim == LIM_MC) col_slopes_char<LIM_MC, CS, DS>(m, c, p, d, l, first, gam);
    else if (lim == LIM_MM) col_slopes_char<LIM_MM, CS, DS>(m, c, p, d, l, first, gam);
    else col_slopes_char<LIM_VL, CS, DS>(m, c, p, d, l, first, gam);
  } else {
    if (lim == LIM_MC) col_slopes<LIM_MC, CP, CS, DS>(m, c, p, d, l, first);
    else if (lim == LIM_MM) col_slopes<LIM_MM, CP, CS, DS>(m, c, p, d, l, first);
    else col_slopes<LIM_VL, CP, CS, DS>(m, c, p, d, l, first);
  }
}

// Fluxes of the AX faces (AX = 1, 2) of `box` (face index along AX = the cell
// on its right), in the global variable order (the normal field entry, which
// nothing reads, is not stored).  ORDER 0: donor cell (reconstr_c.c:8-22);
// ORDER 1: PLM with limiter lim (reconstr_c.c:29-91), in characteristic
// variables with CP.  Normal field from the face array bf.  The columns of the
// (x, other axis) plane of the box are cut into `parts` walks of `len` faces;
// the threads take the walks of all columns part by part, so that a plane of
// few columns still fills its blocks.
template <int AX, int ORDER, int RS, int CP>
__global__ void __launch_bounds__(FLUX_NT, ORDER ? 4 : 5)
    k_flux_march(GridDev g, const double* __restrict__ w, const double* __restrict__ bf, double* __restrict__ F,
                 plain::Box box, int lim, int len, int parts, unsigned* err) {
  using V = RowVars<CP>;
  constexpr int ST = FLUX_NT, RS_ = V::NV * ST;  // stride between a thread's values, between its rows
  constexpr int OAX = AX == 1 ? 2 : 1;
  extern __shared__ __align__(16) double flux_smem[];
  const int nxb = box.hi.x - box.lo.x + 1, no = ax_of(box.hi, OAX) - ax_of(box.lo, OAX) + 1;
  const unsigned t = blockIdx.x * ST + threadIdx.x, ncol = (unsigned)nxb * no;
  const int part = (int)(t / ncol), col = (int)(t - part * ncol);
  if (part >= parts) return;
  const int i = box.lo.x + col % nxb, o = ax_of(box.lo, OAX) + col / nxb;
  const int a0 = ax_of(box.lo, AX) + part * len, a1 = min(a0 + len - 1, ax_of(box.hi, AX));
  const long long sv = g.sv, sy = g.nx, sz = (long long)g.nx * g.ny;
  const long long sa = AX == 1 ? sy : sz, so = AX == 1 ? sz : sy;
  const long long c0 = i + o * so;
  double* r0 = flux_smem + threadIdx.x;  // rows of the cells f-1, f, f+1, in turn
  double* r1 = r0 + RS_;
  double* r2 = r1 + RS_;
  double* d = flux_smem + ColSmem<ORDER, CP>::ROWS + threadIdx.x;
  double* l = d + 8 * ST;
  auto row = [&](double* dst, int a) {
    const double* q = w + c0 + a * sa;
#pragma unroll
    for (int n = 0; n < NM; ++n) {
      if (n == BX && !CP) continue;
      cpa::copy8(dst + V::slot(n) * ST, q + plain::perm<AX>(n) * sv);
    }
    cpa::copy8(dst + V::BF * ST, bf + AX * sv + c0 + a * sa);
  };
  const double gm1i = 1. / (g.gam - 1.);
  unsigned e = 0;
  if (ORDER) {
    // the slope of the first face's left cell
    row(r0, a0 - 2);
    row(r1, a0 - 1);
    row(r2, a0);
    cpa::commit();
    cpa::wait<0>();
    col_slopes_rt<CP, ST, ST>(lim, r0, r1, r2, d, l, true, g.gam);
    row(r0, a0 + 1);
    cpa::commit();
    double* q = r0;
    r0 = r1;
    r1 = r2;
    r2 = q;
  } else {
    row(r0, a0 - 1);
    row(r1, a0);
    cpa::commit();
    if (a0 < a1) row(r2, a0 + 1);
    cpa::commit();
  }
  for (int f = a0; f <= a1; ++f) {
    if (ORDER) {
      // cell f + 1 has arrived: the slope of cell f, the left state of face f;
      // cell f - 1 is not needed any more and makes room for cell f + 2
      cpa::wait<0>();
      col_slopes_rt<CP, ST, ST>(lim, r0, r1, r2, d, l, false, g.gam);
      if (f < a1) row(r0, f + 2);
    } else {
      cpa::wait<1>();  // all but the newest copy: cell f has arrived
    }
    double fl[NM];
    face_flux<RS>(fl, ColFace<ORDER, CP>{ORDER ? l : r0, r1, d}, r1[V::BF * ST], g.gam, gm1i, e);
    double* Fc = F + c0 + f * sa;
#pragma unroll
    for (int n = 0; n < NM; ++n)
      if (n != BX) Fc[plain::perm<AX>(n) * sv] = fl[n];
    if (!ORDER && f + 2 <= a1) row(r0, f + 2);
    cpa::commit();
    double* q = r0;
    r0 = r1;
    r1 = r2;
    r2 = q;
  }
  if (e) atomicOr(err, e);
}

// states of an x face: the cells at p - 1 and p of the warp's segment, their
// slopes at d - 1 and d
template <int ORDER, int CP, int SW>
struct RowFace {
  const double *p, *d;
  __device__ __forceinline__ static int o(int n) { return RowVars<CP>::slot(n) * SW; }
  __device__ __forceinline__ double L(int n) const { return ORDER ? p[o(n) - 1] + d[slot8(n) * 32 - 1] : p[o(n) - 1]; }
  __device__ __forceinline__ double R(int n) const { return ORDER ? p[o(n)] - d[slot8(n) * 32] : p[o(n)]; }
  __device__ __forceinline__ double at(bool left, int n) const {
    const double v = (left ? p - 1 : p)[o(n)];
    if (ORDER == 0) return v;
    return fma(left ? 1. : -1., (left ? d - 1 : d)[slot8(n) * 32], v);
  }
};

template <int ORDER, int CP>
struct RowSmem {
  static constexpr int SW = 34;  // a segment: 32 cells and one on either side
  static constexpr int SEG = RowVars<CP>::NV * SW;
  static constexpr int WARP = 2 * SEG + (ORDER ? 8 * 32 : 0);  // doubles per warp
  static constexpr int BYTES = 8 * WARP * (FLUX_NT / 32);
};

// Fluxes of the x faces of `box`, as k_flux_march forms them.  The rows of the
// box are laid end to end as entries: the cells from one (ORDER 0) or two
// (ORDER 1) left of the first face's right cell to the last one a slope needs.
// A warp takes 32 consecutive entries at a time, the next ones copied in while
// it computes: with PLM every lane forms its cell's slope and lanes 1 .. 31
// the face on its left (the next segment starts at this one's last entry), so
// 31 faces a segment; with donor cells all 32.  Warp q walks `len` segments.
template <int ORDER, int RS, int CP>
__global__ void __launch_bounds__(FLUX_NT, CP ? 4 : 5)
    k_flux_row(GridDev g, const double* __restrict__ w, const double* __restrict__ bf, double* __restrict__ F,
               plain::Box box, int lim, int len, unsigned* err) {
  using V = RowVars<CP>;
  using M = RowSmem<ORDER, CP>;
  constexpr int SW = M::SW, STEP = ORDER ? 31 : 32;
  extern __shared__ __align__(16) double flux_smem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double* seg0 = flux_smem + wid * M::WARP;
  double* d = seg0 + 2 * M::SEG + lane;
  const int x0 = box.lo.x - 1 - ORDER;                  // the cell of entry 0 of a row
  const int P = box.hi.x + ORDER - x0 + 1;              // entries of a row
  const int nyb = box.hi.y - box.lo.y + 1;
  const long long nent = (long long)P * nyb * (box.hi.z - box.lo.z + 1);
  const long long v0 = ((long long)blockIdx.x * (FLUX_NT / 32) + wid) * len * STEP;  // the warp's first entry
  if (v0 >= nent) return;
  const long long sv = g.sv;
  // this lane's entry: position in its row, row's cell index base, row number
  unsigned r = (unsigned)((v0 + lane) / P);
  int ent = (int)((v0 + lane) - (long long)r * P);
  int j = box.lo.y + (int)(r % nyb), k = box.lo.z + (int)(r / nyb);
  long long c = ((long long)k * g.ny + j) * g.nx + x0 + ent;
  auto advance = [&](int by) {
    ent += by;
    c += by;
    while (ent >= P) {
      ent -= P;
      c += g.nx - P;
      if (++j > box.hi.y) {
        j = box.lo.y;
        ++k;
        c += (long long)(g.ny - nyb) * g.nx;
      }
    }
  };
  // copies the lane's entry (and the ones beside the segment) into segment s
  auto load = [&](double* s) {
    if (k > box.hi.z) return;
    const double* q = w + c;
    double* t = s + lane + 1;
#pragma unroll
    for (int n = 0; n < NM; ++n) {
      if (n == BX && !CP) continue;
      cpa::copy8(t + V::slot(n) * SW, q + n * sv);
    }
    if (ent > ORDER) cpa::copy8(t + V::BF * SW, bf + c);
    const int side = lane == 0 && ent > 0 ? -1 : ORDER && lane == 31 && ent < P - 1 ? 1 : 0;
    if (side) {
#pragma unroll
      for (int n = 0; n < NM; ++n) {
        if (n == BX && !CP) continue;
        cpa::copy8(t + V::slot(n) * SW + side, q + n * sv + side);
      }
    }
  };
  const double gm1i = 1. / (g.gam - 1.);
  unsigned e = 0;
  load(seg0);
  cpa::commit();
  for (int m = 0; m < len; ++m) {
    double* s = seg0 + (m & 1) * M::SEG;
    const bool in = k <= box.hi.z;
    const int en = ent;
    const long long cc = c;
    // the next segment (one warp's segments follow each other; the other
    // buffer's last readers passed the barrier that ended the last segment)
    advance(STEP);
    if (m + 1 < len) load(seg0 + ((m & 1) ^ 1) * M::SEG);
    cpa::commit();
    cpa::wait<1>();
    __syncwarp();
    const double* p = s + lane + 1;
    if (ORDER) {
      if (in && en > 0 && en < P - 1)
        col_slopes_rt<CP, SW, 32>(lim, p - 1, p, p + 1, d, nullptr, true, g.gam);
      __syncwarp();
    }
    if (in && (ORDER ? lane > 0 && en > 1 && en < P - 1 : en > 0)) {
      double fl[NM];
      face_flux<RS>(fl, RowFace<ORDER, CP, SW>{p, d}, p[V::BF * SW], g.gam, gm1i, e);
#pragma unroll
      for (int n = 0; n < NM; ++n)
        if (n != BX) F[n * sv + cc] = fl[n];
    }
    __syncwarp();
  }
  if (e) atomicOr(err, e);
}

}  // namespace split
