// bnz_common.h -- structures shared by the host context and the kernels.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include "../../include/bnz_gpu.h"

// Grid geometry as the kernels see it.  Index conventions follow the
// reference's GridCoord (src/coordinates/coord_c.h:19-99): Ntot cells per axis
// including ng ghosts on active axes, active range i1..i2 / j1..j2 / k1..k2,
// per-axis spacing arrays indexed by the cell index along that axis.
struct GridDev {
  int nx, ny, nz;     // Ntot per axis
  int dims, ng;
  int i1, i2, j1, j2, k1, k2;
  long long sv;       // stride between variables: nx*ny*nz
  double gam;
  const double* dlf[3];      // face spacing lf[i+1]-lf[i]
  const double* dlf_inv[3];
  const double* lf[3];       // face coordinates (Ntot+1 entries)
  const double* lv[3];       // volume (centre) coordinates
  const double* dlv_inv[3];  // inverse centre spacing
};

// Device buffers and options used by one step of one grid.
struct StepArgs {
  GridDev g;
  double* prim;
  double* cons;
  double* bfld;
  double* cons_s;  // predictor conserved state (plain path)
  double* bfld_s;  // predictor face field (plain path)
  double* flx[3];  // Godunov fluxes (plain path)
  double* ec;      // cell-centred E (plain path)
  double* ee;      // edge E (plain path)
  double* wnext;   // fused path: output prim buffer
  double* bnext;   // fused path: output face-B buffer
  unsigned* err;   // sticky device error word
  int rsolver, reconstr_order, limiter, charact_proj;
  int bc[3][2];
  int face_aware;
  cudaStream_t stream;
  // source terms: constant gravity and the driving force field (3 x Ntot)
  double grav[3];
  const double* fdriv;
  int src;  // any source term on
  int hydro;  // the reference's hydro build (MFIELD 0): no field, no CT
  // split path, 3D grids with even Ntot_x: the tensor maps of the update
  // kernel's TMA boxes (split::TM_COUNT maps of 128 bytes), or null
  const unsigned char* smaps;
};

// Device time-step record used by graph-captured stepping.
struct DtState {
  double dt;          // step used by the current step
  double time;        // simulation time after the last completed step
  double tmax;        // clip target
  unsigned long long cdsmax_bits;  // max of (|v|+cf)/dx as a bit pattern
  long long step;
  unsigned long long cds_bits[2];  // fused path: CFL max of the state of parity p
  unsigned long long cfl_bits;     // k_cfl_dt: the blocks' maximum so far, zero between launches
  unsigned cfl_done;               // k_cfl_dt: blocks that have added theirs, zero between launches
};

// Fused 2D path: one grid ("instance") of a batch, as the kernels see it.
struct FusedInst {
  int nx, ny;          // Ntot (x, y)
  int N[2];            // active cells
  int ng;
  long long sv;        // variable stride nx*ny
  double gam;
  int bc[2][2];
  int face_aware;
  const double* dlf[2];
  const double* dlf_inv[2];
  const double* lf[2];
  const double* lv[2];
  double dlf2;         // z extent of the single z cell
  double* w[2];        // prim, ping-pong by step parity
  double* b[2];        // face field, ping-pong
  double* ws;          // predictor prim
  double* bs;          // predictor face field
  DtState* ds;
  unsigned* err;       // the instance's sticky error word
  double grav[3];      // source terms (gravity, driving force field or null)
  const double* fdriv;
  int src;
};

// Fused 3D path: one grid of a 3D batch (or a single 3D context).
struct FusedInst3 {
  int nx, ny, nz;      // Ntot per axis
  int N[3];            // active cells
  int ng;
  long long sv;        // variable stride nx*ny*nz
  double gam;
  int bc[3][2];
  int face_aware;
  const double* dlf[3];
  const double* dlf_inv[3];
  const double* lf[3];
  const double* lv[3];
  double* w[2];        // prim, ping-pong by step parity
  double* b[2];        // face field, ping-pong
  double* ws;          // predictor prim
  double* bs;          // predictor face field
  DtState* ds;
  unsigned* err;
  double grav[3];
  const double* fdriv;
  int src;
};

// Chunk shape of the 3D kernels: at most F3_TX x F3_TY cells in x, y and about
// F3_KZ planes (16 x 8 on one 512-thread block per SM: the flux phase of a
// plane is one round, and the halo recompute of x and y faces stays at one
// Riemann solve per cell and direction plus a third); the corrector's TMA box
// of ws covers the chunk plus two cells each side from an even column:
// F3_BW x F3_BH cells, one plane, 9 fields.
constexpr int F3_TX = 16, F3_TY = 8, F3_KZ = 64;
constexpr int F3_BW = (F3_TX + 6) & ~1, F3_BH = F3_TY + 4;

// A column chunk of a 3D grid: cells [x0, x0+wx) x [y0, y0+wy) x [z0, z0+wz).
struct FusedTile3 {
  int inst;
  int x0, y0, z0;
  int wx, wy, wz;
  int tma;  // the corrector stages ws by TMA (the instance has a tensor map)
};

struct Fused3Launch {
  const FusedInst3* insts;
  int ninst;
  const FusedTile3* tilesA;  // predictor chunks (cells 1..Ntot-2 of each axis)
  int ntA;
  const FusedTile3* tilesB;  // corrector chunks (active cells)
  int ntB;
  int rsolver, limiter, charact_proj;
  double cour;
  int dt_mode;
  double dt_fixed;
  const unsigned char* wsmaps;  // per-instance 4D tensor maps of ws (128 bytes each), or null
  cudaStream_t stream;
  cudaEvent_t* events;  // optional: before dt, predictor, corrector and after (timing)
};

// A tile of cells [x0, x0+wx) x [y0, y0+wy) (array coordinates) of one instance.
struct FusedTile {
  int inst;
  int x0, y0;
  int wx, wy;
  int tma;  // the instance has a tensor map of its ws (persistent corrector)
};

// Variants of the fused kernels the autotuner chooses from: tile shape
// (cells along x, y), whether the predictor stages its input cells in shared
// memory, and whether the stages run as persistent TMA-fed kernels.  A batch
// starts on variant 8 (persistent, 15 x 14) or, a large one, on the walks
// (WALK_VARIANT), a single grid on what grid_variant picks.
struct FusedVariant {
  int tx, ty, staged, persistent;
};
// 15 x 14 tiles give 256 x faces and 255 y faces per interior tile: each flux
// phase of a 256-thread block is one full round (32 x 8 leaves 40% of the
// threads idle in the second round of each phase).
// The persistent variants run the corrector (persistent = 1) or both stages
// (2) as one resident grid fed by a tile queue, with TMA double-buffering of
// the staged input (15 x 14 only: two blocks of those kernels fit one SM's
// shared memory).
// 14 x 14 tiles (variant 9) make every phase of the corrector at most one
// round: 256 slope cells, 240 x and 240 y faces, 225 corners, 196 cells.
constexpr int FUSED_NVARIANT = 10;
constexpr FusedVariant FUSED_VARIANTS[FUSED_NVARIANT] = {
    {32, 8, 0, 0}, {32, 8, 1, 0}, {16, 16, 0, 0}, {16, 16, 1, 0}, {15, 14, 0, 0},
    {15, 14, 1, 0}, {15, 14, 0, 1}, {15, 14, 1, 1}, {15, 14, 0, 2}, {14, 14, 0, 2}};

// Variants built for a Riemann solver: all for HLLD; the default and the
// persistent variants 8 and 9 for the others.
inline bool fused_variant_built(int v, bool hlld) {
  return v == 0 || v == 8 || v == 9 || (hlld && v > 0 && v < FUSED_NVARIANT);
}

// Variant number of the strip walks (bnz_walk2d.cuh), which have no tile shape
// of their own: strips of up to WALK_COLS columns and walk_rows rows, for every
// Riemann solver and limiter, without characteristic slopes.
constexpr int WALK_VARIANT = FUSED_NVARIANT, WALK_COLS = 30;
// Tiles of a batch that does not walk, and of the parts of one that does.
constexpr int BATCH_TILE_VARIANT = 8;

// Walks or tiles (no characteristic slopes in the walks): walks need enough
// strips to fill the device, and strips that are not much narrower than a warp.
constexpr long long WALK_MIN_BATCH = 1500000, WALK_MIN_GRID = 250000;
// Rows of a strip: as many as leave every SM's 12 warps five strips each (a
// strip forms its lowest row's faces besides its own), 8 to 32.
inline int walk_rows(long long zones, int nsm) {
  const long long r = zones / ((long long)WALK_COLS * 12 * 5 * nsm);
  return (int)(r < 8 ? 8 : r > 32 ? 32 : r);
}
// Rows that the warps walk over n0 x n1 cells, a strip's two extra ones included.
inline long long walk_steps(int n0, int n1, int rows) {
  return (long long)((n0 + WALK_COLS - 1) / WALK_COLS) * (n1 + 2 * ((n1 + rows - 1) / rows));
}
inline long long tile_count(int n0, int n1, const FusedVariant& v) {
  return (long long)((n0 + v.tx - 1) / v.tx) * ((n1 + v.ty - 1) / v.ty);
}
// A batch walks from WALK_MIN_BATCH zones, when `steps` rows of warps (both
// stages) stand against enough of the `tiles` of variant 8.  Measured, time by
// walks over time by tiles at steps / tiles: HLLD 7.6 0.87 (256^2 grids, 5 M
// zones), 8.2 0.62 (31^2), 8.5 0.93, 8.9 0.99 (64^2, 5 M), 9.1 1.02 (128^2, 1.6
// M) and 0.96 (40^2, 5 M), 9.3 0.67 (31^2, 1.6 M), 9.5 1.03 (64^2, 3 M), 10.0
// 1.07, 11.2 1.10 (40 x 200); HLL 8.5 0.91, 9.1 1.00, 9.5 0.99 and 0.96, 10.0
// 1.05; HLLT, whose walks cost most, 7.6 0.97, 8.0 0.92 (24^2), 8.1 1.04, 8.6
// 1.12, 10.0 1.22.  Below 1.5 M zones the persistent tiles lead: at 0.94 M
// zones of blasts 423 us a step against 441.
inline bool batch_walks(int rsolver, long long zones, long long steps, long long tiles) {
  const double most = rsolver == BNZ_RS_HLLD ? 9.4 : rsolver == BNZ_RS_HLLT ? 8. : 9.6;
  return zones >= WALK_MIN_BATCH && steps <= most * tiles;
}
// What a single grid runs on.
// Walks from WALK_MIN_GRID cells, us a step by walks / by 32 x 8 tiles of one
// grid alone: HLLD 384^2 139 / 104, 500^2 130 / 154, 512^2 133 / 167, 1024^2 411
// / 596, 80000 x 4 196 / 368; where strips are half empty and tiles full, tiles:
// 31 x 10000 283 / 269 (20 steps a tile; the others up to 11).  HLLT 500^2 182 /
// 166, 512^2 186 / 179, 576^2 204 / 225 (1296 tiles), so from 8 tiles an SM.
// Tiles: the kernels end a phase in a barrier, and the phases of 14 x 14 tiles
// are one round of a block's threads, those of 32 x 8 two.  Where 14 x 14 fit
// one wave (two blocks an SM), or neither shape does and there are at most 1.4
// times as many (1.75 on tall grids, whose 32 x 8 tiles are slower), 14 x 14;
// us a step, 32 x 8 / 14 x 14, one grid alone (in brackets three in flight):
// 64^2 52 / 36 (19 / 13), 224^2 58 / 40 (28 / 26), 256^2, 361 tiles against 256,
// 58 / 64 (34 / 35), 288^2 88 / 67 (43 / 42), 384^2 104 / 95 (78 / 78), 4000 x
// 60, 1.43 times, 149 / 153 (138 / 155), 60 x 4000 197 / 162 (173 / 154), 15000
// x 20 with characteristic slopes, 1.52 times, 236 / 282.  Three grids of 2000 x
// 16 at once pay for the one that gains alone: 54 / 39 (24 / 28).
inline int grid_variant(int n0, int n1, int rsolver, bool charact, int nsm) {
  const long long zones = (long long)n0 * n1;
  const long long t14 = tile_count(n0, n1, FUSED_VARIANTS[9]), t32 = tile_count(n0, n1, FUSED_VARIANTS[0]);
  if (zones >= WALK_MIN_GRID && !charact && walk_steps(n0, n1, walk_rows(zones, nsm)) <= 14 * t32 &&
      (rsolver != BNZ_RS_HLLT || t32 >= 8LL * nsm))
    return WALK_VARIANT;
  if (t14 <= 2 * nsm) return 9;
  if (t32 <= 2 * nsm) return 0;
  return t14 <= (n1 > n0 ? 1.75 : 1.4) * t32 ? 9 : 0;
}

// dt modes of the fused step
enum { FDT_CFL = 0, FDT_EXPLICIT = 1, FDT_FIXED = 2 };

struct FusedLaunch {
  const FusedInst* insts;   // indexed by the tiles' instance numbers
  int ninst;                // the per-instance launches cover insts[inst0 .. inst0+ninst-1]
  int inst0;
  const FusedTile* tilesA;  // predictor tiles (cells 1..Ntot-2 of each axis)
  int ntA;
  const FusedTile* tilesB;  // corrector tiles (active cells)
  int ntB;
  int rsolver, limiter, charact_proj;
  int variant;  // of FUSED_VARIANTS, or WALK_VARIANT (the tiles are strips)
  double cour;
  int dt_mode;
  double dt_fixed;
  unsigned* err;
  cudaStream_t stream;
  // persistent kernels: per-instance tensor maps (128 bytes each) of ws
  // (corrector) and of w[0], w[1] (predictor), and the two work-queue
  // counters (corrector, predictor); null where the variant does not use them
  const unsigned char* wsmaps;
  const unsigned char* wmaps;
  unsigned* queue;
  int withhold;  // test switch: the persistent kernels' TMA loads are not issued
  // optional: events recorded before k_dt_batch, before the predictor, before
  // the corrector and after it (kernel timing; null in normal stepping)
  cudaEvent_t* events;
};

// One reverse (adjoint) step of the fused 2D path: the recorded forward
// values, the incoming and outgoing cotangents and the scratch.
struct AdjStep {
  const double* Wn;   // w^n, b^n (the step's input state)
  const double* Bn;
  const double* Ws;   // ws, bs (the predictor's output for that state)
  const double* Bs;
  const double* W1;   // w^(n+1) (the step's output prim)
  double* G1w;        // cotangent of the output (folded in place first)
  double* G1b;
  double* Vw;         // out: cotangent of the input state (9 + 3 fields)
  double* Vb;
  double* Wsb;        // scratch: 9, 3, 9, 1 and 72 fields of Ntot cells
  double* Bsb;
  double* Ub;
  double* Eb;
  double* Q;
  double dt;
  int rsolver, limiter;
  int charact;        // the corrector's slopes are projected (charact_proj)
  int fold_in;        // fold G1 first (it may carry ghost entries)
  int clear_bsb;      // zero Bsb first (the first reverse step of a pass)
  cudaStream_t stream;
};

// Turbulence driving (turb_driv.pyx): force field, this step's mode
// amplitudes (device), base wavenumbers 2 pi / L and the OU parameters.
struct DriveArgs {
  double* fdriv;
  const double* modes;
  int nmod;
  double k0[3];
  double tau, f0;
};

// Conduction scratch (thcond_elec.pyx DiffScratch).
struct DiffArgs {
  double* temp;
  double* fx;
  double* fy;
  double* fz;
  double* pres0;
  double* presm1;
  double* dtemp;
  double* dtemp0;
  double kappa0;
  int aniso, sat;
  double cour_diff;
};
