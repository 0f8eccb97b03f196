// One fused Runge-Kutta stage of the finite-volume step on a structured box:
//   load state (C2P + clip on the fly) -> MUSCL slopes + face states with the
//   reference's revert rules -> numerical fluxes on every face once ->
//   per-cell residual in the reference's summation order -> RK update ->
//   (last stage) primitive output + CFL reduction.
//
// Replaces, per stage, SpaceOperator::ComputeResidual (SpaceOperator.cpp:3351-3409)
// = Reconstructor::Reconstruct (Reconstructor.cpp:332-904) +
//   SpaceOperator::CheckReconstructedStates (SpaceOperator.cpp:3198-3347) +
//   the face loop of SpaceOperator::ComputeAdvectionFluxes (2423-2815),
// and the RK arithmetic of TimeIntegratorRK2/RK3::AdvanceOneTimeStep
// (TimeIntegrator.cpp:291-428, 496-690) with ConservativeToPrimitive,
// ClipDensityAndPressure and ApplyBoundaryConditions (SpaceOperator.cpp:553-649, 1667-1745).
//
// Layout in HBM: structure-of-arrays FP64, interior cells only
// (index (k*ny + j)*px + i, row pitch px); ghost values are never stored:
// they are rebuilt from interior cells by the boundary rule when loaded.
//
// Work decomposition: a CTA owns a 32 x TY column of cells and marches along
// z through a chunk of planes, one warp per row of 32 cells. What the tile
// needs beyond its own cells (the face states of the four halo sides, the
// fluxes of its high x and y faces, the boundary rule on the halo, the plane
// copies) is done by one more warp (StageShape::edge_warp), or spread over
// the row warps as one extra item each.
// The stage's input is a primitive state in the compute type (V^n for stage
// 1; for later stages clip(C2P(U_s)), written by the previous stage's
// update). Its planes lie in a shared-memory ring with a 2-cell x/y halo,
// each brought in by ONE tensor copy of all five components
// (cp.async.bulk.tensor over a 4D map x, y, z, component; box 40 x (TY+4) x
// 1 x 5 starting at x = i0-4, a 16-byte boundary) on an mbarrier per slot
// (and one more copy for the material IDs, box 64 x (TY+4) from x = i0-16).
// Cells outside the domain in x/y arrive as zeros; one warp rewrites
// them from their image or wrapped cell before any other warp reads them.
// Ghost planes in z are not stored: a thread forms its column's ghost value.
//
// Iteration p of the plane pipeline:
//   A(p)  slopes and checked face states of plane p, one direction after the
//         other, into shared memory (the high z state stays in registers)
//   barrier
//   B(p)  the fluxes of plane p's low x and y faces (to shared memory) and of
//         its low z face p-1/2; with it the update of plane p-1 is complete
//   barrier
//   C(p)  the sum of plane p's fluxes but the one of z face p+1/2, kept in
//         registers for B(p+1)
// The three directions and the three faces are loops that are not unrolled:
// the kernel is bound by issue and by instruction fetch, and three copies of
// the flux code cost more in fetch stalls than their selects save.
// Face states follow Reconstructor.cpp: slope-limited primitive values, the
// first face (in the order l,r,b,t,k,f) failing CheckState reverted to the
// cell value, every face needing clipping reverted to the cell value, and a
// remaining CheckState failure reported as an error (never a trap).
#pragma once
#include <cuda.h>  // CUtensorMap

#include <type_traits>

#include "physics.cuh"

namespace m2c {

constexpr int MAXMAT = 4;
constexpr int TX = 32;
// Width of the plane box in x: cells i0-4 .. i0+35 (the tile's loaded
// columns i0-2 .. i0+33 plus two unused columns each side, so that the box
// starts on a 16-byte boundary for 4- and 8-byte elements).
constexpr int STAGE_TMA_BX = 40;
// The same for the material-ID box: cells i0-16 .. i0+47 (one byte each).
constexpr int STAGE_TMA_IX = 64;
// Upper bound of mbarrier polls for one plane copy (a copy from valid
// addresses always lands; the bound turns a fault into an error status).
constexpr int STAGE_TMA_POLLS = 1 << 22;

enum { BC_NONE = 0, BC_INLET = 1, BC_OUTLET = 2, BC_SLIPWALL = 3, BC_STICKWALL = 4, BC_SYMMETRY = 5,
       BC_PERIODIC = 100 };

struct DevError {
  int code;
  int cell;   // linear interior index of the first failing cell (or -1)
  int where;  // stage * 16 + site
  int pad;
};

struct Grid3 {
  int nx, ny, nz;
  long long px, plane;  // row pitch, plane size (elements)
  int bc[6];
  double inlet[5], outlet[5];
  const double* dx;     // per axis cell widths (interior, length n)
  const double* dy;
  const double* dz;
  const double* lA[3];  // limiter coefficient A per axis index
  const double* lB[3];  // limiter coefficient B per axis index
  const int* lK[3];     // van Albada exponent per axis index
  const double* lC[3];  // generalized minmod B/(A+1) per axis index
  // per axis: 1 if A, B, K and C are the same at every index (uniform
  // meshes), which then stand in for the arrays
  int lu[3];
  double lA0[3], lB0[3], lC0[3];
  float fA0[3], fB0[3], fC0[3];  // the same in FP32
  int lK0[3];
};

template <typename T> __device__ __forceinline__ const T* axis_constant(const double* d, const float* f);
template <> __device__ __forceinline__ const double* axis_constant<double>(const double* d, const float*) { return d; }
template <> __device__ __forceinline__ const float* axis_constant<float>(const double*, const float* f) { return f; }

struct SchemeK {
  int flux, limiter, rec_linear, slope_zero_at_interface;
  int rec_var;             // ReconstructionData::VariableType: 0 primitive, 1 conservative,
                           // 2 primitive characteristic, 3 conservative characteristic
  double alpha, delta;
  int nmat;               // material IDs 0..nmat-1; nmat = inactive (enclosed by an embedded surface)
  double dummy[3];         // the inactive cells' fixed state: density, pressure, internal energy per mass
  Eos<double> ed[MAXMAT];  // per-material EOS, FP64 (built on the host)
  Eos<float> ef[MAXMAT];   // the same in FP32 for the mixed path's flux half
};

// Interface faces of a two-material stage: for a cell, the star states of
// the exact Riemann problems on its three low faces (x, y, z), found through
// slot[cell] (written only where a low face separates two materials).
struct IfaceView {
  const int* slot;       // per cell; valid only where a low face is an interface
  const double* Vsm;     // [slot][3 faces][5]: left star state  (Riemann side idl)
  const double* Vsp;     // [slot][3 faces][5]: right star state (Riemann side idr)
  const double* Vmid;    // [slot][3 faces][5]: state at xi = 0 (EXACT flux)
  const int* midid;      // [slot][3 faces]
  int mp_flux;           // 0 EXACT, 1 NUMERICAL, 2 LLF
  int mp_recon;          // 0 CONSTANT (cell states), 1 LINEAR (face states)
  // Face pass (LINEAR interface reconstruction): if set, the kernel only
  // writes the reconstructed states on both sides of every interface face,
  // [slot][3 faces][left, right][5], for the exact Riemann problems solved
  // before the stage proper; no flux, no update.
  double* faces_out;
};

// Viscous face fluxes (area-weighted; momentum x, y, z and energy, the mass
// component being zero): fr[d] is added by the right cell of a face of axis
// d, fl[d] subtracted by its left cell; [4][faces], faces of axis d indexed
// x: (k ny + j)(nx + 1) + i, y: (k (ny + 1) + j) nx + i, z: (k ny + j) nx + i
// with (i, j, k) the face's right cell. fr[0] == NULL: inviscid.
struct ViscView {
  const double* fr[3];
  const double* fl[3];
  const double* fh[3];  // heat-diffusion flux per face (energy only), same indexing; NULL: none
  long long nf[3];
};

// Faces cut by an embedded surface (walls) and the one-sided Riemann star
// states of their two sides for this stage, from the wall pre-pass
// (SpaceOperator.cpp:2438-2484 and the y/z analogues). mask == NULL: no walls.
struct WallView {
  const uint8_t* mask;  // per cell: bit d set where the low face along axis d is a wall
  const int* slot;      // per cell; valid only where mask != 0
  const double* Vsm;    // [slot][3 faces][5]: the low neighbour's star state (its flux against it)
  const double* Vsp;    // [slot][3 faces][5]: this cell's star state
  int linear;           // EmbeddedBoundaryMethodData::recon LINEAR: reconstructed face states
  // Face pass (LINEAR): if set, the kernel writes the reconstructed states
  // on both sides of every cut face, [slot][3 faces][low, high][5], for the
  // one-sided problems solved before the stage proper; no flux, no update.
  double* faces_out;
};

struct StageArgs {
  Grid3 g;
  SchemeK s;
  const void* Pin[5];    // stage input: primitive state in the compute type (see above)
  void* Po[5];           // non-final stages: clip(C2P(U_new)) in the compute type
  float* Vfo[5];         // final stage, FP32 compute type: FP32 copy of the new state
  const double* Vn[5];   // V^n (primitive) - step state
  const double* Us[5];   // flux source of stages >= 2 (conserved, raw)
  double* Uo[5];         // stage output (conserved) for non-final stages
  double* Vo[5];         // final-stage output (primitive)
  const uint8_t* id;     // material id per cell
  int stage;             // 1-based
  int final_stage;
  double a_prev, a_un;   // U_new = a_prev*U_s + a_un*U^n (stages >= 2)
  double bdt_coef;       // U_new += (bdt_coef*dt)*R; 1.0 for stage 1
  const double* clock;   // device clock: [0] t, [1] dt
  const int* us_clipped; // non-zero: U_s := P2C(clip(C2P(U_s))) everywhere (TimeIntegrator.cpp:542-545)
  int* clipped_out;      // set if any cell of this stage's output was clipped
  unsigned long long* dtmin_bits;  // final stage: min dx/(|u|+c) as ordered bits
  DevError* err;
  int ntx, nty;          // tiles in x and y
  int nitems;            // CTAs that share the (tile, plane) units evenly
  double* Ro[5];         // if set: write the residual R only (no RK update)
  IfaceView iface;
  ViscView visc;
  WallView wall;
  CUtensorMap tin;       // 4D map of the stage input (Pin as one five-component buffer)
  CUtensorMap tid;       // 3D map of the material IDs
};

__device__ __forceinline__ void report(DevError* e, int code, int cell, int where) {
  if (atomicCAS(&e->code, 0, code) == 0) {
    e->cell = cell;
    e->where = where;
  }
}

// Planes of the ring: three are read in an iteration (p-1, p, p+1) and one
// is in flight.
constexpr int STAGE_RING = 4;

template <typename T, int TY, bool MULTI>
struct StageSmem {
  static constexpr int RX = TX + 4, RY = TY + 4;  // loaded region: x -2..TX+1, y -2..TY+1
  static constexpr int BX = STAGE_TMA_BX;         // cell (i0 + x, j0 + y) at column x + 4, row y + 2
  // one plane each, on the 128-byte boundary that a tensor copy starts at
  struct alignas(128) Plane { T v[5][RY][BX]; };
  struct alignas(128) IdPlane { uint8_t v[RY][STAGE_TMA_IX]; };  // column x + 16
  Plane v[STAGE_RING];
  IdPlane id[MULTI ? STAGE_RING : 1];
  // of the faces of a row or column of cells: hi the high-side state of the
  // cell left of the face, lo the low-side state of the cell right of it, f
  // the flux
  T hix[5][TY][TX + 1], lox[5][TY][TX + 1], fx[5][TY][TX + 1];
  T hiy[5][TY + 1][TX], loy[5][TY + 1][TX], fy[5][TY + 1][TX];
  T loz[5][TY][TX];
  double red[TY];
  unsigned long long bar[STAGE_RING];  // one mbarrier per ring slot
};

// Resolve a possibly-outside index along one axis (at most two cells out).
// Returns the interior index to read; sets ghost side (-1 none, 0 low, 1 high)
// or far (outside by more than one cell, not periodic).
__device__ __forceinline__ int resolve_axis(int c, int n, bool periodic, int& side, bool& far) {
  side = -1;
  if (c >= 0 && c < n) return c;
  if (periodic) {
    int w = c < 0 ? c + n : c - n;
    if (w < 0) w += n;
    if (w >= n) w -= n;
    return w;
  }
  if (c == -1) { side = 0; return 0; }
  if (c == n) { side = 1; return n - 1; }
  far = true;
  return c < 0 ? 0 : n - 1;
}

__device__ __forceinline__ int wrap_index(int c, int n) {
  if (c < 0) c += n;
  if (c >= n) c -= n;
  if (c < 0) c += n;
  if (c >= n) c -= n;
  return c;
}

template <typename T> struct EosPick;
template <> struct EosPick<double> {
  __device__ static const Eos<double>& get(const SchemeK& s, int id) { return s.ed[id]; }
};
template <> struct EosPick<float> {
  __device__ static const Eos<float>& get(const SchemeK& s, int id) { return s.ef[id]; }
};

// SG: every material is a stiffened gas (the kernel variant then carries no
// other equation of state and no test of the kind).
template <typename T, bool MULTI, bool SG = false>
__device__ __forceinline__ const Eos<T>& eos_of(const SchemeK& s, int id) {
  const Eos<T>& e = EosPick<T>::get(s, MULTI ? (id < s.nmat ? id : 0) : 0);
  if (SG) __builtin_assume(e.kind == EOS_SG);
  return e;
}

// Boundary face state built from the interior neighbour's face state
// (Reconstructor.cpp:822-875) followed by the clip check of
// CheckReconstructedStates on the ghost's inward face (3279-3318).
template <typename T>
__device__ __forceinline__ void ghost_face(int bc, int axis, const T* inner_face, const T* ghost_cell,
                                           const Eos<T>& e, T* out) {
  if (bc == BC_INLET || bc == BC_OUTLET) {
#pragma unroll
    for (int p = 0; p < 5; p++) out[p] = ghost_cell[p];
  } else {
#pragma unroll
    for (int p = 0; p < 5; p++) out[p] = inner_face[p];
    if (bc == BC_STICKWALL) {
      out[1] = -out[1]; out[2] = -out[2]; out[3] = -out[3];
    } else {
      if (axis == 0) out[1] = -out[1];
      else if (axis == 1) out[2] = -out[2];
      else out[3] = -out[3];
    }
  }
  if (e.needs_clip(out)) {
#pragma unroll
    for (int p = 0; p < 5; p++) out[p] = ghost_cell[p];
  }
}

template <typename T, int FLUX, int PIN>
__device__ __forceinline__ int flux_of(const Eos<T>& e, int d, const T* VL, const T* VR, T delta, T* F) {
  if (FLUX == FLUX_HLLC) return flux_hllc<PIN>(e, d, VL, VR, F);
  if (FLUX == FLUX_ROE) return flux_roe<PIN>(e, d, VL, VR, delta, F);
  return flux_llf2<PIN>(e, e, d, VL, VR, F);
}

// Primitive state of a ghost cell beyond a boundary of type bc on `axis`
// from its image cell's (SpaceOperator::ApplyBoundaryConditions).
template <typename T>
__device__ __forceinline__ void ghost_cell(const Grid3& g, int axis, int bc, const T* image, T* out) {
#pragma unroll
  for (int c = 0; c < 5; c++) out[c] = image[c];
  if (bc == BC_INLET) {
#pragma unroll
    for (int c = 0; c < 5; c++) out[c] = T(g.inlet[c]);
  } else if (bc == BC_OUTLET) {
#pragma unroll
    for (int c = 0; c < 5; c++) out[c] = T(g.outlet[c]);
  } else if (bc == BC_STICKWALL) {
    out[1] = -out[1]; out[2] = -out[2]; out[3] = -out[3];
  } else {  // SYMMETRY / SLIPWALL: normal velocity flipped
    if (axis == 0) out[1] = -out[1];
    else if (axis == 1) out[2] = -out[2];
    else out[3] = -out[3];
  }
}

// Tile rows, whether an extra warp does the edge work, and the CTAs per SM
// that the kernel is compiled for. Registers are handed out per quarter of an
// SM, so warps per SM come in fours: 12 (11 rows and the edge warp) leave 168
// registers each, which the FP64 kernel needs to run without spills; 16 leave
// 128, which the FP32 kernel fits as two CTAs of 8 rows. Measured per stage
// launch, before -> now (the kernel before: 32 x 8 tiles in FP64 and 32 x 16
// in FP32 at one CTA per SM, all slopes kept in shared memory, short-cut
// tests and a branch per limiter component): FP64 HLLC channel 161x97x131
// 1.76 -> 0.92 ms, FP64 bubble 101x96x90 1.50 -> 0.64 ms, mixed bubble cluster
// 192^3 1.91 -> 1.41 ms, mixed HLLC box 160^3 0.78 -> 0.60 ms, mixed Roe box
// 256^3 2.47 -> 2.29 ms. FP64 with 8 rows and the edge warp is 1.39 ms on the
// channel, with 7 rows (255 registers) 1.45 ms; FP32 with 16 rows at one CTA
// per SM 8 % slower on the 256^3 box.
template <typename T> struct StageShape {
  static constexpr int ty = 11, warps = ty + 1, occ = 1;
  static constexpr bool edge_warp = true;
};
template <> struct StageShape<float> {
  static constexpr int ty = 8, warps = ty, occ = 2;
  static constexpr bool edge_warp = false;
};

// CONS: reconstruction in conservative or characteristic variables (a
// separate instantiation so the primitive-variable kernels carry none of it).
// WALLS (two-material variant only): the branch of faces cut by an embedded
// surface is compiled in; without it the kernel carries none of its tests.
template <typename T, int FLUX, bool MULTI, bool CONS, bool WALLS, bool SG>
__global__ void __launch_bounds__(TX * StageShape<T>::warps, CONS ? 1 : StageShape<T>::occ)
    stage_kernel(const __grid_constant__ StageArgs a) {
  constexpr int TY = StageShape<T>::ty;
  constexpr bool EW = StageShape<T>::edge_warp;
  constexpr int PIN = PIN_MOMENTUM | PIN_SOUND | (MULTI ? PIN_SUPERSONIC : 0);  // FP32, see physics.cuh
  static_assert(TY >= 6 && TY <= 16, "one warp holds both x-halo columns of the tile; the spread extra items take warps 0 to 5");
  extern __shared__ __align__(128) unsigned char smem_raw[];
  typedef StageSmem<T, TY, MULTI> S;
  S& sm = *reinterpret_cast<S*>(smem_raw);
  constexpr int RING = STAGE_RING;
  constexpr int CS = S::RY * S::BX;  // component stride of a plane
  constexpr int XS = TY * (TX + 1), YS = (TY + 1) * TX, ZS = TY * TX;  // and of the x, y and z face arrays
  const Grid3& g = a.g;
  const int lane = threadIdx.x, row = threadIdx.y;
  const bool edge = EW && row == TY;                // the edge warp
  const bool copier = lane == 0 && row == (EW ? TY : 5);  // the thread that starts the plane copies
  const bool xper = g.bc[0] == BC_PERIODIC, yper = g.bc[2] == BC_PERIODIC, zper = g.bc[4] == BC_PERIODIC;
  const double dt = a.clock[1];
  const double bdt = a.bdt_coef * dt;
  const bool us_clip = (a.stage > 1) && a.us_clipped && *a.us_clipped;
  const T alpha = T(a.s.alpha), delta = T(a.s.delta);
  const int where = a.stage * 16;
  const int limiter = a.s.limiter;
  const bool rec_linear = a.s.rec_linear;
  const bool slope_zero = MULTI && a.s.slope_zero_at_interface;
  const bool face_pass = MULTI && (a.iface.faces_out || (WALLS && a.wall.faces_out));

  int i0 = 0, j0 = 0, pbase = 0;  // tile origin and first plane of the current segment
  constexpr unsigned TMA_BYTES = 5u * S::RY * S::BX * sizeof(T) + (MULTI ? unsigned(S::RY) * STAGE_TMA_IX : 0u);
  unsigned tma_phase = 0;  // bit s: parity of the next completion of slot s's mbarrier
  if (copier) {
    for (int q = 0; q < RING; q++) {
      const unsigned bar = (unsigned)__cvta_generic_to_shared(&sm.bar[q]);
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<unsigned long long>(&a.tin)) : "memory");
  }

  auto slot_of = [&](int p) { return int(unsigned(p - pbase) % unsigned(RING)); };
  auto real_plane = [&](int p) { return zper || (p >= 0 && p < g.nz); };

  // Start copying plane p into its ring slot (one thread,
  // after a barrier that ends every read of the slot's previous plane).
  auto issue_plane = [&](int p) {
    const int s = slot_of(p), kk = zper ? wrap_index(p, g.nz) : p;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&sm.bar[s]);
    const unsigned dst = (unsigned)__cvta_generic_to_shared(&sm.v[s].v[0][0][0]);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(TMA_BYTES) : "memory");
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
        "[%6];" ::"r"(dst), "l"(reinterpret_cast<unsigned long long>(&a.tin)), "r"(i0 - 4), "r"(j0 - 2), "r"(kk),
        "r"(0), "r"(bar)
        : "memory");
    if constexpr (MULTI) {
      const unsigned idst = (unsigned)__cvta_generic_to_shared(&sm.id[s].v[0][0]);
      asm volatile(
          "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
          "[%5];" ::"r"(idst), "l"(reinterpret_cast<unsigned long long>(&a.tid)), "r"(i0 - 16), "r"(j0 - 2), "r"(kk),
          "r"(bar)
          : "memory");
    }
  };

  // Wait for plane p (bounded; a copy that never lands is reported and the
  // CTA stops at the next barrier). Every thread waits for every plane once.
  auto wait_plane = [&](int p) -> bool {
    const int s = slot_of(p);
    const unsigned bar = (unsigned)__cvta_generic_to_shared(&sm.bar[s]);
    const unsigned parity = (tma_phase >> s) & 1u;
    unsigned ok = 0;
    for (int it = 0; it < STAGE_TMA_POLLS && !ok; it++) {
      asm volatile(
          "{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\tselp.b32 %0, 1, 0, P1;\n\t}"
          : "=r"(ok)
          : "r"(bar), "r"(parity)
          : "memory");
    }
    tma_phase ^= 1u << s;
    if (!ok) report(a.err, ERR_ITER_CAP, -1, where + 5);
    return ok != 0;
  };

  // The landed plane p (a real one): the loaded cells outside the domain in
  // x or y, shared by all threads. A cell beyond a periodic boundary takes its wrapped
  // cell's value, one beyond another boundary the value the boundary rule
  // gives it from its image cell; both are read from global memory. Cells
  // outside twice, or by more than one cell, are never read.
  int fcl = 0, frl = 0, fncol = 0, fn = 0;  // columns and rows below 0, cells of the outside columns, of all (per tile)
  auto fix_plane = [&](int p) {
    const int s = slot_of(p), kk = zper ? wrap_index(p, g.nz) : p;
    for (int it = row * TX + lane; it < fn; it += TX * StageShape<T>::warps) {
      int x, y;  // cell relative to the tile's origin
      if (it < fncol) {
        const int q = it / S::RY;
        x = q < fcl ? q - 2 : g.nx - i0 + q - fcl;
        y = it - q * S::RY - 2;
      } else {
        const int q = (it - fncol) / S::RX;
        y = q < frl ? q - 2 : g.ny - j0 + q - frl;
        x = (it - fncol) - q * S::RX - 2;
      }
      int sx, sy;
      bool far = false;
      const int ii = resolve_axis(i0 + x, g.nx, xper, sx, far), jj = resolve_axis(j0 + y, g.ny, yper, sy, far);
      if (far || (sx >= 0 && sy >= 0)) continue;
      const long long off = (long long)kk * g.plane + (long long)jj * g.px + ii;
      T v[5], o[5];
#pragma unroll
      for (int c = 0; c < 5; c++) v[c] = static_cast<const T*>(a.Pin[c])[off];
      if (MULTI) sm.id[s].v[y + 2][x + 16] = a.id[off];
      const int axis = sx >= 0 ? 0 : 1, side = sx >= 0 ? sx : sy;
      if (side >= 0) {
        ghost_cell(g, axis, g.bc[2 * axis + side], v, o);
      } else {
#pragma unroll
        for (int c = 0; c < 5; c++) o[c] = v[c];
      }
#pragma unroll
      for (int c = 0; c < 5; c++) sm.v[s].v[c][y + 2][x + 4] = o[c];
    }
    // order these writes before the tensor copy that refills the slot
    if (fn) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  };

  // Limiter coefficients (Reconstructor::Setup) of the cell at column cx,
  // row cy of plane p along axis d: the axis' constants on a uniform axis,
  // else its per-index arrays. The generalized minmod uses C = B/(A+1) only
  // (carried in B).
  auto limiter_coeffs = [&](int p, int cx, int cy, int d, T& A, T& B, int& K) {
    if (g.lu[d]) {
      if (limiter == LIM_VANALBADA) {
        A = axis_constant<T>(g.lA0, g.fA0)[d]; B = axis_constant<T>(g.lB0, g.fB0)[d]; K = g.lK0[d];
      } else {
        A = T(0); B = axis_constant<T>(g.lC0, g.fC0)[d];
      }
      return;
    }
    const int ix = d == 0 ? wrap_index(i0 + cx - 4, g.nx) : (d == 1 ? wrap_index(j0 + cy - 2, g.ny)
                                                                    : wrap_index(p, g.nz));
    if (limiter == LIM_VANALBADA) {
      A = T(g.lA[d][ix]); B = T(g.lB[d][ix]); K = g.lK[d][ix];
    } else {
      A = T(0); B = T(g.lC[d][ix]);
    }
  };

  // States (and IDs) of the two neighbours along d of the cell at (cx, cy)
  // of plane p, whose own state is v; ghost planes by the boundary rule.
  auto neighbours = [&](int d, int p, int cx, int cy, const T* v, T* vm, T* vp, int& idm, int& idp) {
    const int s0 = slot_of(p);
    int sm1 = s0, sp1 = s0;
    bool rm = true, rp = true;
    if (d == 2) {
      rm = real_plane(p - 1);
      rp = real_plane(p + 1);
      if (rm) sm1 = slot_of(p - 1);
      if (rp) sp1 = slot_of(p + 1);
    }
    const int off = cy * S::BX + cx, step = d == 0 ? 1 : (d == 1 ? S::BX : 0);
    const T* qm = &sm.v[sm1].v[0][0][0] + (off - step);
    const T* qp = &sm.v[sp1].v[0][0][0] + (off + step);
#pragma unroll
    for (int c = 0; c < 5; c++) {
      vm[c] = qm[c * CS];
      vp[c] = qp[c * CS];
    }
    if (!rm) ghost_cell(g, 2, g.bc[4], v, vm);
    if (!rp) ghost_cell(g, 2, g.bc[5], v, vp);
    if (MULTI && (WALLS || CONS || slope_zero)) {
      const int ox = d == 0 ? 1 : 0, oy = d == 1 ? 1 : 0;
      idm = sm.id[sm1].v[cy - oy][cx - ox + 12];
      idp = sm.id[sp1].v[cy + oy][cx + ox + 12];
    }
  };

  // Limited slopes in direction d of the real cell at (cx, cy) of plane p.
  auto slopes = [&](int d, int p, int cx, int cy, int id, const T* v, T* sd) {
    if (!rec_linear) {
#pragma unroll
      for (int c = 0; c < 5; c++) sd[c] = T(0);
      return;
    }
    T vm[5], vp[5];
    int idm = 0, idp = 0;
    neighbours(d, p, cx, cy, v, vm, vp, idm, idp);
    T A, B;
    int K = 0;
    limiter_coeffs(p, cx, cy, d, A, B, K);
    const bool zero = slope_zero && (id != idm || id != idp);
    // no difference toward an inactive neighbour (Reconstructor.cpp:475-502)
    const bool offm = WALLS && idm == a.s.nmat, offp = WALLS && idp == a.s.nmat;
    T dm[5], dp[5];
#pragma unroll
    for (int c = 0; c < 5; c++) {
      dm[c] = offm ? T(0) : v[c] - vm[c];
      dp[c] = offp ? T(0) : vp[c] - v[c];
    }
    limited_slopes(limiter, A, B, K, alpha, dm, dp, sd);
    if (slope_zero && zero) {
#pragma unroll
      for (int c = 0; c < 5; c++) sd[c] = T(0);
    }
  };

  // Face states of the real cell at (cx, cy) of plane p along d: lo = v - s/2
  // on its low face, hi = v + s/2 on its high one, each reverted to the cell
  // value v where the reference reverts it. chain carries "a non-physical
  // face was reverted already" from one direction of the cell to the next
  // (faces in the reference's order l, r, b, t, k, f).
  auto face_states = [&](int d, int p, int cx, int cy, int id, const Eos<T>& e, const T* v, bool& chain, int& err,
                         T* lo, T* hi) {
    T sd[5];
    slopes(d, p, cx, cy, id, v, sd);
#pragma unroll
    for (int c = 0; c < 5; c++) {
      lo[c] = v[c] - T(0.5) * sd[c];
      hi[c] = v[c] + T(0.5) * sd[c];
    }
    if (e.both_fine(v, sd)) return;
#pragma unroll
    for (int side = 0; side < 2; side++) {
      T* f = side ? hi : lo;
      const bool bad = e.bad(f);
      bool reverted = false;
      // Reconstructor.cpp:719-775: only the first non-physical face is reverted.
      if (!chain && bad) { reverted = true; chain = true; }
      // SpaceOperator.cpp:3240-3273: a face needing clipping reverts to the cell value.
      if (!reverted && e.needs_clip(f)) reverted = true;
      // SpaceOperator.cpp:3275-3277: a face still non-physical is fatal.
      if (!reverted && bad) err = ERR_STATE;
      if (reverted) {
#pragma unroll
        for (int c = 0; c < 5; c++) f[c] = v[c];
      }
    }
  };

  // Limited slopes in direction d of the real cell at (cx, cy) of plane p in
  // the scheme's non-primitive variables (Reconstructor.cpp:397-404, 469-651):
  // differences of the conservative variables (rv 1, 3; neighbours converted
  // with their own EOS) or of the primitive ones (rv 2), projected on the
  // characteristic basis at the cell state (rv 2, 3) and limited there, then
  // mapped back. u is the cell's conservative state. Returns false where the
  // basis does not exist (c^2 < 0; the reference aborts).
  auto nonprim_slopes = [&](int d, int p, int cx, int cy, int id, int rv, const Eos<T>& e, const T* v, const T* u,
                            T* sd) -> bool {
    T A, B;
    int K = 0;
    limiter_coeffs(p, cx, cy, d, A, B, K);
    T qm[5], qp[5], dl[5], dr[5];
    int idm = 0, idp = 0;
    neighbours(d, p, cx, cy, v, qm, qp, idm, idp);
    const bool zero = slope_zero && (id != idm || id != idp);
    const bool uspace = rv != 2;
    if (uspace) {
      T t[5];
      eos_of<T, MULTI, SG>(a.s, idm).p2c(qm, t);
#pragma unroll
      for (int c = 0; c < 5; c++) qm[c] = t[c];
      eos_of<T, MULTI, SG>(a.s, idp).p2c(qp, t);
#pragma unroll
      for (int c = 0; c < 5; c++) qp[c] = t[c];
    }
    const T* q0 = uspace ? u : v;
    const bool offm = WALLS && idm == a.s.nmat, offp = WALLS && idp == a.s.nmat;  // Reconstructor.cpp:529-556
#pragma unroll
    for (int c = 0; c < 5; c++) {
      dl[c] = offm ? T(0) : q0[c] - qm[c];
      dr[c] = offp ? T(0) : qp[c] - q0[c];
    }
    bool ok = true;
    if (rv == 1) {
#pragma unroll
      for (int c = 0; c < 5; c++) sd[c] = limited_slope_c(limiter, A, B, K, alpha, dl[c], dr[c]);
    } else {
      CharBasis<T> cb;
      char_basis(e, d, v, cb);
      ok = cb.ok;
      T wl[5], wr[5], sw[5];
      if (rv == 2) {
        prim_to_char(cb, v, dl, wl);
        prim_to_char(cb, v, dr, wr);
      } else {
        char_rinv(cb, v, dl, wl);
        char_rinv(cb, v, dr, wr);
      }
#pragma unroll
      for (int c = 0; c < 5; c++) sw[c] = limited_slope_c(limiter, A, B, K, alpha, wl[c], wr[c]);
      if (rv == 2) char_to_prim(cb, v, sw, sd);
      else char_r(cb, v, sw, sd);
    }
    if (zero) {
#pragma unroll
      for (int c = 0; c < 5; c++) sd[c] = T(0);
    }
    return ok;
  };

  // CONS: the two face states along dir of the real cell at (cx, cy) of plane
  // p. Any non-physical face of the six sends the cell back to primitive
  // variables (the RETRY of Reconstructor.cpp:719-775), so all are formed.
  auto cons_states = [&](int dir, int p, int cx, int cy, int id, const Eos<T>& e, const T* v, int& err, T* lo, T* hi) {
    if (rec_linear) {
      T sx[5], sy[5], sz[5], u[5];
      const int rv = a.s.rec_var;
      const bool uspace = rv != 2;
      e.p2c(v, u);
      bool okb = nonprim_slopes(0, p, cx, cy, id, rv, e, v, u, sx);
      okb = nonprim_slopes(1, p, cx, cy, id, rv, e, v, u, sy) && okb;
      okb = nonprim_slopes(2, p, cx, cy, id, rv, e, v, u, sz) && okb;
      if (!okb) err = ERR_SOUND;
      bool cons = true;
#pragma unroll
      for (int q = 0; q < 6; q++) {
        const T* sg = q < 2 ? sx : (q < 4 ? sy : sz);
        T f[5];
        if (uspace) {
          T uf[5];
#pragma unroll
          for (int c = 0; c < 5; c++) uf[c] = (q & 1) ? u[c] + T(0.5) * sg[c] : u[c] - T(0.5) * sg[c];
          e.c2p(uf, f);
        } else {
#pragma unroll
          for (int c = 0; c < 5; c++) f[c] = (q & 1) ? v[c] + T(0.5) * sg[c] : v[c] - T(0.5) * sg[c];
        }
        const bool bad = e.bad(f);
        if (bad) cons = false;
        if ((q >> 1) != dir) continue;
        const bool rev = !bad && e.needs_clip(f);  // SpaceOperator.cpp:3240-3273
        T* out = (q & 1) ? hi : lo;
#pragma unroll
        for (int c = 0; c < 5; c++) out[c] = rev ? v[c] : f[c];
      }
      if (cons) return;
    }
    bool chain = false;
#pragma unroll 1
    for (int d = 0; d < 3; d++) {
      T l[5], h[5];
      face_states(d, p, cx, cy, id, e, v, chain, err, l, h);
      if (d != dir) continue;
#pragma unroll
      for (int c = 0; c < 5; c++) {
        lo[c] = l[c];
        hi[c] = h[c];
      }
    }
  };

  // Flux across the low face along d of the cell at (cx, cy) of plane p (the
  // face's right cell), as its left cell sees it. VL, VR: the two cells' face
  // states, rL, rR: whether they are real (a ghost's is formed here). At a
  // NUMERICAL interface face the right cell forms its own flux in its update.
  auto face_flux = [&](auto pin, int d, int p, int cx, int cy, bool rL, bool rR, T* VL, T* VR, T* F) {
    const int ox = d == 0 ? 1 : 0, oy = d == 1 ? 1 : 0;
    const int sR = slot_of(p), sL = d == 2 ? slot_of(p - 1) : sR;
    int idL = 0, idR = 0;
    if (MULTI) {
      if (rL) idL = sm.id[sL].v[cy - oy][cx - ox + 12];
      if (rR) idR = sm.id[sR].v[cy][cx + 12];
      if (!rL) idL = idR;
      if (!rR) idR = idL;
    }
    // Boundary face state built from the interior neighbour's face state
    // (Reconstructor.cpp:822-875), and from the ghost cell's where that
    // needs clipping (CheckReconstructedStates, 3279-3318).
    if (!rL || !rR) {
      T im[5], gc[5];
#pragma unroll
      for (int c = 0; c < 5; c++) im[c] = rR ? sm.v[sR].v[c][cy][cx] : sm.v[sL].v[c][cy - oy][cx - ox];
      const int bc = g.bc[2 * d + (rR ? 0 : 1)];
      ghost_cell(g, d, bc, im, gc);
      ghost_face(bc, d, rR ? VR : VL, gc, eos_of<T, MULTI, SG>(a.s, idR), rR ? VL : VR);
    }
    // a face cut by an embedded surface (interior faces only) takes the wall
    // branch, which the reference tests before the material-interface one
    bool wall = false;
    long long offR = 0;
    if (MULTI && rL && rR && (WALLS || idL != idR)) {
      offR = (long long)wrap_index(p, g.nz) * g.plane + (long long)wrap_index(j0 + cy - 2, g.ny) * g.px +
             wrap_index(i0 + cx - 4, g.nx);
      if (WALLS) wall = (a.wall.mask[offR] >> d) & 1;
    }
    if (face_pass) {  // the states a pre-pass solves from, and nothing else
      for (int q = 0; q < 2; q++) {
        if (q == 0 ? !(a.iface.faces_out && idL != idR) : !(WALLS && a.wall.faces_out && wall)) continue;
        const int slot = q == 0 ? a.iface.slot[offR] : a.wall.slot[offR];
        double* o = (q == 0 ? a.iface.faces_out : a.wall.faces_out) + ((long long)slot * 3 + d) * 10;
#pragma unroll
        for (int c = 0; c < 5; c++) {
          o[c] = double(VL[c]);
          o[5 + c] = double(VR[c]);
        }
      }
      return;
    }
    if (WALLS && (idL == a.s.nmat || idR == a.s.nmat) && !(wall && idL != a.s.nmat)) {
      // an inactive side gets no flux, and a face with an inactive cell that
      // no surface cuts carries none (SpaceOperator.cpp:2441-2483, 2537-2551);
      // the right cell of a cut face forms its own flux in its update
#pragma unroll
      for (int c = 0; c < 5; c++) F[c] = T(0);
      return;
    }
    int err = ERR_NONE;
    const Eos<T>* e = &eos_of<T, MULTI, SG>(a.s, idR);  // the right cell's EOS, as the reference's face loop
    if (MULTI && (wall || idL != idR)) {
      // Material interface (SpaceOperator.cpp:2486-2542): two one-sided fluxes
      // against the exact Riemann star states, or LLF across the interface.
      // Wall (2438-2484): the left cell's flux against its one-sided star state.
      const IfaceView& iv = a.iface;
      if (wall ? !a.wall.linear : iv.mp_recon == 0) {  // constant reconstruction: cell-centred states
#pragma unroll
        for (int c = 0; c < 5; c++) {
          VL[c] = sm.v[sL].v[c][cy - oy][cx - ox];
          VR[c] = sm.v[sR].v[c][cy][cx];
        }
      }
      if (!wall && iv.mp_flux == 2) {
        err = flux_llf2(eos_of<T, MULTI, SG>(a.s, idL), eos_of<T, MULTI, SG>(a.s, idR), d, VL, VR, F);
        if (err) report(a.err, err, -1, where + 2);
        return;
      }
      const int slot = wall ? a.wall.slot[offR] : iv.slot[offR];  // held by the right cell
      const long long base = ((long long)slot * 3 + d) * 5;
      if (!wall && iv.mp_flux == 0) {  // Godunov flux of the state at xi = 0
        T Vm[5];
#pragma unroll
        for (int c = 0; c < 5; c++) Vm[c] = T(iv.Vmid[base + c]);
        phys_flux(eos_of<T, MULTI, SG>(a.s, iv.midid[slot * 3 + d]), d, Vm, F);
        return;
      }
      const double* src = wall ? a.wall.Vsm : iv.Vsm;
#pragma unroll
      for (int c = 0; c < 5; c++) VR[c] = T(src[base + c]);
      e = &eos_of<T, MULTI, SG>(a.s, idL);
    }
    err = flux_of<T, FLUX, decltype(pin)::value>(*e, d, VL, VR, delta, F);
    if (err) report(a.err, err, -1, where + 2);
  };

  // per-thread CFL extremes: the largest |u| + c seen against each axis'
  // current width (dx / max is the smallest quotient, rounding being
  // monotonic), turned into a time step when a width changes
  double lmax[3] = {0.0, 0.0, 0.0}, dtmin_local = 1.0e300;
  int clipped_local = 0;
  const int tiles = a.ntx * a.nty;

  // Balanced segments: the (tile, plane) units, ordered tile by tile and
  // plane by plane within a tile, are split evenly over the CTAs; a CTA runs
  // the plane pipeline over each tile segment of its share (at most a few).
  const long long units = (long long)tiles * g.nz;
  const long long ubeg = units * blockIdx.x / gridDim.x, uend = units * (blockIdx.x + 1) / gridDim.x;
  for (long long u = ubeg; u < uend;) {
    const int t2 = (int)(u / g.nz);
    const int kb = (int)(u - (long long)t2 * g.nz);
    const int ke = (int)min((long long)g.nz, kb + (uend - u));
    u += ke - kb;
    const int tyi = t2 / a.ntx, txi = t2 - tyi * a.ntx;
    __syncthreads();  // the previous segment's last reads (and the mbarriers' initialisation)
    i0 = txi * TX;
    j0 = tyi * TY;
    pbase = kb - 2;
    fcl = i0 == 0 ? 2 : 0;
    frl = j0 == 0 ? 2 : 0;
    fncol = (fcl + max(0, min(i0 + TX + 2 - g.nx, 2))) * S::RY;
    fn = fncol + (frl + max(0, min(j0 + TY + 2 - g.ny, 2))) * S::RX;
    const int gi = i0 + lane, gj = j0 + row;
    const bool own = !edge && gi < g.nx && gj < g.ny;
    // Cells this thread reconstructs, and the faces it owns. A row's own
    // cells take all directions; a wrapped cell beyond a periodic boundary
    // inside the tile only the one whose face needs it.
    const bool inx = gi < g.nx, iny = gj < g.ny;
    const bool sx_act = own || (xper && !edge && gi == g.nx && iny), sy_act = own || (yper && !edge && gj == g.ny && inx);
    const bool fx_act = !edge && iny && gi <= g.nx, fy_act = !edge && inx && gj <= g.ny;
    // Extra items: states of the x-halo columns (lanes 0-15 the low one,
    // 16-31 the high one), of the low and the high halo row; fluxes of the
    // tile's high x and y faces.
    const int er = lane & 15, ehi = lane >> 4;
    const bool er_in = er < TY && j0 + er < g.ny;
    const bool hx_act = er_in && (ehi ? (i0 + TX < g.nx || (xper && i0 + TX == g.nx)) : (i0 > 0 || xper));
    const bool ylo_act = inx && (j0 > 0 || yper), yhi_act = inx && (j0 + TY < g.ny || (yper && j0 + TY == g.ny));
    const bool hfx_act = er_in && ehi && i0 + TX <= g.nx, hfy_act = inx && j0 + TY <= g.ny;
    // real cells left and right of this thread's low x (bits 0, 1) and y (bits 2, 3) face
    const int lr = (gi > 0 || xper ? 1 : 0) | (inx || xper ? 2 : 0) | (gj > 0 || yper ? 4 : 0) | (iny || yper ? 8 : 0);
    // first item of this warp's loops (its own directions and faces are 0, 1, 2)
    const int a_first = EW ? (edge ? -3 : 0) : (row < 3 ? -1 : 0), a_end = edge ? 0 : 3;
    const int b_first = EW ? (edge ? -2 : 0) : (row == 3 || row == 4 ? -1 : 0);
    double dxi = 0, dyj = 0, dzc = 0, inv_mvol = 0, ax = 0, ay = 0;
    if (own) { dxi = g.dx[gi]; dyj = g.dy[gj]; }
    const double az = dxi * dyj;
    float axf = 0.f, ayf = 0.f;
    const float azf = float(az);
    // cell offsets fit 32 bits: 2^32 cells would not fit the device
    const unsigned plane32 = unsigned(g.plane), offc = unsigned(gj) * unsigned(g.px) + unsigned(gi);

    // pipeline prologue: RING planes in flight, the halos iteration kb-1 reads ready
    bool landed = true;
    if (copier)
      for (int p = kb - 2; p < kb - 2 + RING; p++)
        if (p <= ke + 1 && real_plane(p)) issue_plane(p);
    for (int p = kb - 2; p <= kb; p++) {
      if (!real_plane(p)) continue;
      landed = wait_plane(p) && landed;
      if (landed && (CONS || p > kb - 2)) fix_plane(p);
    }
    if (__syncthreads_or(!landed)) return;

    T pz[5];             // high z face state of plane p-1
    double part[5];      // FP64: flux sum of plane p-1 without its face p-1/2
    T dxy[5], hl[5];     // mixed: x and y flux differences of plane p-1, flux of face p-3/2
    int idprev = 0;      // material of plane p-1
#pragma unroll
    for (int c = 0; c < 5; c++) {
      pz[c] = dxy[c] = hl[c] = T(0);
      part[c] = 0.0;
    }
    for (int p = kb - 1; p <= ke; p++) {
      const bool rp = real_plane(p), in = p >= kb && p < ke;
      const int s0 = slot_of(p);
      // ---- A(p)
      if (p > kb && own && !face_pass) {  // the update's FP64 inputs of plane p-1 into L1
        const unsigned offp = unsigned(p - 1) * plane32 + offc;
#pragma unroll
        for (int c = 0; c < 5; c++) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.Vn[c] + offp));
        if (a.stage != 1) {
#pragma unroll
          for (int c = 0; c < 5; c++) asm volatile("prefetch.global.L1 [%0];" ::"l"(a.Us[c] + offp));
        }
      }
      T pzn[5];
#pragma unroll
      for (int c = 0; c < 5; c++) pzn[c] = T(0);
      int idp = 0;
      if (rp) {
        int err = ERR_NONE;
        bool chain = false;
        auto item = [&](int it) {
          const int k = EW ? it + 3 : row;  // which extra item (it < 0)
          const int d = it >= 0 ? it : (k == 0 ? 0 : 1);
          const int cx = it < 0 && k == 0 ? (ehi ? TX + 4 : 3) : lane + 4;
          const int cy = it >= 0 ? row + 2 : (k == 0 ? er + 2 : (k == 1 ? 1 : TY + 2));
          if (it >= 0 ? !(it == 0 ? sx_act : (it == 1 ? sy_act : own))
                      : !(in && (k == 0 ? hx_act : (k == 1 ? ylo_act : yhi_act))))
            return;
          T v[5], lo[5], hi[5];
#pragma unroll
          for (int c = 0; c < 5; c++) v[c] = sm.v[s0].v[c][cy][cx];
          const int id = MULTI ? sm.id[s0].v[cy][cx + 12] : 0;
          const Eos<T>& e = eos_of<T, MULTI, SG>(a.s, id);
          int bad = ERR_NONE;
          if (WALLS && id == a.s.nmat) {  // inactive: constant reconstruction, no checks
#pragma unroll
            for (int c = 0; c < 5; c++) lo[c] = hi[c] = v[c];
          } else if constexpr (CONS) {
            cons_states(d, p, cx, cy, id, e, v, bad, lo, hi);
          } else {
            if (it <= 0 || !own) chain = false;  // another cell than in the last iteration
            face_states(d, p, cx, cy, id, e, v, chain, bad, lo, hi);
          }
          if (it >= 0 && bad) err = bad;
          // of a low halo only the high state is read, of a high one only the low state
          const bool put_lo = it >= 0 || (k == 0 ? ehi : k == 2);
          T* plo = d == 0 ? &sm.lox[0][cy - 2][cx - 4] : (d == 1 ? &sm.loy[0][cy - 2][lane] : &sm.loz[0][row][lane]);
          T* phi = d == 0 ? &sm.hix[0][cy - 2][cx - 3] : &sm.hiy[0][cy - 1][lane];
          const int st = d == 0 ? XS : (d == 1 ? YS : ZS);
          if (put_lo) {
#pragma unroll
            for (int c = 0; c < 5; c++) plo[c * st] = lo[c];
          }
          if (it == 2) {
#pragma unroll
            for (int c = 0; c < 5; c++) pzn[c] = hi[c];
          } else if (it >= 0 || !put_lo) {
#pragma unroll
            for (int c = 0; c < 5; c++) phi[c * st] = hi[c];
          }
          if (MULTI && it >= 0) idp = id;
        };
        // Own directions unrolled in the one-material kernel (4% off the FP32
        // stage of a 256^3 box); in the two-material one that spills (3% more).
        if constexpr (MULTI) {
#pragma unroll 1
          for (int it = a_first; it < a_end; it++) item(it);
        } else {
#pragma unroll 1
          for (int it = a_first; it < 0; it++) item(it);
          if (!edge) {
            item(0);
            item(1);
            item(2);
          }
        }
        if (err && own) {
          const int ka = wrap_index(p, g.nz);
          report(a.err, err, (int)(((long long)ka * g.ny + gj) * g.nx + gi), where + 1);
        }
      }
      __syncthreads();
      // ---- B(p): the low x, y and z faces of the cell, last so that F ends as the z flux
      T F[5];
#pragma unroll 1
      for (int it = b_first; it < a_end; it++) {
        const int k = EW ? it + 2 : row - 3;  // which extra item (it < 0): high x faces, high y faces
        const int d = it >= 0 ? it : k;
        if (it >= 0 ? !(it == 0 ? in && fx_act : (it == 1 ? in && fy_act : own && p >= kb))
                    : !(in && (k == 0 ? hfx_act : hfy_act)))
          continue;
        const int cx = it < 0 && k == 0 ? TX + 4 : lane + 4, cy = it >= 0 ? row + 2 : (k == 0 ? er + 2 : TY + 2);
        const int st = d == 0 ? XS : (d == 1 ? YS : ZS);
        const int at = d == 0 ? (cy - 2) * (TX + 1) + cx - 4 : (cy - 2) * TX + lane;
        const T* ph = (d == 0 ? &sm.hix[0][0][0] : &sm.hiy[0][0][0]) + at;
        const T* pl = (d == 0 ? &sm.lox[0][0][0] : (d == 1 ? &sm.loy[0][0][0] : &sm.loz[0][0][0])) + at;
        T VL[5], VR[5];
#pragma unroll
        for (int c = 0; c < 5; c++) {
          VL[c] = d == 2 ? pz[c] : ph[c * st];
          VR[c] = pl[c * st];
        }
        const int f2 = it < 0 ? (1 | ((k == 0 ? hx_act : yhi_act) ? 2 : 0))
                              : (d == 2 ? (real_plane(p - 1) ? 1 : 0) | (rp ? 2 : 0) : lr >> (2 * d));
        const bool rL = f2 & 1, rR = f2 & 2;
        // FP32: faces between blocks of 32 x 16 cells, as their left cells
        // see them, go through a call of their own, whose contraction is the
        // compiler's (see PIN_MOMENTUM): the mixed path's values stay as they were
        if (sizeof(T) == 4 && it < 0 && (k == 0 || ((j0 + TY) & 15) == 0))
          face_flux(std::integral_constant<int, PIN & ~PIN_MOMENTUM>(), k == 0 ? 0 : 1, p, cx, cy, rL, rR, VL, VR, F);
        else
          face_flux(std::integral_constant<int, PIN>(), d, p, cx, cy, rL, rR, VL, VR, F);
        if (d < 2) {
          T* pf = (d == 0 ? &sm.fx[0][0][0] : &sm.fy[0][0][0]) + at;
#pragma unroll
          for (int c = 0; c < 5; c++) pf[c * st] = F[c];
        }
      }
      if (p > kb && own && !face_pass) {
        // F is the flux of face p-1/2: residual + RK update of plane m
        const int m = p - 1;
        const unsigned off = unsigned(m) * plane32 + offc;
        const int id = idprev;
        if (WALLS && id == a.s.nmat) {
          // inactive: no residual (every face gives it a zero flux), and
          // VarFcnDummy's fixed states after every stage (VarFcnDummy.h:44-57)
          const double Vd[5] = {a.s.dummy[0], 0.0, 0.0, 0.0, a.s.dummy[1]};
          const double Ud[5] = {a.s.dummy[0], 0.0, 0.0, 0.0, a.s.dummy[0] * a.s.dummy[2]};
#pragma unroll
          for (int c = 0; c < 5; c++) {
            if (a.Ro[0]) {
              a.Ro[c][off] = 0.0 * inv_mvol;
            } else if (a.final_stage) {
              a.Vo[c][off] = Vd[c];
              if (a.Vfo[0]) a.Vfo[c][off] = float(Vd[c]);
            } else {
              a.Uo[c][off] = Ud[c];
              static_cast<T*>(a.Po[c])[off] = T(Vd[c]);
            }
          }
        } else {
          const Eos<double>& e = eos_of<double, MULTI, SG>(a.s, id);
          double Un[5], Unew[5], Vn[5];
#pragma unroll
          for (int c = 0; c < 5; c++) Vn[c] = a.Vn[c][off];
          e.p2c(Vn, Un);
          if (a.stage == 1) {
#pragma unroll
            for (int c = 0; c < 5; c++) Unew[c] = Un[c];
          } else {
            double Us[5];
#pragma unroll
            for (int c = 0; c < 5; c++) Us[c] = a.Us[c][off];
            if (us_clip) {
              double Vs[5];
              e.c2p(Us, Vs);
              e.clip(Vs);
              e.p2c(Vs, Us);
            }
#pragma unroll
            for (int c = 0; c < 5; c++) Unew[c] = a.a_prev * Us[c] + a.a_un * Un[c];
          }
#pragma unroll
          for (int c = 0; c < 5; c++) {
            double f;
            if constexpr (sizeof(T) == 8) f = part[c] + double(F[c]) * az;
            else f = double(dxy[c] + (F[c] - hl[c]) * azf);
            if (a.visc.fr[0]) {
              // viscous fluxes (ViscosityOperator::AddDiffusionFluxes), added to
              // the flux sum in its cell order: this cell's low x, y, z faces,
              // then the low faces of its +x, +y, +z neighbours
              if (c == 0) {
                f = f + 0.0; f = f + 0.0; f = f + 0.0;
                f = f - 0.0; f = f - 0.0; f = f - 0.0;
              } else {
                const long long Sv = a.visc.nf[0], cc = (long long)(c - 1) * Sv;
                const long long fxi = ((long long)m * g.ny + gj) * (g.nx + 1) + gi;
                const long long fyi = ((long long)m * (g.ny + 1) + gj) * g.nx + gi;
                const long long fzi = ((long long)m * g.ny + gj) * g.nx + gi;
                f = f + a.visc.fr[0][cc + fxi];
                f = f + a.visc.fr[1][cc + fyi];
                f = f + a.visc.fr[2][cc + fzi];
                f = f - a.visc.fl[0][cc + fxi + 1];
                f = f - a.visc.fl[1][cc + fyi + g.nx];
                f = f - a.visc.fl[2][cc + fzi + (long long)g.ny * g.nx];
              }
            }
            if (c == 4 && a.visc.fh[0]) {
              // heat fluxes (HeatDiffusionOperator::AddDiffusionFluxes, after the
              // viscous ones), energy only, in the same cell order
              const long long fxi = ((long long)m * g.ny + gj) * (g.nx + 1) + gi;
              const long long fyi = ((long long)m * (g.ny + 1) + gj) * g.nx + gi;
              const long long fzi = ((long long)m * g.ny + gj) * g.nx + gi;
              f = f + a.visc.fh[0][fxi];
              f = f + a.visc.fh[1][fyi];
              f = f + a.visc.fh[2][fzi];
              f = f - a.visc.fh[0][fxi + 1];
              f = f - a.visc.fh[1][fyi + g.nx];
              f = f - a.visc.fh[2][fzi + (long long)g.ny * g.nx];
            }
            const double R = f * inv_mvol;
            if (a.Ro[0]) a.Ro[c][off] = R;
            Unew[c] = Unew[c] + bdt * R;
          }
          if (!a.Ro[0]) {
            double V[5];
            e.c2p(Unew, V);
            const bool clipped = e.clip(V);
            clipped_local |= clipped ? 1 : 0;
            if (e.bad(V))
              report(a.err, ERR_STATE, (int)((long long)m * g.ny * g.nx + (long long)gj * g.nx + gi), where + 3);
            if (a.final_stage) {
#pragma unroll
              for (int c = 0; c < 5; c++) a.Vo[c][off] = V[c];
              if (a.Vfo[0]) {
#pragma unroll
                for (int c = 0; c < 5; c++) a.Vfo[c][off] = float(V[c]);
              }
              const double ee = e.energy(V[0], V[4]);
              const double c2 = e.c2(V[0], ee);
              if (c2 < 0.0) report(a.err, ERR_SOUND, (int)off, where + 4);
              const double cs = sqrt(c2);
#pragma unroll
              for (int d = 0; d < 3; d++) lmax[d] = smax(lmax[d], fabs(V[1 + d]) + cs);
            } else {
#pragma unroll
              for (int c = 0; c < 5; c++) a.Uo[c][off] = Unew[c];
              // the next stage's input: clip(C2P(U_new)), as it would recompute it
#pragma unroll
              for (int c = 0; c < 5; c++) static_cast<T*>(a.Po[c])[off] = T(V[c]);
            }
          }
        }
      }
      // the halo of the plane after next
      if (p + 2 <= ke + 1 && real_plane(p + 2)) {
        landed = wait_plane(p + 2);
        if (landed) fix_plane(p + 2);
      }
      if (__syncthreads_or(!landed)) return;
      // ---- C(p)
      if (copier && p + RING - 1 <= ke + 1 && real_plane(p + RING - 1)) issue_plane(p + RING - 1);
      if (in && own && !face_pass) {
        const double dzk = g.dz[p];
        if (dzk != dzc) {
          ax = dyj * dzk;
          ay = dxi * dzk;
          axf = float(ax);
          ayf = float(ay);
          if (dzc != 0.0) dtmin_local = smin(dtmin_local, dzc / lmax[2]);
          lmax[2] = 0.0;
          dzc = dzk;
          const double vol = dxi * dyj * dzk;
          // Vec5D::operator/= multiplies by the reciprocal (Vector5D.h:172-181)
          inv_mvol = 1.0 / (-vol);
        }
        // Low faces, the flux this cell sees as the right-hand cell
        // (SpaceOperator.cpp:2555-2556, 2683-2684, 2810-2811). Low faces that
        // are material interfaces under the NUMERICAL interface flux: this
        // cell's flux is its EOS's numerical flux between the right star state
        // and its own cell-centred state (SpaceOperator.cpp:2499-2542), or
        // under LINEAR interface reconstruction its reconstructed state. Low
        // faces cut by an embedded surface likewise take this cell's flux
        // against its one-sided star state (SpaceOperator.cpp:2462-2478).
        T FL[3][5];
#pragma unroll
        for (int c = 0; c < 5; c++) {
          FL[0][c] = sm.fx[c][row][lane];
          FL[1][c] = sm.fy[c][row][lane];
          FL[2][c] = F[c];
        }
        if constexpr (MULTI) {
          const unsigned off = unsigned(p) * plane32 + offc;
          const int wm = WALLS ? a.wall.mask[off] : 0;
          int fm = wm;
          if (a.iface.mp_flux == 1) {  // set only with interface slots (two-material contexts)
            fm |= (idp != sm.id[s0].v[row + 2][lane + 15] ? 1 : 0) | (idp != sm.id[s0].v[row + 1][lane + 16] ? 2 : 0) |
                  (real_plane(p - 1) && idp != idprev ? 4 : 0);
          }
          if (fm) {
            auto own_side = [&](int d) {
              if (!((fm >> d) & 1)) return;
              const bool w = (wm >> d) & 1;
              const T* ps = (w ? a.wall.linear : a.iface.mp_recon)
                                ? (d == 0 ? &sm.lox[0][row][lane] : (d == 1 ? &sm.loy[0][row][lane] : &sm.loz[0][row][lane]))
                                : &sm.v[s0].v[0][row + 2][lane + 4];
              const int st = (w ? a.wall.linear : a.iface.mp_recon) ? (d == 0 ? XS : (d == 1 ? YS : ZS)) : CS;
              const long long sl = w ? a.wall.slot[off] : a.iface.slot[off];
              const double* src = (w ? a.wall.Vsp : a.iface.Vsp) + (sl * 3 + d) * 5;
              T W[5], Sp[5], F2[5];
#pragma unroll
              for (int c = 0; c < 5; c++) {
                W[c] = ps[c * st];
                Sp[c] = T(src[c]);
              }
              const int err2 = flux_of<T, FLUX, PIN>(eos_of<T, MULTI, SG>(a.s, idp), d, Sp, W, delta, F2);
              if (err2) report(a.err, err2, -1, where + 2);
#pragma unroll
              for (int c = 0; c < 5; c++) {
                FL[0][c] = d == 0 ? F2[c] : FL[0][c];
                FL[1][c] = d == 1 ? F2[c] : FL[1][c];
                FL[2][c] = d == 2 ? F2[c] : FL[2][c];
              }
            };
#pragma unroll 1
            for (int d = 0; d < 3; d++) own_side(d);
          }
        }
#pragma unroll
        for (int c = 0; c < 5; c++) {
          const T fr = sm.fx[c][row][lane + 1], gr = sm.fy[c][row + 1][lane];
          if constexpr (sizeof(T) == 8) {
            // FP64: the reference's order, 0 - Fl A - Gl A - Hl A + Fr A + Gr A + Hr A
            double f = 0.0;
            f = f - FL[0][c] * ax;
            f = f - FL[1][c] * ay;
            f = f - FL[2][c] * az;
            f = f + double(fr) * ax;
            f = f + double(gr) * ay;
            part[c] = f;
          } else {
            // mixed: FP32 accumulation of the flux differences (the difference
            // of two nearby FP32 fluxes is exact), one conversion per component
            dxy[c] = (fr - FL[0][c]) * axf + (gr - FL[1][c]) * ayf;
            hl[c] = FL[2][c];
          }
        }
      }
      idprev = idp;
#pragma unroll
      for (int c = 0; c < 5; c++) pz[c] = pzn[c];
    }
    if (own) {
      dtmin_local = smin(dtmin_local, smin(dxi / lmax[0], smin(dyj / lmax[1], dzc / lmax[2])));
      lmax[0] = lmax[1] = lmax[2] = 0.0;
    }
  }

  if (a.clipped_out && __syncthreads_or(clipped_local)) {
    if (lane == 0 && row == 0) atomicOr(a.clipped_out, 1);
  }
  if (a.final_stage && a.dtmin_bits) {
    double v = dtmin_local;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = smin(v, __shfl_xor_sync(0xffffffffu, v, o));
    __syncthreads();
    if (lane == 0 && row < TY) sm.red[row] = v;
    __syncthreads();
    if (lane == 0 && row == 0) {
      double r = sm.red[0];
      for (int q = 1; q < TY; q++) r = smin(r, sm.red[q]);
      if (r < 1.0e300) atomicMin(a.dtmin_bits, (unsigned long long)__double_as_longlong(r));
    }
  }
}

}  // namespace m2c
