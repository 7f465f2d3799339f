// omhd_fused3d.cuh -- one fused kernel per TVD-RK2 stage for 3D grids.
//
// A CTA owns a TX x TY column of interior cells and marches it through a
// chunk of z planes.  A ring of four primitive planes (k-1 .. k+2, each with
// a two-cell x/y halo) lives in shared memory, so the conserved->primitive
// recovery of every plane is done once per CTA; per plane the CTA
//   - loads and converts plane k+2 (u2v.f90, first GLM half in stage 1),
//   - builds x and y face states and fluxes of plane k in shared memory
//     (limiter.f90, flux_solver.f90, bc_for_F/G face fixes),
//   - reconstructs cell k+1 in z and solves the z face k+1/2 in registers,
//     carrying the z flux of face k-1/2 from the previous plane,
//   - updates plane k (rk.f90), fills ghosts by owner writes (bc),
//     applies the second GLM half and the CFL reduction in stage 2.
// Resistive fluxes (3D_reconnection_gpu/flux_resistive.cuf) are added at
// each face from cell-centred B in the ring.
#pragma once
#include "omhd_fused.h"
#include "omhd_step.cuh"

#ifndef OMHD_VARIANT
#error "define OMHD_VARIANT before including omhd_fused3d.cuh"
#endif

namespace omhd {
namespace OMHD_VARIANT {
namespace d3 {

// A column of TX x TY cells and the CTAs per SM its kernel is built for.
template <int TX_, int TY_, int CTAS_, int EXTRA_ = 0>
struct Col {
  static constexpr int TX = TX_, TY = TY_, CTAS = CTAS_, CELLS = TX * TY;
  static constexpr int NT = CELLS + 32 * EXTRA_;  // EXTRA_ warps without cells
  static_assert(TY * NV <= NT - TX, "the x and y wall fixes use disjoint threads");
  static constexpr int RX = TX + 4, RY = TY + 4, PL = RX * RY;  // plane of the halo tile
  static constexpr int XS = TX + 2, NXS3 = TY * XS;             // cells reconstructed in x (a row strip per tile row)
  static constexpr int NYS3 = (TY + 2) * TX;                    // cells reconstructed in y
  static constexpr int XF = TX + 1, NXF3 = TY * XF;             // x faces
  static constexpr int NXFP3 = (NXF3 + 31) / 32 * 32;           // x faces padded to whole warps
  static constexpr int NYF3 = (TY + 1) * TX;                    // y faces
  // ring of NRING primitive planes, then the x and y face states of one plane;
  // each face's flux overwrites the lower-cell face state that only it reads
  template <class T>
  static constexpr size_t smem_bytes() {
    return sizeof(T) * (size_t)NV * (4 * PL + 2 * NXS3 + 2 * NYS3);
  }
};
// The column of the other builds than the FP64 performance one: 32x8, FP32 two
// CTAs per SM (build-time constants, for tuning)
#ifndef OMHD_3D_TILE_X
#define OMHD_3D_TILE_X 32
#endif
#ifndef OMHD_3D_TILE_Y
#define OMHD_3D_TILE_Y 8
#endif
#ifndef OMHD_3D_MIXED_MIN_CTAS  // resident CTAs per SM the FP32-mixed 3D kernel is built for
#define OMHD_3D_MIXED_MIN_CTAS 2
#endif
template <class T>
using DefaultCol = Col<OMHD_3D_TILE_X, OMHD_3D_TILE_Y, sizeof(T) == 4 ? OMHD_3D_MIXED_MIN_CTAS : 1>;
// FP64 HLLD with fused multiply-adds: 16x16, or two 16x8 CTAs per SM
// (small_columns), with a warp more than the cells need.  The 16x16 plane's 288
// pairs of face states and 544 x and y faces are 9 and 17 warps' worth, which eight
// warps did in rounds of 8 and 1: a warp alone on the SM gets a third of the FP64
// pipe, and a quarter of a plane's time went that way (168 registers with 444 bytes
// spilled instead of 255; Harris 256x128x256 33.3 -> 28.6 ms per step, two extra
// warps 28.8, mixed 6.17 -> 6.75: not used there).  16x8: loop 100x100x200 5.70 -> 5.25.
using WideCol = Col<16, 16, 1, 1>;
using SmallCol = Col<16, 8, 2, 1>;
using SquareCol = Col<16, 16, 2>;  // FP32-mixed HLLD, beside 32x8 (square_columns)
constexpr int NRING = 4;
constexpr int ZCHUNK = 64;  // most z planes marched by one CTA

// z planes per CTA for a grid of `columns` columns and nz interior planes on a
// device that runs `slots` CTAs at a time.  Every CTA costs its planes plus a
// prologue (four plane loads and one z face, about kProloguePlanes planes), and
// the launch as many rounds of CTAs as it takes, so the split with the smallest
// rounds x (planes + prologue) is taken: small grids are cut into short chunks
// until every SM has a CTA, large ones so that the last round is nearly full.
// Against fixed chunks of 64 planes (ms per step on GB300): Harris 64x32x64 FP64
// 12.3 -> 0.95 (8 CTAs before), field loop 100x100x200 FP64 15.9 -> 10.4 (208 CTAs
// in two rounds), Harris 256x128x256 mixed 10.5 -> 9.4 (512 CTAs on 304 slots).
constexpr double kProloguePlanes = 1.5;
inline int pick_zchunk(long long columns, int nz, int slots, double* cost_out = nullptr) {
  int best = ZCHUNK;
  double best_cost = 1e300;
  for (int c = nz < ZCHUNK ? nz : ZCHUNK; c >= 1; --c) {
    const long long chunks = (nz + c - 1) / c;
    if (chunks > 65535) break;  // gridDim.z
    const double cost = (double)((columns * chunks + slots - 1) / slots) * (c + kProloguePlanes);
    if (cost < best_cost) {
      best_cost = cost;
      best = c;
    }
  }
  if (cost_out) *cost_out = best_cost;
  return best;
}

__device__ __forceinline__ int map_idx(int g, int n, bool periodic) {
  if (g >= 0 && g < n) return g;
  if (periodic) {
    const int P = n - 2;
    int r = (g - 1) % P;
    if (r < 0) r += P;
    return r + 1;
  }
  return g < 0 ? 0 : n - 1;
}

__device__ __forceinline__ double eta3(int kind, double x, double y, double z) {
  if (kind == OMHD_ETA_RECON2D) {  // 2D_reconnection/flux_resistive.f90:1-16 (as coded in the 3D GPU driver)
    const double Rm1 = 60.0, Rm0 = 1000.0;
    const double eta0 = 1.0 / Rm0;
    const double eta01 = (Rm0 - Rm1) / (Rm0 * Rm1);
    const double c = cosh(fmin2(sqrt(x * x + y * y), 25.0));
    return eta0 + eta01 * (1.0 / (c * c));
  }
  if (kind == OMHD_ETA_HARRIS_XZ) return 1.0e-3 + (1.0 / 60.0) * exp(-(x * x + z * z) / 4.0);
  return 0.0;
}

// eta / dx of the Harris resistivity, eta = 1e-3 + exp(-(x^2+z^2)/4)/60, from
// the factors ex = exp(-x^2/4) and ez = exp(-z^2/4), in the arithmetic type R
template <class R>
__device__ __forceinline__ R harris_eta_dx(R ex, R ez, R inv_dx) {
  return (R(1.0e-3) + R(1.0 / 60.0) * (ex * ez)) * inv_dx;
}

// Resistive terms of the FP32-mixed kernels (flux_resistive.cuf:87-135) in
// binary32, added to the binary32 face flux they belong to.  Each current
// component is a difference of cell-centred B across the face plus a quarter
// of a four-point transverse difference; the four-point sums are formed as two
// neighbour differences, which binary32 subtracts exactly when the neighbours
// are within a factor of two (Sterbenz), so the current keeps its relative
// precision where it is small.  b(var, dx, dy, dz) reads B of the cell at that
// offset from the face's lower cell; the face normal is axis n (1, 2, 3).
template <int n, class BF>
__device__ __forceinline__ void resist_face_f32(const BF& b, float eta_dx, float (&Fo)[NV]) {
  if constexpr (n == 1) {  // x face (:87-101)
    const float JyS = (b(BZ, 0, 0, 0) - b(BZ, 1, 0, 0)) +
                      0.25f * ((b(BX, 0, 0, 1) - b(BX, 0, 0, -1)) + (b(BX, 1, 0, 1) - b(BX, 1, 0, -1)));
    const float JzS = (b(BY, 1, 0, 0) - b(BY, 0, 0, 0)) -
                      0.25f * ((b(BX, 0, 1, 0) - b(BX, 0, -1, 0)) + (b(BX, 1, 1, 0) - b(BX, 1, -1, 0)));
    Fo[EN] += 0.5f * eta_dx * (JyS * (b(BZ, 0, 0, 0) + b(BZ, 1, 0, 0)) - JzS * (b(BY, 0, 0, 0) + b(BY, 1, 0, 0)));
    Fo[BY] -= eta_dx * JzS;
    Fo[BZ] += eta_dx * JyS;
  } else if constexpr (n == 2) {  // y face (:104-118)
    const float JxS = (b(BZ, 0, 1, 0) - b(BZ, 0, 0, 0)) -
                      0.25f * ((b(BY, 0, 0, 1) - b(BY, 0, 0, -1)) + (b(BY, 0, 1, 1) - b(BY, 0, 1, -1)));
    const float JzS = (b(BX, 0, 0, 0) - b(BX, 0, 1, 0)) +
                      0.25f * ((b(BY, 1, 0, 0) - b(BY, -1, 0, 0)) + (b(BY, 1, 1, 0) - b(BY, -1, 1, 0)));
    Fo[EN] += 0.5f * eta_dx * (JzS * (b(BX, 0, 0, 0) + b(BX, 0, 1, 0)) - JxS * (b(BZ, 0, 0, 0) + b(BZ, 0, 1, 0)));
    Fo[BX] += eta_dx * JzS;
    Fo[BZ] -= eta_dx * JxS;
  } else {  // z face (:121-135)
    const float JyS = (b(BX, 0, 0, 1) - b(BX, 0, 0, 0)) -
                      0.25f * ((b(BZ, 1, 0, 0) - b(BZ, -1, 0, 0)) + (b(BZ, 1, 0, 1) - b(BZ, -1, 0, 1)));
    const float JxS = (b(BY, 0, 0, 0) - b(BY, 0, 0, 1)) +
                      0.25f * ((b(BZ, 0, 1, 0) - b(BZ, 0, -1, 0)) + (b(BZ, 0, 1, 1) - b(BZ, 0, -1, 1)));
    Fo[EN] += 0.5f * eta_dx * (JxS * (b(BY, 0, 0, 0) + b(BY, 0, 0, 1)) - JyS * (b(BX, 0, 0, 0) + b(BX, 0, 0, 1)));
    Fo[BX] -= eta_dx * JyS;
    Fo[BY] += eta_dx * JxS;
  }
}

// The same terms of the FP64 kernels, added to the face flux F (grid components);
// b as above, n = 0, 1, 2 the face normal's axis.
template <int n, class BF>
__device__ __forceinline__ void resist_face_f64(const BF& B, double eta_dx, double (&F)[NV]) {
  if constexpr (n == 0) {  // flux_resistive.cuf:87-101
    const double JyS = -(B(BZ, 1, 0, 0) - B(BZ, 0, 0, 0)) +
                       0.25 * (B(BX, 0, 0, 1) + B(BX, 1, 0, 1) - B(BX, 0, 0, -1) - B(BX, 1, 0, -1));
    const double JzS = (B(BY, 1, 0, 0) - B(BY, 0, 0, 0)) -
                       0.25 * (B(BX, 0, 1, 0) + B(BX, 1, 1, 0) - B(BX, 0, -1, 0) - B(BX, 1, -1, 0));
    F[EN] = F[EN] + 0.5 * eta_dx * (JyS * (B(BZ, 0, 0, 0) + B(BZ, 1, 0, 0)) - JzS * (B(BY, 0, 0, 0) + B(BY, 1, 0, 0)));
    F[BY] = F[BY] - eta_dx * JzS;
    F[BZ] = F[BZ] + eta_dx * JyS;
  } else if constexpr (n == 1) {  // flux_resistive.cuf:104-118
    const double JxS = (B(BZ, 0, 1, 0) - B(BZ, 0, 0, 0)) -
                       0.25 * (B(BY, 0, 0, 1) + B(BY, 0, 1, 1) - B(BY, 0, 0, -1) - B(BY, 0, 1, -1));
    const double JzS = -(B(BX, 0, 1, 0) - B(BX, 0, 0, 0)) +
                       0.25 * (B(BY, 1, 0, 0) + B(BY, 1, 1, 0) - B(BY, -1, 0, 0) - B(BY, -1, 1, 0));
    F[EN] = F[EN] + 0.5 * eta_dx * (JzS * (B(BX, 0, 0, 0) + B(BX, 0, 1, 0)) - JxS * (B(BZ, 0, 0, 0) + B(BZ, 0, 1, 0)));
    F[BX] = F[BX] + eta_dx * JzS;
    F[BZ] = F[BZ] - eta_dx * JxS;
  } else {  // flux_resistive.cuf:121-135
    const double JyS = (B(BX, 0, 0, 1) - B(BX, 0, 0, 0)) -
                       0.25 * (B(BZ, 1, 0, 0) + B(BZ, 1, 0, 1) - B(BZ, -1, 0, 0) - B(BZ, -1, 0, 1));
    const double JxS = -(B(BY, 0, 0, 1) - B(BY, 0, 0, 0)) +
                       0.25 * (B(BZ, 0, 1, 0) + B(BZ, 0, 1, 1) - B(BZ, 0, -1, 0) - B(BZ, 0, -1, 1));
    F[EN] = F[EN] + 0.5 * eta_dx * (JxS * (B(BY, 0, 0, 0) + B(BY, 0, 0, 1)) - JyS * (B(BX, 0, 0, 0) + B(BX, 0, 0, 1)));
    F[BX] = F[BX] - eta_dx * JyS;
    F[BY] = F[BY] + eta_dx * JxS;
  }
}

// slot k of a face state rotated into x orientation holds component rot3(n, k) for
// the face normal n = 0, 1, 2 (x, y, z), the component order of flux_solver.f90
__device__ __forceinline__ constexpr int rot3(int n, int k) {
  return (k <= 2) ? (k + n) % 3 : ((k >= 5 && k <= 7) ? 5 + (k - 5 + n) % 3 : k);
}

// Load + convert one z plane (global index gk, any value; mapped by the z bc)
// of the halo tile into ring slot `slot`.
template <class T, class G>
__device__ __forceinline__ void load_plane(const StageArgs& a, T* W, int slot, int gk, int gi0, int gj0, bool perx,
                                           bool pery, bool perz, bool resist, double glmf) {
  constexpr int TX = G::TX, TY = G::TY, NT = G::NT, RX = G::RX, RY = G::RY, PL = G::PL;
  const int ix = a.ix, jx = a.jx, kx = a.kx;
  const size_t N = (size_t)ix * jx * kx;
  const double f1g = a.gm1;  // derived on the host
  const float f1g32 = a.gm1_f;
  const int mk = map_idx(gk, kx, perz);
  T* Ws = W + (size_t)slot * NV * PL;
  for (int q = threadIdx.x; q < PL; q += NT) {
    const int rx = q % RX, ry = q / RX;
    const bool cx_in = rx >= 2 && rx < TX + 2, cy_in = ry >= 2 && ry < TY + 2;
    if (!cx_in && !cy_in) {
      if (!resist || rx == 0 || rx == RX - 1 || ry == 0 || ry == RY - 1) continue;
    }
    const int gi = gi0 - 2 + rx, gj = gj0 - 2 + ry;
    const size_t c = (size_t)map_idx(gi, ix, perx) + (size_t)ix * ((size_t)map_idx(gj, jx, pery) + (size_t)jx * mk);
    const double* U = a.Uin;
    double u[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) u[v] = U[v * N + c];
    double ps = u[PS];
    if (a.stage == 1) ps = glmf * ps;
    T w[NV];
    double pr, ro;
    u2v_cell<T, OMHD_FAST, OMHD_FAST && sizeof(T) == 8>(u, f1g, f1g32, ps, w, pr, ro);  // 3D_basic/u2v.f90
#pragma unroll
    for (int v = 0; v < NV; ++v) Ws[v * PL + q] = w[v];
  }
}

// FP32 face arithmetic: two CTAs per SM (registers capped at 128, 97 KB of
// shared memory each), so that one CTA's FP64 loads, updates and barriers
// overlap the other's face work.
template <class T, int FLUX, class G>
__global__ void __launch_bounds__(G::NT, G::CTAS) k_stage3d(const StageArgs a, const int zchunk) {
  constexpr int TX = G::TX, TY = G::TY, NT = G::NT, RX = G::RX, PL = G::PL, XS = G::XS, XF = G::XF;
  constexpr int NXS3 = G::NXS3, NYS3 = G::NYS3, NXF3 = G::NXF3, NXFP3 = G::NXFP3, NYF3 = G::NYF3;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* W = reinterpret_cast<T*>(smem_raw);  // [NRING][NV][PL]
  T* SLx = W + NRING * NV * PL;  // [NV][NXS3]; x fluxes in place
  T* SRx = SLx + NV * NXS3;
  T* SLy = SRx + NV * NXS3;      // [NV][NYS3]; y fluxes in place
  T* SRy = SLy + NV * NYS3;
  __shared__ double red32[32];
  __shared__ int skip;

  StepState* st = a.st;
  // one thread decides, so that the whole CTA leaves together
  if (threadIdx.x == 0) skip = st->done || *(volatile int*)&a.err->code;
  __syncthreads();
  if (skip) return;
  const double dt = st->dt, chd = st->ch, glmf = st->glm_f;
  const int ix = a.ix, jx = a.jx, kx = a.kx;
  const size_t N = (size_t)ix * jx * kx;
  const int tid = threadIdx.x;
  const int gi0 = 1 + blockIdx.x * TX, gj0 = 1 + blockIdx.y * TY;
  const int k0 = 1 + blockIdx.z * zchunk;
  const int k1 = min(k0 + zchunk - 1, kx - 2);
  const bool perx = a.bc_kind[0] == OMHD_BC_PERIODIC, pery = a.bc_kind[2] == OMHD_BC_PERIODIC;
  const bool perz = a.bc_kind[4] == OMHD_BC_PERIODIC;
  const bool resist = a.eta_kind != OMHD_ETA_NONE;
  const double gamma = a.gamma;
  // gamma constants derived on the host (stage_args_derived)
  const double f1g = a.gm1;
  const T ch = to_face<T>(chd);
  T gam, r1, r2;
  if constexpr (sizeof(T) == 4) {
    gam = a.gamma_f;
    r1 = a.r1_f;
    r2 = a.r2_f;
  } else {
    gam = gamma;
    r1 = a.r1;
    r2 = a.r2;
  }
  const int lm = a.lm_type;
  // the thread's cell; a warp without cells keeps the indices of some and owns none
  const int tx = tid % TX, ty = tid % G::CELLS / TX;
  const int gi = gi0 + tx, gj = gj0 + ty;
  const bool own = tid < G::CELLS && gi <= ix - 2 && gj <= jx - 2;
  const int oc = (ty + 2) * RX + (tx + 2);  // own column in a ring plane
  // dt/dx as dt * (dtx_scale/dx) in the FAST builds (within an ulp), the
  // reference's division in the parity build
  const double dtx = OMHD_FAST ? dt * a.sdx : a.dtx_scale * dt / a.dx;
  const double dty = OMHD_FAST ? dt * a.sdy : a.dtx_scale * dt / a.dy;
  const double dtz = OMHD_FAST ? dt * a.sdz : a.dtx_scale * dt / a.dz;
  auto slot = [](int k) { return ((k % NRING) + NRING) % NRING; };
  auto Wv = [&](int k, int v, int o) -> T { return W[(size_t)slot(k) * NV * PL + v * PL + o]; };

  // The Harris resistivity is separable in x and z: in the FAST builds its
  // exponential is tabulated over this CTA's x columns (cell centres ex_c and
  // x faces ex_f, index q = i - gi0 + 1) and z chunk (ez_c, ez_f at z faces,
  // index p = k - k0 + 1), one exp per entry instead of one per face.
  __shared__ T ex_c[TX + 2], ex_f[TX + 2], ez_c[ZCHUNK + 2], ez_f[ZCHUNK + 2];
  const bool sep_eta = OMHD_FAST && a.eta_kind == OMHD_ETA_HARRIS_XZ;
  const double inv_dx = 1.0 / a.dx;
  const T inv_dx_t = T(inv_dx);
  if (sep_eta) {
    const int nez = k1 - k0 + 3;  // planes k0-1 .. k1+1
    for (int q = tid; q < 2 * (TX + 2) + 2 * nez; q += NT) {
      if (q < 2 * (TX + 2)) {
        const int p = q % (TX + 2);
        const double x = a.xc[min(gi0 - 1 + p, ix - 1)] + (q >= TX + 2 ? 0.5 * a.dx : 0.0);
        (q < TX + 2 ? ex_c : ex_f)[p] = to_face<T>(exp(-(x * x) / 4.0));
      } else {
        const int r = q - 2 * (TX + 2), p = r < nez ? r : r - nez;
        const double z = a.zc[min(k0 - 1 + p, kx - 1)] + (r >= nez ? 0.5 * a.dx : 0.0);
        (r < nez ? ez_c : ez_f)[p] = to_face<T>(exp(-(z * z) / 4.0));
      }
    }
  }

  // ---- prologue: planes k0-2 .. k0+1, then the z face k0-1/2 ----
  for (int p = k0 - 2; p <= k0 + 1; ++p)
    load_plane<T, G>(a, W, slot(p), p, gi0, gj0, perx, pery, perz, resist, glmf);
  __syncthreads();
  T sLc[NV];  // z-upper face state of the current cell (k)
  double Fzp[NV] = {};  // z flux through face k-1/2
  // The face below the chunk's first plane is solved by the loop's own code in a
  // leading iteration k0-1 that does nothing else, so that a run's results do not
  // depend on where the chunks begin.
  const bool lead_in = sizeof(T) == 8 || (k0 - 1) % ZCHUNK != 0;
  if (lead_in) {
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      T r;
      reconstruct_t<T, OMHD_FAST>(lm, Wv(k0 - 2, v, oc), Wv(k0 - 1, v, oc), Wv(k0, v, oc), sLc[v], r);
    }
  }
  double vloc = 0.0;
  // the FP64 performance build solves all faces in one loop (the FP32 and parity
  // builds keep a copy of the solver per direction: another component order changes
  // their rounding)
  constexpr bool kOneSolver = OMHD_FAST && sizeof(T) == 8;

  for (int k = lead_in ? k0 - 1 : k0; k <= k1; ++k) {
    const bool lead = k < k0;  // only the z face k+1/2 (uniform over the CTA)
    const float known = OMHD_FAST && a.stage == 2 ? cfl_known(st) : 0.0f;  // read a plane ahead of its use
    // Three CTA barriers per plane (plus one where a wall fix is needed).  The
    // ring slot of plane k+2 held plane k-2, whose last readers (the resistive
    // terms of plane k-1) finished before the previous plane's flux barrier;
    // the face arrays are rewritten only after the barrier that follows this
    // load, which every thread reaches after its reads of the previous plane's
    // fluxes.  The chunk's first z face (and a seam's) reads plane k-2: one
    // barrier before the load.
    if (!lead) {
      // FP32: the z face below every ZCHUNK-th plane enters that plane's update
      // through this second copy of the solver, which the compiler contracts
      // differently from the loop's; with chunks of ZCHUNK planes it was the first
      // face of a chunk, and keeping it there gives a mixed run the same bits for
      // every split
      const bool every = (k - 1) % ZCHUNK == 0, seam = sizeof(T) == 4 && every;
      if constexpr (sizeof(T) == 4) {
        if (seam) {
          T L[NV], R[NV], Fo[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            T l, r;
            reconstruct_t<T, OMHD_FAST>(lm, Wv(k - 2, v, oc), Wv(k - 1, v, oc), Wv(k, v, oc), l, r);
            L[v] = l;  // upper state of cell k-1
            reconstruct_t<T, OMHD_FAST>(lm, Wv(k - 1, v, oc), Wv(k, v, oc), Wv(k + 1, v, oc), l, r);
            R[v] = r;  // lower state of cell k
            sLc[v] = l;
          }
          if (!perz && k == 1) {  // bottom wall: VL = flip(VR)  (3D_reconnection_gpu/bc.cuf bc_for_H pattern)
#pragma unroll
            for (int v = 0; v < NV; ++v) L[v] = ((a.bc_flip[4] >> v) & 1) ? -R[v] : R[v];
          }
          riemann_flux<T, 3, FLUX, OMHD_FAST>(L, R, ch, gam, r1, r2, Fo);
#pragma unroll
          for (int v = 0; v < NV; ++v) Fzp[v] = to_f64<T>(Fo[v]);
          if (resist && own) {  // z face k-1/2 (flux_resistive.cuf:121-135)
            const int kl = k - 1;
            auto b = [&](int var, int dxo, int dyo, int dzo) { return Wv(kl + dzo, var, oc + dxo + dyo * RX); };
            const float eta_dx = sep_eta ? harris_eta_dx<T>(ex_c[tx + 1], ez_f[k - k0], inv_dx_t)
                                         : narrow_f64(eta3(a.eta_kind, a.xc[gi], a.yc[gj], a.zc[kl] + 0.5 * a.dx) / a.dx);
            resist_face_f32<3>(b, eta_dx, Fo);
#pragma unroll
            for (int v = 0; v < NV; ++v) Fzp[v] = to_f64<T>(Fo[v]);
          }
        }
      }
      if (k == k0 || seam) __syncthreads();
      load_plane<T, G>(a, W, slot(k + 2), k + 2, gi0, gj0, perx, pery, perz, resist, glmf);
      __syncthreads();
      // positivity of the plane's own cells (u2v.f90:36-45).  NaN counts on every
      // ZCHUNK-th plane, where the FP32 build also judges the FP64 values: wherever the
      // chunks begin, so that which states a run refuses does not depend on the cut
      if (own) {
        double ro, pr;
        if (seam) {
          double u[NV];
          T w[NV];
          const size_t c = (size_t)gi + (size_t)ix * ((size_t)gj + (size_t)jx * k);
#pragma unroll
          for (int v = 0; v < NV; ++v) u[v] = a.Uin[v * N + c];
          u2v_cell<T, OMHD_FAST, OMHD_FAST && sizeof(T) == 8>(u, a.gm1, a.gm1_f, u[PS], w, pr, ro);
        } else {
          ro = to_f64<T>(Wv(k, RO, oc));
          pr = to_f64<T>(Wv(k, PR, oc));
        }
        auto refused = [&](double x) { return !gt0_<true>(x) && (every || x == x); };
        if (refused(pr))
          raise_error(a.err, OMHD_NEG_PRESSURE, gi + 1, gj + 1, k + 1, 0, pr);
        else if (refused(ro))
          raise_error(a.err, OMHD_NEG_DENSITY, gi + 1, gj + 1, k + 1, 0, ro);
      }
      const T* Wk = W + (size_t)slot(k) * NV * PL;

      // ---- x and y face states of plane k, one phase ----
      bool paired = false;
      if constexpr (kOneSolver) {
        if (lm == LM_MINMOD || lm == LM_MC) {
          // two neighbouring cells of a strip per item, their shared slope once
          paired = true;
          constexpr int XP = XS / 2, NXP = NXS3 / 2, NYP = NYS3 / 2;
          static_assert(XS % 2 == 0 && (TY + 2) % 2 == 0, "cell pairs need even strip lengths");
#pragma unroll 1
          for (int p = tid; p < NXP + NYP; p += NT) {
            const bool xd = p < NXP;
            const int pp = xd ? p : p - NXP;
            const int ca = xd ? 2 * (pp % XP) : pp % TX, cb = xd ? pp / XP : 2 * (pp / TX);
            const int o = xd ? (cb + 2) * RX + (ca + 1) : (cb + 1) * RX + (ca + 2);
            const int st = xd ? 1 : RX, i0 = xd ? cb * XS + ca : cb * TX + ca, di = xd ? 1 : TX;
            T* dl = xd ? SLx : SLy;
            T* dr = xd ? SRx : SRy;
            const int sv = xd ? NXS3 : NYS3;
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              const T* w = Wk + v * PL + o;
              const T wm = w[-st], w0 = w[0], w1 = w[st], w2 = w[2 * st];
              const T d0 = w0 - wm, d1 = w1 - w0, d2 = w2 - w1;
              reconstruct_fp64_g(lm, d0, d1, wm, w0, w1, dl[v * sv + i0], dr[v * sv + i0]);
              reconstruct_fp64_g(lm, d1, d2, w0, w1, w2, dl[v * sv + i0 + di], dr[v * sv + i0 + di]);
            }
          }
        }
      }
      for (int q = tid; !paired && q < NXS3 + NYS3; q += NT) {
        const bool xd = q < NXS3;
        const int qq = xd ? q : q - NXS3;
        int o, st;
        if (xd) {  // x row cy, cells cx = 0..TX+1 (tile columns -1..TX)
          const int cx = qq % XS, cy = qq / XS;
          o = (cy + 2) * RX + (cx + 1);
          st = 1;
        } else {  // y column cx, cells cy = 0..TY+1 (tile rows -1..TY)
          const int cx = qq % TX, cy = qq / TX;
          o = (cy + 1) * RX + (cx + 2);
          st = RX;
        }
        T* dl = xd ? SLx : SLy;
        T* dr = xd ? SRx : SRy;
        const int sv = xd ? NXS3 : NYS3;
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          T l, r;
          reconstruct_t<T, OMHD_FAST>(lm, Wk[v * PL + o - st], Wk[v * PL + o], Wk[v * PL + o + st], l, r);
          dl[v * sv + qq] = l;
          dr[v * sv + qq] = r;
        }
      }
      __syncthreads();
      if (!perx || !pery) {  // wall face fixes, x by the first threads, y by the last
        if (!perx && tid < TY * NV) {
          const int cy = tid % TY, v = tid / TY;
          if (gi0 == 1) {
            const T s = SRx[v * NXS3 + cy * XS + 1];
            SLx[v * NXS3 + cy * XS + 0] = ((a.bc_flip[0] >> v) & 1) ? -s : s;
          }
          const int cl = (ix - 2) - gi0 + 1;
          if (cl >= 1 && cl <= TX) {
            const T s = SLx[v * NXS3 + cy * XS + cl];
            SRx[v * NXS3 + cy * XS + cl + 1] = ((a.bc_flip[1] >> v) & 1) ? -s : s;
          }
        }
        if (!pery && tid >= NT - TX) {
          const int cx = tid - (NT - TX);
          const int cl = (jx - 2) - gj0 + 1;
          for (int v = 0; v < NV; ++v) {
            if (gj0 == 1) {
              const T s = SRy[v * NYS3 + 1 * TX + cx];
              SLy[v * NYS3 + 0 * TX + cx] = ((a.bc_flip[2] >> v) & 1) ? -s : s;
            }
            if (cl >= 1 && cl <= TY) {
              const T s = SLy[v * NYS3 + cl * TX + cx];
              SRy[v * NYS3 + (cl + 1) * TX + cx] = ((a.bc_flip[3] >> v) & 1) ? -s : s;
            }
          }
        }
        __syncthreads();
      }

      // ---- x and y fluxes of plane k, one phase (x faces padded to whole
      // warps, so that no warp mixes directions); each flux replaces the
      // lower-cell face state that only its own face reads ----
      if constexpr (!kOneSolver)
      for (int q = tid; q < NXFP3 + NYF3; q += NT) {
        if (q < NXFP3) {
          if (q >= NXF3) continue;  // padding lanes
          const int fx = q % XF, cy = q / XF;
          T L[NV], R[NV], Fo[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            L[v] = SLx[v * NXS3 + cy * XS + fx];
            R[v] = SRx[v * NXS3 + cy * XS + fx + 1];
          }
          riemann_flux<T, 1, FLUX, OMHD_FAST>(L, R, ch, gam, r1, r2, Fo);
          if (resist) {  // flux_resistive.cuf:87-101
            const int g = gi0 - 1 + fx, gjj = gj0 + cy;
            if (g >= 0 && g <= ix - 2 && gjj <= jx - 2) {
              const int o = (cy + 2) * RX + (fx + 1);
              if constexpr (sizeof(T) == 4) {
                auto b = [&](int var, int dxo, int dyo, int dzo) { return Wv(k + dzo, var, o + dxo + dyo * RX); };
                const float eta_dx = sep_eta ? harris_eta_dx<T>(ex_f[fx], ez_c[k - k0 + 1], inv_dx_t)
                                             : narrow_f64(eta3(a.eta_kind, a.xc[g] + 0.5 * a.dx, a.yc[gjj], a.zc[k]) / a.dx);
                resist_face_f32<1>(b, eta_dx, Fo);
              } else {
                auto B = [&](int var, int dxo, int dyo, int dzo) { return to_f64<T>(Wv(k + dzo, var, o + dxo + dyo * RX)); };
                const double eta_dx = sep_eta ? harris_eta_dx<double>(ex_f[fx], ez_c[k - k0 + 1], inv_dx)
                                              : eta3(a.eta_kind, a.xc[g] + 0.5 * a.dx, a.yc[gjj], a.zc[k]) / a.dx;
                resist_face_f64<0>(B, eta_dx, Fo);
              }
            }
          }
#pragma unroll
          for (int v = 0; v < NV; ++v) SLx[v * NXS3 + cy * XS + fx] = Fo[v];
        } else {
          const int qq = q - NXFP3;
          const int cx = qq % TX, fy = qq / TX;
          T L[NV], R[NV], Fo[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            L[v] = SLy[v * NYS3 + fy * TX + cx];
            R[v] = SRy[v * NYS3 + (fy + 1) * TX + cx];
          }
          riemann_flux<T, 2, FLUX, OMHD_FAST>(L, R, ch, gam, r1, r2, Fo);
          if (resist) {  // flux_resistive.cuf:104-118
            const int gii = gi0 + cx, g = gj0 - 1 + fy;
            if (g >= 0 && g <= jx - 2 && gii <= ix - 2) {
              const int o = (fy + 1) * RX + (cx + 2);
              if constexpr (sizeof(T) == 4) {
                auto b = [&](int var, int dxo, int dyo, int dzo) { return Wv(k + dzo, var, o + dxo + dyo * RX); };
                const float eta_dx = sep_eta ? harris_eta_dx<T>(ex_c[cx + 1], ez_c[k - k0 + 1], inv_dx_t)
                                             : narrow_f64(eta3(a.eta_kind, a.xc[gii], a.yc[g] + 0.5 * a.dx, a.zc[k]) / a.dx);
                resist_face_f32<2>(b, eta_dx, Fo);
              } else {
                auto B = [&](int var, int dxo, int dyo, int dzo) { return to_f64<T>(Wv(k + dzo, var, o + dxo + dyo * RX)); };
                const double eta_dx = sep_eta ? harris_eta_dx<double>(ex_c[cx + 1], ez_c[k - k0 + 1], inv_dx)
                                              : eta3(a.eta_kind, a.xc[gii], a.yc[g] + 0.5 * a.dx, a.zc[k]) / a.dx;
                resist_face_f64<1>(B, eta_dx, Fo);
              }
            }
          }
#pragma unroll
          for (int v = 0; v < NV; ++v) SLy[v * NYS3 + fy * TX + cx] = Fo[v];
        }
      }
    }
    // ---- z face k+1/2 in registers: it reads only the ring, so the FP64 build
    // solves it before the flux barrier (threads with no face left in the last
    // round of x/y faces solve their z face meanwhile: 1 % faster on Harris
    // 512x256x512); the FP32 build, after the barrier (3 % faster there) ----
    double Fzc[NV];
    T sLn[NV];
    auto z_face = [&]() {
      T L[NV], R[NV], Fo[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        T l, r;
        reconstruct_t<T, OMHD_FAST>(lm, Wv(k, v, oc), Wv(k + 1, v, oc), Wv(k + 2, v, oc), l, r);
        L[v] = sLc[v];
        R[v] = r;
        sLn[v] = l;
      }
      if constexpr (sizeof(T) == 8) {
        if (!perz && k == 0) {  // bottom wall: VL = flip(VR)
#pragma unroll
          for (int v = 0; v < NV; ++v) L[v] = ((a.bc_flip[4] >> v) & 1) ? -R[v] : R[v];
        }
      }
      if (!perz && k == kx - 2) {  // top wall: VR = flip(VL)
#pragma unroll
        for (int v = 0; v < NV; ++v) R[v] = ((a.bc_flip[5] >> v) & 1) ? -L[v] : L[v];
      }
      riemann_flux<T, 3, FLUX, OMHD_FAST>(L, R, ch, gam, r1, r2, Fo);
#pragma unroll
      for (int v = 0; v < NV; ++v) Fzc[v] = to_f64<T>(Fo[v]);
      if (resist && own) {  // flux_resistive.cuf:121-135
        if constexpr (sizeof(T) == 4) {
          auto b = [&](int var, int dxo, int dyo, int dzo) { return Wv(k + dzo, var, oc + dxo + dyo * RX); };
          const float eta_dx = sep_eta ? harris_eta_dx<T>(ex_c[tx + 1], ez_f[k - k0 + 1], inv_dx_t)
                                       : narrow_f64(eta3(a.eta_kind, a.xc[gi], a.yc[gj], a.zc[k] + 0.5 * a.dx) / a.dx);
          resist_face_f32<3>(b, eta_dx, Fo);
#pragma unroll
          for (int v = 0; v < NV; ++v) Fzc[v] = to_f64<T>(Fo[v]);
        } else {
          auto B = [&](int var, int dxo, int dyo, int dzo) { return to_f64<T>(Wv(k + dzo, var, oc + dxo + dyo * RX)); };
          const double eta_dx = sep_eta ? harris_eta_dx<double>(ex_c[tx + 1], ez_f[k - k0 + 1], inv_dx)
                                        : eta3(a.eta_kind, a.xc[gi], a.yc[gj], a.zc[k] + 0.5 * a.dx) / a.dx;
          resist_face_f64<2>(B, eta_dx, Fzc);
        }
      }
    };
    if constexpr (kOneSolver) {
      // x and y faces of the plane, then this thread's z face k+1/2 (in registers;
      // it reads only the ring), through one x-oriented solver in one rolled loop:
      // with a copy per direction a fifth of the warps' time went into instruction
      // fetches.  Fluxes replace the lower-cell face states that only they read.
      constexpr int RXY = (NXF3 + NYF3 + NT - 1) / NT;
#pragma unroll 1
      for (int r = lead ? RXY : 0; r <= RXY; ++r) {
        const bool zf = r == RXY;
        const int q = tid + r * NT, n = zf ? 2 : (q < NXF3 ? 0 : 1);
        if (zf ? tid >= G::CELLS : q >= NXF3 + NYF3) continue;
        const int qq = n == 0 ? q : q - NXF3;
        const int fa = n == 0 ? qq % XF : qq % TX, fb = n == 0 ? qq / XF : qq / TX;
        double* const bl = n == 0 ? SLx + fb * XS + fa : SLy + fb * TX + fa;
        const double* const br = n == 0 ? SRx + fb * XS + fa + 1 : SRy + (fb + 1) * TX + fa;
        const int sv = n == 0 ? NXS3 : NYS3;
        double L[NV], R[NV], Fo[NV], F[NV];
        if (zf) {
          double Rg[NV];
#pragma unroll
          for (int v = 0; v < NV; ++v)
            reconstruct_t<T, OMHD_FAST>(lm, Wv(k, v, oc), Wv(k + 1, v, oc), Wv(k + 2, v, oc), sLn[v], Rg[v]);
          if (!perz && k == 0) {  // bottom wall: VL = flip(VR)
#pragma unroll
            for (int v = 0; v < NV; ++v) sLc[v] = ((a.bc_flip[4] >> v) & 1) ? -Rg[v] : Rg[v];
          }
          if (!perz && k == kx - 2) {  // top wall: VR = flip(VL)
#pragma unroll
            for (int v = 0; v < NV; ++v) Rg[v] = ((a.bc_flip[5] >> v) & 1) ? -sLc[v] : sLc[v];
          }
#pragma unroll
          for (int c = 0; c < NV; ++c) {
            L[c] = sLc[rot3(2, c)];
            R[c] = Rg[rot3(2, c)];
          }
        } else {
#pragma unroll
          for (int c = 0; c < NV; ++c) {
            const int pv = (n == 0 ? c : rot3(1, c)) * sv;
            L[c] = bl[pv];
            R[c] = br[pv];
          }
        }
        riemann_flux<double, 1, FLUX, true>(L, R, ch, gam, r1, r2, Fo);
#pragma unroll
        for (int v = 0; v < NV; ++v) {  // back to grid components: v = rot3(1, rot3(2, v)) = rot3(2, rot3(1, v))
          F[v] = n == 0 ? Fo[v] : (n == 1 ? Fo[rot3(2, v)] : Fo[rot3(1, v)]);
        }
        if (resist) {
          const int gx = zf ? gi : (n == 0 ? gi0 - 1 + fa : gi0 + fa), gy = zf ? gj : (n == 0 ? gj0 + fb : gj0 - 1 + fb);
          if (gx >= 0 && gy >= 0 && gx <= ix - 2 && gy <= jx - 2) {
            const int o = zf ? oc : (n == 0 ? (fb + 2) * RX + (fa + 1) : (fb + 1) * RX + (fa + 2));
            const int ex_i = zf ? tx + 1 : (n == 0 ? fa : fa + 1);
            auto B = [&](int var, int dxo, int dyo, int dzo) { return Wv(k + dzo, var, o + dxo + dyo * RX); };
            const double eta_dx =
                sep_eta ? harris_eta_dx<double>((n == 0 ? ex_f : ex_c)[ex_i], (zf ? ez_f : ez_c)[k - k0 + 1], inv_dx)
                        : eta3(a.eta_kind, a.xc[gx] + (n == 0 ? 0.5 * a.dx : 0.0), a.yc[gy] + (n == 1 ? 0.5 * a.dx : 0.0),
                               a.zc[k] + (zf ? 0.5 * a.dx : 0.0)) / a.dx;
            if (zf)
              resist_face_f64<2>(B, eta_dx, F);
            else if (n == 0)
              resist_face_f64<0>(B, eta_dx, F);
            else
              resist_face_f64<1>(B, eta_dx, F);
          }
        }
        if (zf) {
#pragma unroll
          for (int v = 0; v < NV; ++v) Fzc[v] = F[v];
        } else {
#pragma unroll
          for (int v = 0; v < NV; ++v) bl[v * sv] = F[v];
        }
      }
    } else if constexpr (sizeof(T) == 8) {
      z_face();
    }

    double acc[NV] = {}, gm[NV] = {}, gp[NV] = {};
    if (!lead) {
      __syncthreads();
#pragma unroll
      for (int v = 0; v < NV; ++v) {  // mixed: off the FP64 pipe, and stage 2's halving (14.8 to 14.1 ms for 2 steps of 256x128x256)
        acc[v] = sub_f64<T>(SLx[v * NXS3 + ty * XS + tx], SLx[v * NXS3 + ty * XS + tx + 1]);
        gm[v] = to_f64<T>(SLy[v * NYS3 + ty * TX + tx]);
        gp[v] = to_f64<T>(SLy[v * NYS3 + (ty + 1) * TX + tx]);
      }
    }
    if constexpr (sizeof(T) == 4) z_face();

    // ---- update plane k ----
    if (own && !lead) {
      const size_t c = (size_t)gi + (size_t)ix * ((size_t)gj + (size_t)jx * k);
      double out[NV];
      // the alternatives outside the loops over the variables: predicated-off FP64
      // instructions hold the FP64 pipe (164 of its instructions a cell and stage
      // in the mixed kernel for 89 operations, with the choices inside)
      const bool rk2 = a.stage == 1 || a.time_type == OMHD_TIME_RK2;
      auto ub = [&](int v) { return v == PS ? glmf * a.Ubase[v * N + c] : a.Ubase[v * N + c]; };
      if constexpr (OMHD_FAST && sizeof(T) == 8) {  // U + dt/dx (dF + dx/dy dG + dx/dz dH)
        auto d = [&](int v) { return fma(a.rzx, Fzp[v] - Fzc[v], fma(a.ryx, gm[v] - gp[v], acc[v])); };
        if (rk2) {
#pragma unroll
          for (int v = 0; v < NV; ++v) out[v] = fma(dtx, d(v), ub(v));
        } else {
#pragma unroll
          for (int v = 0; v < NV; ++v) out[v] = half_rn(fma(dtx, d(v), ub(v) + a.U1[v * N + c]));
        }
      } else {
        double d[NV];
        if (a.iso) {
#pragma unroll
          for (int v = 0; v < NV; ++v) d[v] = dtx * (acc[v] + gm[v] - gp[v] + Fzp[v] - Fzc[v]);  // 3D_basic/rk.f90:26-35 order
        } else {
#pragma unroll
          for (int v = 0; v < NV; ++v) d[v] = dtx * acc[v] + dty * (gm[v] - gp[v]) + dtz * (Fzp[v] - Fzc[v]);
        }
        if (rk2) {
#pragma unroll
          for (int v = 0; v < NV; ++v) out[v] = ub(v) + d[v];
        } else {
#pragma unroll
          for (int v = 0; v < NV; ++v) out[v] = half_<OMHD_FAST>(ub(v) + a.U1[v * N + c] + d[v]);
        }
      }
      if (a.stage == 2) out[PS] = glmf * out[PS];
      int xt[3], yt[3], zt[3], xf[3], yf[3], zf[3], nxt = 1, nyt = 1, nzt = 1;
      xt[0] = gi; xf[0] = 0; yt[0] = gj; yf[0] = 0; zt[0] = k; zf[0] = 0;
      if (gi == 1) { xt[nxt] = perx ? ix - 1 : 0; xf[nxt] = perx ? 0 : a.bc_flip[0]; ++nxt; }
      if (gi == ix - 2) { xt[nxt] = perx ? 0 : ix - 1; xf[nxt] = perx ? 0 : a.bc_flip[1]; ++nxt; }
      if (gj == 1) { yt[nyt] = pery ? jx - 1 : 0; yf[nyt] = pery ? 0 : a.bc_flip[2]; ++nyt; }
      if (gj == jx - 2) { yt[nyt] = pery ? 0 : jx - 1; yf[nyt] = pery ? 0 : a.bc_flip[3]; ++nyt; }
      if (k == 1) { zt[nzt] = perz ? kx - 1 : 0; zf[nzt] = perz ? 0 : a.bc_flip[4]; ++nzt; }
      if (k == kx - 2) { zt[nzt] = perz ? 0 : kx - 1; zf[nzt] = perz ? 0 : a.bc_flip[5]; ++nzt; }
      for (int e = 0; e < nzt; ++e)
        for (int b = 0; b < nyt; ++b)
          for (int q = 0; q < nxt; ++q) {
            const size_t cc = (size_t)xt[q] + (size_t)ix * ((size_t)yt[b] + (size_t)jx * zt[e]);
            const int fm = xf[q] ^ yf[b] ^ zf[e];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              const double o = ((fm >> v) & 1) ? -out[v] : out[v];
              a.Uout[v * N + cc] = o;
              if (a.Uhost) a.Uhost[v * N + cc] = o;  // result straight to host memory
            }
          }
      // 3D_basic/set_dt.f90:27-43 on the new state
      if (a.stage == 2 && !(OMHD_FAST && known > 0.0f && cfl_upper<3>(out, a.gamma_f, a.gm1_f) < known)) {
        const double ro = out[RO];
        const double iro = rcp_<double, OMHD_FAST, sizeof(T) == 4>(ro);  // one reciprocal for the three velocities
        const double vx = divr_<double, OMHD_FAST>(out[MX], ro, iro), vy = divr_<double, OMHD_FAST>(out[MY], ro, iro), vz = divr_<double, OMHD_FAST>(out[MZ], ro, iro);
        const double rv2 = vx * out[MX] + vy * out[MY] + vz * out[MZ];
        const double B2 = out[BX] * out[BX] + out[BY] * out[BY] + out[BZ] * out[BZ];
        const double pr = f1g * (out[EN] - 0.5 * (rv2 + B2));
        const double f1 = gamma * pr;
        // fmax2 of the three speeds and of the running max, the comparisons on
        // the integer pipe in the FAST builds (same results)
        const double sx = fabs(vx) + fast_speed<double, OMHD_FAST, sizeof(T) == 4>(f1, B2, out[BX], ro);
        const double sy = fabs(vy) + fast_speed<double, OMHD_FAST, sizeof(T) == 4>(f1, B2, out[BY], ro);
        const double sz = fabs(vz) + fast_speed<double, OMHD_FAST, sizeof(T) == 4>(f1, B2, out[BZ], ro);
        double s = lt_<double, OMHD_FAST>(sx, sy) ? sy : sx;
        s = lt_<double, OMHD_FAST>(s, sz) ? sz : s;
        vloc = lt_<double, OMHD_FAST>(s, vloc) ? vloc : s;
        if (OMHD_FAST) cfl_publish(st, s, known);
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      Fzp[v] = Fzc[v];
      sLc[v] = sLn[v];
    }
  }
  if (a.stage == 2) {
    const double bm = block_max_pos(vloc, red32);
    StepConsts sc{a.cfl, a.dmin, a.dx, a.eta_kind};
    reduce_and_finalize(st, sc, a.err, bm, gridDim.x * gridDim.y * gridDim.z, 1);
  }
}

template <class G>
inline long long columns_of(const StageArgs& a) {
  return (long long)((a.ix - 2 + G::TX - 1) / G::TX) * ((a.jx - 2 + G::TY - 1) / G::TY);
}

template <class G>
Tiling tiling_of(const StageArgs& a, int nsm) {
  return {G::TX, G::TY, pick_zchunk(columns_of<G>(a), a.kx - 2, nsm * G::CTAS), G::CTAS};
}

template <class T, int FLUX, class G = DefaultCol<T>>
int launch_one3d(const StageArgs& a, cudaStream_t s) {
  const size_t bytes = G::template smem_bytes<T>();
  static std::atomic<unsigned long long> configured{0};
  int r = set_smem_attr_once(k_stage3d<T, FLUX, G>, bytes, configured);
  int nsm = 0;
  if (!r) r = sm_count(&nsm);
  if (r) return r;
  const int zc = tiling_of<G>(a, nsm).tz;
  dim3 grid((a.ix - 2 + G::TX - 1) / G::TX, (a.jx - 2 + G::TY - 1) / G::TY, (a.kx - 2 + zc - 1) / zc);
  k_stage3d<T, FLUX, G><<<grid, G::NT, bytes, s>>>(a, zc);
  return (int)cudaGetLastError();
}

// FP64 HLLD: 16x16 columns, one CTA per SM, or two CTAs of 16x8 columns, the
// cheaper by the rounds x (planes + prologue) of pick_zchunk.  For grids that both
// cover alike an SM takes longer for a plane of two 16x8 columns, whose halo is
// larger and with resistivity has corners: 10-12 % on Harris (96x48x96 1.91 against
// 1.74 ms per step, 256x128x256 32.0 / 28.6), 2 % on the field loop (64x64x128 1.338 /
// 1.315).  They cover ragged grids better (loop 100x100x200: 5.25 / 5.70).
inline bool small_columns(const StageArgs& a, int nsm) {
  double wide = 0.0, small = 0.0;
  pick_zchunk(columns_of<WideCol>(a), a.kx - 2, nsm * WideCol::CTAS, &wide);
  pick_zchunk(columns_of<SmallCol>(a), a.kx - 2, nsm * SmallCol::CTAS, &small);
  return (a.eta_kind != OMHD_ETA_NONE ? 1.11 : 1.02) * small < wide;
}

// FP32-mixed HLLD.  Resistive runs: 16x16 columns, whose smaller halo saves corner loads,
// unless 32x8 columns cover the grid in fewer rounds x (planes + prologue), as they do
// where ny is no multiple of 16: half of a 16x16 column's faces may then be outside the
// grid and are solved all the same.  Harris-type grids, us per step with 32x8 / 16x16:
// 1024x8x1024 6585 / 11306, 512x24x512 5018 / 6399, 512x40x512 8373 / 9540, 300x72x300
// 5476 / 5725; at equal cost 128x64x128 934 / 870, 256x128x256 6605 / 6475, 512x256x512
// 51304 / 50946, 96x48x96 393 / 394 (48x24x200 272 / 300, the worst of 25 grids).  Other
// runs: 16x16 only where fewer of them cover the grid (field loop 100x100x200 2130 /
// 1949, 64x64x128 449 / 473).
inline bool square_columns(const StageArgs& a, int nsm) {
  using Flat = DefaultCol<float>;
  if (a.eta_kind == OMHD_ETA_NONE) return columns_of<SquareCol>(a) < columns_of<Flat>(a);
  double square = 0.0, flat = 0.0;
  pick_zchunk(columns_of<SquareCol>(a), a.kx - 2, nsm * SquareCol::CTAS, &square);
  pick_zchunk(columns_of<Flat>(a), a.kx - 2, nsm * Flat::CTAS, &flat);
  return square <= flat;
}

// calls f with the column of an HLLD launch of face arithmetic T
template <class T, class F>
auto with_hlld_column(const StageArgs& a, int nsm, F&& f) {
  if constexpr (OMHD_FAST && sizeof(T) == 8) {
    return small_columns(a, nsm) ? f(SmallCol{}) : f(WideCol{});
  } else if constexpr (sizeof(T) == 4) {
    return square_columns(a, nsm) ? f(SquareCol{}) : f(DefaultCol<float>{});
  } else {
    return f(DefaultCol<T>{});
  }
}

template <class T>
Tiling tiling3d(const StageArgs& a, int nsm) {
  if (a.flux_type != FX_HLLD) return tiling_of<DefaultCol<T>>(a, nsm);
  return with_hlld_column<T>(a, nsm, [&](auto col) { return tiling_of<decltype(col)>(a, nsm); });
}

template <class T>
int launch_variant3d(const StageArgs& a, cudaStream_t s) {
  switch (a.flux_type) {
    case FX_LLF: return launch_one3d<T, FX_LLF>(a, s);
    case FX_HLL: return launch_one3d<T, FX_HLL>(a, s);
    case FX_HLLC: return launch_one3d<T, FX_HLLC>(a, s);
    case FX_HLLD: {
      int nsm = 0;
      const int r = sm_count(&nsm);
      if (r) return r;
      return with_hlld_column<T>(a, nsm, [&](auto col) { return launch_one3d<T, FX_HLLD, decltype(col)>(a, s); });
    }
    default: return launch_one3d<T, FX_LHLLD>(a, s);
  }
}

}  // namespace d3
}  // namespace OMHD_VARIANT
}  // namespace omhd
