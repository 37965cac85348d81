// ugks_fused.cu -- the whole UGKS time step in a few launches (FP64 four for one
// limiter and velocity grid; mixed seven, ugks_delta.cuh), for every block of every
// solve of a device-resident block table.
//
// Per FP64 step (UGKSim.one_step, ugks_sim.py:407-501):
//   face pass   a face per warp, in either direction: reconstruction (iFace),
//               face moments (getFaceCons/getAL/getAR), slopes (getPLR),
//               initMacroFlux, calcFaceQ, macroFlux and distFlux fused; wall
//               faces a CTA each: accommodatingWallDist | adsorbingWall_P1 + P2,
//               then wallFlux and wallMassEnergyFluxes.
//   wall faces  again, only for solves whose dt changed (updateTimeStep inside
//               the dt loop, ugks_sim.py:430-441); an interior face takes the dt of
//               the last pass at once.
//   cell pass   a cell per warp: calcQ, updateMacro and UGKS_update fused, plus
//               the cell's CFL frequency (clFindDT).
//   ghost pass  one CTA per ghost cell of every block face (updateBC), and the
//               end of the step: calcTimeStep, updateTimeStep, time advance.
// Nothing reads the host in between, so a step can be captured in a graph.
#include <cuda_runtime.h>
#include <float.h>

#include <algorithm>
#include <mutex>
#include <optional>
#include <type_traits>
#include <vector>

#include <nvtx3/nvToolsExt.h>

#include "ugks_device.cuh"

using namespace ugks;

namespace {

constexpr int FT = 128;  // threads per face / cell / ghost CTA
// velocities (or pairs) per thread whose loads are in flight together in
// the ghost copies, issued before the first store (a store may alias a later
// load, so the compiler keeps them in program order)
constexpr int GHOST_U = 4;
// Launch shapes a face-pass segment can run with (ugks_fused_sizes.seg_variant;
// the tuner in pyugks_b200/tuner.py picks them by timing): variant 0 is the
// default 1, 1..4 are (warps per CTA, CTAs per SM of the register budget).
// FP64 face pass (a face per warp; measured at face_item_fp64):
template <int V> struct FaceShape;
template <> struct FaceShape<1> { static constexpr int wpc = 4, minb = 4; };
template <> struct FaceShape<2> { static constexpr int wpc = 4, minb = 5; };
template <> struct FaceShape<3> { static constexpr int wpc = 8, minb = 2; };
template <> struct FaceShape<4> { static constexpr int wpc = 4, minb = 3; };
// launch shapes of the mixed moments sweep (a face per warp): warps per CTA x
// CTAs per SM
template <int V> struct MomentsShape;
template <> struct MomentsShape<1> { static constexpr int wpc = 4, minb = 4; };
template <> struct MomentsShape<2> { static constexpr int wpc = 4, minb = 5; };
template <> struct MomentsShape<3> { static constexpr int wpc = 8, minb = 3; };
template <> struct MomentsShape<4> { static constexpr int wpc = 4, minb = 6; };
// and of the mixed flux sweep
constexpr int FLUX_WPC = 4;
#ifndef UGKS_FLUX_TMA_MINB
#define UGKS_FLUX_TMA_MINB 5
#endif
constexpr int FLUX_TMA_MINB = UGKS_FLUX_TMA_MINB;
// cell pass: CELL_MINB x 8 cell warps per SM by default, 16 at 128 registers (24
// at 80 spill: FP64 1.06 -> 1.22 ms a step on the 2x2-block cavity, mixed 0.720
// -> 0.730), and the depth of the per-warp ring of asynchronous copies that
// stream the f and flux rows of the FP64 update into shared memory (with the
// 16-byte pairs of the mixed storage the ring was 18% slower than plain loads)
constexpr int CELL_MINB = 2, CELL_RING_F64 = 3;
// shared memory of the cell-update ring: per warp, ring stages x 5 rows
// (f, S face j, S face j+1, W face i, W face i+1) x 32 lanes
constexpr size_t cell_ring_bytes() { return (size_t)CELL_RING_F64 * 5 * 32 * sizeof(double2); }

// cp.async (sm_80+ asynchronous global -> shared copy of 8 or 16 bytes per
// thread; a thread waits only for its own groups)
template <int BYTES, bool CA = false>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if constexpr (BYTES == 16 && !CA)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" ::"r"(d), "l"(src), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

inline cudaStream_t S(void *s) { return reinterpret_cast<cudaStream_t>(s); }
// Where a step's kernels are launched: a stream, and for steps of few faces
// (`carve` > 0) programmatic launches, that share one split of L1 and shared
// memory, `carve` percent.  An SM changes that split only when it is idle, so a
// kernel that starts beside its predecessor runs with the predecessor's, and with
// one that suits neither the reconfiguration costs more than the early launch
// gives.  On large grids each pass is better off with the split that fits it.
// There only the launches of a face pass after its first are programmatic
// (`chained`): they fill the SMs that the last CTAs of the one before leave idle
// (16 cavities of eight velocity grids and limiters, step in us without and with:
// FP64 7029 and 6430, mixed 3934 and 3900).
struct StepStream {
  cudaStream_t st;
  int carve = 0;
  bool chained = false;
};
template <typename... P, typename... A>
void launch(void (*kernel)(P...), unsigned grid, unsigned block, size_t smem, StepStream to, A... args) {
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributePreferredSharedMemoryCarveout;
  attr[1].val.sharedMemCarveout = (unsigned)to.carve;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = to.st;
  cfg.attrs = attr;
  cfg.numAttrs = to.carve > 0 ? 2 : to.chained ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}
inline int launch_status() {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? 0 : -(int)e;
}

// block of work item w: the last block whose begin <= w (begins are ascending)
template <int WHICH>
__device__ __forceinline__ int find_block(const ugks_fused_block *B, int nb, int w) {
  int lo = 0, hi = nb - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    int beg = WHICH == 0 ? B[mid].face_begin
                         : (WHICH == 1 ? B[mid].cell_begin : (WHICH == 2 ? B[mid].ghost_begin : B[mid].wall_begin));
    if (beg <= w) lo = mid; else hi = mid - 1;
  }
  return lo;
}

__device__ __forceinline__ bool is_wall(int bc) { return bc == BC_DIFFUSE || bc == BC_ADSORBING; }

// UGKS_CHECKED builds (python -m pyugks_b200.build --checked): every work
// item is checked against the block it was found in -- inside the block's
// range of items, and the block's sizes consistent with its ghost layers and
// its limiter's stencil -- and an item that fails (a table corrupted on the
// device after ugks_fused_layout validated it) flags its solve with status 9
// and is skipped instead of indexing outside the block's arrays.
#ifndef UGKS_CHECKED
#define UGKS_CHECKED 0
#endif
constexpr int STATUS_INDEX_CHECK = 9;
template <int WHICH>
__device__ __forceinline__ bool item_in_block(const ugks_fused_block &b, int w) {
  const ugks_block_desc &d = b.d;
  long begin = 0, count = 0;
  if (WHICH == 0) { begin = b.face_begin; count = 2l * (d.ni + 1) * (d.nj + 1); }
  if (WHICH == 1) { begin = b.cell_begin; count = (long)d.ni * d.nj; }
  if (WHICH == 2) { begin = b.ghost_begin; count = 2l * d.ghost * (d.ni + d.nj); }
  if (WHICH == 3) { begin = b.wall_begin; count = 2l * (d.ni + d.nj); }
  return w >= begin && w < begin + count && d.ghost >= (d.flux_method == 1 ? 3 : 2) &&
         d.Ni == d.ni + 2 * d.ghost && d.Nj == d.nj + 2 * d.ghost;
}
#define UGKS_CHECK_ITEM(WHICH, blk, w, solves, ...)                                                       \
  do {                                                                                                     \
    if (UGKS_CHECKED && !item_in_block<WHICH>((blk), (w))) {                                               \
      atomicExch(const_cast<int *>(&(solves)[(blk).solve].status), STATUS_INDEX_CHECK);                     \
      return __VA_ARGS__;                                                                                  \
    }                                                                                                      \
  } while (0)

// The launches of a face pass depend on the step before, not on one another: those
// after the first (`chained`) start at once, since the first has waited before it
// let them start, and have one CTA more, which waits, so that their completion
// stands for the first's.  (A wait at the end of the last working CTA cost the
// mixed moments sweep 3%: no warp left before its CTA's last.)
__device__ __forceinline__ void pdl_begin_face(int chained) {
  if (!chained) pdl_wait();
  pdl_trigger();
  if (!chained) return;
  if (blockIdx.x == gridDim.x - 1) pdl_wait();
  else __threadfence();  // acquire: nothing this SM cached before the first launch's wait
}

// dt update of updateTimeStep (ugks_sim.py:285-311) with limit = True
__device__ __forceinline__ double limited_dt(double dt_old, double dt_new, double delta) {
  if (dt_old != dt_new) {
    if (dt_new > (1.0 + delta) * dt_old) dt_new = (1.0 + delta) * dt_old;
    return dt_new;
  }
  return dt_old;
}

// The time steps of one fused step (the dt loop of one_step, ugks_sim.py:430-446):
// the first flux pass runs at `first`; when the limiter changes dt the pass is
// redone at `flux` and dt is limited once more for the cell update.  A pure
// function of the solve record, which only finish_step writes, so that every
// kernel of the step evaluates it for itself.
struct StepDt {
  double first, flux, cell;
  bool retry;
};
__device__ __forceinline__ StepDt step_dt(const ugks_solve_state &x) {
  StepDt t;
  t.first = x.dt;
  t.flux = limited_dt(x.dt, x.max_dt, x.delta_dt);
  t.retry = t.flux != x.dt;
  t.cell = t.retry ? limited_dt(t.flux, x.max_dt, x.delta_dt) : t.flux;
  return t;
}

// ---------------------------------------------------------------------------
// face pass
// ---------------------------------------------------------------------------
// The per-face and per-cell coefficient helpers below restate getPrimary,
// microSlope, momentU, relaxTime and the time weights (clUGKS.c:16-80,
// 497-503, clFunctions.c:8-32) with every division by rho, lambda, tau or a
// constant replaced by one Newton-Raphson reciprocal (nr_rcp) and products:
// branch-free, so the independent chains of a face overlap.  Results differ
// from the dividing forms by a few ulp.
struct Rcp {
  double rho, lam;  // 1/rho, 1/lambda
};

__device__ __forceinline__ P4 to_primary_rcp(const ugks_block_desc &d, P4 w, Rcp &r) {
  const double r0 = nr_rcp(w.s0);
  P4 p = w;
  p.s1 = w.s1 * r0;
  p.s2 = w.s2 * r0;
  const double e = w.s3 - 0.5 * (w.s1 * w.s1 + w.s2 * w.s2) * r0;
  p.s3 = (0.5 * w.s0) * nr_rcp((d.gam - 1.0) * e);
  r.rho = r0;
  r.lam = nr_rcp(p.s3);
  return p;
}

__device__ __forceinline__ P4 micro_slope_rcp(double K, P4 prim, Rcp r, P4 sw) {
  const double k2 = 0.5 * (K + 2.0) * r.lam;  // (K + 2) / (2 lambda)
  const double c3 = 4.0 * (prim.s3 * prim.s3) * nr_rcp(K + 2.0) * r.rho;
  const double cl = 2.0 * prim.s3 * r.rho;
  const double uv2 = prim.s1 * prim.s1 + prim.s2 * prim.s2;
  P4 a;
  a.s3 = c3 * (2.0 * sw.s3 - 2.0 * prim.s1 * sw.s1 - 2.0 * prim.s2 * sw.s2 + sw.s0 * (uv2 - k2));
  a.s2 = cl * (sw.s2 - prim.s2 * sw.s0) - prim.s2 * a.s3;
  a.s1 = cl * (sw.s1 - prim.s1 * sw.s0) - prim.s1 * a.s3;
  a.s0 = sw.s0 * r.rho - prim.s1 * a.s1 - prim.s2 * a.s2 - 0.5 * (uv2 + k2) * a.s3;
  return a;
}

// momentU (clUGKS.c:47-80) over one half range: sg = +1 gives the moments
// <u^k> over u > 0 (MuL), sg = -1 those over u < 0 (MuR); Mv and Mxi are the
// full-range moments of v and xi.  The two halves are the same instruction
// stream with the sign flipped, so two lanes compute them side by side.
__device__ __forceinline__ void half_moments_rcp(double PI, double K, P4 prim, Rcp r, double sg,
                                                 double Mh[MNUM], double Mv[MTUM], double Mxi[3]) {
  const double sl = sqrt(prim.s3);
  const double g = 0.5 * exp(-prim.s3 * (prim.s1 * prim.s1)) * nr_rcp(sqrt(PI * prim.s3));
  const double hl = 0.5 * r.lam;
  Mh[0] = 0.5 * erfc((-sg * sl) * prim.s1);
  Mh[1] = prim.s1 * Mh[0] + sg * g;
#pragma unroll
  for (int i = 2; i < MNUM; ++i) Mh[i] = prim.s1 * Mh[i - 1] + ((i - 1) * hl) * Mh[i - 2];
  Mv[0] = 1.0;
  Mv[1] = prim.s2;
#pragma unroll
  for (int i = 2; i < MTUM; ++i) Mv[i] = prim.s2 * Mv[i - 1] + ((i - 1) * hl) * Mv[i - 2];
  Mxi[0] = 1.0;
  Mxi[1] = K * hl;
  Mxi[2] = (K * K + 2.0 * K) * (hl * hl);
}

// raw moments of a distribution up to third order: sums over the velocities
// of h u^a v^b (RMab) and of b u^a v^b (RBab)
enum { RM00, RM10, RM01, RM20, RM11, RM02, RM30, RM21, RM12, RM03, RB00, RB10, RB01, RNMOM };

// Heat flux (calcQ, clKernel.c:480-543) relative to velocity U of a
// distribution given by its raw moments M (the RM* / RB* sums over v of h u^a
// v^b and of b u^a v^b), in the frame of the moments:
//   q = 1/2 sum (c |c|^2 h + c b / K),  c = (u, v) - U.
__device__ __forceinline__ V2 heat_flux_from_moments(const double *M, double K, V2 U) {
  const double Ux = U.x, Uy = U.y;
  const double cx3 = M[RM30] - 3.0 * Ux * M[RM20] + 3.0 * Ux * Ux * M[RM10] - Ux * Ux * Ux * M[RM00] + M[RM12] -
                     2.0 * Uy * M[RM11] + Uy * Uy * M[RM10] - Ux * M[RM02] + 2.0 * Ux * Uy * M[RM01] -
                     Ux * Uy * Uy * M[RM00];
  const double cy3 = M[RM03] - 3.0 * Uy * M[RM02] + 3.0 * Uy * Uy * M[RM01] - Uy * Uy * Uy * M[RM00] + M[RM21] -
                     2.0 * Ux * M[RM11] + Ux * Ux * M[RM01] - Uy * M[RM20] + 2.0 * Ux * Uy * M[RM10] -
                     Uy * Ux * Ux * M[RM00];
  return v2(0.5 * (cx3 + (M[RB10] - Ux * M[RB00]) / K), 0.5 * (cy3 + (M[RB01] - Uy * M[RB00]) / K));
}

// 1 / relaxTime
__device__ __forceinline__ double inv_relax_time_rcp(const ugks_block_desc &d, P4 prim, Rcp r) {
  // exp((1 - omega) ln lambda) has half of pow's dependent chain and its error grows
  // with the exponent: 2.7 ulp against 1.3 for lambda in 1e-3..1e3, omega 0.66, 0.58
  // against 0.56 for 0.8..1.3, omega 0.81
  const double p = pow(prim.s3, 1.0 - d.omega);
  double c = 1.0;
  switch (d.relax_type) {
    case 0: c = 0.79788456080286541; break;
    case 1: c = (5. / 8.) * sqrt(d.PI); break;
    case 3: c = 2.2567583341910251; break;
    default: break;
  }
  return nr_rcp((d.Kn_eff * r.rho) * c * p);
}

__device__ __forceinline__ void time_weights_rcp(double inv_tau, double dt, double Mt[5]) {
  const double tau = nr_rcp(inv_tau);
  const double e = exp(-dt * inv_tau);
  Mt[3] = tau * (1.0 - e);
  Mt[4] = -tau * dt * e + tau * Mt[3];
  Mt[0] = dt - Mt[3];
  Mt[1] = -tau * Mt[0] + Mt[4];
  Mt[2] = 0.5 * (dt * dt) - tau * Mt[0];
}

// shared memory of a wall CTA: block-sum scratch, a broadcast
template <int NT>
struct FaceShared {
  double scratch[16 * (NT / 32)];
  double bcast[2];
};

// WENO5 (clFunctions.c:266-313) of one component, up to the final division:
// slope * dx = num / den.  Written in the first and second differences
// D_k = S_{k+1} - S_k, p_k = D_{k+1} - D_k:
//   4 beta_k = 13/3 p_k^2 + r_k^2,  r = (2 D1 + p0, D1 + D2, p2 - 2 D2)
//   6 (f_k - S2) = (2 r0 - D1, r1 + D2, D2 - r2)  (f_k: the candidates)
// and the weights c_k / (eps + beta_k)^2 multiplied through by
// prod_j (eps + beta_j)^2 (a common factor of num and den; eps scales with
// beta); the 1/6 is left to the caller.  35 FP64 operations per component
// against 44 with the candidates and smoothness terms spelled out.
__device__ __forceinline__ void weno5_part(const double (&S)[5], double &num6, double &den) {
  const double D0 = S[1] - S[0], D1 = S[2] - S[1], D2 = S[3] - S[2], D3 = S[4] - S[3];
  const double p0 = D1 - D0, p1 = D2 - D1, p2 = D3 - D2;
  const double r0 = fma(2.0, D1, p0), r1 = D1 + D2, r2 = fma(-2.0, D2, p2);
  constexpr double c = 13.0 / 3.0, eps = 4e-16;
  const double e0 = fma(c * p0, p0, fma(r0, r0, eps));
  const double e1 = fma(c * p1, p1, fma(r1, r1, eps));
  const double e2 = fma(c * p2, p2, fma(r2, r2, eps));
  const double q0 = e0 * e0, q1 = e1 * e1, q2 = e2 * e2;
  const double t0 = 3.0 * q0;
  const double a0 = q1 * q2, a1 = (t0 + t0) * q2, a2 = t0 * q1;  // 1 : 6 : 3
  num6 = fma(a0, fma(2.0, r0, -D1), fma(a1, r1 + D2, a2 * (D2 - r2)));
  den = (a0 + a1) + a2;
}

template <int L, typename VEC>
__device__ __forceinline__ void load_stencil(const VEC *p, int st, VEC (&x)[L]) {
#pragma unroll
  for (int s = 0; s < L; ++s) x[s] = p[s * st];
}

// iFace (clUGKS.c:148-194) for one velocity: face value and slope of (h, b).
// The two components share one reciprocal: 1/x = y * 1/(x y).
// The stencil runs upwind to downwind: cells MID+1 .. 1 before the face and
// 0 .. L-MID-2 after it for u > 0, mirrored for u <= 0; `p` points at stencil
// cell 0 and `st` is the signed cell stride in (h, b) pairs.
template <int FM>
__device__ __forceinline__ void reconstruct(const double2 (&x)[FM == 1 ? 5 : 3], double inv_l, double ds,
                                            double inv_ds, double &fh, double &fb, double &sh, double &sb) {
  constexpr int L = FM == 1 ? 5 : 3, MID = FM == 1 ? 2 : 1;
  double Sh[L], Sb[L];
#pragma unroll
  for (int s = 0; s < L; ++s) {
    Sh[s] = x[s].x;
    Sb[s] = x[s].y;
  }
  if constexpr (FM == 0) {
    // vanLeer (clFunctions.c:255-261)
    const double h1 = (Sh[1] - Sh[0]) * inv_l, h2 = (Sh[2] - Sh[1]) * inv_l;
    const double b1 = (Sb[1] - Sb[0]) * inv_l, b2 = (Sb[2] - Sb[1]) * inv_l;
    const double dh = fabs(h1) + fabs(h2) + 1e-16, db = fabs(b1) + fabs(b2) + 1e-16;
    const double r = nr_rcp(dh * db);
    sh = (ocl_sign(h1) + ocl_sign(h2)) * (fabs(h1) * fabs(h2)) * (db * r);
    sb = (ocl_sign(b1) + ocl_sign(b2)) * (fabs(b1) * fabs(b2)) * (dh * r);
  } else if constexpr (FM == 1) {
    double nh, dh, nb, db;
    weno5_part(Sh, nh, dh);
    weno5_part(Sb, nb, db);
    const double r = nr_rcp(dh * db) * ((1.0 / 6.0) * inv_ds);
    sh = nh * (db * r);
    sb = nb * (dh * r);
  } else {
    sh = (0.5 * minmod(Sh[2] - Sh[1], Sh[1] - Sh[0])) * inv_ds;
    sb = (0.5 * minmod(Sb[2] - Sb[1], Sb[1] - Sb[0])) * inv_ds;
  }
  fh = Sh[MID] + sh * ds;
  fb = Sb[MID] + sb * ds;
}

// The FP32 flux path (FP32 storage of h and b): the same reconstructions in
// single precision.  WENO5 keeps the difference form above, with the three
// smoothness terms e_k (>= 12e-16) divided by their sum before the products:
// the weights only enter as ratios, the largest scaled e_k is >= 1/3 and the
// smallest >= 1e-17, so the weight of the smoothest stencil stays a normal
// FP32 number (>= 1e-35) while only negligible weights can underflow.
// 1 / x by the hardware's approximate reciprocal (rcp.approx.ftz.f32, within
// about an ulp; denormal results flush to zero): the FP32 limiter and WENO5
// weights divide only by sums that are at least 1e-16 or normalised to 1
#ifndef UGKS_FRCP_APPROX
#define UGKS_FRCP_APPROX 1
#endif
__device__ __forceinline__ float frcp(float x) {
#if UGKS_FRCP_APPROX
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
#else
  return __fdividef(1.0f, x);
#endif
}
__device__ __forceinline__ float fsign(float a) {
  return a > 0.0f ? 1.0f : (a < 0.0f ? -1.0f : (a == 0.0f ? a : 0.0f));
}
__device__ __forceinline__ float fminmod(float a, float b) {
  float out = 0.0f;
  if ((fabsf(a) < fabsf(b)) && (a * b > 0.0f)) out = a;
  else if ((fabsf(b) < fabsf(a)) && (a * b > 0.0f)) out = b;
  else if (a == b) out = a;
  return out;
}
__device__ __forceinline__ void weno5_part_f(const float (&S)[5], float &num, float &den) {
  const float D0 = S[1] - S[0], D1 = S[2] - S[1], D2 = S[3] - S[2], D3 = S[4] - S[3];
  const float p0 = D1 - D0, p1 = D2 - D1, p2 = D3 - D2;
  const float r0 = fmaf(3.0f, D1, -D0), r1 = D1 + D2, r2 = fmaf(-3.0f, D2, D3);
  float e0 = 12e-16f + fmaf(13.0f * p0, p0, (3.0f * r0) * r0);
  float e1 = 12e-16f + fmaf(13.0f * p1, p1, (3.0f * r1) * r1);
  float e2 = 12e-16f + fmaf(13.0f * p2, p2, (3.0f * r2) * r2);
  const float sc = frcp((e0 + e1) + e2);
  e0 *= sc;
  e1 *= sc;
  e2 *= sc;
  const float q0 = e0 * e0, q1 = e1 * e1, q2 = e2 * e2;
  const float a0 = q1 * q2, a1 = 6.0f * (q0 * q2), a2 = 3.0f * (q0 * q1);
  const float f0 = fmaf(-1.0f / 3.0f, D0, (5.0f / 6.0f) * D1);
  const float f1 = fmaf(1.0f / 6.0f, D1, (1.0f / 3.0f) * D2);
  const float f2 = fmaf(2.0f / 3.0f, D2, (-1.0f / 6.0f) * D3);
  num = fmaf(a0, f0, fmaf(a1, f1, a2 * f2));
  den = (a0 + a1) + a2;
}
template <int FM>
__device__ __forceinline__ void reconstruct_f(const float2 (&xs)[FM == 1 ? 5 : 3], float inv_l, float ds, float inv_ds,
                                              float &fh, float &fb, float &sh, float &sb) {
  constexpr int L = FM == 1 ? 5 : 3, MID = FM == 1 ? 2 : 1;
  float Sh[L], Sb[L];
#pragma unroll
  for (int s = 0; s < L; ++s) {
    const float2 x = xs[s];
    Sh[s] = x.x;
    Sb[s] = x.y;
  }
  if constexpr (FM == 0) {
    const float h1 = (Sh[1] - Sh[0]) * inv_l, h2 = (Sh[2] - Sh[1]) * inv_l;
    const float b1 = (Sb[1] - Sb[0]) * inv_l, b2 = (Sb[2] - Sb[1]) * inv_l;
    sh = (fsign(h1) + fsign(h2)) * (fabsf(h1) * fabsf(h2)) * frcp(fabsf(h1) + fabsf(h2) + 1e-16f);
    sb = (fsign(b1) + fsign(b2)) * (fabsf(b1) * fabsf(b2)) * frcp(fabsf(b1) + fabsf(b2) + 1e-16f);
  } else if constexpr (FM == 1) {
    float nh, dh, nb, db;
    weno5_part_f(Sh, nh, dh);
    weno5_part_f(Sb, nb, db);
    sh = nh * frcp(dh) * inv_ds;
    sb = nb * frcp(db) * inv_ds;
  } else {
    sh = (0.5f * fminmod(Sh[2] - Sh[1], Sh[1] - Sh[0])) * inv_ds;
    sb = (0.5f * fminmod(Sb[2] - Sb[1], Sb[1] - Sb[0])) * inv_ds;
  }
  fh = fmaf(sh, ds, Sh[MID]);
  fb = fmaf(sb, ds, Sb[MID]);
}

// exp(-lambda (x - c)^2) over the nodes of one velocity axis
template <typename R>
__device__ __forceinline__ void axis_exp(R *out, const double *quad, int n, int stride,
                                         int comp, double c, double lambda, int t, int nt) {
  for (int i = t; i < n; i += nt) {
    const double x = quad[2 * (size_t)i * stride + comp] - c;
    out[i] = (R)exp(-lambda * (x * x));
  }
}

// stencil geometry of a face for both upwind directions (iFace,
// clUGKS.c:148-176): |mid - c|, 1/|mid - c| and 1/|c - c'| with c, c' the
// cells MID and MID-1 from the face (u <= 0), then the cells before the face
// (u > 0)
__device__ __forceinline__ void stencil_geometry(const ugks_fused_block &blk, long gi, long gj, int dir, V2 mid,
                                                 double *out) {
  const ugks_block_desc &d = blk.d;
  auto geo = [&](long c0, long c1, double *o) {
    const long c0i = dir == SOUTH ? gi : gi + c0, c0j = dir == SOUTH ? gj + c0 : gj;
    const long c1i = dir == SOUTH ? gi : gi + c1, c1j = dir == SOUTH ? gj + c1 : gj;
    const V2 a = ld2(blk.centre, gidx(d, c0i, c0j)), b = ld2(blk.centre, gidx(d, c1i, c1j));
    o[0] = sqrt((mid.x - a.x) * (mid.x - a.x) + (mid.y - a.y) * (mid.y - a.y));
    o[1] = 1.0 / o[0];
    o[2] = 1.0 / sqrt((a.x - b.x) * (a.x - b.x) + (a.y - b.y) * (a.y - b.y));
  };
  geo(0, 1, out);        // u <= 0
  geo(-1, -2, out + 3);  // u > 0
}

// the same for every face, once at set-up (read by the FP64 face pass)
__global__ void face_geometry(const ugks_fused_block *__restrict__ B, int nb, int n_faces) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= n_faces) return;
  const int bi = find_block<0>(B, nb, w);
  const ugks_fused_block &blk = B[bi];
  const ugks_block_desc &d = blk.d;
  int lf = w - blk.face_begin;
  const int dir = lf & 1;
  lf >>= 1;
  const int mi = lf / (d.nj + 1), mj = lf % (d.nj + 1);
  if (dir == SOUTH ? (mi >= d.ni) : (mj >= d.nj)) return;
  const long gi = mi + d.ghost, gj = mj + d.ghost;
  stencil_geometry(blk, gi, gj, dir, ld2(blk.mid_side, faceidx(d, gi, gj, dir)),
                   blk.face_geo + 6 * faceidx(d, gi, gj, dir));
}

// whether wall is the last adsorbing wall in the order N, S, E, W with a face ci
__device__ __forceinline__ bool last_on_row(const ugks_fused_block &blk, int wall, long ci) {
  auto rank = [](int f) { return ((f & 1) << 1) | (f >> 1); };
  for (int f = 0; f < 4; ++f)
    if (blk.bc_type[f] == BC_ADSORBING && rank(f) > rank(wall) && ci < ((f & 1) ? blk.d.nj : blk.d.ni)) return false;
  return true;
}

// The wall procedure of one wall face (all threads of the CTA take part):
// accommodatingWallDist (clUGKS.c:774-906) or adsorbingWall_P1 (clAdsorb.c:253-482)
// followed by the re-emission stage (adsorbingWallD_P2 / S_P2 / CL_P2,
// clAdsorb.c:488-975), then wallFlux (clUGKS.c:910-1011) and
// wallMassEnergyFluxes (1019-1147).  face_value(v, h, b) gives the reconstructed
// face distribution; fw holds Nv (h, b) pairs (each thread reads back only what
// it wrote); rin is scratch of this face alone, Nv (h, b) pairs, from which
// specular and Cercignani-Lampis walls gather the reflected incoming
// distribution; store_flux(v, h, b) writes the face-flux row of velocity v.
// wall_dist has one row per ci for all four walls of the block, whose CTAs run
// side by side, so nothing is read back from it: the wall the reference treats
// last (N, S, E, W) leaves its reflected distribution there, the others nothing.
// A diffuse wall takes two sweeps: the face values of the incoming half and the
// wall Maxwellian of the outgoing half (one exp each) with their two sums, then
// the fluxes with their eight sums.
template <int NT, typename RIN, typename FaceValue, typename StoreFlux>
__device__ __forceinline__ void wall_face(const ugks_fused_block &blk, ugks_solve_state &sol, FaceShared<NT> &sh,
                                          double *fw, RIN *rin, const int wall, const int dir, const long gi,
                                          const long gj, const long mi, const long mj, const V2 n, const double len,
                                          const double dt, FaceValue face_value, StoreFlux store_flux) {
  using R = double;
  const ugks_block_desc &d = blk.d;
  const int Nv = d.Nv;
  const double2 *__restrict__ qd = reinterpret_cast<const double2 *>(d.quad);
  const double *__restrict__ wt = d.weight;
  auto fvel = [&](int vv) {
    const double2 e = qd[vv];
    return v2(e.x * n.x + e.y * n.y, e.x * (-n.y) + e.y * n.x);
  };
  const int rot = (wall == GNORTH || wall == GEAST) ? -1 : 1;
  const long ci = dir == SOUTH ? mi : mj;
  P4 wl = ld4(blk.wall_prop, ci * 4 + wall);
  {
    const V2 t = to_local(v2(wl.s1, wl.s2), n);
    wl.s1 = t.x;
    wl.s2 = t.y;
  }
  double ratio_out = 1.0;  // diffuse: the outgoing half of fw is scaled by this
  if (blk.bc_type[wall] == BC_DIFFUSE) {
    // accommodatingWallDist (clUGKS.c:774-906)
    double s[2] = {0.0, 0.0};
    for (int v = threadIdx.x; v < Nv; v += NT) {
      const V2 uv = fvel(v);
      double h, b;
      if (upwind_flag(uv.x, rot)) {
        const V2 M = maxwellian(d, wl, uv, v);
        h = M.x;
        b = M.y;
        s[1] -= uv.x * h;
      } else {
        face_value(v, h, b);
        s[0] += uv.x * h;
      }
      fw[2 * v] = h;
      fw[2 * v + 1] = b;
    }
    block_sum_spread<2>(s, sh.scratch);
    ratio_out = s[0] / s[1];
  } else {
    for (int v = threadIdx.x; v < Nv; v += NT) face_value(v, fw[2 * v], fw[2 * v + 1]);
    // adsorbingWall_P1 (clAdsorb.c:253-482)
    const long ti = dir == SOUTH ? mi : (wall == GEAST ? d.ni - 1 : 0);
    const long tj = dir == SOUTH ? (wall == GNORTH ? d.nj - 1 : 0) : mj;
    const double Tw = 1.0 / blk.macro[4 * midx(d, ti, tj) + 3], Dw = blk.macro[4 * midx(d, ti, tj)];
    double *cover = blk.wall_cover + 4 * (ci * 4 + wall);
    const double theta = cover[0];
    const double gf = d.gamma_f[wall];
    double s[3] = {0.0, 0.0, 0.0};
    // the parts of the incoming flux of velocity v: reflected, adsorbed, beta times all
    auto incoming = [&](int v, V2 uv, V2 &refl, V2 &ads, double &stick) {
      const int delta = upwind_flag(uv.x, rot);
      const double k = -rot * uv.x * (1 - delta);
      const V2 total = v2(k * fw[2 * v], k * fw[2 * v + 1]);
      const double beta = sticking(d, uv, Tw, wall);
      ads = v2(beta * total.x * gf * (1.0 - theta), beta * total.y * gf * (1.0 - theta));
      const double fs = ocl_sign(total.x);
      if ((fs * ads.x) > (fs * total.x)) ads = total;
      refl = v2(total.x - ads.x, total.y - ads.y);
      stick = beta * total.x;
    };
    for (int v = threadIdx.x; v < Nv; v += NT) {
      V2 refl, ads;
      double stick;
      incoming(v, fvel(v), refl, ads, stick);
      s[0] += refl.x;
      s[1] += ads.x;
      s[2] += stick;
    }
    block_sum<3>(s, sh.scratch);
    if (threadIdx.x == 0) {
      double ads_final = s[1], dvt = 0.0, des = 0.0;
      bool ok = true;
      if (gf > 0.0) {
        if (d.dynamic[wall] == 1) {
          dvt = dt * d.alpha_p[wall] * s[1];
          if (dvt > (1 - theta)) {
            dvt = 1 - theta;
            ads_final = dvt / dt * d.alpha_p[wall];  // the reference's form (clAdsorb.c:420)
          }
        }
        if (d.k_des[wall] > 0.0) {
          des = d.k_des[wall] * theta / d.alpha_p[wall];
        } else {
          const V2 veq = vartheta_langmuir(d, Dw, Tw, wall);
          if (veq.y == 1.0) {
            atomicExch(&sol.status, 4);  // outside the tabulated isotherm
            ok = false;
          } else {
            des = gf * (1.0 / veq.x - 1.0) * s[2] * theta;
          }
        }
        if (ok) {
          if (d.dynamic[wall] == 1) {
            dvt -= dt * d.alpha_p[wall] * des;
            if ((theta + dvt) < 0.0) des = theta / (dt * d.alpha_p[wall]);
          }
        }
      }
      double corr = 1.0;
      if (ok) {
        const double refl_final = s[0] + s[1] - ads_final;
        corr = refl_final / s[0];
        cover[0] += dvt;
        cover[1] = refl_final;
        cover[2] = ads_final;
        cover[3] = des;
      }
      sh.bcast[0] = corr;
      sh.bcast[1] = ok ? 1.0 : 0.0;
    }
    __syncthreads();
    const double corr = sh.bcast[0];
    const bool ok = sh.bcast[1] != 0.0;
    const int kind = d.reflect[wall];
    const bool keep = last_on_row(blk, wall, ci), gather = ok && kind != UGKS_REFLECT_DIFFUSE;
    if (keep || gather)
      for (int v = threadIdx.x; v < Nv; v += NT) {
        const V2 uv = fvel(v);
        V2 x, ads;
        double stick;
        incoming(v, uv, x, ads, stick);
        x = v2(x.x / uv.x, x.y / uv.x);
        if (corr != 1.0) x = v2(x.x * corr, x.y * corr);
        if (keep) st2(blk.wall_dist, (size_t)ci * Nv + v, x);
        if (gather) {
          rin[v].x = x.x;
          rin[v].y = x.y;
        }
      }
    if (!ok) {
      // the reference skips the rest of this wall face and carries on
      // (ugks_block.py:949-950, 1084): its flux row keeps what iFace wrote
      // there, the face values of (h, b), and its face macro flux is not
      // written this step
      for (int v = threadIdx.x; v < Nv; v += NT) store_flux(v, fw[2 * v], fw[2 * v + 1]);
      return;
    }
    // re-emission of the reflected flux: adsorbingWallD_P2 (clAdsorb.c:821-975,
    // diffuse), adsorbingWallS_P2 (656-816, specular) or adsorbingWallCL_P2
    // (488-651, Cercignani-Lampis)
    const double refl = cover[1], des = cover[3], ads = cover[2];
    double ratio = 1.0;
    if (refl > 0.0) {
      __syncthreads();  // rin is complete
      const double an = d.alpha_n[wall], at = d.alpha_t[wall], Tw = 1.0 / wl.s3;
      double r[1] = {0.0};
      for (int v = threadIdx.x; v < Nv; v += NT) {
        const V2 uv = fvel(v);
        const int delta = upwind_flag(uv.x, rot);
        V2 out = v2(0.0, 0.0);
        if (delta) {
          if (kind == UGKS_REFLECT_DIFFUSE) {
            out = maxwellian(d, wl, uv, v);
          } else if (kind == UGKS_REFLECT_CL) {
            for (int va = 0; va < Nv; ++va) {
              const V2 uv_in = fvel(va);
              if (!upwind_flag(uv_in.x, rot) && uv_in.x != 0.0) {
                const auto fi = rin[va];
                const V2 c = cercignani_lampis(d.PI, uv_in, uv, v2(fi.x, fi.y), an, at, Tw, wl.s3);
                out.x += c.x;
                out.y += c.y;
              }
            }
            out.x *= wt[v];
            out.y *= wt[v];
          } else {
            const auto x = rin[dir == WEST ? d.mirror_EW[v] : d.mirror_NS[v]];
            out = v2(x.x, x.y);
          }
        }
        fw[2 * v] = (R)(delta * out.x + (1 - delta) * fw[2 * v]);
        fw[2 * v + 1] = (R)(delta * out.y + (1 - delta) * fw[2 * v + 1]);
        r[0] += rot * uv.x * out.x;
      }
      block_sum<1>(r, sh.scratch);
      ratio = refl / r[0];
    }
    const int account = ((des == 0.0) && (ads > 0.0) && (refl == 0.0)) ? 1 : 0;
    P4 wd = wl;
    wd.s0 = 2 * des * sqrt(d.PI * wl.s3);
    for (int v = threadIdx.x; v < Nv; v += NT) {
      const V2 uv = fvel(v);
      const int delta = upwind_flag(uv.x, rot);
      const double sc = 1 - delta * (1 - ratio);
      double x = fw[2 * v] * sc, y = fw[2 * v + 1] * sc;
      const V2 M = maxwellian(d, wd, uv, v);
      x += delta * M.x;
      y += delta * M.y;
      x -= account * delta * x;
      y -= account * delta * y;
      fw[2 * v] = (R)x;
      fw[2 * v + 1] = (R)y;
    }
  }
  // wallFlux (clUGKS.c:910-1011) and wallMassEnergyFluxes (1019-1147): the
  // incoming and outgoing sums; the face macro flux is both together
  double s[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) s[k] = 0.0;
  const double ld = len * dt;
  for (int v = threadIdx.x; v < Nv; v += NT) {
    const V2 uv = fvel(v);
    const bool out = upwind_flag(uv.x, rot) != 0;
    const double k = uv.x * ld * (out ? ratio_out : 1.0);
    const double oh = k * fw[2 * v], ob = k * fw[2 * v + 1];
    store_flux(v, oh, ob);
    const double e = 0.5 * ((uv.x * uv.x + uv.y * uv.y) * oh + ob), px = uv.x * oh, py = uv.y * oh;
    s[0] += out ? 0.0 : oh; s[1] += out ? 0.0 : px; s[2] += out ? 0.0 : py; s[3] += out ? 0.0 : e;
    s[4] += out ? oh : 0.0; s[5] += out ? px : 0.0; s[6] += out ? py : 0.0; s[7] += out ? e : 0.0;
  }
  block_sum_spread_to0<8>(s, sh.scratch);
  if (threadIdx.x == 0) {
    const V2 g = to_global(v2(s[1] + s[5], s[2] + s[6]), n);
    st4(dir == SOUTH ? blk.flux_macro_S : blk.flux_macro_W, gidx(d, gi, gj), p4(s[0] + s[4], g.x, g.y, s[3] + s[7]));
    double *wf = blk.wall_fluxes + 8 * (ci * 4 + wall);
    wf[0] = -rot * s[0]; wf[1] = rot * s[4]; wf[2] = -rot * s[1]; wf[3] = rot * s[5];
    wf[4] = -rot * s[2]; wf[5] = rot * s[6]; wf[6] = -rot * s[3]; wf[7] = rot * s[7];
  }
}

// face work item -> (block, i, j, direction, wall face); false when the item
// is skipped (inactive solve, retry pass of a solve without retry, another flux
// method than FM >= 0, or the unused S face of the last column / W face of the
// last row).  S and W faces of one corner (i, j) are adjacent work items so that
// both directions read f while it is in L2; with STRIPS a block's items are
// ordered in strips of FACE_STRIP columns i, in each first the S faces with j
// running fastest, then the W faces with i running fastest: consecutive items
// (the warps of a CTA) are neighbours along their normal and share most of
// their stencil rows in L1.
struct FaceWork {
  int bi, dir, mi, mj, wall;
  long gi, gj;
};
constexpr int FACE_STRIP = 4;
template <int FM, bool STRIPS = false>
__device__ __forceinline__ bool face_work(const ugks_fused_block *__restrict__ B, int nb,
                                          const ugks_solve_state *__restrict__ solves, const int w, int retry_pass,
                                          FaceWork &fw) {
  fw.bi = find_block<0>(B, nb, w);
  const ugks_fused_block &blk = B[fw.bi];
  const ugks_block_desc &d = blk.d;
  UGKS_CHECK_ITEM(0, blk, w, solves, false);
  const ugks_solve_state &sol = solves[blk.solve];
  if (!sol.active) return false;
  if (retry_pass && !step_dt(sol).retry) return false;
  if (FM >= 0 && d.flux_method != FM) return false;  // FM < 0: any flux method
  int lf = w - blk.face_begin;
  if (STRIPS) {
    const int c = d.nj + 1, strip = 2 * FACE_STRIP * c, s = lf / strip;
    const int wd = min(FACE_STRIP, d.ni + 1 - s * FACE_STRIP);
    lf -= s * strip;
    fw.dir = lf >= wd * c ? WEST : SOUTH;
    if (fw.dir == WEST) lf -= wd * c;
    fw.mi = s * FACE_STRIP + (fw.dir == SOUTH ? lf / c : lf % wd);
    fw.mj = fw.dir == SOUTH ? lf % c : lf / wd;
  } else {
    fw.dir = lf & 1;
    lf >>= 1;
    fw.mi = lf / (d.nj + 1);
    fw.mj = lf % (d.nj + 1);
  }
  if (fw.dir == SOUTH ? (fw.mi >= d.ni) : (fw.mj >= d.nj)) return false;
  fw.gi = fw.mi + d.ghost;
  fw.gj = fw.mj + d.ghost;
  fw.wall = -1;
  if (fw.dir == SOUTH) {
    if (fw.mj == 0 && is_wall(blk.bc_type[GSOUTH])) fw.wall = GSOUTH;
    else if (fw.mj == d.nj && is_wall(blk.bc_type[GNORTH])) fw.wall = GNORTH;
  } else {
    if (fw.mi == 0 && is_wall(blk.bc_type[GWEST])) fw.wall = GWEST;
    else if (fw.mi == d.ni && is_wall(blk.bc_type[GEAST])) fw.wall = GEAST;
  }
  return true;
}

// ---------------------------------------------------------------------------
// FP64 interior faces: a face per warp, its lanes over the velocities
// ---------------------------------------------------------------------------
// Any velocity grid and any face normal; no barrier, no shared memory per
// velocity: 16 faces are in flight on an SM whatever the velocity grid, each at
// its own phase, and the serial middle part of one hides behind the sweeps of
// the others.  On the 2x2-block cavity (Nv 1089, WENO5) 0.976 -> 0.716 ms, on a
// 96x96 cavity with Nv 2401 (vanLeer) 1.154 -> 0.868 ms, against a CTA per face
// that kept face values and slopes in shared memory over three velocity sweeps
// (six, at Nv 2401 two, faces per SM, with barriers around its serial part).
// Bound by the L1 / shared data pipe (71%: the stencil rows pass it once as
// cp.async and once as loads) and FP64 issue (50%) at 16 warps per SM.  Measured
// and not kept (against 0.730 ms then): no face values stored, the reconstruction run
// again in sweep 2, 0.917; stencil rows by plain loads a trip ahead, 0.840;
// rings of 3 or 4 stages, 0.750-0.790; 20 and 24 warps per SM at 96 and 80
// registers, 0.775 and 1.016 (the rows in flight outgrow L2); two velocities
// per lane side by side, 0.813; the three parts as launches of their own, 0.866;
// a CTA per face with threads that hold their v node, 0.801.
//
//   sweep 1  reconstruction (iFace); the face values into the face's flux row
//            (an L2 round trip of 16 bytes a velocity),
//            nine raw moments that give the face state (getFaceCons) and heat
//            flux (calcFaceQ);
//   once     slopes (getPLR), initMacroFlux, time weights: the two sides of the
//            face on even and odd lanes;
//   sweep 2  macroFlux and distFlux over the stored values, the slope taken
//            again as (face value - upwind cell) / distance.
//
// Face record (per warp, shared memory): polynomials a0 + ax x + ay y + a3 (x^2
// + y^2) in the global velocity components, time weights, face state.  It
// takes the place of the moments.
enum {
  FK_L = 0, FK_R = 6, FK_T = 12, FK_MT3 = 18, FK_MT4, FK_SX, FK_SY, FK_G0, FK_UX = FK_G0 + 4, FK_UY, FK_LAM, FK_KB,
  FK_CHL, FK_NUM
};
constexpr int FACE_MOM = 9;    // h, xh, yh, xxh, xyh, yyh, b, x t, y t with t = (x^2 + y^2) h + b / K
constexpr int FACE_TAB = 32;   // doubles of a record
static_assert(FK_NUM <= FACE_TAB && FACE_MOM <= FACE_TAB, "face record layout");

// what both sweeps of a face need
template <int FM>
struct FaceRows {
  V2 n;
  double dist0, idist0, il0, dist1, idist1, il1;
  int step;
  const double2 *fcell;  // cell (gi, gj), velocity 0
  double2 *row;          // the face's flux row
  static constexpr int L = FM == 1 ? 5 : 3, MID = FM == 1 ? 2 : 1;
  __device__ __forceinline__ FaceRows(const ugks_fused_block &blk, const FaceWork &w) {
    const ugks_block_desc &d = blk.d;
    const size_t fk = faceidx(d, w.gi, w.gj, w.dir), base = fidx(d, w.gi, w.gj, 0);
    n = ld2(blk.normal, fk);
    const double *g = blk.face_geo + 6 * fk;
    dist0 = g[0]; idist0 = g[1]; il0 = g[2]; dist1 = g[3]; idist1 = g[4]; il1 = g[5];
    step = w.dir == SOUTH ? d.Nv : d.Nj * d.Nv;
    fcell = reinterpret_cast<const double2 *>(blk.f) + base;
    row = reinterpret_cast<double2 *>(w.dir == SOUTH ? blk.flux_S : blk.flux_W) + base;
  }
  __device__ __forceinline__ bool up(double2 e) const { return fma(e.x, n.x, e.y * n.y) > 0.0; }
  // stencil cell 0 and the signed stride of velocity v
  __device__ __forceinline__ const double2 *stencil(int v, bool u, int &st) const {
    st = u ? step : -step;
    return fcell + (v + (u ? -(MID + 1) * step : MID * step));
  }
  __device__ __forceinline__ void value(const double2 (&x)[L], bool u, double &h, double &b, double &sh,
                                        double &sb) const {
    reconstruct<FM>(x, u ? il1 : il0, u ? dist1 : dist0, u ? idist1 : idist0, h, b, sh, sb);
  }
};
__device__ __forceinline__ void add_moments(double2 e, double Kinv, double h, double b, double (&m)[FACE_MOM]) {
  const double xh = e.x * h, yh = e.y * h;
  const double t = fma(fma(e.x, e.x, e.y * e.y), h, b * Kinv);
  m[0] += h;
  m[1] += xh;
  m[2] += yh;
  m[3] = fma(e.x, xh, m[3]);
  m[4] = fma(e.y, xh, m[4]);
  m[5] = fma(e.y, yh, m[5]);
  m[6] += b;
  m[7] = fma(e.x, t, m[7]);
  m[8] = fma(e.y, t, m[8]);
}

// calcQ of a distribution from its raw moments M about 0 (add_moments), relative
// to velocity U, global frame
__device__ __forceinline__ V2 face_heat_flux(const double (&M)[FACE_MOM], double Kinv, V2 U) {
  const double cu = fma(U.x, M[1], U.y * M[2]), U2 = fma(U.x, U.x, U.y * U.y);
  const double T = fma(Kinv, M[6], M[3] + M[5]) - 2.0 * cu + U2 * M[0];
  return v2(0.5 * (M[7] - 2.0 * fma(U.x, M[3], U.y * M[4]) + U2 * M[1] - U.x * T),
            0.5 * (M[8] - 2.0 * fma(U.x, M[4], U.y * M[5]) + U2 * M[2] - U.y * T));
}

// stages of cp.async in flight per lane: the stencil rows of FACE_RING
// velocities in sweep 1, (face value, upwind cell) of as many as fit in the
// same memory in sweep 2; a lane reads back only what it copied
constexpr int FACE_RING = 2;
template <int FM>
constexpr int face_ring_elems() { return FACE_RING * FaceRows<FM>::L * 32; }

// The per-face coefficients, by the face's warp: `rec` holds the moments and
// receives the record.  Even lanes compute the side before the face, odd lanes
// the side after it (the same instructions with one sign flipped).  Not
// inlined: it runs once per face, and its registers would weigh on the sweeps (128
// in the default shape, 96 and 168 in shapes 2 and 4).
__device__ __noinline__ void face_coefficients(const ugks_fused_block &blk, double dt, const FaceWork fwk,
                                               double *rec) {
  const ugks_block_desc &d = blk.d;
  const int lane = threadIdx.x & 31, side = lane & 1;
  double M[FACE_MOM];
#pragma unroll
  for (int k = 0; k < FACE_MOM; ++k) M[k] = rec[k];
  __syncwarp();  // every lane has the moments before the record takes their place
  const int dir = fwk.dir;
  const long gi = fwk.gi, gj = fwk.gj;
  const size_t fk = faceidx(d, gi, gj, dir);
  const size_t ck = side == 0 ? gidx(d, gi - dir, gj - (1 - dir)) : gidx(d, gi, gj);
  const P4 mc = ld4(blk.cell_mom, ck);
  const V2 cc = ld2(blk.centre, ck), mid = ld2(blk.mid_side, fk), n = ld2(blk.normal, fk);
  const double len = blk.side_length[fk], Kinv = nr_rcp(d.K);
  const V2 Wm = to_local(v2(M[1], M[2]), n);
  const P4 W = p4(M[0], Wm.x, Wm.y, 0.5 * (M[3] + M[5] + M[6]));
  Rcp rc;
  const P4 prim = to_primary_rcp(d, W, rc);  // getPLR (clUGKS.c:421-422)
  const V2 Ug = to_global(v2(prim.s1, prim.s2), n);
  const double kb = (0.5 * d.K) * rc.lam, sg = side == 0 ? 1.0 : -1.0;
  double Mh[MNUM], Mv[MTUM], Mxi[3];
  half_moments_rcp(d.PI, d.K, prim, rc, sg, Mh, Mv, Mxi);
  // left: (W - W_L) / |mid - c_L|; right: (W_R - W) / |mid - c_R|
  const V2 uc = to_local(v2(mc.s1, mc.s2), n);
  const double id = sg * nr_rcp(sqrt((mid.x - cc.x) * (mid.x - cc.x) + (mid.y - cc.y) * (mid.y - cc.y)));
  const P4 a = micro_slope_rcp(d.K, prim, rc,
                               p4((W.s0 - mc.s0) * id, (W.s1 - uc.x) * id, (W.s2 - uc.y) * id, (W.s3 - mc.s3) * id));
  // sums over both sides, by exchange with the neighbouring lane
  auto both = [](double z) { return z + __shfl_xor_sync(0xffffffffu, z, 1); };
  auto both4 = [&](P4 z) { return p4(both(z.s0), both(z.s1), both(z.s2), both(z.s3)); };
  const P4 t1 = both4(moment_au(a, Mh, Mv, Mxi, 1, 0)), t2 = both4(moment_au(a, Mh, Mv, Mxi, 2, 0));
  double Mu[MNUM];
#pragma unroll
  for (int k = 0; k < MNUM; ++k) Mu[k] = both(Mh[k]);
  const P4 aT = micro_slope_rcp(d.K, prim, rc, scale(-prim.s0, t1));
  double Mt[5];
  time_weights_rcp(inv_relax_time_rcp(d, prim, rc), dt, Mt);
  const P4 g0 = scale(prim.s0, add(add(scale(Mt[0], moment_uv(Mu, Mv, Mxi, 1, 0, 0)), scale(Mt[1], t2)),
                                   scale(Mt[2], moment_au(aT, Mu, Mv, Mxi, 1, 0))));
  // calcQ of the face values (calcFaceQ, clUGKS.c:522-585) from their raw
  // moments about 0, global frame; times the Shakhov factor and Mt0
  const V2 q = face_heat_flux(M, Kinv, Ug);
  const double s0 = 0.8 * (1 - d.Pr) * (prim.s3 * prim.s3) * rc.rho * Mt[0];
  const double xk = Mxi[2] - kb * kb;
  // a1 u + a2 v = x (a1 n.x - a2 n.y) + y (a1 n.y + a2 n.x)
  auto put = [&](double *c, P4 z, double w, double w0) {
    c[0] = fma(w, fma(0.5 * z.s3, kb, z.s0), w0);
    c[1] = w * (z.s1 * n.x - z.s2 * n.y);
    c[2] = w * (z.s1 * n.y + z.s2 * n.x);
    c[3] = w * (0.5 * z.s3);
    c[4] = w * (0.5 * z.s3 * xk);
  };
  if (lane < 2) put(rec + FK_L + 6 * side, a, Mt[1], 0.0);
  if (lane == 2) put(rec + FK_T, aT, Mt[2], Mt[0]);
  if (lane == 3) {
    rec[FK_MT3] = Mt[3] * len;
    rec[FK_MT4] = Mt[4] * len;
    rec[FK_SX] = s0 * q.x;
    rec[FK_SY] = s0 * q.y;
    const V2 g = to_global(v2(g0.s1, g0.s2), n);
    rec[FK_G0] = len * g0.s0;
    rec[FK_G0 + 1] = len * g.x;
    rec[FK_G0 + 2] = len * g.y;
    rec[FK_G0 + 3] = len * g0.s3;
    rec[FK_UX] = Ug.x;
    rec[FK_UY] = Ug.y;
    rec[FK_LAM] = prim.s3;
    rec[FK_KB] = kb;
    // Maxwellian prefactor rho lambda / pi (fM, clFunctions.c:49-58) times the
    // face length: every per-velocity flux carries the length
    rec[FK_CHL] = prim.s0 * prim.s3 * nr_rcp(d.PI) * len;
  }
}

// the Maxwellian factor of a velocity on a grid that is not a tensor product
__device__ __noinline__ double plain_exp(double x) { return exp(x); }

// Sweep 2.  With h0 = weight * fM (times the face length), kb = K / (2 lambda),
// S = Mt0 s (c . Q) (the Shakhov factor of fS, clFunctions.c:64-77, times
// Mt0), P4 = 2 lambda c^2 - 4, the upwind slope a (aL for u > 0, else aR),
//   Ph = a0 + a1 u + a2 v + a3 (|u|^2 + kb) / 2, and Th likewise with aT,
//   Rh = Mt3 fh - Mt4 u sh,   Rb = Mt3 fb - Mt4 u sb,
//   Zh = u (S P4 h0 + Rh),    Zb = u (S (P4 + 2) kb h0 + Rb),
//   B  = Mt0 + Mt1 u Ph + Mt2 Th,
// distFlux's (clUGKS.c:683-772) two components are
//   hx = Zh + u h0 B,
//   hy = Zb + u h0 (kb B + Mt1 u a3 X / 2 + Mt2 aT3 X / 2),  X = Mxi2 - kb^2,
// and macroFlux's (587-681) discrete part sums (Zh, x Zh, y Zh, (|u|^2 Zh + Zb) / 2)
// in the global frame.
template <int FM>
__device__ __forceinline__ void face_item_fp64(const ugks_fused_block &blk, const double dt, double *rec,
                                               double2 *ring, const FaceWork &fwk) {
  const ugks_block_desc &d = blk.d;
  const int lane = threadIdx.x & 31, Nv = d.Nv, un = d.u_num, vn = d.v_num;
  const FaceRows<FM> F(blk, fwk);
  constexpr int L = FaceRows<FM>::L, D = FACE_RING, D2 = face_ring_elems<FM>() / 64;
  const double2 *__restrict__ qd = reinterpret_cast<const double2 *>(d.quad);
  ring += lane;
  {
    auto issue = [&](int v, int stage) {
      if (v < Nv) {
        int st;
        const double2 *p = F.stencil(v, F.up(qd[v]), st);
        double2 *r = ring + stage * (L * 32);
#pragma unroll
        for (int s = 0; s < L; ++s) cp_async<16, true>(r + 32 * s, p + s * st);
      }
      cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < D; ++s) issue(lane + 32 * s, s);
    double m[FACE_MOM] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
    const double Kinv = nr_rcp(d.K);
    int stage = 0;
#pragma unroll 1
    for (int v = lane; v < Nv; v += 32) {
      const double2 e = qd[v];
      cp_async_wait<D - 1>();
      double2 xs[L];
      const double2 *r = ring + stage * (L * 32);
#pragma unroll
      for (int s = 0; s < L; ++s) xs[s] = r[32 * s];
      double h, b, sh, sb;
      F.value(xs, F.up(e), h, b, sh, sb);
      F.row[v] = make_double2(h, b);
      issue(v + 32 * D, stage);
      stage = stage + 1 == D ? 0 : stage + 1;
      add_moments(e, Kinv, h, b, m);
    }
    cp_async_wait<0>();
    const double t = warp_spread_sum<FACE_MOM>(m);
    constexpr int S = spread_shift<FACE_MOM>();
    if ((lane & ((1 << S) - 1)) == 0 && (lane >> S) < FACE_MOM) rec[lane >> S] = t;
  }
  __threadfence_block();  // this lane's row[] before its copies of it
  __syncwarp();
  auto up_at = [&](int v) { return v < Nv && F.up(qd[v]); };
  auto issue = [&](int v, int stage, bool u) {
    if (v < Nv) {
      double2 *r = ring + stage * 64;
      cp_async<16>(r, F.row + v);
      cp_async<16>(r + 32, F.fcell + v - (u ? F.step : 0));
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < D2; ++s) issue(lane + 32 * s, s, up_at(lane + 32 * s));  // under the coefficients
  face_coefficients(blk, dt, fwk, rec);
  __syncwarp();
  const bool sep = un > 0 && un * vn == Nv && un + vn <= 512;
  double *Eu = rec + FACE_TAB, *Ev = Eu + un;
  const double lam = rec[FK_LAM], Ux = rec[FK_UX], Uy = rec[FK_UY], kb = rec[FK_KB];
  if (sep) {
    // axis factors of the face Maxwellian, the prefactor on the u axis
    const double chl = rec[FK_CHL];
    for (int k = lane; k < un + vn; k += 32) {
      const double z = k < un ? qd[(size_t)k * vn].x - Ux : qd[k - un].y - Uy;
      Eu[k] = (k < un ? chl : 1.0) * exp(-lam * (z * z));
    }
    __syncwarp();
  }
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  {
    const double lam2 = 2.0 * lam, sx = rec[FK_SX], sy = rec[FK_SY], Mt3 = rec[FK_MT3], Mt4 = rec[FK_MT4];
    const double T0 = rec[FK_T], T1 = rec[FK_T + 1], T2 = rec[FK_T + 2], T3 = rec[FK_T + 3], CT = rec[FK_T + 4];
    const double *__restrict__ wt = d.weight;
    const int qs = sep ? 32 / vn : 0, rs = sep ? 32 % vn : 0;
    int iu = sep ? lane / vn : 0, jv = sep ? lane % vn : 0;
    int stage = 0;
#pragma unroll 1
    for (int v = lane; v < Nv; v += 32) {
      const double2 e = qd[v];
      const double wv = wt[v];
      // the side of the velocity copied at the end of this trip: taken there, its load
      // stood before the copy (2x2-block cavity, face pass 0.758 against 0.715 ms)
      const bool next_up = up_at(v + 32 * D2);
      const double u = fma(e.x, F.n.x, e.y * F.n.y), uu = fma(e.x, e.x, e.y * e.y);
      const double cx = e.x - Ux, cy = e.y - Uy, c2 = fma(cx, cx, cy * cy);
      double E;
      if (sep) {
        E = Eu[iu] * Ev[jv];
        jv += rs;
        iu += qs;
        if (jv >= vn) { jv -= vn; ++iu; }
      } else {
        E = rec[FK_CHL] * plain_exp(-lam * c2);
      }
      const double h0 = wv * E;
      const double Sp = fma(cx, sx, cy * sy);
      const double S4 = Sp * fma(lam2, c2, -4.0), S2 = fma(2.0, Sp, S4);
      const double *A = rec + (u > 0.0 ? FK_L : FK_R);
      const double MP = fma(A[3], uu, fma(A[2], e.y, fma(A[1], e.x, A[0])));
      const double Bk = fma(u, MP, fma(T3, uu, fma(T2, e.y, fma(T1, e.x, T0))));
      cp_async_wait<D2 - 1>();
      const double2 fd = ring[stage * 64], fc = ring[stage * 64 + 32];
      const double mu = (Mt4 * u) * (u > 0.0 ? F.idist1 : F.idist0);
      const double Rh = fma(-mu, fd.x - fc.x, Mt3 * fd.x), Rb = fma(-mu, fd.y - fc.y, Mt3 * fd.y);
      const double Zh = u * fma(S4, h0, Rh), Zb = u * fma(S2, h0 * kb, Rb);
      const double uh = u * h0;
      const double hx = fma(uh, Bk, Zh);
      const double hy = fma(uh, fma(kb, Bk, fma(A[4], u, CT)), Zb);
      acc[0] += Zh;
      acc[1] = fma(e.x, Zh, acc[1]);
      acc[2] = fma(e.y, Zh, acc[2]);
      acc[3] = fma(uu, Zh, acc[3]) + Zb;
      // streamed: read next by the cell pass, a gigabyte of other traffic later
      __stcs(F.row + v, make_double2(hx, hy));
      // refilled only after the store that consumed the stage's values: a copy is
      // not ordered after loads of its target that are still under way
      issue(v + 32 * D2, stage, next_up);
      stage = stage + 1 == D2 ? 0 : stage + 1;
    }
    cp_async_wait<0>();
  }
  acc[3] *= 0.5;
  const double t = warp_spread_sum<4>(acc);
  constexpr int S = spread_shift<4>();
  if ((lane & ((1 << S) - 1)) == 0) {
    const int k = lane >> S;
    (fwk.dir == SOUTH ? blk.flux_macro_S : blk.flux_macro_W)[4 * gidx(d, fwk.gi, fwk.gj) + k] = t + rec[FK_G0 + k];
  }
  __syncwarp();  // the record is free again
}

// A wall face in FP64 (all NT threads of the CTA take part): the face values
// live in the face's flux row, which the wall procedure works on in place; the
// reflected incoming distribution it gathers from lies in the row behind the
// wall, a ghost face that nothing else touches (there are two ghost layers or more).
template <int FM, int NT>
__device__ __noinline__ void wall_item_fp64(const ugks_fused_block &blk, ugks_solve_state &sol, const double dt,
                                            FaceShared<NT> &sh, const FaceWork fwk) {
  const ugks_block_desc &d = blk.d;
  const int dir = fwk.dir, Nv = d.Nv;
  const long gi = fwk.gi, gj = fwk.gj;
  const size_t fk = faceidx(d, gi, gj, dir), base = fidx(d, gi, gj, 0);
  const V2 n = ld2(blk.normal, fk);
  const double *fg = blk.face_geo + 6 * fk;
  const int step = dir == SOUTH ? Nv : d.Nj * Nv;
  constexpr int L = FM == 1 ? 5 : 3, MID = FM == 1 ? 2 : 1;
  const double2 *fcell = reinterpret_cast<const double2 *>(blk.f) + base;
  const double2 *up1 = fcell - (MID + 1) * step, *up0 = fcell + MID * step;
  const double2 *qd = reinterpret_cast<const double2 *>(d.quad);
  double2 *row = reinterpret_cast<double2 *>(dir == SOUTH ? blk.flux_S : blk.flux_W) + base;
  auto face_value = [&](int v, double &h, double &b) {
    const double2 e = qd[v];
    const bool up = fma(e.x, n.x, e.y * n.y) > 0.0;
    const double *g = fg + (up ? 3 : 0);
    double2 xs[L];
    load_stencil((up ? up1 : up0) + v, up ? step : -step, xs);
    double sx, sy;
    reconstruct<FM>(xs, g[2], g[0], g[1], h, b, sx, sy);
  };
  double2 *behind = row + (fwk.wall == GNORTH || fwk.wall == GEAST ? step : -step);
  wall_face<NT>(blk, sol, sh, reinterpret_cast<double *>(row), behind, fwk.wall, dir, gi, gj, fwk.mi, fwk.mj, n,
                blk.side_length[fk], dt, face_value, [&](int v, double hx, double hy) { row[v] = make_double2(hx, hy); });
}

// wall work item (2 (ni + nj) per block: the S faces of rows 0 and nj, then
// the W faces of columns 0 and ni) -> the face work item of that face
__device__ __forceinline__ int wall_to_face(const ugks_fused_block &blk, int w) {
  const ugks_block_desc &d = blk.d;
  int lw = w - blk.wall_begin, mi, mj, dir;
  if (lw < 2 * d.ni) {
    dir = SOUTH;
    mi = lw % d.ni;
    mj = lw < d.ni ? 0 : d.nj;
  } else {
    lw -= 2 * d.ni;
    dir = WEST;
    mj = lw % d.nj;
    mi = lw < d.nj ? 0 : d.ni;
  }
  return blk.face_begin + ((mi * (d.nj + 1) + mj) << 1) + dir;
}

// Cercignani-Lampis walls of more than WIDE_NV velocities, FP64: the Nv^2 loop of
// such a face is as long as its CTA is narrow, so that tables that have any (a
// segment of method UGKS_SEG_CL_WALLS) take them in a launch of their own, in CTAs
// of WIDE_NT threads, beside which the faces run.  Step in ms with these walls in
// the face pass's CTAs of 128 threads and so: 32 wall faces of 1681 velocities 11.2
// and 3.8, 256 of 1369 8.7 and 5.4, 256 of 2401 25.0 and 14.3.
constexpr int WALL_NT = 128, WIDE_NV = 1100, WIDE_NT = 512;
__host__ __device__ inline bool wide_cl_wall(const ugks_fused_block &blk, int wall) {
  return blk.d.Nv > WIDE_NV && blk.bc_type[wall] == BC_ADSORBING && blk.d.reflect[wall] == UGKS_REFLECT_CL;
}
inline bool has_cl_walls(const ugks_fused_sizes *z) {
  return z->n_segments > 0 && z->seg_method[z->n_segments - 1] == UGKS_SEG_CL_WALLS;
}

// a wall work item of any flux method (all threads of the CTA): every wall, the wide
// Cercignani-Lampis walls only, or the others only
enum WallKind { WALL_ANY, WALL_WIDE_CL, WALL_OTHER };
template <int NT>
__device__ __forceinline__ void wall_work_fp64(const ugks_fused_block *__restrict__ B, int nb,
                                               ugks_solve_state *__restrict__ solves, const int w, int retry_pass,
                                               WallKind kind) {
  __shared__ FaceShared<NT> sh;
  const ugks_fused_block &blk = B[find_block<3>(B, nb, w)];
  UGKS_CHECK_ITEM(3, blk, w, solves);
  FaceWork fwk;
  if (!face_work<-1>(B, nb, solves, wall_to_face(blk, w), retry_pass, fwk) || fwk.wall < 0) return;
  if (kind != WALL_ANY && wide_cl_wall(blk, fwk.wall) != (kind == WALL_WIDE_CL)) return;
  ugks_solve_state &sol = solves[blk.solve];
  const double dt = retry_pass ? step_dt(sol).flux : sol.dt;
  switch (blk.d.flux_method) {
    case 0: wall_item_fp64<0, NT>(blk, sol, dt, sh, fwk); break;
    case 1: wall_item_fp64<1, NT>(blk, sol, dt, sh, fwk); break;
    case 3: wall_item_fp64<3, NT>(blk, sol, dt, sh, fwk); break;
    default: break;
  }
}

__global__ void __launch_bounds__(WIDE_NT) cl_wall_pass_fp64(const ugks_fused_block *__restrict__ B, int nb,
                                                             ugks_solve_state *__restrict__ solves) {
  pdl_begin();
  wall_work_fp64<WIDE_NT>(B, nb, solves, (int)blockIdx.x, 0, WALL_WIDE_CL);
}

// FP64 face pass: the first n_wall CTAs take a wall work item each (they are
// the longest, so they start first), the others WPC interior faces, one per warp
template <int FM, int WPC>
__device__ __forceinline__ double2 *face_ring(double *dyn, int wstride, int warp) {
  return reinterpret_cast<double2 *>(dyn + WPC * wstride) + warp * face_ring_elems<FM>();
}
template <int FM, int WPC, int MINB>
__global__ void __launch_bounds__(WPC * 32, MINB) face_pass_fp64(const ugks_fused_block *__restrict__ B, int nb,
                                                                 ugks_solve_state *__restrict__ solves, int n_wall,
                                                                 WallKind kind, int first, int count, int wstride,
                                                                 int chained) {
  extern __shared__ double dyn[];
  pdl_begin_face(chained);
  const int warp = threadIdx.x >> 5;
  const int item = ((int)blockIdx.x - n_wall) * WPC + warp;
  FaceWork fwk;
  if ((int)blockIdx.x < n_wall) {
    wall_work_fp64<WPC * 32>(B, nb, solves, (int)blockIdx.x, 0, kind);
  } else if (item < count && face_work<FM, true>(B, nb, solves, first + item, 0, fwk) && fwk.wall < 0) {
    const ugks_fused_block &blk = B[fwk.bi];
    // the dt of the step's final flux pass: the reference's first pass, when it is
    // redone, leaves nothing of an interior face
    face_item_fp64<FM>(blk, step_dt(solves[blk.solve]).flux, dyn + warp * wstride, face_ring<FM, WPC>(dyn, wstride, warp),
                       fwk);
  }
}

// The walls' flux pass redone after a dt change (ugks_sim.py:432-441), for few solves
// in few steps.  An interior face has nothing to redo, a wall has: its coverage moves
// in both passes.  Every CTA finds the solves that retry, and their walls count through
// as one list, dealt to the CTAs in turn.  Against a pass over all faces of these
// solves, a step whose dt grows by its limit: 64x64 cells of 625 velocities 497 -> 206
// us, 32x16 of 2401 435 -> 261, 16 solves of 48x48 and 625 2453 -> 1523.
inline unsigned retry_grid(int ns) { return (unsigned)std::min(592l, 148l * ns); }
__device__ __forceinline__ bool retries(const ugks_solve_state &x) { return x.active && x.nblocks > 0 && step_dt(x).retry; }
template <typename Work>
__device__ __forceinline__ void redo_walls(const ugks_fused_block *__restrict__ B,
                                           const ugks_solve_state *__restrict__ solves, int ns, Work work) {
  int before = 0;  // walls of the solves before
  auto solve = [&](int s) {
    const ugks_solve_state &x = solves[s];
    const ugks_fused_block &b = B[x.first_block], &e = B[x.first_block + x.nblocks - 1];
    const int n = e.wall_begin + 2 * (e.d.ni + e.d.nj) - b.wall_begin, ctas = gridDim.x;
    for (int w = ((int)blockIdx.x + ctas - before % ctas) % ctas; w < n; w += ctas) {
      work(b.wall_begin + w);
      __syncthreads();  // the next item reuses the shared tables
    }
    before += n;
  };
  if (ns == 1) {  // the usual table
    if (retries(solves[0])) solve(0);
    return;
  }
  // a lane per solve, by every warp for itself: all of a CTA with the same result
  const int lane = threadIdx.x & 31;
  bool any = false;
  for (int s = lane; s < ns; s += 32) any |= retries(solves[s]);
  if (!__any_sync(0xffffffffu, any)) return;
  for (int s0 = 0; s0 < ns; s0 += 32)
    for (unsigned m = __ballot_sync(0xffffffffu, s0 + lane < ns && retries(solves[s0 + lane])); m; m &= m - 1)
      solve(s0 + __ffs(m) - 1);
}
template <int NT>
__global__ void __launch_bounds__(NT, 512 / NT) wall_retry_fp64(const ugks_fused_block *__restrict__ B, int nb,
                                                                ugks_solve_state *__restrict__ solves, int ns) {
  pdl_begin();
  redo_walls(B, solves, ns, [&](int w) { wall_work_fp64<NT>(B, nb, solves, w, 1, WALL_ANY); });
}
// ---------------------------------------------------------------------------
// cell pass: calcQ (clKernel.c:480-543) + updateMacro (clUGKS.c:1158-1187) +
// UGKS_update (clUGKS.c:1189-1257) + clFindDT (clKernel.c:224-308)
// ---------------------------------------------------------------------------
// clFindDT with the descriptor's Kn (the host's unrounded Kn, ugks_block.py:1421)
__device__ __forceinline__ double cfl_freq(const ugks_fused_block &blk, P4 m, long mi, long mj) {
  return cfl_frequency(blk.d, blk.xy, blk.area, m, mi, mj, blk.d.Kn_eff);
}

// One warp per cell, CW cells per CTA.  The serial per-cell part (updateMacro,
// two relaxation times, the CFL frequency: some 1500 instructions) of the CTA's
// cells runs on CW lanes of its first warp, one cell each, while the others
// build the old states' tables and the first rows are on their way; every warp
// running it for its own cell on one lane cost 2x2-block FP64 0.320 ms against
// 0.301, a 24x24 cavity 18.4 us against 16.8.  The moments of f^{n+1} are summed
// in the update loop (a second sweep over f: 0.314 ms).  Bound by memory latency:
// 1.2 GB at 4 TB/s with 16 warps per SM.
constexpr int CW = 4;
// per-warp shared memory: the axis tables of the old and new state
// (2 (u_num + v_num) doubles) and CELL_COEF coefficient slots
constexpr int CELL_COEF = 14;
enum { CC_U, CC_V, CC_LAM, CC_A1, CC_A2, CC_A3, CC_A4, CC_P, CC_KN, CC_SN, CC_LNP };

template <int N>
__device__ __forceinline__ void warp_sum(double (&x)[N]) {
#pragma unroll
  for (int k = 0; k < N; ++k) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x[k] += __shfl_xor_sync(0xffffffffu, x[k], o);
  }
}

// a cell warp's cell: false when the warp has none (past the end, or a solve
// that is switched off)
struct CellWork {
  int bi;
  long mi, mj, gi, gj;
};
__device__ __forceinline__ bool cell_work(const ugks_fused_block *__restrict__ B, int nb,
                                          const ugks_solve_state *__restrict__ solves, int w, int n_cells, CellWork &c) {
  if (w >= n_cells) return false;
  c.bi = find_block<1>(B, nb, w);
  const ugks_fused_block &blk = B[c.bi];
  UGKS_CHECK_ITEM(1, blk, w, solves, false);
  if (!solves[blk.solve].active) return false;
  const int lc = w - blk.cell_begin;
  c.mi = lc / blk.d.nj;
  c.mj = lc % blk.d.nj;
  c.gi = c.mi + blk.d.ghost;
  c.gj = c.mj + blk.d.ghost;
  return true;
}

// updateMacro, the relaxation weights of UGKS_update and the CFL frequency of
// one cell (a thread), its coefficients into bc:
//   a1 = (1 - dt/2 /tau_old) / D, a2 = 1 / (A D), a3 = dt/2 / (tau D),
//   a4 = dt/2 / (tau_old D), D = 1 + dt/2 / tau  (a1 + a3 + a4 = 1)
__device__ __forceinline__ double cell_coefficients(const ugks_fused_block &blk, const ugks_solve_state &sol,
                                                    const CellWork &c, double *bc, double P0pi) {
  const ugks_block_desc &d = blk.d;
  const size_t m = midx(d, c.mi, c.mj);
  const P4 old = ld4(blk.macro, m);
  const P4 s0 = ld4(blk.flux_macro_S, gidx(d, c.gi, c.gj)), s1 = ld4(blk.flux_macro_S, gidx(d, c.gi, c.gj + 1));
  const P4 w0 = ld4(blk.flux_macro_W, gidx(d, c.gi, c.gj)), w1 = ld4(blk.flux_macro_W, gidx(d, c.gi + 1, c.gj));
  const double iA = 1.0 / blk.area[gidx(d, c.gi, c.gj)], dt = step_dt(sol).cell;
  // calcQ of f^n with the macro of f^n: accumulated by the previous cell pass
  // (or the initialisation) in Q_next
  st2(blk.Q, m, ld2(blk.Q_next, m));
  const P4 wc = to_conserved(d, old);
  const P4 nw = p4(wc.s0 + (s0.s0 - s1.s0 + w0.s0 - w1.s0) * iA, wc.s1 + (s0.s1 - s1.s1 + w0.s1 - w1.s1) * iA,
                   wc.s2 + (s0.s2 - s1.s2 + w0.s2 - w1.s2) * iA, wc.s3 + (s0.s3 - s1.s3 + w0.s3 - w1.s3) * iA);
  Rcp rn, ro;
  const P4 prim = to_primary_rcp(d, nw, rn);
  ro.rho = nr_rcp(old.s0);
  ro.lam = nr_rcp(old.s3);
  st4(blk.macro, m, prim);
  st4(blk.prim_old, m, old);
  const double itau_old = inv_relax_time_rcp(d, old, ro), itau = inv_relax_time_rcp(d, prim, rn);
  const double hdt = 0.5 * dt, iden = nr_rcp(1.0 + hdt * itau);
  bc[CC_U] = prim.s1;
  bc[CC_V] = prim.s2;
  bc[CC_LAM] = prim.s3;
  bc[CC_A1] = (1.0 - hdt * itau_old) * iden;
  bc[CC_A2] = iden * iA;
  bc[CC_A3] = hdt * itau * iden;
  bc[CC_A4] = hdt * itau_old * iden;
  bc[CC_P] = prim.s0 * prim.s3;                                  // pi times the prefactor of fM
  bc[CC_KN] = (0.5 * d.K) * rn.lam;                              // K / (2 lambda)
  bc[CC_SN] = 0.8 * (1 - d.Pr) * (prim.s3 * prim.s3) * rn.rho;   // Shakhov factor
  if (P0pi > 0.0) bc[CC_LNP] = log((prim.s0 * prim.s3) / P0pi);  // mixed: ln(P / P0)
  return cfl_freq(blk, prim, c.mi, c.mj);
}
// the same for the CTA's cells, one per lane of its first warp
template <bool MIXED>
__device__ __forceinline__ void cta_cell_coefficients(const ugks_fused_block *__restrict__ B, int nb,
                                                      ugks_solve_state *__restrict__ solves, int n_cells, double *dyn,
                                                      int wstride) {
  if (threadIdx.x >= CW) return;
  CellWork c;
  if (!cell_work(B, nb, solves, (int)blockIdx.x * CW + (int)threadIdx.x, n_cells, c)) return;
  const ugks_fused_block &blk = B[c.bi];
  const double P0pi = MIXED ? blk.ref[UGKS_REF_P0] * blk.d.PI : 0.0;
  const double fq = cell_coefficients(blk, solves[blk.solve], c,
                                      dyn + (size_t)threadIdx.x * wstride + (wstride - CELL_COEF), P0pi);
  atomicMax(&solves[blk.solve].max_freq, (unsigned long long)__double_as_longlong(fq));
}

template <int MINB>
__global__ void __launch_bounds__(CW * 32, MINB * 8 / CW) cell_pass_fp64(const ugks_fused_block *__restrict__ B, int nb,
                                                                ugks_solve_state *__restrict__ solves, int n_cells,
                                                                int wstride) {
  pdl_begin();
  extern __shared__ double dyn[];
  using St = Store<double>;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  CellWork cw;
  const bool on = cell_work(B, nb, solves, (int)blockIdx.x * CW + warp, n_cells, cw);
  const ugks_fused_block &blk = B[on ? cw.bi : 0];
  const ugks_block_desc &d = blk.d;
  const int Nv = on ? d.Nv : 0, un = d.u_num, vn = d.v_num;
  const bool sep = un > 0 && un * vn == d.Nv && un + vn <= 512;
  double *Eou = dyn + (size_t)warp * wstride, *Eov = Eou + un, *Enu = Eov + vn, *Env = Enu + un;
  const double *bc = dyn + (size_t)warp * wstride + (wstride - CELL_COEF);
  const size_t base = on ? fidx(d, cw.gi, cw.gj, 0) : 0;
  const size_t sj = (size_t)d.Nv, si = (size_t)d.Nj * d.Nv, m = on ? midx(d, cw.mi, cw.mj) : 0;
  // the five rows this lane reads run D velocities (of this lane) ahead
  // through a ring of cp.async stages; a stage is refilled only after the
  // store that consumed its values, whose operands are the stage's loads
  constexpr int D = CELL_RING_F64;
  using E = double2;
  E *ring = reinterpret_cast<E *>(dyn + (size_t)CW * wstride) + (size_t)warp * (D * 5 * 32) + lane;
  const E *gf = reinterpret_cast<const E *>(blk.f), *gS = reinterpret_cast<const E *>(blk.flux_S),
          *gW = reinterpret_cast<const E *>(blk.flux_W);
  auto issue = [&](int vv, int stage) {
    if (vv < Nv) {
      const size_t k = base + vv;
      E *r = ring + stage * (5 * 32);
      cp_async<16>(r, gf + k);
      cp_async<16>(r + 32, gS + k);
      cp_async<16>(r + 64, gS + k + sj);
      cp_async<16>(r + 96, gW + k);
      cp_async<16>(r + 128, gW + k + si);
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < D; ++s) issue(lane + 32 * s, s);
  P4 old = p4(1.0, 0.0, 0.0, 1.0);
  V2 Q = v2(0.0, 0.0);
  if (on) {
    old = ld4(blk.macro, m);
    Q = ld2(blk.Q_next, m);
  }
  __syncthreads();  // every warp has its cell's old state before it is updated
  cta_cell_coefficients<false>(B, nb, solves, n_cells, dyn, wstride);
  __syncwarp();
  if (on && sep) {
    axis_exp(Eou, d.quad, un, vn, 0, old.s1, old.s3, lane, 32);
    axis_exp(Eov, d.quad, vn, 1, 1, old.s2, old.s3, lane, 32);
  }
  __syncthreads();
  if (!on) return;
  const double nU = bc[CC_U], nV = bc[CC_V], nl = bc[CC_LAM], ipi = nr_rcp(d.PI);
  const double a1 = bc[CC_A1], a2 = bc[CC_A2], kn = bc[CC_KN], sn = bc[CC_SN];
  const double cn = bc[CC_P] * ipi * bc[CC_A3], co = old.s0 * (old.s3 * ipi) * bc[CC_A4];
  if (sep) {
    axis_exp(Enu, d.quad, un, vn, 0, nU, nl, lane, 32);
    axis_exp(Env, d.quad, vn, 1, 1, nV, nl, lane, 32);
    __syncwarp();
  }
  const double ko = (0.5 * d.K) * nr_rcp(old.s3);
  const double so = 0.8 * (1 - d.Pr) * (old.s3 * old.s3) * nr_rcp(old.s0);
  const int qs = sep ? 32 / vn : 0, rs = sep ? 32 % vn : 0;
  int iu = sep ? lane / vn : 0, jv = sep ? lane % vn : 0;
  bool nan = false;
  int stage = 0;
  const double Kinv = nr_rcp(d.K);
  // moments of f^{n+1} for the next face pass, and calcQ (clKernel.c:480-543)
  // of f^{n+1} with the new macro for the next cell pass
  double mom[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  // UGKS_update (clUGKS.c:1189-1257) per velocity, regrouped:
  //   f' = f a1 + (sum of face fluxes) a2 + fEQ(new) a3 + fEQ(old) a4,
  // a3 and a4 in the Maxwellian prefactors rho lambda / pi of fEQ
#pragma unroll 1
  for (int v = lane; v < Nv; v += 32) {
    const size_t k = base + v;
    cp_async_wait<D - 1>();
    const E *r = ring + stage * (5 * 32);
    const E f = r[0], s0 = r[32], s1 = r[64], w0 = r[96], w1 = r[128];
    const V2 e = quad_at(d, v);
    const double wv = d.weight[v];
    const double ox = e.x - old.s1, oy = e.y - old.s2, o2 = fma(ox, ox, oy * oy);
    const double nx = e.x - nU, ny = e.y - nV, n2 = fma(nx, nx, ny * ny);
    double Eo, En;
    if (sep) {
      Eo = Eou[iu] * Eov[jv];
      En = Enu[iu] * Env[jv];
      jv += rs;
      iu += qs;
      if (jv >= vn) { jv -= vn; ++iu; }
    } else {
      Eo = plain_exp(-old.s3 * o2);
      En = plain_exp(-nl * n2);
    }
    // fEQ (clFunctions.c:79-86) at the old and the new macro state, scaled
    const double ho = wv * co * Eo, hn = wv * cn * En;
    const double So = so * fma(ox, Q.x, oy * Q.y), Sn = sn * fma(nx, Q.x, ny * Q.y);
    const double po = fma(2.0 * old.s3, o2, -4.0), pn = fma(2.0 * nl, n2, -4.0);
    const double eh = fma(So * po, ho, ho) + fma(Sn * pn, hn, hn);
    const double eb = ko * fma(So * (po + 2.0), ho, ho) + kn * fma(Sn * (pn + 2.0), hn, hn);
    const double flh = (s0.x - s1.x) + (w0.x - w1.x), flb = (s0.y - s1.y) + (w0.y - w1.y);
    const V2 out = v2(fma(f.x, a1, fma(flh, a2, eh)), fma(f.y, a1, fma(flb, a2, eb)));
    nan |= isnan(out.x) || isnan(out.y);
    St::store(blk.f, k, out);
    issue(v + 32 * D, stage);
    stage = stage + 1 == D ? 0 : stage + 1;
    mom[0] += out.x;
    mom[1] = fma(e.x, out.x, mom[1]);
    mom[2] = fma(e.y, out.x, mom[2]);
    mom[3] += fma(fma(e.x, e.x, e.y * e.y), out.x, out.y);
    const double t = fma(n2, out.x, out.y * Kinv);
    mom[4] = fma(nx, t, mom[4]);
    mom[5] = fma(ny, t, mom[5]);
  }
  cp_async_wait<0>();
  if (nan) atomicExch(&solves[blk.solve].status, 1);
  const double t = warp_spread_sum<6>(mom);
  constexpr int S = spread_shift<6>();
  if ((lane & ((1 << S) - 1)) == 0 && (lane >> S) < 6) {
    const int k = lane >> S;
    if (k < 4) blk.cell_mom[4 * gidx(d, cw.gi, cw.gj) + k] = k == 3 ? 0.5 * t : t;
    else blk.Q_next[2 * m + (k - 4)] = 0.5 * t;
  }
}

// ---------------------------------------------------------------------------
// dt control (ugks_sim.py:285-311, 430-446, 458-460, 491): after the cell pass
// the dt of the step, calcTimeStep + updateTimeStep, time += dt
// ---------------------------------------------------------------------------
__device__ __forceinline__ void finish_step(ugks_solve_state &x) {
  if (!x.active) return;
  const StepDt t = step_dt(x);
  if (t.retry) x.retries += 1;
  const double fq = __longlong_as_double((long long)x.max_freq);
  x.max_dt = x.CFL / fq;
  x.dt = limited_dt(t.cell, x.max_dt, x.delta_dt);
  x.time += x.dt;
  x.steps += 1;
  x.max_freq = 0ull;
  x.retry = 0;
}
// every solve, by the threads of a whole launch (the ghost pass, which needs
// none of what this writes)
__device__ __forceinline__ void finish_steps(ugks_solve_state *solves, int ns) {
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < ns; s += gridDim.x * blockDim.x) finish_step(solves[s]);
}
__global__ void dt_update(ugks_solve_state *solves, int ns) {
  pdl_begin();
  finish_steps(solves, ns);
}

// ---------------------------------------------------------------------------
// ghost pass (UGKSBlock.updateBC, ugks_block.py:621-665): one CTA per ghost
// cell of every block face
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(FT) ghost_pass(const ugks_fused_block *__restrict__ B, int nb,
                                                 ugks_solve_state *solves, int finish) {
  pdl_begin();
  __shared__ double scratch[4 * (FT / 32)];
  finish_steps(solves, finish);
  using St = Store<T>;
  const int w = blockIdx.x;
  const int bi = find_block<2>(B, nb, w);
  const ugks_fused_block &blk = B[bi];
  const ugks_block_desc &d = blk.d;
  UGKS_CHECK_ITEM(2, blk, w, solves);
  if (!solves[blk.solve].active) return;
  const int G = d.ghost, Nv = d.Nv;
  // strips in face order N, E, S, W: N/S have ni*G cells, E/W G*nj
  int lc = w - blk.ghost_begin;
  int face = 0;
  const int ns_cells = d.ni * G, ew_cells = G * d.nj;
  for (face = 0; face < 4; ++face) {
    const int c = (face == GNORTH || face == GSOUTH) ? ns_cells : ew_cells;
    if (lc < c) break;
    lc -= c;
  }
  long a, b;  // NDRange ids of the reference edge kernels
  if (face == GNORTH || face == GSOUTH) { a = lc / G; b = lc % G; }
  else { a = lc / d.nj; b = lc % d.nj; }
  long gi = a, gj = b;
  switch (face) {
    case GNORTH: gi += G; gj += d.Nj - G; break;
    case GEAST: gi += d.Ni - G; gj += G; break;
    case GSOUTH: gi += G; break;
    default: gj += G; break;
  }
  const size_t dst = fidx(d, gi, gj, 0);
  const int t = blk.bc_type[face];
  // every branch writes the ghost cell through put(), which also sums the
  // cell moments the next face pass reads
  double mom[4] = {0.0, 0.0, 0.0, 0.0};
  auto put = [&](int v, V2 x) {
    St::store(blk.f, dst + v, x);
    const V2 o = St::as_stored(x);
    const V2 e = quad_at(d, v);
    mom[0] += o.x;
    mom[1] = fma(e.x, o.x, mom[1]);
    mom[2] = fma(e.y, o.x, mom[2]);
    mom[3] += fma(fma(e.x, e.x, e.y * e.y), o.x, o.y);
  };
  // load(v) for every velocity, put in the same order as a plain loop
  auto copy = [&](auto load) {
    for (int v0 = threadIdx.x; v0 < Nv; v0 += GHOST_U * FT) {
      V2 x[GHOST_U];
#pragma unroll
      for (int u = 0; u < GHOST_U; ++u)
        if (v0 + u * FT < Nv) x[u] = load(v0 + u * FT);
#pragma unroll
      for (int u = 0; u < GHOST_U; ++u)
        if (v0 + u * FT < Nv) put(v0 + u * FT, x[u]);
    }
  };
  if (t == BC_ADJACENT || t == BC_PERIODIC) {
    // edgeExchange (clGhostRoutines.c:407-538)
    const ugks_fused_block &ob = B[blk.bc_block[face]];
    const int that = blk.bc_face[face], NI = d.Ni, NJ = d.Nj, NIB = ob.d.Ni, NJB = ob.d.Nj;
    int a1i, a1j, a2i, a2j, b1i, b1j, b2i, b2j;
    auto corners = [&](int f, int NI_, int NJ_, int &p, int &q, int &r, int &s) {
      switch (f) {
        case GNORTH: p = G; q = NJ_ - G; r = NI_ - G; s = NJ_ - G; break;
        case GEAST: p = NI_ - G; q = G; r = NI_ - G; s = NJ_ - G; break;
        case GSOUTH: p = G; q = G; r = NI_ - G; s = G; break;
        default: p = G; q = G; r = G; s = NJ_ - G; break;
      }
    };
    corners(face, NI, NJ, a1i, a1j, a2i, a2j);
    corners(that, NIB, NJB, b1i, b1j, b2i, b2j);
    const V2 A1 = ld2(blk.xy, (size_t)a1i * (NJ + 1) + a1j), A2 = ld2(blk.xy, (size_t)a2i * (NJ + 1) + a2j);
    const V2 B1 = ld2(ob.xy, (size_t)b1i * (NJB + 1) + b1j), B2 = ld2(ob.xy, (size_t)b2i * (NJB + 1) + b2j);
    const bool misalign = !(fabs(A1.x - B1.x) <= 1e-6) || !(fabs(A1.y - B1.y) <= 1e-6) ||
                          !(fabs(A2.x - B2.x) <= 1e-6) || !(fabs(A2.y - B2.y) <= 1e-6);
    int iB = (int)gi, jB = (int)gj;
    if (misalign && blk.bc_ori[face]) {
      if (face == GEAST || face == GWEST) jB = (NJ - 1) - jB;
      else iB = (NI - 1) - iB;
    }
    swap_cell_index(NI, NJ, G, face, iB, jB, that, NIB, NJB);
    if (iB < 0 || iB >= NIB || jB < 0 || jB >= NJB || ob.d.Nv != Nv) {
      // connection that does not map onto the neighbour: flag, do not read
      if (threadIdx.x == 0) atomicExch(&solves[blk.solve].status, 6);
      return;
    }
    const size_t src = ((size_t)iB * NJB + jB) * (size_t)Nv;
    const int flip = blk.bc_flip[face];
    const int32_t *perm = flip == FLIP_NS ? d.mirror_NS : (flip == FLIP_D ? d.mirror_D : d.mirror_EW);
    if (flip == NO_FLIP) copy([&](int v) { return St::load(ob.f, src + v); });
    else copy([&](int v) { return St::load(ob.f, src + perm[v]); });
  } else if (t == BC_DIFFUSE || t == BC_ADSORBING) {
    // edgeConstGrad (clGhostRoutines.c:967-1048)
    long ei0, ej0, ei1, ej1;
    double m;
    switch (face) {
      case GNORTH: ei1 = gi; ej1 = d.Nj - G - 1; ei0 = ei1; ej0 = ej1 - 1; m = (double)(gj - ej1); break;
      case GEAST: ei1 = d.Ni - G - 1; ej1 = gj; ei0 = ei1 - 1; ej0 = ej1; m = (double)(gi - ei1); break;
      case GSOUTH: ei1 = gi; ej1 = G; ei0 = ei1; ej0 = ej1 + 1; m = (double)(ej1 - gj); break;
      default: ei1 = G; ej1 = gj; ei0 = ei1 + 1; ej0 = ej1; m = (double)(ei1 - gi); break;
    }
    const size_t k0 = fidx(d, ei0, ej0, 0), k1 = fidx(d, ei1, ej1, 0);
    copy([&](int v) {
      const V2 f0 = St::load(blk.f, k0 + v), f1 = St::load(blk.f, k1 + v);
      return v2(__dadd_rn(f1.x, __dmul_rn(m, __dsub_rn(f1.x, f0.x))),
                __dadd_rn(f1.y, __dmul_rn(m, __dsub_rn(f1.y, f0.y))));
    });
  } else if (t == BC_EXTRAPOLATE_OUT || t == BC_REFLECT || t == BC_BOUNCE_BACK) {
    long si, sj;
    const int32_t *perm = nullptr;
    if (t == BC_EXTRAPOLATE_OUT) {  // edgeExtrapolate (544-597)
      switch (face) {
        case GNORTH: si = gi; sj = d.Nj - G - 1; break;
        case GEAST: si = d.Ni - G - 1; sj = gj; break;
        case GSOUTH: si = gi; sj = G; break;
        default: si = G; sj = gj; break;
      }
    } else {  // edgeMirror / edgeBounceBack (845-961)
      switch (face) {
        case GNORTH: si = gi; sj = 2 * (d.Nj - G) - gj - 1; perm = d.mirror_NS; break;
        case GEAST: si = 2 * (d.Ni - G) - gi - 1; sj = gj; perm = d.mirror_EW; break;
        case GSOUTH: si = gi; sj = 2 * G - gj - 1; perm = d.mirror_NS; break;
        default: si = 2 * G - gi - 1; sj = gj; perm = d.mirror_EW; break;
      }
      if (t == BC_BOUNCE_BACK) perm = d.mirror_D;
    }
    const size_t src = fidx(d, si, sj, 0);
    if (perm) copy([&](int v) { return St::load(blk.f, src + perm[v]); });
    else copy([&](int v) { return St::load(blk.f, src + v); });
  } else if (t == BC_CONSTANT || t == BC_INFLOW || t == BC_OUTFLOW) {
    const long ci = (face == GNORTH || face == GSOUTH) ? a : b;
    const P4 wp = ld4(blk.wall_prop, ci * 4 + face);
    P4 prim = wp;
    V2 Q = v2(0.0, 0.0);
    if (t != BC_CONSTANT) {
      // edgeInflow / edgeOutflow (664-839)
      long ei, ej, noi, noj;
      int fid;
      switch (face) {
        case GNORTH: ei = gi; ej = d.Nj - G - 1; noi = gi; noj = gj; fid = SOUTH; break;
        case GEAST: ei = d.Ni - G - 1; ej = gj; noi = gi; noj = gj; fid = WEST; break;
        case GSOUTH: ei = gi; ej = G; noi = ei; noj = ej; fid = SOUTH; break;
        default: ei = G; ej = gj; noi = ei; noj = ej; fid = WEST; break;
      }
      Q = ld2(blk.Q, midx(d, ei - G, ej - G));
      prim = ld4(blk.macro, midx(d, ei - G, ej - G));
      const V2 uv = to_local(v2(prim.s1, prim.s2), ld2(blk.normal, faceidx(d, noi, noj, fid)));
      prim.s1 = uv.x;
      prim.s2 = uv.y;
      if (t == BC_OUTFLOW) {
        prim.s3 = prim.s0 / (wp.s0 / wp.s3);
      } else {
        prim.s0 = wp.s0;
        prim.s3 = wp.s3;
      }
    }
    for (int v = threadIdx.x; v < Nv; v += FT) put(v, shakhov_eq(d, prim, Q, quad_at(d, v), v));
  }
  block_sum<4>(mom, scratch);
  if (threadIdx.x == 0) st4(blk.cell_mom, gidx(d, gi, gj), p4(mom[0], mom[1], mom[2], 0.5 * mom[3]));
}

// ---------------------------------------------------------------------------
// initial state (ugks_block.py:411-429, ugks_sim.py:88-92)
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(FT) init_cells(const ugks_fused_block *__restrict__ B, int nb,
                                                 ugks_solve_state *__restrict__ solves) {
  __shared__ double scratch[4 * (FT / 32)];
  using St = Store<T>;
  const int w = blockIdx.x;
  const int bi = find_block<1>(B, nb, w);
  const ugks_fused_block &blk = B[bi];
  const ugks_block_desc &d = blk.d;
  UGKS_CHECK_ITEM(1, blk, w, solves);
  ugks_solve_state &sol = solves[blk.solve];
  if (!sol.active) return;
  const int lc = w - blk.cell_begin;
  const long mi = lc / d.nj, mj = lc % d.nj;
  const size_t base = fidx(d, mi + d.ghost, mj + d.ghost, 0);
  // initFunctions
  P4 prim = ld4(blk.macro, midx(d, mi, mj));
  V2 Q = ld2(blk.Q, midx(d, mi, mj));
  double m[4] = {0.0, 0.0, 0.0, 0.0};
  for (int v = threadIdx.x; v < d.Nv; v += FT) {
    const V2 e = quad_at(d, v);
    const V2 f = shakhov_eq(d, prim, Q, e, v);
    St::store(blk.f, base + v, f);
    const V2 fs = St::load(blk.f, base + v);  // moments of f as stored
    m[0] += fs.x;
    m[1] += e.x * fs.x;
    m[2] += e.y * fs.x;
    m[3] += 0.5 * ((e.x * e.x + e.y * e.y) * fs.x + fs.y);
  }
  // calcMacro
  block_sum<4>(m, scratch);
  const P4 mom = p4(m[0], m[1], m[2], m[3]);
  prim = to_primary(d, mom);
  // calcQ
  double q[2] = {0.0, 0.0};
  for (int v = threadIdx.x; v < d.Nv; v += FT) {
    const V2 f = St::load(blk.f, base + v);
    const V2 e = quad_at(d, v);
    const double cx = e.x - prim.s1, cy = e.y - prim.s2, c2 = cx * cx + cy * cy;
    const double t = c2 * f.x + f.y / d.K;
    q[0] += 0.5 * (cx * t);
    q[1] += 0.5 * (cy * t);
  }
  block_sum<2>(q, scratch);
  if (threadIdx.x == 0) {
    st4(blk.macro, midx(d, mi, mj), prim);
    st4(blk.cell_mom, gidx(d, mi + d.ghost, mj + d.ghost), mom);
    st2(blk.Q, midx(d, mi, mj), v2(q[0], q[1]));
    st2(blk.Q_next, midx(d, mi, mj), v2(q[0], q[1]));
    const double fq = cfl_freq(blk, prim, mi, mj);
    atomicMax(&sol.max_freq, (unsigned long long)__double_as_longlong(fq));
  }
}

// restart from saved f, macro and Q (initFunctions with a restart file and
// f present, ugks_block.py:274-300, 347-349): f and macro stay as loaded; the
// fused path's own per-cell state is rebuilt from them (the moments of f for
// the face pass, calcQ of f with the macro for the next cell pass) and the CFL
// frequency of every cell is taken as at start-up (calcTimeStep)
template <typename T>
__global__ void __launch_bounds__(FT) restart_cells(const ugks_fused_block *__restrict__ B, int nb,
                                                    ugks_solve_state *__restrict__ solves) {
  __shared__ double scratch[6 * (FT / 32)];
  using St = Store<T>;
  const int w = blockIdx.x;
  const int bi = find_block<1>(B, nb, w);
  const ugks_fused_block &blk = B[bi];
  const ugks_block_desc &d = blk.d;
  UGKS_CHECK_ITEM(1, blk, w, solves);
  ugks_solve_state &sol = solves[blk.solve];
  if (!sol.active) return;
  const int lc = w - blk.cell_begin;
  const long mi = lc / d.nj, mj = lc % d.nj;
  const size_t base = fidx(d, mi + d.ghost, mj + d.ghost, 0);
  const P4 prim = ld4(blk.macro, midx(d, mi, mj));
  const double Kinv = 1.0 / d.K;
  double m[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  for (int v = threadIdx.x; v < d.Nv; v += FT) {
    const V2 f = St::load(blk.f, base + v);
    const V2 e = quad_at(d, v);
    m[0] += f.x;
    m[1] = fma(e.x, f.x, m[1]);
    m[2] = fma(e.y, f.x, m[2]);
    m[3] += fma(fma(e.x, e.x, e.y * e.y), f.x, f.y);
    const double cx = e.x - prim.s1, cy = e.y - prim.s2;
    const double t = fma(fma(cx, cx, cy * cy), f.x, f.y * Kinv);
    m[4] = fma(cx, t, m[4]);
    m[5] = fma(cy, t, m[5]);
  }
  block_sum<6>(m, scratch);
  if (threadIdx.x == 0) {
    st4(blk.cell_mom, gidx(d, mi + d.ghost, mj + d.ghost), p4(m[0], m[1], m[2], 0.5 * m[3]));
    st2(blk.Q_next, midx(d, mi, mj), v2(0.5 * m[4], 0.5 * m[5]));
    const double fq = cfl_freq(blk, prim, mi, mj);
    atomicMax(&sol.max_freq, (unsigned long long)__double_as_longlong(fq));
  }
}

// paraBC (clKernel.c:141-218) for constant wall values, every block
__global__ void init_walls(const ugks_fused_block *B, int nb) {
  const ugks_fused_block &blk = B[blockIdx.x];
  const ugks_block_desc &d = blk.d;
  const int wl = max(d.ni, d.nj);
  for (int ci = threadIdx.x; ci < wl; ci += blockDim.x)
    for (int f = 0; f < 4; ++f) {
      const bool ns = (f == GNORTH || f == GSOUTH);
      if (ns ? !(ci < d.ni) : !(ci < d.nj)) continue;
      const double l = (d.wall_P[f] != -1) ? d.wall_P[f] / d.wall_D[f] : d.wall_T[f];
      st4(blk.wall_prop, ci * 4 + f, p4(d.wall_D[f], d.wall_U[f], d.wall_V[f], l));
    }
}

// calcTimeStep + updateTimeStep(limit=False) at start-up
__global__ void dt_init(ugks_solve_state *solves, int ns) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ns) return;
  ugks_solve_state &x = solves[s];
  if (!x.active) return;
  x.max_dt = x.CFL / __longlong_as_double((long long)x.max_freq);
  if (x.dt != x.max_dt) x.dt = x.max_dt;
  x.max_freq = 0ull;
  x.retry = 0;
}

// the mixed-precision (FP32 deviation) kernels
#include "ugks_delta.cuh"

// the ghost update of every block of the table, and with finish = the number of
// solves the end of their step
template <typename T>
void launch_ghosts(const ugks_fused_block *B, int nb, const ugks_fused_sizes *z, ugks_solve_state *solves,
                   int finish, StepStream st) {
  if (!z->n_ghost) {
    if (finish) launch(dt_update, (finish + 127) / 128, 128, 0, st, solves, finish);
    return;
  }
  launch(std::is_same<T, float>::value ? ghost_pass_delta : ghost_pass<double>, z->n_ghost, FT, 0, st, B, nb, solves, finish);
}

template <typename T>
int init_impl(const ugks_fused_block *B, int nb, const ugks_fused_sizes *z, ugks_solve_state *solves,
              int ns, void *stream) {
  cudaStream_t st = S(stream);
  init_walls<<<nb, 128, 0, st>>>(B, nb);
  if (z->n_faces) face_geometry<<<(z->n_faces + 127) / 128, 128, 0, st>>>(B, nb, z->n_faces);
  if (z->n_cells) {
    if (std::is_same<T, float>::value) setup_cells_delta<true><<<z->n_cells, FT, 0, st>>>(B, nb, solves);
    else init_cells<double><<<z->n_cells, FT, 0, st>>>(B, nb, solves);
  }
  dt_init<<<(ns + 127) / 128, 128, 0, st>>>(solves, ns);
  launch_ghosts<T>(B, nb, z, solves, 0, {st});
  return launch_status();
}

template <typename T>
int restart_impl(const ugks_fused_block *B, int nb, const ugks_fused_sizes *z, ugks_solve_state *solves,
                 int ns, void *stream) {
  cudaStream_t st = S(stream);
  init_walls<<<nb, 128, 0, st>>>(B, nb);
  if (z->n_faces) face_geometry<<<(z->n_faces + 127) / 128, 128, 0, st>>>(B, nb, z->n_faces);
  if (z->n_cells) {
    if (std::is_same<T, float>::value) setup_cells_delta<false><<<z->n_cells, FT, 0, st>>>(B, nb, solves);
    else restart_cells<double><<<z->n_cells, FT, 0, st>>>(B, nb, solves);
  }
  dt_init<<<(ns + 127) / 128, 128, 0, st>>>(solves, ns);
  launch_ghosts<T>(B, nb, z, solves, 0, {st});
  return launch_status();
}

template <typename K>
cudaError_t allow_smem(K kernel) {
  return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}
template <int V>
cudaError_t set_face_shape() {
  constexpr int W = FaceShape<V>::wpc, M = FaceShape<V>::minb;
  cudaError_t r[3] = {allow_smem(face_pass_fp64<0, W, M>), allow_smem(face_pass_fp64<1, W, M>),
                      allow_smem(face_pass_fp64<3, W, M>)};
  for (cudaError_t e : r)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}
template <typename T>
cudaError_t set_wall_attributes() {
  if constexpr (std::is_same<T, double>::value) {
    cudaError_t r[4] = {set_face_shape<1>(), set_face_shape<2>(), set_face_shape<3>(), set_face_shape<4>()};
    for (cudaError_t e : r)
      if (e != cudaSuccess) return e;
  }
  if constexpr (std::is_same<T, float>::value) {
    cudaError_t r[3] = {allow_smem(wall_pass_delta), allow_smem(wall_retry_delta<WALL_NT>),
                        allow_smem(wall_retry_delta<WIDE_NT>)};
    for (cudaError_t e : r)
      if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
template <int V>
cudaError_t set_moments_shape() {
  constexpr int W = MomentsShape<V>::wpc, M = MomentsShape<V>::minb;
  cudaError_t r[3] = {allow_smem(face_moments_warp<0, W, M>), allow_smem(face_moments_warp<1, W, M>),
                      allow_smem(face_moments_warp<3, W, M>)};
  for (cudaError_t e : r)
    if (e != cudaSuccess) return e;
  return cudaSuccess;
}
template <typename T>
cudaError_t set_flux_attributes() {
  if constexpr (std::is_same<T, float>::value) {
    cudaError_t r[4] = {set_moments_shape<1>(), set_moments_shape<2>(), set_moments_shape<3>(), set_moments_shape<4>()};
    for (cudaError_t x : r)
      if (x != cudaSuccess) return x;
    cudaError_t e = cudaFuncSetAttribute(face_flux_tma<FLUX_WPC, FLUX_TMA_MINB>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(face_flux_tma<FLUX_WPC, FLUX_TMA_MINB>, cudaFuncAttributePreferredSharedMemoryCarveout,
                               cudaSharedmemCarveoutMaxShared);
    return e;
  }
  return cudaSuccess;
}
template <typename T, int MINB>
cudaError_t set_cell_attributes() {
  if (std::is_same<T, float>::value)
    return cudaFuncSetAttribute(cell_pass_delta<MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
  return cudaFuncSetAttribute(cell_pass_fp64<MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
}

// Kernel attributes (the dynamic shared memory above 48 KB that the face and
// cell passes of large velocity grids need) hold per device: they are set
// once for each device a step runs on, with that device current.
constexpr int kMaxDevices = 64;

// A large mixed step's wall launch runs on a side stream beside the moments sweep
// (it needs only this step's f and writes only wall faces): a fork and a join by
// events, which stream capture turns into graph edges.  One side stream per
// device, created with the device's kernel attributes (before any capture:
// ugks_prepare); `lock` keeps the record-wait pairs of concurrent host threads
// from interleaving.
struct WallStream {
  cudaStream_t s = nullptr;
  cudaEvent_t fork = nullptr, join = nullptr;
  std::mutex lock;
};
inline WallStream &wall_stream(int dev) {
  static WallStream ws[kMaxDevices];
  return ws[dev];
}
inline cudaError_t make_wall_stream(int dev) {
  WallStream &w = wall_stream(dev);
  if (w.s) return cudaSuccess;
  cudaError_t e = cudaStreamCreateWithFlags(&w.s, cudaStreamNonBlocking);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&w.fork, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&w.join, cudaEventDisableTiming);
  return e;
}

template <typename T>
cudaError_t set_step_attributes() {
  static std::mutex lock;
  static bool done[kMaxDevices] = {false};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> guard(lock);
  if (done[dev]) return cudaSuccess;
  cudaError_t r[4] = {set_cell_attributes<T, 2>(), set_cell_attributes<T, 3>(), set_wall_attributes<T>(),
                      set_flux_attributes<T>()};
  for (cudaError_t x : r)
    if (x != cudaSuccess) return x;
  if (std::is_same<T, float>::value) {
    e = make_wall_stream(dev);
    if (e != cudaSuccess) return e;
  }
  done[dev] = true;
  return cudaSuccess;
}

// The largest velocity grid a step accepts, as bytes against 200 KB.  Mixed: a wall
// face's values, which its CTA holds in shared memory.  FP64: the bound (6400
// velocities) of a face pass that held a face's values and slopes there; nothing of
// that size is left in shared memory, and grids above it stay refused as before.
template <typename T>
inline size_t face_limit_bytes(int max_nv, int max_axes) {
  if (std::is_same<T, float>::value) return delta_wall_smem(max_nv);
  return 4 * sizeof(double) * (size_t)max_nv + sizeof(double) * (size_t)max_axes;
}

// doubles of shared memory per FP64 face warp beside its ring: the face record
// and the axis factors (of grids with up to 512 axis nodes; larger ones go without)
inline int face_stride(int max_axes) { return FACE_TAB + ((std::min(max_axes, 512) + 1) & ~1); }
// the mixed kernels keep axis tables of any tensor grid
inline int mixed_axes(const ugks_fused_sizes *z) {
  int n = z->max_axes;
  for (int k = 0; k < z->n_segments && k < UGKS_MAX_FACE_SEGMENTS; ++k) n = std::max(n, (int)z->seg_max_axes[k]);
  return n;
}
template <int FM, int WPC>
size_t face_smem(int wstride) {
  return (size_t)WPC * (wstride * sizeof(double) + face_ring_elems<FM>() * sizeof(double2));
}

// the FP64 face pass of one segment (one flux method) in launch shape v; the
// first segment's launch takes the wall faces of the whole table with it
template <int WPC, int MINB>
void launch_faces_shape(const ugks_fused_block *B, int nb, ugks_solve_state *solves, int method, int n_wall, WallKind kind, int first,
                        int count, int axes, int chained, StepStream st) {
  const int ws = face_stride(axes);
  const unsigned g = (unsigned)(n_wall + (count + WPC - 1) / WPC + chained), t = WPC * 32;
  switch (method) {
    case 0: launch(face_pass_fp64<0, WPC, MINB>, g, t, face_smem<0, WPC>(ws), st, B, nb, solves, n_wall, kind, first, count, ws, chained); break;
    case 1: launch(face_pass_fp64<1, WPC, MINB>, g, t, face_smem<1, WPC>(ws), st, B, nb, solves, n_wall, kind, first, count, ws, chained); break;
    case 3: launch(face_pass_fp64<3, WPC, MINB>, g, t, face_smem<3, WPC>(ws), st, B, nb, solves, n_wall, kind, first, count, ws, chained); break;
    default: break;
  }
}
inline void launch_faces(int v, const ugks_fused_block *B, int nb, ugks_solve_state *solves, int method, int n_wall,
                         WallKind kind, int first, int count, int axes, int chained, StepStream st) {
  switch (v) {
    case 2: launch_faces_shape<FaceShape<2>::wpc, FaceShape<2>::minb>(B, nb, solves, method, n_wall, kind, first, count, axes, chained, st); break;
    case 3: launch_faces_shape<FaceShape<3>::wpc, FaceShape<3>::minb>(B, nb, solves, method, n_wall, kind, first, count, axes, chained, st); break;
    case 4: launch_faces_shape<FaceShape<4>::wpc, FaceShape<4>::minb>(B, nb, solves, method, n_wall, kind, first, count, axes, chained, st); break;
    default: launch_faces_shape<FaceShape<1>::wpc, FaceShape<1>::minb>(B, nb, solves, method, n_wall, kind, first, count, axes, chained, st); break;
  }
}

// the walls redone after a dt change (rare)
template <typename T>
void launch_retry(const ugks_fused_block *B, int nb, const ugks_fused_sizes *z, ugks_solve_state *solves, int ns,
                  StepStream st) {
  if (!z->n_wall) return;
  const bool wide = has_cl_walls(z);
  const unsigned g = retry_grid(ns), nt = wide ? WIDE_NT : WALL_NT;
  if constexpr (std::is_same<T, float>::value)
    launch(wide ? wall_retry_delta<WIDE_NT> : wall_retry_delta<WALL_NT>, g, nt, delta_wall_smem(z->max_nv), st, B, nb, solves, ns);
  else
    launch(wide ? wall_retry_fp64<WIDE_NT> : wall_retry_fp64<WALL_NT>, g, nt, 0, st, B, nb, solves, ns);
}

// the mixed moments sweep of one segment, in launch shape v (ugks_fused_sizes.seg_variant)
template <int WPC, int MINB>
void launch_moments_shape(const ugks_fused_block *B, int nb, ugks_solve_state *solves, int method, int first,
                          int count, int axes, int chained, StepStream st) {
  const int ws = delta_moments_stride(axes);
  const unsigned g = (unsigned)((count + WPC - 1) / WPC + chained);
  const size_t sm = (size_t)WPC * ws * sizeof(double);
  switch (method) {
    case 0: launch(face_moments_warp<0, WPC, MINB>, g, WPC * 32, sm + WPC * delta_ring_bytes<0>(), st, B, nb, solves, first, count, ws, chained); break;
    case 1: launch(face_moments_warp<1, WPC, MINB>, g, WPC * 32, sm + WPC * delta_ring_bytes<1>(), st, B, nb, solves, first, count, ws, chained); break;
    case 3: launch(face_moments_warp<3, WPC, MINB>, g, WPC * 32, sm + WPC * delta_ring_bytes<3>(), st, B, nb, solves, first, count, ws, chained); break;
    default: break;
  }
}
inline void launch_moments(int v, const ugks_fused_block *B, int nb, ugks_solve_state *solves, int method,
                           int first, int count, int axes, int chained, StepStream st) {
  switch (v) {
    case 2: launch_moments_shape<MomentsShape<2>::wpc, MomentsShape<2>::minb>(B, nb, solves, method, first, count, axes, chained, st); break;
    case 3: launch_moments_shape<MomentsShape<3>::wpc, MomentsShape<3>::minb>(B, nb, solves, method, first, count, axes, chained, st); break;
    case 4: launch_moments_shape<MomentsShape<4>::wpc, MomentsShape<4>::minb>(B, nb, solves, method, first, count, axes, chained, st); break;
    default: launch_moments_shape<MomentsShape<1>::wpc, MomentsShape<1>::minb>(B, nb, solves, method, first, count, axes, chained, st); break;
  }
}

// NVTX range over a phase's launches on the host timeline (a profiler shows
// them beside the kernels; without one attached a range costs a few ns)
struct NvtxRange {
  explicit NvtxRange(const char *name) { nvtxRangePushA(name); }
  ~NvtxRange() { nvtxRangePop(); }
  NvtxRange(const NvtxRange &) = delete;
  NvtxRange &operator=(const NvtxRange &) = delete;
};

// The line between the two ways to launch a step.  A boundary saves about 2 us
// whatever the work; the shared split costs a share of the passes it fits less
// well.  Mixed: by work, faces times velocities.  FP64: up to as many cells as the
// cell pass holds in one wave of the 3 CTAs an SM has with that split (4 with its
// own).  Step in us without and with programmatic launches, square cavities (cells
// a side, velocities), vanLeer: mixed 24, 17^2 (0.4 M) 52.5 and 42.5; 56, 25^2 (4.1 M)
// 117 and 104; 80, 25^2 (8.2 M) 193 and 184; 62, 33^2 (8.6 M) 183 and 180; 88, 33^2
// (17 M) 304 and 315.  FP64 24, 17^2 46.3 and 38.1; 40, 25^2 93 and 86; 36, 41^2 196
// and 193; 44, 33^2 149 and 173; 63, 33^2 279 and 301.  Tables of small cavities (17^2
// velocities, two limiters): mixed 8 of 24 (2.9 M) 133 and 131, 16 of 24 (5.8 M) 245
// and 252, 64 of 12 (6.3 M) 304 and 311; FP64 4 of 12 54 and 47, 4 of 24 91.7 and
// 92.2, 64 of 12 387 and 399.
template <typename T>
inline StepStream step_stream(cudaStream_t st, const ugks_fused_sizes *z) {
  if (std::is_same<T, float>::value) return {st, (double)z->n_faces * z->max_nv <= 1e7 ? 70 : 0};
  return {st, z->n_cells <= 3 * 148 * CW ? 50 : 0};
}

template <typename T>
int step_impl(const ugks_fused_block *B, int nb, const ugks_fused_sizes *z, ugks_solve_state *solves,
              int ns, void *stream, void *const *events = nullptr) {
  const StepStream st = step_stream<T>(S(stream), z);
  // cell pass: the axis factor tables of the old and new macro state
  constexpr bool mixed = std::is_same<T, float>::value;
  // doubles of shared memory per cell warp
  const int axes = mixed ? mixed_axes(z) : z->max_axes;
  const int cstride = mixed ? delta_cell_stride(axes) : 2 * axes + CELL_COEF;
  const size_t csmem = (size_t)CW * cstride * sizeof(double) + (mixed ? (size_t)CW * CELL_RING_F32 * 160 * 16 : (size_t)CW * cell_ring_bytes());
  const cudaError_t attr = set_step_attributes<T>();
  if (attr != cudaSuccess) return -(int)attr;
  const size_t fsmem = mixed ? FLUX_WPC * flux_tma_warp_bytes(axes) : 0;
  if (face_limit_bytes<T>(z->max_nv, z->max_axes) > 200 * 1024 || csmem > 200 * 1024 || fsmem > 200 * 1024)
    return -(int)cudaErrorInvalidValue;
  auto mark = [&](int k) {
    if (events && events[k]) cudaEventRecord(reinterpret_cast<cudaEvent_t>(events[k]), st.st);
  };
  // NVTX: the step, and within it the face, cell and ghost phases
  NvtxRange step_range(mixed ? "ugks step (mixed)" : "ugks step (fp64)");
  std::optional<NvtxRange> phase;
  phase.emplace("ugks face pass");
  mark(0);
  // the launches of the face pass depend only on the step before: all but the
  // first are chained.  Mixed: the wall faces first, beside which the moments run,
  // chained or, on large tables, with the wall faces on the side stream
  int chained = 0;
  WallStream *ws = nullptr;
  std::unique_lock<std::mutex> ws_guard;
  if (mixed && z->n_wall) {
    StepStream to = st;
    if (!st.carve) {
      int dev = 0;
      const cudaError_t e = cudaGetDevice(&dev);
      if (e != cudaSuccess) return -(int)e;
      ws = &wall_stream(dev);
      ws_guard = std::unique_lock<std::mutex>(ws->lock);
      cudaEventRecord(ws->fork, st.st);
      cudaStreamWaitEvent(ws->s, ws->fork, 0);
      to = {ws->s};
    }
    launch(wall_pass_delta, z->n_wall, WALL_NT, delta_wall_smem(z->max_nv), to, B, nb, solves);
    if (ws) cudaEventRecord(ws->join, ws->s);
    chained = st.carve > 0;
  }
  int walls = z->n_wall;
  const bool cl_walls = !mixed && walls && has_cl_walls(z);
  if (cl_walls) {
    launch(cl_wall_pass_fp64, walls, WIDE_NT, 0, st, B, nb, solves);
    chained = 1;
  }
  for (int k = 0; k < z->n_segments && k < UGKS_MAX_FACE_SEGMENTS; ++k) {
    if (z->seg_count[k] <= 0 || z->seg_method[k] == UGKS_SEG_CL_WALLS) continue;
    int v = z->seg_variant[k];
    StepStream to = st;
    to.chained = chained;
    const int m = z->seg_method[k], b0 = z->seg_begin[k], n = z->seg_count[k];
    if (v <= 0 || v > 4) v = 1;
    if constexpr (mixed) {
      launch_moments(v, B, nb, solves, m, b0, n, z->seg_max_axes[k], chained, to);
    } else {
      launch_faces(v, B, nb, solves, m, walls, cl_walls ? WALL_OTHER : WALL_ANY, b0, n, z->seg_max_axes[k], chained, to);
      walls = 0;
    }
    chained = 1;
  }
  if (ws) {
    cudaStreamWaitEvent(st.st, ws->join, 0);
    ws_guard.unlock();
  }
  // mixed: the interior faces' coefficient and flux launches take the dt of the
  // final flux pass, and the events bracket all of the face pass
  if (!mixed) {
    mark(1);
    mark(2);
  }
  launch_retry<T>(B, nb, z, solves, ns, st);
  if (mixed && z->n_faces) {
    launch(face_coef_delta, (unsigned)((2l * z->n_faces + COEF_NT - 1) / COEF_NT), COEF_NT, 0, st, B, nb, solves, z->n_faces);
    const int wb = (int)flux_tma_warp_bytes(axes);
    launch(face_flux_tma<FLUX_WPC, FLUX_TMA_MINB>, (unsigned)((z->n_faces + FLUX_WPC - 1) / FLUX_WPC), FLUX_WPC * 32,
           fsmem, st, B, nb, solves, z->n_faces, wb);
  }
  if (mixed) {
    mark(1);
    mark(2);
  }
  mark(3);
  phase.reset();
  mark(4);
  phase.emplace("ugks cell pass");
  if (z->n_cells) {
    // cell_variant: 0 the default register budget, 2 or 3 times 8 warps per SM
    const unsigned cg = (unsigned)((z->n_cells + CW - 1) / CW);
    const int cv = z->cell_variant == 2 || z->cell_variant == 3 ? z->cell_variant : CELL_MINB;
    if (mixed) launch(cv == 3 ? cell_pass_delta<3> : cell_pass_delta<2>, cg, CW * 32, csmem, st, B, nb, solves, z->n_cells, cstride);
    else launch(cv == 3 ? cell_pass_fp64<3> : cell_pass_fp64<2>, cg, CW * 32, csmem, st, B, nb, solves, z->n_cells, cstride);
  }
  mark(5);
  phase.reset();
  mark(6);
  phase.emplace("ugks ghost pass");
  launch_ghosts<T>(B, nb, z, solves, ns, st);
  mark(7);
  return launch_status();
}

// the stop rule of an active solve (ugks_stop_check)
__device__ __forceinline__ void stop_rule(ugks_solve_state &x) {
  int why = 0;
  if (x.status != 0) why = UGKS_STOP_ERROR;
  else if (x.stop_residual > 0.0 && x.steps >= x.stop_after && x.residual[0] < x.stop_residual)
    why = UGKS_STOP_CONVERGED;
  else if (x.stop_steps > 0 && x.steps >= x.stop_steps) why = UGKS_STOP_STEPS;
  if (why) {
    x.stopped = why;
    x.active = 0;
  }
}

// residual (getResidual, clUGKS.c:1259-1277, and ugks_block.py:1316-1327): one CTA
// per solve walks its blocks, and with STOP applies the solve's stop rule.  The
// sums are short (a few cells per thread), so the CTA is as wide as it can be: with
// 128 threads six solves of up to 48 x 48 cells took 17 us, with 1024 and the stop
// rule in it 7.
constexpr int RES_NT = 1024;
template <bool STOP>
__global__ void __launch_bounds__(RES_NT) residual_kernel(const ugks_fused_block *B, int nb, ugks_solve_state *solves,
                                                          int ns) {
  pdl_begin();
  __shared__ double scratch[8 * (RES_NT / 32)];
  const int s = blockIdx.x;
  if (s >= ns || !solves[s].active) return;  // a stopped solve keeps its last residual
  double r[4] = {0.0, 0.0, 0.0, 0.0};
  int n = 0;
  for (int b = 0; b < nb; ++b) {
    if (B[b].solve != s) continue;
    const ugks_fused_block &blk = B[b];
    const int cells = blk.d.ni * blk.d.nj;
    double a[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int c = threadIdx.x; c < cells; c += RES_NT) {
      const P4 p = ld4(blk.macro, c), o = ld4(blk.prim_old, c);
      a[0] += (p.s0 - o.s0) * (p.s0 - o.s0);
      a[1] += (p.s1 - o.s1) * (p.s1 - o.s1);
      a[2] += (p.s2 - o.s2) * (p.s2 - o.s2);
      a[3] += (p.s3 - o.s3) * (p.s3 - o.s3);
      a[4] += fabs(p.s0);
      a[5] += fabs(p.s1);
      a[6] += fabs(p.s2);
      a[7] += fabs(p.s3);
    }
    block_sum_spread_to0<8>(a, scratch);
    if (threadIdx.x == 0)
      for (int k = 0; k < 4; ++k) {
        const double v = sqrt((double)cells * a[k]) / (a[4 + k] + DBL_MIN);
        r[k] += v <= 0.0 ? 1.0 : v;
      }
    ++n;
  }
  if (threadIdx.x == 0) {
    for (int k = 0; k < 4; ++k) solves[s].residual[k] = n ? r[k] / n : 0.0;
    if (STOP) stop_rule(solves[s]);
  }
}

// The bounded wait of the face pass's bulk copies, exercised on its own: a
// warp arms an mbarrier for 512 bytes and copies them from `src` (global, 16-
// byte aligned), or, with src null, never does; it then waits at most `polls`
// times and writes 0 when the copy completed, STATUS_COPY_TIMEOUT when the
// wait ran out (what the face pass writes into a solve's status)
__global__ void copy_wait_check(const float4 *src, unsigned polls, int *status) {
  __shared__ __align__(128) float4 buf[32];
  __shared__ __align__(8) uint64_t bar;
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
    mbar_arrive_expect_tx(&bar, 512u);
    if (src) bulk_g2s(buf, src, 512u, &bar);
  }
  __syncwarp();
  const bool ok = __all_sync(0xffffffffu, mbar_wait(&bar, 0u, polls));
  // the copied values read back (a lane's float4 must equal the source's)
  const bool same = ok && src ? __all_sync(0xffffffffu, buf[lane].x == src[lane].x && buf[lane].w == src[lane].w)
                              : true;
  if (lane == 0) *status = !ok ? STATUS_COPY_TIMEOUT : (same ? 0 : -1);
}

// the reciprocal of the face and cell coefficients, on its own (ugks_check_reciprocal)
__global__ void reciprocal_check(const double *x, int64_t n, double *y) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k < n) y[k] = nr_rcp(x[k]);
}

// and the relaxation rate of gas at density 1 (ugks_check_relax_rate)
__global__ void relax_rate_check(const ugks_block_desc d, const double *lambda, int64_t n, double *rate) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const Rcp rc = {1.0, nr_rcp(lambda[k])};
  rate[k] = inv_relax_time_rcp(d, p4(1.0, 0.0, 0.0, lambda[k]), rc);
}

// the stop rule of every active solve (ugks_stop_check)
__global__ void stop_check(ugks_solve_state *solves, int ns) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= ns) return;
  if (solves[s].active) stop_rule(solves[s]);
}

}  // namespace

extern "C" {

int ugks_step_fp64(const ugks_fused_block *blocks_dev, int nblocks, const ugks_fused_sizes *sizes,
                   ugks_solve_state *solves_dev, int nsolves, void *stream) {
  return step_impl<double>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream);
}
int ugks_step_mixed(const ugks_fused_block *blocks_dev, int nblocks, const ugks_fused_sizes *sizes,
                    ugks_solve_state *solves_dev, int nsolves, void *stream) {
  return step_impl<float>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream);
}
int ugks_step_profiled(int mixed, const ugks_fused_block *blocks_dev, int nblocks,
                       const ugks_fused_sizes *sizes, ugks_solve_state *solves_dev, int nsolves,
                       void *const *events, void *stream) {
  return mixed ? step_impl<float>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream, events)
               : step_impl<double>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream, events);
}
int ugks_step_launches(const ugks_fused_sizes *z, int mixed) {
  int n = 0;
  if (mixed && z->n_faces) n += 2;  // the mixed face pass's coefficient and flux launches
  if (mixed && z->n_wall) n += 1;   // and its wall launch
  for (int k = 0; k < z->n_segments && k < UGKS_MAX_FACE_SEGMENTS; ++k)
    n += z->seg_count[k] > 0 && !(mixed && z->seg_method[k] == UGKS_SEG_CL_WALLS) ? 1 : 0;
  n += z->n_wall ? 1 : 0;  // retry pass
  n += z->n_cells ? 1 : 0;
  n += 1;                                                          // ghost pass (or the dt update alone)
  return n;
}

int ugks_residual(const ugks_fused_block *blocks_dev, int nblocks, ugks_solve_state *solves_dev,
                  int nsolves, void *stream) {
  if (nsolves <= 0) return 0;
  launch(residual_kernel<false>, nsolves, RES_NT, 0, {S(stream)}, blocks_dev, nblocks, solves_dev, nsolves);
  return launch_status();
}

int ugks_stop_check(ugks_solve_state *solves_dev, int nsolves, void *stream) {
  if (nsolves <= 0) return 0;
  stop_check<<<(nsolves + 127) / 128, 128, 0, S(stream)>>>(solves_dev, nsolves);
  return launch_status();
}

int ugks_serve_steps(int mixed, const ugks_fused_block *blocks_dev, int nblocks, const ugks_fused_sizes *sizes,
                     ugks_solve_state *solves_dev, int nsolves, int nsteps, void *stream) {
  const StepStream st = mixed ? step_stream<float>(S(stream), sizes) : step_stream<double>(S(stream), sizes);
  for (int k = 0; k < nsteps; ++k) {
    int rc = mixed ? step_impl<float>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream)
                   : step_impl<double>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream);
    if (rc == 0 && nsolves > 0) {
      launch(residual_kernel<true>, nsolves, RES_NT, 0, st, blocks_dev, nblocks, solves_dev, nsolves);
      rc = launch_status();
    }
    if (rc != 0) return rc;
  }
  return 0;
}

int ugks_check_copy_wait(const void *src_dev, unsigned polls, int *status_dev, void *stream) {
  copy_wait_check<<<1, 32, 0, S(stream)>>>(reinterpret_cast<const float4 *>(src_dev), polls, status_dev);
  return launch_status();
}

int ugks_check_reciprocal(const double *x_dev, int64_t n, double *y_dev, void *stream) {
  if (n <= 0) return 0;
  reciprocal_check<<<(unsigned)((n + 255) / 256), 256, 0, S(stream)>>>(x_dev, n, y_dev);
  return launch_status();
}

int ugks_check_relax_rate(const ugks_block_desc *d, const double *lambda_dev, int64_t n, double *rate_dev, void *stream) {
  if (n <= 0) return 0;
  relax_rate_check<<<(unsigned)((n + 255) / 256), 256, 0, S(stream)>>>(*d, lambda_dev, n, rate_dev);
  return launch_status();
}

int ugks_prepare(int mixed) {
  const cudaError_t e = mixed ? set_step_attributes<float>() : set_step_attributes<double>();
  return e == cudaSuccess ? 0 : -(int)e;
}

// A block the fused kernels can index safely: sizes consistent with the
// ghost layers the flux method's stencil needs, the arrays every pass
// touches present, block connections inside the table and on a face of the
// same extent.  (A corrupted entry would otherwise send a kernel outside its
// arrays: the table is rejected on the host before any launch.)
static bool block_valid(const ugks_fused_block *blocks, int nblocks, int b) {
  const ugks_fused_block &x = blocks[b];
  const ugks_block_desc &d = x.d;
  const int need = d.flux_method == 1 ? 3 : 2;  // stencil half-width of WENO5 / vanLeer, minmod
  if (d.ni <= 0 || d.nj <= 0 || d.Nv <= 0 || d.ghost < need) return false;
  if (d.Ni != d.ni + 2 * d.ghost || d.Nj != d.nj + 2 * d.ghost) return false;
  if (d.u_num < 0 || d.v_num < 0 || (d.u_num > 0 && (int64_t)d.u_num * d.v_num != d.Nv)) return false;
  if (!d.quad || !d.weight || !d.mirror_NS || !d.mirror_EW || !d.mirror_D) return false;
  if (!x.f || !x.flux_S || !x.flux_W || !x.flux_macro_S || !x.flux_macro_W || !x.macro || !x.Q || !x.prim_old ||
      !x.area || !x.centre || !x.mid_side || !x.normal || !x.side_length || !x.xy || !x.cell_mom || !x.Q_next ||
      !x.face_geo || !x.wall_prop || !x.wall_cover || !x.wall_fluxes || !x.wall_dist)
    return false;
  for (int f = 0; f < 4; ++f) {
    if (x.bc_type[f] < BC_ADJACENT || x.bc_type[f] > BC_BOUNCE_BACK) return false;
    if (x.bc_type[f] == BC_ADJACENT || x.bc_type[f] == BC_PERIODIC) {
      const int o = x.bc_block[f], of = x.bc_face[f];
      if (o < 0 || o >= nblocks || of < 0 || of > 3) return false;
      const ugks_block_desc &od = blocks[o].d;
      const int n_here = (f == GNORTH || f == GSOUTH) ? d.ni : d.nj;
      const int n_there = (of == GNORTH || of == GSOUTH) ? od.ni : od.nj;
      if (n_here != n_there || od.Nv != d.Nv || od.ghost != d.ghost || blocks[o].solve != x.solve) return false;
    }
  }
  return true;
}

int ugks_fused_layout(ugks_fused_block *blocks, int nblocks, ugks_fused_sizes *z) {
  if (nblocks < 0 || (nblocks > 0 && !blocks) || !z) return -3;
  for (int b = 0; b < nblocks; ++b)
    if (!block_valid(blocks, nblocks, b)) return -3;
  int64_t f = 0, c = 0, g = 0, wl = 0;
  int32_t max_nv = 0, max_axes = 0;
  int64_t fb[4] = {0, 0, 0, 0}, fc[4] = {0, 0, 0, 0};
  struct Run {
    int method, nv, max_nv, axes;
    int64_t begin, count;
  };
  std::vector<Run> runs;
  int last_method = -1, seen = 0, last_solve = -1;
  bool cl_walls = false;
  for (int b = 0; b < nblocks; ++b) {
    ugks_fused_block &x = blocks[b];
    const int m = x.d.flux_method;
    if (m < 0 || m > 3) return -2;
    if (m != last_method) {
      if (seen & (1 << m)) return -2;  // methods must be contiguous
      seen |= 1 << m;
      fb[m] = f;
      last_method = m;
    }
    if (x.solve != last_solve) {
      if (x.solve != last_solve + 1) return -2;  // solves contiguous and in order
      last_solve = x.solve;
    }
    x.face_begin = (int32_t)f;
    x.cell_begin = (int32_t)c;
    x.ghost_begin = (int32_t)g;
    x.wall_begin = (int32_t)wl;
    wl += 2ll * (x.d.ni + x.d.nj);
    for (int w = 0; w < 4; ++w) cl_walls |= wide_cl_wall(x, w);
    const int64_t nf = 2ll * (x.d.ni + 1) * (x.d.nj + 1);
    const int axes_b = x.d.u_num > 0 ? x.d.u_num + x.d.v_num : 0;
    if (runs.empty() || runs.back().method != m || runs.back().nv != x.d.Nv)
      runs.push_back(Run{m, x.d.Nv, x.d.Nv, axes_b, f, 0});
    runs.back().count += nf;
    runs.back().axes = std::max(runs.back().axes, axes_b);
    f += nf;
    fc[m] += nf;
    c += (int64_t)x.d.ni * x.d.nj;
    g += 2ll * x.d.ghost * (x.d.ni + x.d.nj);
    if (x.d.Nv > max_nv) max_nv = x.d.Nv;
    const int axes = x.d.u_num + x.d.v_num;
    if (x.d.u_num > 0 && x.d.u_num * x.d.v_num == x.d.Nv && axes <= 512 && axes > max_axes) max_axes = axes;
  }
  if (f > INT32_MAX || c > INT32_MAX || g > INT32_MAX || wl > INT32_MAX) return -1;
  z->n_wall = (int32_t)wl;
  z->n_faces = (int32_t)f;
  z->n_cells = (int32_t)c;
  z->n_ghost = (int32_t)g;
  z->max_nv = max_nv;
  z->max_axes = max_axes;
  // at most UGKS_MAX_FACE_SEGMENTS launches: merge the adjacent pair of one
  // method whose merged Nv is smallest (methods are contiguous, so this ends
  // at one run per method at worst)
  const int limit = UGKS_MAX_FACE_SEGMENTS - (cl_walls ? 1 : 0);
  while ((int)runs.size() > limit) {
    int best = -1;
    for (int k = 0; k + 1 < (int)runs.size(); ++k)
      if (runs[k].method == runs[k + 1].method &&
          (best < 0 || std::max(runs[k].max_nv, runs[k + 1].max_nv) <
                           std::max(runs[best].max_nv, runs[best + 1].max_nv)))
        best = k;
    if (best < 0) return -2;
    runs[best].max_nv = std::max(runs[best].max_nv, runs[best + 1].max_nv);
    runs[best].axes = std::max(runs[best].axes, runs[best + 1].axes);
    runs[best].count += runs[best + 1].count;
    runs.erase(runs.begin() + best + 1);
  }
  if (cl_walls) runs.push_back(Run{UGKS_SEG_CL_WALLS, 0, max_nv, 0, 0, wl});
  z->n_segments = (int32_t)runs.size();
  for (int k = 0; k < UGKS_MAX_FACE_SEGMENTS; ++k) {
    const bool on = k < (int)runs.size();
    z->seg_begin[k] = on ? (int32_t)runs[k].begin : 0;
    z->seg_count[k] = on ? (int32_t)runs[k].count : 0;
    z->seg_method[k] = on ? runs[k].method : 0;
    z->seg_max_nv[k] = on ? runs[k].max_nv : 0;
    z->seg_max_axes[k] = on ? runs[k].axes : 0;
  }
  for (int m = 0; m < 4; ++m) {
    z->face_begin[m] = (int32_t)fb[m];
    z->face_count[m] = (int32_t)fc[m];
  }
  for (int k = 0; k < UGKS_MAX_FACE_SEGMENTS; ++k) z->seg_variant[k] = 0;
  z->cell_variant = 0;
  return 0;
}

int ugks_init_fp64(const ugks_fused_block *blocks_dev, int nblocks, const ugks_fused_sizes *sizes,
                   ugks_solve_state *solves_dev, int nsolves, void *stream) {
  return init_impl<double>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream);
}
int ugks_init_mixed(const ugks_fused_block *blocks_dev, int nblocks, const ugks_fused_sizes *sizes,
                    ugks_solve_state *solves_dev, int nsolves, void *stream) {
  return init_impl<float>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream);
}
int ugks_restart_fp64(const ugks_fused_block *blocks_dev, int nblocks, const ugks_fused_sizes *sizes,
                      ugks_solve_state *solves_dev, int nsolves, void *stream) {
  return restart_impl<double>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream);
}
int ugks_restart_mixed(const ugks_fused_block *blocks_dev, int nblocks, const ugks_fused_sizes *sizes,
                       ugks_solve_state *solves_dev, int nsolves, void *stream) {
  return restart_impl<float>(blocks_dev, nblocks, sizes, solves_dev, nsolves, stream);
}

}  // extern "C"
