// common.cuh -- device data layout and the reconstruction + Riemann-flux
// kernels shared by the FP64 translation unit (harm_gpu.cu, built with
// -fmad=false for bit-identity with the reference) and the FP32 one of the
// mixed-precision path (flux_f32.cu, built with FMA contraction and fast
// FP32 division/square root, which leave FP64 arithmetic untouched).
#pragma once
#include <cuda_runtime.h>

#include "harm_device.cuh"
#include "harmgpu.h"
#include "weno5.cuh"

namespace hg {

// geometry component offsets
constexpr int GLOC = 34;                  // per location: gcov 16, gcon 16, gcovpert_tt, gdet
// What derive_metric forms at upload.  The face kernels read gcon's upper
// triangle alone, so at the faces its lower triangle (planes 16 + 4a + b, b <
// a) holds alpha, 1/alpha, beta^1..3, 1/gdet; the inversion reads all of gcon
// at CENT, where alpha and 1/alpha have planes of their own.
__host__ __device__ constexpr int g_derived(int q) { return 16 + (q == 0 ? 4 : (q == 1 ? 8 : (q == 2 ? 9 : 9 + q))); }
constexpr int G_FACE1 = 0, G_FACE2 = 1, G_FACE3 = 2, G_CENT = 3;
constexpr int G_CORN = 4 * GLOC;          // CORN1, CORN2, CORN3 gdet
constexpr int G_CONN = G_CORN + 3;        // 64
constexpr int G_FLOOR = G_CONN + 64;      // 2
constexpr int G_LAPSE = G_FLOOR + 2;      // CENT: alpha, 1/alpha
constexpr int G_NCOMP = G_LAPSE + 2;      // 207

// reference location ids (global.h:948-955)
constexpr int R_FACE1 = 0, R_FACE2 = 1, R_FACE3 = 2, R_CORN1 = 3, R_CORN2 = 4, R_CORN3 = 5, R_CENT = 7;

struct Dims {
  int n1, n2, n3;
  int g1, g2, g3;
  int nt1, nt2, nt3;
  int s1, s2, s3;
  int gt1, gt2;
  long long nz, nij;
};

// One instance of a batch: a 1D problem occupying the x1 cells
// i0-ng .. i0+n+ng-1 of the concatenated line (its own ghosts included),
// with its own gamma, dx, time and dt (step_ch's t, dt, tf per problem).
struct Inst {
  int i0, n;
  double dx, gam, tf;
  double t, dt;
  unsigned long long ndtbits;  // x1 min of cour*dx/ctop as ordered bits
  int done;                    // t reached tf: the instance no longer advances
  int nsteps;                  // time steps this instance has taken
};

struct Params {
  double gam, cour, gammamax, gammafail, rhominlimit, uuminlimit, defcon, safe, tf;
  double dx1, dx2, dx3;
  int lim, flux;
  int bc[6];
  // finite-volume scheme: faces beyond one zone across the grid (its flux
  // loops run over all transverse ghosts) feed only the dt minimum
  int fvring;
  // batch of independent 1D instances (nullptr: one domain)
  const int *cell_inst;  // instance of every cell of the line
  Inst *inst;
  int ninst;
  // failure and floor counters per zone, NFFC planes of nz (failfloorcount,
  // fixup.c:206): incremented where the reference's diag_fixup counts
  unsigned int *ffc;
  // Bondi-integral x1 boundaries: [2][g1+1][n2][49] coordinate data (nullptr: none)
  const double *bondi;
};

// counter categories (global.h:769-779)
enum {
  CNT_UTOPRIMFAILCONV = 0,
  CNT_FLOORACT = 1,
  CNT_LIMITGAMMAACT = 2,
  CNT_INFLOWACT = 3,
  CNT_UTOPRIMFAILRHONEG = 4,
  CNT_UTOPRIMFAILUNEG = 5,
  CNT_UTOPRIMFAILRHOUNEG = 6,
  CNT_GAMMAPERC = 7,
  CNT_UPERC = 8,
  NFFC = 9
};

__device__ __forceinline__ void ffc_count(const Params &P, long long nz, long long z, int what) {
  if (P.ffc) P.ffc[(long long)what * nz + z] += 1u;
}

// device scalars
struct Scalars {
  double t, dt;
  unsigned long long ndtbits[4];   // per-direction min of cour*dx/ctop as ordered bits
  unsigned long long iters;        // Newton iterations
  int err;
  int nfail;                       // failures after Utoprimgen in the last stage
  int ncand;                       // checksolution candidates
  int ndep;                        // checksolution candidates that depend on earlier ones
  int nfixlist;                    // fixup_utoprim list length
  int nfixed;
  int overflow;
  int done;                        // t reached tf: later steps leave the state unchanged
  int nsteps;                      // time steps taken since the last upload
  unsigned long long nfloor;       // zone floorings by fixup1zone (summed over a call's final substeps)
  unsigned int blocks_done;        // blocks of a bound kernel that are through (wraps to 0 with the last)
  int nonfinite;                   // a stage of this call left an infinity or NaN in uf
};

__device__ __forceinline__ long long zix(const Dims &d, int i, int j, int k) {
  return ((long long)(i + d.g1) * d.nt2 + (j + d.g2)) * d.nt3 + (k + d.g3);
}
__device__ __forceinline__ long long gix(const Dims &d, int i, int j) {
  return (long long)(i + d.g1) * d.gt2 + (j + d.g2);
}

// metric of one location converted to the arithmetic type of a kernel
template <typename T>
__device__ __forceinline__ void load_metric_t(const double *__restrict__ G, const Dims &d, long long ij, int slot,
                                              MetricT<T> &m) {
  const double *b = G + (long long)slot * GLOC * d.nij + ij;
#pragma unroll
  for (int q = 0; q < 16; q++) m.gcov[q] = (T)__ldg(b + (long long)q * d.nij);
#pragma unroll
  for (int q = 0; q < 16; q++)
    if (slot == G_CENT || (q & 3) >= (q >> 2)) m.gcon[q] = (T)__ldg(b + (long long)(16 + q) * d.nij);
  m.gcovpert_tt = (T)__ldg(b + (long long)32 * d.nij);
  m.g = (T)__ldg(b + (long long)33 * d.nij);
  if (slot == G_CENT) {
    m.alpha = (T)__ldg(G + (long long)G_LAPSE * d.nij + ij);
    m.ralpha = (T)__ldg(G + (long long)(G_LAPSE + 1) * d.nij + ij);
    derive_shift(m);
    m.rg = kept_rcp(m.g);
  } else {
    m.alpha = (T)__ldg(b + (long long)g_derived(0) * d.nij);
    m.ralpha = (T)__ldg(b + (long long)g_derived(1) * d.nij);
#pragma unroll
    for (int q = 0; q < 3; q++) m.beta[q] = (T)__ldg(b + (long long)g_derived(2 + q) * d.nij);
    m.rg = (T)__ldg(b + (long long)g_derived(5) * d.nij);
  }
}
__device__ __forceinline__ void load_metric(const double *__restrict__ G, const Dims &d, long long ij, int slot,
                                            Metric &m) {
  load_metric_t(G, d, ij, slot, m);
}

// poison() of a state at a location
template <typename T>
__device__ __forceinline__ unsigned poison_at(const T *pr, const double *G, long long nij, long long ij, int slot) {
  Dims d;
  d.nij = nij;
  MetricT<T> m;
  load_metric_t(G, d, ij, slot, m);
  StateT<T> q;
  EMT<T> e;
  get_state(pr, m, q);
  em_prepare<0>(pr, m, q, e);
  return poison(pr, q, e);
}

__device__ __forceinline__ void load_prim(const double *__restrict__ P, const Dims &d, long long z, double *pr) {
#pragma unroll
  for (int v = 0; v < NPR; v++) pr[v] = P[(long long)v * d.nz + z];
}
__device__ __forceinline__ void store_prim(double *__restrict__ P, const Dims &d, long long z, const double *pr) {
#pragma unroll
  for (int v = 0; v < NPR; v++) P[(long long)v * d.nz + z] = pr[v];
}

// box iteration helper: flat index -> (i,j,k) with k fastest
struct Box {
  int i0, j0, k0, ni, nj, nk;
  __host__ __device__ long long size() const { return (long long)ni * nj * nk; }
};
// (a context's zones number below 2^32 -- each takes over 600 bytes of device
// memory -- so the index is divided in 32 bits, not by 64-bit routines)
__device__ __forceinline__ void box_ijk(const Box &b, long long t, int &i, int &j, int &k) {
  const unsigned u = (unsigned)t;
  const unsigned r = u / (unsigned)b.nk;
  k = (int)(u - r * b.nk);
  i = (int)(r / (unsigned)b.nj);
  j = (int)(r - (unsigned)i * b.nj);
  i += b.i0;
  j += b.j0;
  k += b.k0;
}

__device__ __forceinline__ void warp_min_atomic(unsigned long long *dst, double v, bool active) {
  unsigned long long bits = active ? (unsigned long long)__double_as_longlong(v) : 0xFFFFFFFFFFFFFFFFull;
  // NaN is never selected by the reference's `if (dtij < ndt)`: map it out
  if (active && !(v == v)) bits = 0xFFFFFFFFFFFFFFFFull;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    unsigned long long ob = __shfl_xor_sync(0xffffffffu, bits, o);
    bits = ob < bits ? ob : bits;
  }
  if ((threadIdx.x & 31) == 0 && bits != 0xFFFFFFFFFFFFFFFFull) atomicMin(dst, bits);
}

// one value from global to shared memory, asynchronously
template <typename V>
__device__ __forceinline__ void copy_async(double *to, const V *from) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(to)), "l"(from),
               "n"(sizeof(V)));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;"); }
template <int PENDING>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

// MC / VANL / MINM / DONOR slopes (interppoint.c:387-443)
template <typename T>
__device__ __forceinline__ T slope3(int lim, T yl, T yc, T yr) {
  if (lim == HGPU_LIM_MC) {
    T Dqm = T(2.0) * (yc - yl);
    T Dqp = T(2.0) * (yr - yc);
    T Dqc = T(0.5) * (yr - yl);
    T mm = ((Dqm) * (Dqp) <= T(0)) ? T(0.0) : ((fabs(Dqm) < fabs(Dqp)) ? (Dqm) : (Dqp));
    return ((Dqc) * (mm) <= T(0)) ? T(0.0) : ((fabs(Dqc) < fabs(mm)) ? (Dqc) : (mm));
  } else if (lim == HGPU_LIM_VANL) {
    T Dqm = (yc - yl);
    T Dqp = (yr - yc);
    T s = Dqm * Dqp;
    if (s <= T(0.)) return T(0.);
    return (T(2.0) * s / (Dqm + Dqp));
  } else if (lim == HGPU_LIM_MINM) {
    T Dqm = T(1.0) * (yc - yl);
    T Dqp = T(1.0) * (yr - yc);
    T Dqc = T(0.5) * (yr - yl);
    T mm = ((Dqm) * (Dqc) <= T(0)) ? T(0.0) : ((fabs(Dqm) < fabs(Dqc)) ? (Dqm) : (Dqc));
    return ((mm) * (Dqp) <= T(0)) ? T(0.0) : ((fabs(mm) < fabs(Dqp)) ? (mm) : (Dqp));
  }
  return T(0.0);
}

// para4 (interppoint.c:736-869) with PARA2LIM=MC and JONPARAREDUCE=0: face
// values of the cell at y[0] from y[-2..2]
template <typename T>
__device__ __forceinline__ void para4(const T *y, T *lout, T *rout) {
  T dq[3];
#pragma unroll
  for (int mm = -1; mm <= 1; mm++) {
    T Dqm = T(2.0) * (y[mm] - y[mm - 1]);
    T Dqp = T(2.0) * (y[mm + 1] - y[mm]);
    T Dqc = T(0.5) * (y[mm + 1] - y[mm - 1]);
    T aDqm = fabs(Dqm), aDqp = fabs(Dqp), aDqc = fabs(Dqc);
    T s = Dqm * Dqp;
    T sg = (Dqc > T(0.0)) ? T(1.0) : ((Dqc < T(0.0)) ? T(-1.0) : T(0.0));
    dq[mm + 1] = (s <= T(0.)) ? T(0.) : min_ref(aDqc, min_ref(aDqm, aDqp)) * sg;
  }
  T l = T(0.5) * (y[0] + y[-1]) - (dq[1] - dq[0]) / T(8.0);
  T r = T(0.5) * (y[1] + y[0]) - (dq[2] - dq[1]) / T(8.0);
  l = max_ref(min_ref(y[0], y[-1]), l);
  l = min_ref(max_ref(y[0], y[-1]), l);
  r = max_ref(min_ref(y[0], y[1]), r);
  r = min_ref(max_ref(y[0], y[1]), r);
  T qa = (r - y[0]) * (y[0] - l);
  T qd = (r - l);
  T qe = T(6.0) * (y[0] - T(0.5) * (l + r));
  if (qa <= T(0.)) {
    l = y[0];
    r = y[0];
  } else {
    if (qd * (qd - qe) < T(0.0)) l = T(3.0) * y[0] - T(2.0) * r;
    if (qd * (qd + qe) < T(0.0)) r = T(3.0) * y[0] - T(2.0) * l;
  }
  *lout = l;
  *rout = r;
}

// Minimum resident blocks per SM asked of the register allocator for the
// FP64-heavy kernels (launch_bounds' second argument).  With 64K registers
// per SM, B blocks of 128 threads cap a thread at 65536 / (128 B) registers:
// 1-2 -> 255 (8 warps/SM), 3 -> 170 (12 warps), 4 -> 128 (16 warps), more
// warps to hide FP64 latency at the price of spills to local memory.
// Measured on the B200, us per step: flux 4 against 3 blocks 3438 / 3679 on
// the 256x128x128 WENO5 torus, 237 / 259 on 97x51x33 MC, 58 / 54 on 64x64
// (there the few warps gain nothing from the fourth block and pay its
// spills); WENO5 4 against 3 blocks 8921 / 9716 on 256x128x128, 1008 / 1100 on
// 128x64x32; update 4 against 3 blocks 154 / 85 on 97x51x33,
// 36 / 27 on 64x64 (its spills sit in the contraction with the connection), but
// for the staged form (conserve_kernel), which takes 4.
#ifndef HG_MINB_FLUX
#define HG_MINB_FLUX 4
#endif
#ifndef HG_MINB_UPDATE
#define HG_MINB_UPDATE 3
#endif
#ifndef HG_MINB_INVERT
#define HG_MINB_INVERT 1
#endif
#ifndef HG_MINB_WENO
#define HG_MINB_WENO 4
#endif
// the same for the FP32 kernels of the mixed-precision path (B200 sweep of
// 4/6/8 for flux: 8 -4%)
#ifndef HG_MINB_FLUX_F32
#define HG_MINB_FLUX_F32 8
#endif
#ifndef HG_MINB_WENO_F32
#define HG_MINB_WENO_F32 4
#endif
template <typename T> struct MinBlocks;
template <> struct MinBlocks<double> {
  static constexpr int flux = HG_MINB_FLUX, weno = HG_MINB_WENO;
};
template <> struct MinBlocks<float> {
  static constexpr int flux = HG_MINB_FLUX_F32, weno = HG_MINB_WENO_F32;
};

// the FP64 variants the autotuner chooses between (resident blocks per SM
// for each heavy kernel; variant 0 is the default above)
constexpr int kFluxMB[2] = {HG_MINB_FLUX, HG_MINB_FLUX - 1};
constexpr int kWenoMB[2] = {HG_MINB_WENO, HG_MINB_WENO - 1};
constexpr int kConserveMB[2] = {HG_MINB_UPDATE, HG_MINB_UPDATE + 1};
// (1 and 2 name the inversion's variants for hgpu_tuning: as many blocks as its
// registers were cut for, 4 or, with Jon's inverter or the finite-volume scheme,
// 3, and one less)
constexpr int kInvertMB[2] = {HG_MINB_INVERT, 2};

template <int DIR>
__device__ __forceinline__ long long dir_stride(const Dims &d) {
  return (DIR == 1) ? (long long)d.nt2 * d.nt3 : ((DIR == 2) ? (long long)d.nt3 : 1);
}

// ---------------------------------------------------------------------------
// WENO5 line reconstruction (slope_lim_linetype_c2e, interpline.c:517-678),
// one kernel per direction.  The reference sweeps whole lines serially; here
// one thread marches one primitive along a segment of `lb` output cells of
// one line, keeping in registers what neighbouring cells share, so that every
// per-cell quantity is formed once (but for six cells where a segment starts):
//   y  the line at cells s-7..s
//   A  cell s-2: SMONO class (cusp test and indicator) and unoptimised order-3
//      weights (compute_cf_stencil_weights + mono_adjust_unoptimized_weights)
//   R  cell s-4: lower-order fraction of compute_weights_ratios from the
//      weights of cells s-6, s-4, s-2
//   F  output cell s-5: the final fraction (the cell's own, and the shock
//      factor times its neighbours'), optimised and order-2 weights and the
//      two face values -> pL, pR
// The shock factor, the post/pre-shock reduction of
// apply_additional_reduction_to_weights (reconstructeno.c:650-700) from the
// dP/P jump of compute_df_line_new (interpline.c:2148-2222), is the same for
// the eight primitives: w5_state_kernel and w5_shock_kernel form it once per
// zone and direction.
// The output cells of a direction are the line cells -1..n (the box), every
// line across it that the flux loop covers.  Every quantity has the bits of
// the reference's expressions in FP64.  T = float is the reconstruction of
// the mixed-precision path: its line is kept in FP64, it works on differences
// from each cell's own value and writes FP64 face values (the cell's value
// plus the FP32 offset), which the FP64 Riemann kernel reads.
//
// Bound by instruction issue, FP64 first (issue slots 58-68% and FP64 pipe
// 56-60% active, about 200 FP64 instructions a cell and primitive).  Staging
// tiles of a line in shared memory, one stage at a time between barriers,
// holds 1.7 other instructions (addresses, shared memory, selects, the branches
// of its divisions) to an FP64 one: 2.63 against 1.09 ms a launch on
// 256x128x128.
// The loop stays rolled: unrolled by 2 or 4, to spare the moves of its windows
// (a fifth of its instructions), it ran 15% and 52% longer.
// ---------------------------------------------------------------------------
constexpr int W5_THREADS = 128;
constexpr int W5_CHUNK = 8;               // FS: line cells staged per warp and turn
constexpr int W5_RING = 4;                // not FS: cells of a thread's ring
constexpr int W5_PITCH = W5_CHUNK + 1;    // odd, so that lanes on different rows meet different banks

struct W5Tile {
  Box box;      // output cells
  int lb;       // output cells per segment
  int w;        // lines a caller chose for a tile (kept for hgpu_tuning; rows fill the warps by themselves)
  int nseg;     // segments along the direction
  int nlines;   // lines of the box
  int fast_s;   // 1: a line's cells are contiguous in memory, 0: neighbouring lines are
};

// The dP/P pieces of compute_df_line_new (interpline.c:2148-2222) of one
// zone, (1 + u_t) u^t and gam u (u^t u_t) + (gam - 1) u, into PU[0][z] and
// PU[1][z]: they depend on the zone's state only, so one pass serves the
// WENO5 reconstruction of every direction.
template <typename T>
__global__ void __launch_bounds__(128) w5_state_kernel(Dims d, Params P, Box box, const double *__restrict__ pb,
                                                       const double *__restrict__ G, T *__restrict__ PU) {
  long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= box.size()) return;
  int i, j, k;
  box_ijk(box, t, i, j, k);
  const long long z = zix(d, i, j, k);
  const T gam = (T)(P.cell_inst ? P.inst[P.cell_inst[z]].gam : P.gam);
  T pc[NPR];
#pragma unroll
  for (int v = 0; v < NPR; v++) pc[v] = (T)pb[(long long)v * d.nz + z];
  MetricT<T> m;
  load_metric_t(G, d, gix(d, i, j), G_CENT, m);
  StateT<T> q;
  get_state(pc, m, q);
  const T a = compute_1plusud0(m, q);
  PU[z] = a * (q.ucon[0]);
  PU[d.nz + z] = gam * pc[UU] * (q.ucon[0] * q.ucov[0]) + (gam - T(1.0)) * pc[UU];
}

// The shock factor of every output cell along each direction, SS[dir-1][z],
// from the state pieces of cells -1, 0, +1 (five planes read, up to three
// written: HBM).  A zone outside a direction's cells -1..n has none there.
template <typename T>
__global__ void __launch_bounds__(256) w5_shock_kernel(Dims d, Box box, const double *__restrict__ pb,
                                                       const T *__restrict__ PU, T *__restrict__ SS) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= box.size()) return;
  int ijk[3];
  box_ijk(box, t, ijk[0], ijk[1], ijk[2]);
  const long long z = zix(d, ijk[0], ijk[1], ijk[2]);
  const long long o[3] = {(long long)d.nt2 * d.nt3, d.nt3, 1};
  const int n[3] = {d.n1, d.n2, d.n3};
  const T r0 = (T)pb[z], par = PU[z], upar = PU[d.nz + z];
#pragma unroll
  for (int q = 0; q < 3; q++) {
    if (n[q] == 1 || ijk[q] < -1 || ijk[q] > n[q]) continue;
    const T parl = PU[z - o[q]], parr = PU[z + o[q]];
    const T uparl = PU[d.nz + z - o[q]], uparr = PU[d.nz + z + o[q]];
    const T dP = (fabs(r0 * (parr - parl)) + fabs(uparr - uparl)) / (fabs(r0 * par) + fabs(upar) + w5::K<T>::tiny);
    // (x / 0.25 is the exact multiplication by 4)
    SS[q * d.nz + z] = w5::wmin((fabs(dP) - T(0.5 * w5::kDpFrac)) * T(1.0 / (0.5 * w5::kDpFrac)), T(1.));
  }
}

// zone index of cell 0 of line `line` of box b (along the line the index
// steps by dir_stride)
template <int DIR>
__device__ __forceinline__ long long w5_line(const Dims &d, const Box &b, int line) {
  int i = 0, j = 0, k = 0;
  if (DIR == 1) {
    j = b.j0 + line / b.nk;
    k = b.k0 + line % b.nk;
  } else if (DIR == 2) {
    i = b.i0 + line / b.nk;
    k = b.k0 + line % b.nk;
  } else {
    i = b.i0 + line / b.nj;
    j = b.j0 + line % b.nj;
  }
  return zix(d, i, j, k);
}

// Lines next to one another in memory (not FS): neighbouring lanes are
// neighbouring lines; each thread keeps the next three cells of its line and
// of the shock factor on their way into a ring of its own in shared memory
// (loaded into registers a step ahead, they were waited for: 2 of 6.6 stall
// cycles an instruction).  FS (a line's cells are contiguous): a warp's 32
// rows (segments of lines) lie far apart, so it brings W5_CHUNK cells of each
// at a time, a row's cells by neighbouring lanes, the next chunk while one is
// worked on, and the face values go back the same way through the slots of
// the cells they came from.
template <int DIR, bool FS, typename T, int MB = MinBlocks<T>::weno>
__global__ void __launch_bounds__(W5_THREADS, MB) weno5_kernel(Dims d, W5Tile tl, const double *__restrict__ pb,
                                                               const T *__restrict__ SS, double *__restrict__ pL,
                                                               double *__restrict__ pR) {
  // FS: [warp][buffer][Y, S][row][cell]; otherwise [slot][Y, S][thread]
  __shared__ double stage[FS ? W5_THREADS / 32 * 4 * 32 * W5_PITCH : W5_RING * 2 * W5_THREADS];
  const unsigned lane = threadIdx.x & 31;
  const unsigned rows = (unsigned)tl.nlines * tl.nseg;
  unsigned t = blockIdx.x * W5_THREADS + threadIdx.x;
  const bool on = t < rows * NPR;
  if (!on) t = rows * NPR - 1;
  const int v = (int)(t / rows);
  const unsigned r = t - v * rows;
  const int seg = FS ? (int)(r % tl.nseg) : (int)(r / tl.nlines);
  const int line = FS ? (int)(r / tl.nseg) : (int)(r % tl.nlines);
  const int nout = (DIR == 1) ? tl.box.ni : ((DIR == 2) ? tl.box.nj : tl.box.nk);
  const int nv = on ? min(tl.lb, nout - seg * tl.lb) : 0;  // output cells of this thread
  const long long o = dir_stride<DIR>(d);
  const long long zc = w5_line<DIR>(d, tl.box, line) +
                       (((DIR == 1) ? tl.box.i0 : ((DIR == 2) ? tl.box.j0 : tl.box.k0)) + seg * tl.lb) * o;
  const long long zv = zc + (long long)v * d.nz;
  const double *src = pb + zv;
  const T *ssrc = SS + (long long)(DIR - 1) * d.nz + zc;
  const int slast = nv + 4;  // the last cell this thread's output reads
  double *buf = FS ? stage + (threadIdx.x >> 5) * 4 * 32 * W5_PITCH : stage + threadIdx.x;
  // FS: cells s .. s+CHUNK-1 of the warp's rows, and of the shock factor s-5 ..
  auto bring_chunk = [&](int s, int which) {
    double *Yb = buf + which * 2 * 32 * W5_PITCH, *Sb = Yb + 32 * W5_PITCH;
#pragma unroll
    for (int it = 0; it < W5_CHUNK; it++) {
      const int row = it * (32 / W5_CHUNK) + (int)(lane / W5_CHUNK), c = (int)(lane % W5_CHUNK);
      const double *rs = (const double *)__shfl_sync(0xffffffffu, (unsigned long long)src, row);
      const T *rss = (const T *)__shfl_sync(0xffffffffu, (unsigned long long)ssrc, row);
      const int last = __shfl_sync(0xffffffffu, slast, row);
      copy_async(Yb + row * W5_PITCH + c, rs + min(s + c, last));
      copy_async(Sb + row * W5_PITCH + c, rss + max(min(s + c - 5, last - 5), 0));
    }
    copy_commit();
  };
  // otherwise: cell s of this thread's line
  auto bring = [&](int s) {
    double *slot = buf + ((s + 5) % W5_RING) * 2 * W5_THREADS;
    copy_async(slot, src + (long long)min(s, slast) * o);
    copy_async(slot + W5_THREADS, ssrc + (long long)max(min(s - 5, nv - 1), 0) * o);
    copy_commit();
  };

  double y[8];  // the line at cells s-7 .. s
  T w0[5], w1[4], w2[4];  // weights of cells s-6 .. s-2 (w0), s-5 .. s-2
  T Rm = T(0.), Rc = T(0.), Rp = T(0.);  // lower-order fractions of cells s-6, s-5, s-4
  unsigned codes = 0;     // classes, two bits a cell, s-2 lowest
#pragma unroll
  for (int q = 0; q < 8; q++) y[q] = 0.;
#pragma unroll
  for (int q = 0; q < 5; q++) w0[q] = T(0.);
#pragma unroll
  for (int q = 0; q < 4; q++) w1[q] = w2[q] = T(0.);
  if (FS) {
    bring_chunk(-5, 0);
  } else {
#pragma unroll
    for (int s = 0; s < W5_RING - 1; s++) bring(s - 5);
  }
  // (FS: whole chunks, whose face values leave with their last step)
  const int send = FS ? (tl.lb + 10 + W5_CHUNK - 1) / W5_CHUNK * W5_CHUNK - 5 : tl.lb + 5;
  for (int s = -5; s < send; s++) {
    const int slot = (s + 5) % W5_CHUNK, half = ((s + 5) / W5_CHUNK) & 1;
    double *ys = FS ? buf + half * 2 * 32 * W5_PITCH + lane * W5_PITCH + slot
                    : buf + ((s + 5) % W5_RING) * 2 * W5_THREADS;
    double *sst = ys + (FS ? 32 * W5_PITCH : W5_THREADS);
    if (FS) {
      if (slot == 0) {
        // this chunk has come; the other buffer's face values are out
        copy_wait<0>();
        __syncwarp();
        if (s + W5_CHUNK < send) bring_chunk(s + W5_CHUNK, half ^ 1);
      }
    } else {
      copy_wait<W5_RING - 2>();
    }
#pragma unroll
    for (int q = 0; q < 7; q++) y[q] = y[q + 1];
    y[7] = *ys;
    const T ss = *(const T *)sst;
    // (into the slot read a step ago)
    if (!FS) bring(s + W5_RING - 1);
    // the stencil of the cell at y[q]: values for FP64; in FP32 offsets from
    // the cell's own value, and the values for magnitudes
    auto stencil = [&](int q, T *yd, T *yn) {
#pragma unroll
      for (int e = 0; e < 5; e++) {
        if constexpr (sizeof(T) == 4) {
          yd[e] = (T)(y[q - 2 + e] - y[q]);
          yn[e] = (T)y[q - 2 + e];
        } else {
          yd[e] = yn[e] = y[q - 2 + e];
        }
      }
    };
    // (the steps that only fill the last chunk compute nothing)
    const bool live = !FS || s < tl.lb + 5;
    if (s >= -1 && live) {
      T ya[5], yb[5], w[3];
      stencil(5, ya, yb);
      const int code = w5::code_of(ya + 2, yb + 2);
      w5::weights3(code, ya + 2, yb + 2, w);
      codes = (codes << 2) | (unsigned)code;
#pragma unroll
      for (int q = 0; q < 4; q++) w0[q] = w0[q + 1];
#pragma unroll
      for (int q = 0; q < 3; q++) {
        w1[q] = w1[q + 1];
        w2[q] = w2[q + 1];
      }
      w0[4] = w[0];
      w1[3] = w[1];
      w2[3] = w[2];
    }
    if (s >= 3 && live) {
      Rm = Rc;
      Rc = Rp;
      Rp = w5::lower_fraction((int)(codes >> 4) & 3, w0[2], w2[1], w0[0], w2[3]);
    }
    if (s >= 5 && live) {
      T lof = Rc;
      lof = w5::wmax(lof, ss * Rp);
      lof = w5::wmax(lof, ss * Rm);
      T ya[5], yb[5], yl, yr;
      stencil(2, ya, yb);
      const T w[3] = {w0[1], w1[0], w2[0]};
      w5::face_values((int)(codes >> 6) & 3, ya + 2, yb + 2, w, lof, &yl, &yr);
      const double fl = sizeof(T) == 4 ? y[2] + (double)yl : (double)yl;
      const double fr = sizeof(T) == 4 ? y[2] + (double)yr : (double)yr;
      if (FS) {
        *ys = fl;
        *sst = fr;
      } else if (s - 5 < nv) {
        pL[zv + (long long)(s - 5) * o] = fl;
        pR[zv + (long long)(s - 5) * o] = fr;
      }
    }
    if (FS && slot == W5_CHUNK - 1) {
      // the face values of this chunk's output cells, s-5-slot ..
      __syncwarp();
      const double *Lb = buf + half * 2 * 32 * W5_PITCH, *Rb = Lb + 32 * W5_PITCH;
#pragma unroll
      for (int it = 0; it < W5_CHUNK; it++) {
        const int row = it * (32 / W5_CHUNK) + (int)(lane / W5_CHUNK), c = (int)(lane % W5_CHUNK);
        const long long rz = __shfl_sync(0xffffffffu, zv, row);
        const int rnv = __shfl_sync(0xffffffffu, nv, row);
        const int cell = s - 5 - slot + c;
        if (cell >= 0 && cell < rnv) {
          pL[rz + cell] = Lb[row * W5_PITCH + c];
          pR[rz + cell] = Rb[row * W5_PITCH + c];
        }
      }
    }
  }
  copy_wait<0>();
}

// the two states of face z of direction DIR
template <int DIR, int RECON, typename T, typename TR>
__device__ __forceinline__ void face_states(int lim, long long nz, long long z, long long o, const double *__restrict__ pb,
                                            const TR *__restrict__ pL, const TR *__restrict__ pR, T *p_l, T *p_r) {
  if (RECON == 1) {
    // getp2interplr (flux.c:788-808), line-type branch
#pragma unroll
    for (int v = 0; v < NPR; v++) {
      p_l[v] = (T)__ldg(pR + (long long)v * nz + z - o);
      p_r[v] = (T)__ldg(pL + (long long)v * nz + z);
    }
  } else if (RECON == 2) {
    // PARA: pright of the cell on the left, pleft of the cell on the right
#pragma unroll
    for (int v = 0; v < NPR; v++) {
      const double *q = pb + (long long)v * nz + z;
      T y[6];
#pragma unroll
      for (int l = 0; l < 6; l++) y[l] = (T)__ldg(q + (l - 3) * o);
      T dummy;
      para4(y + 2, &dummy, &p_l[v]);
      para4(y + 3, &p_r[v], &dummy);
    }
  } else {
#pragma unroll
    for (int v = 0; v < NPR; v++) {
      const double *q = pb + (long long)v * nz + z;
      T ym2 = (T)__ldg(q - 2 * o), ym1 = (T)__ldg(q - o), y0 = (T)__ldg(q), yp1 = (T)__ldg(q + o);
      T dqm = slope3(lim, ym2, ym1, y0);
      T dq0 = slope3(lim, ym1, y0, yp1);
      // getp2interplr (flux.c:788-808)
      p_l[v] = ym1 + T(0.5) * dqm;
      p_r[v] = y0 - T(0.5) * dq0;
    }
  }
  // BDIRCONT (flux.c:629-633)
  p_l[B1 + DIR - 1] = p_r[B1 + DIR - 1] = T(0.5) * (p_l[B1 + DIR - 1] + p_r[B1 + DIR - 1]);
}

// A stored flux that is not finite: the components that a NaN product of
// either state reaches.  Out of line and from the states' sources: few faces
// come here, and what the products need, kept beside two states, cost the
// Riemann kernels 400 B of spills a thread.
template <int DIR, int RECON, typename T, typename TR>
static __device__ __noinline__ void poison_face(int lim, long long nz, long long z, long long o, const double *pb,
                                                const TR *pL, const TR *pR, const double *G, long long nij, long long ij,
                                                double *F) {
  T p_l[NPR], p_r[NPR], nans[NPR] = {};
  face_states<DIR, RECON>(lim, nz, z, o, pb, pL, pR, p_l, p_r);
  const unsigned l = poison_at(p_l, G, nij, ij, DIR - 1), r = poison_at(p_r, G, nij, ij, DIR - 1);
  put_poison(l, DIR, nans);
  put_poison(l, 0, nans);
  put_poison(r, DIR, nans);
  put_poison(r, 0, nans);
#pragma unroll
  for (int v = UU; v <= U3; v++)
    if (nans[v] != T(0.)) F[(long long)v * nz + z] = NAN;
}

// ---------------------------------------------------------------------------
// face flux kernel (one per direction); RECON 0: MC-type slopes in the
// kernel, RECON 1: Riemann states from the WENO5 face values pL/pR (stored
// as TR), RECON 2: PARA
// ---------------------------------------------------------------------------
// MIX = 1: the mixed-precision variant of the FP64 kernel (wave speeds in
// FP32, vchar_f32; instantiated only in flux_f32.cu, whose FP64 arithmetic
// may contract a*b+c into FMA).
// Bound by FP64 issue and by the registers of two states.  On the
// 256x128x128 WENO5 torus one direction takes 0.57 ms a launch, 1.14 ms
// while every quotient was a division of its own and the tensors' zero
// diagonals and the unit vectors of simplefast were multiplied out.
template <int DIR, int RECON, typename T, typename TR, int MIX>
__device__ __forceinline__ void flux_block(unsigned block, const Dims &d, const Params &P, const Box &box,
                                           const double *__restrict__ pb, const TR *__restrict__ pL,
                                           const TR *__restrict__ pR, const double *__restrict__ G,
                                           double *__restrict__ F, Scalars *sc) {
  long long t = (long long)block * blockDim.x + threadIdx.x;
  bool active = t < box.size();
  double dtij = 0.0;
  bool bad = false;
  if (active) {
    int i, j, k;
    box_ijk(box, t, i, j, k);
    long long z = zix(d, i, j, k);
    const long long o = dir_stride<DIR>(d);
    T p_l[NPR], p_r[NPR];
    face_states<DIR, RECON>(P.lim, d.nz, z, o, pb, pL, pR, p_l, p_r);
    MetricT<T> m;
    load_metric_t(G, d, gix(d, i, j), DIR - 1, m);
    int b = P.cell_inst ? P.cell_inst[z] : -1;
    const T gam = (T)(b >= 0 ? P.inst[b].gam : P.gam);
    int err = 0;
    // a face that only feeds the dt minimum needs the wave speeds alone
    bool ring = false;
    if (P.fvring) {
      if (DIR != 1 && (i < -d.s1 || i > d.n1 - 1 + d.s1)) ring = true;
      if (DIR != 2 && (j < -d.s2 || j > d.n2 - 1 + d.s2)) ring = true;
      if (DIR != 3 && (k < -d.s3 || k > d.n3 - 1 + d.s3)) ring = true;
    }
    T cmaxl = T(0.), cminl = T(0.), cmaxr = T(0.), cminr = T(0.);
    T Fl[NPR], Fr[NPR], Ul[NPR], Ur[NPR];
    {
      StateT<T> q;
      if (get_state(p_l, m, q)) err |= ERR_UTCALC_DISCR;
      if constexpr (MIX != 0) err |= vchar_f32(p_l, q, DIR, m, gam, &cmaxl, &cminl);
      else err |= vchar(p_l, q, DIR, m, gam, &cmaxl, &cminl);
      if (!ring) {
        EMT<T> e;
        em_prepare<DIR>(p_l, m, q, e);
        primtoflux<DIR>(p_l, q, e, m, gam, Fl);
        primtoflux<0>(p_l, q, e, m, gam, Ul);
      }
    }
    {
      StateT<T> q;
      if (get_state(p_r, m, q)) err |= ERR_UTCALC_DISCR;
      if constexpr (MIX != 0) err |= vchar_f32(p_r, q, DIR, m, gam, &cmaxr, &cminr);
      else err |= vchar(p_r, q, DIR, m, gam, &cmaxr, &cminr);
      if (!ring) {
        EMT<T> e;
        em_prepare<DIR>(p_r, m, q, e);
        primtoflux<DIR>(p_r, q, e, m, gam, Fr);
        primtoflux<0>(p_r, q, e, m, gam, Ur);
      }
    }
    // cminmax_calc (wavespeeds.c:325-385)
    T lmin = min_ref(cminl, cminr);
    T lmax = max_ref(cmaxl, cmaxr);
    lmin = fabs(max_ref(T(0.), -lmin));
    lmax = fabs(max_ref(T(0.), lmax));
    T cmin = lmin, cmax = lmax, ctop = max_ref(lmax, lmin);
    if (!ring) {
      double Fo[NPR];
      if (P.flux == HGPU_FLUX_HLL && (cmax + cmin != T(0.0))) {
        T num[NPR], quo[NPR];
#pragma unroll
        for (int v = 0; v < NPR; v++) num[v] = (cmax * Fl[v] + cmin * Fr[v]) - (cmax * cmin) * (Ur[v] - Ul[v]);
        div_n<NPR>(num, make_divisor(cmax + cmin), quo);
#pragma unroll
        for (int v = 0; v < NPR; v++) Fo[v] = (double)quo[v];
      } else {
#pragma unroll
        for (int v = 0; v < NPR; v++) Fo[v] = (double)(T(0.5) * ((Fl[v] + Fr[v]) - ctop * (Ur[v] - Ul[v])));
      }
      // flux_ct gdet strip (fluxct.c:74-96), in FP64 in both precision modes
      const double *gf = G + (long long)((DIR - 1) * GLOC) * d.nij + gix(d, i, j);
      double Fs[3];
      div_n<3>(Fo + B1, known_divisor(__ldg(gf + 33 * d.nij), __ldg(gf + g_derived(5) * d.nij)), Fs);
      Fo[B1] = Fs[0];
      Fo[B2] = Fs[1];
      Fo[B3] = Fs[2];
      store_prim(F, d, z, Fo);
      bad = not_finite(Fo[UU + DIR]);
    }
    double dxd = (DIR == 1) ? P.dx1 : ((DIR == 2) ? P.dx2 : P.dx3);
    if (b >= 0) {
      // batch: faces 0..n of a running instance feed its own dt
      const Inst &I = P.inst[b];
      int loc = i - I.i0;
      active = false;
      if (loc >= 0 && loc <= I.n && !I.done) {
        dtij = P.cour * I.dx / (double)ctop;
        if (dtij == dtij) atomicMin(&P.inst[b].ndtbits, (unsigned long long)__double_as_longlong(dtij));
        if (err) atomicOr(&sc->err, err);
      }
    } else {
      dtij = P.cour * dxd / (double)ctop;
      if (err) atomicOr(&sc->err, err);
    }
  }
  warp_min_atomic(&sc->ndtbits[DIR], dtij, active);
  if (bad) {
    int i, j, k;
    box_ijk(box, t, i, j, k);
    poison_face<DIR, RECON, T>(P.lim, d.nz, zix(d, i, j, k), dir_stride<DIR>(d), pb, pL, pR, G, d.nij, gix(d, i, j), F);
  }
}

template <int DIR, int RECON, typename T, int MB = MinBlocks<T>::flux, typename TR = T, int MIX = 0>
__global__ void __launch_bounds__(128, MB) flux_kernel(Dims d, Params P, Box box,
                                                                 const double *__restrict__ pb,
                                                                 const TR *__restrict__ pL, const TR *__restrict__ pR,
                                                                 const double *__restrict__ G, double *__restrict__ F,
                                                                 Scalars *sc) {
  flux_block<DIR, RECON, T, TR, MIX>(blockIdx.x, d, P, box, pb, pL, pR, G, F, sc);
}

// get_bsqflags (fixup.c:1751-1849), which pre_fixup runs on the stage's
// input state at the start of every RK stage (step_ch.c:117-120): per zone,
// with the CENT metric, b^2/rho against BSQORHOLIMIT and b^2/u against
// BSQOULIMIT (initbase.c:465-466), 2 above the limit, 1 above 0.9 of it,
// else 0: the FLAGBSQORHO and FLAGBSQOU slots of pflag, packed as
// FLAGBSQORHO | FLAGBSQOU << 2.  With LIMADJUST = FLUXADJUST = 0 they change
// no state; the last stage's values are what the reference leaves in pflag.
// A state whose u^t has no real solution sets ERR_UTCALC_DISCR, as the
// reference's FAILSTATEMENT ends the step.
constexpr double BSQORHOLIMIT = 20.0, BSQOULIMIT = 100.0;
__device__ __forceinline__ void bsqflags_zone(long long z, const Dims &d, const double *__restrict__ pv,
                                              const double *__restrict__ G, unsigned char *__restrict__ bf,
                                              Scalars *sc) {
  if (z >= d.nz) return;
  const long long r = z / d.nt3;
  const int j = (int)(r % d.nt2) - d.g2;
  const int i = (int)(r / d.nt2) - d.g1;
  double pr[NPR];
  load_prim(pv, d, z, pr);
  Metric m;
  load_metric(G, d, gix(d, i, j), G_CENT, m);
  State q;
  if (get_state(pr, m, q)) {
    atomicOr(&sc->err, ERR_UTCALC_DISCR);
    bf[z] = 0;
    return;
  }
  const double bsq = dot4(q.bcon, q.bcov);
  int f0, f3;
  if (bsq / pr[RHO] > BSQORHOLIMIT) f0 = 2;
  else if (bsq / pr[RHO] > 0.9 * BSQORHOLIMIT) f0 = 1;
  else f0 = 0;
  if (bsq / pr[UU] > BSQOULIMIT) f3 = 2;
  else if (bsq / pr[UU] > 0.9 * BSQOULIMIT) f3 = 1;
  else f3 = 0;
  bf[z] = (unsigned char)(f0 | (f3 << 2));
}

// The faces of every direction in one launch (point reconstructions, whose
// states need no pass of their own), and behind them, on the last RK stage,
// the b^2 flags of the state pi.  The directions and the flags do not depend
// on one another: on a 64x64 grid one direction's 33 blocks take 11 us on 148
// SMs, all of it latency, so that two directions at once cost the time of
// one; on large grids the last wave of one direction fills with the next.
//
// The finite-volume scheme's faces beyond one zone across the grid feed only
// the dt minimum and stop after the wave speeds.  They come as boxes of their
// own: in rows of 34 full and 20 such faces (11 ghosts on 32 zones along x3) a
// third of every warp waited on the others.
constexpr int FACE_BOXES = 5;  // the faces with fluxes, and the ring on four sides
struct FaceBoxes {
  Box box[FACE_BOXES];
  unsigned first[FACE_BOXES + 1];  // first block of each box, and the number of blocks
};
struct FluxJob {
  FaceBoxes faces[4];     // per direction
  unsigned first[5];      // first block of direction 1, 2, 3, of the flags, and the number of blocks
  double *F[4];
  const double *pi;
  unsigned char *bsqf;
};
template <int DIR, int RECON, typename T>
__device__ __forceinline__ void flux_boxes(unsigned block, const Dims &d, const Params &P, const FaceBoxes &B,
                                           const double *__restrict__ pb, const double *__restrict__ G,
                                           double *__restrict__ F, Scalars *sc) {
  int s = 0;
  while (s < FACE_BOXES - 1 && block >= B.first[s + 1]) s++;
  flux_block<DIR, RECON, T, T, 0>(block - B.first[s], d, P, B.box[s], pb, nullptr, nullptr, G, F, sc);
}
template <int RECON, typename T, int MB = MinBlocks<T>::flux>
__global__ void __launch_bounds__(128, MB) fluxes_kernel(Dims d, Params P, FluxJob J, const double *__restrict__ pb,
                                                         const double *__restrict__ G, Scalars *sc) {
  const unsigned b = blockIdx.x;
  if (b < J.first[1])
    flux_boxes<1, RECON, T>(b, d, P, J.faces[1], pb, G, J.F[1], sc);
  else if (b < J.first[2])
    flux_boxes<2, RECON, T>(b - J.first[1], d, P, J.faces[2], pb, G, J.F[2], sc);
  else if (b < J.first[3])
    flux_boxes<3, RECON, T>(b - J.first[2], d, P, J.faces[3], pb, G, J.F[3], sc);
  else if constexpr (sizeof(T) == 8)  // (of the FP64 unit; see launch_fluxes_t)
    bsqflags_zone((long long)(b - J.first[3]) * blockDim.x + threadIdx.x, d, J.pi, G, J.bsqf, sc);
}


}  // namespace hg
