// Plain FP64 kernels of the Eulerian hydro step (sm_103a).
//
// This translation unit is compiled with --fmad=false: every multiply and add
// below rounds separately, in the order the reference writes them, so the
// results are bit-identical to the reference arithmetic of
//   evaluate_time_step  apps/hydro/tasks.h:331-376
//   evaluate_gradients  apps/hydro/tasks.h:145-321
//   evaluate_fluxes     apps/hydro/tasks.h:385-464
//   apply_update        apps/hydro/tasks.h:589-659
// with the physics of flecsale/eqns/euler_eqns.h and flecsale/eqns/flux.h and
// the ideal gas of flecsale/eos/ideal_gas.h (IEEE division and square root are
// correctly rounded on both CPU and GPU).
//
// Layout: every field component is its own FP64 plane (SoA), so a warp's 32
// consecutive cells or faces read 256 contiguous bytes per plane.  Neighbour
// gathers follow the CSR lists in the reference's iteration order; with
// lexicographic numbering the neighbours of a warp's cells share cache lines and
// are served from L1/L2 after the first touch.
//
// Pipes: GB300 issues 2 FP64 operations per clock per SM.  Most products and
// every quotient below are computed on the integer/FP32 pipes by the
// correctly rounded routines of fvh_sf64.cuh, while most sums and differences
// stay on the FP64 pipe; each kernel moves a part of one kind to the other
// pipe so that both are loaded alike (fp64_products, add_call).  Comparisons,
// minima and maxima run on integer order keys.  Both pipes round to
// nearest-even exactly as IEEE binary64 does, so the bits are unchanged, and
// they work at the same time.  Each unit of work (a cell or a
// face) is evaluated optimistically with the branch-free integer forms
// (arith_opt); if any operand was of a kind they do not handle (subnormal,
// infinite, NaN, beyond 2^+-500) the unit is evaluated again with the FP64
// instructions (arith_hw) and that result is kept.
//
// Code size: the integer forms inline to tens of instructions per product, so
// a fully unrolled kernel outgrows the SM's instruction cache and its warps
// stall on instruction fetch.  The kernels for many cells keep their neighbour
// and vertex loops rolled, evaluate each physical flux once per side (selecting
// the state instead of branching into copies), and take the fluxes' products, the
// quotients and the FP64 redo of a rare unit in out-of-line calls.  Inlined and
// unrolled the 1024^2 step took 2.27 ms, so arranged 1.77, with the work below
// 1.19.
//
// What bounds them: with many cells the FP64 and the integer pipes, loaded alike
// (1024^2: FP64 66-79 % busy, ALU 59-64 %; the gradients 85-90 % on a flow with waves
// everywhere); with few cells the chain of loads and operations of one thread, so
// those kernels (gradients_few_kernel and the others named so) spread a cell's
// variables over threads and use the FP64 instructions.
#include <cuda_runtime.h>

#include <cstdint>
#include <type_traits>

#include "flecsale_gb300.h"
#include "fvh_kernels.h"
#include "fvh_sf64.cuh"

namespace fvh {
namespace plain {

// Few cells or faces leave most of the chip idle and a kernel's time is one
// thread's chain of loads and operations.  The FP64 instructions are then the
// shorter chain (their pipe is shared by few warps), small blocks reach more SMs
// and unrolled loops load ahead.  Where the lines lie:
constexpr int kFewThreads = 64;
// Gradients with tables: a step takes 58 us at 64^2 against 60 with the integer forms
// one variable a thread and 68 in pairs, at 112^2 71, 68 and 75; in 3D at 16^3 107,
// 115 and 132, at 20^3 139, 130 and 152.
constexpr int kFewCells = 6144;
// ... and without (us a launch, few and many cells' kernel; gas at rest, and waves):
// 2D with the limiter 13.3 and 23.0, 14.4 and 45.5 at 64^2, 29.4 and 29.3, 29.9 and
// 46.6 at 112^2, 38.5 and 29.4, 39.8 and 46.4 at 127x129; without it 13.3 and 16.2,
// 13.3 and 19.9 at 80^2, 19.1 and 16.1, 19.0 and 19.5 at 90^2; 3D 93 and 107, 92 and
// 163 at 20^3, 159 and 109, 152 and 162 at 22x23x23, 186 and 111, 187 and 164 at
// 25x25x26.
constexpr int few_cells_no_tables(int dim, bool limited) {
  return dim == 3 ? 8000 : limited ? 15360 : 6400;
}
// Fluxes: a step with tables takes 44.0 us against 48.1 (HLLE), 45.1 and 45.7 (HLLC),
// 43.2 and 44.7 (Rusanov) at 64^2, 58.1 and 59.7, 59.4 and 57.4, 56.1 and 56.0 at
// 100^2; in 3D 71.5 and 74.7, 71.6 and 72.8, 70.9 and 71.8 at 12^3.  First order 5.8
// us a launch against 6.8, 6.1 and 6.2, 5.1 and 5.8 at 64^2.  Second order without
// tables only Rusanov gains (7.1 and 7.7, in 3D 10.1 and 10.5): HLLC takes 8.7 and
// 7.0 on a gas at rest and 8.2 and 8.4 with waves at 64^2, 11.7 and 8.2, 11.1 and
// 10.9 at 12^3, HLLE 7.8 and 7.8, 11.0 and 9.4.
constexpr int kFewFaces = 10000;
constexpr bool few_faces_form(int kind, bool second, bool pre) {
  return pre || !second || kind == FVH_FLUX_RUSANOV;
}
// Update, a launch in a graph: 4.96 us against 5.57 with 1,024 cells, 5.34 and 5.92
// with 14,400, 6.56 and 7.02 with 20,022, 6.79 and 7.00 with 28,900, 9.88 and 8.06
// with 44,100; in 3D 6.27 against 7.48 with 4,096, 8.60 and 9.15 with 19,683, 10.7 and
// 9.24 with 32,768.
constexpr int kFewUpdateCells = 20000;

// Products and quotients in out-of-line calls (a call costs a few
// instructions; inlining them everywhere made the kernels too large for the
// instruction cache).  Each returns its result with the flag that an operand
// was left to the hardware.
struct flagged {
  double q;
  unsigned rare;
};
__device__ __noinline__ flagged mul_call(double a, double b) {
  flagged r;
  r.rare = 0;
  r.q = sf64::mul_opt(a, b, r.rare);
  return r;
}
__device__ __noinline__ flagged div_call(double a, double b) {
  flagged r;
  r.rare = 0;
  r.q = sf64::div_opt(a, b, r.rare);
  return r;
}
// A sum on the integer pipe (correctly rounded; rare operands inside go to the
// hardware instruction), for a kernel whose FP64 pipe is the busier one.
__device__ __noinline__ double add_call(double a, double b) { return sf64::add(a, b); }

// Products and quotients of one unit of work: on the integer pipes, noting
// any operand they leave to the hardware ...
struct arith_opt {
  static constexpr bool wide_issue = true;  // many warps: skip what adds nothing
  using part = sf64::parts;
  unsigned rare = 0;
  // an operand of several products is taken apart once
  __device__ __forceinline__ part take(double x) { return sf64::take(x, rare); }
  // an entry of the solver's tables, known to be moderate or zero
  __device__ __forceinline__ part take_entry(double x) { return sf64::take_plain(x); }
  __device__ __forceinline__ double prod(const part &a, const part &b) {
    return sf64::mul_parts(a, b);
  }
  // s + a * b for a sum s that started at +0 (so it is never -0 and a zero
  // product leaves it as it is); the first product is the sum 0 + a * b
  __device__ __forceinline__ void add_first(double &s, const part &a, const part &b) {
    const double q = sf64::mul_core(a, b);
    s = (a.zero | b.zero) ? 0.0 : q;
  }
  __device__ __forceinline__ void add(double &s, const part &a, const part &b) {
    const double q = sf64::mul_core(a, b);
    if (!(a.zero | b.zero)) s += q;
  }
  __device__ __forceinline__ double mul(double a, double b) {
    const flagged r = mul_call(a, b);
    rare |= r.rare;
    return r.q;
  }
  __device__ __forceinline__ double quo(double a, double b) {
    const flagged r = div_call(a, b);
    rare |= r.rare;
    return r.q;
  }
  // x * 0.5 and x / 2, the same correctly rounded value: exact while the
  // half is a normal number, so the exponent field drops by one; zeros keep
  // their bits; tiny, infinite and NaN operands are left to the hardware
  __device__ __forceinline__ double half(double x) {
    unsigned lo, hi;
    sf64::halves(x, lo, hi);
    const unsigned e = sf64::expo(hi);
    rare |= (unsigned)((e <= 1u) & !sf64::is_zero(lo, hi)) | (unsigned)(e == 0x7ffu);
    return e > 1u ? sf64::join(lo, hi - (1u << 20)) : x;
  }
};
// ... and with the FP64 instructions (the evaluation kept when `rare`)
struct arith_hw {
  static constexpr bool wide_issue = false;  // few warps: independent loads, no branches
  static constexpr unsigned rare = 0;
  using part = double;
  __device__ __forceinline__ part take(double x) { return x; }
  __device__ __forceinline__ part take_entry(double x) { return x; }
  __device__ __forceinline__ double prod(part a, part b) { return __dmul_rn(a, b); }
  __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  __device__ __forceinline__ double quo(double a, double b) { return __ddiv_rn(a, b); }
  __device__ __forceinline__ double half(double x) { return __dmul_rn(x, 0.5); }
};

// Products of a part of a unit's work on the FP64 pipe (the same correctly
// rounded bits), the rest of the arithmetic as the unit's policy does it: a
// kernel whose integer pipe is the busier one moves some products back: in the
// fluxes one side's physical flux and the area scaling, in dt the dot products.
// Four steps at 1024^2 (HLLC) and two at 80^3 (Rusanov) take 4.739 and 4.033 ms so;
// with the area scaling on the integer pipe 4.718 and 4.047, the physical flux
// there 4.723 and 4.050, the normal velocities on the FP64 pipe 4.833 and 4.067.
template <class A>
struct fp64_products {
  A &ar;
  __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  __device__ __forceinline__ double quo(double a, double b) { return ar.quo(a, b); }
  __device__ __forceinline__ double half(double x) { return ar.half(x); }
};

// IEEE comparisons decided on the integer pipe (an FP64 compare would take an
// FP64 issue slot): order keys of the two's-complement kind, NaN unordered.
__device__ __forceinline__ bool is_nan(unsigned lo, unsigned hi) {
  const unsigned h = hi & 0x7fffffffu;
  return h > 0x7ff00000u || (h == 0x7ff00000u && lo != 0u);
}
__device__ __forceinline__ long long cmp_key(unsigned lo, unsigned hi) {
  // -0 and +0 share a key; a < b exactly when key(a) < key(b) for non-NaN
  long long b = (long long)(((unsigned long long)hi << 32) | lo);
  b = (b == (long long)0x8000000000000000ull) ? 0ll : b;
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
// a < b
__device__ __forceinline__ bool lt(double a, double b) {
  unsigned al, ah, bl, bh;
  sf64::halves(a, al, ah);
  sf64::halves(b, bl, bh);
  return !is_nan(al, ah) && !is_nan(bl, bh) && cmp_key(al, ah) < cmp_key(bl, bh);
}
// x >= 0, x <= 0, x < 0
__device__ __forceinline__ bool ge0(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return !is_nan(lo, hi) && ((hi >> 31) == 0u || sf64::is_zero(lo, hi));
}
__device__ __forceinline__ bool le0(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return !is_nan(lo, hi) && ((hi >> 31) != 0u || sf64::is_zero(lo, hi));
}
__device__ __forceinline__ bool lt0(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return !is_nan(lo, hi) && (hi >> 31) != 0u && !sf64::is_zero(lo, hi);
}
// x == +-0
__device__ __forceinline__ bool is_zero(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return sf64::is_zero(lo, hi);
}
// neither -0 nor a NaN (x + (+-0) == x bit for bit)
__device__ __forceinline__ bool ordinary(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return !is_nan(lo, hi) && !(hi == 0x80000000u && lo == 0u);
}
// |x| by clearing the sign bit
__device__ __forceinline__ double absval(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return sf64::join(lo, hi & 0x7fffffffu);
}

// std::max / std::min semantics of the reference (a < b ? b : a)
__device__ __forceinline__ double smax(double a, double b) { return lt(a, b) ? b : a; }
__device__ __forceinline__ double smin(double a, double b) { return lt(b, a) ? b : a; }

// x with a negative zero made positive: 0 + x without an FP64 addition.
__device__ __forceinline__ double plus_zero(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return sf64::join(lo, (hi ^ 0x80000000u | lo) == 0u ? 0u : hi);
}

// The reference sums from zero in index order.  Starting from the first
// product instead gives the same sum except that it can be -0 (all products
// -0), where the sum from zero is +0.  The FP64 pipe is the bound of these
// kernels, and this takes one addition off every dot product.
template <int D, class A>
__device__ __forceinline__ double dot(A &ar, const double *a, const double *b) {
  double s = ar.mul(a[0], b[0]);
#pragma unroll
  for (int i = 1; i < D; ++i) s += ar.mul(a[i], b[i]);
  return plus_zero(s);
}

// Same slots as pack_copy(c, d, v, p, e, T, a) (tasks.h:420).  T is carried by
// the reference but never used in a flux, so it is not loaded here.
template <int D>
struct prim {
  double d, v[D], p, e, a;
};

template <int D, class A>
__device__ __forceinline__ double total_energy(A &ar, const prim<D> &u) {
  // 0.5 * |v|^2; squares are never -0
  double s = ar.mul(u.v[0], u.v[0]);
#pragma unroll
  for (int i = 1; i < D; ++i) s += ar.mul(u.v[i], u.v[i]);
  return u.e + ar.half(s);
}

// The physical flux of u along n from its normal velocity vn = v.n and total
// energy et, which the Riemann fluxes also use themselves.
template <int D, class A>
__device__ __forceinline__ void phys_flux(A &ar, const prim<D> &u, const double *n, double vn,
                                          double et, double *f) {
  const double mass_flux = ar.mul(u.d, vn);
  f[0] = mass_flux;
#pragma unroll
  for (int i = 0; i < D; ++i) f[1 + i] = ar.mul(mass_flux, u.v[i]) + ar.mul(u.p, n[i]);
  f[D + 1] = ar.mul(mass_flux, et + ar.quo(u.p, u.d));
}

// a or b, value by value (a reference to either would put both in memory)
template <int D>
__device__ __forceinline__ prim<D> pick(bool first, const prim<D> &a, const prim<D> &b) {
  prim<D> u;
  u.d = first ? a.d : b.d;
#pragma unroll
  for (int i = 0; i < D; ++i) u.v[i] = first ? a.v[i] : b.v[i];
  u.p = first ? a.p : b.p;
  u.e = first ? a.e : b.e;
  u.a = first ? a.a : b.a;
  return u;
}

// ur - ul of the conserved variables, from the total energies
template <int D, class A>
__device__ __forceinline__ void solution_delta(A &ar, const prim<D> &l, const prim<D> &r,
                                               double et_l, double et_r, double *du) {
  const double ener_l = ar.mul(l.d, et_l);
  const double ener_r = ar.mul(r.d, et_r);
  du[0] = r.d - l.d;
#pragma unroll
  for (int i = 0; i < D; ++i) du[1 + i] = ar.mul(r.d, r.v[i]) - ar.mul(l.d, l.v[i]);
  du[D + 1] = ener_r - ener_l;
}

template <int D, class A>
__device__ __forceinline__ void hlle(A &ar, const prim<D> &l, const prim<D> &r,
                                     const double *n, double *f) {
  const double vnl = dot<D>(ar, l.v, n), vnr = dot<D>(ar, r.v, n);
  const double lambda_l = smin(vnl - l.a, vnr - r.a);
  const double lambda_r = smax(vnl + l.a, vnr + r.a);
  // one physical-flux evaluation per side: the upwind side's (or the left
  // side's when both are needed), then the right side's if both are
  const bool up_l = ge0(lambda_l), up_r = !up_l && le0(lambda_r);
  const prim<D> u = pick<D>(up_r, r, l);
  const double et = total_energy<D>(ar, u);
  phys_flux<D>(ar, u, n, up_r ? vnr : vnl, et, f);
  if (up_l || up_r) return;
  double fr[D + 2], du[D + 2];
  const double et_r = total_energy<D>(ar, r);
  phys_flux<D>(ar, r, n, vnr, et_r, fr);
  const double c1 = ar.mul(lambda_l, lambda_r);
  const double c2 = lambda_r - lambda_l;
  const double c2inv = ar.quo(1, c2);
  solution_delta<D>(ar, l, r, et, et_r, du);
#pragma unroll
  for (int i = 0; i < D + 2; ++i)
    f[i] = ar.mul(c2inv, ar.mul(lambda_r, f[i]) - ar.mul(lambda_l, fr[i]) + ar.mul(c1, du[i]));
}

template <int D, class A>
__device__ __forceinline__ void rusanov(A &ar, const prim<D> &l, const prim<D> &r,
                                        const double *n, double *f) {
  double fl[D + 2], fr[D + 2], du[D + 2];
  const double vnl = dot<D>(ar, l.v, n), vnr = dot<D>(ar, r.v, n);
  const double et_l = total_energy<D>(ar, l), et_r = total_energy<D>(ar, r);
  {
    fp64_products<A> pp{ar};
    phys_flux<D>(pp, l, n, vnl, et_l, fl);
  }
  phys_flux<D>(ar, r, n, vnr, et_r, fr);
  const double s = smax(l.a + absval(vnl), r.a + absval(vnr));
  solution_delta<D>(ar, l, r, et_l, et_r, du);
  const double half_s = ar.half(s);  // s / 2
#pragma unroll
  for (int i = 0; i < D + 2; ++i) f[i] = ar.half(fl[i] + fr[i]) - ar.mul(du[i], half_s);
}

// Toro's HLLC (sec. 10.4) with the hlle_flux wave-speed estimates.
template <int D, class A>
__device__ __forceinline__ void hllc(A &ar, const prim<D> &l, const prim<D> &r,
                                     const double *n, double *f) {
  const double vnl = dot<D>(ar, l.v, n), vnr = dot<D>(ar, r.v, n);
  const double sL = smin(vnl - l.a, vnr - r.a);
  const double sR = smax(vnl + l.a, vnr + r.a);
  // one physical-flux evaluation: of the upwind side, or of the star
  // region's side, which then takes its correction
  const bool up_l = ge0(sL), up_r = !up_l && le0(sR), star = !(up_l || up_r);
  double ml = 0, mr = 0, sM = 0;
  bool left = up_l;
  if (star) {
    ml = ar.mul(l.d, sL - vnl);
    mr = ar.mul(r.d, sR - vnr);
    sM = ar.quo(r.p - l.p + ar.mul(ml, vnl) - ar.mul(mr, vnr), ml - mr);
    left = ge0(sM);
  }
  const prim<D> u = pick<D>(left, l, r);
  const double vnK = left ? vnl : vnr;
  const double et = total_energy<D>(ar, u);
  {
    fp64_products<A> pp{ar};
    phys_flux<D>(pp, u, n, vnK, et, f);
  }
  if (!star) return;
  const double sK = left ? sL : sR;
  const double mK = left ? ml : mr;
  const double EK = ar.mul(u.d, et);
  const double fac = ar.quo(mK, sK - sM);
  const double dvn = sM - vnK;
  f[0] = f[0] + ar.mul(sK, fac - u.d);
#pragma unroll
  for (int i = 0; i < D; ++i)
    f[1 + i] = f[1 + i] +
               ar.mul(sK, ar.mul(fac, u.v[i] + ar.mul(dvn, n[i])) - ar.mul(u.d, u.v[i]));
  f[D + 1] = f[D + 1] +
             ar.mul(sK, ar.mul(fac, ar.quo(EK, u.d) + ar.mul(dvn, sM + ar.quo(u.p, mK))) - EK);
}

// ---------------------------------------------------------------------------
// Order-preserving integer keys of doubles.  Minima and maxima of doubles run
// on the integer pipe through these keys.  key(a) < key(b) exactly when a < b
// for non-NaN values; -0 and +0 share the key of +0, so a minimum or maximum
// can differ from the floating-point one only in the sign of a zero.
// ---------------------------------------------------------------------------
__device__ __forceinline__ long long okey(double x) {
  long long b = __double_as_longlong(x);
  b = (b == (long long)0x8000000000000000ull) ? 0ll : b;
  return b ^ ((b >> 63) & 0x7fffffffffffffffll);
}
__device__ __forceinline__ double from_okey(long long k) {
  return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffll));
}

// ---------------------------------------------------------------------------
// dt: per-block maxima of (a + |v.n|) / (V/A), then one block finishes.
// With PRE the V/A of each (cell, face) slot comes from a table built once per
// mesh by the same division.
// ---------------------------------------------------------------------------
template <int D, bool PRE, class A>
__device__ __forceinline__ double cell_dt_inv(A &ar, const fvh_mesh_view &m, int c,
                                              const double *v, double a,
                                              const double *__restrict__ slot_dx) {
  const double vol = PRE ? 0.0 : m.cell_volume[c];
  double dt_inv = 0;
  const int q0 = m.cell_face_offsets[c], q1 = m.cell_face_offsets[c + 1];
  constexpr int U = A::wide_issue ? 1 : 4;
#pragma unroll U
  for (int q = q0; q < q1; ++q) {
    int f = m.cell_faces[q];
    f = f < 0 ? ~f : f;
    double n[D];
#pragma unroll
    for (int i = 0; i < D; ++i) n[i] = m.face_normal[i][f];
    const double delta_x = PRE ? slot_dx[q] : ar.quo(vol, m.face_area[f]);
    fp64_products<A> pp{ar};
    const double dti = ar.quo(a + absval(dot<D>(pp, v, n)), delta_x);
    dt_inv = smax(dti, dt_inv);
  }
  return dt_inv;
}

// the same, evaluated again with the FP64 instructions where an operand is rare
template <int D, bool PRE>
__device__ __forceinline__ double cell_dt_inv_any(const fvh_mesh_view &m, int c, const double *v,
                                                  double a, const double *__restrict__ slot_dx) {
  arith_opt ar;
  const double r = cell_dt_inv<D, PRE>(ar, m, c, v, a, slot_dx);
  if (!ar.rare) return r;
  arith_hw hw;
  return cell_dt_inv<D, PRE>(hw, m, c, v, a, slot_dx);
}

// With has_src the state is read from src (e.g. host-mapped planes of a caller
// that holds its state in host memory) and stored into s as it goes, all but
// the temperature, which no kernel of the step reads.
template <int D, bool PRE>
__global__ void __launch_bounds__(kDtThreads)
dt_partial_kernel(const fvh_mesh_view m, const fvh_state_view s, double *partial,
                  const double *__restrict__ slot_dx, const fvh_state_view src, int has_src) {
  double dt_inv = 0;
  for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < m.num_cells;
       c += gridDim.x * blockDim.x) {
    if (has_src) {
      s.density[c] = src.density[c];
#pragma unroll
      for (int i = 0; i < D; ++i) s.velocity[i][c] = src.velocity[i][c];
      s.internal_energy[c] = src.internal_energy[c];
      s.pressure[c] = src.pressure[c];
      s.sound_speed[c] = src.sound_speed[c];
    }
    double v[D];
#pragma unroll
    for (int i = 0; i < D; ++i) v[i] = s.velocity[i][c];
    // the reference's running maximum over cells and faces, taken cell by
    // cell (a maximum of maxima: the same value)
    dt_inv = smax(cell_dt_inv_any<D, PRE>(m, c, v, s.sound_speed[c], slot_dx), dt_inv);
  }
  dt_inv = block_max(dt_inv);
  if (threadIdx.x == 0) partial[blockIdx.x] = dt_inv;
}

// dt = min(CFL / maximum, t_f - t)
__device__ __forceinline__ void write_dt(double dt_inv, double cfl, double final_time,
                                         const double *soln_time, double *dt_out,
                                         fvh_device_status *status) {
  const double max_dt = final_time - soln_time[0];
  if (le0(dt_inv)) {
    atomicMin(status, status_key(0, FVH_ERR_INFINITE_DT));
    dt_out[0] = 0;
  } else {
    double time_step = __ddiv_rn(1, dt_inv);
    time_step = __dmul_rn(time_step, cfl);
    dt_out[0] = smin(time_step, max_dt);
  }
}

__global__ void __launch_bounds__(kDtThreads)
dt_final_kernel(const double *partial, int nblocks, fvh_params p, const double *soln_time,
                double *dt_out, fvh_device_status *status, unsigned long long *maximum) {
  double dt_inv = 0;
  for (int i = threadIdx.x; i < nblocks; i += blockDim.x) dt_inv = smax(partial[i], dt_inv);
  dt_inv = block_max(dt_inv);
  if (threadIdx.x == 0) {
    write_dt(dt_inv, p.cfl, p.final_time, soln_time, dt_out, status);
    if (maximum) *maximum = 0ull;  // (a run that failed half-way may have left one)
  }
}

// Inside a run the last update of a step also takes the CFL maximum of the new
// state (next_dt::maximum, the order of positive doubles is that of their
// bits, and a NaN ranks above them all), and the first kernel of the following
// step, which does not read dt, turns it into dt and clears it.
constexpr unsigned long long kInfinity = 0x7ff0000000000000ull;
__device__ __forceinline__ unsigned block_index() { return blockIdx.y * gridDim.x + blockIdx.x; }
__device__ __forceinline__ void finish_dt(const next_dt &nd) {
  if (!nd.maximum || block_index() != 0 || threadIdx.x != 0) return;
  const unsigned long long max_bits = *nd.maximum;
  if (max_bits > kInfinity) return;  // (left to redo_dt)
  *nd.maximum = 0ull;
  write_dt(__longlong_as_double((long long)max_bits), nd.cfl, nd.final_time, nd.soln_time, nd.dt,
           nd.status);
}
// Whether it was a NaN, asked in the fluxes kernels by their first nd.nblocks
// blocks: all of these find the NaN, or a number or the zero it is cleared to.
__device__ __forceinline__ bool carried_nan(const next_dt &nd) {
  return nd.maximum && block_index() < (unsigned)nd.nblocks &&
         *(const volatile unsigned long long *)nd.maximum > kInfinity;
}

// The maximum of dt_partial_kernel's or dt_final_kernel's block of kDtThreads
// threads, of which this block, of any whole number of warps, takes one warp
// after another: value(i) is what its thread i holds.  Valid in thread 0.
template <class V>
__device__ __forceinline__ double dt_block_max(V value) {
  constexpr int NW = kDtThreads / 32;
  __shared__ double warps[NW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll 1
  for (int w = warp; w < NW; w += blockDim.x >> 5) {
    const double v = warp_max(value(32 * w + lane));
    if (lane == 0) warps[w] = v;
  }
  __syncthreads();
  const double v = warp == 0 ? warp_max(lane < NW ? warps[lane] : 0.0) : 0.0;
  __syncthreads();
  return v;
}

// dt of a state with NaNs.  A maximum in the reference's order (a < b ? b : a)
// keeps a NaN or drops it by the place where it stands, so the cells are folded
// exactly as the two dt kernels fold them: the first blocks of the grid take
// dt_partial_kernel's blocks, and the last of them to finish does
// dt_final_kernel's work.  All threads of those blocks call it; nothing waits for
// another block.
template <int D>
__device__ __noinline__ void redo_dt(const fvh_mesh_view &m, const fvh_state_view &s,
                                     const next_dt &nd) {
  __shared__ bool last;
  const unsigned blocks = min(gridDim.x * gridDim.y, (unsigned)nd.nblocks);
  for (unsigned b = block_index(); b < (unsigned)nd.nblocks; b += blocks) {
    const double dt_inv = dt_block_max([&](int i) {
      double most = 0;
      for (int c = b * kDtThreads + i; c < m.num_cells; c += nd.nblocks * kDtThreads) {
        double v[D];
#pragma unroll
        for (int j = 0; j < D; ++j) v[j] = s.velocity[j][c];
        arith_hw hw;
        most = smax(cell_dt_inv<D, true>(hw, m, c, v, s.sound_speed[c], nd.slot_dx), most);
      }
      return most;
    });
    if (threadIdx.x == 0) nd.partial[b] = dt_inv;
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) last = atomicInc(nd.done, blocks - 1) == blocks - 1;  // (back to zero)
  __syncthreads();
  if (!last) return;
  __threadfence();
  const double dt_inv = dt_block_max([&](int i) {
    double most = 0;
    for (int b = i; b < nd.nblocks; b += kDtThreads) most = smax(__ldcg(nd.partial + b), most);
    return most;
  });
  if (threadIdx.x == 0) {
    *nd.maximum = 0ull;
    write_dt(dt_inv, nd.cfl, nd.final_time, nd.soln_time, nd.dt, nd.status);
  }
}
__device__ __forceinline__ void add_to_maximum(const next_dt &nd, double dt_inv) {
  unsigned lo, hi;
  sf64::halves(dt_inv, lo, hi);
  if (is_nan(lo, hi)) atomicMax(nd.maximum, kInfinity + 1);
  dt_inv = block_max(dt_inv);
  if (threadIdx.x == 0 && lt(0.0, dt_inv))
    atomicMax(nd.maximum, (unsigned long long)__double_as_longlong(dt_inv));
}

// ---------------------------------------------------------------------------
// Geometry-only tables built once per mesh for the solver (same operations in
// the same order as the on-the-fly code, so the values are identical).
// ---------------------------------------------------------------------------
// lsq record per cell: 2D (a00 a01 a11 denom); 3D (a00 a01 a02 a11 a12 a22
// min1 min2 min3 denom), tasks.h:210-228 and :250-261
template <int D>
struct lsq_width {
  static constexpr int value = D == 2 ? 4 : 10;
};

template <int D, class A>
__device__ __forceinline__ void lsq_matrix(A &ar, const fvh_mesh_view &m, int c0, double *r) {
  double x0[D];
#pragma unroll
  for (int i = 0; i < D; ++i) x0[i] = m.cell_centroid[i][c0];
  double dxdx[6] = {0, 0, 0, 0, 0, 0};
  for (int q = m.cell_nbr_offsets[c0]; q < m.cell_nbr_offsets[c0 + 1]; ++q) {
    const int c1 = m.cell_nbrs[q];
    double dx[D];
#pragma unroll
    for (int d = 0; d < D; ++d) dx[d] = m.cell_centroid[d][c1] - x0[d];
    if (D == 2) {
      dxdx[0] += ar.mul(dx[0], dx[0]);
      dxdx[1] += ar.mul(dx[0], dx[1]);
      dxdx[2] += ar.mul(dx[1], dx[1]);
    } else {
      dxdx[0] += ar.mul(dx[0], dx[0]);
      dxdx[1] += ar.mul(dx[0], dx[1]);
      dxdx[2] += ar.mul(dx[0], dx[D - 1]);
      dxdx[3] += ar.mul(dx[1], dx[1]);
      dxdx[4] += ar.mul(dx[1], dx[D - 1]);
      dxdx[5] += ar.mul(dx[D - 1], dx[D - 1]);
    }
  }
  if (D == 2) {
    r[0] = dxdx[0];
    r[1] = dxdx[1];
    r[2] = dxdx[2];
    r[3] = ar.quo(1, ar.mul(dxdx[0], dxdx[2]) - ar.mul(dxdx[1], dxdx[1]));
  } else {
    const double a00 = dxdx[0], a01 = dxdx[1], a02 = dxdx[2], a11 = dxdx[3],
                 a12 = dxdx[4], a22 = dxdx[5];
    const double min1 = ar.mul(a11, a22) - ar.mul(a12, a12);
    const double min2 = ar.mul(a01, a22) - ar.mul(a12, a02);
    const double min3 = ar.mul(a01, a12) - ar.mul(a11, a02);
    for (int k = 0; k < 6; ++k) r[k] = dxdx[k];
    r[6] = min1;
    r[7] = min2;
    r[8] = min3;
    r[9] = ar.quo(1, ar.mul(a00, min1) - ar.mul(a01, min2) + ar.mul(a02, min3));
  }
}

// notes an offset that is neither zero nor within 2^+-500 (take_entry)
__device__ __forceinline__ void note_odd(double x, unsigned *odd) {
  unsigned rare = 0;
  sf64::take(x, rare);
  if (rare) atomicOr(odd, 1u);
}

template <int D>
__global__ void cell_tables_kernel(const fvh_mesh_view m, double *lsq, double *slot_dx,
                                   double *nbr_dx, double *vtx_dx, unsigned *odd) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= m.num_cells) return;
  arith_hw hw;  // set-up, once per mesh
  constexpr int W = lsq_width<D>::value;
  double r[W];
  lsq_matrix<D>(hw, m, c, r);
#pragma unroll
  for (int k = 0; k < W; ++k) lsq[(size_t)k * m.num_cells + c] = r[k];
  const double vol = m.cell_volume[c];
  for (int q = m.cell_face_offsets[c]; q < m.cell_face_offsets[c + 1]; ++q) {
    int f = m.cell_faces[q];
    f = f < 0 ? ~f : f;
    slot_dx[q] = hw.quo(vol, m.face_area[f]);
  }
  double x0[D];
#pragma unroll
  for (int i = 0; i < D; ++i) x0[i] = m.cell_centroid[i][c];
  for (int q = m.cell_nbr_offsets[c]; q < m.cell_nbr_offsets[c + 1]; ++q) {
    const int c1 = m.cell_nbrs[q];
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const double dx = m.cell_centroid[d][c1] - x0[d];
      nbr_dx[(size_t)q * D + d] = dx;
      note_odd(dx, odd);
    }
  }
  const int r0 = m.cell_vertex_offsets[c], r1 = m.cell_vertex_offsets[c + 1];
  if (r0 == r1) atomicOr(odd, 1u);  // a cell without vertices (limiter_side)
  for (int q = r0; q < r1; ++q) {
    const int v = m.cell_vertices[q];
#pragma unroll
    for (int d = 0; d < D; ++d) vtx_dx[(size_t)q * D + d] = m.vertex_coord[d][v] - x0[d];
  }
}

template <int D>
__global__ void face_tables_kernel(const fvh_mesh_view m, double *face_dx, unsigned *odd) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.num_faces) return;
  const int2 cc = reinterpret_cast<const int2 *>(m.face_cells)[f];
#pragma unroll
  for (int side = 0; side < 2; ++side) {
    const int c = side == 0 ? cc.x : cc.y;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      const double dx = c >= 0 ? m.face_centroid[i][f] - m.cell_centroid[i][c] : 0.0;
      face_dx[(size_t)f * 2 * D + side * D + i] = dx;
      note_odd(dx, odd);
    }
  }
}

// ---------------------------------------------------------------------------
// gradients + Barth-Jespersen vertex limiter (tasks.h:145-321)
// With PRE the geometry-only terms (matrix, neighbour and vertex offsets) come
// from the solver's tables.
// ---------------------------------------------------------------------------
template <int D>
__device__ __forceinline__ void load_dx(const double *__restrict__ p, double *dx) {
  if (D == 2) {
    const double2 v = __ldg(reinterpret_cast<const double2 *>(p));
    dx[0] = v.x;
    dx[D - 1] = v.y;
  } else {
#pragma unroll
    for (int d = 0; d < D; ++d) dx[d] = __ldg(p + d);
  }
}

// Plane k of the reconstructed variables (d, v.., e, p, a) of a state, and the
// planes of its gradient.  Both views hold their plane pointers one after another,
// so a variable that is only known at run time is an index.
template <int D>
__device__ __forceinline__ const double *state_plane_at(const fvh_state_view &s, int k) {
  // density, velocity[3], internal_energy, pressure, temperature, sound_speed
  return reinterpret_cast<const double *const *>(&s)[k <= D ? k : k == D + 3 ? 7 : k + 3 - D];
}
template <int D>
__device__ __forceinline__ double *const *grad_planes_at(const fvh_gradient_view &g, int k) {
  // density[3], velocity[3][3], internal_energy[3], pressure[3], sound_speed[3]
  return reinterpret_cast<double *const *>(&g) + 3 * (k <= D ? k : k + 3 - D);
}
static_assert(sizeof(fvh_state_view) == 8 * sizeof(double *) &&
                  sizeof(fvh_gradient_view) == 21 * sizeof(double *),
              "plane pointers stand one after another");

template <int D, bool PRE>
__device__ __forceinline__ void vertex_offset(const fvh_mesh_view &m, const tables &t, int rr,
                                              const double *x0, double *dxv) {
  if (PRE) {
    load_dx<D>(t.vtx_dx + (size_t)rr * D, dxv);
  } else {
    const int vtx = m.cell_vertices[rr];
#pragma unroll
    for (int i = 0; i < D; ++i) dxv[i] = m.vertex_coord[i][vtx] - x0[i];
  }
}

// The limiter factor phi of one variable (tasks.h:267-299) with the reference's
// arithmetic: u0 and the gradient g of cell c0, `plane` the variable's values.
// Out of line: the kernel calls it only where its FP32 bounds do not decide.
//
// phi = min over vertices of (umax-u0)/du or (umin-u0)/du.  Correctly rounded
// division is monotone in the divisor, so only the largest du > tol and the
// smallest du < -tol can set the minimum; the result equals the reference's
// per-vertex minimum.
template <int D, bool PRE>
__device__ __noinline__ double limiter_exact(const fvh_mesh_view &m, const tables &t,
                                             const double *plane, int c0, double u0,
                                             double g0, double g1, double g2) {
  constexpr double tol = 1.e-9;
  const long long ktol = okey(tol), kntol = okey(-tol);
  const double g[3] = {g0, g1, g2};
  double x0[D];
  if (!PRE) {
#pragma unroll
    for (int i = 0; i < D; ++i) x0[i] = m.cell_centroid[i][c0];
  }
  long long kpos = 0, kneg = 0;
  const int r0 = m.cell_vertex_offsets[c0], r1 = m.cell_vertex_offsets[c0 + 1];
#pragma unroll 1
  for (int rr = r0; rr < r1; ++rr) {
    double dxv[D];
    vertex_offset<D, PRE>(m, t, rr, x0, dxv);
    double u1 = u0;
#pragma unroll
    for (int i = 0; i < D; ++i) u1 += __dmul_rn(dxv[i], g[i]);
    const long long kd = okey(u1 - u0);
    if (kd > ktol) kpos = (kpos < kd) ? kd : kpos;
    else if (kd < kntol) kneg = (kd < kneg) ? kd : kneg;
  }
  long long kphi = okey(1.0);
  if (kpos > ktol || kneg < kntol) {
    // the neighbour extrema umin / umax (tasks.h:232-236)
    long long kmin = okey(u0), kmax = kmin;
    const int q0 = m.cell_nbr_offsets[c0], q1 = m.cell_nbr_offsets[c0 + 1];
#pragma unroll 4
    for (int q = q0; q < q1; ++q) {
      const long long k1 = okey(plane[m.cell_nbrs[q]]);
      kmin = (k1 < kmin) ? k1 : kmin;  // std::min(u1, umin)
      kmax = (kmax < k1) ? k1 : kmax;  // std::max(u1, umax)
    }
    // RN(N / du) >= 1 exactly when |N| >= |du| (N and du of one sign, du
    // normal), so the quotient is formed only when it can lower phi below 1
    if (kpos > ktol) {
      const double num = from_okey(kmax) - u0;
      if (okey(num) < kpos) {
        const long long kq = okey(__ddiv_rn(num, from_okey(kpos)));
        kphi = (kq < kphi) ? kq : kphi;
      }
    }
    if (kneg < kntol) {
      const double num = from_okey(kmin) - u0;
      if (okey(num) > kneg) {
        const long long kq = okey(__ddiv_rn(num, from_okey(kneg)));
        kphi = (kq < kphi) ? kq : kphi;
      }
    }
  }
  kphi = (kphi < 0) ? 0 : kphi;  // std::max(phi, 0)
  return from_okey(kphi);
}

// x truncated to FP32 (relative error below 2^-23; 0 for |x| < 2^-60); `wide`
// collects whether |x| >= 2^60 or x is a NaN.
__device__ __forceinline__ float truncated(double x, unsigned &wide) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  const unsigned h = hi & 0x7fffffffu;
  wide |= (unsigned)(h >= (1083u << 20));
  const unsigned mag = __funnelshift_l(lo, h - (896u << 20), 3);
  return __uint_as_float(h < (963u << 20) ? 0u : mag | (hi & 0x80000000u));
}

// Order key of the high half of a double: for differences it finds the largest
// and smallest up to 20 bits of their significands.
__device__ __forceinline__ int high_key(double x) {
  unsigned lo, hi;
  sf64::halves(x, lo, hi);
  return (int)(hi ^ (unsigned)(((int)hi >> 31) & 0x7fffffff));
}
// A lower bound in FP32 of the magnitude whose high half is h (0 for an
// infinity or a NaN, which bound nothing).
__device__ __forceinline__ float at_least(unsigned h) {
  const unsigned f = (h - (896u << 20)) << 3;
  return __uint_as_float(h < (897u << 20) || h >= 0x7ff00000u ? 0u
                         : h >= (1150u << 20)                 ? 0x7f000000u
                                                              : f);
}

struct side_limit {
  long long key;
  unsigned rare;
};

// Whether the sides that FP32 does not decide are taken one by one (limiter_side)
// or both in limiter_exact.  In 3D without tables each pass gathers the offsets of
// eight vertices again, and two passes a side cost more than the FP64 sums they
// save (us, sides and exact: uniform mesh with waves, 28^3 218 and 182, 36^3 272
// and 239, 54x83x48 851 and 840, 80^3 1,907 and 1,813; jittered 184 and 183, 238
// and 238, 795 and 836, 1,777 and 1,807; before the FP32 bounds 213, 258, 879 and
// 1,892).  In 2D the sides win where there are many (800^2 367 and 382).
template <int D, bool PRE>
constexpr bool limit_by_sides() { return PRE || D == 2; }

// What one side of the limiter allows a variable whose largest vertex
// difference above u0 (UP, below u0 otherwise) may exceed the room that the
// neighbours leave: the order key of min(1, (umax-u0)/du) or of
// min(1, (umin-u0)/du).  g32 and E are the FP32 gradient and error bound of
// cell_gradients: a vertex whose FP32 difference is more than 2 E below the
// largest cannot be the largest, so the reference's arithmetic runs at the
// largest one and at those within 2 E of it, with products and the quotient on
// the integer pipes.  `rare` notes operands these leave to the hardware.
template <int D, bool PRE, bool UP>
__device__ __noinline__ side_limit limiter_side(const fvh_mesh_view &m, const tables &t,
                                                const double *plane, int c0,
                                                double u0, double g0, double g1, double g2,
                                                float E) {
  const double g[3] = {g0, g1, g2};
  unsigned wide = 0, rare = 0;
  float gf[D];
#pragma unroll
  for (int i = 0; i < D; ++i) gf[i] = UP ? truncated(g[i], wide) : -truncated(g[i], wide);
  double x0[D];
  if (!PRE) {
#pragma unroll
    for (int i = 0; i < D; ++i) x0[i] = m.cell_centroid[i][c0];
  }
  const int r0 = m.cell_vertex_offsets[c0], r1 = m.cell_vertex_offsets[c0 + 1];
  auto estimate = [&](int rr) {
    double dxv[D];
    vertex_offset<D, PRE>(m, t, rr, x0, dxv);
    float du = __fmul_rn(truncated(dxv[0], wide), gf[0]);
#pragma unroll
    for (int i = 1; i < D; ++i) du = __fmaf_rn(truncated(dxv[i], wide), gf[i], du);
    return du;
  };
  long long kbest = 0;
  auto exact = [&](int rr) {
    double dxv[D];
    vertex_offset<D, PRE>(m, t, rr, x0, dxv);
    double u1 = u0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      const flagged p = mul_call(dxv[i], g[i]);
      rare |= p.rare;
      u1 += p.q;
    }
    const long long kd = okey(u1 - u0);
    kbest = (UP ? kbest < kd : kd < kbest) ? kd : kbest;
  };
  int best = r0;
  float top = -1.f, next = -1.f;  // the two largest estimates (of those above 0)
#pragma unroll 1
  for (int rr = r0; rr < r1; ++rr) {
    const float du = estimate(rr);
    next = fmaxf(next, fminf(du, top));
    if (du > top) {
      top = du;
      best = rr;
    }
  }
  exact(best);
  const float near = top - 2.0001f * E;
  if (next >= near) {
#pragma unroll 1
    for (int rr = r0; rr < r1; ++rr)
      if (rr != best && estimate(rr) >= near) exact(rr);
  }
  constexpr double tol = 1.e-9;
  const long long one = okey(1.0);
  if (UP ? !(kbest > okey(tol)) : !(kbest < okey(-tol))) return {one, rare};
  long long kn = okey(u0);
  const int q0 = m.cell_nbr_offsets[c0], q1 = m.cell_nbr_offsets[c0 + 1];
#pragma unroll 4
  for (int q = q0; q < q1; ++q) {
    const long long k1 = okey(plane[m.cell_nbrs[q]]);
    kn = (UP ? kn < k1 : k1 < kn) ? k1 : kn;
  }
  const double num = from_okey(kn) - u0;
  if (UP ? !(okey(num) < kbest) : !(okey(num) > kbest)) return {one, rare};  // (see limiter_exact)
  const flagged f = div_call(num, from_okey(kbest));
  rare |= f.rare;
  const long long kq = okey(f.q);
  return {kq < one ? kq : one, rare};
}

// closed-form solve of the least-squares system from the sums b (tasks.h:238-262)
template <class A>
__device__ __forceinline__ void solve(A &ar, const double (&r)[4], const double (&b)[2],
                                      double (&g)[2]) {
  const auto a00 = ar.take(r[0]), a01 = ar.take(r[1]), a11 = ar.take(r[2]), den = ar.take(r[3]);
  const auto b0 = ar.take(b[0]), b1 = ar.take(b[1]);
  g[0] = ar.prod(ar.take(ar.prod(b0, a11) - ar.prod(b1, a01)), den);
  g[1] = ar.prod(ar.take(ar.prod(b1, a00) - ar.prod(b0, a01)), den);
}
// 3D: products of the same two operands are formed once
template <class A>
__device__ __forceinline__ void solve(A &ar, const double (&r)[10], const double (&b)[3],
                                      double (&g)[3]) {
  const auto a00 = ar.take(r[0]), a01 = ar.take(r[1]), a02 = ar.take(r[2]), a11 = ar.take(r[3]),
             a12 = ar.take(r[4]), a22 = ar.take(r[5]), den = ar.take(r[9]);
  const auto b0 = ar.take(b[0]), b1 = ar.take(b[1]), b2 = ar.take(b[2]);
  const double b1a12 = ar.prod(b1, a12), b2a11 = ar.prod(a11, b2);
  const auto s = ar.take(ar.prod(b1, a22) - ar.prod(a12, b2));
  const auto u = ar.take(ar.prod(b2, a01) - ar.prod(a02, b1));
  g[0] = ar.prod(ar.take(ar.prod(b0, ar.take(r[6])) - ar.prod(a01, s) +
                         ar.prod(a02, ar.take(b1a12 - b2a11))), den);
  g[1] = ar.prod(ar.take(ar.prod(a00, s) - ar.prod(b0, ar.take(r[7])) + ar.prod(a02, u)), den);
  g[2] = ar.prod(ar.take(ar.prod(a00, ar.take(b2a11 - b1a12)) - ar.prod(a01, u) +
                         ar.prod(b0, ar.take(r[8]))), den);
}

// The limited gradients gu of cell c0 for the NK reconstructed variables from
// k0 on (of d, v.., e, p, a); r: the cell's least-squares terms (read from the
// table with PRE).  Each variable's gradient and limiter depend on that variable alone, so the
// variables are taken in groups, each in its own pass over the neighbours.
//
// The limiter is decided in FP32 where FP32 can decide it: with every vertex
// difference du within E of its FP32 estimate, a variable is not limited when
// du <= tol, or du <= umax - u0 (RN(umax - u0) is the largest neighbour
// difference, of which the key of the high half gives a lower bound), and
// likewise below; phi is then 1 exactly.  The other variables take limiter_side
// or limiter_exact.  In flows that are smooth or at rest up to rounding nearly
// all are decided, which saves their vertex products and sums and the second
// pass over the neighbours.
template <int D, int NK, bool LIMIT, bool PRE>
__device__ __forceinline__ void cell_gradients(arith_opt &ar, const fvh_mesh_view &m,
                                               const fvh_state_view &s, const tables &t, int c0,
                                               int k0, const double (&r)[lsq_width<D>::value],
                                               double (&gu)[NK][D]) {
  double x0[D];
  if (!PRE) {
#pragma unroll
    for (int i = 0; i < D; ++i) x0[i] = m.cell_centroid[i][c0];
  }
  const double *plane[NK];
  double u0[NK], dudx[NK][D];
  int kmax[NK], kmin[NK];
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    plane[k] = state_plane_at<D>(s, k0 + k);
    u0[k] = plane[k][c0];
    kmax[k] = kmin[k] = 0;
#pragma unroll
    for (int j = 0; j < D; ++j) dudx[k][j] = 0;
  }
  const int q0 = m.cell_nbr_offsets[c0], q1 = m.cell_nbr_offsets[c0 + 1];
  auto neighbour = [&](int q, bool first) {
    const int c1 = m.cell_nbrs[q];
    double du[NK], dx[D];
#pragma unroll
    for (int k = 0; k < NK; ++k) du[k] = plane[k][c1];
    if (PRE) {
      load_dx<D>(t.nbr_dx + (size_t)q * D, dx);
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d) dx[d] = m.cell_centroid[d][c1] - x0[d];
    }
    bool same = true;
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      du[k] -= u0[k];
      same = same && is_zero(du[k]);
      if (LIMIT) {
        const int key = high_key(du[k]);
        kmax[k] = max(kmax[k], key);
        kmin[k] = min(kmin[k], key);
      }
    }
    // a neighbour equal to the cell in every variable adds (+-0) * dx = +-0 to
    // each sum, which leaves it as it is: cells inside a uniform region skip it
    if (same) return;
    sf64::parts px[D];
#pragma unroll
    for (int j = 0; j < D; ++j) px[j] = PRE ? ar.take_entry(dx[j]) : ar.take(dx[j]);
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      const auto pu = ar.take(du[k]);
#pragma unroll
      for (int j = 0; j < D; ++j) {
        if (first)
          ar.add_first(dudx[k][j], pu, px[j]);
        else
          ar.add(dudx[k][j], pu, px[j]);
      }
    }
  };
  if (q0 < q1) neighbour(q0, true);
#pragma unroll 1
  for (int q = q0 + 1; q < q1; ++q) neighbour(q, false);
  {
    double lsq[lsq_width<D>::value];
#pragma unroll
    for (int w = 0; w < lsq_width<D>::value; ++w)
      lsq[w] = PRE ? t.lsq[(size_t)w * m.num_cells + c0] : r[w];
#pragma unroll
    for (int k = 0; k < NK; ++k) solve(ar, lsq, dudx[k], gu[k]);
  }
  if (!LIMIT) return;
  float gf[NK][D], top[NK], low[NK], reach[D];
  unsigned wide[NK], far = 0;
#pragma unroll
  for (int i = 0; i < D; ++i) reach[i] = 0.f;
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    wide[k] = 0;
    top[k] = low[k] = 0.f;
#pragma unroll
    for (int i = 0; i < D; ++i) gf[k][i] = truncated(gu[k][i], wide[k]);
  }
  const int r0 = m.cell_vertex_offsets[c0], r1 = m.cell_vertex_offsets[c0 + 1];
#pragma unroll 1
  for (int rr = r0; rr < r1; ++rr) {
    double dxv[D];
    float f[D];
    vertex_offset<D, PRE>(m, t, rr, x0, dxv);
#pragma unroll
    for (int i = 0; i < D; ++i) {
      f[i] = truncated(dxv[i], far);
      reach[i] = fmaxf(reach[i], fabsf(f[i]));
    }
#pragma unroll
    for (int k = 0; k < NK; ++k) {
      float du = __fmul_rn(f[0], gf[k][0]);
#pragma unroll
      for (int i = 1; i < D; ++i) du = __fmaf_rn(f[i], gf[k][i], du);
      top[k] = fmaxf(top[k], du);
      low[k] = fminf(low[k], du);
    }
  }
  // E: truncating g and dx and the FP32 roundings move sum |dx g| by less than
  // 2^-21 of itself; values below 2^-60 taken as zero; the reference's own
  // roundings about u0 by less than 2^-50 |u0|.  Each term is taken double.
  // (A cell without vertices, which a mesh with tables does not have, is free.)
  float tiny = !PRE && r0 == r1 ? -INFINITY : 1e-30f;
#pragma unroll
  for (int i = 0; i < D; ++i) tiny = __fmaf_rn(reach[i], 0x1p-59f, tiny);
#pragma unroll
  for (int k = 0; k < NK; ++k) {
    float E = __fmaf_rn(fabsf(truncated(u0[k], wide[k])), 0x1p-49f, tiny);
#pragma unroll
    for (int i = 0; i < D; ++i)
      E = __fmaf_rn(__fmaf_rn(reach[i], 0x1p-20f, 0x1p-59f), fabsf(gf[k][i]), E);
    const float up = top[k] + E, down = E - low[k];
    const float room = at_least((unsigned)kmax[k]);
    const float floor = at_least((unsigned)~kmin[k] & 0x7fffffffu);
    constexpr float tol = 0.9999e-9f;
    const bool free_up = up <= tol || up <= room, free_down = down <= tol || down <= floor;
    unsigned odd = wide[k] | far;
    if (free_up && free_down && !odd) continue;
    long long kphi = okey(1.0);
    const double *gk = gu[k];
    if (limit_by_sides<D, PRE>() && !odd) {
      if (!free_up) {
        const side_limit l = limiter_side<D, PRE, true>(m, t, plane[k], c0, u0[k], gk[0], gk[1],
                                                        gk[D - 1], E);
        kphi = l.key;
        odd = l.rare;
      }
      if (!free_down) {
        const side_limit l = limiter_side<D, PRE, false>(m, t, plane[k], c0, u0[k], gk[0], gk[1],
                                                         gk[D - 1], E);
        kphi = l.key < kphi ? l.key : kphi;
        odd |= l.rare;
      }
      kphi = (kphi < 0) ? 0 : kphi;  // std::max(phi, 0)
    }
    if (!limit_by_sides<D, PRE>() || odd)
      kphi = okey(limiter_exact<D, PRE>(m, t, plane[k], c0, u0[k], gk[0], gk[1], gk[D - 1]));
    if (kphi != okey(1.0)) {
      const auto phi = ar.take(from_okey(kphi));
#pragma unroll
      for (int i = 0; i < D; ++i) gu[k][i] = ar.prod(ar.take(gu[k][i]), phi);
    }
  }
}

template <int D, int NK>
__device__ __forceinline__ void store_gradients(const fvh_gradient_view &g, int c0, int k0,
                                                const double (&gu)[NK][D]) {
#pragma unroll
  for (int k = 0; k < NK; ++k)
#pragma unroll
    for (int i = 0; i < D; ++i) grad_planes_at<D>(g, k0 + k)[i][c0] = gu[k][i];
}

// The limited gradient of variable k of cell c0 with the FP64 instructions,
// stored: the reference's arithmetic in as short a chain as it has.  The vertex
// offsets are read ahead, the neighbour extrema taken beside the sums, and every
// vertex tested (limiter_exact says why the extreme differences suffice).
// `ready` is called between reading the cell's lists and offsets and its state.
template <int D, bool LIMIT, bool PRE, class READY>
__device__ __forceinline__ void gradient_fp64(const fvh_mesh_view &m, const fvh_state_view &s,
                                              const fvh_gradient_view &g, const tables &t, int c0,
                                              int k, READY ready) {
  arith_hw hw;
  const int q0 = m.cell_nbr_offsets[c0], q1 = m.cell_nbr_offsets[c0 + 1];
  const int r0 = LIMIT ? m.cell_vertex_offsets[c0] : 0, r1 = LIMIT ? m.cell_vertex_offsets[c0 + 1] : 0;
  double x0[D], r[lsq_width<D>::value];
  if (!PRE) {
#pragma unroll
    for (int i = 0; i < D; ++i) x0[i] = m.cell_centroid[i][c0];
  }
  constexpr int AHEAD = D == 2 ? 4 : 8;
  double ahead[AHEAD][D];
  if (LIMIT) {
#pragma unroll
    for (int v = 0; v < AHEAD; ++v)
      if (r0 + v < r1) vertex_offset<D, PRE>(m, t, r0 + v, x0, ahead[v]);
  }
  if (PRE) {
#pragma unroll
    for (int w = 0; w < lsq_width<D>::value; ++w) r[w] = t.lsq[(size_t)w * m.num_cells + c0];
  }
  constexpr int LISTED = 8;
  int listed[LISTED];
#pragma unroll
  for (int i = 0; i < LISTED; ++i) listed[i] = q0 + i < q1 ? m.cell_nbrs[q0 + i] : 0;
  ready();
  const double *plane = state_plane_at<D>(s, k);
  const double u0 = plane[c0];
  double b[D];
#pragma unroll
  for (int j = 0; j < D; ++j) b[j] = 0;
  long long kmin = okey(u0), kmax = kmin;
  auto neighbour = [&](int q, int c1) {
    const double u1 = plane[c1], du = u1 - u0;
    double dx[D];
    if (PRE) {
      load_dx<D>(t.nbr_dx + (size_t)q * D, dx);
    } else {
#pragma unroll
      for (int d = 0; d < D; ++d) dx[d] = m.cell_centroid[d][c1] - x0[d];
    }
#pragma unroll
    for (int j = 0; j < D; ++j) b[j] += __dmul_rn(du, dx[j]);
    if (LIMIT) {
      const long long k1 = okey(u1);
      kmin = (k1 < kmin) ? k1 : kmin;
      kmax = (kmax < k1) ? k1 : kmax;
    }
  };
#pragma unroll
  for (int i = 0; i < LISTED; ++i)
    if (q0 + i < q1) neighbour(q0 + i, listed[i]);
#pragma unroll 4
  for (int q = q0 + LISTED; q < q1; ++q) neighbour(q, m.cell_nbrs[q]);
  if (!PRE) lsq_matrix<D>(hw, m, c0, r);
  double gu[D];
  solve(hw, r, b, gu);
  if (LIMIT) {
    constexpr double tol = 1.e-9;
    const long long ktol = okey(tol), kntol = okey(-tol), one = okey(1.0);
    long long kpos = 0, kneg = 0;
    auto vertex = [&](const double *dxv) {
      double u1 = u0;
#pragma unroll
      for (int i = 0; i < D; ++i) u1 += __dmul_rn(dxv[i], gu[i]);
      const long long kd = okey(u1 - u0);
      if (kd > ktol) kpos = (kpos < kd) ? kd : kpos;
      else if (kd < kntol) kneg = (kd < kneg) ? kd : kneg;
    };
#pragma unroll
    for (int v = 0; v < AHEAD; ++v)
      if (r0 + v < r1) vertex(ahead[v]);
#pragma unroll 1
    for (int rr = r0 + AHEAD; rr < r1; ++rr) {
      double dxv[D];
      vertex_offset<D, PRE>(m, t, rr, x0, dxv);
      vertex(dxv);
    }
    long long kphi = one;
    if (kpos > ktol) {
      const double num = from_okey(kmax) - u0;
      if (okey(num) < kpos) {
        const long long kq = okey(__ddiv_rn(num, from_okey(kpos)));
        kphi = (kq < kphi) ? kq : kphi;
      }
    }
    if (kneg < kntol) {
      const double num = from_okey(kmin) - u0;
      if (okey(num) > kneg) {
        const long long kq = okey(__ddiv_rn(num, from_okey(kneg)));
        kphi = (kq < kphi) ? kq : kphi;
      }
    }
    kphi = (kphi < 0) ? 0 : kphi;  // std::max(phi, 0)
    if (kphi != one) {
#pragma unroll
      for (int i = 0; i < D; ++i) gu[i] = __dmul_rn(gu[i], from_okey(kphi));
    }
  }
#pragma unroll
  for (int i = 0; i < D; ++i) grad_planes_at<D>(g, k)[i][c0] = gu[i];
}

// the FP64 redo of a cell whose operands left the integer-pipe range, out of
// line (it is rare and would otherwise double the kernel's code)
template <int D, int NK, bool LIMIT, bool PRE>
__device__ __noinline__ void gradient_group_hw(const fvh_mesh_view &m, const fvh_state_view &s,
                                               const fvh_gradient_view &g, const tables &t,
                                               int c0, int k0) {
#pragma unroll 1
  for (int k = k0; k < k0 + NK; ++k) gradient_fp64<D, LIMIT, PRE>(m, s, g, t, c0, k, [] {});
}

// the gradients of NK variables from k0 on of cell c0, stored
template <int D, int NK, bool LIMIT, bool PRE>
__device__ __forceinline__ void gradient_group(const fvh_mesh_view &m, const fvh_state_view &s,
                                               const fvh_gradient_view &g, const tables &t,
                                               int c0, int k0,
                                               const double (&r)[lsq_width<D>::value],
                                               unsigned rare) {
  double gu[NK][D];
  arith_opt ar;
  ar.rare = rare;
  cell_gradients<D, NK, LIMIT, PRE>(ar, m, s, t, c0, k0, r, gu);
  if (ar.rare) {
    gradient_group_hw<D, NK, LIMIT, PRE>(m, s, g, t, c0, k0);
    return;
  }
  store_gradients<D, NK>(g, c0, k0, gu);
}

// Blocks of 128 per SM the kernels are compiled for.  2D (1024^2 four-quadrant
// workload, 4 steps): fluxes 7 (72 registers) 4.88 ms against 4.98 with 6 and
// 4.89 with 8; gradients 10 4.74 against 4.77 with 9 and 4.81 with 8 (a flow
// with waves everywhere 5.78, 5.79 and 5.84); update 10 (48 registers).  3D
// (80^3 hex, 2 steps): fluxes 5 (96 registers) 0.311 ms a launch against 0.320
// with 4 and 0.329 with 6; gradients 8 4.02 ms against 4.08 with 7 and 4.18
// with 6; update the compiler's choice.  Gradients without tables: 3D 6.
template <int D>
constexpr int min_blocks() { return D == 2 ? 7 : 5; }
template <int D, bool PRE>
constexpr int grad_min_blocks() { return PRE ? (D == 2 ? 10 : 8) : (D == 2 ? 7 : 6); }
template <int D>
constexpr int update_min_blocks() { return D == 2 ? 10 : 1; }
// Variables of a cell per thread.  The blocks of a cell's groups of variables
// follow one another, so the offsets and lists they share come from memory once
// (1024^2: 255 -> 249 us, with waves 344 -> 338; 32^3 one variable a thread 94 -> 92;
// a whole sweep over the cells per group moved 732 MB instead of 391 at 1024^2).
// Sharing by spans of 32 to 1,520 blocks: 249 to 251 and 96 to 100.  Pairs in 3D
// sweep all cells for one pair and then the next, where the values of 26 neighbours
// count for more than the offsets (80^3, 2 steps 4.03 ms, side by side 4.07).
// In pairs the offsets
// x_nbr - x_c are read and taken apart once for both; one by one gives twice the
// threads, which wins until the chip is full: 10 steps at 360^2 2.58 ms against
// 2.68 in pairs, at 512^2 4.71 and 4.71, at 1024^2 (4 steps) 4.97 and 4.74; in
// 3D 5 steps 2.93 against 2.94 at 44^3, 4.24 against 4.08 at 50^3.  All of a
// cell's variables in one thread: 4.28 ms against 4.08 (80^3, 2 steps); threes
// 4.51.  Without tables a thread takes all of them, as it builds the
// least-squares matrix itself.
constexpr int kSingleCells2D = 262144, kSingleCells3D = 92160;
constexpr bool groups_side_by_side(int dim, int group) { return dim == 2 || group == 1; }

template <int D, bool LIMIT, bool PRE, int G>
__global__ void __launch_bounds__(kCellThreads, grad_min_blocks<D, PRE>())
gradients_kernel(const __grid_constant__ fvh_mesh_view m, const __grid_constant__ fvh_state_view s,
                 const __grid_constant__ fvh_gradient_view g, const __grid_constant__ tables t,
                 const __grid_constant__ next_dt nd) {
  after_previous();
  finish_dt(nd);
  constexpr int NV = D + 4, R = NV % G, NG = PRE ? (NV + G - 1) / G : 1;
  constexpr bool NEXT_TO = groups_side_by_side(D, G);
  const int c0 = (NEXT_TO ? blockIdx.x / NG : blockIdx.x) * blockDim.x + threadIdx.x;
  if (c0 >= m.num_cells) return;
  double r[lsq_width<D>::value];
  arith_opt ar;
  int k0 = (NEXT_TO ? blockIdx.x % NG : blockIdx.y) * G;
  if (!PRE) lsq_matrix<D>(ar, m, c0, r);
#pragma unroll 1
  for (; k0 + G <= NV; k0 += PRE ? NV + 1 : G)
    gradient_group<D, G, LIMIT, PRE>(m, s, g, t, c0, k0, r, ar.rare);
  if constexpr (R != 0)
    if (k0 == NV - R) gradient_group<D, R, LIMIT, PRE>(m, s, g, t, c0, k0, r, ar.rare);
  let_next_start();
}

// Few cells (kFewCells): one variable of one cell per thread (blockIdx.y), with
// the FP64 instructions.
template <int D, bool LIMIT, bool PRE>
__global__ void __launch_bounds__(kFewThreads)
gradients_few_kernel(const __grid_constant__ fvh_mesh_view m,
                     const __grid_constant__ fvh_state_view s,
                     const __grid_constant__ fvh_gradient_view g,
                     const __grid_constant__ tables t, const __grid_constant__ next_dt nd) {
  const int c0 = blockIdx.x * blockDim.x + threadIdx.x;
  if (c0 >= m.num_cells) return;
  gradient_fp64<D, LIMIT, PRE>(m, s, g, t, c0, blockIdx.y, [&] {
    after_previous();
    finish_dt(nd);
  });
  let_next_start();
}

// ---------------------------------------------------------------------------
// face fluxes (tasks.h:385-464)
// ---------------------------------------------------------------------------
template <int D, bool SECOND, bool PRE, class A>
__device__ __forceinline__ prim<D> reconstruct(A &ar, const fvh_state_view &s,
                                               const fvh_gradient_view &g, int c,
                                               const double *dx, bool swap) {
  prim<D> w;
  w.d = s.density[c];
#pragma unroll
  for (int i = 0; i < D; ++i) w.v[i] = s.velocity[i][c];
  w.p = s.pressure[c];
  w.e = s.internal_energy[c];
  w.a = s.sound_speed[c];
  if (SECOND) {
    double *const *gp = swap ? g.internal_energy : g.pressure;
    double *const *ge = swap ? g.pressure : g.internal_energy;
    double gd[D], gv[D][D], gpp[D], gee[D], ga[D];
    unsigned nonzero = 0;
#pragma unroll
    for (int i = 0; i < D; ++i) {
      gd[i] = g.density[i][c];
      nonzero |= (unsigned)!is_zero(gd[i]);
#pragma unroll
      for (int d = 0; d < D; ++d) {
        gv[d][i] = g.velocity[d][i][c];
        nonzero |= (unsigned)!is_zero(gv[d][i]);
      }
      gpp[i] = gp[i][c];
      gee[i] = ge[i][c];
      ga[i] = g.sound_speed[i][c];
      nonzero |= (unsigned)(!is_zero(gpp[i]) | !is_zero(gee[i]) | !is_zero(ga[i]));
    }
    // zero gradients add dx * (+-0) = +-0 to each value (dx is finite), which
    // leaves it as it is unless the value is -0 or a NaN: cells with uniform
    // neighbourhoods skip the products when no value is one of those
    unsigned plain = (unsigned)(ordinary(w.d) & ordinary(w.p) & ordinary(w.e) & ordinary(w.a));
#pragma unroll
    for (int d = 0; d < D; ++d) plain &= (unsigned)ordinary(w.v[d]);
    if (!A::wide_issue || (nonzero | !plain)) {
#pragma unroll
      for (int i = 0; i < D; ++i) {
        // dx is taken apart once for all of its products
        const auto px = PRE ? ar.take_entry(dx[i]) : ar.take(dx[i]);
        auto step = [&](double &u, double gr) { u += ar.prod(px, ar.take(gr)); };
        step(w.d, gd[i]);
#pragma unroll
        for (int d = 0; d < D; ++d) step(w.v[d], gv[d][i]);
        step(w.p, gpp[i]);
        step(w.e, gee[i]);
        step(w.a, ga[i]);
      }
    }
  }
  return w;
}

// x_f - x_c of one side of face f, from the table or on the fly
template <int D, bool PRE>
__device__ __forceinline__ void face_offset(const fvh_mesh_view &m, const double *face_dx,
                                            int f, int side, int c, double *dx) {
  if (PRE) {
    load_dx<D>(face_dx + (size_t)f * 2 * D + side * D, dx);
  } else {
#pragma unroll
    for (int i = 0; i < D; ++i) dx[i] = m.face_centroid[i][f] - m.cell_centroid[i][c];
  }
}

// the area-weighted flux of face f (tasks.h:405-461)
struct at_once {
  __device__ __forceinline__ void operator()() const {}
};
// `ready` is called between reading the face's geometry and its cells' state
template <int D, int KIND, bool SECOND, bool PRE, class A, class READY = at_once>
__device__ __forceinline__ void face_flux(A &ar, const fvh_mesh_view &m,
                                          const fvh_state_view &s, const fvh_gradient_view &g,
                                          int f, int2 cc, bool swap, bool outflow,
                                          const double *face_dx, double *F,
                                          READY ready = READY()) {
  double n[D];
#pragma unroll
  for (int i = 0; i < D; ++i) n[i] = m.face_normal[i][f];
  double dx[D] = {}, dx1[D] = {};
  if (SECOND) face_offset<D, PRE>(m, face_dx, f, 0, cc.x, dx);
  // (many warps: the second offset is read where it is used)
  if (SECOND && !A::wide_issue && cc.y >= 0) face_offset<D, PRE>(m, face_dx, f, 1, cc.y, dx1);
  ready();
  const prim<D> wl = reconstruct<D, SECOND, PRE>(ar, s, g, cc.x, dx, swap);
  if (cc.y >= 0) {
    if (SECOND && A::wide_issue) face_offset<D, PRE>(m, face_dx, f, 1, cc.y, dx1);
    const prim<D> wr = reconstruct<D, SECOND, PRE>(ar, s, g, cc.y, dx1, swap);
    if (KIND == FVH_FLUX_RUSANOV)
      rusanov<D>(ar, wl, wr, n, F);
    else if (KIND == FVH_FLUX_HLLC)
      hllc<D>(ar, wl, wr, n, F);
    else
      hlle<D>(ar, wl, wr, n, F);
  } else if (outflow) {
    phys_flux<D>(ar, wl, n, dot<D>(ar, wl.v, n), total_energy<D>(ar, wl), F);
  } else {
    F[0] = 0;
#pragma unroll
    for (int i = 0; i < D; ++i) F[1 + i] = ar.mul(wl.p, n[i]);
    F[D + 1] = 0;
  }
  const double area = m.face_area[f];
#pragma unroll
  for (int k = 0; k < D + 2; ++k) F[k] = __dmul_rn(F[k], area);
}

template <int D>
__device__ __forceinline__ void store_flux(const fvh_flux_view &fl, int f, const double *F) {
  fl.mass[f] = F[0];
#pragma unroll
  for (int i = 0; i < D; ++i) fl.momentum[i][f] = F[1 + i];
  fl.energy[f] = F[D + 1];
}

// the FP64 redo of a face whose operands left the integer-pipe range, out of
// line
template <int D, int KIND, bool SECOND, bool PRE>
__device__ __noinline__ void face_flux_hw(const fvh_mesh_view &m, const fvh_state_view &s,
                                          const fvh_gradient_view &g, const fvh_flux_view &fl,
                                          int f, int2 cc, int swap, int outflow,
                                          const double *face_dx) {
  double F[D + 2];
  arith_hw hw;
  face_flux<D, KIND, SECOND, PRE>(hw, m, s, g, f, cc, swap != 0, outflow != 0, face_dx, F);
  store_flux<D>(fl, f, F);
}

template <int D, int KIND, bool SECOND, bool PRE>
__global__ void __launch_bounds__(kFaceThreads, min_blocks<D>())
fluxes_kernel(const __grid_constant__ fvh_mesh_view m, const __grid_constant__ fvh_state_view s,
              const __grid_constant__ fvh_gradient_view g, const __grid_constant__ fvh_flux_view fl,
              int swap, int outflow, const double *__restrict__ face_dx,
              const __grid_constant__ next_dt nd) {
  after_previous();
  if (!SECOND) finish_dt(nd);  // (first order has no gradients)
  if (carried_nan(nd)) redo_dt<D>(m, s, nd);
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  if (f >= m.num_faces) return;
  const int2 cc = reinterpret_cast<const int2 *>(m.face_cells)[f];
  double F[D + 2];
  arith_opt ar;
  face_flux<D, KIND, SECOND, PRE>(ar, m, s, g, f, cc, swap != 0, outflow != 0, face_dx, F);
  if (ar.rare) {
    face_flux_hw<D, KIND, SECOND, PRE>(m, s, g, fl, f, cc, swap, outflow, face_dx);
    return;
  }
  let_next_start();
  store_flux<D>(fl, f, F);
}

// Few faces (kFewFaces): with the FP64 instructions.
template <int D, int KIND, bool SECOND, bool PRE>
__global__ void __launch_bounds__(kFewThreads)
fluxes_few_kernel(const __grid_constant__ fvh_mesh_view m, const __grid_constant__ fvh_state_view s,
                  const __grid_constant__ fvh_gradient_view g,
                  const __grid_constant__ fvh_flux_view fl, int swap, int outflow,
                  const double *__restrict__ face_dx, const __grid_constant__ next_dt nd) {
  const int f = blockIdx.x * blockDim.x + threadIdx.x;
  bool nan = false;
  auto ready = [&] {
    after_previous();
    nan = carried_nan(nd);
    if (!SECOND) finish_dt(nd);
  };
  if (f < m.num_faces) {
    double F[D + 2];
    arith_hw hw;
    face_flux<D, KIND, SECOND, PRE>(hw, m, s, g, f, reinterpret_cast<const int2 *>(m.face_cells)[f],
                                    swap != 0, outflow != 0, face_dx, F, ready);
    let_next_start();
    store_flux<D>(fl, f, F);
  } else {
    ready();
  }
  if (nan) redo_dt<D>(m, s, nd);
}

// ---------------------------------------------------------------------------
// gather + conservative update + EOS (tasks.h:589-659)
// ---------------------------------------------------------------------------
// 0 - F or 0 + F: F with that sign, +0 for a zero
__device__ __forceinline__ double signed_flux(double F, bool minus) {
  unsigned lo, hi;
  sf64::halves(F, lo, hi);
  return sf64::join(lo, sf64::is_zero(lo, hi) ? 0u : hi ^ (minus ? 0x80000000u : 0u));
}

// the new state of cell c: w = (d, v.., e, p, T, a^2)
// gm1 = gamma - 1 and ggm1 = gamma * (gamma - 1), rounded once on the host
// exactly as the reference rounds them per cell (euler_eqns.h / ideal_gas.h)
// The lists are read before `ready` is called and the time increment
// delta_t = dt * factor and the state after it.
template <int D, class A, class READY = at_once>
__device__ __forceinline__ void cell_update(A &ar, const fvh_mesh_view &m,
                                            const fvh_flux_view &fl, const fvh_state_view &s,
                                            int c, const double *dt, double factor, double gm1,
                                            double ggm1, double cv, double *w,
                                            READY ready = READY()) {
  double du[D + 2];
#pragma unroll
  for (int k = 0; k < D + 2; ++k) du[k] = 0;
  const int q0 = m.cell_face_offsets[c], q1 = m.cell_face_offsets[c + 1];
  const double vol = m.cell_volume[c];
  auto face = [&](int i, int sf) {
    const int f = sf < 0 ? ~sf : sf;
    double F[D + 2];
    F[0] = fl.mass[f];
#pragma unroll
    for (int i = 0; i < D; ++i) F[1 + i] = fl.momentum[i][f];
    F[D + 1] = fl.energy[f];
    if (i == 0) {  // the first sum, 0 -+ F, is F with its sign
#pragma unroll
      for (int k = 0; k < D + 2; ++k) du[k] = signed_flux(F[k], sf >= 0);
    } else if (A::wide_issue && i == 1) {
      // the update kernel's FP64 pipe is its bound: these sums run on the
      // integer pipe; a - b is a + (-b) exactly
#pragma unroll
      for (int k = 0; k < D + 2; ++k) du[k] = add_call(du[k], sf >= 0 ? -F[k] : F[k]);
    } else if (sf >= 0) {
#pragma unroll
      for (int k = 0; k < D + 2; ++k) du[k] -= F[k];
    } else {
#pragma unroll
      for (int k = 0; k < D + 2; ++k) du[k] += F[k];
    }
  };
  if (A::wide_issue) {
    ready();
#pragma unroll 2
    for (int q = q0; q < q1; ++q) face(q - q0, m.cell_faces[q]);
  } else {
    constexpr int LISTED = 2 * D;
    int listed[LISTED];
#pragma unroll
    for (int i = 0; i < LISTED; ++i) listed[i] = q0 + i < q1 ? m.cell_faces[q0 + i] : 0;
    ready();
#pragma unroll
    for (int i = 0; i < LISTED; ++i)
      if (q0 + i < q1) face(i, listed[i]);
#pragma unroll 1
    for (int q = q0 + LISTED; q < q1; ++q) face(q - q0, m.cell_faces[q]);
  }
  const double scale = ar.quo(__dmul_rn(dt[0], factor), vol);
#pragma unroll
  for (int k = 0; k < D + 2; ++k) du[k] = ar.mul(du[k], scale);
  double vel[D];
#pragma unroll
  for (int i = 0; i < D; ++i) vel[i] = s.velocity[i][c];
  const double den0 = s.density[c];
  const double mass = den0 + du[0];
  const double ener =
      ar.mul(den0, s.internal_energy[c] + ar.half(dot<D>(ar, vel, vel))) + du[D + 1];
  const double inv_mass = ar.quo(1, mass);
#pragma unroll
  for (int i = 0; i < D; ++i) vel[i] = ar.mul(ar.mul(den0, vel[i]) + du[1 + i], inv_mass);
  const double e = ar.mul(ener, inv_mass) - ar.half(dot<D>(ar, vel, vel));
  w[0] = mass;
#pragma unroll
  for (int i = 0; i < D; ++i) w[1 + i] = vel[i];
  w[D + 1] = e;
  w[D + 2] = ar.mul(ar.mul(gm1, mass), e);
  w[D + 3] = cv == 1.0 ? e : ar.quo(e, cv);  // x / 1 == x exactly
  w[D + 4] = ar.mul(ggm1, e);                 // a^2; its root is taken once
}

// FEW (kFewUpdateCells): with the FP64 instructions.  NEXT: the last update of a step that
// another one follows; slot_dx the table of V / A.
template <int D, bool FEW, bool NEXT>
__global__ void __launch_bounds__(FEW ? kFewThreads : kCellThreads, FEW ? 1 : update_min_blocks<D>())
update_kernel(const __grid_constant__ fvh_mesh_view m, const __grid_constant__ fvh_flux_view fl,
              const __grid_constant__ fvh_state_view s, const double *dt, double factor, double gm1,
              double ggm1, double cv, double *soln_time, fvh_device_status *status,
              const __grid_constant__ fvh_state_view out, int has_out,
              const double *__restrict__ slot_dx, const __grid_constant__ next_dt nd) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (!NEXT && c >= m.num_cells) return;
  double dt_inv = 0;
  if (!NEXT || c < m.num_cells) {
    double w[D + 5];
    arith_opt ar;
    if (!FEW) cell_update<D>(ar, m, fl, s, c, dt, factor, gm1, ggm1, cv, w, after_previous);
    if (FEW || ar.rare) {
      arith_hw hw;
      cell_update<D>(hw, m, fl, s, c, dt, factor, gm1, ggm1, cv, w, after_previous);
    }
    if (c == 0) soln_time[0] = 0.0 + soln_time[0] + __dmul_rn(dt[0], factor);
    let_next_start();
    const double a = sqrt(w[D + 4]);
    s.density[c] = w[0];
#pragma unroll
    for (int i = 0; i < D; ++i) s.velocity[i][c] = w[1 + i];
    s.internal_energy[c] = w[D + 1];
    s.pressure[c] = w[D + 2];
    s.temperature[c] = w[D + 3];
    s.sound_speed[c] = a;
    if (has_out) {
      out.density[c] = w[0];
#pragma unroll
      for (int i = 0; i < D; ++i) out.velocity[i][c] = w[1 + i];
      out.internal_energy[c] = w[D + 1];
      out.pressure[c] = w[D + 2];
      out.temperature[c] = w[D + 3];
      out.sound_speed[c] = a;
    }
    if (lt0(w[D + 1]) || lt0(w[0])) atomicMin(status, status_key(c, FVH_ERR_NEGATIVE_STATE));
    if (NEXT) {
      if (FEW) {
        arith_hw hw;
        dt_inv = cell_dt_inv<D, true>(hw, m, c, w + 1, a, slot_dx);
      } else {
        dt_inv = cell_dt_inv_any<D, true>(m, c, w + 1, a, slot_dx);
      }
    }
  }
  if (NEXT) add_to_maximum(nd, dt_inv);
}

// ---------------------------------------------------------------------------
// the integer-pipe arithmetic against the FP64 instructions (diagnostic)
// ---------------------------------------------------------------------------
__global__ void sf64_kernel(int op, const double *a, const double *b, int64_t n, double *out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x) {
    const double x = a[i], y = b[i];
    double r;
    unsigned rare = 0;
    switch (op) {
      case 0: r = sf64::mul(x, y); break;
      case 1: r = sf64::add(x, y); break;
      case 2: r = sf64::sub(x, y); break;
      case 3: r = sf64::div(x, y); break;
      case 4: r = __dmul_rn(x, y); break;
      case 5: r = __dadd_rn(x, y); break;
      case 6: r = __dsub_rn(x, y); break;
      case 7: r = __ddiv_rn(x, y); break;
      case 8:  // the optimistic forms with their redo, as the kernels use them
        r = sf64::mul_opt(x, y, rare);
        if (rare) r = __dmul_rn(x, y);
        break;
      case 10: {  // the kernels' halving of x (0.5 * x and x / 2), with its redo
        arith_opt ar;
        r = ar.half(x);
        if (ar.rare) r = __dmul_rn(x, 0.5);
        break;
      }
      default:
        r = sf64::div_opt(x, y, rare);
        if (rare) r = __ddiv_rn(x, y);
        break;
    }
    out[i] = r;
  }
}

cudaError_t debug_sf64(int op, const double *a, const double *b, int64_t n, double *out,
                       cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int64_t nb64 = (n + 255) / 256;
  const int nb = (int)(nb64 < 4096 ? nb64 : 4096);
  sf64_kernel<<<nb, 256, 0, st>>>(op, a, b, n, out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------------------
// host launchers
// ---------------------------------------------------------------------------
static int blocks_of(int n, int threads) { return (n + threads - 1) / threads; }

template <int D>
cudaError_t launch_dt(const fvh_mesh_view &m, const fvh_state_view &s,
                      const fvh_params &p, const double *soln_time, double *dt,
                      double *partial, int nblocks, fvh_device_status *status,
                      cudaStream_t st, const double *slot_dx, const fvh_state_view *src,
                      unsigned long long *maximum) {
  const fvh_state_view from = src ? *src : s;
  if (slot_dx)
    dt_partial_kernel<D, true><<<nblocks, kDtThreads, 0, st>>>(m, s, partial, slot_dx, from,
                                                               src ? 1 : 0);
  else
    dt_partial_kernel<D, false><<<nblocks, kDtThreads, 0, st>>>(m, s, partial, nullptr, from,
                                                                src ? 1 : 0);
  dt_final_kernel<<<1, kDtThreads, 0, st>>>(partial, nblocks, p, soln_time, dt, status, maximum);
  return cudaGetLastError();
}

template <int D>
cudaError_t launch_gradients(const fvh_mesh_view &m, const fvh_state_view &s,
                             const fvh_gradient_view &g, const fvh_params &p,
                             cudaStream_t st, const tables &t, const next_dt &nd,
                             bool overlap) {
  const bool lim = p.limiter != FVH_LIMITER_NONE, pre = t.lsq && t.nbr_dx && t.vtx_dx;
  if (m.num_cells <= (pre ? kFewCells : few_cells_no_tables(D, lim))) {
    const dim3 grid(blocks_of(m.num_cells, kFewThreads), D + 4);
    auto go = [&](auto kernel) { launch(kernel, grid, kFewThreads, st, overlap, m, s, g, t, nd); };
    if (pre)
      lim ? go(gradients_few_kernel<D, true, true>) : go(gradients_few_kernel<D, false, true>);
    else
      lim ? go(gradients_few_kernel<D, true, false>) : go(gradients_few_kernel<D, false, false>);
    return cudaGetLastError();
  }
  auto go = [&](auto kernel, int groups, int group_size = 2) {
    const unsigned nb = blocks_of(m.num_cells, kCellThreads);
    const dim3 grid = groups_side_by_side(D, group_size) ? dim3(nb * groups) : dim3(nb, groups);
    launch(kernel, grid, kCellThreads, st, overlap, m, s, g, t, nd);
  };
  const int pairs = blocks_of(D + 4, 2);
  if (!pre)
    lim ? go(gradients_kernel<D, true, false, 2>, 1) : go(gradients_kernel<D, false, false, 2>, 1);
  else if (m.num_cells <= (D == 2 ? kSingleCells2D : kSingleCells3D))
    lim ? go(gradients_kernel<D, true, true, 1>, D + 4, 1)
        : go(gradients_kernel<D, false, true, 1>, D + 4, 1);
  else
    lim ? go(gradients_kernel<D, true, true, 2>, pairs) : go(gradients_kernel<D, false, true, 2>, pairs);
  return cudaGetLastError();
}

size_t table_doubles(int dim, int64_t nc, int64_t nf, int64_t nnz_cf, int64_t nnz_nb,
                     int64_t nnz_cv) {
  const int64_t w = dim == 2 ? lsq_width<2>::value : lsq_width<3>::value;
  // each table starts on a 256-byte boundary (32 doubles)
  auto up = [](int64_t x) { return (x + 31) / 32 * 32; };
  return (size_t)(up(w * nc) + up(nnz_cf) + up(dim * nnz_nb) + up(dim * nnz_cv) +
                  up(2 * dim * nf) + 32);
}

template <int D>
cudaError_t build_tables(const fvh_mesh_view &m, double *base, int64_t nnz_cf,
                         int64_t nnz_nb, int64_t nnz_cv, tables *t) {
  auto up = [](int64_t x) { return (x + 31) / 32 * 32; };
  double *lsq = base;
  double *slot_dx = lsq + up((int64_t)lsq_width<D>::value * m.num_cells);
  double *nbr_dx = slot_dx + up(nnz_cf);
  double *vtx_dx = nbr_dx + up(D * nnz_nb);
  double *face_dx = vtx_dx + up(D * nnz_cv);
  unsigned *d_odd = reinterpret_cast<unsigned *>(face_dx + up(2 * D * (int64_t)m.num_faces));
  unsigned odd = 0;
  cudaError_t e = cudaMemset(d_odd, 0, sizeof(unsigned));
  if (e != cudaSuccess) return e;
  const int th = 128;
  cell_tables_kernel<D><<<(m.num_cells + th - 1) / th, th>>>(m, lsq, slot_dx, nbr_dx, vtx_dx,
                                                             d_odd);
  face_tables_kernel<D><<<(m.num_faces + th - 1) / th, th>>>(m, face_dx, d_odd);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(&odd, d_odd, sizeof(unsigned), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return e;
  t->lsq = lsq;
  t->slot_dx = slot_dx;
  t->nbr_dx = nbr_dx;
  t->vtx_dx = vtx_dx;
  t->face_dx = face_dx;
  // the kernels take these offsets unchecked: a mesh with others, or with cells
  // without vertices, computes them on the fly
  if (odd) t->nbr_dx = t->face_dx = nullptr;
  return cudaSuccess;
}

template <int D, bool SECOND, bool PRE>
static void launch_fluxes_kind(const fvh_mesh_view &m, const fvh_state_view &s,
                               const fvh_gradient_view &g, const fvh_flux_view &fl,
                               const fvh_params &p, cudaStream_t st, const double *face_dx,
                               const next_dt &nd, bool overlap) {
  auto go = [&](auto kernel, int threads) {
    launch(kernel, blocks_of(m.num_faces, threads), threads, st, overlap, m, s, g, fl,
           p.recon_swap_ep, p.boundary, face_dx, nd);
  };
  auto kind = [&](auto k) {
    constexpr int KIND = decltype(k)::value;
    if constexpr (few_faces_form(KIND, SECOND, PRE)) {
      if (m.num_faces <= kFewFaces) {
        go(fluxes_few_kernel<D, KIND, SECOND, PRE>, kFewThreads);
        return;
      }
    }
    go(fluxes_kernel<D, KIND, SECOND, PRE>, kFaceThreads);
  };
  if (p.flux_kind == FVH_FLUX_RUSANOV)
    kind(std::integral_constant<int, FVH_FLUX_RUSANOV>());
  else if (p.flux_kind == FVH_FLUX_HLLC)
    kind(std::integral_constant<int, FVH_FLUX_HLLC>());
  else
    kind(std::integral_constant<int, FVH_FLUX_HLLE>());
}

template <int D>
cudaError_t launch_fluxes(const fvh_mesh_view &m, const fvh_state_view &s,
                          const fvh_gradient_view &g, const fvh_flux_view &fl,
                          const fvh_params &p, cudaStream_t st, const tables &t,
                          const next_dt &nd, bool overlap) {
  if (p.order == 1)
    launch_fluxes_kind<D, false, false>(m, s, g, fl, p, st, nullptr, nd, overlap);
  else if (t.face_dx)
    launch_fluxes_kind<D, true, true>(m, s, g, fl, p, st, t.face_dx, nd, overlap);
  else
    launch_fluxes_kind<D, true, false>(m, s, g, fl, p, st, nullptr, nd, overlap);
  return cudaGetLastError();
}

template <int D>
cudaError_t launch_update(const fvh_mesh_view &m, const fvh_params &p, const double *dt,
                          double factor, const fvh_flux_view &fl,
                          const fvh_state_view &s, double *soln_time,
                          fvh_device_status *status, cudaStream_t st,
                          const fvh_state_view *out, const double *slot_dx, const next_dt &nd,
                          bool overlap) {
  // the same two roundings as (gamma - 1.0) and gamma * (gamma - 1.0) per cell
  const double gamma = p.gamma;
  const double gm1 = gamma - 1.0;
  const double ggm1 = gamma * gm1;
  auto go = [&](auto kernel, int threads) {
    launch(kernel, blocks_of(m.num_cells, threads), threads, st, overlap, m, fl, s, dt, factor, gm1,
           ggm1, p.cv, soln_time, status, out ? *out : s, out ? 1 : 0, slot_dx, nd);
  };
  if (m.num_cells <= kFewUpdateCells)
    nd.maximum ? go(update_kernel<D, true, true>, kFewThreads)
               : go(update_kernel<D, true, false>, kFewThreads);
  else
    nd.maximum ? go(update_kernel<D, false, true>, kCellThreads)
               : go(update_kernel<D, false, false>, kCellThreads);
  return cudaGetLastError();
}

#define FVH_INSTANTIATE(D)                                                              \
  template cudaError_t launch_dt<D>(const fvh_mesh_view &, const fvh_state_view &,     \
                                    const fvh_params &, const double *, double *,      \
                                    double *, int, fvh_device_status *, cudaStream_t,  \
                                    const double *, const fvh_state_view *,            \
                                    unsigned long long *);                             \
  template cudaError_t launch_gradients<D>(const fvh_mesh_view &, const fvh_state_view &, \
                                           const fvh_gradient_view &, const fvh_params &, \
                                           cudaStream_t, const tables &, const next_dt &, bool);              \
  template cudaError_t build_tables<D>(const fvh_mesh_view &, double *, int64_t, int64_t, \
                                       int64_t, tables *);                             \
  template cudaError_t launch_fluxes<D>(const fvh_mesh_view &, const fvh_state_view &, \
                                        const fvh_gradient_view &, const fvh_flux_view &, \
                                        const fvh_params &, cudaStream_t, const tables &, \
                                        const next_dt &, bool); \
  template cudaError_t launch_update<D>(const fvh_mesh_view &, const fvh_params &,     \
                                        const double *, double, const fvh_flux_view &, \
                                        const fvh_state_view &, double *,              \
                                        fvh_device_status *, cudaStream_t,             \
                                        const fvh_state_view *, const double *,        \
                                        const next_dt &, bool);
FVH_INSTANTIATE(2)
FVH_INSTANTIATE(3)

}  // namespace plain
}  // namespace fvh
