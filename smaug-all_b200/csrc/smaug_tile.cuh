// smaug_tile.cuh -- what the production stage kernels share (arithmetic in the
// stencil type, the advance pass with its ghost images and wave-speed maxima, the
// divergence-of-B terms), and the FP64 tile kernel that runs a whole stage of one
// simulation by itself: single-step runs, and 3-D RK4 without a workspace.
//
// Same operator as smaug_stage.cuh (the term-by-term restatement used for
// bit-exact parity), reorganised for throughput.  In the tile kernel
//  * a block owns a TX x TY (x TZ) tile of inner cells, one thread per cell;
//  * fluxes of every field along `dir` are evaluated once on the tile widened
//    by 2 along dir and kept in shared memory for the 5-point divergence;
//  * for each dimension d the hyperviscosity inputs q (rho, internal energy,
//    velocities, B components) are evaluated once on the tile widened by 3
//    along d and 1 across, then nu_R / nu_L once per cell (and on the +-1
//    ring the off-diagonal terms need), all in shared memory;
//  * divisions become multiplications by per-cell reciprocals.
// Results match the reference operator to rounding (the FMA-free restatement
// in smaug_stage.cuh is the bit-exact one).
//
// The template parameter T is the type of the stage states and of the stencil
// arithmetic: double (the FP64 path) or float (the mixed path).  The mixed
// path keeps FP64 where accuracy needs it: the background fields, the total
// pressure p_T and the internal energy (both recovered by cancellation), the
// RK base state (an FP32 value plus an FP32 compensation), the RK combination
// itself and the dt reductions.
#pragma once
#include <type_traits>
#include "smaug_device.cuh"

namespace SMAUG_NS {
using namespace smaug;

// A tile of inner cells, one thread per cell (TZ = 1 in 2-D).
template <int X, int Y, int Z>
struct Tile {
  static constexpr int TX = X, TY = Y, TZ = Z, NT = X * Y * Z;
};
// the single-instance kernels' tiles
template <int D>
struct TileShape;
template <>
struct TileShape<2> : Tile<16, 16, 1> {};
template <>
struct TileShape<3> : Tile<8, 8, 4> {};

template <int D>
struct TileBox {
  // a box in grid coordinates: lo[d] .. lo[d]+ext[d]-1
  int lo[3], ext[3];
  __device__ __forceinline__ int size() const { return ext[0] * ext[1] * (D == 3 ? ext[2] : 1); }
  __device__ __forceinline__ void at(int r, int *c) const {
    c[0] = lo[0] + r % ext[0];
    r /= ext[0];
    c[1] = lo[1] + r % ext[1];
    c[2] = D == 3 ? lo[2] + r / ext[1] : 0;
  }
  __device__ __forceinline__ int index(const int *c) const {
    return (c[0] - lo[0]) + ext[0] * ((c[1] - lo[1]) + (D == 3 ? ext[1] * (c[2] - lo[2]) : 0));
  }
};

template <int D>
__device__ __forceinline__ long long gidx(const Geo &g, const int *c) {
  return c[0] + (long long)c[1] * g.st[1] + (D == 3 ? (long long)c[2] * g.st[2] : 0);
}

__device__ __forceinline__ double vmax(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float vmax(float a, float b) { return fmaxf(a, b); }
__device__ __forceinline__ double vabs(double a) { return fabs(a); }
__device__ __forceinline__ float vabs(float a) { return fabsf(a); }
// a * b + c with one rounding (never left to contraction)
__device__ __forceinline__ double vfma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float vfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
// Conversions between the stencil type and FP64 (none when it is FP64).  The
// plain casts of the -ftz=true build flush subnormals around the conversion
// (a multiply before it, a compare and a select after it), which in the mixed
// kernels was a tenth of all instructions; the FP32 arithmetic that reads a
// converted value flushes it anyway.
__device__ __forceinline__ double dbl(double x) { return x; }
__device__ __forceinline__ double dbl(float x) {
  double r;
  asm("cvt.f64.f32 %0, %1;" : "=d"(r) : "f"(x));
  return r;
}
template <typename T>
__device__ __forceinline__ T num(double x) {
  if constexpr (sizeof(T) == sizeof(float)) {
    float r;
    asm("cvt.rn.f32.f64 %0, %1;" : "=f"(r) : "d"(x));
    return r;
  } else {
    return x;
  }
}
// The hyperviscosity ratio a / b (b > 0): IEEE division in FP64; in FP32 the
// reciprocal-based quotient (within 2 ulp), the ratio being a limiter weight.
__device__ __forceinline__ double vratio(double a, double b) { return a / b; }
__device__ __forceinline__ float vratio(float a, float b) { return __fdividef(a, b); }

// Offset of field f at cell i in 32-bit arithmetic (the host rejects grids
// whose NVAR * N does not fit 31 bits): one multiply-add per access instead
// of a 64-bit product.
__device__ __forceinline__ unsigned fo32(int f, long long N, long long i) {
  return (unsigned)f * (unsigned)N + (unsigned)i;
}

// State accessor: evolved fields of type T, background fields FP64.
template <int D, typename T>
struct CellT {
  const T *__restrict__ in;
  const double *__restrict__ bg;
  long long N;
  // field f at cell i in the stencil type
  __device__ __forceinline__ T v(int f, long long i) const {
    return f < Lay<D>::NW ? ldw(in + fo32(f, N, i)) : num<T>(__ldg(bg + fo32(f - Lay<D>::NW, N, i)));
  }
  // field f at cell i in FP64
  __device__ __forceinline__ double vd(int f, long long i) const {
    return f < Lay<D>::NW ? dbl(ldw(in + fo32(f, N, i))) : __ldg(bg + fo32(f - Lay<D>::NW, N, i));
  }
};

template <int D>
__device__ __forceinline__ bool in_grid(const Geo &g, const int *c) {
#pragma unroll
  for (int d = 0; d < D; ++d)
    if (c[d] < 0 || c[d] >= g.n[d]) return false;
  return true;
}

// Fluxes along dir with reciprocal arithmetic (the same physical fluxes as
// fluxes_at): rho, momentum, energy, induction.  rho_t, its reciprocal and
// the total pressure are formed in FP64.  bgb = 0: e_b and B_b are zero
// everywhere (not read).
template <int D, typename T>
__device__ __forceinline__ void fluxes_fast(const CellT<D, T> &c, long long i, int dir, double gam, bool bgb, T *F) {
  using L = Lay<D>;
  const T rho = c.v(L::RHO, i);
  const double rt = dbl(rho) + c.vd(L::RHOB, i);
  const double irtd = __drcp_rn(rt);
  const T irt = num<T>(irtd);
  T m[D], b[D], bb[D];
#pragma unroll
  for (int k = 0; k < D; ++k) {
    m[k] = c.v(L::M0 + k, i);
    b[k] = c.v(L::B0 + k, i);
    bb[k] = bgb ? c.v(L::BB0 + k, i) : T(0);
  }
  const T e = c.v(L::EN, i), eb = bgb ? c.v(L::EB, i) : T(0);
  double bbb = 0, b2 = 0, m2 = 0;
  T bbm = 0, bm = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    bbb += dbl(b[k]) * dbl(bb[k]);
    b2 += dbl(b[k]) * dbl(b[k]);
    m2 += dbl(m[k]) * dbl(m[k]);
    bbm += bb[k] * m[k];
    bm += b[k] * m[k];
  }
  const T pt = num<T>((gam - 1.0) * (dbl(e) - 0.5 * m2 * irtd) - (gam - 2.0) * (bbb + 0.5 * b2));
  const T md = m[dir], vd = md * irt;
  const T bd = b[dir], bbd = bb[dir];
  F[L::RHO] = md;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    T f = vd * m[k] - (b[k] * bbd + bb[k] * bd) - b[k] * bd;
    if (k == dir) f += pt;
    F[L::M0 + k] = f;
  }
  F[L::EN] = vd * (e + eb) + (md * pt - bd * bbm - bbd * bm - bd * bm) * irt;
#pragma unroll
  for (int k = 0; k < D; ++k)
    F[L::B0 + k] = (k == dir) ? T(0) : vd * (b[k] + bb[k]) - (bd + bbd) * m[k] * irt;
}

// q values for the hyperviscosity of all fields of one dimension d:
// slot 0 rho, 1 internal energy q_e (formed in FP64), 2..2+D-1 velocities,
// then B_f (f != d).
template <int D, typename T>
__device__ __forceinline__ void q_all(const CellT<D, T> &c, long long i, int d, T *q) {
  using L = Lay<D>;
  const T rho = c.v(L::RHO, i);
  const double irtd = __drcp_rn(dbl(rho) + c.vd(L::RHOB, i));
  const T irt = num<T>(irtd);
  double b2 = 0, m2 = 0;
  q[0] = rho;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const T m = c.v(L::M0 + k, i), b = c.v(L::B0 + k, i);
    b2 += dbl(b) * dbl(b);
    m2 += dbl(m) * dbl(m);
    q[2 + k] = m * irt;
  }
  q[1] = num<T>(c.vd(L::EN, i) - 0.5 * (b2 + m2 * irtd));
  int s = 2 + D;
#pragma unroll
  for (int f = 0; f < D; ++f)
    if (f != d) q[s++] = c.v(L::B0 + f, i);
}

// cfast/courant maxima as reduce_cell (computec3, dervfields.cu:241-309), for
// the mixed path: the state is FP32 there, so the wave speeds are formed in
// FP32 from a correctly rounded reciprocal of rho_t (the pressure recovery's
// rounding stays at the level of the FP32 inputs); the courant number divides
// by the metric through a correctly rounded reciprocal too.  Explicitly
// rounded operations, never contracted: every build variant of the stage
// kernel gives the same bits.  b: eb, rho_b, B_b (zeros when the simulation
// has no energy background).  The maxima are FP32 values and kept in FP32.
//
// A fast pass comes first. It takes the square roots and the metric's
// reciprocal from the hardware approximations (x rsqrtf(x), __fdividef); every
// other operation is the same as in the exact pass. That puts each approximate
// speed within about 8 ulp (1e-6 relative) of its correctly rounded value: the
// terms under the roots are identical, and the sums after them add
// non-negative terms. If every approximate speed of the cell stays more than
// 1e-5 below the thread's running maximum, the cell cannot raise it and is
// done. Any other cell, a NaN included, takes the correctly rounded pass. The
// maxima come out the same bits either way.
__device__ __forceinline__ float sqrt_approx(float x) { return x > 0.0f ? x * rsqrtf(x) : 0.0f; }

// Returns the correctly rounded speed of the last dim, or -1 if the cell was
// done after the fast pass.
template <int D>
__device__ __forceinline__ float reduce_cell_mixed(const Geo &g, const Phys &p, const float *o, const double *b,
                                                   long long idx, float *r) {
  using L = Lay<D>;
  const float irt = __frcp_rn(num<float>(dbl(o[L::RHO]) + b[1]));
  float m2 = 0.0f, b2 = 0.0f, bbb = 0.0f, bb2 = 0.0f;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    const float m = o[L::M0 + k], bf = o[L::B0 + k], bb = num<float>(b[2 + k]);
    m2 = __fmaf_rn(m, m, m2);
    b2 = __fmaf_rn(bf, bf, b2);
    bbb = __fmaf_rn(bb, bf, bbb);
    bb2 = __fmaf_rn(bb, bb, bb2);
  }
  const float gm1 = (float)(p.gamma - 1.0), gam = (float)p.gamma;
  // p_k = (gamma-1) (e - m^2/(2 rho_t) - B^2/2 - B.B_b)
  const float ek = __fsub_rn(__fsub_rn(__fsub_rn(o[L::EN], __fmul_rn(__fmul_rn(0.5f, m2), irt)),
                                       __fmul_rn(0.5f, b2)), bbb);
  const float pk = __fmul_rn(gm1, ek);
  // c_s^2 = gamma (p_k + (gamma-1)(e_b - B_b^2/2)) / rho_t
  const float pbg = __fmul_rn(gm1, __fsub_rn(num<float>(b[0]), __fmul_rn(0.5f, bb2)));
  const float cs2 = __fmul_rn(__fmul_rn(gam, __fadd_rn(pk, pbg)), irt);
  const float cf = __fadd_rn(__fmul_rn(__fadd_rn(__fadd_rn(b2, bb2), __fmul_rn(2.0f, bbb)), irt), cs2);
  {
    constexpr float kBelow = 1.0f - 1e-5f;
    const float rdx = __fdividef(1.0f, num<float>(__ldg(g.dxlast + idx)));
    bool need = false;
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const float bd = num<float>(b[2 + d] + dbl(o[L::B0 + d]));
      const float disc =
          __fsub_rn(__fmul_rn(cf, cf), __fmul_rn(__fmul_rn(__fmul_rn(4.0f, cs2), __fmul_rn(bd, bd)), irt));
      const float cfi = __fmul_rn(0.5f, __fadd_rn(cf, sqrt_approx(fmaxf(disc, 0.0f))));
      const float cff = __fadd_rn(sqrt_approx(cfi), fabsf(__fmul_rn(o[L::M0 + d], irt)));
      need |= !(cff < r[d] * kBelow);
      if (d == D - 1) {
        const float cour = cff * rdx;
        need |= !(cour < r[3] * kBelow);
        if (idx >= g.K) need |= !(cour < r[4] * kBelow);
      }
    }
    if (!need) return -1.0f;
  }
  float last = 0.0f;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const float bd = num<float>(b[2 + d] + dbl(o[L::B0 + d]));
    const float disc = __fsub_rn(__fmul_rn(cf, cf), __fmul_rn(__fmul_rn(__fmul_rn(4.0f, cs2), __fmul_rn(bd, bd)), irt));
    const float cfi = __fmul_rn(0.5f, __fadd_rn(cf, __fsqrt_rn(fmaxf(disc, 0.0f))));
    const float cff = __fadd_rn(__fsqrt_rn(cfi), fabsf(__fmul_rn(o[L::M0 + d], irt)));
    if (cff > r[d] || cff != cff) r[d] = cff;
    if (d == D - 1) {
      const float cour = __fmul_rn(cff, __frcp_rn(num<float>(__ldg(g.dxlast + idx))));
      if (cour > r[3] || cour != cour) r[3] = cour;
      if (idx >= g.K && (cour > r[4] || cour != cour)) r[4] = cour;
      last = cff;
    }
  }
  return last;
}

// reduce_cell (FP64) behind a screen, as in reduce_cell_mixed: the speeds with
// one reciprocal of rho_t, hardware-approximated square roots and metric
// reciprocal lie within 1e-5 of the exact ones (the terms under the roots carry
// a few roundings of cf^2, at most 1e-7 of cf after the root; the
// approximations themselves 2^-20), so a cell that stays more than 1e-5 below
// the running maxima cannot raise them.  Any other cell, a NaN included, takes
// reduce_cell: the maxima keep their bits.  So does a cell whose discriminant is
// zero but for rounding (sound and Alfven speed along d agree): reduce_cell's
// may be negative there and its speed NaN, which has to be seen whatever the
// thread has seen before.  (Nine divisions and six square roots in software per
// 3-D cell otherwise.)
__device__ __forceinline__ double rsqrt_approx(double x) {
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}
__device__ __forceinline__ double rcp_approx(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  return r;
}
// Returns the exact speed of the last dim, or -1 if the cell was done after the
// screen.
template <int D>
__device__ __forceinline__ double reduce_cell_screened(const Geo &g, const Phys &p, const double *o, const double *b,
                                                       long long idx, double *r) {
  using L = Lay<D>;
  const double irt = __drcp_rn(o[L::RHO] + b[1]);
  double m2 = 0, b2 = 0, bbb = 0, bb2 = 0;
#pragma unroll
  for (int k = 0; k < D; ++k) {
    m2 += o[L::M0 + k] * o[L::M0 + k];
    b2 += o[L::B0 + k] * o[L::B0 + k];
    bbb += b[2 + k] * o[L::B0 + k];
    bb2 += b[2 + k] * b[2 + k];
  }
  const double pk = (p.gamma - 1) * (o[L::EN] - 0.5 * m2 * irt - 0.5 * b2 - bbb);
  const double cs2 = p.gamma * (pk + (p.gamma - 1) * (b[0] - 0.5 * bb2)) * irt;
  const double cf = (b2 + bb2 + 2.0 * bbb) * irt + cs2;
  constexpr double kBelow = 1.0 - 1e-5;
  const double rdx = rcp_approx(__ldg(g.dxlast + idx));
  // How small the root of the discriminant |b_d^2 / rho_t - c_s^2| may be before
  // rounding decides its sign: in either evaluation the discriminant carries a
  // few roundings of cf^2 (its root 3e-8 of cf), and c_s^2 a few of the energies
  // that p_k is recovered from (1e-13: 450 units of 2^-52).
  const double low =
      1e-6 * cf + 1e-13 * p.gamma * (fabs(o[L::EN]) + fabs(b[0]) + m2 * irt + b2 + bb2) * irt;
  bool need = false;
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const double bd = b[2 + d] + o[L::B0 + d];
    const double disc = cf * cf - 4.0 * cs2 * (bd * bd) * irt;
    const double cfi = 0.5 * (cf + disc * rsqrt_approx(disc));
    const double cff = cfi * rsqrt_approx(cfi) + fabs(o[L::M0 + d] * irt);
    need |= !(disc > low * low) || !(cff < r[d] * kBelow);
    if (d == D - 1) {
      const double cour = cff * rdx;
      need |= !(cour < r[3] * kBelow);
      if (idx >= g.K) need |= !(cour < r[4] * kBelow);
    }
  }
  return need ? reduce_cell<D>(g, p, o, b, idx, r) : -1.0;
}

// The courant number of a cell of speed cff at cell j, taken into the maxima,
// with the operations of the two reductions.
__device__ __forceinline__ void courant_at(const Geo &g, float cff, long long j, float *r) {
  const float cour = __fmul_rn(cff, __frcp_rn(num<float>(__ldg(g.dxlast + j))));
  if (cour > r[3] || cour != cour) r[3] = cour;
  if (j >= g.K && (cour > r[4] || cour != cour)) r[4] = cour;
}
__device__ __forceinline__ void courant_at(const Geo &g, double cff, long long j, double *r) {
  const double cour = cff / __ldg(g.dxlast + j);
  if (cour > r[3] || cour != cour) r[3] = cour;
  if (j >= g.K && (cour > r[4] || cour != cour)) r[4] = cour;
}

// Loads and stores of the advance pass: every value is touched once, so it
// passes by L1 (and the instructions are global ones: the buffer pointers come
// from a table in memory, where the compiler does not know their space).
__device__ __forceinline__ float ldq(const float *p) { return __ldcg(p); }
__device__ __forceinline__ double ldq(const double *p) { return __ldcg(p); }
__device__ __forceinline__ void stq(float *p, float v) { __stcg(p, v); }
__device__ __forceinline__ void stq(double *p, double v) { __stcg(p, v); }

// The sources dL of one inner cell on their way from the stage kernel to the
// advance pass.
template <int D, typename T>
__device__ __forceinline__ void store_sources(const StageArgs &a, const Geo &g, long long idx, const T *dL) {
  T *o = sizeof(T) == sizeof(float) ? (T *)(void *)a.src32 : (T *)(void *)a.src;
#pragma unroll
  for (int f = 0; f < Lay<D>::NW; ++f) stq(o + fo32(f, g.N, idx), dL[f]);
}
template <int D, typename T>
__device__ __forceinline__ void load_sources(const StageArgs &a, const Geo &g, long long idx, T *dL) {
  const T *o = sizeof(T) == sizeof(float) ? (const T *)(const void *)a.src32 : (const T *)(const void *)a.src;
#pragma unroll
  for (int f = 0; f < Lay<D>::NW; ++f) dL[f] = ldq(o + fo32(f, g.N, idx));
}

// Wave-speed maxima of the state v (of the inner cell or one of its images)
// at cell j, with that cell's backgrounds (e_b and B_b are zero everywhere
// without an energy background: only rho_b is read then).
// Returns the speed of the last dim as the functions above.
template <int D, typename T>
__device__ __forceinline__ T reduce_at(const StageArgs &a, const Geo &g, const Phys &p, const T *v, long long j,
                                       T *red) {
  using L = Lay<D>;
  constexpr int NW = L::NW, NB = L::NVAR - NW;
  double bgv[NB];
#pragma unroll
  for (int b = 0; b < NB; ++b)
    bgv[b] = (b == L::RHOB - NW || p.has_bgb) ? __ldg(a.bg + fo32(b, g.N, j)) : 0.0;
  if constexpr (sizeof(T) == sizeof(float))
    return reduce_cell_mixed<D>(g, p, v, bgv, j, red);
  else
    return reduce_cell_screened<D>(g, p, v, bgv, j, red);
}

// The end of a stage for one inner cell: the stage output base + h dL with the
// driver, the RK combination of the stage (KIND: StageArgs::kind), the write of
// the cell and of its ghost images (the reference's boundary pass after each
// step, iosmaug.cpp:1157-1166; a stage reads no buffer that it writes beyond
// the cell itself), and the wave-speed maxima of all of them (the reference's
// c_max covers the ghosts), taken into the thread's running maxima red[5] (in
// the stencil type: FP32 values in the mixed path; the caller flushes them to
// the simulation's reduction slot).  Everything the cell reads is loaded
// before its first store: a load behind a store to another buffer waits for it
// (the buffers may alias as far as the compiler knows), and field by field
// that was one memory latency per field.
template <int D, typename T, int KIND>
__device__ __forceinline__ void advance_cell(const StageArgs &a, const Geo &g, const Phys &p, const int *c,
                                             long long idx, double h, double tdep, const T *dL, T *red) {
  using L = Lay<D>;
  constexpr int NW = L::NW;
  constexpr bool MIXED = sizeof(T) == sizeof(float);
  T o[NW];   // the stage output (mixed: FP32 value)
  T lo[NW];  // what goes with it: the sum so far, in mixed stage 4 the compensation
  if constexpr (!MIXED) {
    double bv[NW], iv[NW];
#pragma unroll
    for (int f = 0; f < NW; ++f) bv[f] = ldq(a.base + fo32(f, g.N, idx));
    if (KIND >= 3) {
#pragma unroll
      for (int f = 0; f < NW; ++f) lo[f] = ldq(a.acc + fo32(f, g.N, idx));
    }
    if (KIND == 3) {
#pragma unroll
      for (int f = 0; f < NW; ++f) iv[f] = ldq(a.in + fo32(f, g.N, idx));
    }
#pragma unroll
    for (int f = 0; f < NW; ++f) o[f] = bv[f] + h * dL[f];
    if (p.drv_on) {  // momentum driver on the stage output (before the RK combination)
      const double vvz = driver_vvz<D>(g, p, tdep, c);
      const double rb = __ldg(a.bg + (long long)(L::RHOB - NW) * g.N + idx);
      // (unrolled compare: a runtime index would push o to local memory)
#pragma unroll
      for (int k = 0; k < D; ++k)
        if (k == p.drv_dir) o[L::M0 + k] = o[L::M0 + k] + h * vvz * (o[L::RHO] + rb);
    }
    if (KIND == 3) {
#pragma unroll
      for (int f = 0; f < NW; ++f)
        stq(a.acc + fo32(f, g.N, idx), (lo[f] + 2.0 * iv[f] + o[f] - 4.0 * bv[f]) * (1.0 / 3.0));
    } else if (KIND == 4) {
#pragma unroll
      for (int f = 0; f < NW; ++f) o[f] += lo[f];
    }
  } else {
    // RK4 in increment form, W = w32 + c32:
    //   stages k = 1..3: S_k = W + h_k L_k (FP32), A += c_k h_k L_k with
    //   c = 1/3, 2/3, 1/3, so A = (S1 + 2 S2 + S3 - 4 W) / 3 as the FP64 path;
    //   stage 4: W <- W + h_4 L_4 + A, kept as value + compensation.
    // Stages 1..3 round to FP32 anyway, so they take the base without c32.
    float wv[NW], cv[NW], av[NW];
#pragma unroll
    for (int f = 0; f < NW; ++f) wv[f] = ldq(a.w32 + fo32(f, g.N, idx));
    if (KIND != 1) {
#pragma unroll
      for (int f = 0; f < NW; ++f) av[f] = ldq(a.acc32 + fo32(f, g.N, idx));
    }
    if (KIND == 4) {
#pragma unroll
      for (int f = 0; f < NW; ++f) cv[f] = ldq(a.c32 + fo32(f, g.N, idx));
    }
    // momentum driver with the stage output's density, added to the
    // increment of m along drv_dir (dm = 0 without a driver)
    double dm = 0.0;
    int dm_f = -1;
    if (p.drv_on) {
      const double wr = KIND == 4 ? dbl(wv[0]) + dbl(cv[0]) : dbl(wv[0]);
      const double rb = __ldg(a.bg + (long long)(L::RHOB - NW) * g.N + idx);
      dm = h * driver_vvz<D>(g, p, tdep, c) * ((wr + h * dbl(dL[L::RHO])) + rb);
      dm_f = L::M0 + p.drv_dir;
    }
#pragma unroll
    for (int f = 0; f < NW; ++f) {
      double inc = h * dbl(dL[f]);
      if (f == dm_f) inc += dm;
      if (KIND == 4) {
        const double wn = (dbl(wv[f]) + dbl(cv[f])) + (inc + dbl(av[f]));
        o[f] = num<float>(wn);
        lo[f] = num<float>(wn - dbl(o[f]));
      } else {
        o[f] = num<float>(dbl(wv[f]) + inc);
        const float sum = num<float>((KIND == 1 ? 0.0 : dbl(av[f])) + (KIND == 2 ? 2.0 : 1.0) * (1.0 / 3.0) * inc);
        stq(a.acc32 + fo32(f, g.N, idx), sum);
      }
    }
  }
  // the cell (image 0) and its ghost images, all of cells within four cells of
  // an end (images(): the rules of every direction composed)
  bool near = false;
#pragma unroll
  for (int d = 0; d < D; ++d) near |= c[d] < 5 || c[d] > g.n[d] - 6;
  int n0 = 1, n1 = 1, n2 = 1;
  int xa = 0, xb = 0, ya = 0, yb = 0, za = 0, zb = 0;  // image coordinates per dimension
  unsigned g0 = 0, g1 = 0, g2 = 0;
  if (near) {
    int x[3];
    n0 = images<D>(g, 0, c[0], x, &g0);
    xa = x[1];
    xb = x[2];
    n1 = images<D>(g, 1, c[1], x, &g1);
    ya = x[1];
    yb = x[2];
    if (D == 3) {
      n2 = images<D>(g, D - 1, c[D - 1], x, &g2);
      za = x[1];
      zb = x[2];
    }
  }
  const int count = n0 * n1 * n2;
  long long j = idx;
  unsigned neg = 0;
  T cff = 0;  // the cell's own speed along the last dim, if it was formed exactly
#pragma unroll 1
  for (int k = 0;;) {
    T v[NW];
    T *w = MIXED ? (T *)(void *)(KIND == 4 ? a.w32 : a.out32) : (T *)(void *)a.out;
#pragma unroll
    for (int f = 0; f < NW; ++f) {
      const unsigned q = fo32(f, g.N, j);
      const bool m = (neg >> f) & 1u;
      v[f] = m ? -o[f] : o[f];
      stq(w + q, v[f]);
      if (MIXED && KIND == 4) stq(a.c32 + q, m ? -(float)lo[f] : (float)lo[f]);
    }
    // What the next stage reads.  An image without negated fields over the
    // cell's own background has the cell's speeds: only its courant number,
    // over the metric there, can differ (and the exact pass again, once per
    // image, would be most of a small grid's advance).
    if (k > 0 && neg == 0 && cff > T(0) && !p.has_bgb &&
        __ldg(a.bg + fo32(L::RHOB - NW, g.N, j)) == __ldg(a.bg + fo32(L::RHOB - NW, g.N, idx))) {
      courant_at(g, cff, j, red);
    } else {
      const T c0 = reduce_at<D, T>(a, g, p, v, j, red);
      if (k == 0) cff = c0;
    }
    if (++k >= count) break;
    const int i0 = k % n0, r = k / n0, i1 = r % n1, i2 = r / n1;
    j = (i0 == 0 ? c[0] : i0 == 1 ? xa : xb) + (i1 == 0 ? c[1] : i1 == 1 ? ya : yb) * g.st[1] +
        (D == 3 ? (i2 == 0 ? c[2] : i2 == 1 ? za : zb) * g.st[2] : 0);
    neg = (i0 ? g0 : 0u) ^ (i1 ? g1 : 0u) ^ (i2 ? g2 : 0u);
  }
}
// The same in FP64 with the kind at run time (tile_body).
template <int D>
__device__ __forceinline__ void advance_cell_any(const StageArgs &a, const Geo &g, const Phys &p, const int *c,
                                                 long long idx, double h, const double *dL, double *red) {
  const double tdep = p.drv_on ? driver_tdep(p, a.sc, a.tfrac) : 0.0;
  if (a.kind == 3)
    advance_cell<D, double, 3>(a, g, p, c, idx, h, tdep, dL, red);
  else if (a.kind == 4)
    advance_cell<D, double, 4>(a, g, p, c, idx, h, tdep, dL, red);
  else
    advance_cell<D, double, 0>(a, g, p, c, idx, h, tdep, dL, red);
}

// Divergence-of-B source terms at an inner cell (cudivb, divb.cu:165-336 with
// divbon = divbfix = 1; 2-D): at cells 3..n-3 of both dims, divB from the
// 4th-order difference over the uniform spacing (zero at the first and last
// two inner cells, as grad3d of gradops.cu:132-237), then -divB (0, B, B.v,
// v) per unit time with B.v = B_total . m / rho_t; NaN momentum and field
// sources count as 0 (dbsourcemom, dbsourceb).
template <typename T>
__device__ __forceinline__ void divb_sources(const CellT<2, T> &C, const Geo &g, const Phys &p, const int *c,
                                             long long idx, T *dL) {
  using L = Lay<2>;
  if (c[0] <= 2 || c[1] <= 2) return;
  T divb = 0;
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    const int x = c[d], n = g.n[d];
    if (x == 3 || x == n - 4 || x == n - 3) continue;
    const long long s = g.st[d];
    T b[4];  // B_d + B_bd at -2, -1, +1, +2
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long j = idx + (k < 2 ? k - 2 : k - 1) * s;
      b[k] = C.v(L::B0 + d, j) + (p.has_bgb ? C.v(L::BB0 + d, j) : T(0));
    }
    divb += ((T)8 * (b[2] - b[1]) - (b[3] - b[0])) * num<T>(1.0 / (12.0 * p.dxs[d]));
  }
  const T irt = num<T>(1.0 / (C.vd(L::RHO, idx) + C.vd(L::RHOB, idx)));
  T bdotv = 0;
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const T bk = C.v(L::B0 + k, idx), mk = C.v(L::M0 + k, idx);
    bdotv += (bk + (p.has_bgb ? C.v(L::BB0 + k, idx) : T(0))) * mk;
    T sm = divb * bk, sb = divb * mk * irt;
    if (sm != sm) sm = 0;
    if (sb != sb) sb = 0;
    dL[L::M0 + k] += sm;
    dL[L::B0 + k] += sb;
  }
  dL[L::EN] += divb * bdotv * irt;
}

// One RK stage on the tile (bx, by, bz) of one simulation; every thread of
// the block calls it (it synchronises the block).  sm: tile_smem_elems<D, S>()
// doubles.  (Single-step runs, and 3-D runs without the workspace of
// smaug_pass3.cuh; FP64: mixed runs are RK4 through the batch kernels.)
template <int D, typename S>
__device__ __forceinline__ void tile_body(const StageArgs &a, const Geo &g, const Phys &p, int bx, int by, int bz,
                                          double *sm, double *red) {
  using T = double;
  using L = Lay<D>;
  constexpr int TX = S::TX, TY = S::TY, TZ = S::TZ, NT = TX * TY * TZ;
  constexpr int NW = L::NW, NB = L::NVAR - NW;
  constexpr int NQ = 2 * D + 1;  // q slots per cell for one dimension

  const int t = threadIdx.x;
  const int tc[3] = {t % TX, (t / TX) % TY, D == 3 ? t / (TX * TY) : 0};
  const int org[3] = {2 + bx * TX, 2 + by * TY, D == 3 ? 2 + bz * TZ : 0};
  int c[3] = {org[0] + tc[0], org[1] + tc[1], org[2] + tc[2]};
  bool active = true;
#pragma unroll
  for (int d = 0; d < D; ++d)
    if (c[d] > g.n[d] - 3) active = false;
  const long long idx = active ? gidx<D>(g, c) : 0;
  const CellT<D, T> C{a.in, a.bg, g.N};
  const double dt = a.sc->dt;
  const double h = a.hslot > 0 ? a.sc->hst[a.hslot] : dt / a.hdiv;
  T cm[3] = {0, 0, 0};
#pragma unroll
  for (int d = 0; d < D; ++d) cm[d] = num<T>(red_get(a.sc->red[a.red_in], d));
  int tile_ext[3] = {TX, TY, D == 3 ? TZ : 1};
  T idx1[3] = {0, 0, 0};
  if (active) {
#pragma unroll
    for (int d = 0; d < D; ++d) idx1[d] = num<T>(__ldg(g.rdx1[d] + c[d]));
  }
  T dL[NW];
#pragma unroll
  for (int f = 0; f < NW; ++f) dL[f] = 0;
  T numax = 0;

  // ------------------------------------------------ flux divergences
#pragma unroll
  for (int dir = 0; dir < D; ++dir) {
    TileBox<D> box;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      box.lo[e] = org[e] - (e == dir ? 2 : 0);
      box.ext[e] = tile_ext[e] + (e == dir ? 4 : 0);
    }
    const int nbox = box.size();
    for (int r = t; r < nbox; r += NT) {
      int cc[3];
      box.at(r, cc);
      T F[NW];
      if (in_grid<D>(g, cc)) {
        fluxes_fast<D, T>(C, gidx<D>(g, cc), dir, p.gamma, p.has_bgb, F);
      } else {
#pragma unroll
        for (int f = 0; f < NW; ++f) F[f] = 0;
      }
#pragma unroll
      for (int f = 0; f < NW; ++f) sm[f * nbox + r] = F[f];
    }
    __syncthreads();
    if (active) {
      const bool zr = z4(g, c, dir);
      int cc[3] = {c[0], c[1], c[2]};
      const int r0 = box.index(cc);
      const int st = dir == 0 ? 1 : dir == 1 ? box.ext[0] : box.ext[0] * box.ext[1];
      const T w12 = idx1[dir] * (T)(1.0 / 12.0);
#pragma unroll
      for (int f = 0; f < NW; ++f) {
        const T *Fp = sm + f * nbox + r0;
        T gr = ((T)8 * (Fp[st] - Fp[-st]) - (Fp[2 * st] - Fp[-2 * st])) * w12;
        if (!zr) dL[f] -= gr;
      }
    }
    __syncthreads();
  }

  // ------------------------------------------------ gravity
  if (active && p.has_grav) {
    const T rho = C.v(L::RHO, idx), irt = num<T>(__drcp_rn(dbl(rho) + C.vd(L::RHOB, idx)));
#pragma unroll
    for (int k = 0; k < D; ++k) {
      dL[L::M0 + k] += num<T>(p.g[k]) * rho;
      dL[L::EN] += rho * num<T>(p.g[k]) * C.v(L::M0 + k, idx) * irt;
    }
  }
  if constexpr (D == 2) {
    if (active && p.divb) divb_sources<T>(C, g, p, c, idx, dL);
  }

  // ------------------------------------------------ per-dimension hyperdiffusion
  // (one call per dimension, d a compile-time constant in each)
  auto dim_pass = [&](auto dc) {
    constexpr int d = decltype(dc)::value;
    // q box: tile widened by 3 along d and 1 across
    TileBox<D> qb;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const int w = e >= D ? 0 : (e == d ? 3 : 1);
      qb.lo[e] = org[e] - w;
      qb.ext[e] = tile_ext[e] + 2 * w;
    }
    const int nq = qb.size();
    // face box: the faces along d of the tile (face j between cells j and
    // j+1, j from -1), widened by 1 across d (the off-diagonal terms need nu
    // there); it holds the hyperviscosity ratio max|d3 q| / max|d1 q| per face
    constexpr int TD = d == 0 ? TX : d == 1 ? TY : TZ;
    TileBox<D> fb;
#pragma unroll
    for (int e = 0; e < 3; ++e) {
      const int w = (e >= D || e == d) ? 0 : 1;
      fb.lo[e] = org[e] - (e == d ? 1 : w);
      fb.ext[e] = e == d ? TD + 1 : tile_ext[e] + 2 * w;
    }
    const int nf = fb.size();
    T *Q = sm;            // [NQ][nq]
    T *V = sm + NQ * nq;  // [NQ][nf]
    for (int r = t; r < nq; r += NT) {
      int cc[3];
      qb.at(r, cc);
      T q[NQ];
      const int x = cc[d];
      bool ok = true;
#pragma unroll
      for (int e = 0; e < D; ++e)
        if (e != d && (cc[e] < 0 || cc[e] >= g.n[e])) ok = false;
      if (!ok || x >= g.n[d]) {  // x == n: right pad of the padded q copy (0)
#pragma unroll
        for (int k = 0; k < NQ; ++k) q[k] = 0;
      } else {
        int src[3] = {cc[0], cc[1], cc[2]};
        if (x < 0) src[d] = 5;  // left pad: q(-1) = q(5)
        q_all<D, T>(C, gidx<D>(g, src), d, q);
      }
#pragma unroll
      for (int k = 0; k < NQ; ++k) Q[k * nq + r] = q[k];
    }
    __syncthreads();
    const int sd = d == 0 ? 1 : d == 1 ? qb.ext[0] : qb.ext[0] * qb.ext[1];
    if (p.hyperdif) {
      // runs of SEG faces along d of one q slot on one line: the line's q
      // values are read once, each first and third difference is formed once
      // (explicit FMA), every face takes its windowed maxima; the last run of
      // a line is shifted back to end at the line's last face (shared faces
      // are written twice with the same value)
      constexpr int SEG = TD + 1 < 5 ? TD + 1 : 5;
      constexpr int NS = (TD + 1 + SEG - 1) / SEG;
      const int lines = nf / (TD + 1);
      const int fs = d == 0 ? 1 : d == 1 ? fb.ext[0] : fb.ext[0] * fb.ext[1];  // face stride along d
      for (int u = t; u < NQ * lines * NS; u += NT) {
        const int sg = u % NS, rest = u / NS;
        const int ln = rest % lines, k = rest / lines;
        const int f0 = min(-1 + sg * SEG, TD - SEG);  // first face of the run, tile-relative
        // the line's cross coordinates (tile-relative, -1 .. T_e): decode ln
        int cr[3] = {0, 0, 0}, rem = ln;
#pragma unroll
        for (int e = 0; e < 3; ++e) {
          if (e == d || e >= D) continue;
          const int ex = tile_ext[e] + 2;
          cr[e] = rem % ex - 1;
          rem /= ex;
        }
        // q at the cells f0-2 .. f0+SEG+2 along d
        int qc[3] = {org[0] + cr[0], org[1] + cr[1], org[2] + cr[2]};
        qc[d] = org[d] + f0 - 2;
        const T *qq = Q + k * nq + qb.index(qc);
        T qv[SEG + 5], t1[SEG + 4], t3[SEG + 3];
#pragma unroll
        for (int jx = 0; jx < SEG + 5; ++jx) qv[jx] = qq[jx * sd];
#pragma unroll
        for (int jx = 0; jx < SEG + 4; ++jx) t1[jx] = qv[jx + 1] - qv[jx];
#pragma unroll
        for (int jx = 1; jx <= SEG + 2; ++jx) t3[jx] = vabs(vfma((T)3, t1[jx], -(qv[jx + 2] - qv[jx - 1])));
        int fc[3] = {org[0] + cr[0], org[1] + cr[1], org[2] + cr[2]};
        fc[d] = org[d] + f0;
        T *dst = V + k * nf + fb.index(fc);
#pragma unroll
        for (int m = 0; m < SEG; ++m) {
          T m1 = 0, m3 = 0;
#pragma unroll
          for (int jx = m; jx <= m + 4; ++jx) m1 = vmax(m1, vabs(t1[jx]));
#pragma unroll
          for (int jx = m + 1; jx <= m + 3; ++jx) m3 = vmax(m3, t3[jx]);
          dst[m * fs] = m1 > 0 ? vratio(m3, m1) : T(0);
        }
      }
    }
    __syncthreads();
    if (active) {
      int cc[3] = {c[0], c[1], c[2]};
      const int r0 = qb.index(cc);
      const int fr = fb.index(cc);  // the cell's right face along d; its left face is fr - fs
      const int fs = d == 0 ? 1 : d == 1 ? fb.ext[0] : fb.ext[0] * fb.ext[1];
      const T dxd = num<T>(__ldg(g.dx1[d] + c[d]));
      // nu_R, nu_L of slot k at the cell shifted by `off` faces across d: dx
      // c_max c_hyp times the face ratios (0 off the inner cells, as the
      // reference's viscosity arrays are)
      auto nu_at = [&](int k, int off, bool in, T &nr, T &nl) {
        int fid = k == 0 ? L::RHO : k == 1 ? L::EN : k < 2 + D ? L::M0 + (k - 2) : 0;
        if (k >= 2 + D) {
          const int ff = k - (2 + D);
          fid = L::B0 + (ff >= d ? ff + 1 : ff);
        }
        const T kk = dxd * cm[d] * num<T>(p.chyp[fid]);
        nr = in ? kk * V[k * nf + fr + off] : T(0);
        nl = in ? kk * V[k * nf + fr - fs + off] : T(0);
      };
      const long long sg = g.st[d];
      const bool zd = z1(g, c, d);
      const T i1 = idx1[d], i2 = idx1[d] * idx1[d];
      if (p.has_bgb) {  // background energy terms along d (addenergyterms_cd2)
        double bb2 = 0;
#pragma unroll
        for (int k = 0; k < D; ++k) bb2 += C.vd(L::BB0 + k, idx) * C.vd(L::BB0 + k, idx);
        const T ptb = num<T>((p.gamma - 1) * C.vd(L::EB, idx) - 0.5 * (p.gamma - 2) * bb2);
        const bool z4d = z4(g, c, d);
#pragma unroll
        for (int dir = 0; dir < D; ++dir) {
          const T *v = Q + (2 + dir) * nq + r0;
          T gv = z4d ? T(0) : ((T)8 * (v[sd] - v[-sd]) - (v[2 * sd] - v[-2 * sd])) * (i1 * (T)(1.0 / 12.0));
          if (d == dir) dL[L::EN] -= ptb * gv;
          dL[L::EN] += C.v(L::BB0 + d, idx) * C.v(L::BB0 + dir, idx) * gv;
        }
      }
      if (p.hyperdif) {
#pragma unroll
        for (int k = 0; k < NQ; ++k) {
          T nr, nl;
          nu_at(k, 0, true, nr, nl);
          numax = vmax(numax, vmax(nr, nl));
        }
        // rho and internal energy: f += (nu_R dq+ - nu_L dq-) / dx^2
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const T *q = Q + k * nq + r0;
          T nr, nl;
          nu_at(k, 0, true, nr, nl);
          const T dp = zd ? T(0) : q[sd] - q[0], dm = zd ? T(0) : q[0] - q[-sd];
          dL[k == 0 ? L::RHO : L::EN] += (nr * dp - nl * dm) * i2;
        }
        // momentum
        const T rt0 = C.v(L::RHO, idx) + C.v(L::RHOB, idx);
        const T rtp = C.v(L::RHO, idx + sg) + C.v(L::RHOB, idx + sg);
        const T rtm = C.v(L::RHO, idx - sg) + C.v(L::RHOB, idx - sg);
#pragma unroll
        for (int f = 0; f < D; ++f) {
          const int k = 2 + f;
          const T *v = Q + k * nq + r0;
          T nr, nl;
          nu_at(k, 0, true, nr, nl);
          const T dvp = zd ? T(0) : v[sd] - v[0], dvm = zd ? T(0) : v[0] - v[-sd];
          const T m0 = C.v(L::M0 + f, idx), mp = C.v(L::M0 + f, idx + sg), mm = C.v(L::M0 + f, idx - sg);
          const T fac = (f == d ? (T)1 : (T)0.5) * i2;
          dL[L::M0 + f] += ((rt0 + rtp) * nr * dvp - (rt0 + rtm) * nl * dvm) * (T)0.5 * fac;
          dL[L::EN] += ((m0 + mp) * nr * dvp - (m0 + mm) * nl * dvm) * (T)0.5 * fac;
          if (f != d) {  // off-diagonal: m_d += d_f( rho_t (nu_R+nu_L)/4 d_d v_f )
            const int sf = f == 0 ? 1 : f == 1 ? qb.ext[0] : qb.ext[0] * qb.ext[1];
            const int ff = f == 0 ? 1 : f == 1 ? fb.ext[0] : fb.ext[0] * fb.ext[1];
            const long long gf = g.st[f];
            T t1[2], t2[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              const int o = s ? sf : -sf;
              const int on = s ? ff : -ff;
              const long long go = s ? gf : -gf;
              int cx[3] = {c[0], c[1], c[2]};
              cx[f] += s ? 1 : -1;
              T nr2, nl2;
              nu_at(k, on, cx[f] >= 2 && cx[f] <= g.n[f] - 3, nr2, nl2);
              const T nsum = nr2 + nl2;
              const T tmp5 = z1(g, cx, d) ? T(0) : (v[o + sd] - v[o - sd]) * (T)0.5 * i1;
              const T tmp6 = tmp5 * nsum * (T)0.25;
              t1[s] = (C.v(L::RHO, idx + go) + C.v(L::RHOB, idx + go)) * tmp6;
              t2[s] = tmp6 * C.v(L::M0 + d, idx + go);
            }
            const bool zf = z1(g, c, f);
            const T hf = (T)0.5 * idx1[f];
            if (!zf) {
              dL[L::M0 + d] += (t1[1] - t1[0]) * hf;
              dL[L::EN] += (t2[1] - t2[0]) * hf;
            }
          }
        }
        // magnetic field, f != d
        int ks = 2 + D;
#pragma unroll
        for (int f = 0; f < D; ++f) {
          if (f == d) continue;
          const int k = ks++;
          const T *b = Q + k * nq + r0;
          T nr, nl;
          nu_at(k, 0, true, nr, nl);
          {  // off-diagonal: B_d -= d_f( (nu_L+nu_R)/2 d_d B_f ), e likewise with B_d
            const int sf = f == 0 ? 1 : f == 1 ? qb.ext[0] : qb.ext[0] * qb.ext[1];
            const int ff = f == 0 ? 1 : f == 1 ? fb.ext[0] : fb.ext[0] * fb.ext[1];
            const long long gf = g.st[f];
            T t1[2], t2[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              const int o = s ? sf : -sf;
              const int on = s ? ff : -ff;
              const long long go = s ? gf : -gf;
              int cx[3] = {c[0], c[1], c[2]};
              cx[f] += s ? 1 : -1;
              T nr2, nl2;
              nu_at(k, on, cx[f] >= 2 && cx[f] <= g.n[f] - 3, nr2, nl2);
              const T nsum = nr2 + nl2;
              const T tmp2 = z1(g, cx, d) ? T(0) : (b[o + sd] - b[o - sd]) * (T)0.5 * i1;
              t1[s] = tmp2 * nsum * (T)0.5;
              t2[s] = t1[s] * C.v(L::B0 + d, idx + go);
            }
            if (!z1(g, c, f)) {
              const T hf = (T)0.5 * idx1[f];
              dL[L::B0 + d] -= (t1[1] - t1[0]) * hf;
              dL[L::EN] -= (t2[1] - t2[0]) * hf;
            }
          }
          {  // diagonal: B_f += (nu_R dB+ - nu_L dB-)/dx^2 and Ohmic heating
            const T dbp = zd ? T(0) : b[sd] - b[0], dbm = zd ? T(0) : b[0] - b[-sd];
            dL[L::B0 + f] += (nr * dbp - nl * dbm) * i2;
            dL[L::EN] += ((T)0.5 * (b[0] + b[sd]) * nr * dbp - (T)0.5 * (b[0] + b[-sd]) * nl * dbm) * i2;
          }
        }
      }
    }
    __syncthreads();
  };
  if (p.hyperdif || p.has_bgb) {
    dim_pass(std::integral_constant<int, 0>{});
    dim_pass(std::integral_constant<int, 1>{});
    if constexpr (D == 3) dim_pass(std::integral_constant<int, 2>{});
  }

  if (numax > red[5] || numax != numax) red[5] = numax;
  if (active) advance_cell_any<D>(a, g, p, c, idx, h, dL, red);
}

// One launch = one RK stage of one simulation, one block per tile.
template <int D>
__global__ void __launch_bounds__(256, 2) tile_stage_kernel(StageArgs a, Geo g, Phys p) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double red[6] = {0, 0, 0, 0, 0, 0};
  tile_body<D, TileShape<D>>(a, g, p, blockIdx.x, blockIdx.y, blockIdx.z, reinterpret_cast<double *>(smraw), red);
  block_max_flush<0, 6>(red, &a.sc->red[a.red_out]);
}

// shared memory elements the tile body needs
template <int D, typename S = TileShape<D>>
__host__ __device__ constexpr int tile_smem_elems() {
  constexpr int NW = 2 + 2 * D, NQ = 2 * D + 1;
  constexpr int ex[3] = {S::TX, S::TY, D == 3 ? S::TZ : 1};
  // flux box, largest over dir
  int fl = 0, qv = 0;
  for (int dir = 0; dir < D; ++dir) {
    int n = 1, m = 1, u = 1;
    for (int e = 0; e < D; ++e) {
      n *= ex[e] + (e == dir ? 4 : 0);
      m *= ex[e] + (e == dir ? 6 : 2);
      u *= ex[e] + (e == dir ? 1 : 2);  // face box
    }
    fl = fl > NW * n ? fl : NW * n;
    qv = qv > NQ * m + NQ * u ? qv : NQ * m + NQ * u;
  }
  return fl > qv ? fl : qv;
}

}  // namespace SMAUG_NS
