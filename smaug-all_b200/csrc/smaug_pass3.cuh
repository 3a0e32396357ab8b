// smaug_pass3.cuh -- the 3-D RK stage in three passes over slabs of planes.
//
// Same operator as tile_body (smaug_tile.cuh).  A 3-D tile that keeps its own
// neighbourhood in shared memory forms every derived quantity, flux and face
// ratio of a wide halo again (272 warp instructions per cell at 8x8x8 tiles,
// 103 here).  Here each is formed once per cell and handed on through a
// workspace:
//   derive   every cell of the slab +-3 planes: what the stencils read, from
//            the stage input and the backgrounds;
//   faces    every face of every line of inner cells: the hyperviscosity
//            ratio max|d3 q| / max|d1 q| of all seven slots;
//   terms    every inner cell: flux divergences, gravity, background energy
//            terms and hyperdiffusion; the sources go to the advance pass.
// A slab is a range of planes: it bounds the workspace (kSlabBytes).
// Blast wave 128^3, mixed (ncu, one stage): derive 38 us, faces 88 us and terms
// 226 us with the workspace partly from HBM (0.85 KB of traffic per cell), where
// the tile kernel took 740 us with its epilogue.
//
// Workspace of a slab (elements of the stencil type T, vectors so that a
// neighbour costs five loads instead of thirteen; a 32-cell row of one vector
// array is contiguous, so every load is coalesced):
//   derived, NP cells (planes pz0 ..):  H_k = (b_k, v_k) pairs for k = 0..2,
//     MP = (m_0, m_1, m_2, p_T), R = (rho_t, e, rho, e_int), and with an
//     energy background BG = (B_b,0, B_b,1, B_b,2, e_b)
//   faces, NV cells (planes vz0 ..), per dimension d, at the cell left of the
//     face: X = (b_f, v_f, b_g, v_g) with f < g the other dimensions, and
//     Y = (rho, e_int, v_d, unused)
#pragma once
#include <type_traits>

#include "smaug_batch.cuh"
#include "smaug_tile.cuh"

namespace SMAUG_NS {
using namespace smaug;

template <typename T>
struct alignas(2 * sizeof(T)) Two {
  T x, y;
};
template <typename T>
struct alignas(16) Four {
  T x, y, z, w;
};
// Loads from the workspace (global, read-only in the pass that reads them).
// Volatile, so that the compiler keeps them in the order they are written in:
// hoisted together, the loads of a cell's neighbours take more registers than
// there are.
__device__ __forceinline__ Two<float> ldv(const Two<float> *p) {
  Two<float> v;
  asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ Two<double> ldv(const Two<double> *p) {
  Two<double> v;
  asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ Four<float> ldv4(const Two<float> *p) {
  Four<float> v;
  asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
  return v;
}
__device__ __forceinline__ Four<double> ldv4(const Two<double> *p) {
  const Two<double> a = ldv(p), b = ldv(p + 1);
  return {a.x, a.y, b.x, b.y};
}
__device__ __forceinline__ void stv(Two<float> *p, float x, float y) {
  *reinterpret_cast<float2 *>(p) = make_float2(x, y);
}
__device__ __forceinline__ void stv(Two<double> *p, double x, double y) {
  *reinterpret_cast<double2 *>(p) = make_double2(x, y);
}
__device__ __forceinline__ void stv(Four<float> *p, float x, float y, float z, float w) {
  *reinterpret_cast<float4 *>(p) = make_float4(x, y, z, w);
}
__device__ __forceinline__ void stv(Four<double> *p, double x, double y, double z, double w) {
  reinterpret_cast<double2 *>(p)[0] = make_double2(x, y);
  reinterpret_cast<double2 *>(p)[1] = make_double2(z, w);
}

// The workspace of a slab, for the stencil type T.  Offsets count pairs of T in
// 32 bits (a grid's NVAR * N stays below 2^31), so that an address is one
// multiply-add on one of two base pointers.
template <typename T>
struct Work3 {
  Two<T> *P, *V;
  unsigned NP, NV;
  __device__ __forceinline__ Work3(const Slab3 &s) : P((Two<T> *)s.P), V((Two<T> *)s.V), NP(s.NP), NV(s.NV) {}
  // derived arrays at cell i
  __device__ __forceinline__ unsigned H(int k, unsigned i) const { return k * NP + i; }
  __device__ __forceinline__ unsigned MP(unsigned i) const { return 3 * NP + 2 * i; }
  __device__ __forceinline__ unsigned R(unsigned i) const { return 5 * NP + 2 * i; }
  __device__ __forceinline__ unsigned BG(unsigned i) const { return 7 * NP + 2 * i; }
  // face arrays at the cell i left of the face along d
  __device__ __forceinline__ unsigned X(int d, unsigned i) const { return (4 * d) * NV + 2 * i; }
  __device__ __forceinline__ unsigned Y(int d, unsigned i) const { return (4 * d + 2) * NV + 2 * i; }
};

// ---------------------------------------------------------------- derive
// kDeriveChunk / 256 cells per thread; bound by its loads and stores (36 B in and
// 56 B out per cell in mixed precision).  The FP64 parts (p_T and the internal
// energy, both recovered by cancellation) are formed here once per cell and
// stage.  An ordinary load stays behind the stores before it, so where a block
// has an SM to itself, the state of all four cells is loaded before the first
// of them is stored (blast wave 26^3 mixed, us per launch: 10.3, so 8.5); where
// other warps cover a load's latency, the registers of that cost more than it
// gives (128^3 mixed 43.4 and 49.5, 85^3 FP64 24.4 and 28.0).
template <typename T>
struct Raw3 {
  T rho, e, m[3], b[3];
};
template <typename T>
__device__ __forceinline__ void derive_load(const CellT<3, T> &C, int idx, Raw3<T> &r) {
  using L = Lay<3>;
  r.rho = C.v(L::RHO, idx);
  r.e = C.v(L::EN, idx);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    r.m[k] = C.v(L::M0 + k, idx);
    r.b[k] = C.v(L::B0 + k, idx);
  }
}
template <typename T>
__device__ __forceinline__ void derive_cell(const CellT<3, T> &C, const Phys &p, const Work3<T> &W, const Raw3<T> &r,
                                            int idx, int pi) {
  using L = Lay<3>;
  const double rhob = C.vd(L::RHOB, idx);
  const double irtd = __drcp_rn(dbl(r.rho) + rhob);
  const T irt = num<T>(irtd);
  T bb[3] = {0, 0, 0};
  double b2 = 0, m2 = 0, bbb = 0;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    if (p.has_bgb) bb[k] = C.v(L::BB0 + k, idx);
    b2 += dbl(r.b[k]) * dbl(r.b[k]);
    m2 += dbl(r.m[k]) * dbl(r.m[k]);
    bbb += dbl(r.b[k]) * dbl(bb[k]);
  }
  const T ei = num<T>(dbl(r.e) - 0.5 * (b2 + m2 * irtd));
  const T pt = num<T>((p.gamma - 1.0) * (dbl(r.e) - 0.5 * m2 * irtd) - (p.gamma - 2.0) * (bbb + 0.5 * b2));
#pragma unroll
  for (int k = 0; k < 3; ++k) stv(W.P + W.H(k, pi), r.b[k], r.m[k] * irt);
  stv((Four<T> *)(W.P + W.MP(pi)), r.m[0], r.m[1], r.m[2], pt);
  stv((Four<T> *)(W.P + W.R(pi)), r.rho + num<T>(rhob), r.e, r.rho, ei);
  if (p.has_bgb) stv((Four<T> *)(W.P + W.BG(pi)), bb[0], bb[1], bb[2], C.v(L::EB, idx));
}

// ---------------------------------------------------------------- faces
// Face j of a line along d lies between its cells j and j+1; faces 1 .. n-3
// bound the inner cells.  A thread takes SEG consecutive faces of one line
// (along x one face, its neighbours being the neighbouring lanes' cells), one
// pair of slots at a time, each cell's q read once per pair and each first and
// third difference formed once.  q outside the grid: 0 on the right, q(5) on
// the left, as the reference's padded copies.
template <typename T, int SEG>
__device__ __forceinline__ void face_run2(const Two<T> (&q)[SEG + 5], T (&rx)[SEG], T (&ry)[SEG]) {
  auto run = [&](auto get, T(&out)[SEG]) {
    T t1[SEG + 4], t3[SEG + 2];
#pragma unroll
    for (int j = 0; j < SEG + 4; ++j) t1[j] = get(j + 1) - get(j);
#pragma unroll
    for (int j = 0; j < SEG + 2; ++j) t3[j] = vabs(vfma((T)3, t1[j + 1], -(get(j + 3) - get(j))));
#pragma unroll
    for (int m = 0; m < SEG; ++m) {
      T m1 = vabs(t1[m]);
#pragma unroll
      for (int j = m + 1; j <= m + 4; ++j) m1 = vmax(m1, vabs(t1[j]));
      const T m3 = vmax(vmax(t3[m], t3[m + 1]), t3[m + 2]);
      out[m] = m1 > 0 ? vratio(m3, m1) : T(0);
    }
  };
  run([&](int j) { return q[j].x; }, rx);
  run([&](int j) { return q[j].y; }, ry);
}

// Faces f0 .. f0+SEG-1 (at most f1) of the line along d whose cell 0 has the
// workspace offsets p0 (derived) and v0 (faces); s: the cell stride along d.
// q is read at the cells up to chi only: beyond it lies the end of the grid
// (q = 0), or cells that no kept face reads.
template <int d, typename T, int SEG>
__device__ __forceinline__ void line_faces(const Work3<T> &W, int p0, int v0, int s, int f0, int f1, int chi) {
  constexpr int f = d == 0 ? 1 : 0, h = d == 2 ? 1 : 2;  // the other dimensions, f < h
  const bool whole = f0 >= 2 && f0 + SEG + 2 <= chi;     // no pad in reach
  auto load = [&](unsigned off, int mul, Two<T>(&q)[SEG + 5]) {
    if (whole) {
      unsigned o = off + (unsigned)((p0 + (f0 - 2) * s) * mul);
#pragma unroll
      for (int j = 0; j < SEG + 5; ++j, o += (unsigned)(s * mul)) q[j] = ldv(W.P + o);
    } else {
#pragma unroll
      for (int j = 0; j < SEG + 5; ++j) {
        const int c = f0 - 2 + j;
        if (c <= chi)
          q[j] = ldv(W.P + (off + (unsigned)((p0 + (c < 0 ? 5 : c) * s) * mul)));
        else
          q[j] = {T(0), T(0)};
      }
    }
  };
  auto store = [&](unsigned o, const T(&a)[SEG], const T(&b)[SEG], const T(&c)[SEG], const T *e) {
#pragma unroll
    for (int m = 0; m < SEG; ++m, o += (unsigned)(2 * s))
      if (f0 + m <= f1) stv((Four<T> *)(W.V + o), a[m], b[m], c[m], e ? e[m] : T(0));
  };
  // (rho, e_int) first: in this order the ratios that wait for a store are the
  // fewest registers (72 -> 56 in mixed precision; blast wave 128^3 94.1 -> 87.1 us
  // per launch)
  T r[4][SEG];
  {
    Two<T> q[SEG + 5];
    load(W.R(0) + 1, 2, q);  // (rho, e_int): the second half of R
    face_run2<T, SEG>(q, r[0], r[1]);
  }
  {
    Two<T> q[SEG + 5];
    load(W.H(d, 0), 1, q);
    face_run2<T, SEG>(q, r[3], r[2]);  // (b_d's ratio is not used)
  }
  store(W.Y(d, v0 + f0 * s), r[0], r[1], r[2], nullptr);
  {
    Two<T> q[SEG + 5];
    load(W.H(f, 0), 1, q);
    face_run2<T, SEG>(q, r[0], r[1]);
  }
  {
    Two<T> q[SEG + 5];
    load(W.H(h, 0), 1, q);
    face_run2<T, SEG>(q, r[2], r[3]);
  }
  store(W.X(d, v0 + f0 * s), r[0], r[1], r[2], r[3]);
}

// ---------------------------------------------------------------- terms
// One cell's values: what its fluxes and the terms towards it are formed from.
template <typename T>
struct Nb3 {
  T b[3], v[3], m[3], pt, rt, e, rho, ei, bb[3], eb;
};
template <bool BGB, typename T>
__device__ __forceinline__ void load_nb(const Work3<T> &W, unsigned i, Nb3<T> &n) {
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const Two<T> h = ldv(W.P + W.H(k, i));
    n.b[k] = h.x;
    n.v[k] = h.y;
  }
  const Four<T> mp = ldv4(W.P + W.MP(i));
  n.m[0] = mp.x;
  n.m[1] = mp.y;
  n.m[2] = mp.z;
  n.pt = mp.w;
  const Four<T> r = ldv4(W.P + W.R(i));
  n.rt = r.x;
  n.e = r.y;
  n.rho = r.z;
  n.ei = r.w;
  if (BGB) {
    const Four<T> q = ldv4(W.P + W.BG(i));
    n.bb[0] = q.x;
    n.bb[1] = q.y;
    n.bb[2] = q.z;
    n.eb = q.w;
  }
}

// The physical fluxes along d (those of fluxes_at, in terms of v = m / rho_t):
// F[0] rho, F[1..3] momentum, F[4] e, F[5..7] B_k (none for k = d).
template <int d, bool BGB, typename T>
__device__ __forceinline__ void flux_nb(const Nb3<T> &n, T *F) {
  const T vd = n.v[d], bd = n.b[d], bdt = BGB ? bd + n.bb[d] : bd;
  F[0] = n.m[d];
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    F[1 + k] = vfma(vd, n.m[k], -(BGB ? vfma(n.b[k], bdt, n.bb[k] * bd) : n.b[k] * bdt));
    F[5 + k] = k == d ? T(0) : vfma(vd, BGB ? n.b[k] + n.bb[k] : n.b[k], -(bdt * n.v[k]));
  }
  F[1 + d] += n.pt;
  const T bv = vfma(n.b[2], n.v[2], vfma(n.b[1], n.v[1], n.b[0] * n.v[0]));
  T x = bdt * bv;
  if (BGB) x = vfma(bd, vfma(n.bb[2], n.v[2], vfma(n.bb[1], n.v[1], n.bb[0] * n.v[0])), x);
  F[4] = vfma(vd, (BGB ? n.e + n.eb : n.e) + n.pt, -x);
}

// What the terms pass reads of a simulation's descriptor, in the stencil type
// and in shared memory (converted once per block and slab).
template <typename T>
struct Consts3 {
  T chyp[8], cm[3], g[3];
};

// The sources dL of one inner cell and the maximum of its viscosities.  One
// neighbour is held at a time: its flux goes into the divergence's sum, its
// face ratio and differences into the diagonal terms, and its neighbours
// across into the off-diagonal terms differenced towards it.
template <bool BGB, typename T>
__device__ __forceinline__ void terms_cell(const Geo &g, const Phys &p, const Consts3<T> &K, const Work3<T> &W,
                                           const int *c, int pi, int vi, T *dL, T &numax) {
  using L = Lay<3>;
  const bool hyp = p.hyperdif;
  T i1[3], kd[3];
  bool zd[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    i1[d] = num<T>(__ldg(g.rdx1[d] + c[d]));
    kd[d] = num<T>(__ldg(g.dx1[d] + c[d])) * K.cm[d];  // nu = kd c_hyp * face ratio
    zd[d] = z1(g, c, d);
  }
  const int st[3] = {1, (int)g.st[1], (int)g.st[2]};
  Nb3<T> z;  // the cell
  load_nb<BGB>(W, pi, z);
  T ptb = 0;
  if (BGB) {  // the background's total pressure term (addenergyterms_cd2)
    const double bb2 = dbl(z.bb[0]) * dbl(z.bb[0]) + dbl(z.bb[1]) * dbl(z.bb[1]) + dbl(z.bb[2]) * dbl(z.bb[2]);
    ptb = num<T>((p.gamma - 1) * dbl(z.eb) - 0.5 * (p.gamma - 2) * bb2);
  }
  if (p.has_grav) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
      dL[L::M0 + k] += K.g[k] * z.rho;
      dL[L::EN] += z.rho * K.g[k] * z.v[k];
    }
  }
  auto dim = [&](auto dc) {
    constexpr int d = decltype(dc)::value;
    constexpr int f1 = d == 0 ? 1 : 0, f2 = d == 2 ? 1 : 2;
    const int s = st[d];
    // dF: F_+1 - F_-1, then 8 (F_+1 - F_-1) - (F_+2 - F_-2); gv: v likewise
    T dF[8], gv[3];
    // the terms towards the neighbour at pi + o, face ratios at vi + fo
    auto side = [&](auto sc) {
      constexpr bool plus = decltype(sc)::value;
      const int o = plus ? s : -s, fo = plus ? 0 : -s;
      Nb3<T> n;
      load_nb<BGB>(W, pi + o, n);
      {
        T F[8];
        flux_nb<d, BGB>(n, F);
#pragma unroll
        for (int k = 0; k < 8; ++k) dF[k] = plus ? F[k] : dF[k] - F[k];
        if (BGB) {
#pragma unroll
          for (int k = 0; k < 3; ++k) gv[k] = plus ? n.v[k] : gv[k] - n.v[k];
        }
      }
      if (!hyp) return;
      // diagonal terms: nu_R (q_+ - q) - nu_L (q - q_-), so the same form on
      // both sides
      const Four<T> y = ldv4(W.V + W.Y(d, vi + fo)), x = ldv4(W.V + W.X(d, vi + fo));
      const T wr = K.chyp[L::RHO] * y.x, we = K.chyp[L::EN] * y.y, wd = K.chyp[L::M0 + d] * y.z;
      const T w1 = K.chyp[L::M0 + f1] * x.y, w2 = K.chyp[L::M0 + f2] * x.w;
      const T u1 = K.chyp[L::B0 + f1] * x.x, u2 = K.chyp[L::B0 + f2] * x.z;
      numax = vmax(numax, kd[d] * vmax(vmax(vmax(wr, we), wd), vmax(vmax(w1, w2), vmax(u1, u2))));
      if (!zd[d]) {
        const T k2 = kd[d] * (i1[d] * i1[d]);
        dL[L::RHO] = vfma(wr * k2, n.rho - z.rho, dL[L::RHO]);
        T de = (we * k2) * (n.ei - z.ei);
        const T rs = z.rt + n.rt;
        // momentum m_f: the face values of rho_t and m_f times nu dv_f
        auto mom = [&](int f, T w) {
          const T t = (w * (k2 * (f == d ? (T)0.5 : (T)0.25))) * (n.v[f] - z.v[f]);
          dL[L::M0 + f] = vfma(rs, t, dL[L::M0 + f]);
          de = vfma(z.m[f] + n.m[f], t, de);
        };
        mom(d, wd);
        mom(f1, w1);
        mom(f2, w2);
        // field B_f, f != d, and Ohmic heating
        auto mag = [&](int f, T u) {
          const T t = (u * k2) * (n.b[f] - z.b[f]);
          dL[L::B0 + f] += t;
          de = vfma((T)0.5 * (z.b[f] + n.b[f]), t, de);
        };
        mag(f1, u1);
        mag(f2, u2);
        dL[L::EN] += de;
        // off-diagonal terms differenced along d: for each other dimension t,
        //   m_t += d_d( rho_t (nu_R + nu_L)/4 d_t v_d ),  B_t -= d_d( (nu_R + nu_L)/2 d_t B_d )
        // with nu of v_d and B_d along t, zero where the neighbour along d is
        // not an inner cell; the gradient along t counts as zero at a closed end
        const bool in = plus ? c[d] + 1 <= g.n[d] - 3 : c[d] - 1 >= 2;
        auto off = [&](auto tc) {
          constexpr int t = decltype(tc)::value;
          constexpr int sec = d == (t == 0 ? 1 : 0) ? 0 : 1;  // d's place among t's other dimensions
          if (zd[t] || !in) return;
          const int q = st[t];
          const Two<T> hp = ldv(W.P + W.H(d, pi + o + q)), hm = ldv(W.P + W.H(d, pi + o - q));
          const Two<T> nr = ldv(W.V + (W.X(t, vi + o) + sec)), nl = ldv(W.V + (W.X(t, vi + o - q) + sec));
          const T kt = (kd[t] * i1[t]) * ((plus ? (T)0.25 : (T)-0.25) * i1[d]);
          const T tb = (kt * (K.chyp[L::B0 + d] * (T)0.5)) * ((hp.x - hm.x) * (nr.x + nl.x));
          const T tm = (kt * (K.chyp[L::M0 + d] * (T)0.25)) * ((hp.y - hm.y) * (nr.y + nl.y));
          dL[L::M0 + t] = vfma(n.rt, tm, dL[L::M0 + t]);
          dL[L::B0 + t] -= tb;
          dL[L::EN] += vfma(n.m[t], tm, -(n.b[t] * tb));
        };
        off(std::integral_constant<int, f1>{});
        off(std::integral_constant<int, f2>{});
      }
    };
    side(std::true_type{});
    side(std::false_type{});
    // flux divergence -(8 (F_+1 - F_-1) - (F_+2 - F_-2)) / (12 dx), and the
    // background energy terms' velocity gradients
    if (z4(g, c, d)) return;
    const T w12 = i1[d] * (T)(1.0 / 12.0);
    {
      T F2[8], F[8];
      Nb3<T> n;
      load_nb<BGB>(W, pi + 2 * s, n);
      flux_nb<d, BGB>(n, F2);
      if (BGB) {
#pragma unroll
        for (int k = 0; k < 3; ++k) gv[k] = vfma((T)8, gv[k], -n.v[k]);
      }
      load_nb<BGB>(W, pi - 2 * s, n);
      flux_nb<d, BGB>(n, F);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if (k == 5 + d) continue;
        dL[k] = vfma(-vfma((T)8, dF[k], -(F2[k] - F[k])), w12, dL[k]);
      }
      if (BGB) {
        T sum = -ptb * (gv[d] + n.v[d]);
#pragma unroll
        for (int k = 0; k < 3; ++k) sum = vfma(z.bb[d] * z.bb[k], gv[k] + n.v[k], sum);
        dL[L::EN] = vfma(sum, w12, dL[L::EN]);
      }
    }
  };
  dim(std::integral_constant<int, 0>{});
  dim(std::integral_constant<int, 1>{});
  dim(std::integral_constant<int, 2>{});
}

}  // namespace SMAUG_NS
