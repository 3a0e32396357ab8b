// smaug_pairs2.cuh -- the 2-D mixed stage body on pairs of cells.
//
// The three phases of tile_body2 (smaug_tile2.cuh) with two cells per thread,
// TY/2 rows apart, as the two lanes of packed FP32 instructions (f32x2,
// smaug_pair.cuh).  The boxes in shared memory hold such pairs: entry (x, r)
// is the q of rows r and r + TY/2 of the tile widened by 3, so that every
// neighbour of both cells is one 64-bit load with nothing to repack, free of
// bank conflicts (16 lanes take 16 consecutive pairs).  The six rows in the
// middle of the box are stored twice.  The scalar body was bound by
// instruction issue (69 % of the slots busy, 54 warp instructions per cell);
// this one needs 34 and is bound by the latency of its chains at 16 warps per
// SM (50 % busy): 1531x1022 vortex, stage kernel 124 -> 104 us (ncu), ensemble
// of 24 2.02 -> 1.82 ms per step.
//
// The lane type P is f2, or f1 (one cell per thread): the same operations, so
// the same bits, with twice the threads per tile where a grid is too small to
// fill the chip and a thread's own chain of instructions is what it waits for
// (the rule is in BatchLaunch).
//
// FP32 only: FP64 has no packed form.  All tile shapes and lane types give the
// same bits: no product is added to anything but by an explicit fma (prod below
// for sums of products), because ptxas contracts packed mul and add (.rn ones
// too) where it sees fit.
#pragma once
#include <type_traits>

#include "smaug_pair.cuh"
#include "smaug_tile2.cuh"

namespace SMAUG_NS {
using namespace smaug;

// Box sizes of the body for a TX x TY tile (in elements of P).
template <typename S, typename P>
struct Box2P {
  static constexpr int LANES = sizeof(P) / sizeof(float);
  static constexpr int TX = S::TX, H = S::TY / LANES, NT = TX * H;
  static constexpr int NQS = 14;                        // q slots per cell (q_from)
  static constexpr int QX = TX + 6, QN = QX * (H + 6);  // q: tile +-3
  // face ratios along x: faces x+1/2 for x in [-1, TX), rows -1 .. H; along y:
  // faces y+1/2 for y in [-1, H), columns -1 .. TX
  static constexpr int V0X = TX + 1, V0N = (TX + 1) * (H + 2);
  static constexpr int V1X = TX + 2, V1N = (TX + 2) * (H + 1);
  static constexpr int OV0 = NQS * QN, OV1 = OV0 + 5 * V0N, ELEMS = OV1 + 5 * V1N;
};

// The fluxes along dir of a pair from its q slots (flux_q's): F[0] rho, F[1]
// m_x, F[2] m_y, F[3] e, F[4] B of the other dimension.
template <int dir, int QN, bool BGB, typename P>
__device__ __forceinline__ void flux_pair(const P *Q, int r, P *F) {
  const P v0 = Q[2 * QN + r], v1 = Q[3 * QN + r], b0 = Q[4 * QN + r], b1 = Q[5 * QN + r];
  const P m0 = Q[7 * QN + r], m1 = Q[8 * QN + r], e = Q[9 * QN + r], pt = Q[10 * QN + r];
  P bb0, bb1, eb;
  if (BGB) {
    bb0 = Q[11 * QN + r];
    bb1 = Q[12 * QN + r];
    eb = Q[13 * QN + r];
  }
  const P vd = dir == 0 ? v0 : v1, bd = dir == 0 ? b0 : b1;
  const P nbt = pneg(BGB ? bd + (dir == 0 ? bb0 : bb1) : bd);  // -(B_dir with the background)
  F[0] = dir == 0 ? m0 : m1;
  F[1] = pfma(b0, nbt, vd * m0);
  F[2] = pfma(b1, nbt, vd * m1);
  P x = nbt * pfma(b1, v1, b0 * v0);
  if (BGB) {
    const P nb = pneg(bd);
    F[1] = pfma(bb0, nb, F[1]);
    F[2] = pfma(bb1, nb, F[2]);
    x = pfma(nb, pfma(bb1, v1, bb0 * v0), x);
  }
  if (dir == 0)
    F[1] = F[1] + pt;
  else
    F[2] = F[2] + pt;
  F[3] = pfma(vd, (BGB ? e + eb : e) + pt, x);
  const P bf = dir == 0 ? b1 : b0;
  F[4] = pfma(vd, BGB ? bf + (dir == 0 ? bb1 : bb0) : bf, nbt * (dir == 0 ? v1 : v0));
}

// The face ratios of SEG consecutive faces of a line of pairs at q (stride s)
// into dst (stride ds).
template <int SEG, typename P>
__device__ __forceinline__ void face_run_pair(const P *q, int s, P *dst, int ds) {
  const P three = splat<P>(3.0f);
  P v[SEG + 5], t1[SEG + 4], t3[SEG + 2];
#pragma unroll
  for (int j = 0; j < SEG + 5; ++j) v[j] = q[j * s];
#pragma unroll
  for (int j = 0; j < SEG + 4; ++j) t1[j] = v[j + 1] - v[j];
#pragma unroll
  for (int j = 0; j < SEG + 2; ++j) t3[j] = pfma(three, t1[j + 1], v[j] - v[j + 3]);
#pragma unroll
  for (int m = 0; m < SEG; ++m) {
    float r[2];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k * sizeof(float) >= sizeof(P)) continue;
      auto g = [&](P x) { return fabsf(lane(x, k)); };
      const float m1 = fmaxf(fmaxf(fmaxf(g(t1[m]), g(t1[m + 1])), g(t1[m + 2])), fmaxf(g(t1[m + 3]), g(t1[m + 4])));
      const float m3 = fmaxf(fmaxf(g(t3[m]), g(t3[m + 1])), g(t3[m + 2]));
      r[k] = m1 > 0.0f ? vratio(m3, m1) : 0.0f;
    }
    dst[m * ds] = pack<P>(r[0], r[1]);
  }
}

template <bool BGB, typename P, typename S>
__device__ __forceinline__ void pairs_body2(const StageArgs &a, const Geo &g, const Phys &p, const float *scm, int bx,
                                            int by, int nbx, int nby, P *sm, float &red) {
  using L = Lay<2>;
  using B = Box2P<S, P>;
  constexpr int LANES = B::LANES;
  constexpr int TX = B::TX, H = B::H, TY = S::TY, NT = B::NT, QN = B::QN, QX = B::QX;
  P *Q = sm, *V0 = sm + B::OV0, *V1 = sm + B::OV1;
  const int t = threadIdx.x;
  const int ox = 2 + bx * TX, oy = 2 + by * TY;
  const int n0 = g.n[0], n1 = g.n[1];
  const CellT<2, float> C{a.in32, a.bg, g.N};
  if (nbx >= 0) prefetch_qbox_rows<float, TX, TY, NT>(a, g, p, nbx, nby);

  // ------------------------------------------------ phase A: q on the tile +-3
  {
    float *Qs = reinterpret_cast<float *>(Q);
    constexpr int N = QX * (TY + 6), NA = (N + NT - 1) / NT;
#pragma unroll
    for (int u = 0; u < NA; ++u) {
      const int rr = t + u * NT;
      if (rr >= N) continue;
      const int row = rr / QX, col = rr - row * QX;
      int cx = ox - 3 + col, cy = oy - 3 + row;
      const bool inx = cx >= 0 && cx < n0, iny = cy >= 0 && cy < n1;
      float q[B::NQS];
      // pads of the padded copies: right 0, left q(5); corners never read
      if ((!inx && !iny) || cx >= n0 || cy >= n1) {
#pragma unroll
        for (int k = 0; k < B::NQS; ++k) q[k] = 0;
      } else {
        if (cx < 0) cx = 5;
        if (cy < 0) cy = 5;
        QRaw<float> raw;
        q_load<float>(C, cx + (long long)cy * g.st[1], BGB, raw);
        q_from<float>(raw, p.gamma, q);
      }
      float *lo = Qs + LANES * (col + QX * row), *hi = lo - LANES * QX * H + 1;
      if (LANES == 1 || row < H + 6) {
#pragma unroll
        for (int k = 0; k < (BGB ? 14 : 11); ++k) lo[LANES * k * QN] = q[k];
      }
      if (LANES == 2 && row >= H) {
#pragma unroll
        for (int k = 0; k < (BGB ? 14 : 11); ++k) hi[LANES * k * QN] = q[k];
      }
    }
  }
  __syncthreads();

  // ------------------------------------------------ phase B: face ratios along x and y
  if (p.hyperdif) {
    // (runs of at most nine faces; the last run of a line is shifted back to
    // end at its last face, the shared faces written twice with the same value)
    constexpr int RUN = 9;
    constexpr int SEG0 = RUN < TX + 1 ? RUN : TX + 1, SEG1 = RUN < H + 1 ? RUN : H + 1;
    constexpr int NS0 = (TX + 1 + SEG0 - 1) / SEG0, NS1 = (H + 1 + SEG1 - 1) / SEG1;
    constexpr int NU0 = 5 * (H + 2) * NS0, NU1 = 5 * (TX + 2) * NS1;
    for (int u = t; u < NU0 + NU1; u += NT) {
      if (u < NU0) {  // along x: slots rho, e_int, v_x, v_y, B_y
        const int s = u % NS0, line = (u / NS0) % (H + 2), k = u / (NS0 * (H + 2));
        const int f0 = min(s * SEG0, TX + 1 - SEG0);
        face_run_pair<SEG0>(Q + (k < 4 ? k : 5) * QN + f0 + QX * (line + 2), 1, V0 + k * B::V0N + f0 + B::V0X * line, 1);
      } else {  // along y: B_x in the last slot
        const int w = u - NU0, line = w % (TX + 2), s = (w / (TX + 2)) % NS1, k = w / ((TX + 2) * NS1);
        const int f0 = min(s * SEG1, H + 1 - SEG1);
        face_run_pair<SEG1>(Q + k * QN + (line + 2) + QX * f0, QX, V1 + k * B::V1N + line + B::V1X * f0, B::V1X);
      }
    }
  }
  __syncthreads();

  // ------------------------------------------------ phase C: the pair's sources
  const int tx = t % TX, ty = t / TX;
  const int c0 = ox + tx, cl = oy + ty, ch = cl + H;  // x, and y of the two cells
  const bool al = c0 <= n0 - 3 && cl <= n1 - 3, ah = LANES == 2 && c0 <= n0 - 3 && ch <= n1 - 3;
  if (!al) return;
  // -0 in a form ptxas cannot see through (grids have fewer than 2^24 cells a
  // side): a product formed as fma(a, b, -0) is rounded by itself, so sums over
  // the two sides of a cell do not depend on their order and mirror images stay
  // mirror images.
  const P nz = splat<P>(__int_as_float((int)(0x80000000u | ((unsigned)n0 >> 24))));
  auto prod = [&](P x, P y) { return pfma(x, y, nz); };
  const int gl = cl, gh = LANES == 2 ? min(ch, n1 - 3) : cl;  // (a missing second cell repeats an inner row: in bounds, not stored)
  const int r0 = (tx + 3) + QX * (ty + 3);
  const int idl = c0 + gl * (int)g.st[1], idh = c0 + gh * (int)g.st[1];
  const float ix = num<float>(__ldg(g.rdx1[0] + c0));
  const P i1[2] = {splat<P>(ix), pack<P>(num<float>(__ldg(g.rdx1[1] + gl)), num<float>(__ldg(g.rdx1[1] + gh)))};
  // where gradients count as zero near a closed end (z4, z1), per lane; all
  // false in tiles that touch none
  const bool closed = (g.btype[0] != 0 && (ox == 2 || ox + TX > n0 - 4)) || (g.btype[1] != 0 && (oy == 2 || oy + TY > n1 - 4));
  const int zl[3] = {c0, gl, 0}, zh[3] = {c0, gh, 0};
  P dL[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) dL[f] = splat<P>(0.0f);
  float numl = 0.0f, numh = 0.0f;
  const P zrho = Q[r0], zei = Q[QN + r0], zrt = Q[6 * QN + r0];
  const P zv[2] = {Q[2 * QN + r0], Q[3 * QN + r0]}, zb[2] = {Q[4 * QN + r0], Q[5 * QN + r0]};
  const P zm[2] = {Q[7 * QN + r0], Q[8 * QN + r0]};
  if (p.has_grav) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const P gk = splat<P>(num<float>(p.g[k]));
      dL[L::M0 + k] = pfma(gk, zrho, dL[L::M0 + k]);
      dL[L::EN] = pfma(gk * zrho, zv[k], dL[L::EN]);
    }
  }
  P ptb, bbz[2];
  if (BGB) {  // the background's total pressure term (addenergyterms_cd2)
    float pl[2] = {0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      if (k >= LANES) continue;
      const int i = k ? idh : idl;
      const double x = C.vd(L::BB0, i), y = C.vd(L::BB0 + 1, i);
      pl[k] = num<float>((p.gamma - 1) * C.vd(L::EB, i) - 0.5 * (p.gamma - 2) * (x * x + y * y));
    }
    ptb = pack<P>(pl[0], pl[1]);
    bbz[0] = Q[11 * QN + r0];
    bbz[1] = Q[12 * QN + r0];
  }
  auto dim = [&](auto dc) {
    constexpr int d = decltype(dc)::value, fo = 1 - d;
    constexpr int sd = d == 0 ? 1 : QX, sq = d == 0 ? QX : 1;  // q strides along d and across
    const P w12 = i1[d] * splat<P>(1.0f / 12.0f);
    {
      // flux divergence: -(8 (F_+1 - F_-1) - (F_+2 - F_-2)) / (12 dx)
      P Fp[5], Fm[5], e[5];
      flux_pair<d, QN, BGB>(Q, r0 + 2 * sd, Fp);
      flux_pair<d, QN, BGB>(Q, r0 - 2 * sd, Fm);
#pragma unroll
      for (int k = 0; k < 5; ++k) e[k] = Fp[k] - Fm[k];
      flux_pair<d, QN, BGB>(Q, r0 + sd, Fp);
      flux_pair<d, QN, BGB>(Q, r0 - sd, Fm);
#pragma unroll
      for (int k = 0; k < 5; ++k) e[k] = pfma(splat<P>(-8.0f), Fp[k] - Fm[k], e[k]);
      if (BGB) {  // background energy terms along d
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          const P *v = Q + (2 + k) * QN + r0;
          const P gv = pfma(splat<P>(8.0f), v[sd] - v[-sd], v[-2 * sd] - v[2 * sd]);
          if (k == d) e[3] = pfma(pneg(ptb), gv, e[3]);
          e[3] = pfma(bbz[d] * bbz[k], gv, e[3]);
        }
      }
      if (closed) {
        const bool l = !z4(g, zl, d), h = !z4(g, zh, d);
#pragma unroll
        for (int k = 0; k < 5; ++k) e[k] = keep(l, h, e[k]);
      }
#pragma unroll
      for (int k = 0; k < 5; ++k) {
        const int f = k < 4 ? k : L::B0 + fo;
        dL[f] = pfma(e[k], w12, dL[f]);
      }
    }
    if (!p.hyperdif) return;
    const P *V = d == 0 ? V0 : V1;
    constexpr int VN = d == 0 ? B::V0N : B::V1N;
    constexpr int fs = d == 0 ? 1 : B::V1X, sv = d == 0 ? B::V0X : 1;  // face strides along d and across
    const int fr = d == 0 ? (tx + 1) + B::V0X * (ty + 1) : (tx + 1) + B::V1X * (ty + 1);
    const P dx = d == 0 ? splat<P>(num<float>(__ldg(g.dx1[0] + c0)))
                         : pack<P>(num<float>(__ldg(g.dx1[1] + gl)), num<float>(__ldg(g.dx1[1] + gh)));
    const P kd = dx * splat<P>(scm[d]);
    const P kr = kd * splat<P>(num<float>(p.chyp[L::RHO])), ke = kd * splat<P>(num<float>(p.chyp[L::EN]));
    const P km[2] = {kd * splat<P>(num<float>(p.chyp[L::M0])), kd * splat<P>(num<float>(p.chyp[L::M0 + 1]))};
    const P kb = kd * splat<P>(num<float>(p.chyp[L::B0 + fo]));
    const P i2 = i1[d] * i1[d];
    // diagonal terms nu_R (q_+ - q) - nu_L (q - q_-): the same form on both
    // sides; D: rho, m_x, m_y, e, B_f
    P D[5];
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int o = r0 + (side ? -sd : sd), fv = fr - (side ? fs : 0);
      const P nr = kr * V[fv], ne = ke * V[VN + fv], nm[2] = {km[0] * V[2 * VN + fv], km[1] * V[3 * VN + fv]};
      const P nb = kb * V[4 * VN + fv];
      numl = fmaxf(fmaxf(numl, fmaxf(lane(nr, 0), lane(ne, 0))), fmaxf(fmaxf(lane(nm[0], 0), lane(nm[1], 0)), lane(nb, 0)));
      if (LANES == 2)
        numh = fmaxf(fmaxf(numh, fmaxf(lane(nr, 1), lane(ne, 1))), fmaxf(fmaxf(lane(nm[0], 1), lane(nm[1], 1)), lane(nb, 1)));
      const P dr = Q[o] - zrho;
      const P rs = zrt + Q[6 * QN + o];
      P es = ne * (Q[QN + o] - zei);
#pragma unroll
      for (int f = 0; f < 2; ++f) {
        const P tv = (nm[f] * splat<P>(f == d ? 0.5f : 0.25f)) * (Q[(2 + f) * QN + o] - zv[f]);
        const P tm = prod(rs, tv);
        D[1 + f] = side ? D[1 + f] + tm : tm;
        es = pfma(zm[f] + Q[(7 + f) * QN + o], tv, es);
      }
      const P qb = Q[(4 + fo) * QN + o];
      const P db = qb - zb[fo];
      es = pfma(splat<P>(0.5f) * (zb[fo] + qb), nb * db, es);
      const P tr = prod(nr, dr), tb = prod(nb, db);
      D[0] = side ? D[0] + tr : tr;
      D[3] = side ? D[3] + es : es;
      D[4] = side ? D[4] + tb : tb;
    }
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int f = k < 4 ? k : L::B0 + fo;
      if (closed) D[k] = keep(!z1(g, zl, d), !z1(g, zh, d), D[k]);
      dL[f] = pfma(D[k], i2, dL[f]);
    }
    // off-diagonal terms: the gradients along d of v and B of the other
    // dimension with nu along d, differenced across:
    //   m_d += d_f( rho_t (nu_R + nu_L)/4 d_d v_f ),  B_d -= d_f( (nu_R + nu_L)/2 d_d B_f )
    // and the energy with m_d and B_d; nu is zero off the inner cells
    P O[3];
    const P hq = i1[d] * (splat<P>(0.125f) * i1[fo]);
    const P cv = km[fo] * (splat<P>(0.5f) * hq), cb = pneg(kb * hq);
    const P nv = pneg(cv), mb = pneg(cb);
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int o = r0 + (side ? -sq : sq), fv = fr + (side ? -sv : sv);
      const int x = (d == 0 ? gl : c0) + (side ? -1 : 1), xh = (d == 0 ? gh : c0) + (side ? -1 : 1);
      const int hi = (d == 0 ? n1 : n0) - 3;
      const bool l = x >= 2 && x <= hi, h = xh >= 2 && xh <= hi;
      const P vv = V[(2 + fo) * VN + fv] + V[(2 + fo) * VN + fv - fs], vb = V[4 * VN + fv] + V[4 * VN + fv - fs];
      const P *qv = Q + (2 + fo) * QN + o, *qb = Q + (4 + fo) * QN + o;
      const P tv = keep(l, h, (side ? nv : cv) * ((qv[sd] - qv[-sd]) * vv));
      const P tb = keep(l, h, (side ? mb : cb) * ((qb[sd] - qb[-sd]) * vb));
      const P om = prod(Q[6 * QN + o], tv);
      O[0] = side ? O[0] + om : om;
      O[1] = side ? O[1] + tb : tb;
      const P oe = pfma(Q[(7 + d) * QN + o], tv, Q[(4 + d) * QN + o] * tb);
      O[2] = side ? O[2] + oe : oe;
    }
    if (closed) {
      const bool l = !z1(g, zl, 0) && !z1(g, zl, 1), h = !z1(g, zh, 0) && !z1(g, zh, 1);
#pragma unroll
      for (int k = 0; k < 3; ++k) O[k] = keep(l, h, O[k]);
    }
    dL[L::M0 + d] = dL[L::M0 + d] + O[0];
    dL[L::B0 + d] = dL[L::B0 + d] + O[1];
    dL[L::EN] = dL[L::EN] + O[2];
  };
  // (y first: one of eight orders of these sums that are equally exact.  After
  // 100 steps of a 96^2 vortex they lie between 8.4e-4 and 1.4e-3 of the FMA-free
  // FP64 build, this one at 1.19e-3, as the scalar kernel before it; after 1000
  // steps, a chaotic run by then, between 1.65e-2 and 1.2e-1, this one at 1.65e-2:
  // the lowest, which is why it was taken and says nothing about its exactness.)
  dim(std::integral_constant<int, 1>{});
  dim(std::integral_constant<int, 0>{});
  float dl[6], dh[6];
#pragma unroll
  for (int f = 0; f < 6; ++f) {
    dl[f] = lane(dL[f], 0);
    dh[f] = lane(dL[f], 1);
  }
  if (p.divb) {
    divb_sources<float>(C, g, p, zl, idl, dl);
    if (LANES == 2) divb_sources<float>(C, g, p, zh, idh, dh);
  }
  store_sources<2>(a, g, idl, dl);
  if (numl > red || numl != numl) red = numl;
  if (ah) {
    store_sources<2>(a, g, idh, dh);
    if (numh > red || numh != numh) red = numh;
  }
}

}  // namespace SMAUG_NS
