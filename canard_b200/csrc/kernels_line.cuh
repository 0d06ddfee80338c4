// One-lane line solves (k_line): one warp per 32 lines, one line per lane, the
// tile of whole lines in shared memory. Included by kernels.cuh.
//
// Both sweeps run in blocks of eight rows that follow one another without a
// break: the closure rows and the leftover rows that do not fill a block stand
// at the line's ends, the block loop only checks that the next rows have
// arrived, and a finished chunk is stored as soon as a block has passed it.
// The rows of the factor tables that are not constant (the first 30 to 70, and
// the last three) are staged in shared memory while the tile's copies are in
// flight. With the tables read from L1/L2 and the sweeps cut at every chunk, a
// 257-point FP64 derivative tile spent 6 of its 10.7 thousand forward cycles and
// 4 of its 10.1 thousand backward cycles on 36 table rows and some 30 rows
// outside the blocks (per-CTA clock stamps); a row inside a block costs 24
// cycles forward and 21 backward.
#pragma once

// Where a line's factors are: rows [0, T) staged in shared memory as (l1, l2)
// and (u1, u2, u3, unused), rows [c0, c1] in registers (bitwise constant
// there), the others in the tables in global memory (only where the constant
// range starts above row T).
template <class RS>
struct LineFac {
  const RS* fl;
  const RS* bu;
  const RS* __restrict__ g;  // l1, l2, u1, u2, u3, each L long
  RS cl1, cl2, cu1, cu2, cu3;
  int T, c0, c1, L;
  __device__ __forceinline__ void row_l(int i, RS& a, RS& b) const {
    if (i < T) { a = fl[2 * i]; b = fl[2 * i + 1]; }
    else if (i >= c0 && i <= c1) { a = cl1; b = cl2; }
    else { a = __ldg(g + i); b = __ldg(g + L + i); }
  }
  __device__ __forceinline__ void row_u(int i, RS& a, RS& b, RS& c) const {
    if (i < T) { a = bu[4 * i]; b = bu[4 * i + 1]; c = bu[4 * i + 2]; }
    else if (i >= c0 && i <= c1) { a = cu1; b = cu2; c = cu3; }
    else { a = __ldg(g + 2 * L + i); b = __ldg(g + 3 * L + i); c = __ldg(g + 4 * L + i); }
  }
  // rows i..i+B-1, all staged or all read from the tables (a block that
  // straddles the two is read from the tables)
  template <int B>
  __device__ __forceinline__ void rows_l(int i, RS (&a)[B], RS (&b)[B]) const {
    if (i + B <= T) {
#pragma unroll
      for (int k = 0; k < B; ++k) { a[k] = fl[2 * (i + k)]; b[k] = fl[2 * (i + k) + 1]; }
    } else {
#pragma unroll
      for (int k = 0; k < B; ++k) { a[k] = __ldg(g + i + k); b[k] = __ldg(g + L + i + k); }
    }
  }
  // rows i, i-1, ..., i-B+1
  template <int B>
  __device__ __forceinline__ void rows_u(int i, RS (&a)[B], RS (&b)[B], RS (&c)[B]) const {
    if (i < T) {
#pragma unroll
      for (int k = 0; k < B; ++k) { a[k] = bu[4 * (i - k)]; b[k] = bu[4 * (i - k) + 1]; c[k] = bu[4 * (i - k) + 2]; }
    } else {
#pragma unroll
      for (int k = 0; k < B; ++k) {
        a[k] = __ldg(g + 2 * L + i - k); b[k] = __ldg(g + 3 * L + i - k); c[k] = __ldg(g + 4 * L + i - k);
      }
    }
  }
};

// A tile arrives in NC chunks of CR positions (rows), chunk 0 and the last
// chunk first (the closures read both ends), then 1, 2, ...
struct ChunkIn {
  uint64_t* bars;
  int CR, NC, L;
  int next;   // next middle chunk to wait for
  int ready;  // rows [0, ready) and the last chunk have arrived
  __device__ __forceinline__ bool wait_next(int* err) {
    if (next >= NC - 1) { ready = L; return true; }
    if (!mbar_wait(bars + next, 0)) { atomicExch(err, kErrTimeout); return false; }
    ++next;
    ready = (next >= NC - 1) ? L : next * CR;
    return true;
  }
  // rows up to `row` have arrived
  __device__ __forceinline__ bool need(int row, int* err) {
    while (row >= ready && ready < L) {
      if (!wait_next(err)) return false;
      __syncwarp();
    }
    return true;
  }
};

// One lane's line in a tile. ST 32: [row][32 lines]. ST 1: an xi tile, one or
// two boxes of [line][W] positions (row i >= W lies D elements further on);
// blocks of rows then move in 16-byte accesses, free of bank conflicts because
// a box's line pitch W is an odd number of 16-byte units. A block starts at a
// multiple of 16 bytes, and W is one too, so no access straddles two boxes.
template <int ST, class TT>
struct LineTile {
  TT* p;
  int W, D;
  __device__ __forceinline__ TT& operator()(int i) const { return ST == 1 ? p[i + (i >= W ? D : 0)] : p[i * ST]; }
  template <int B>
  __device__ __forceinline__ void ld(int i, TT* v) const {
    if constexpr (ST == 1 && sizeof(TT) == 8) {
#pragma unroll
      for (int k = 0; k < B; k += 2) {
        const double2 d = *reinterpret_cast<const double2*>(&(*this)(i + k));
        v[k] = d.x; v[k + 1] = d.y;
      }
    } else if constexpr (ST == 1) {
#pragma unroll
      for (int k = 0; k < B; k += 4) {
        const float4 d = *reinterpret_cast<const float4*>(&(*this)(i + k));
        v[k] = d.x; v[k + 1] = d.y; v[k + 2] = d.z; v[k + 3] = d.w;
      }
    } else {
#pragma unroll
      for (int k = 0; k < B; ++k) v[k] = p[(i + k) * ST];
    }
  }
  template <int B>
  __device__ __forceinline__ void st(int i, const TT* v) const {
    if constexpr (ST == 1 && sizeof(TT) == 8) {
#pragma unroll
      for (int k = 0; k < B; k += 2) *reinterpret_cast<double2*>(&(*this)(i + k)) = make_double2(v[k], v[k + 1]);
    } else if constexpr (ST == 1) {
#pragma unroll
      for (int k = 0; k < B; k += 4)
        *reinterpret_cast<float4*>(&(*this)(i + k)) = make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]);
    } else {
#pragma unroll
      for (int k = 0; k < B; ++k) p[(i + k) * ST] = v[k];
    }
  }
};

// The interior right-hand sides of rows i..i+B-1. The window w holds the
// originals s[i-LO .. i+LO-1+CY] on entry (rows up to i-1 are overwritten by
// then) and the same moved by B rows on return; rows i+LO+CY.. are read. CY
// rows of extra look-ahead keep the reads of a row-major tile aligned.
template <int OP, class TT>
struct Stencil {
  TT fa, fb, fc, al, be;  // the filter's weights; the interior left-hand side where DIRECT
};
template <int OP, int CY>
struct WinSize {
  static constexpr int LO = OP == 0 ? 2 : 3, N = 2 * LO + CY;
};
template <int OP, bool DIRECT, class TT>
__device__ __forceinline__ TT rhs_row(const TT* w, const Stencil<OP, TT>& c) {
  if constexpr (OP == 0) {
    return TT(CA_AA) * (w[3] - w[1]) + TT(CA_AB) * (w[4] - w[0]);
  } else {
    const TT rk = w[3] + w[3];
    TT r = (c.fa * ((w[2] + w[4]) - rk) + c.fb * ((w[1] + w[5]) - rk)) + c.fc * ((w[0] + w[6]) - rk);
    // the filtered values' own right-hand side (B x)_i = (A x)_i + ((B - A) x)_i
    if constexpr (DIRECT) r = r + ((w[3] + c.al * (w[2] + w[4])) + c.be * (w[1] + w[5]));
    return r;
  }
}
template <int B, int OP, int ST, int CY, bool DIRECT, class TT>
__device__ __forceinline__ void rhs_rows(const LineTile<ST, TT>& s, int i, const Stencil<OP, TT>& c,
                                         TT (&w)[WinSize<OP, CY>::N], TT (&r)[B]) {
  constexpr int NW = WinSize<OP, CY>::N, LO = WinSize<OP, CY>::LO;
  TT win[NW + B];
#pragma unroll
  for (int k = 0; k < NW; ++k) win[k] = w[k];
  s.template ld<B>(i + LO + CY, win + NW);
#pragma unroll
  for (int k = 0; k < B; ++k) r[k] = rhs_row<OP, DIRECT, TT>(win + k, c);
#pragma unroll
  for (int k = 0; k < NW; ++k) w[k] = win[B + k];
}

// Forward elimination of rows i..i+B-1 from their right-hand sides r and
// factors l1, l2.
template <int B, int ST, class TT, class RS>
__device__ __forceinline__ void chain_fwd(const LineTile<ST, TT>& s, int i, const RS (&l1)[B], const RS (&l2)[B],
                                          const TT (&r)[B], RS& am2, RS& am1) {
  TT a[B];
#pragma unroll
  for (int k = 0; k < B; ++k) {
    const RS v = (RS(r[k]) - l1[k] * am2) - l2[k] * am1;
    a[k] = TT(v);
    am2 = am1;
    am1 = v;
  }
  s.template st<B>(i, a);
}
// The same for eight rows, with the right-hand sides (and, FAC 1 or 2, the
// factors) of the next eight formed row by row in between: a scheduler that
// holds one warp fills the chain's latency only with work that stands next to
// it in the program. FAC: 0 the factors stay, 1 the next rows' staged ones, 2
// the next rows' from the tables.
template <int FAC, int OP, int ST, int CY, bool DIRECT, class TT, class RS>
__device__ __forceinline__ void fwd_pipe(const LineTile<ST, TT>& s, int i, const LineFac<RS>& F, const Stencil<OP, TT>& c,
                                         TT (&w)[WinSize<OP, CY>::N], RS (&l1)[8], RS (&l2)[8], TT (&r)[8], RS& am2,
                                         RS& am1) {
  constexpr int NW = WinSize<OP, CY>::N, LO = WinSize<OP, CY>::LO;
  TT win[NW + 8], a[8];
#pragma unroll
  for (int k = 0; k < NW; ++k) win[k] = w[k];
  s.template ld<8>(i + 8 + LO + CY, win + NW);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const RS v = (RS(r[k]) - l1[k] * am2) - l2[k] * am1;
    a[k] = TT(v);
    am2 = am1;
    am1 = v;
    if (ST != 1) s(i + k) = a[k];
    r[k] = rhs_row<OP, DIRECT, TT>(win + k, c);
    if (FAC == 1) { l1[k] = F.fl[2 * (i + 8 + k)]; l2[k] = F.fl[2 * (i + 8 + k) + 1]; }
    if (FAC == 2) { l1[k] = __ldg(F.g + i + 8 + k); l2[k] = __ldg(F.g + F.L + i + 8 + k); }
  }
  if (ST == 1) s.template st<8>(i, a);
#pragma unroll
  for (int k = 0; k < NW; ++k) w[k] = win[8 + k];
}
// V 0: the reference's order; 1: the products in the order of the shorter
// dependent chain (the units that contract multiply-adds)
template <int V, class RS>
__device__ __forceinline__ RS back_row(RS p, RS u2, RS u3, RS cp1, RS cp2) {
  return V == 0 ? (p - u2 * cp1) - u3 * cp2 : (p - u3 * cp2) - u2 * cp1;
}
// Back substitution of rows i, i-1, ..., i-B+1 from p = u1 * (forward result).
// ADD: each row is stored as original + increment, the originals in o.
template <int B, int ST, int V, int ADD, class TT, class RS>
__device__ __forceinline__ void chain_bwd(const LineTile<ST, TT>& s, int i, const RS (&u2)[B], const RS (&u3)[B],
                                          const RS (&p)[B], const TT (&o)[B], RS& cp1, RS& cp2) {
  TT out[B];
#pragma unroll
  for (int k = 0; k < B; ++k) {
    const RS c = back_row<V, RS>(p[k], u2[k], u3[k], cp1, cp2);
    out[B - 1 - k] = ADD ? o[k] + TT(c) : TT(c);
    cp2 = cp1;
    cp1 = c;
  }
  s.template st<B>(i - B + 1, out);
}
// The same for eight rows with the next eight rows' products u1 * (forward
// result), factors (FAC as in fwd_pipe) and originals formed in between.
template <int FAC, int ST, int V, int ADD, class TT, class RS, class Org>
__device__ __forceinline__ void bwd_pipe(const LineTile<ST, TT>& s, int i, const LineFac<RS>& F, RS (&u2)[8],
                                         RS (&u3)[8], RS (&p)[8], TT (&o)[8], RS& cp1, RS& cp2, Org&& org) {
  TT v[8], out[8];
  s.template ld<8>(i - 15, v);
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int r = i - 8 - k;
    const RS c = back_row<V, RS>(p[k], u2[k], u3[k], cp1, cp2);
    out[7 - k] = ADD ? o[k] + TT(c) : TT(c);
    cp2 = cp1;
    cp1 = c;
    if (ST != 1) s(i - k) = out[7 - k];
    const RS u1 = FAC == 0 ? F.cu1 : FAC == 1 ? F.bu[4 * r] : __ldg(F.g + 2 * F.L + r);
    p[k] = u1 * RS(v[7 - k]);
    if (FAC == 1) { u2[k] = F.bu[4 * r + 1]; u3[k] = F.bu[4 * r + 2]; }
    if (FAC == 2) { u2[k] = __ldg(F.g + 3 * F.L + r); u3[k] = __ldg(F.g + 4 * F.L + r); }
    if (ADD) o[k] = org(r);
  }
  if (ST == 1) s.template st<8>(i - 7, out);
}

// One line in shared memory (element stride ST): the compact derivative
// (OP 0, src/mo_numerics.f90:742-792) or the compact filter (OP 1,
// src/mo_numerics.f90:922-977). On return the line holds the derivative or
// the filtered values; done(ch) is called as chunks become final. The filter
// solves for the increment and adds it to the original, org(row) (ADD 1), or
// leaves it in the tile (ADD 0), or solves for the filtered values themselves
// (DIRECT). q0, q1: interface sums received by the two ends.
// tl: the factors of the last three rows. Returns false if a bounded wait gave
// up.
template <int OP, int ST, class TT, class RS, int V, int ADD, bool DIRECT, class Done, class Org>
__device__ __forceinline__ bool sweep_line(const LineTile<ST, TT>& s, const LineFac<RS>& F, const RS* tl, int ndf0, int ndf1,
                                           const DevScheme* __restrict__ sc, const TT (&q0)[3], const TT (&q1)[3],
                                           ChunkIn& CI, int* err, Done&& done, Org&& org) {
#define S(i) s(i)
  constexpr int NE = OP == 0 ? 2 : 3;  // closure rows at each end
  constexpr int CY = ST != 1 ? 0 : OP == 1 ? 1 : (sizeof(TT) == 8 ? 0 : 2);
  constexpr int LO = WinSize<OP, CY>::LO, NW = WinSize<OP, CY>::N, LA = LO + CY;
  constexpr int START = (ST == 1 && (OP == 1 || sizeof(TT) == 4)) ? 4 : NE;  // first row of the aligned blocks
  constexpr int AL = ST == 1 ? 16 / (int)sizeof(TT) : 1;
  const int N = F.L - 1;
  Stencil<OP, TT> c{};
  if (OP == 1) {
    c.fa = TT(sc->fa); c.fb = TT(sc->fb); c.fc = TT(sc->fc);
    if (DIRECT) { c.al = TT(sc->alphf); c.be = TT(sc->betf); }
  }
  auto fbc = [&](int r, int k) { return TT(sc->fbc[r][k]); };
  // closure right-hand sides of the rows at both ends: b[side][0] the end row
  TT b[2][3];
#pragma unroll
  for (int sd = 0; sd < 2; ++sd) {
    const int e0 = sd ? N : 0, de = sd ? -1 : 1;
    const int ndf = sd ? ndf1 : ndf0;
    const TT(&q)[3] = sd ? q1 : q0;
    auto E = [&](int k) { return S(e0 + de * k); };
    b[sd][2] = 0;
    if (OP == 0) {
      if (ndf == 0) {
        const TT v0 = E(0), v1 = E(1), v2 = E(2), v3 = E(3), v4 = E(4);
        // the differences of the far end keep the reference's sign order
        if (sd == 0) {
          b[0][0] = ((TT(CA_A01) * (v1 - v0) + TT(CA_A02) * (v2 - v0)) + TT(CA_A03) * (v3 - v0)) + TT(CA_A04) * (v4 - v0);
          b[0][1] = ((TT(CA_A10) * (v0 - v1) + TT(CA_A12) * (v2 - v1)) + TT(CA_A13) * (v3 - v1)) + TT(CA_A14) * (v4 - v1);
        } else {
          b[1][0] = ((TT(CA_A01) * (v0 - v1) + TT(CA_A02) * (v0 - v2)) + TT(CA_A03) * (v0 - v3)) + TT(CA_A04) * (v0 - v4);
          b[1][1] = ((TT(CA_A10) * (v1 - v0) + TT(CA_A12) * (v1 - v2)) + TT(CA_A13) * (v1 - v3)) + TT(CA_A14) * (v1 - v4);
        }
      } else {
        TT t0 = 0, t1 = 0;
#pragma unroll
        for (int i = 0; i < 12; ++i) {
          const TT v = E(i);
          t0 = t0 + TT(sc->pbci[0][0][i]) * v;
          t1 = t1 + TT(sc->pbci[0][1][i]) * v;
        }
        b[sd][0] = sd ? -t0 - q[0] : t0 + q[0];
        b[sd][1] = sd ? -t1 - q[1] : t1 + q[1];
      }
    } else {
      const TT v0 = E(0), v1 = E(1), v2 = E(2), v3 = E(3), v4 = E(4), v5 = E(5);
      if (ndf == 0) {
        b[sd][0] = (((fbc(0, 0) * (v1 - v0) + fbc(0, 1) * (v2 - v0)) + fbc(0, 2) * (v3 - v0)) + fbc(0, 3) * (v4 - v0)) +
                   fbc(0, 4) * (v5 - v0);
        b[sd][1] = (((fbc(1, 0) * (v0 - v1) + fbc(1, 1) * (v2 - v1)) + fbc(1, 2) * (v3 - v1)) + fbc(1, 3) * (v4 - v1)) +
                   fbc(1, 4) * (v5 - v1);
        b[sd][2] = (((fbc(2, 0) * (v0 - v2) + fbc(2, 1) * (v1 - v2)) + fbc(2, 2) * (v3 - v2)) + fbc(2, 3) * (v4 - v2)) +
                   fbc(2, 4) * (v5 - v2);
      } else {
        TT t0 = 0, t1 = 0;
#pragma unroll
        for (int i = 0; i < 12; ++i) {
          const TT v = E(i);
          t0 = t0 + TT(sc->pbci[1][0][i]) * v;
          t1 = t1 + TT(sc->pbci[1][1][i]) * v;
        }
        const TT ra2 = v2 + v2;
        b[sd][0] = t0 + q[0];
        b[sd][1] = t1 + q[1];
        // the neighbour's value stands outside its end; the sums of pairs keep
        // the reference's order (they commute, so both ends read alike)
        b[sd][2] = (c.fa * ((v1 + v3) - ra2) + c.fb * ((v0 + v4) - ra2)) + c.fc * ((q[2] + v5) - ra2);
      }
      if (DIRECT) {  // (A x) of the three closure rows
        const double* a = &sc->albef[ndf][0][0];
        b[sd][0] = b[sd][0] + ((v0 + TT(a[3]) * v1) + TT(a[4]) * v2);
        b[sd][1] = b[sd][1] + (((TT(a[6]) * v0 + v1) + TT(a[8]) * v2) + TT(a[9]) * v3);
        b[sd][2] = b[sd][2] + ((((TT(a[10]) * v0 + TT(a[11]) * v1) + v2) + TT(a[13]) * v3) + TT(a[14]) * v4);
      }
    }
  }
  // ---- forward elimination, in place; the originals that later rows need are in w
  TT w[NW];
#pragma unroll
  for (int k = 0; k < NW; ++k) w[k] = S(NE - LO + k);
  RS am2 = RS(b[0][0]), am1, l1, l2;
  F.row_l(1, l1, l2);
  am1 = RS(b[0][1]) - l2 * am2;
  S(0) = TT(am2);
  S(1) = TT(am1);
  if (OP == 1) {
    F.row_l(2, l1, l2);
    const RS a2 = (RS(b[0][2]) - l1 * am2) - l2 * am1;
    S(2) = TT(a2);
    am2 = am1;
    am1 = a2;
  }
  int i = NE;
  auto step = [&](RS f1, RS f2) {
    TT x[2 * LO + 1];
    const TT nx = S(i + LA);  // inside the allocation for every i <= N - 2
#pragma unroll
    for (int k = 0; k <= 2 * LO; ++k) x[k] = k < NW ? w[k < NW ? k : 0] : nx;
    const RS a = (RS(rhs_row<OP, DIRECT, TT>(x, c)) - f1 * am2) - f2 * am1;
    S(i) = TT(a);
#pragma unroll
    for (int k = 0; k + 1 < NW; ++k) w[k] = w[k + 1];
    w[NW - 1] = nx;
    am2 = am1;
    am1 = a;
    ++i;
  };
  while (i < START && i <= N - 3) {
    F.row_l(i, l1, l2);
    step(l1, l2);
  }
  if (((N - 2 - i) & 4) && i + 3 <= N - 3) {
    if (!CI.need(min(N, i + 3 + LA), err)) return false;
    TT r[4];
    RS f1[4], f2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) F.row_l(i + k, f1[k], f2[k]);
    rhs_rows<4, OP, ST, CY, DIRECT, TT>(s, i, c, w, r);
    chain_fwd<4, ST, TT, RS>(s, i, f1, f2, r, am2, am1);
    i += 4;
  }
  {
    const int nb = max(0, (N - 2 - i) >> 3);                        // blocks of rows up to N - 3
    const int tb = min(nb, max(0, (F.c0 - i + 7) >> 3));            // the first tb have rows below c0
    TT rr[8];
    RS f1[8], f2[8];
    if (nb > 0) {
      if (!CI.need(min(N, i + 7 + LA), err)) return false;
      rhs_rows<8, OP, ST, CY, DIRECT, TT>(s, i, c, w, rr);
      if (tb > 0) F.template rows_l<8>(i, f1, f2);
      for (int k = 1; k < tb; ++k) {
        if (!CI.need(min(N, i + 15 + LA), err)) return false;
        if (i + 16 <= F.T) fwd_pipe<1, OP, ST, CY, DIRECT, TT, RS>(s, i, F, c, w, f1, f2, rr, am2, am1);
        else fwd_pipe<2, OP, ST, CY, DIRECT, TT, RS>(s, i, F, c, w, f1, f2, rr, am2, am1);
        i += 8;
      }
      if (tb > 0 && tb < nb) {
        if (!CI.need(min(N, i + 15 + LA), err)) return false;
        fwd_pipe<0, OP, ST, CY, DIRECT, TT, RS>(s, i, F, c, w, f1, f2, rr, am2, am1);
        i += 8;
      }
      if (tb < nb) {
#pragma unroll
        for (int j = 0; j < 8; ++j) { f1[j] = F.cl1; f2[j] = F.cl2; }
        for (int k = tb + 1; k < nb; ++k) {
          if (!CI.need(min(N, i + 15 + LA), err)) return false;
          fwd_pipe<0, OP, ST, CY, DIRECT, TT, RS>(s, i, F, c, w, f1, f2, rr, am2, am1);
          i += 8;
        }
      }
      chain_fwd<8, ST, TT, RS>(s, i, f1, f2, rr, am2, am1);
      i += 8;
    }
  }
  if (!CI.need(N, err)) return false;
  while (i <= N - 3) {
    F.row_l(i, l1, l2);
    step(l1, l2);
  }
  if (OP == 0) {
    step(tl[0], tl[1]);  // row N - 2
  } else {
    const RS a = (RS(b[1][2]) - tl[0] * am2) - tl[1] * am1;
    S(N - 2) = TT(a);
    am2 = am1;
    am1 = a;
  }
  const RS a1 = (RS(b[1][1]) - tl[2] * am2) - tl[3] * am1;
  const RS a0 = (RS(b[1][0]) - tl[4] * am1) - tl[5] * a1;
  TRACE(3)
  // ---- back substitution: the last three rows, then blocks down to row 0
  auto put = [&](int r, RS v) { S(r) = ADD ? org(r) + TT(v) : TT(v); };
  RS cp2 = tl[6] * RS(TT(a0));
  RS cp1 = tl[7] * RS(TT(a1)) - tl[8] * cp2;
  {
    const RS x = back_row<0, RS>(tl[9] * RS(S(N - 2)), tl[10], tl[11], cp1, cp2);
    put(N, cp2);
    put(N - 1, cp1);
    put(N - 2, x);
    cp2 = cp1;
    cp1 = x;
  }
  i = N - 3;
  int ch = CI.NC - 1, lo = ch * CI.CR;
  auto passed = [&]() {  // rows above i are final
    while (i < lo) {
      done(ch);
      --ch;
      lo = ch >= 0 ? ch * CI.CR : -1000;
    }
  };
  auto back = [&]() {
    RS u1, u2, u3;
    F.row_u(i, u1, u2, u3);
    const RS x = back_row<V, RS>(u1 * RS(S(i)), u2, u3, cp1, cp2);
    put(i, x);
    cp2 = cp1;
    cp1 = x;
    --i;
  };
  while (((i + 1) & (AL - 1)) != 0 && i >= 0) back();
  passed();
  {
    RS p[8], u1[8], u2[8], u3[8];
    TT o[8] = {};
    auto first = [&]() {  // products and originals of rows i..i-7
      TT v[8];
      s.template ld<8>(i - 7, v);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        p[k] = u1[k] * RS(v[7 - k]);
        if (ADD) o[k] = org(i - k);
      }
    };
    auto finish = [&]() {
      chain_bwd<8, ST, V, ADD, TT, RS>(s, i, u2, u3, p, o, cp1, cp2);
      i -= 8;
      passed();
    };
    const int nc = max(0, (i - F.c0 + 1) >> 3);
    if (nc > 0) {
#pragma unroll
      for (int k = 0; k < 8; ++k) { u1[k] = F.cu1; u2[k] = F.cu2; u3[k] = F.cu3; }
      first();
      for (int k = 1; k < nc; ++k) {
        bwd_pipe<0, ST, V, ADD, TT, RS>(s, i, F, u2, u3, p, o, cp1, cp2, org);
        i -= 8;
        passed();
      }
      finish();
    }
    const int tb = (i + 1) >> 3;
    if (tb > 0) {
      F.template rows_u<8>(i, u1, u2, u3);
      first();
      for (int k = 1; k < tb; ++k) {
        if (i - 8 < F.T) bwd_pipe<1, ST, V, ADD, TT, RS>(s, i, F, u2, u3, p, o, cp1, cp2, org);
        else bwd_pipe<2, ST, V, ADD, TT, RS>(s, i, F, u2, u3, p, o, cp1, cp2, org);
        i -= 8;
        passed();
      }
      finish();
    }
    if ((i + 1) & 4) {
      RS u1[4], u2[4], u3[4], p4[4];
      TT v[4], o4[4] = {};
#pragma unroll
      for (int k = 0; k < 4; ++k) F.row_u(i - k, u1[k], u2[k], u3[k]);
      s.template ld<4>(i - 3, v);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        p4[k] = u1[k] * RS(v[3 - k]);
        if (ADD) o4[k] = org(i - k);
      }
      chain_bwd<4, ST, V, ADD, TT, RS>(s, i, u2, u3, p4, o4, cp1, cp2);
      i -= 4;
      passed();
    }
    while (i >= 0) back();
    passed();
  }
#undef S
  return true;
}

// shared memory ahead of the tile: the chunks' barriers (64 bytes), then the
// twelve factors of the last three rows
constexpr int kLineHead = 256;
// bytes of `rows` staged rows of factors
template <class RS>
__host__ __device__ constexpr size_t line_tab_bytes(int rows) {
  return (size_t)rows * 6 * sizeof(RS);
}
constexpr int kLineStage = 96;  // factor rows staged at most
constexpr int kLineSlack = 32;  // a row-major tile's reads may touch one row past its last line

// One CTA = one warp = 32 lines. DIR: 1 xi, 2 eta, 3 zeta. OP: 0 derivative,
// 1 filter (in place). TT: field and tile type, RS: type of the elimination.
// V: 0 the reference's order (FP64 without contraction: bit-exact), 1 the
// units with contraction; the FP64 filter then solves for the filtered values.
// Eta/zeta tiles are [row][32 lines] and move in chunks (loads overlap the
// forward sweep, stores the back substitution); xi tiles are one or two
// [line][pitch] boxes (T.xt, lines of up to 508 FP64 or 504 FP32 points; one box,
// up to 254 points, for a filter that solves for the increment, whose store is
// one add per line) or, for longer lines, one bulk copy per line: 32 bulk copies
// cost a CTA 3.0 thousand cycles to issue and 32 bulk stores 5.6 thousand, a box
// 1.4 thousand with its task's start-up.
//
// A filter that solves for the increment adds the originals row by row along
// eta and zeta; along xi the tile keeps the increment and one bulk FP64
// reduce-add per line adds it to the field (the same single rounding). FP64
// reductions straight from the registers, without the originals' loads, ran at
// 0.73 / 0.56 ms along eta / zeta against 0.63 / 0.59 (five fields, 257 points),
// and at 0.65 against 0.51 along xi.
template <int DIR, int OP, class TT, class RS, int V>
__global__ void __maxnreg__(168) k_line(const LineTask* __restrict__ tasks, const int* __restrict__ tile_task,
                                        int tdiv, const CUtensorMap* __restrict__ maps, int* __restrict__ err) {
  constexpr int kVec = 16 / (int)sizeof(TT);  // elements per 16 bytes
  constexpr bool DIRECT = OP == 1 && V == 1 && sizeof(RS) == 8;
  constexpr bool kInc = OP == 1 && !DIRECT;  // the sweep solves for the increment
  constexpr bool kRedAdd = kInc && DIR == 1;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem_raw);
  RS* tl = reinterpret_cast<RS*>(smem_raw + 64);
  TT* s = reinterpret_cast<TT*>(smem_raw + kLineHead);
  const int lane = threadIdx.x;
  TRACE(0)
  // the tile's task and the error flag load together (independent)
  const int ti = tile_of(tile_task, tdiv);
  const int eflag = error_flag_early(err);
  const LineTask& T = tasks[ti];
  const TT* in = static_cast<const TT*>(T.in);
  TT* out = static_cast<TT*>(T.out);
  const int lt = blockIdx.x - T.tile0;
  const int L = T.L;
  const int X = T.X, Y = T.Y, Z = T.Z, Xp = T.Xp;
  const int NC = T.nbox, CR = T.by;
  const int P = T.pitch;
  const bool box = DIR != 1 || T.xt != 0;
  int nval, x0 = 0, r0 = 0, fix = 0;  // fix: z for dir 2, y for dir 3
  if (DIR == 1) {
    r0 = lt * kLanes;
    nval = min(kLanes, Y * Z - r0);
  } else {
    fix = lt / T.ntx;
    x0 = (lt % T.ntx) * kLanes;
    nval = min(kLanes, X - x0);
  }
  const long long pstride = (DIR == 2) ? (long long)Xp : (long long)Xp * Y;  // dir 2/3 position stride
  const long long base = (DIR == 1) ? (long long)r0 * Xp
                                    : ((DIR == 2) ? (long long)fix * Y * Xp + x0 : (long long)fix * Xp + x0);
  const CUtensorMap* map_in = maps + 2 * ti;
  const CUtensorMap* map_out = maps + 2 * ti + 1;
  if (lane == 0) {
    for (int c = 0; c < NC; ++c) mbar_init(bars + c, 1);
    mbar_init_done();
  }
  // a kernel launched after a bounded wait gave up does no work
  if (__shfl_sync(0xffffffffu, eflag, 0) != 0) return;
  __syncwarp();
  // issue the loads: chunk 0, the last chunk, then the middle ones
  const uint32_t lbytes = (uint32_t)((L + kVec - 1) / kVec * kVec * sizeof(TT));  // one xi line
  if (DIR == 1 && !box) {
    if (lane == 0) mbar_expect_tx(bars, lbytes * nval);
    __syncwarp();
    if (lane < nval) bulk_g2s(s + lane * P, in + base + (long long)lane * Xp, lbytes, bars);
  } else if (lane == 0) {
    for (int k = 0; k < NC; ++k) {
      const int c = (k == 0) ? 0 : (k == 1 ? NC - 1 : k - 1);
      mbar_expect_tx(bars + c, (uint32_t)(CR * kLanes * sizeof(TT)));
      if (DIR == 1) tma_load_3d(s + c * CR * kLanes, map_in, c * CR, r0, 0, bars + c);
      else if (DIR == 2) tma_load_3d(s + c * CR * kLanes, map_in, x0, c * CR, fix, bars + c);
      else tma_load_3d(s + c * CR * kLanes, map_in, x0, fix, c * CR, bars + c);
    }
  }
  TRACE(1)
  // while the copies are in flight: the received interface sums (the periodic
  // contraction below reads the tile instead) and the staged factors
  const bool has = lane < nval;
  int jk = 0;
  if (DIR == 1) jk = r0 + lane;
  else if (DIR == 2) jk = (x0 + lane) * Z + fix;
  else jk = fix * X + x0 + lane;
  const int nbs = T.nbs;
  const TT* recv = static_cast<const TT*>(T.recv);
  constexpr int NQ = OP == 0 ? 2 : 3;
  TT q0[3] = {}, q1[3] = {};
  if (OP == 1 || !T.selfp) {
#pragma unroll
    for (int k = 0; k < NQ; ++k) {
      if (has && T.ndf0) q0[k] = recv[k * nbs + jk];
      if (has && T.ndf1) q1[k] = recv[(NQ + k) * nbs + jk];
    }
  }
  const int TR = T.ts;
  RS* fl = reinterpret_cast<RS*>(s + (DIR == 1 && !box ? P : NC * CR) * kLanes);
  RS* bu = fl + 2 * TR;
  const RS* lu = static_cast<const RS*>(T.lu);
  {
    // lanes 0..11: l1, l2 of rows N-2, N-1, N, then u1(N), u1(N-1), u2(N-1), u1..u3(N-2)
    const int k = lane, N = L - 1;
    if (k < 12) {
      const int row = k < 6 ? N - 2 + k / 2 : k == 6 ? N : k < 9 ? N - 1 : N - 2;
      const int tab = k < 6 ? k % 2 : k < 8 ? 2 : k == 8 ? 3 : k - 7;
      tl[k] = __ldg(lu + tab * L + row);
    }
    static_assert(kLineStage <= 3 * kLanes, "rows staged per lane");
    RS v[3][5];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int r = lane + j * kLanes;
#pragma unroll
      for (int q = 0; q < 5; ++q) v[j][q] = r < TR ? __ldg(lu + q * L + r) : RS(0);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int r = lane + j * kLanes;
      if (r < TR) {
        fl[2 * r] = v[j][0]; fl[2 * r + 1] = v[j][1];
        bu[4 * r] = v[j][2]; bu[4 * r + 1] = v[j][3]; bu[4 * r + 2] = v[j][4];
      }
    }
    // the scheme's coefficients (1.2 KB), read by the closures
    if (lane >= 16 && lane < 26) prefetch_l1(reinterpret_cast<const char*>(T.sc) + 128 * (lane - 16));
  }
  const LineFac<RS> F{fl, bu, lu, RS(T.cl1), RS(T.cl2), RS(T.cu1), RS(T.cu2), RS(T.cu3), TR, T.c0, L - 4, L};
  if (!mbar_wait(bars, 0) || !mbar_wait(bars + NC - 1, 0)) {
    if (lane == 0) atomicExch(err, kErrTimeout);
    // copies may still be landing: wait for the other chunks, the last among
    // them where the first gave up (bounded), before exit
    for (int c = 1; c < NC; ++c) mbar_wait(bars + c, 0);
    return;
  }
  __syncwarp();
  TRACE(2)
  ChunkIn CI{bars, CR, NC, L, 1, (NC > 1 ? CR : L)};
  if (NC <= 2) CI.ready = L;
  if (kRedAdd && (L & 1)) s[lane * P + L] = TT(0);  // the 16-byte tail's pad element adds 0
  // chunk c is final: store it
  auto done = [&](int c) {
    fence_proxy_async();
    __syncwarp();
    if (DIR == 1 && (kRedAdd || !box)) {  // kRedAdd: one box at most
      if (lane < nval) {
        TT* d = out + base + (long long)lane * Xp;
        if (kRedAdd) bulk_s2g_add_f64(d, s + lane * P, lbytes);
        else bulk_s2g(d, s + lane * P, lbytes);
        bulk_commit();
      }
    } else if (lane == 0) {
      // positions past the block edge (and x past X) are not written
      if (DIR == 1) tma_store_3d(map_out, c * CR, r0, 0, s + c * CR * kLanes);
      else if (DIR == 2) tma_store_3d(map_out, x0, c * CR, fix, s + c * CR * kLanes);
      else tma_store_3d(map_out, x0, fix, c * CR, s + c * CR * kLanes);
      bulk_commit();
    }
  };
  bool ok = true;
  // every lane runs the sweep (lanes past the tile edge on zero-filled or
  // stale columns) so the chunk hand-offs stay warp-uniform; only lanes with a
  // line read the receive buffers or write drva
  constexpr int ST = (DIR == 1) ? 1 : kLanes;
  const LineTile<ST, TT> sl{(DIR == 1) ? s + lane * P : s + lane, box && NC > 1 ? CR : (1 << 30),
                            (kLanes - 1) * CR};
  if (OP == 0) {
    if (T.selfp) {
      // The line is periodic onto itself, so the interface contraction the
      // other end would send (src/mo_numerics.f90:503-518 with n45 = 0) is
      // formed here from the tile: side 0 receives the sums over positions
      // N-1..N-12, side 1 over positions 1..12, accumulated in the same order.
      const DevScheme* __restrict__ sc = T.sc;
      const int N = L - 1;
#pragma unroll
      for (int i = 0; i < 12; ++i) {
        const TT v = sl(N - 1 - i), w = sl(1 + i);
        q0[0] = q0[0] + TT(sc->pbco[0][0][i]) * v;
        q0[1] = q0[1] + TT(sc->pbco[0][1][i]) * v;
        q1[0] = q1[0] + TT(sc->pbco[0][0][i]) * w;
        q1[1] = q1[1] + TT(sc->pbco[0][1][i]) * w;
      }
    }
    ok = sweep_line<OP, ST, TT, RS, V, 0, false>(sl, F, tl, T.ndf0, T.ndf1, T.sc, q0, q1, CI, err, done,
                                                 [](int) { return TT(0); });
    if (ok && has && T.drva) {
      TT* drva = static_cast<TT*>(T.drva);
      drva[jk + (long long)nbs * (T.m - 1)] = sl(0);
      drva[jk + (long long)nbs * ((T.m - 1) + 5)] = sl(L - 1);
    }
  } else {
    // this lane's line of the unfiltered field (lanes without a line read
    // lane 0's, whose results are not stored)
    const TT* og = in + base + (has ? lane : 0);
    ok = sweep_line<OP, ST, TT, RS, V, kInc && DIR != 1 ? 1 : 0, DIRECT>(
        sl, F, tl, T.ndf0, T.ndf1, T.sc, q0, q1, CI, err, done, [&](int r) { return __ldg(og + r * pstride); });
  }
  // every issued bulk store has to finish reading shared memory before exit;
  // after a timeout, wait for the chunks still in flight (bounded) instead
  if (!ok) {
    for (int c = CI.next; c < NC - 1; ++c) mbar_wait(bars + c, 0);
    return;
  }
  TRACE(4)
  bulk_wait_read0();
  TRACE(5)
#ifdef CANARD_TRACE
  if (threadIdx.x == 0) {
    unsigned smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    g_trace[(long long)blockIdx.x * 8 + 6] = smid;
  }
#endif
}
