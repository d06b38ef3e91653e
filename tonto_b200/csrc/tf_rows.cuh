// tf_rows.cuh — lane-group quartets for the classes whose (e0|f0) block does not fit one
// thread: the ket pairs beyond the thread kernels of tf_thread.cuh (pp, dp, dd, and
// every class with an f shell except those whose ket block is small).
//
// A group of lanes computes one contracted quartet: NF <= 32 lanes (the ket's (f0|
// components), 32 / NF groups to a warp; for (fd| and (ff| kets, 46 and 74 components,
// a block of two or three warps.
//   * Per primitive quartet the group builds the 3 x NROOT 2D recurrence tables in shared
//     memory (make_esfs_XX, shell1quartet.foo:7418-7609) and lane f accumulates (e0|f0)
//     for all e in registers (form_esfs :7615-7649).
//   * Lane f holds a whole column, so the bra's horizontal transfer (transfer_ab
//     :8310-11134) stays in its registers; the column X(ab, f) is written to shared memory
//     once, with J~(f) = sum_ab X(ab, f) P(ab) summed on the way.
//   * Lane r then reads row ab = r of X, so the ket's transfer stays in registers too, and
//     digests the row as a thread kernel digests a quartet: J(ab) whole, the row's shares
//     of K(ac), K(ad), K(bc), K(bd) back into the row's place, summed over rows at the end.
// What bounds such kernels on this GPU is the shared-memory and L1 pipe, not FP64: the
// layout reads every integral from shared memory once (the row read), where transfers and
// digestion element by element in shared memory read each about ten times.  Measured,
// class-by-class builds, against that form of the kernels: (H2O)32 cc-pVDZ (dp|dp) 1.22 ->
// 0.72 ms, (dd|pp) 1.26 -> 0.56, (dd|dp) 1.01 -> 0.28, (dp|pp) 3.44 -> 2.77.  For the f classes,
// against one warp a quartet with run-time angular momenta in global scratch: (H2O)5 cc-pVTZ
// (fd|dp) 3.26 -> 0.14 ms, (ff|ff) 1.08 -> 0.02.  The classes of tf_jk_l*.cu come here with
// short lists only (dispatch_jk has both sides' times).
#pragma once
#include "tf_device.cuh"
#include "tf_host.h"

#include <algorithm>

namespace tf {

__host__ __device__ constexpr int cmax(int a, int b) { return a > b ? a : b; }

struct RowArgs {
  const int2* quartets;
  long long n;
  const PrimPair* prim_full;
  const PrimPair* prim_skip;
  const double* P;
  double* J;
  double* K;
  const MolInfo* mols;
  unsigned long long* prim_count;
  const long long* range;       // graph builds: see resolve_range
  long long base, cap;
  const int4* jkrec;            // packed pair records (load_pair_jk)
  const double4* xyz4;          // atom positions (load_pair_jk)
  const double* P2;             // unrestricted: beta density and its J, K (else null)
  double* J2;
  double* K2;
  int want;                     // bit 0 J, bit 1 K
  unsigned long long* qcount;   // quartets counted per class (the launch's FP64 or FP32 half)
  long long fx_lo;              // deterministic builds: offset of the lo words (fock_add), else 0
  long long groups;             // lane groups of the full grid (see k_jk_rows)
  long long expect;             // entries the launch will probably have (chooses the instantiation)
};

template <int LA, int LB, int LC, int LD>
struct RowCfg {
  using Q = Quartet<LA, LB, LC, LD>;
  static constexpr int NR = Q::NROOT, D1 = Q::LAB + 1, D2 = Q::LCD + 1;
  static constexpr int NAB = Q::NA * Q::NB, NCD = Q::NC * Q::ND, NY = Q::NC + Q::ND, NX = Q::NA + Q::NB;
  static constexpr int GW = (Q::NF + 31) / 32;           // warps per quartet
  static constexpr int G = GW == 1 ? Q::NF : 32 * GW;    // lanes per quartet
  static constexpr int QPW = GW == 1 ? 32 / G : 1;       // quartets per warp (GW > 1: per block)
  // a 2D table's column and the table itself, odd: lanes that read several columns or write
  // several tables hit different banks (as do a warp's groups, per_group)
  static constexpr int CS = D1 | 1, TS = (CS * D2) | 1;
  static constexpr int T2D = 3 * NR * TS;
  // row stride (odd: rows on different banks): the row, or in its place the row's K shares
  __host__ __device__ static constexpr int rs(int ns) { return cmax(Q::NF, 2 * NY * ns) | 1; }
  static constexpr int YS = NY | 1;
  __host__ __device__ static constexpr int area(int ns) { return cmax(T2D, NAB * rs(ns)); }
  // per density: P(a|b, c|d), P(ab), P(cd), J~
  static constexpr int STAGE = NX * YS + NAB + NCD + Q::NF;
  __host__ __device__ static constexpr int per_group(int ns) { return (area(ns) + ns * STAGE) | 1; }
};

struct CompBytes {
  unsigned char x[NCOMP_ALL], y[NCOMP_ALL], z[NCOMP_ALL];
};
__host__ __device__ constexpr CompBytes make_comp_bytes() {
  CompBytes b{};
  for (int i = 0; i < NCOMP_ALL; ++i) {
    b.x[i] = (unsigned char)CT.x[i];
    b.y[i] = (unsigned char)CT.y[i];
    b.z[i] = (unsigned char)CT.z[i];
  }
  return b;
}
static __device__ const CompBytes g_comp_bytes = make_comp_bytes();

// The ket transfer of one (c, d) as a sum over the 2^LD subsets t of d's unit steps:
// (c, d) = sum_t prod_{s not in t} R(dir_s) f[c + the steps in t].
template <int LC, int LD>
struct KetPlan {
  unsigned char f[ncart(LC) * ncart(LD)][1 << LD];
  unsigned char dir[ncart(LD)][LD > 0 ? LD : 1];
};
template <int LC, int LD>
constexpr KetPlan<LC, LD> make_ket_plan() {
  KetPlan<LC, LD> p{};
  for (int d = 0; d < ncart(LD); ++d) {
    int st[4] = {0, 0, 0, 0}, n = 0;
    for (int k = 0; k < cx(LD, d); ++k) st[n++] = 0;
    for (int k = 0; k < cy(LD, d); ++k) st[n++] = 1;
    for (int k = 0; k < cz(LD, d); ++k) st[n++] = 2;
    for (int s = 0; s < LD; ++s) p.dir[d][s] = (unsigned char)st[s];
    for (int c = 0; c < ncart(LC); ++c)
      for (int t = 0; t < (1 << LD); ++t) {
        int v[3] = {cx(LC, c), cy(LC, c), cz(LC, c)};
        for (int s = 0; s < LD; ++s)
          if (t >> s & 1) v[st[s]]++;
        p.f[c * ncart(LD) + d][t] = (unsigned char)(gidx(v[0], v[1], v[2]) - CT.first[LC]);
      }
  }
  return p;
}
template <int LC, int LD>
static __device__ const KetPlan<LC, LD> g_ket_plan = make_ket_plan<LC, LD>();

// One element of the bra transfer from the column es[e] in registers:
// (e, b + 1_i) = (e + 1_i, b) + R_i (e, b).
template <int EX, int EY, int EZ, int BX, int BY, int BZ, int FE, int NE>
__device__ __forceinline__ double bra_value(const double (&es)[NE], const double (&R)[3]) {
  if constexpr (BX > 0)
    return fma(R[0], bra_value<EX, EY, EZ, BX - 1, BY, BZ, FE>(es, R),
               bra_value<EX + 1, EY, EZ, BX - 1, BY, BZ, FE>(es, R));
  else if constexpr (BY > 0)
    return fma(R[1], bra_value<EX, EY, EZ, BX, BY - 1, BZ, FE>(es, R),
               bra_value<EX, EY + 1, EZ, BX, BY - 1, BZ, FE>(es, R));
  else if constexpr (BZ > 0)
    return fma(R[2], bra_value<EX, EY, EZ, BX, BY, BZ - 1, FE>(es, R),
               bra_value<EX, EY, EZ + 1, BX, BY, BZ - 1, FE>(es, R));
  else
    return es[gidx(EX, EY, EZ) - FE];
}

// Rys nodes and weights of a lane group's primitive quartet: the 2 N polynomial
// pieces (u_1..u_N, w_1..w_N at the interval of x) are spread over the group's
// lanes (G of a warp), each evaluated once, then exchanged with shuffles.  x is
// uniform within a group; every lane of the warp takes part.  gbase: the group's
// first lane.
template <int N, int G>
__device__ __forceinline__ void group_rys(double x, int gl, int gbase, double (&u)[N], double (&w)[N]) {
  static_assert(TF_RYS_NCOEF == 12 && rys_offset(N) % 4 == 0, "three 32-byte words a polynomial");
  constexpr int NF2 = 2 * N, PER = (NF2 + G - 1) / G;
  constexpr int XMAX = rys_xmax(N), OFF = rys_offset(N), HOFF = rys_hoffset(N);
  const bool tab = x < (double)XMAX;
  const int j = tab ? (int)x : 0;
  const double s = x - (double)j;
  double val[PER];
#pragma unroll
  for (int q = 0; q < PER; ++q) {
    const int f = gl + q * G;
    double v = 0.0;
    if (tab && f < NF2) {
      const double* cf = tf_rys_coef + OFF + j * (NF2 * TF_RYS_NCOEF) + f * TF_RYS_NCOEF;
      const double4 c2 = ldg256(cf + 8), c1 = ldg256(cf + 4), c0 = ldg256(cf);
      v = fma(fma(fma(c2.w, s, c2.z), s, c2.y), s, c2.x);
      v = fma(fma(fma(fma(v, s, c1.w), s, c1.z), s, c1.y), s, c1.x);
      v = fma(fma(fma(fma(v, s, c0.w), s, c0.z), s, c0.y), s, c0.x);
    }
    val[q] = v;
  }
#pragma unroll
  for (int f = 0; f < NF2; ++f) {
    const double v = __shfl_sync(0xffffffffu, val[f / G], gbase + f % G);
    if (f < N) u[f] = v;
    else w[f - N] = v;
  }
  if (!tab) {
    const double ix = rcp_nr(x), isx = rsqrt_nr(x);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      u[i] = tf_rys_hroot2[HOFF + i] * ix;
      w[i] = tf_rys_hweight[HOFF + i] * isx;
    }
  }
}

__device__ __forceinline__ void fock_add_rt(double* addr, double v, long long fx_lo) {
  if (fx_lo) fock_add<true>(addr, v, fx_lo);
  else fock_add<false>(addr, v, 0);
}

// SHARED: a list with fewer quartets than the GPU has lane groups; several groups of a warp
// share a quartet.  Each takes every share-th primitive quartet, their (e0|f0) columns are
// summed by shuffles, the first group transfers them and all lanes take rows: (H2O)2 STO-3G's
// 81-primitive (pp|pp) quartets 66 -> 28 us, (H2O)2 cc-pVTZ (ff|ps) 93 -> 44.  An instantiation of
// its own: with run-time lane counts (H2O)32's (pp|pp) took 2.97 instead of 2.55 ms.
template <int LA, int LB, int LC, int LD, int WPB, bool SHARED>
__global__ void __launch_bounds__(32 * WPB) k_jk_rows(RowArgs a) {
  using C = RowCfg<LA, LB, LC, LD>;
  using Q = typename C::Q;
  constexpr int G = C::G, GW = C::GW, QPW = C::QPW, NR = C::NR, D1 = C::D1, D2 = C::D2;
  constexpr int NE = Q::NE, NF = Q::NF, NA = Q::NA, NB = Q::NB, NC = Q::NC, ND = Q::ND;
  constexpr int NAB = C::NAB, NCD = C::NCD, NY = C::NY, NX = C::NX, YS = C::YS;
  static_assert(GW == 1 || GW == WPB, "a quartet wider than a warp takes a block");
  extern __shared__ double smem[];
  const int ns = a.P2 ? 2 : 1;
  const int rs = C::rs(ns);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto group_sync = [] {
    if constexpr (GW == 1) __syncwarp();
    else __syncthreads();
  };
  // gl: lane within the group; lanes outside every group keep the warp in step
  const int gq = GW == 1 ? lane / G : 0;
  const bool in_group = GW > 1 || gq < QPW;
  const int gl = GW > 1 ? (int)threadIdx.x : (in_group ? lane - gq * G : 0x40000000);
  const int slot = GW > 1 ? 0 : warp * QPW + (in_group ? gq : 0);
  double* const T2 = smem + (size_t)slot * C::per_group(ns);      // the group's 2D tables
  const bool has_f = in_group && gl < NF;
  const int2* quartets = a.quartets;
  long long nq = a.n;
  resolve_range(a.range, a.base, a.cap, quartets, nq);
  if (nq <= 0) return;
  // (from the list length and the full grid alone, so that a deterministic build does not
  // depend on the launch)
  const int share = SHARED ? (int)max(1LL, min((long long)QPW, a.groups / nq)) : 1;
  const int per_warp = QPW / share;                    // quartets of a warp at a time
  const int qs = in_group ? gq / share : 0, member = in_group ? gq - qs * share : 0;
  const bool used = in_group && qs < per_warp;
  const int ql = used ? member * G + gl : 0x40000000;  // lane within the quartet, and its lanes
  const int QL = share * G;
  const int gf = Q::FF + (has_f ? gl : 0);
  const int fx = g_comp_bytes.x[gf], fy = g_comp_bytes.y[gf], fz = g_comp_bytes.z[gf];
  const long long nslots = GW > 1 ? gridDim.x : (long long)gridDim.x * WPB;   // warps or blocks at work
  // the quartet's rows and density blocks, in its first group's area
  double* const X = smem + (size_t)(slot - member) * C::per_group(ns);
  double* const stage = X + C::area(ns);
  unsigned long long nprim = 0, nquart = 0;
  for (long long base = (GW > 1 ? (long long)blockIdx.x : (long long)blockIdx.x * WPB + warp) * per_warp; base < nq;
       base += nslots * per_warp) {
    const long long t = base + qs;
    const bool act = used && t < nq;
    const int2 qd = act ? quartets[t] : make_int2(0, 0);
    const PairJK b = load_pair_jk(a.jkrec, a.xyz4, qd.x);
    const PairJK k = load_pair_jk(a.jkrec, a.xyz4, qd.y);
    const bool any_same = b.atom_hi == b.atom_lo || k.atom_hi == k.atom_lo || b.atom_hi == k.atom_hi ||
                          b.atom_hi == k.atom_lo || b.atom_lo == k.atom_hi || b.atom_lo == k.atom_lo;
    const PrimPair* bp = any_same ? a.prim_full + b.full_off : a.prim_skip + b.skip_off;
    const PrimPair* kp = any_same ? a.prim_full + k.full_off : a.prim_skip + k.skip_off;
    const int nbp = any_same ? b.n_full : b.n_skip;
    const int nkp = any_same ? k.n_full : k.n_skip;
    const int npq = act ? nbp * nkp : 0;
    if (act && ql == 0) { nprim += (unsigned long long)npq; nquart += 1; }
    const MolInfo mi = a.mols[act ? b.mol : 0];
    const int n = mi.n_cart;
    const int oa = b.cart_hi, ob = b.cart_lo, oc = k.cart_hi, od = k.cart_lo;
    // density blocks of the quartet, read while the primitive loop runs
    if (act) {
      for (int s = 0; s < ns; ++s) {
        const double* __restrict__ P = (s ? a.P2 : a.P) + mi.cmat;
        double* st = stage + s * C::STAGE;
        for (int e = ql; e < NX * NY; e += QL) {
          const int x = e / NY, y = e - x * NY;
          const int row = x < NA ? oa + x : ob + x - NA, col = y < NC ? oc + y : od + y - NC;
          st[x * YS + y] = __ldg(P + (size_t)row * n + col);
        }
        for (int e = ql; e < NAB; e += QL) st[NX * YS + e] = __ldg(P + (size_t)(oa + e / NB) * n + ob + e % NB);
        for (int e = ql; e < NCD; e += QL)
          st[NX * YS + NAB + e] = __ldg(P + (size_t)(oc + e / ND) * n + od + e % ND);
      }
    }
    const int mine = npq > member ? (npq - member + share - 1) / share : 0;   // this group's primitive quartets
    const int maxnpq = GW > 1 ? npq : (int)__reduce_max_sync(0xffffffffu, mine);
    const QuartetGeom geom = quartet_geom(b, k);
    double es[NE];
#pragma unroll
    for (int e = 0; e < NE; ++e) es[e] = 0.0;
    int ib = 0, ik = member;
    for (int p = 0; p < maxnpq; ++p) {
      const bool v = p < mine;
      if constexpr (SHARED)
        while (v && ik >= nkp) { ik -= nkp; ++ib; }
      double u[NR], w[NR];
      double4 b0 = make_double4(1, 0, 0, 0), k0 = make_double4(1, 0, 0, 0);
      double inv = 0.0, r_z = 0.0, r_e = 0.0, scale = 0.0, xx = 0.0;
      if (v) {
        b0 = load_prim(bp, ib);
        k0 = load_prim(kp, ik);
        const double bcc = b0.y * TWOPI5ON2, kcc = k0.y;
        const double sq = rsqrt_nr(b0.x + k0.x);
        inv = sq * sq;
        const double rho = b0.x * k0.x * inv;
        const PrimGeom pg = prim_geom(b0, k0, geom);
        xx = rho * (pg.QP[0] * pg.QP[0] + pg.QP[1] * pg.QP[1] + pg.QP[2] * pg.QP[2]);
        scale = bcc * kcc * sq;                  // (cc holds the pair's sqrt(zeta))
        r_z = k0.x * inv;
        r_e = b0.x * inv;
      }
      if constexpr (GW > 1) group_rys<NR, 32>(xx, lane, 0, u, w);
      else group_rys<NR, G>(xx, in_group ? gl : G, lane - (in_group ? gl : 0), u, w);
      group_sync();                              // the tables of the previous primitive quartet have been read
      if (v) {
        for (int task = gl; task < 3 * NR; task += G) {
          const int d = task / NR, r = task - d * NR;
          double t2 = 0.0, wr = 0.0;
#pragma unroll
          for (int i = 0; i < NR; ++i)
            if (i == r) { t2 = u[i]; wr = w[i]; }
          const double Rb = d == 0 ? geom.Rab[0] : (d == 1 ? geom.Rab[1] : geom.Rab[2]);
          const double Rk = d == 0 ? geom.Rcd[0] : (d == 1 ? geom.Rcd[1] : geom.Rcd[2]);
          const double PA = b0.z * Rb, QC = k0.z * Rk;
          const double QPd = fma(-b0.z, Rb, fma(k0.z, Rk, d == 0 ? geom.CA[0] : (d == 1 ? geom.CA[1] : geom.CA[2])));
          const double t2_rz = t2 * r_z, t2_re = t2 * r_e;
          const double B10 = (1.0 - t2_rz) * b0.w, B01 = (1.0 - t2_re) * k0.w, B00 = 0.5 * t2 * inv;
          const double c00 = PA + t2_rz * QPd, d00 = QC - t2_re * QPd;
          double* out = T2 + task * C::TS;
          // one ket column at a time: I[e][f + 1] from columns f and f - 1
          double I0[D1], I1[D1];
          I0[0] = d == 2 ? wr * scale : 1.0;
          if (D1 > 1) I0[1] = c00 * I0[0];
#pragma unroll
          for (int e = 1; e + 1 < D1; ++e) I0[e + 1] = c00 * I0[e] + e * B10 * I0[e - 1];
#pragma unroll
          for (int e = 0; e < D1; ++e) { out[e] = I0[e]; I1[e] = 0.0; }
#pragma unroll
          for (int f = 0; f + 1 < D2; ++f) {
            double nx[D1];
#pragma unroll
            for (int e = 0; e < D1; ++e) {
              double vv = d00 * I0[e];
              if (f > 0) vv += f * B01 * I1[e];
              if (e > 0) vv += e * B00 * I0[e - 1];
              nx[e] = vv;
            }
#pragma unroll
            for (int e = 0; e < D1; ++e) {
              I1[e] = I0[e];
              I0[e] = nx[e];
              out[(f + 1) * C::CS + e] = nx[e];
            }
          }
        }
      }
      group_sync();
      if (v && has_f) {
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          // (8-byte loads: lanes that share a word are served together, half a warp at a
          // time; 16-byte ones a quarter warp at a time, measured 2-4 cycles against 0.6-1.3)
          double cxv[D1], cyv[D1], czv[D1];
          const double* tx = T2 + (0 * NR + r) * C::TS + fx * C::CS;
          const double* ty = T2 + (1 * NR + r) * C::TS + fy * C::CS;
          const double* tz = T2 + (2 * NR + r) * C::TS + fz * C::CS;
#pragma unroll
          for (int e = 0; e < D1; ++e) {
            cxv[e] = tx[e];
            cyv[e] = ty[e];
            czv[e] = tz[e];
          }
          static_for<NE>([&](auto ee) {
            constexpr int e = decltype(ee)::value;
            constexpr int ge = Q::FE + e;
            es[e] += cxv[gx(ge)] * cyv[gy(ge)] * czv[gz(ge)];
          });
        }
      }
      if constexpr (SHARED) ik += share;
      else if (++ik == nkp) { ik = 0; ++ib; }
    }
    group_sync();                                // the tables have been read, the density blocks written
    if constexpr (SHARED) {                      // the sharing groups' sums, halving
      for (int o = share; o > 1; o = (o + 1) / 2) {
        const int h = (o + 1) / 2;
        const bool add = used && member + h < o;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
          const double x = __shfl_sync(0xffffffffu, es[e], (lane + h * G) & 31);
          if (add) es[e] += x;
        }
      }
    }
    const double (&Rab)[3] = geom.Rab;
    const double (&Rcd)[3] = geom.Rcd;
    if (act && has_f && member == 0) {           // column f: bra transfer, J~(f)
      double jt = 0.0, jt2 = 0.0;
      const double* pab = stage + NX * YS;
      static_for<NA>([&](auto aa) {
        static_for<NB>([&](auto bb) {
          constexpr int ia = decltype(aa)::value, ibb = decltype(bb)::value, ab = ia * NB + ibb;
          const double xv = bra_value<cx(LA, ia), cy(LA, ia), cz(LA, ia), cx(LB, ibb), cy(LB, ibb), cz(LB, ibb),
                                      Q::FE>(es, Rab);
          X[ab * rs + gl] = xv;
          jt = fma(xv, pab[ab], jt);
          if (ns > 1) jt2 = fma(xv, pab[C::STAGE + ab], jt2);
        });
      });
      stage[NX * YS + NAB + NCD + gl] = jt;
      if (ns > 1) stage[C::STAGE + NX * YS + NAB + NCD + gl] = jt2;
    }
    group_sync();
    double f = 1.0;
    if (b.same) f *= 0.5;
    if (k.same) f *= 0.5;
    if (qd.x == qd.y) f *= 0.5;
    if (act) {
      for (int r = ql; r < NAB; r += QL) {        // row ab: ket transfer, J(ab), the row's shares of K
        const int ia = r / NB, ibb = r - ia * NB;
        double* row = X + r * rs;
        double g[1][NF], I[1][NC][ND];
#pragma unroll
        for (int q = 0; q < NF; ++q) g[0][q] = row[q];
        hrr_ket<LC, LD, 1, double>(g, Rcd, I);
        for (int s = 0; s < ns; ++s) {
          const double* st = stage + s * C::STAGE;
          const double* pa = st + ia * YS;
          const double* pb = st + (NA + ibb) * YS;
          const double* pcd = st + NX * YS + NAB;
          double* out = row + 2 * NY * s;
          if (a.want & 1) {
            double j = 0.0;
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
              for (int d = 0; d < ND; ++d) j = fma(I[0][c][d], pcd[c * ND + d], j);
            fock_add_rt((s ? a.J2 : a.J) + mi.cmat + (size_t)(oa + ia) * n + ob + ibb, f * j, a.fx_lo);
          }
          if (a.want & 2) {
            double kad[ND], kbd[ND], pad[ND], pbd[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              kad[d] = kbd[d] = 0.0;
              pad[d] = pa[NC + d];
              pbd[d] = pb[NC + d];
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) {
              const double pac = pa[c], pbc = pb[c];
              double kac = 0.0, kbc = 0.0;
#pragma unroll
              for (int d = 0; d < ND; ++d) {
                const double v = I[0][c][d];
                kac = fma(v, pbd[d], kac);
                kbc = fma(v, pad[d], kbc);
                kad[d] = fma(v, pbc, kad[d]);
                kbd[d] = fma(v, pac, kbd[d]);
              }
              out[c] = kac;
              out[NY + c] = kbc;
            }
#pragma unroll
            for (int d = 0; d < ND; ++d) {
              out[NC + d] = kad[d];
              out[NY + NC + d] = kbd[d];
            }
          }
        }
      }
      if (a.want & 1) {                          // J(cd) = ket transfer of J~
        const KetPlan<LC, LD>& kp2 = g_ket_plan<LC, LD>;
        for (int s = 0; s < ns; ++s) {
          const double* jt = stage + s * C::STAGE + NX * YS + NAB + NCD;
          double* Jm = (s ? a.J2 : a.J) + mi.cmat;
          for (int cd = ql; cd < NCD; cd += QL) {
            const int c = cd / ND, d = cd - c * ND;
            double sum = 0.0;
#pragma unroll
            for (int q = 0; q < (1 << LD); ++q) {
              double cf = jt[kp2.f[cd][q]];
#pragma unroll
              for (int st = 0; st < LD; ++st)
                if (!(q >> st & 1)) {
                  const int dir = kp2.dir[d][st];
                  cf *= dir == 0 ? Rcd[0] : (dir == 1 ? Rcd[1] : Rcd[2]);
                }
              sum += cf;
            }
            fock_add_rt(Jm + (size_t)(oc + c) * n + od + d, f * sum, a.fx_lo);
          }
        }
      }
    }
    group_sync();
    if (act && (a.want & 2)) {                   // K: the rows' shares summed over b (rows of K at a) or a (at b)
      for (int s = 0; s < ns; ++s) {
        double* Km = (s ? a.K2 : a.K) + mi.cmat;
        const double* part = X + 2 * NY * s;
        for (int e = ql; e < NX * NY; e += QL) {
          const int x = e / NY, y = e - x * NY;
          double sum = 0.0;
          if (x < NA) {
            const double* q = part + x * NB * rs + y;
#pragma unroll
            for (int ibb = 0; ibb < NB; ++ibb) sum += q[ibb * rs];
          } else {
            const double* q = part + (x - NA) * rs + NY + y;
#pragma unroll
            for (int ia = 0; ia < NA; ++ia) sum += q[ia * NB * rs];
          }
          const int row = x < NA ? oa + x : ob + x - NA, col = y < NC ? oc + y : od + y - NC;
          fock_add_rt(Km + (size_t)row * n + col, f * sum, a.fx_lo);
        }
      }
    }
    group_sync();
  }
  if (GW == 1) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nprim += __shfl_xor_sync(0xffffffffu, nprim, o);
      nquart += __shfl_xor_sync(0xffffffffu, nquart, o);
    }
  }
  if ((GW == 1 ? lane : (int)threadIdx.x) == 0) {
    const int cls = ((LA * 5 + LB) * 5 + LC) * 5 + LD;
    if (nprim) atomicAdd(a.prim_count + cls, nprim);
    if (nquart) atomicAdd(a.qcount + cls, nquart);
  }
}

// Warps per block: one where a warp's groups take more than 12 KB, so that blocks fill
// an SM's shared memory closely, else four; a quartet wider than a warp is a block.
template <int LA, int LB, int LC, int LD>
constexpr int rows_wpb() {
  using C = RowCfg<LA, LB, LC, LD>;
  return C::GW > 1 ? C::GW : C::QPW * C::per_group(1) * 8 > 12288 ? 1 : 4;
}

// Launches the class (false: the launch could not be set up, which is done once per device).
// n <= 0 without a range only sets up.
template <int LA, int LB, int LC, int LD>
static bool launch_rows_t(const RowArgs& a, cudaStream_t s) {
  using C = RowCfg<LA, LB, LC, LD>;
  constexpr int WPB = rows_wpb<LA, LB, LC, LD>();
  constexpr int QPB = C::GW > 1 ? 1 : C::QPW * WPB;
  const size_t smem = (size_t)QPB * C::per_group(a.P2 ? 2 : 1) * sizeof(double);
  constexpr bool CAN_SHARE = C::QPW > 1;
  struct Resident {
    long long blocks[2];                      // restricted, unrestricted
  };
  static PerDevice<Resident> resident;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  Resident r_dev{};
  const bool ready = resident.get(dev, r_dev, [&](Resident& v) {
    const int top = (int)(QPB * C::per_group(2) * sizeof(double));
    int nsm = 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(k_jk_rows<LA, LB, LC, LD, WPB, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, top) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_jk_rows<LA, LB, LC, LD, WPB, CAN_SHARE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             top) != cudaSuccess)
      return false;
    for (int u = 0; u < 2; ++u) {
      int nb = 0;
      if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_jk_rows<LA, LB, LC, LD, WPB, false>, 32 * WPB,
                                                        (size_t)QPB * C::per_group(1 + u) * sizeof(double)) != cudaSuccess)
        return false;
      v.blocks[u] = (long long)nsm * std::max(nb, 1);
    }
    return true;
  });
  if (!ready) return false;
  if (a.n <= 0 && !a.range) return true;
  RowArgs r = a;
  const long long full = r_dev.blocks[a.P2 ? 1 : 0];
  r.groups = full * QPB;
  // sharing groups where the list is expected to leave half of them idle; always in a
  // deterministic build, whose sums must not depend on an expectation
  const bool shared = CAN_SHARE && (a.fx_lo || 2 * a.expect <= r.groups);
  const long long per_block = shared ? WPB : QPB, need = (a.n + per_block - 1) / per_block;
  const long long blocks = a.range || need > full ? full : need;
  if (shared) k_jk_rows<LA, LB, LC, LD, WPB, CAN_SHARE><<<(unsigned)blocks, 32 * WPB, smem, s>>>(r);
  else k_jk_rows<LA, LB, LC, LD, WPB, false><<<(unsigned)blocks, 32 * WPB, smem, s>>>(r);
  return true;
}

// The classes of one translation unit each (tf_rows_*.cu); 1: launched, 0: not a
// class of that unit, -1: the launch could not be set up.
int launch_rows_d(int key, const RowArgs& a, cudaStream_t s);
int launch_rows_fs(int key, const RowArgs& a, cudaStream_t s);
int launch_rows_fd(int key, const RowArgs& a, cudaStream_t s);
int launch_rows_ff(int key, const RowArgs& a, cudaStream_t s);

#define TF_ROWS_CASE(A, B, C, D) \
  case class_key(A, B, C, D): return launch_rows_t<A, B, C, D>(a, s) ? 1 : -1;

}  // namespace tf
