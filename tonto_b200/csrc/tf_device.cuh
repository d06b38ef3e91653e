// tf_device.cuh — device-side building blocks of the B200 Rys J/K builder.
//
// Everything that depends on angular momentum is resolved at compile time:
// Cartesian component tables (Tonto's lexical order, gaussian_data.foo:295-479)
// are constexpr, loops over components are unrolled with static_for, and the
// integral arrays therefore live in registers.  One thread computes one
// contracted shell quartet:
//   primitive quartets -> Rys nodes/weights (piecewise tables, FP64)
//   -> 2D recurrences on the higher-l centre of each pair (make_esfs_XX,
//      shell1quartet.foo:7418-7609) -> (e0|f0) accumulation (form_esfs :7615)
//   -> horizontal transfer ket then bra (transfer_cd / transfer_ab :8310-11134)
//   -> digestion into J and K with Tonto's coincidence factors
//      (molecule.fock.foo:1296-1338).
// The spherical transform of make_ERI (:433-563) is not applied per quartet:
// the density is taken to the Cartesian basis once per build and J, K are taken
// back once (the transforms commute with the contraction).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>
#include <utility>
#include <type_traits>

// (32-byte aligned: a polynomial's twelve coefficients are three 32-byte loads)
#define TF_RYS_CONST __device__ const __align__(32)
// the asymptotic-rule tables in the constant bank: read at compile-time indices,
// they become immediate operands instead of global loads
#define TF_RYS_SMALL_CONST __constant__ const
#include "rys_tables.inc"
#include "boys_table.inc"
#include "boys2_table.inc"

namespace tf {

// ---------------------------------------------------------------------------
// Reciprocal and reciprocal square root by one third-order step, seeded by the PTX
// approximate instructions rcp.approx.ftz.f64 / rsqrt.approx.ftz.f64 (about 20 correct
// bits).  With the residual e the truncated binomial series
//   1/x:       e = 1 - x y,    y <- y + y (e + e^2)
//   1/sqrt(x): e = 1 - x y^2,  y <- y + y e (1/2 + 3/8 e)
// leaves an error of order e^3, some 2^-59, below the double-precision rounding (a few
// ulp; checked against IEEE division and square root by tests/fast_math_check.cu): three
// and five operations where two Newton steps take four and seven.  Used for the
// exponent sums, rho, the Boys-function ratio and 1/x of the asymptotic rules: positive
// normal numbers far from the overflow range.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double rcp_nr(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double rsqrt_nr(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
}

// ---------------------------------------------------------------------------
// Fock accumulation.  FX = false: an FP64 atomic add.  Deterministic builds
// (FX = true, a kernel instantiation of its own so that the default kernels carry
// none of this code): the contribution v is split into two 64-bit fixed-point words,
// hi = round(v 2^32) and lo = round((v - hi 2^-32) 2^60), added with integer
// atomics to the element's hi word (the accumulator itself, read as an integer)
// and to its lo word, fx_lo elements further on.  v - hi 2^-32 is exact (the two
// are within a factor of two of each other, or hi = 0), so each contribution is
// kept to 2^-61; integer sums are exact and wrap modulo 2^64, so the totals do
// not depend on the order of the additions, and k_finalize reads them as
// hi 2^-32 + lo 2^-60.  Contributions and totals below 2^31 in magnitude.
// ---------------------------------------------------------------------------
template <bool FX>
__device__ __forceinline__ void fock_add(double* addr, double v, long long fx_lo) {
  if constexpr (!FX) {
    atomicAdd(addr, v);
  } else {
    const double h = rint(v * 0x1p32);
    const long long hi = (long long)h;
    const long long lo = __double2ll_rn((v - h * 0x1p-32) * 0x1p60);
    atomicAdd(reinterpret_cast<unsigned long long*>(addr), (unsigned long long)hi);
    atomicAdd(reinterpret_cast<unsigned long long*>(addr + fx_lo), (unsigned long long)lo);
  }
}

// The value of a Fock accumulator element (see fock_add).
__device__ __forceinline__ double fock_value(const double* m, size_t i, long long fx_lo) {
  if (fx_lo == 0) return m[i];
  const long long* q = reinterpret_cast<const long long*>(m);
  return (double)q[i] * 0x1p-32 + (double)q[i + fx_lo] * 0x1p-60;
}

// ---------------------------------------------------------------------------
// compile-time helpers
// ---------------------------------------------------------------------------
template <int... Is, class F>
__device__ __forceinline__ void static_for_impl(std::integer_sequence<int, Is...>, F&& f) {
  (f(std::integral_constant<int, Is>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
  static_for_impl(std::make_integer_sequence<int, N>{}, f);
}

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int ncart_upto(int l) { return l < 0 ? 0 : (l + 1) * (l + 2) * (l + 3) / 6; }

// Switch key of a class (la lb|lc ld), l <= 3.
__host__ __device__ constexpr int class_key(int la, int lb, int lc, int ld) { return ((la * 4 + lb) * 4 + lc) * 4 + ld; }

constexpr int LCOMP = 8;                         // components tabulated up to l = 8
constexpr int NCOMP_ALL = ncart_upto(LCOMP);     // 165

struct CompTable {
  int x[NCOMP_ALL], y[NCOMP_ALL], z[NCOMP_ALL];
  int first[LCOMP + 2];
  int idx[LCOMP + 1][LCOMP + 1][LCOMP + 1];      // position within its own l
};

__host__ __device__ constexpr void comp_push(CompTable& t, int& i, int X, int Y, int Z) {
  t.x[i] = X; t.y[i] = Y; t.z[i] = Z; ++i;
}

// Tonto's lexical Cartesian order: for L, the highest power a descends, then the
// second b, each pattern expanded in a fixed permutation order.
__host__ __device__ constexpr CompTable make_comp_table() {
  CompTable t{};
  int i = 0;
  for (int L = 0; L <= LCOMP; ++L) {
    t.first[L] = i;
    for (int a = L; a >= (L + 2) / 3; --a) {
      for (int b = (L - a < a ? L - a : a); b >= (L - a + 1) / 2; --b) {
        int c = L - a - b;
        if (a == b && b == c) {
          comp_push(t, i, a, a, a);
        } else if (a > b && b == c) {
          comp_push(t, i, a, b, b); comp_push(t, i, b, a, b); comp_push(t, i, b, b, a);
        } else if (a == b && b > c) {
          comp_push(t, i, a, a, c); comp_push(t, i, a, c, a); comp_push(t, i, c, a, a);
        } else {
          comp_push(t, i, a, b, c); comp_push(t, i, a, c, b); comp_push(t, i, b, a, c);
          comp_push(t, i, c, a, b); comp_push(t, i, b, c, a); comp_push(t, i, c, b, a);
        }
      }
    }
  }
  t.first[LCOMP + 1] = i;
  for (int k = 0; k < NCOMP_ALL; ++k) {
    int L = t.x[k] + t.y[k] + t.z[k];
    t.idx[t.x[k]][t.y[k]][t.z[k]] = k - t.first[L];
  }
  return t;
}

constexpr CompTable CT = make_comp_table();
static_assert(CT.first[LCOMP + 1] == NCOMP_ALL, "component table size");

__host__ __device__ constexpr int cx(int l, int i) { return CT.x[CT.first[l] + i]; }
__host__ __device__ constexpr int cy(int l, int i) { return CT.y[CT.first[l] + i]; }
__host__ __device__ constexpr int cz(int l, int i) { return CT.z[CT.first[l] + i]; }
// global lexical index -> powers
__host__ __device__ constexpr int gx(int g) { return CT.x[g]; }
__host__ __device__ constexpr int gy(int g) { return CT.y[g]; }
__host__ __device__ constexpr int gz(int g) { return CT.z[g]; }
__host__ __device__ constexpr int gidx(int x, int y, int z) { return CT.first[x + y + z] + CT.idx[x][y][z]; }

// ---------------------------------------------------------------------------
// data layouts shared with the host code
// ---------------------------------------------------------------------------
// One primitive pair (Gaussian product), positioned.  cc holds
// c_a c_b zeta^(-1) exp(-a b |AB|^2 / zeta): the prefactor c_a c_b zeta^(-3/2) exp(...)
// times sqrt(zeta), so that a primitive quartet's
// 2 pi^(5/2) cc_ab zeta^(-3/2) cc_cd eta^(-3/2) sqrt(rho), rho = zeta eta / (zeta + eta),
// becomes 2 pi^(5/2) cc_ab cc_cd / sqrt(zeta + eta): one reciprocal square root of
// zeta + eta gives both it and 1/(zeta + eta) (its square).
// Positions are not stored: P - A (A: the centre of the higher-l shell) is f (A - B),
// f = -b / zeta, so a record is one 32-byte word, one sector and one load instruction
// (ldg256).  The thread kernels are bound by the sectors their lanes' loads touch (one L1 data
// cycle each; every lane has its own ket): with 64-byte records (P and zeta, the rest) a ket
// primitive cost two, with 80-byte ones read 16 bytes at a time three to five.
struct __align__(32) PrimPair {
  double zeta, cc, f, half_zinv;     // cc: prefactor, half_zinv: 1/(2 zeta)
};
static_assert(sizeof(PrimPair) == 32, "primitive-pair record layout");

// One 32-byte read-only load (p 32-byte aligned).
__device__ __forceinline__ double4 ldg256(const void* p) {
  double4 v;
  asm("ld.global.nc.v4.f64 {%0, %1, %2, %3}, [%4];" : "=d"(v.x), "=d"(v.y), "=d"(v.z), "=d"(v.w) : "l"(p));
  return v;
}

// One shell pair, oriented so that shell "hi" has the higher l (ties: the
// shell with the larger index, as Tonto's pair (a >= b) orientation).
struct __align__(16) PairRec {
  int sh_hi, sh_lo;          // shell indices (Tonto order)
  int atom_hi, atom_lo;
  int cart_hi, cart_lo;      // first Cartesian function of each shell
  int full_off, n_full;      // primitive pairs without the pair cutoff
  int skip_off, n_skip;      // primitive pairs with the pair cutoff (atoms differ)
  int mol, tonto_ab;         // molecule (batched contexts), Tonto pair index a(a+1)/2+b within it
  double Rx, Ry, Rz;         // hi centre - lo centre
  double imax;               // Schwarz bound sqrt(max |(ab|ab)|)
};

// What the ERI kernels read of a shell pair, packed into one 32-byte word: {cart_hi,
// cart_lo, full_off, skip_off, atom_hi, atom_lo, n_full | n_skip << 16, mol | (shell hi ==
// shell lo) << 31}; the centres come from the atom positions (32 bytes an atom), which the
// neighbouring kets of a warp share.
struct PairJK {
  int cart_hi, cart_lo, full_off, skip_off;
  int atom_hi, atom_lo, n_full, n_skip, mol;
  bool same;                 // both shells the same (coincidence factor 1/2)
  double Ax, Ay, Az;         // hi centre
  double Rx, Ry, Rz;         // hi centre - lo centre
};

__device__ __forceinline__ PairJK load_pair_jk(const int4* __restrict__ rec, const double4* __restrict__ xyz4, int id) {
  int4 x, y;
  asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w), "=r"(y.x), "=r"(y.y), "=r"(y.z), "=r"(y.w)
      : "l"(rec + 2 * id));
  PairJK p;
  p.cart_hi = x.x; p.cart_lo = x.y; p.full_off = x.z; p.skip_off = x.w;
  p.atom_hi = y.x; p.atom_lo = y.y;
  p.n_full = y.z & 0xffff; p.n_skip = (int)((unsigned)y.z >> 16);
  p.mol = y.w & 0x7fffffff; p.same = y.w < 0;
  const double4 A = ldg256(xyz4 + p.atom_hi), B = ldg256(xyz4 + p.atom_lo);
  p.Ax = A.x; p.Ay = A.y; p.Az = A.z;
  p.Rx = A.x - B.x; p.Ry = A.y - B.y; p.Rz = A.z - B.z;
  return p;
}

// Quartet range of a launch in a graph-captured build: list[range[0] - base,
// range[1] - base), read on the device and clamped to the list capacity.
__device__ __forceinline__ void resolve_range(const long long* range, long long base, long long cap,
                                              const int2*& q, long long& n) {
  if (range) {
    const long long s0 = range[0], s1 = min(range[1], base + cap);
    q += s0 - base;
    n = s1 > s0 ? s1 - s0 : 0;
  }
}

// Cost buckets of the primitive-quartet count npq: npq itself below 8, then quarter
// octaves (counts within a factor 1.19 share a bucket), so that the lanes of a warp
// loop over nearly the same number of primitive quartets.
constexpr int NCOST = 47;
constexpr int NBUCKET = 2 * NCOST;         // FP64 buckets, then FP32 buckets

// Work of one thread-kernel launch, computed on the device from the list's bucket counts
// (k_group_offsets): the buckets, heaviest first, each cut into warps.  Bucket j holds
// list entries [item0[j], item0[j] + count[j]); 2^lg[j] neighbouring lanes share one
// entry's primitive quartets; warps [warp0[j], warp0[j + 1]) work on it.
struct LaunchPlan {
  long long item0[NCOST], count[NCOST], warp0[NCOST + 1];
  int lg[NCOST];
};

// One molecule of a (possibly batched) context: its shells are a contiguous
// global range; its matrices sit at fixed offsets in the concatenated buffers.
struct __align__(16) MolInfo {
  int shell0, n_shell;       // global shell range
  int cart0, bf0;            // first global Cartesian / basis function
  int n_cart, n_bf;
  int atom0, n_atom;         // global atom range
  long long cmat;            // offset of its n_cart x n_cart Cartesian block
  long long bmat;            // offset of its n_bf x n_bf Tonto-basis block
  long long pmax;            // offset of its n_shell x n_shell pair-maximum block
};

// molecule owning element t of a concatenated buffer with offsets off[0..n_mol]
__device__ __forceinline__ int find_mol(const long long* __restrict__ off, int n_mol, long long t) {
  int lo = 0, hi = n_mol - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (off[mid] <= t) lo = mid; else hi = mid - 1;
  }
  return lo;
}

constexpr double TWOPI5ON2 = 34.9868366552497256925;   // 2 pi^(5/2)

// ---------------------------------------------------------------------------
// Rys nodes and weights (FP64 always)
// ---------------------------------------------------------------------------
__host__ __device__ constexpr int rys_xmax(int n) { const int t[] = TF_RYS_XMAX_INIT; return t[n]; }
__host__ __device__ constexpr int rys_offset(int n) { const int t[] = TF_RYS_OFFSET_INIT; return t[n]; }
__host__ __device__ constexpr int rys_hoffset(int n) { const int t[] = TF_RYS_HOFFSET_INIT; return t[n]; }

template <int N>
__device__ __forceinline__ void rys_eval(double x, double (&u)[N], double (&w)[N]) {
  constexpr int XMAX = rys_xmax(N), OFF = rys_offset(N), HOFF = rys_hoffset(N);
  if (x < (double)XMAX) {
    const int j = (int)x;
    const double s = x - (double)j;
    const double* c = tf_rys_coef + OFF + j * (2 * N * TF_RYS_NCOEF);
#pragma unroll
    for (int f = 0; f < 2 * N; ++f) {
      const double* cf = c + f * TF_RYS_NCOEF;
      double v = __ldg(cf + TF_RYS_DEG);
#pragma unroll
      for (int k = TF_RYS_DEG - 1; k >= 0; --k) v = fma(v, s, __ldg(cf + k));
      if (f < N) u[f] = v; else w[f - N] = v;
    }
  } else {
    const double ix = rcp_nr(x);
    const double isx = rsqrt_nr(x);
#pragma unroll
    for (int i = 0; i < N; ++i) {
      u[i] = tf_rys_hroot2[HOFF + i] * ix;
      w[i] = tf_rys_hweight[HOFF + i] * isx;
    }
  }
}

// The same tables staged in shared memory, transposed to [coef][function][interval]
// so that lanes evaluating different intervals hit different banks.
template <int N>
struct RysPoly {
  static constexpr int NI = rys_xmax(N);              // intervals
  static constexpr int SIZE = TF_RYS_NCOEF * 2 * N * NI;
  // layout [k][j][i] with the pairs (u_i, w_i) adjacent: one 16-byte load per
  // (coefficient, root)
  static __device__ __forceinline__ void load(double* t) {
    constexpr int OFF = rys_offset(N);
    for (int q = threadIdx.x; q < SIZE; q += blockDim.x) {
      // q = ((k * NI + j) * N + i) * 2 + (0: node, 1: weight)
      const int uw = q & 1, i = (q >> 1) % N, kj = (q >> 1) / N, j = kj % NI, k = kj / NI;
      const int f = uw ? N + i : i;
      t[q] = tf_rys_coef[OFF + j * (2 * N * TF_RYS_NCOEF) + f * TF_RYS_NCOEF + k];
    }
  }
  static __device__ __forceinline__ void eval(const double* __restrict__ t, double x, double (&u)[N], double (&w)[N]) {
    if (x < (double)NI) {
      const int j = (int)x;
      const double s = x - (double)j;
      const double2* c = reinterpret_cast<const double2*>(t) + j * N;
      constexpr int KS = NI * N;                     // stride between coefficients (double2)
#pragma unroll
      for (int i = 0; i < N; ++i) {
        const double2 v = c[TF_RYS_DEG * KS + i];
        u[i] = v.x;
        w[i] = v.y;
      }
#pragma unroll
      for (int k = TF_RYS_DEG - 1; k >= 0; --k)
#pragma unroll
        for (int i = 0; i < N; ++i) {
          const double2 v = c[k * KS + i];
          u[i] = fma(u[i], s, v.x);
          w[i] = fma(w[i], s, v.y);
        }
    } else {
      constexpr int HOFF = rys_hoffset(N);
      const double ix = rcp_nr(x);
      const double isx = rsqrt_nr(x);
#pragma unroll
      for (int i = 0; i < N; ++i) {
        u[i] = tf_rys_hroot2[HOFF + i] * ix;
        w[i] = tf_rys_hweight[HOFF + i] * isx;
      }
    }
  }
};

template <int N>
struct RysSmem : RysPoly<N> {};

// One root: the rule is exact for f linear in t^2, so w = F0(x) and u = F1(x)/F0(x).
// F0 and F1 come from an 8-term Taylor step about the nearest point k/8 of a grid
// of F_0..F_8 (gen_boys_table.py; dF_m/dx = -F_{m+1}): five 16-byte table loads
// per evaluation instead of one per polynomial coefficient.
template <>
struct RysSmem<1> {
  static constexpr int SIZE = TF_BOYS_NPTS * TF_BOYS_NM;
  static __device__ __forceinline__ void load(double* t) {
    for (int q = threadIdx.x; q < SIZE; q += blockDim.x) t[q] = tf_boys_grid[q];
  }
  static __device__ __forceinline__ void eval(const double* __restrict__ t, double x, double (&u)[1], double (&w)[1]) {
    static_assert(TF_BOYS_NTERM == 8 && TF_BOYS_NM == 10, "Taylor step written for 8 terms");
    if (x < (double)TF_BOYS_XMAX) {
      const int k = (int)(x * (double)TF_BOYS_H_INV + 0.5);
      const double d = (double)k * (1.0 / TF_BOYS_H_INV) - x;
      const double2* g = reinterpret_cast<const double2*>(t + k * TF_BOYS_NM);
      const double2 f01 = g[0], f23 = g[1], f45 = g[2], f67 = g[3], f89 = g[4];
      const double d2 = d * 0.5, d3 = d * (1.0 / 3.0), d4 = d * 0.25, d5 = d * 0.2, d6 = d * (1.0 / 6.0),
                   d7 = d * (1.0 / 7.0);
      double a = fma(d7, f67.y, f67.x);      // F0 = f0 + d (f1 + d/2 (f2 + ... + d/7 f7))
      double b = fma(d7, f89.x, f67.y);      // F1 = f1 + d (f2 + d/2 (f3 + ... + d/7 f8))
      a = fma(d6, a, f45.y);
      b = fma(d6, b, f67.x);
      a = fma(d5, a, f45.x);
      b = fma(d5, b, f45.y);
      a = fma(d4, a, f23.y);
      b = fma(d4, b, f45.x);
      a = fma(d3, a, f23.x);
      b = fma(d3, b, f23.y);
      a = fma(d2, a, f01.y);
      b = fma(d2, b, f23.x);
      a = fma(d, a, f01.x);
      b = fma(d, b, f01.y);
      w[0] = a;
      u[0] = b * rcp_nr(a);
    } else {
      constexpr int HOFF = rys_hoffset(1);
      u[0] = tf_rys_hroot2[HOFF] * rcp_nr(x);
      w[0] = tf_rys_hweight[HOFF] * rsqrt_nr(x);
    }
  }
};

#ifndef TF_RYS2_MOMENTS
#define TF_RYS2_MOMENTS 1
#endif
#if TF_RYS2_MOMENTS
// Two roots: the Gauss rule of the moments F_0..F_3 (gen_boys_table.py): u_1, u_2
// are the roots of u^2 + a u + b, the monic polynomial orthogonal to 1 and u,
//   a = (F0 F3 - F1 F2) / (F1^2 - F0 F2),  b = (F2^2 - F1 F3) / (F1^2 - F0 F2),
// taken as q = (sqrt(a^2 - 4b) - a) / 2 (a < 0: no cancellation), u_1 = q,
// u_2 = b / q; w_1 = (F0 u_2 - F1) / (u_2 - u_1), w_2 = F0 - w_1.  F0..F3 by the
// 8-term Taylor step from a 1/8 grid of F_0..F_10: six 16-byte loads instead of 24.
template <>
struct RysSmem<2> {
  static constexpr int SIZE = TF_BOYS2_NPTS * TF_BOYS2_NM;
  static __device__ __forceinline__ void load(double* t) {
    for (int q = threadIdx.x; q < SIZE; q += blockDim.x) t[q] = tf_boys2_grid[q];
  }
  static __device__ __forceinline__ void eval(const double* __restrict__ t, double x, double (&u)[2], double (&w)[2]) {
    static_assert(TF_BOYS_NTERM == 8 && TF_BOYS2_NM == 12 && TF_BOYS2_XMAX == 50, "grid for the two-point rule");
    if (x < (double)TF_BOYS2_XMAX) {
      const int k = (int)(x * (double)TF_BOYS_H_INV + 0.5);
      const double d = (double)k * (1.0 / TF_BOYS_H_INV) - x;
      const double2* g = reinterpret_cast<const double2*>(t + k * TF_BOYS2_NM);
      double f[12];
#pragma unroll
      for (int q = 0; q < 6; ++q) {
        const double2 v = g[q];
        f[2 * q] = v.x;
        f[2 * q + 1] = v.y;
      }
      const double dj[8] = {0.0, d, d * 0.5, d * (1.0 / 3.0), d * 0.25, d * 0.2, d * (1.0 / 6.0), d * (1.0 / 7.0)};
      double m[4];
#pragma unroll
      for (int r = 0; r < 4; ++r) {              // F_r = f_r + d (f_{r+1} + d/2 (... + d/7 f_{r+7}))
        double v = f[r + 7];
#pragma unroll
        for (int j = 7; j >= 1; --j) v = fma(dj[j], v, f[r + j - 1]);
        m[r] = v;
      }
      const double r = rcp_nr(m[1] * m[1] - m[0] * m[2]);
      const double a = (m[0] * m[3] - m[1] * m[2]) * r;
      const double b = (m[2] * m[2] - m[1] * m[3]) * r;
      const double disc = fma(a, a, -4.0 * b);
      const double q = 0.5 * (disc * rsqrt_nr(disc) - a);
      u[0] = q;
      u[1] = b * rcp_nr(q);
      const double w0 = (m[0] * u[1] - m[1]) * rcp_nr(u[1] - u[0]);
      w[0] = w0;
      w[1] = m[0] - w0;
    } else {
      constexpr int HOFF = rys_hoffset(2);
      const double ix = rcp_nr(x);
      const double isx = rsqrt_nr(x);
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        u[i] = tf_rys_hroot2[HOFF + i] * ix;
        w[i] = tf_rys_hweight[HOFF + i] * isx;
      }
    }
  }
};
#endif

// Boys functions F_0 .. F_M, M <= 3, of the classes evaluated by the vertical recurrence
// (prim_quartet_vrr): the 8-term Taylor step of the grids above about the nearest point
// k/8; beyond the grid (42, or 50 for M >= 2) F_0 = sqrt(pi/x)/2 and F_{m+1} = (2m+1)/(2x)
// F_m, where exp(-x)/(2x) is below rounding.  M = 0, 1: the table holds F_j(k/8)/j!, the
// coefficients of F_0 in d = k/8 - x; F_1 is that polynomial's derivative, one Horner scheme
// for both (15 operations against 20 with the factors d/j).  M = 2, 3: one independent chain per
// order, shorter in latency and no longer in operations.
template <int M>
struct BoysSmem {
  static constexpr bool WIDE = M >= 2;
  static constexpr int NM = WIDE ? TF_BOYS2_NM : TF_BOYS_NM, NPTS = WIDE ? TF_BOYS2_NPTS : TF_BOYS_NPTS;
  static constexpr int XMAX = WIDE ? TF_BOYS2_XMAX : TF_BOYS_XMAX;
  static constexpr int SIZE = NPTS * NM;
  static __device__ __forceinline__ void load(double* t) {
    if constexpr (WIDE) {
      for (int q = threadIdx.x; q < SIZE; q += blockDim.x) t[q] = tf_boys2_grid[q];
    } else {
      for (int q = threadIdx.x; q < SIZE; q += blockDim.x) {
        const int j = q % NM;
        const double f = j < 2 ? 1.0 : j == 2 ? 2.0 : j == 3 ? 6.0 : j == 4 ? 24.0 : j == 5 ? 120.0 : j == 6 ? 720.0
                         : j == 7 ? 5040.0 : 40320.0;
        t[q] = tf_boys_grid[q] / f;
      }
    }
  }
  static __device__ __forceinline__ void eval(const double* __restrict__ t, double x, double (&F)[M + 1]) {
    static_assert(M <= 3 && TF_BOYS_NTERM == 8, "grids of F_0 .. F_8 and F_0 .. F_10");
    if (x < (double)XMAX) {
      const int k = (int)(x * (double)TF_BOYS_H_INV + 0.5);
      const double d = (double)k * (1.0 / TF_BOYS_H_INV) - x;
      const double2* g = reinterpret_cast<const double2*>(t + k * NM);
      double f[2 * ((M + 9) / 2)];
#pragma unroll
      for (int q = 0; q < (M + 9) / 2; ++q) {
        const double2 v = g[q];
        f[2 * q] = v.x;
        f[2 * q + 1] = v.y;
      }
      if constexpr (M == 0) {
        double p = f[7];
#pragma unroll
        for (int j = 6; j >= 0; --j) p = fma(p, d, f[j]);
        F[0] = p;
      } else if constexpr (M == 1) {
        double p = fma(f[8], d, f[7]), q = f[8];       // value and derivative
#pragma unroll
        for (int j = 6; j >= 0; --j) {
          q = fma(q, d, p);
          p = fma(p, d, f[j]);
        }
        F[0] = p;
        F[1] = q;
      } else {
        const double dj[8] = {0.0, d, d * 0.5, d * (1.0 / 3.0), d * 0.25, d * 0.2, d * (1.0 / 6.0), d * (1.0 / 7.0)};
#pragma unroll
        for (int m = 0; m <= M; ++m) F[m] = f[m + 7];
#pragma unroll
        for (int j = 7; j >= 1; --j)
#pragma unroll
          for (int m = 0; m <= M; ++m) F[m] = fma(dj[j], F[m], f[m + j - 1]);
      }
    } else {
      const double r = rsqrt_nr(x), ix = r * r;
      F[0] = tf_rys_hweight[rys_hoffset(1)] * r;
#pragma unroll
      for (int m = 0; m < M; ++m) F[m + 1] = (m + 0.5) * ix * F[m];
    }
  }
};

// ---------------------------------------------------------------------------
// One contracted shell quartet (LA LB | LC LD), LA >= LB, LC >= LD, in
// arithmetic type T for the 2D recurrences and (e0|f0) sums (double, or float
// for the mixed-precision path); nodes/weights and the final integrals FP64.
// ---------------------------------------------------------------------------
template <int LA, int LB, int LC, int LD>
struct Quartet {
  static constexpr int LAB = LA + LB, LCD = LC + LD;
  static constexpr int NROOT = (LAB + LCD) / 2 + 1;
  static constexpr int FE = CT.first[LA], NE = CT.first[LAB + 1] - CT.first[LA];   // e: l in [LA, LA+LB]
  static constexpr int FF = CT.first[LC], NF = CT.first[LCD + 1] - CT.first[LC];
  static constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
  static constexpr int NINT = NA * NB * NC * ND;
};

// (e0|f0) accumulation over all primitive quartets of a contracted quartet.
#ifndef TF_PRIM_UNROLL
#define TF_PRIM_UNROLL 1
#endif

constexpr int kPrimUnroll = TF_PRIM_UNROLL;

// A loaded primitive-pair record: (zeta, cc, f, 1/(2 zeta)).
typedef double4 PrimRegs;
__device__ __forceinline__ PrimRegs load_prim(const PrimPair* __restrict__ q, int i) { return ldg256(q + i); }

// Geometry of a quartet: A - B, C - D, and C - A.
struct QuartetGeom {
  double Rab[3], Rcd[3], CA[3];
};
__device__ __forceinline__ QuartetGeom quartet_geom(const PairJK& b, const PairJK& k) {
  return QuartetGeom{{b.Rx, b.Ry, b.Rz}, {k.Rx, k.Ry, k.Rz}, {k.Ax - b.Ax, k.Ay - b.Ay, k.Az - b.Az}};
}

// P - A, Q - C and Q - P of a primitive quartet; QA = Q - A of its ket, which a loop over
// bras keeps.
struct PrimGeom {
  double PA[3], QC[3], QP[3];
};
struct KetPos {
  double QA[3];
};
__device__ __forceinline__ KetPos ket_pos(const PrimRegs& K, const QuartetGeom& g) {
  return KetPos{{fma(K.z, g.Rcd[0], g.CA[0]), fma(K.z, g.Rcd[1], g.CA[1]), fma(K.z, g.Rcd[2], g.CA[2])}};
}
__device__ __forceinline__ PrimGeom prim_geom(const PrimRegs& B, const PrimRegs& K, const KetPos& q,
                                              const QuartetGeom& g) {
  PrimGeom r;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    r.PA[i] = B.z * g.Rab[i];
    r.QC[i] = K.z * g.Rcd[i];
    r.QP[i] = fma(-B.z, g.Rab[i], q.QA[i]);
  }
  return r;
}
__device__ __forceinline__ PrimGeom prim_geom(const PrimRegs& B, const PrimRegs& K, const QuartetGeom& g) {
  return prim_geom(B, K, ket_pos(K, g), g);
}

// 1/x and 1/sqrt(x) in FP32 (the PTX approximate instructions, about 23 correct
// bits: the rounding level of the FP32 arithmetic they feed).
__device__ __forceinline__ float rcp_f32(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_f32(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// Classes evaluated by the vertical recurrence over Boys functions (Obara and Saika, J. Chem.
// Phys. 84, 3963 (1986)) instead of Rys quadrature: up to three quanta in all and an ss or ps
// ket.  There the recurrence takes a third to a half of the quadrature's FP64 operations
// ((ps|ps) 33 against about 120 after the Boys functions: no root finding, no sum over
// roots) with as few live values; from four quanta on, its tables no longer fit the
// registers beside the (e0|f0) block.  T = float (mixed precision) keeps the quadrature: an
// incremental build is nearly all FP32 quartets, and its rounding is part of its result.
// Measured: (H2O)32 cc-pVDZ (ps|ps) 10.17 -> 9.31 ms, (pp|ss) 5.28 -> 4.73, (ds|ss) 4.27 ->
// 3.86, (ps|ss) 12.63 -> 12.45, the build 73.2 -> 71.0; 24 clusters batched 191 -> 184 ms.
template <int LA, int LB, int LC, int LD, typename T>
__host__ __device__ constexpr bool use_vrr() {
  return std::is_same<T, double>::value && LC + LD <= 1 && LA + LB + LC + LD <= 3;
}

// The table a thread kernel's primitive loop reads in shared memory.
template <int LA, int LB, int LC, int LD, typename T>
using RootTable = std::conditional_t<use_vrr<LA, LB, LC, LD, T>(),
                                     BoysSmem<(use_vrr<LA, LB, LC, LD, T>() ? LA + LB + LC + LD : 0)>,
                                     RysSmem<(LA + LB + LC + LD) / 2 + 1>>;

// Direction along which Cartesian component g is raised from a lower one: the smallest
// non-zero power, so that most components need no third term.
__host__ __device__ constexpr int vrr_dir(int g) {
  const int v[3] = {gx(g), gy(g), gz(g)};
  int d = -1;
  for (int i = 0; i < 3; ++i)
    if (v[i] > 0 && (d < 0 || v[i] < v[d])) d = i;
  return d;
}
__host__ __device__ constexpr int comp_power(int g, int i) { return i == 0 ? gx(g) : (i == 1 ? gy(g) : gz(g)); }
__host__ __device__ constexpr int comp_lower(int g, int i) {
  return gidx(gx(g) - (i == 0), gy(g) - (i == 1), gz(g) - (i == 2));
}

// [e0|f0] of one primitive quartet, added to esfs, from S[m] = [00|00]^(m):
//   [e+1_i, 0]^m = PA_i [e]^m + WP_i [e]^(m+1) + e_i/(2 zeta) ([e-1_i]^m - r_z [e-1_i]^(m+1)),
//   [e, 1_j] = QC_j [e]^0 + WQ_j [e]^1 + e_j/(2(zeta+eta)) [e-1_j]^1,
// WP = r_z QP, WQ = -r_e QP, r_z = rho/zeta, r_e = rho/eta.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void vrr_add(const double (&S)[LA + LB + LC + LD + 1], const double (&PA)[3], const double (&WP)[3],
                                        const double (&QC)[3], const double (&WQ)[3], double half_zinv, double r_z, double half_inv,
                                        double (&esfs)[Quartet<LA, LB, LC, LD>::NE][Quartet<LA, LB, LC, LD>::NF]) {
  using Q = Quartet<LA, LB, LC, LD>;
  constexpr int L = Q::LAB + Q::LCD, LAB = Q::LAB, LCD = Q::LCD, NG = ncart_upto(LAB);
  double v[NG][L + 1], dz[NG][L + 1];             // [e]^m, and 1/(2 zeta) ([e]^m - r_z [e]^(m+1))
#pragma unroll
  for (int m = 0; m <= L; ++m) v[0][m] = S[m];
  static_for<NG>([&](auto gg) {
    constexpr int g = decltype(gg)::value, l = gx(g) + gy(g) + gz(g);
    if constexpr (l > 0) {
      constexpr int i = vrr_dir(g), p = comp_lower(g, i), e = comp_power(p, i);
      // the highest level without a ket step is only added up
      constexpr int MM = (LAB - l) + LCD;
      constexpr bool sum_only = MM == 0;
      static_for<MM + 1>([&](auto mm) {
        constexpr int m = decltype(mm)::value;
        double t = sum_only ? esfs[g - Q::FE >= 0 ? g - Q::FE : 0][0] : 0.0;
        t = sum_only ? fma(PA[i], v[p][m], t) : PA[i] * v[p][m];
        t = fma(WP[i], v[p][m + 1], t);
        if constexpr (e > 0) {
          constexpr int pp = comp_lower(p, i);
          t = fma(double(e), dz[pp][m], t);
        }
        if constexpr (sum_only) esfs[g - Q::FE][0] = t;
        else v[g][m] = t;
      });
    }
    if constexpr (l + 2 <= LAB) {            // raised twice along one direction later
      static_for<LAB - l - 2 + LCD + 1>([&](auto mm) {
        constexpr int m = decltype(mm)::value;
        dz[g][m] = half_zinv * fma(-r_z, v[g][m + 1], v[g][m]);
      });
    }
  });
  static_for<Q::NE>([&](auto ee) {
    constexpr int e = decltype(ee)::value, g = Q::FE + e, l = gx(g) + gy(g) + gz(g);
    if constexpr (LCD == 0) {
      if constexpr (l < LAB || LAB == 0) esfs[e][0] += v[g][0];
    } else {
      static_for<3>([&](auto jj) {
        constexpr int j = decltype(jj)::value, ej = comp_power(g, j);
        double t = fma(QC[j], v[g][0], esfs[e][j]);
        t = fma(WQ[j], v[g][1], t);
        if constexpr (ej > 0) t = fma(double(ej) * half_inv, v[comp_lower(g, j)][1], t);
        esfs[e][j] = t;
      });
    }
  });
}

// F_0 .. F_M at x from the table in shared memory, or (null) from the Rys rule, which is
// exact for them.
template <int M>
__device__ __forceinline__ void boys_eval(const double* __restrict__ tab, double x, double (&F)[M + 1]) {
  if (tab) {
    BoysSmem<M>::eval(tab, x, F);
  } else {
    constexpr int N = M / 2 + 1;
    double u[N], w[N];
    rys_eval<N>(x, u, w);
#pragma unroll
    for (int m = 0; m <= M; ++m) F[m] = 0.0;
#pragma unroll
    for (int r = 0; r < N; ++r) {
      double p = w[r];
#pragma unroll
      for (int m = 0; m <= M; ++m) { F[m] += p; p *= u[r]; }
    }
  }
}

// One primitive quartet by the vertical recurrence.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void prim_quartet_vrr(const PrimRegs& B, const PrimRegs& K, const KetPos& q,
                                                 const QuartetGeom& g,
                                                 double (&esfs)[Quartet<LA, LB, LC, LD>::NE][Quartet<LA, LB, LC, LD>::NF],
                                                 const double* __restrict__ tab) {
  constexpr int L = LA + LB + LC + LD;
  const PrimGeom p = prim_geom(B, K, q, g);
  const double zeta = B.x, eta = K.x;
  const double sq = rsqrt_nr(zeta + eta);      // 1/sqrt(zeta + eta)
  const double inv = sq * sq, r_z = eta * inv, r_e = zeta * inv;
  const double xx = zeta * r_z * (p.QP[0] * p.QP[0] + p.QP[1] * p.QP[1] + p.QP[2] * p.QP[2]);
  double F[L + 1];
  boys_eval<L>(tab, xx, F);
  const double scale = B.y * K.y * TWOPI5ON2 * sq;
  double S[L + 1], WP[3], WQ[3];
#pragma unroll
  for (int m = 0; m <= L; ++m) S[m] = F[m] * scale;
  if constexpr (L == 1) {                      // one step: r_z with S[1] instead of with Q - P
    const double s1 = r_z * S[1];
#pragma unroll
    for (int i = 0; i < 3; ++i) esfs[i][0] = fma(p.QP[i], s1, fma(p.PA[i], S[0], esfs[i][0]));
    return;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    WP[i] = r_z * p.QP[i];
    WQ[i] = -r_e * p.QP[i];
  }
  vrr_add<LA, LB, LC, LD>(S, p.PA, WP, p.QC, WQ, B.w, r_z, 0.5 * inv, esfs);
}

// One primitive quartet in the mixed-precision path: the Boys-function argument
// and everything after the Rys nodes and weights in FP32 (exponent sums, rho, the
// prefactor, the recurrence coefficients, the 2D recurrences and the (e0|f0)
// products); P - Q in FP64 (a difference of positions), then the nodes and weights
// themselves in FP64 from the FP64 tables, as for the FP64 path.
// The order of every FP32 operation is written out (no contraction left to the compiler):
// an incremental build is nearly all FP32 quartets, so a different rounding shows in its
// result, and all kernel variants of a class should give the same one.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void prim_quartet_f32(const PrimRegs& B, const PrimRegs& K, const KetPos& q,
                                                 const QuartetGeom& g,
                                                 float (&esfs)[Quartet<LA, LB, LC, LD>::NE][Quartet<LA, LB, LC, LD>::NF],
                                                 const double* __restrict__ rys_smem) {
  using Q = Quartet<LA, LB, LC, LD>;
  constexpr int D1 = Q::LAB + 1, D2 = Q::LCD + 1, NR = Q::NROOT;
  const PrimGeom p = prim_geom(B, K, q, g);
  const float zeta = (float)B.x, eta = (float)K.x;
  const float half_zinv = (float)B.w, half_einv = (float)K.w;
  const float sq = rsqrt_f32(__fadd_rn(zeta, eta));
  const float inv = __fmul_rn(sq, sq);
  const float rho = __fmul_rn(__fmul_rn(zeta, eta), inv);
  const float QP[3] = {(float)p.QP[0], (float)p.QP[1], (float)p.QP[2]};
  const float xx = __fmul_rn(rho, __fmaf_rn(QP[2], QP[2], __fmaf_rn(QP[0], QP[0], __fmul_rn(QP[1], QP[1]))));
  double u[NR], w[NR];
  if (rys_smem) RysSmem<NR>::eval(rys_smem, (double)xx, u, w);
  else rys_eval<NR>((double)xx, u, w);
  const float scale = __fmul_rn((float)(B.y * K.y * TWOPI5ON2), sq);
  const float r_z = __fmul_rn(eta, inv);     // rho / zeta
  const float r_e = __fmul_rn(zeta, inv);    // rho / eta
  const float PA[3] = {(float)p.PA[0], (float)p.PA[1], (float)p.PA[2]};
  const float QC[3] = {(float)p.QC[0], (float)p.QC[1], (float)p.QC[2]};
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const float t2 = (float)u[r];
    const float t2_rz = __fmul_rn(t2, r_z), t2_re = __fmul_rn(t2, r_e);
    const float B10 = __fmul_rn(__fsub_rn(1.0f, t2_rz), half_zinv);
    const float B01 = __fmul_rn(__fsub_rn(1.0f, t2_re), half_einv);
    const float B00 = __fmul_rn(__fmul_rn(0.5f, t2), inv);
    const float wt = __fmul_rn((float)w[r], scale);
    float I[3][D1][D2];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const float c00 = __fmaf_rn(t2_rz, QP[d], PA[d]);
      const float d00 = __fmaf_rn(-t2_re, QP[d], QC[d]);
      I[d][0][0] = (d == 2) ? wt : 1.0f;
      if (D1 > 1) I[d][1][0] = d == 2 ? __fmul_rn(c00, wt) : c00;
#pragma unroll
      for (int e = 1; e + 1 < D1; ++e)
        I[d][e + 1][0] = d == 2 && D1 == 3 ? __fmaf_rn(B10, I[d][0][0], __fmul_rn(c00, I[d][1][0]))
                                : __fmaf_rn(c00, I[d][e][0], __fmul_rn(__fmul_rn(float(e), B10), I[d][e - 1][0]));
#pragma unroll
      for (int f = 0; f + 1 < D2; ++f) {
#pragma unroll
        for (int e = 0; e < D1; ++e) {
          const float i0 = I[d][e][f];
          float v;
          if (f > 0) {
            v = __fmaf_rn(d00, i0, __fmul_rn(__fmul_rn(float(f), B01), I[d][e][f - 1]));
            if (e > 0) v = __fmaf_rn(__fmul_rn(float(e), B00), I[d][e - 1][f], v);
          } else if (e > 0) {
            v = __fmaf_rn(d00, i0, __fmul_rn(__fmul_rn(float(e), B00), I[d][e - 1][f]));
          } else {
            v = __fmul_rn(d00, i0);
          }
          I[d][e][f + 1] = v;
        }
      }
    }
    if constexpr (Q::LAB == 1 && Q::LCD == 0) {      // one product per element, none rounded by itself
      esfs[0][0] = __fmaf_rn(I[0][1][0], wt, esfs[0][0]);
      esfs[1][0] = __fmaf_rn(I[1][1][0], wt, esfs[1][0]);
      esfs[2][0] = __fmaf_rn(__fmaf_rn(t2_rz, QP[2], PA[2]), wt, esfs[2][0]);
    } else {
      static_for<Q::NE>([&](auto e) {
        constexpr int ge = Q::FE + decltype(e)::value;
        static_for<Q::NF>([&](auto f) {
          constexpr int gf = Q::FF + decltype(f)::value;
          float& es = esfs[decltype(e)::value][decltype(f)::value];
          es = __fmaf_rn(__fmul_rn(I[0][gx(ge)][gx(gf)], I[1][gy(ge)][gy(gf)]), I[2][gz(ge)][gz(gf)], es);
        });
      });
    }
  }
}

// One primitive quartet: Rys nodes and weights, the 2D recurrences and the
// (e0|f0) products, added to esfs.
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ void prim_quartet(const PrimRegs& B, const PrimRegs& K, const KetPos& q,
                                             const QuartetGeom& g,
                                             T (&esfs)[Quartet<LA, LB, LC, LD>::NE][Quartet<LA, LB, LC, LD>::NF],
                                             const double* __restrict__ rys_smem) {
  if constexpr (use_vrr<LA, LB, LC, LD, T>()) {
    prim_quartet_vrr<LA, LB, LC, LD>(B, K, q, g, esfs, rys_smem);
    return;
  } else if constexpr (std::is_same<T, float>::value) {
    prim_quartet_f32<LA, LB, LC, LD>(B, K, q, g, esfs, rys_smem);
    return;
  } else {
  using Q = Quartet<LA, LB, LC, LD>;
  constexpr int D1 = Q::LAB + 1, D2 = Q::LCD + 1, NR = Q::NROOT;
  const PrimGeom p = prim_geom(B, K, q, g);
  const double bcc = B.y * TWOPI5ON2, kcc = K.y;
  const double zeta = B.x, half_zinv = B.w;
  const double eta = K.x, half_einv = K.w;
  const double sq = rsqrt_nr(zeta + eta);     // 1/sqrt(zeta + eta)
  const double inv = sq * sq;
  const double rho = zeta * eta * inv;
  const double xx = rho * (p.QP[0] * p.QP[0] + p.QP[1] * p.QP[1] + p.QP[2] * p.QP[2]);
  double u[NR], w[NR];
  if (rys_smem) RysSmem<NR>::eval(rys_smem, xx, u, w);
  else rys_eval<NR>(xx, u, w);
  const double scale = bcc * kcc * sq;
  const double r_z = eta * inv;     // rho / zeta
  const double r_e = zeta * inv;    // rho / eta
#pragma unroll
  for (int r = 0; r < NR; ++r) {
    const double t2 = u[r];
    const double t2_rz = t2 * r_z, t2_re = t2 * r_e;
    const T B10 = T((1.0 - t2_rz) * half_zinv);
    const T B01 = T((1.0 - t2_re) * half_einv);
    const T B00 = T(0.5 * t2 * inv);
    const T wt = T(w[r] * scale);
    T I[3][D1][D2];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      const T c00 = T(p.PA[d] + t2_rz * p.QP[d]);
      const T d00 = T(p.QC[d] - t2_re * p.QP[d]);
      I[d][0][0] = (d == 2) ? wt : T(1);
      if (D1 > 1) I[d][1][0] = c00 * I[d][0][0];
#pragma unroll
      for (int e = 1; e + 1 < D1; ++e) I[d][e + 1][0] = c00 * I[d][e][0] + T(e) * B10 * I[d][e - 1][0];
#pragma unroll
      for (int f = 0; f + 1 < D2; ++f) {
#pragma unroll
        for (int e = 0; e < D1; ++e) {
          T v = d00 * I[d][e][f];
          if (f > 0) v += T(f) * B01 * I[d][e][f - 1];
          if (e > 0) v += T(e) * B00 * I[d][e - 1][f];
          I[d][e][f + 1] = v;
        }
      }
    }
    static_for<Q::NE>([&](auto e) {
      constexpr int ge = Q::FE + decltype(e)::value;
      static_for<Q::NF>([&](auto f) {
        constexpr int gf = Q::FF + decltype(f)::value;
        esfs[decltype(e)::value][decltype(f)::value] +=
            I[0][gx(ge)][gx(gf)] * I[1][gy(ge)][gy(gf)] * I[2][gz(ge)][gz(gf)];
      });
    });
  }
}
}

// One flat loop over the nbp x nkp primitive quartets: lanes with the same count but
// different (nbp, nkp) splits stay converged.  Kets are the outer index and bras the
// inner one: the lanes of a warp share the bra pair (bra-major lists), so the
// per-iteration bra loads are warp-wide broadcasts and each lane's ket record is
// read once per ket primitive, one iteration ahead.  (Two primitive quartets per
// iteration as independent chains measured no faster on (H2O)32.)
// p0, npq: the share of the quartet's nbp x nkp primitive quartets to add up (flat
// indices p0 .. p0 + npq - 1, p = ket * nbp + bra): all of them, or one lane's part where
// several lanes share a quartet.
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ void accumulate_esfs(const PrimPair* __restrict__ bp, int nbp,
                                                const PrimPair* __restrict__ kp, int nkp, int p0, int npq,
                                                const QuartetGeom& g,
                                                T (&esfs)[Quartet<LA, LB, LC, LD>::NE][Quartet<LA, LB, LC, LD>::NF],
                                                const double* __restrict__ rys_smem = nullptr) {
  using Q = Quartet<LA, LB, LC, LD>;
#pragma unroll
  for (int e = 0; e < Q::NE; ++e)
#pragma unroll
    for (int f = 0; f < Q::NF; ++f) esfs[e][f] = T(0);
  if (npq <= 0) return;
  int ik = p0 ? p0 / nbp : 0, ib = p0 - ik * nbp;
  // (the one-root classes, at 20 resident warps, have no registers for it)
  constexpr bool KEEP = Q::LAB + Q::LCD >= 2;
  PrimRegs k = load_prim(kp, ik);
  KetPos q = ket_pos(k, g);
#pragma unroll(kPrimUnroll)
  for (int p = 0; p < npq; ++p) {
    const PrimRegs b = load_prim(bp, ib);
    const bool last = ++ib == nbp;             // the ket's last bra: its successor is loaded meanwhile
    PrimRegs kc = k;
    if (last) {
      ib = 0;
      ++ik;
      if (ik < nkp) kc = load_prim(kp, ik);
    }
    prim_quartet<LA, LB, LC, LD, T>(b, k, KEEP ? q : ket_pos(k, g), g, esfs, rys_smem);
    if (last) {
      k = kc;
      if (KEEP) q = ket_pos(k, g);
    }
  }
}

// Horizontal transfer on the ket: esfs[e][f] (f over l in [LC, LC+LD]) ->
// out[e][c][d], (c, d+1_i) = (c+1_i, d) + R_i (c, d), R = C - D.
// Level k holds d over comps(k) and c over l in [LC, LC+LD-k].
template <int LC, int LD, int NE, typename T>
__device__ __forceinline__ void hrr_ket(const T (&G)[NE][CT.first[LC + LD + 1] - CT.first[LC]], const double* R,
                                        T (&out)[NE][ncart(LC)][ncart(LD)]) {
  if constexpr (LD == 0) {
#pragma unroll
    for (int e = 0; e < NE; ++e)
#pragma unroll
      for (int c = 0; c < ncart(LC); ++c) out[e][c][0] = G[e][c];
  } else {
    // level tables: lev[k][c_global_offset][d], c over l in [LC, LC+LD-k]
    constexpr int NCR = CT.first[LC + LD + 1] - CT.first[LC];
    T cur[NE][NCR][ncart(LD)];
#pragma unroll
    for (int e = 0; e < NE; ++e)
#pragma unroll
      for (int c = 0; c < NCR; ++c) cur[e][c][0] = G[e][c];
    static_for<LD>([&](auto kk) {
      constexpr int k = decltype(kk)::value;           // building d level k+1
      constexpr int NCN = CT.first[LC + LD - k] - CT.first[LC];
      T nxt[NE][NCN > 0 ? NCN : 1][ncart(k + 1)];
      static_for<ncart(k + 1)>([&](auto dd) {
        constexpr int d1 = decltype(dd)::value;
        constexpr int px = cx(k + 1, d1), py = cy(k + 1, d1), pz = cz(k + 1, d1);
        constexpr int dir = px > 0 ? 0 : (py > 0 ? 1 : 2);
        constexpr int d0 = CT.idx[px - (dir == 0)][py - (dir == 1)][pz - (dir == 2)];
        static_for<NCN>([&](auto ci) {
          constexpr int c = decltype(ci)::value;
          constexpr int g = CT.first[LC] + c;
          constexpr int gp = gidx(gx(g) + (dir == 0), gy(g) + (dir == 1), gz(g) + (dir == 2)) - CT.first[LC];
#pragma unroll
          for (int e = 0; e < NE; ++e) nxt[e][c][d1] = cur[e][gp][d0] + T(R[dir]) * cur[e][c][d0];
        });
      });
#pragma unroll
      for (int e = 0; e < NE; ++e)
#pragma unroll
        for (int c = 0; c < NCN; ++c)
#pragma unroll
          for (int d = 0; d < ncart(k + 1); ++d) cur[e][c][d] = nxt[e][c][d];
    });
#pragma unroll
    for (int e = 0; e < NE; ++e)
#pragma unroll
      for (int c = 0; c < ncart(LC); ++c)
#pragma unroll
        for (int d = 0; d < ncart(LD); ++d) out[e][c][d] = cur[e][c][d];
  }
}

// Horizontal transfer on the bra: G[e][r] (e over l in [LA, LA+LB]) ->
// out[a][b][r] with R = A - B.
template <int LA, int LB, int NR, typename T>
__device__ __forceinline__ void hrr_bra(const T (&G)[CT.first[LA + LB + 1] - CT.first[LA]][NR], const double* R,
                                        T (&out)[ncart(LA)][ncart(LB)][NR]) {
  if constexpr (LB == 0) {
#pragma unroll
    for (int a = 0; a < ncart(LA); ++a)
#pragma unroll
      for (int r = 0; r < NR; ++r) out[a][0][r] = G[a][r];
  } else {
    constexpr int NAR = CT.first[LA + LB + 1] - CT.first[LA];
    T cur[NAR][ncart(LB)][NR];
#pragma unroll
    for (int a = 0; a < NAR; ++a)
#pragma unroll
      for (int r = 0; r < NR; ++r) cur[a][0][r] = G[a][r];
    static_for<LB>([&](auto kk) {
      constexpr int k = decltype(kk)::value;
      constexpr int NAN_ = CT.first[LA + LB - k] - CT.first[LA];
      T nxt[NAN_ > 0 ? NAN_ : 1][ncart(k + 1)][NR];
      static_for<ncart(k + 1)>([&](auto bb) {
        constexpr int b1 = decltype(bb)::value;
        constexpr int px = cx(k + 1, b1), py = cy(k + 1, b1), pz = cz(k + 1, b1);
        constexpr int dir = px > 0 ? 0 : (py > 0 ? 1 : 2);
        constexpr int b0 = CT.idx[px - (dir == 0)][py - (dir == 1)][pz - (dir == 2)];
        static_for<NAN_>([&](auto ai) {
          constexpr int a = decltype(ai)::value;
          constexpr int g = CT.first[LA] + a;
          constexpr int gp = gidx(gx(g) + (dir == 0), gy(g) + (dir == 1), gz(g) + (dir == 2)) - CT.first[LA];
#pragma unroll
          for (int r = 0; r < NR; ++r) nxt[a][b1][r] = cur[gp][b0][r] + T(R[dir]) * cur[a][b0][r];
        });
      });
#pragma unroll
      for (int a = 0; a < NAN_; ++a)
#pragma unroll
        for (int b = 0; b < ncart(k + 1); ++b)
#pragma unroll
          for (int r = 0; r < NR; ++r) cur[a][b][r] = nxt[a][b][r];
    });
#pragma unroll
    for (int a = 0; a < ncart(LA); ++a)
#pragma unroll
      for (int b = 0; b < ncart(LB); ++b)
#pragma unroll
        for (int r = 0; r < NR; ++r) out[a][b][r] = cur[a][b][r];
  }
}

// (e0|f0) of a bra family: the primitive loop runs once over the positioned
// primitive pairs the members share (bp, the first member's), each primitive
// quartet evaluated with a unit bra coefficient and added into every member's block
// with that member's coefficient product (bm[m][ib].cc; bm[m] null: no member m).
template <int LA, int LB, int LC, int LD, typename T, int MB>
__device__ __forceinline__ void accumulate_esfs_fam(const PrimPair* __restrict__ bp, int nbp,
                                                    const PrimPair* __restrict__ kp, int nkp, int p0, int npq,
                                                    const QuartetGeom& g,
                                                    const PrimPair* const (&bm)[MB],
                                                    T (&esfs)[MB][Quartet<LA, LB, LC, LD>::NE][Quartet<LA, LB, LC, LD>::NF],
                                                    const double* __restrict__ rys_smem) {
  using Q = Quartet<LA, LB, LC, LD>;
#pragma unroll
  for (int m = 0; m < MB; ++m)
#pragma unroll
    for (int e = 0; e < Q::NE; ++e)
#pragma unroll
      for (int f = 0; f < Q::NF; ++f) esfs[m][e][f] = T(0);
  if (npq <= 0) return;
  int ik = p0 ? p0 / nbp : 0, ib = p0 - ik * nbp;
  // (the one-root classes, at 20 resident warps, have no registers for it)
  constexpr bool KEEP = Q::LAB + Q::LCD >= 2;
  PrimRegs k = load_prim(kp, ik);
  KetPos q = ket_pos(k, g);
  for (int p = 0; p < npq; ++p) {
    PrimRegs b = load_prim(bp, ib);
    double cb[MB];
#pragma unroll
    for (int m = 0; m < MB; ++m) cb[m] = bm[m] ? __ldg(&bm[m][ib].cc) : 0.0;
    b.y = 1.0;
    const bool last = ++ib == nbp;
    PrimRegs kc = k;
    if (last) {
      ib = 0;
      ++ik;
      if (ik < nkp) kc = load_prim(kp, ik);
    }
    T one[Q::NE][Q::NF];
#pragma unroll
    for (int e = 0; e < Q::NE; ++e)
#pragma unroll
      for (int f = 0; f < Q::NF; ++f) one[e][f] = T(0);
    prim_quartet<LA, LB, LC, LD, T>(b, k, KEEP ? q : ket_pos(k, g), g, one, rys_smem);
    if (last) {
      k = kc;
      if (KEEP) q = ket_pos(k, g);
    }
#pragma unroll
    for (int m = 0; m < MB; ++m) {
      const T w = T(cb[m]);
#pragma unroll
      for (int e = 0; e < Q::NE; ++e)
#pragma unroll
        for (int f = 0; f < Q::NF; ++f) esfs[m][e][f] += w * one[e][f];
    }
  }
}

// Horizontal transfers of one (e0|f0) block to the Cartesian (ab|cd), as double.
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ void hrr_quartet(const T (&esfs)[Quartet<LA, LB, LC, LD>::NE][Quartet<LA, LB, LC, LD>::NF],
                                            const double* Rab, const double* Rcd,
                                            double (&abcd)[ncart(LA)][ncart(LB)][ncart(LC) * ncart(LD)]) {
  using Q = Quartet<LA, LB, LC, LD>;
  double ed[Q::NE][Q::NF];
#pragma unroll
  for (int e = 0; e < Q::NE; ++e)
#pragma unroll
    for (int f = 0; f < Q::NF; ++f) ed[e][f] = (double)esfs[e][f];
  double ket[Q::NE][Q::NC][Q::ND];
  hrr_ket<LC, LD, Q::NE, double>(ed, Rcd, ket);
  double flat[Q::NE][Q::NC * Q::ND];
#pragma unroll
  for (int e = 0; e < Q::NE; ++e)
#pragma unroll
    for (int c = 0; c < Q::NC; ++c)
#pragma unroll
      for (int d = 0; d < Q::ND; ++d) flat[e][c * Q::ND + d] = ket[e][c][d];
  hrr_bra<LA, LB, Q::NC * Q::ND, double>(flat, Rab, abcd);
}

}  // namespace tf
