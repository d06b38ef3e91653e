// tf_thread.cuh — one thread per contracted quartet: the J/K kernels of the classes whose
// (e0|f0) block fits a thread's registers, their launch arguments and launches.  The
// classes are shared out over translation units (tf_jk_*.cu), which build in parallel.
#pragma once
#include "tf_device.cuh"
#include "tf_host.h"

#include <algorithm>

namespace tf {

constexpr int LMAX_SUPPORTED = 3;                 // s, p, d, f shells
constexpr int NPAIRCLS = (LMAX_SUPPORTED + 1) * (LMAX_SUPPORTED + 2) / 2;
constexpr int NQCLS = 625;                        // (la lb lc ld) counter slots, l <= 4
// Counters of a build, zeroed with it and read back after it: primitive quartets per
// class [0, NQCLS), the non-finite-density flag [NQCLS], contracted quartets per class
// of the FP64 buckets [NQCLS + 1, 2 NQCLS + 1) and of the FP32 buckets after them.
constexpr int BUILD_COUNTERS = 3 * NQCLS + 1;
__host__ __device__ constexpr int pair_class(int lh, int ll) { return lh * (lh + 1) / 2 + ll; }
__host__ __device__ constexpr int qclass_id(int la, int lb, int lc, int ld) { return ((la * 5 + lb) * 5 + lc) * 5 + ld; }
// Bra-family members the thread kernel of a class holds at once (accumulator
// capacity), for the classes that evaluate a bra family's primitive quartets once.
// Measured on (H2O)32 cc-pVDZ, one member per entry -> families: (ss|ss) 7.65 -> 7.21 ms,
// (ds|ss) 2.72 -> 2.84, the build 56.65 -> 56.43.  With capacity 2 (ps|ss), (ps|ps) and
// (ds|ps) are slower (10.2 -> 11.2, 6.4 -> 7.5 and 4.1 -> 6.1 ms: the extra accumulators
// cost registers, the coefficient loads and products every primitive quartet, and few of
// their bras are families), so they, like every other class, take one member per list
// entry (capacity 1).
__host__ __device__ constexpr int fam_cap_l(int la, int lb, int lc, int ld) {
  return (la == 0 && lb == 0 && lc == 0 && ld == 0) ? 4 : (la == 2 && lb == 0 && lc == 0 && ld == 0) ? 2 : 1;
}

// ---------------------------------------------------------------------------
// kernel: ERIs + digestion (one thread per contracted quartet)
// ---------------------------------------------------------------------------
struct JKArgs {
  const int2* quartets;
  long long n;
  const PrimPair* prim_full;
  const PrimPair* prim_skip;
  const double* P;              // Cartesian density (per-molecule blocks)
  double* J;                    // Cartesian accumulators
  double* K;
  const MolInfo* mols;
  unsigned long long* prim_count;   // per quartet class
  // the list's memory (quartets) starts at list entry base; a thread kernel reads its
  // entries from its plan, a lane-group kernel takes list[range[0] - base, range[1] - base)
  // (graph builds: read on the device and clamped to base + cap) or n entries from first
  const LaunchPlan* plan;
  const long long* range;
  long long base, cap, first;
  const int4* jkrec;            // packed pair records (load_pair_jk)
  const double4* xyz4;          // atom positions (load_pair_jk)
  // unrestricted builds: the beta density and its J, K (else null); P, J, K above
  // are then the alpha ones.  want: bit 0 J, bit 1 K.
  const double* P2;
  double* J2;
  double* K2;
  int want;
  // bra families (family groups): per list entry the members' mask, per pair its
  // family members; member quartets counted per class, FP64 buckets then FP32
  const unsigned char* qmask;
  const int4* fam_mem;
  unsigned long long* qcount;
  int fam;                      // bra-family capacity of the launch's kernel (1: none)
  int bucket32;                 // 1: the launch covers the FP32 buckets
  long long fx_lo;              // deterministic builds: offset of the lo words (fock_add), else 0
  long long expect;             // entries the launch will probably have (the lane-group kernels' choice)
};


#ifndef TF_JK_MINB_N1
#define TF_JK_MINB_N1 5
#endif
#ifndef TF_JK_MINB
#define TF_JK_MINB 1
#endif
// Resident warps per SM, in units of four (bounds the registers per thread).
// Variant 0 leaves the registers to the compiler (one-root classes: 20 warps);
// variant 1 asks for more resident warps (24 for one root, 16 otherwise), at the
// price of fewer registers.  The autotuner times the variants per class.
template <int LA, int LB, int LC, int LD, int V>
constexpr int jk_min_blocks() {
  return Quartet<LA, LB, LC, LD>::NROOT == 1 ? ((V & 1) ? 6 : TF_JK_MINB_N1) : ((V & 1) ? 4 : TF_JK_MINB);
}
// Variant bits: 1 = more resident warps (see above); 2 = K atomics of lanes that hit
// the same element summed first (segmented warp sums over lanes of one bra); 4 =
// deterministic accumulation (fock_add), set by the context, not by the autotuner.
constexpr int JK_VARIANTS = 4;
// Threads per block: the resident warps of an SM form one block, so the SM holds
// one copy of the shared Rys/Boys grid and leaves the rest of its shared storage to
// the L1 cache, which serves the bra primitive records every iteration re-reads
// (measured on (H2O)32, (ps|ss): L1 hit rate 42% -> 62%, 14.8 -> 13.7 ms against
// five blocks of 128 threads).  A variant with no register bound uses up to 255
// registers: 256 threads per SM.
template <int LA, int LB, int LC, int LD, int V>
constexpr int jk_threads() {
  return jk_min_blocks<LA, LB, LC, LD, V>() == 1 ? 256 : 128 * jk_min_blocks<LA, LB, LC, LD, V>();
}

// N consecutive doubles of a density row at a shell's first column: p, d and f shells start
// on 32-byte boundaries and are padded to whole words (the context's Cartesian order).
template <int N>
__device__ __forceinline__ void load_row(const double* __restrict__ p, double (&v)[N]) {
  if constexpr (N == 1) {
    v[0] = __ldg(p);
  } else {
#pragma unroll
    for (int i = 0; i < N; i += 4) {
      const double4 x = ldg256(p + i);
      v[i] = x.x;
      if (i + 1 < N) v[i + 1] = x.y;
      if (i + 2 < N) v[i + 2] = x.z;
      if (i + 3 < N) v[i + 3] = x.w;
    }
  }
}

// Block (x, y) of the (symmetric) density, shells of NX and NY components at ox and oy,
// read along the wider one: a gather touches a sector per lane and row, whatever of
// its 32 bytes is used.
template <int NX, int NY>
__device__ __forceinline__ void load_block(const double* __restrict__ P, int n, int ox, int oy, double (&v)[NX][NY]) {
  if constexpr (NY >= NX) {
#pragma unroll
    for (int x = 0; x < NX; ++x) load_row<NY>(P + (size_t)(ox + x) * n + oy, v[x]);
  } else {
#pragma unroll
    for (int y = 0; y < NY; ++y) {
      double r[NX];
      load_row<NX>(P + (size_t)(oy + y) * n + ox, r);
#pragma unroll
      for (int x = 0; x < NX; ++x) v[x][y] = r[x];
    }
  }
}

// Sums of N <= 32 values over the warp: at each of the five steps a lane keeps half of its
// values and gets its partner's sums of those, so that about N + 5 exchanges do the work of
// 5 N.  On return v[0] is the warp's sum of value e, the returned index (N or more: none).
template <int N>
__device__ __forceinline__ int warp_sums(double (&v)[N]) {
  static_assert(N >= 1 && N <= 32, "at most a value per lane");
  const int lane = threadIdx.x & 31;
  int e = 0;
  static_for<5>([&](auto ss) {
    constexpr int st = decltype(ss)::value, o = 16 >> st;
    constexpr int P2 = N <= 1 ? 1 : N <= 2 ? 2 : N <= 4 ? 4 : N <= 8 ? 8 : N <= 16 ? 16 : 32;
    constexpr int held = (P2 >> st) > 1 ? (P2 >> st) : 1;
    constexpr int valid = held < N ? held : N;               // held values that exist in some lane
    const bool up = lane & o;
    if constexpr (held > 1) {
      constexpr int h = held / 2;
#pragma unroll
      for (int i = 0; i < h; ++i) {
        const double lo = i < valid ? v[i] : 0.0, hi = i + h < valid ? v[i + h < N ? i + h : 0] : 0.0;
        const double got = __shfl_xor_sync(0xffffffffu, up ? lo : hi, o);
        if (i < N) v[i] = (up ? hi : lo) + got;
      }
      if (up) e += h;
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  });
  // lanes that took part in the last, unsplit steps hold the same sum: one of them adds it
  constexpr int P2 = N <= 1 ? 1 : N <= 2 ? 2 : N <= 4 ? 4 : N <= 8 ? 8 : N <= 16 ? 16 : 32;
  return (lane & (32 / P2 - 1)) == 0 ? e : 32;
}

// Digestion of one quartet's Cartesian integrals I into J and K with the coincidence
// factor f (f = 0: the lane adds nothing but still takes part in the warp sums):
// bid is the bra pair (lanes of one bra are summed together), ob/oa the bra's and
// oc/od the ket's first Cartesian functions.
//   J(ab) += f sum_cd I P(cd);  J(cd) += f sum_ab I P(ab)  (per spin when unrestricted)
//   K(ac) += f sum_bd I P(bd);  K(ad) += f sum_bc I P(bc)
//   K(bc) += f sum_ad I P(ad);  K(bd) += f sum_ac I P(ac)
// The lists are bra-major, so the lanes of a warp usually share the bra pair: then
// J(ab) is summed over the warp and added once, and P(ab) is a broadcast.  Otherwise
// the lanes of one bra are neighbours (a bra's kets of one cost bucket are
// consecutive) and J(ab) is summed over each run of equal bras by a segmented warp
// scan, then added by the run's last lane.  Variant bit 2: the K rows a and b are the
// same for all lanes of one bra, and lanes whose kets share the c (or d) shell add to
// the same K elements; such lanes are neighbours (pair-id order), so each run of
// equal (bra, shell) keys is summed with a segmented warp scan and added once, by its
// last lane.  K(bc), K(bd) are summed over a's components in registers first.
template <int LA, int LB, int LC, int LD, int V>
__device__ __forceinline__ void digest_jk(const JKArgs& a, const MolInfo& mi,
                                          const double (&I)[ncart(LA)][ncart(LB)][ncart(LC) * ncart(LD)], double f,
                                          int bid, int oa, int ob, int oc, int od) {
  using Q = Quartet<LA, LB, LC, LD>;
  constexpr bool FX = (V & 4) != 0;
  const int lane = threadIdx.x & 31;
  const bool live = f != 0.0;
  const int n = mi.n_cart;
  const bool uni = __all_sync(0xffffffffu, bid == __shfl_sync(0xffffffffu, bid, 0));
  const unsigned lt_mask = lane == 31 ? 0xffffffffu : ((2u << lane) - 1u);
  // (every lane executes the shuffle: none may be skipped by a short-circuit)
  const int upx = __shfl_up_sync(0xffffffffu, bid, 1);
  const bool headx = lane == 0 || bid != upx;
  const unsigned heada = __ballot_sync(0xffffffffu, headx);
  const int sega = 31 - __clz(heada & lt_mask);
  const bool taila = lane == 31 || ((heada >> (lane + 1)) & 1u);
  auto digest_j = [&](const double* __restrict__ P, double* __restrict__ Jm) {
    double Pcd[Q::NC][Q::ND];
    load_block<Q::NC, Q::ND>(P, n, oc, od, Pcd);
    double Jab[Q::NA * Q::NB];
#pragma unroll
    for (int ia = 0; ia < Q::NA; ++ia)
#pragma unroll
      for (int ib = 0; ib < Q::NB; ++ib) {
        double s = 0.0;
#pragma unroll
        for (int c = 0; c < Q::NC; ++c)
#pragma unroll
          for (int d = 0; d < Q::ND; ++d) s += I[ia][ib][c * Q::ND + d] * Pcd[c][d];
        Jab[ia * Q::NB + ib] = s * f;
      }
    if (uni) {
      static_for<(Q::NA * Q::NB + 31) / 32>([&](auto cc) {
        constexpr int e0 = 32 * decltype(cc)::value, m = Q::NA * Q::NB - e0 < 32 ? Q::NA * Q::NB - e0 : 32;
        double v[m];
#pragma unroll
        for (int i = 0; i < m; ++i) v[i] = Jab[e0 + i];
        const int i = warp_sums<m>(v), e = e0 + i;
        if (i < m && v[0] != 0.0) fock_add<FX>(Jm + (size_t)(oa + e / Q::NB) * n + ob + e % Q::NB, v[0], a.fx_lo);
      });
    } else {                           // idle lanes join the last run with s = 0
#pragma unroll
      for (int e = 0; e < Q::NA * Q::NB; ++e) {
        double s = Jab[e];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const double t = __shfl_up_sync(0xffffffffu, s, o);
          if (lane - o >= sega) s += t;
        }
        if (taila && s != 0.0) fock_add<FX>(Jm + (size_t)(oa + e / Q::NB) * n + ob + e % Q::NB, s, a.fx_lo);
      }
    }
    if (live) {
      double Pab[Q::NA][Q::NB];
      load_block<Q::NA, Q::NB>(P, n, oa, ob, Pab);
#pragma unroll
      for (int c = 0; c < Q::NC; ++c)
#pragma unroll
        for (int d = 0; d < Q::ND; ++d) {
          double s = 0.0;
#pragma unroll
          for (int ia = 0; ia < Q::NA; ++ia)
#pragma unroll
            for (int ib = 0; ib < Q::NB; ++ib) s += I[ia][ib][c * Q::ND + d] * Pab[ia][ib];
          fock_add<FX>(Jm + (size_t)(oc + c) * n + od + d, f * s, a.fx_lo);
        }
    }
  };
  if (a.want & 1) {                    // uniform over the warp (the J(ab) sums shuffle)
    digest_j(a.P + mi.cmat, a.J + mi.cmat);
    if (a.P2) digest_j(a.P2 + mi.cmat, a.J2 + mi.cmat);
  }
  constexpr bool SEG = (V & 2) != 0;
  int segc = lane, segd = lane;
  bool tailc = true, taild = true;
  if constexpr (SEG) {
    // (every lane executes both shuffles: none may be skipped by a short-circuit)
    const int upc = __shfl_up_sync(0xffffffffu, oc, 1), upd = __shfl_up_sync(0xffffffffu, od, 1);
    const unsigned headc = __ballot_sync(0xffffffffu, headx || oc != upc);
    const unsigned headd = __ballot_sync(0xffffffffu, headx || od != upd);
    segc = 31 - __clz(headc & lt_mask);
    segd = 31 - __clz(headd & lt_mask);
    tailc = lane == 31 || ((headc >> (lane + 1)) & 1u);
    taild = lane == 31 || ((headd >> (lane + 1)) & 1u);
  }
  auto kadd = [&](double* addr, double v, int seg, bool tail) {
    if constexpr (SEG) {
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const double t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane - o >= seg) v += t;
      }
      if (tail && v != 0.0) fock_add<FX>(addr, v, a.fx_lo);
    } else {
      fock_add<FX>(addr, v, a.fx_lo);
    }
  };
#define TF_KADD_C(addr, v) kadd((addr), (v), segc, tailc)
#define TF_KADD_D(addr, v) kadd((addr), (v), segd, taild)
  auto digest_k = [&](const double* __restrict__ P, double* __restrict__ Km) {
    double Pbd[Q::NB][Q::ND], Pbc[Q::NB][Q::NC];
    double Kbc[Q::NB][Q::NC], Kbd[Q::NB][Q::ND];
#pragma unroll
    for (int ib = 0; ib < Q::NB; ++ib) {
#pragma unroll
      for (int c = 0; c < Q::NC; ++c) Kbc[ib][c] = 0.0;
#pragma unroll
      for (int d = 0; d < Q::ND; ++d) Kbd[ib][d] = 0.0;
    }
    load_block<Q::NB, Q::ND>(P, n, ob, od, Pbd);
    load_block<Q::NB, Q::NC>(P, n, ob, oc, Pbc);
    // (a, c) and (a, d): whole blocks when read along a, else row by row with a
    constexpr bool ALONG_A_D = Q::NA > Q::ND, ALONG_A_C = Q::NA > Q::NC;
    double PadA[ALONG_A_D ? Q::NA : 1][Q::ND], PacA[ALONG_A_C ? Q::NA : 1][Q::NC];
    if constexpr (ALONG_A_D) load_block<Q::NA, Q::ND>(P, n, oa, od, PadA);
    if constexpr (ALONG_A_C) load_block<Q::NA, Q::NC>(P, n, oa, oc, PacA);
#pragma unroll
    for (int ia = 0; ia < Q::NA; ++ia) {
      double Pad[Q::ND], Pac[Q::NC];
      if constexpr (ALONG_A_D) {
#pragma unroll
        for (int d = 0; d < Q::ND; ++d) Pad[d] = PadA[ia][d];
      } else {
        load_row<Q::ND>(P + (size_t)(oa + ia) * n + od, Pad);
      }
      if constexpr (ALONG_A_C) {
#pragma unroll
        for (int c = 0; c < Q::NC; ++c) Pac[c] = PacA[ia][c];
      } else {
        load_row<Q::NC>(P + (size_t)(oa + ia) * n + oc, Pac);
      }
#pragma unroll
      for (int c = 0; c < Q::NC; ++c) {
        double s = 0.0;
#pragma unroll
        for (int ib = 0; ib < Q::NB; ++ib)
#pragma unroll
          for (int d = 0; d < Q::ND; ++d) s += I[ia][ib][c * Q::ND + d] * Pbd[ib][d];
        TF_KADD_C(Km + (size_t)(oa + ia) * n + oc + c, f * s);
      }
#pragma unroll
      for (int d = 0; d < Q::ND; ++d) {
        double s = 0.0;
#pragma unroll
        for (int ib = 0; ib < Q::NB; ++ib)
#pragma unroll
          for (int c = 0; c < Q::NC; ++c) s += I[ia][ib][c * Q::ND + d] * Pbc[ib][c];
        TF_KADD_D(Km + (size_t)(oa + ia) * n + od + d, f * s);
      }
#pragma unroll
      for (int ib = 0; ib < Q::NB; ++ib) {
#pragma unroll
        for (int c = 0; c < Q::NC; ++c)
#pragma unroll
          for (int d = 0; d < Q::ND; ++d) Kbc[ib][c] += I[ia][ib][c * Q::ND + d] * Pad[d];
#pragma unroll
        for (int d = 0; d < Q::ND; ++d)
#pragma unroll
          for (int c = 0; c < Q::NC; ++c) Kbd[ib][d] += I[ia][ib][c * Q::ND + d] * Pac[c];
      }
    }
    // K(bc), K(bd): summed over the a components first, one atomic per element
#pragma unroll
    for (int ib = 0; ib < Q::NB; ++ib) {
#pragma unroll
      for (int c = 0; c < Q::NC; ++c) TF_KADD_C(Km + (size_t)(ob + ib) * n + oc + c, f * Kbc[ib][c]);
#pragma unroll
      for (int d = 0; d < Q::ND; ++d) TF_KADD_D(Km + (size_t)(ob + ib) * n + od + d, f * Kbd[ib][d]);
    }
  };
  // with segmented sums every lane takes part (idle lanes add f = 0)
  if ((SEG || live) && (a.want & 2)) {
    digest_k(a.P + mi.cmat, a.K + mi.cmat);
    if (a.P2) digest_k(a.P2 + mi.cmat, a.K2 + mi.cmat);
  }
#undef TF_KADD_C
#undef TF_KADD_D
}

// Per-class counters of a launch, summed over the warp: primitive quartets, and
// contracted (member) quartets of the FP64 or the FP32 buckets.
__device__ __forceinline__ void count_quartets(const JKArgs& a, int cls, unsigned long long nprim,
                                               unsigned long long nq) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    nprim += __shfl_xor_sync(0xffffffffu, nprim, o);
    nq += __shfl_xor_sync(0xffffffffu, nq, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (nprim) atomicAdd(a.prim_count + cls, nprim);
    if (nq) atomicAdd(a.qcount + (a.bucket32 ? NQCLS : 0) + cls, nq);
  }
}

// One thread per contracted quartet, or, in the buckets whose quartets have so many
// primitive quartets that they would outlast the rest of the launch, 2, 4, .. 32
// neighbouring lanes (LaunchPlan): each adds up a share, the shares are summed by
// shuffles and one lane digests.  MB = 1: a list entry is one quartet.  MB > 1
// (family groups): a list entry is a bra family (its first member's pair id) with a
// ket, and the mask of the members whose quartet passed the screen; the primitive
// loop runs once for all members (accumulate_esfs_fam), then each member quartet of
// the mask is transferred and digested with its own Cartesian offsets and
// coincidence factors (molecule.fock.foo:1296-1300).
template <int LA, int LB, int LC, int LD, typename T, int V, int MB>
__global__ void __launch_bounds__(jk_threads<LA, LB, LC, LD, V>(), 1) k_jk(JKArgs a) {
  using Q = Quartet<LA, LB, LC, LD>;
  using RS = RootTable<LA, LB, LC, LD, T>;
  extern __shared__ double rys_tab[];
  __shared__ LaunchPlan plan;
  const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
  const long long n_warps = a.plan->warp0[NCOST], stride = (long long)gridDim.x * (blockDim.x >> 5);
  // a long list: the warps of an SM take neighbouring entries (one bra's records serve them
  // all from L1); a short one is spread over the SMs
  const bool spread = n_warps < 4 * stride;
  if ((spread ? (long long)blockIdx.x : (long long)blockIdx.x * (blockDim.x >> 5)) >= n_warps) return;
  for (int q = threadIdx.x; q < (int)(sizeof(LaunchPlan) / sizeof(int)); q += blockDim.x)
    reinterpret_cast<int*>(&plan)[q] = __ldg(reinterpret_cast<const int*>(a.plan) + q);
  RS::load(rys_tab);
  __syncthreads();
  unsigned long long nprim = 0, nquart = 0;
  int seg = 0;
  for (long long w = spread ? (long long)wib * gridDim.x + blockIdx.x : (long long)blockIdx.x * (blockDim.x >> 5) + wib;
       w < n_warps; w += stride) {
    while (w >= plan.warp0[seg + 1]) ++seg;
    const int lg = plan.lg[seg], sub = lane & ((1 << lg) - 1);
    const long long at = (w - plan.warp0[seg]) * (32 >> lg) + (lane >> lg);
    // lanes past the end repeat the bucket's last entry with weight 0, so that whole warps
    // take part in the warp reductions below
    const bool in_list = at < plan.count[seg];
    const bool active = in_list && sub == 0;          // the lane that digests and counts the entry
    const long long te = plan.item0[seg] + (in_list ? at : plan.count[seg] - 1) - a.base;
    const int2 qd = a.quartets[te];
    const PairJK b = load_pair_jk(a.jkrec, a.xyz4, qd.x);
    const PairJK k = load_pair_jk(a.jkrec, a.xyz4, qd.y);
    const bool any_same = b.atom_hi == b.atom_lo || k.atom_hi == k.atom_lo || b.atom_hi == k.atom_hi ||
                          b.atom_hi == k.atom_lo || b.atom_lo == k.atom_hi || b.atom_lo == k.atom_lo;
    const PrimPair* bp = any_same ? a.prim_full + b.full_off : a.prim_skip + b.skip_off;
    const PrimPair* kp = any_same ? a.prim_full + k.full_off : a.prim_skip + k.skip_off;
    const int nbp = any_same ? b.n_full : b.n_skip;
    const int nkp = any_same ? k.n_full : k.n_skip;
    const QuartetGeom geom = quartet_geom(b, k);
    // this lane's share of the primitive quartets
    const int npq = nbp * nkp;
    const int p0 = lg ? (int)((long long)npq * sub >> lg) : 0;
    const int np = lg ? (int)((long long)npq * (sub + 1) >> lg) - p0 : npq;
    const MolInfo mi = a.mols[b.mol];
    double fk = 1.0;
    if (k.same) fk *= 0.5;
    if constexpr (MB == 1) {
      if (active) { nprim += (unsigned long long)nbp * nkp; nquart += 1; }
      double f = active ? fk : 0.0;
      if (b.same) f *= 0.5;
      if (qd.x == qd.y) f *= 0.5;
      double I[Q::NA][Q::NB][Q::NC * Q::ND];
      T esfs[Q::NE][Q::NF];
      accumulate_esfs<LA, LB, LC, LD, T>(bp, nbp, kp, nkp, p0, np, geom, esfs, rys_tab);
      for (int o = 1; o < 1 << lg; o <<= 1)
#pragma unroll
        for (int e = 0; e < Q::NE; ++e)
#pragma unroll
          for (int q = 0; q < Q::NF; ++q) esfs[e][q] += __shfl_xor_sync(0xffffffffu, esfs[e][q], o);
      hrr_quartet<LA, LB, LC, LD, T>(esfs, geom.Rab, geom.Rcd, I);
      digest_jk<LA, LB, LC, LD, V>(a, mi, I, f, qd.x, b.cart_hi, b.cart_lo, k.cart_hi, k.cart_lo);
    } else {
      const unsigned mask = active ? a.qmask[te] : 0u;
      nprim += (unsigned long long)nbp * nkp * __popc(mask);
      nquart += __popc(mask);
      const int4 mv = a.fam_mem[qd.x];
      const int mid[4] = {mv.x, mv.y, mv.z, mv.w};
      PairJK bm[MB];
      const PrimPair* bmp[MB];
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        bm[m] = load_pair_jk(a.jkrec, a.xyz4, mid[m] >= 0 ? mid[m] : qd.x);
        bmp[m] = mid[m] < 0 ? nullptr : (any_same ? a.prim_full + bm[m].full_off : a.prim_skip + bm[m].skip_off);
      }
      T esfs[MB][Q::NE][Q::NF];
      accumulate_esfs_fam<LA, LB, LC, LD, T, MB>(bp, nbp, kp, nkp, p0, np, geom, bmp, esfs, rys_tab);
      for (int o = 1; o < 1 << lg; o <<= 1)
#pragma unroll
        for (int m = 0; m < MB; ++m)
#pragma unroll
          for (int e = 0; e < Q::NE; ++e)
#pragma unroll
            for (int q = 0; q < Q::NF; ++q) esfs[m][e][q] += __shfl_xor_sync(0xffffffffu, esfs[m][e][q], o);
#pragma unroll
      for (int m = 0; m < MB; ++m) {
        if (!__any_sync(0xffffffffu, (mask >> m) & 1u)) continue;      // uniform over the warp
        double f = ((mask >> m) & 1u) ? fk : 0.0;
        if (bm[m].same) f *= 0.5;
        if (mid[m] == qd.y) f *= 0.5;
        double I[Q::NA][Q::NB][Q::NC * Q::ND];
        hrr_quartet<LA, LB, LC, LD, T>(esfs[m], geom.Rab, geom.Rcd, I);
        digest_jk<LA, LB, LC, LD, V>(a, mi, I, f, mid[m] >= 0 ? mid[m] : qd.x, bm[m].cart_hi, bm[m].cart_lo,
                                     k.cart_hi, k.cart_lo);
      }
    }
  }
  count_quartets(a, qclass_id(LA, LB, LC, LD), nprim, nquart);
}

// Launch set-up (shared-memory attribute, resident blocks of the GPU), done once per
// kernel and device and before any graph capture: a JKArgs without a plan only sets up.
// false: the set-up failed.
template <int LA, int LB, int LC, int LD, typename T, int V, int MB>
static bool launch_jk_t(const JKArgs& a, cudaStream_t s) {
  constexpr int thr = jk_threads<LA, LB, LC, LD, V>();
  constexpr size_t smem = RootTable<LA, LB, LC, LD, T>::SIZE * sizeof(double);
  static PerDevice<long long> resident;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return false;
  long long full = 0;
  const bool ready = resident.get(dev, full, [&](long long& blocks) {
    auto* const kernel = k_jk<LA, LB, LC, LD, T, V, MB>;
    int nsm = 0, per_sm = 0, nb = 0;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess)
      return false;
    // shared storage for one block, the rest to L1
    const int pct = per_sm > 0 ? std::min(100, (int)((smem + 2048) * 100 / per_sm) + 1) : 100;
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, pct) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, kernel, thr, smem) != cudaSuccess)
      return false;
    blocks = (long long)nsm * std::max(nb, 1);
    return true;
  });
  if (!ready) return false;
  if (!a.plan) return true;
  // (n known: at most a warp an entry)
  const long long blocks = a.range ? full : std::min<long long>((a.n * 32 + thr - 1) / thr, full);
  k_jk<LA, LB, LC, LD, T, V, MB><<<(unsigned)blocks, thr, smem, s>>>(a);
  return true;
}

template <int LA, int LB, int LC, int LD, int V, int MB>
static bool launch_jk_v(const JKArgs& a, cudaStream_t s, bool fp32) {
  return fp32 ? launch_jk_t<LA, LB, LC, LD, float, V, MB>(a, s) : launch_jk_t<LA, LB, LC, LD, double, V, MB>(a, s);
}

template <int LA, int LB, int LC, int LD, int MB>
static bool launch_jk_m(const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  switch (variant & 7) {
    case 1: return launch_jk_v<LA, LB, LC, LD, 1, MB>(a, s, fp32);
    case 2: return launch_jk_v<LA, LB, LC, LD, 2, MB>(a, s, fp32);
    case 3: return launch_jk_v<LA, LB, LC, LD, 3, MB>(a, s, fp32);
    case 4: case 6: return launch_jk_v<LA, LB, LC, LD, 6, MB>(a, s, fp32);   // deterministic: always bit 2
    case 5: case 7: return launch_jk_v<LA, LB, LC, LD, 7, MB>(a, s, fp32);
    default: return launch_jk_v<LA, LB, LC, LD, 0, MB>(a, s, fp32);
  }
}

// The bra-family kernel of the class (fam_cap_l) when the launch is a family group.
template <int LA, int LB, int LC, int LD>
static bool launch_jk(const JKArgs& a, cudaStream_t s, bool fp32, int variant) {
  constexpr int CAP = fam_cap_l(LA, LB, LC, LD);
  if constexpr (CAP > 1) {
    if (a.fam > 1) return launch_jk_m<LA, LB, LC, LD, CAP>(a, s, fp32, variant);
  }
  return launch_jk_m<LA, LB, LC, LD, 1>(a, s, fp32, variant);
}

// Classes whose (e0|f0) block and integrals do not fit a thread's registers: FP64 for the
// FP32 buckets too, and the two instantiations that differ in their results' bits only
// (deterministic or not; a register-bounded variant would spill more).
template <int LA, int LB, int LC, int LD>
static bool launch_jk_f64(const JKArgs& a, cudaStream_t s, bool, int variant) {
  return variant & 4 ? launch_jk_t<LA, LB, LC, LD, double, 6, 1>(a, s) : launch_jk_t<LA, LB, LC, LD, double, 0, 1>(a, s);
}

// The classes of one translation unit each (tf_jk_*.cu); 1: launched, 0: not a class of
// that unit, -1: the launch could not be set up.
int launch_jk_ss(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant);
int launch_jk_ps(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant);
int launch_jk_d(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant);
int launch_jk_l(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant);
int launch_jk_l2(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant);
int launch_jk_f(int key, const JKArgs& a, cudaStream_t s, bool fp32, int variant);

#define TF_JK_CASE(LAUNCH, A, B, C, D) \
  case class_key(A, B, C, D): return LAUNCH<A, B, C, D>(a, s, fp32, variant) ? 1 : -1;

}  // namespace tf
